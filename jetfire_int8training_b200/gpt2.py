"""GPT-2 with the Jetfire INT8 data flow, as the caller of the hot path.

This is the integration harness for the operators of this package: a nanoGPT-shaped decoder (no biases) whose linear layers,
LayerNorms, GELU and residual adds run on the per-block INT8 operators, following the data flow of the reference's quantised
model (INT8_GPT2/qmodel.py:35-362): between blocks the activations travel as (fp residual, int8 payload, fp16 block scales,
row mean, row rstd); in the backward pass the gradient travels as (fp residual gradient, int8 payload, fp16 scales) with
stochastic rounding.  int8 payloads cross autograd boundaries viewed as float8_e4m3fn, as in the reference, because autograd
only tracks floating tensors.  Attention itself (scaled-dot-product), the embedding, the final LayerNorm and the LM head stay
in floating point, as they do in the reference.

Differences from the reference's module, none of which touch the operators' semantics: weight gradients are produced in fp32
(the reference's fp16 overflows under its 2^24 loss scale), the materialised dY^T copies are not made (the GEMMs read dY
in place), and the weight matrices are quantised eight per kernel launch at the start of the forward pass.
"""
import contextlib
import math
from dataclasses import dataclass

import torch
import torch.nn as nn
from torch.nn import functional as F

from . import Linear as L
from . import Nonlinear as NL
from ._lib import host
from .lm_loss import lm_cross_entropy

QB = 32
F8 = torch.float8_e4m3fn


@dataclass
class GPTConfig:
    block_size: int = 1024
    vocab_size: int = 50304
    n_layer: int = 12
    n_head: int = 12
    n_embd: int = 768


def _f8(t):
    return t.view(F8)


def quantized_weight(w):
    """(int8 payload, fp16 scales) of a weight matrix for the forward pass that is running: the pair that
    quantise_weights() stored on the parameter at the start of this pass, else a fresh quantisation."""
    hit = getattr(w, "_jf_q", None)
    if hit is not None:
        return hit
    return NL.int8_quantize(w.detach(), QB)


def quantise_weights(weights, reuse=False):
    """Quantise the weight matrices of a model for one forward pass, eight tensors per kernel launch, and store the results
    where quantized_weight finds them (the reference quantises each weight where it is used, INT8_GPT2/qmodel.py:92, 139,
    199-200: 4 * n_layer launches, each smaller than one wave of the GPU at GPT-2 124M sizes).

    `reuse=True` keeps the quantisations of the previous pass.  Only the caller knows that the weights have not changed since --
    the further micro-steps of a gradient-accumulation step -- and has to say so: a parameter's version counter is NOT a safe
    key, because fused optimisers (torch.optim.AdamW(fused=True)) update parameters without advancing it."""
    if reuse and all(getattr(w, "_jf_q", None) is not None for w in weights):
        return
    for w, pair in zip(weights, NL.int8_quantize_many([w.detach() for w in weights], QB)):
        w._jf_q = pair


def _i8(t):
    return t.view(torch.int8)


# A model's pass is one autograd node per part: embedding, each block, the final LayerNorm, the LM head.  With a node for each group of
# operators and torch's views, splits and casts between them, a 2-layer 256-wide model spent 2.3 ms per step on the host around 0.6 ms of
# device work, and GPT-2 124M ~0.7 ms on narrowing copies of the residual stream and concatenations of the QKV gradient.  A node per block (not one for all) keeps the gradients of a block available to DDP while the earlier ones run.


def _add(x1, q, s, dtype, mean_var=False, stochastic=False):
    """Residual add whose fp output the residual stream carries in `dtype` (an operator module without the one-pass form: add, then cast)."""
    fused = getattr(NL, "int8_add_out", None)
    if fused is not None:
        return fused(x1, q, s, QB, dtype, mean_var=mean_var, stochastic=stochastic)
    if mean_var:
        y, *rest = NL.int8_add_Ifp_Ig16_Ofp_Og_MeanVar(x1, q, s, QB)
    else:
        y, *rest = NL.int8_add_Ifp_Ig16_Ofp_Og(x1, q, s, QB, stochastic=stochastic)
    return (y.to(dtype), *rest)


def _quantise_parts(parts):
    """Stochastically rounded block quantisation of the concatenated parts."""
    fused = getattr(NL, "int8_quantize_parts", None)
    if fused is not None:
        return fused(parts, QB, stochastic=True)
    return NL.int8_quantize(torch.cat(parts, dim=-1), QB, stochastic=True)


def _attention(qkv, n_head):
    B, T, C = qkv.shape[0], qkv.shape[1], qkv.shape[2] // 3
    q, k, v = [t.view(B, T, n_head, C // n_head).transpose(1, 2) for t in qkv.split(C, dim=2)]
    return F.scaled_dot_product_attention(q, k, v, is_causal=True).transpose(1, 2).contiguous().view(B, T, C)


class _Embed(torch.autograd.Function):
    """Token + position embedding and the entry of the INT8 stream: quantise their sum, row mean and 1 / std (reference:
    QModel_bgn_func, qmodel.py:309-326).  `tied` carries the LM head's gradient of the shared token matrix from the head's backward
    pass, which always runs first, so that the two are added without a widened copy of either."""

    @staticmethod
    def forward(ctx, idx, wte, wpe, tied):
        x, mean, rstd = host().embed_forward(idx, wte, wpe)
        qx, sx = NL.int8_quantize(x, QB)
        ctx.save_for_backward(idx)
        ctx.sizes, ctx.tied = (wte.shape[0], wpe.shape[0]), tied
        ctx.set_materialize_grads(False)
        ctx.mark_non_differentiable(mean, rstd)
        return x, _f8(qx), sx, mean, rstd

    @staticmethod
    def backward(ctx, g, qg, sg, _m, _r):
        idx, = ctx.saved_tensors
        dwte, dwpe = host().embed_backward(idx, g, ctx.tied.pop("dw", None), *ctx.sizes)
        return None, dwte, dwpe, None


class _Block(torch.autograd.Function):
    """One transformer block, forward and backward over the operators (reference: _QAttentionPart1 / _QAttentionPart2 / _QMLPResidual,
    qmodel.py:86-267): LayerNorm + QKV projection (dequantised fp16) -> attention -> quantise -> output projection + residual add with row
    statistics -> LayerNorm + FC1 + GELU + FC2 + residual add with row statistics.  In the backward pass the gradient travels as (fp
    residual gradient in the residual's type, int8 payload, scales)."""

    @staticmethod
    def forward(ctx, x, qx, sx, mean, rstd, ln1, w_qkv, w_proj, ln2, w1, w2, n_head):
        qx = _i8(qx)
        (qwq, swq), (qwp, swp), (qw1, sw1), (qw2, sw2) = [quantized_weight(w) for w in (w_qkv, w_proj, w1, w2)]
        qn, sn, _ = NL.int8_layernorm_forward(qx, sx, ln1, mean, rstd, QB)
        qkv = L.int8_linear_forward(qn, sn, qwq, swq, False, QB)
        fused = host().attention_forward(qkv, n_head)
        if fused is not None:
            y, max_q, max_k, *att = fused
            ctx.graph = None
        else:                                        # another attention backend: through its own autograd graph
            with torch.enable_grad():
                leaf = qkv.detach().requires_grad_()
                out = _attention(leaf, n_head)
            y, max_q, max_k, att = out.detach(), 0, 0, []
            ctx.graph = (leaf, out)
        qy, sy = NL.int8_quantize(y, QB)
        qo, so = L.int8_linear_forward(qy, sy, qwp, swp, True, QB)
        x1, qx1, sx1, mean1, rstd1 = NL.int8_add_Ifp_Ig16_Ofp_Og_MeanVar(x.contiguous(), qo, so, QB)
        qn1, sn1, _ = NL.int8_layernorm_forward(qx1, sx1, ln2, mean1, rstd1, QB)
        qh, sh = L.int8_linear_forward(qn1, sn1, qw1, sw1, True, QB)
        qa, sa = NL.int8_gelu_forward(qh, sh, QB)
        qo, so = L.int8_linear_forward(qa, sa, qw2, sw2, True, QB)
        x2, qx2, sx2, mean2, rstd2 = _add(x1, qo, so, torch.bfloat16, mean_var=True)
        ctx.save_for_backward(qx, sx, mean, rstd, ln1, qn, sn, qwq, swq, qkv, qy, sy, qwp, swp, qx1, sx1, mean1, rstd1, ln2, qn1, sn1, qw1, sw1,
                              qh, sh, qa, sa, qw2, sw2, *att)
        ctx.meta = (n_head, max_q, max_k, x.dtype)
        ctx.set_materialize_grads(False)
        ctx.mark_non_differentiable(mean2, rstd2)
        return x2, _f8(qx2), sx2, mean2, rstd2

    @staticmethod
    def backward(ctx, fpg, qg, sg, _m, _r):
        (qx, sx, mean, rstd, ln1, qn, sn, qwq, swq, qkv, qy, sy, qwp, swp, qx1, sx1, mean1, rstd1, ln2, qn1, sn1, qw1, sw1,
         qh, sh, qa, sa, qw2, sw2, *att) = ctx.saved_tensors
        n_head, max_q, max_k, dtype = ctx.meta
        qg, sg, dw2 = _linear_backward(qa, sa, _i8(qg), sg, qw2, sw2)
        qg, sg = NL.int8_gelu_backward(qh, sh, qg, sg, QB, stochastic=True)
        qg, sg, dw1 = _linear_backward(qn1, sn1, qg, sg, qw1, sw1)
        qg, sg, dln2 = NL.int8_layernorm_backward(qx1, sx1, qg, sg, ln2, QB, mean1, rstd1, stochastic=True)
        fpg, qg, sg = _add(fpg.contiguous(), qg, sg, dtype, stochastic=True)
        g16, dwp = _linear_backward(qy, sy, qg, sg, qwp, swp, dgrad_quantize=False)
        if ctx.graph is None:
            gq, gk, gv = host().attention_backward(g16, qkv, n_head, max_q, max_k, *att)
            qg, sg = _quantise_parts([gq, gk, gv])
        else:
            leaf, out = ctx.graph
            gqkv, = torch.autograd.grad(out, leaf, g16, retain_graph=True)
            qg, sg = NL.int8_quantize(gqkv.contiguous(), QB, stochastic=True)
        qg, sg, dwq = _linear_backward(qn, sn, qg, sg, qwq, swq)
        qg, sg, dln1 = NL.int8_layernorm_backward(qx, sx, qg, sg, ln1, QB, mean, rstd, stochastic=True)
        fpg, qg, sg = _add(fpg, qg, sg, dtype, stochastic=True)
        return fpg, _f8(qg), sg, None, None, dln1, dwq, dwp, dln2, dw1, dw2, None


class _Final(torch.autograd.Function):
    """Exit of the INT8 stream and final LayerNorm, whose bf16 output is what the LM head reads: in the backward pass the fp gradient is
    block-quantised with stochastic rounding and seeds the INT8 gradient stream (reference: QModel_end_func, qmodel.py:343-362)."""

    @staticmethod
    def forward(ctx, x, qx, sx, ln_f):
        y, xf, mean, rstd = host().final_norm_forward(x, ln_f, 1e-5)
        ctx.save_for_backward(xf, ln_f, mean, rstd)
        ctx.narrow = x.dtype == torch.bfloat16
        return y

    @staticmethod
    def backward(ctx, gy):
        xf, ln_f, mean, rstd = ctx.saved_tensors
        g, dln = host().final_norm_backward(gy, xf, ln_f, mean, rstd, ctx.narrow)
        qg, sg = NL.int8_quantize(g, QB, stochastic=True)
        return g, _f8(qg), sg, dln


class _Head(torch.autograd.Function):
    """LM head: bf16 logits = x W^T on the shared token matrix.  Its bf16 weight gradient is handed to _Embed's backward pass through
    `tied`."""

    @staticmethod
    def forward(ctx, x, wte, tied):
        x2, w = x.reshape(-1, x.shape[-1]), wte.to(torch.bfloat16)
        ctx.save_for_backward(x2, w)
        ctx.shape, ctx.tied = x.shape, tied
        return torch.mm(x2, w.t()).view(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, g):
        x2, w = ctx.saved_tensors
        g2 = g.reshape(-1, w.shape[0]).to(torch.bfloat16)
        ctx.tied["dw"] = torch.mm(g2.t(), x2)
        return torch.mm(g2, w).view(ctx.shape), None, None


def _linear_backward(qx, sx, qg, sg, qw, sw, dgrad_quantize=True):
    """Input gradient (stochastically rounded INT8, or dequantised fp16) and fp32 weight gradient of one linear layer."""
    return L.int8_linear_backward(qx, sx, qg, sg, None, qw, sw, QB, stochastic=True, dgrad_quantize=dgrad_quantize,
                                  wgrad_out_dtype=torch.float32)


class Block(nn.Module):
    def __init__(self, cfg):
        super().__init__()
        C = cfg.n_embd
        self.n_head = cfg.n_head
        self.ln_1 = nn.Parameter(torch.ones(C))
        self.c_attn = nn.Parameter(torch.empty(3 * C, C))
        self.c_proj = nn.Parameter(torch.empty(C, C))
        self.ln_2 = nn.Parameter(torch.ones(C))
        self.c_fc = nn.Parameter(torch.empty(4 * C, C))
        self.c_proj2 = nn.Parameter(torch.empty(C, 4 * C))

    def forward(self, x, qx, sx, mean, rstd):
        return _Block.apply(x, qx, sx, mean, rstd, self.ln_1, self.c_attn, self.c_proj, self.ln_2, self.c_fc, self.c_proj2, self.n_head)


class QGPT(nn.Module):
    def __init__(self, cfg: GPTConfig):
        super().__init__()
        self.cfg = cfg
        self.wte = nn.Embedding(cfg.vocab_size, cfg.n_embd)
        self.wpe = nn.Embedding(cfg.block_size, cfg.n_embd)
        self.blocks = nn.ModuleList([Block(cfg) for _ in range(cfg.n_layer)])
        self.ln_f = nn.Parameter(torch.ones(cfg.n_embd))
        std = 0.02
        nn.init.normal_(self.wte.weight, 0.0, std)
        nn.init.normal_(self.wpe.weight, 0.0, std)
        for b in self.blocks:
            nn.init.normal_(b.c_attn, 0.0, std)
            nn.init.normal_(b.c_fc, 0.0, std)
            nn.init.normal_(b.c_proj, 0.0, std / math.sqrt(2 * cfg.n_layer))
            nn.init.normal_(b.c_proj2, 0.0, std / math.sqrt(2 * cfg.n_layer))

    def num_params(self):
        return sum(p.numel() for p in self.parameters()) - self.wpe.weight.numel()

    def forward(self, idx, targets, reuse_quantised_weights=False):
        """`reuse_quantised_weights`: the weights have not changed since the previous forward pass (micro-steps 2.. of a
        gradient-accumulation step), keep their quantisations."""
        quantise_weights([w for b in self.blocks for w in (b.c_attn, b.c_proj, b.c_fc, b.c_proj2)], reuse=reuse_quantised_weights)
        tied = {}
        with torch.autocast("cuda", enabled=False) if torch.is_autocast_enabled("cuda") else contextlib.nullcontext():
            state = _Embed.apply(idx, self.wte.weight, self.wpe.weight, tied)
            for blk in self.blocks:
                state = blk(*state)
            x, qx, sx, _, _ = state
            logits = _Head.apply(_Final.apply(x, qx, sx, self.ln_f), self.wte.weight, tied)
        return lm_cross_entropy(logits, targets)       # no fp32 copy of the [tokens, vocab] logits; gradient written in place
