"""INT8-in / INT8-out nonlinear operators with the reference's names, signatures and return conventions
(Jetfire/Nonlinear/__init__.py:1-8 of thu-ml/Jetfire-INT8Training), executed by hand-written sm_100a kernels
through the C ABI in include/jetfire_b200.h.

Conventions kept from the reference: tensors are CUDA tensors, 2-D or 3-D (3-D inputs are flattened over the leading
dimensions and outputs get the leading batch dimension back); outputs are freshly allocated; everything runs on the
current stream; QB must be 32.

Extras not in the reference (keyword-only): `noise=` feeds an explicit fp32 noise tensor to a stochastic operator
(used to reproduce the reference's rounding bit for bit), `sr_key=(seed, offset)` pins the Philox key of one call.
`set_sr_noise("torch")` makes every stochastic operator draw its noise the way the reference does -- one fp32 tensor
`uniform_(-0.5, 0.5)` per call from torch's CUDA generator (Jetfire/Nonlinear/quantize.py:143-144, gelu_bwd.py:192,
layernorm.py:493, add.py:185) -- so that a run seeded with `torch.manual_seed` rounds exactly like the reference run with the
same seed, at the price of writing and reading 4 bytes of noise per element; the default "philox" generates 16 noise bits per
element inside the kernel.
"""
import torch

from .. import rng
from .._lib import host

__all__ = [
    "int8_quantize", "int8_quantize_many", "int8_quantize_parts", "int8_quantize_transpose", "int8_transpose", "int8_dequantize",
    "int8_gelu_forward", "int8_gelu_backward", "int8_layernorm_forward", "int8_layernorm_backward",
    "int8_add_Ifp_Ig16_Ofp_Og", "int8_add_Ifp_Ig16_Ofp_Og_MeanVar", "int8_add_out", "set_sr_noise",
]

_SR_NOISE = "philox"


def set_sr_noise(mode):
    """"philox": in-kernel Philox4x32-10 keyed by rng.next_key() (default).  "torch": the reference's noise stream."""
    global _SR_NOISE
    if mode not in ("philox", "torch"):
        raise ValueError("sr noise mode is 'philox' or 'torch'")
    previous, _SR_NOISE = _SR_NOISE, mode
    return previous


def _qb(QB):
    if QB != 32:
        raise ValueError("only the 32x32 quantisation block of the reference recipe is implemented")


def _sr(stochastic, noise, sr_key, like):
    """(noise, seed, offset) of one stochastic call."""
    if not stochastic or noise is not None:
        return noise, 0, 0
    if sr_key is None:
        if _SR_NOISE == "torch" and like.is_cuda:
            return torch.empty(like.shape, dtype=torch.float32, device=like.device).uniform_(-0.5, 0.5), 0, 0
        sr_key = rng.next_key()
    return None, sr_key[0], sr_key[1]


def int8_quantize(x, QB, stochastic=False, *, noise=None, sr_key=None):
    """Jetfire/Nonlinear/quantize.py:128-164.  Returns (q int8, scale fp16)."""
    _qb(QB)
    return host().quantize(x, False, False, stochastic, *_sr(stochastic, noise, sr_key, x))


def int8_quantize_many(tensors, QB):
    """Round-to-nearest int8_quantize of several 2-D tensors (same dtype and device) with one kernel launch per 8 tensors: the
    weight matrices that the reference quantises one by one at the start of every forward pass (INT8_GPT2/qmodel.py:92, 139,
    199-200).  Returns [(q, scale), ...], bit-identical to int8_quantize on each tensor."""
    _qb(QB)
    return host().quantize_many(tensors)


def int8_quantize_parts(parts, QB, stochastic=False, *, sr_key=None):
    """int8_quantize of torch.cat(parts, -1) for one to four parts of one shape and dtype, without the concatenation (the gradients of
    Q, K and V in front of the QKV projection's backward pass)."""
    _qb(QB)
    if stochastic and sr_key is None and _SR_NOISE == "torch":
        return int8_quantize(torch.cat(tuple(parts), dim=-1), QB, stochastic=True)
    return host().quantize_parts(parts, stochastic, *_sr(stochastic, None, sr_key, parts[0]))


def int8_quantize_transpose(x, QB, stochastic=False, transpose_output_2d=False, *, noise=None, sr_key=None):
    """Jetfire/Nonlinear/quantize_transpose.py:131-171.  Returns (q, scale, q^T)."""
    _qb(QB)
    return host().quantize(x, True, transpose_output_2d, stochastic, *_sr(stochastic, noise, sr_key, x))


def int8_transpose(x, transpose_output_2d=False):
    """Jetfire/Nonlinear/transpose.py:69-97."""
    return host().transpose(x, transpose_output_2d)


def int8_dequantize(x, s_x, QB):
    """Jetfire/Nonlinear/dequantize.py:86-116.  Returns fp32."""
    _qb(QB)
    return host().dequantize(x, s_x)


def int8_gelu_forward(x, s_x, QB):
    """Jetfire/Nonlinear/gelu_fwd.py:128-162."""
    _qb(QB)
    return host().gelu_forward(x, s_x)


def int8_gelu_backward(x, s_x, g, s_g, QB, stochastic=False, *, noise=None, sr_key=None):
    """Jetfire/Nonlinear/gelu_bwd.py:173-215."""
    _qb(QB)
    return host().gelu_backward(x, s_x, g, s_g, stochastic, *_sr(stochastic, noise, sr_key, x))


def int8_layernorm_forward(x, sx, weight, mean, rstd, QB, eps=1e-6):
    """Jetfire/Nonlinear/layernorm.py:430-465.  mean / rstd are inputs; no bias; eps is accepted and unused,
    exactly as in the reference.  Returns (y, sy, (mean, rstd))."""
    _qb(QB)
    y, sy = host().layernorm_forward(x, sx, weight, mean, rstd)
    return y, sy, (mean, rstd)


def int8_layernorm_backward(x, sx, g, sg, w, QB, m, v, stochastic=False, eps=1e-6, *, noise=None, sr_key=None):
    """Jetfire/Nonlinear/layernorm.py:467-526.  Returns (dx int8, sdx fp16, dw).  The two row reductions of dx are taken
    over 128-column slabs, as the reference's kernel does."""
    _qb(QB)
    return host().layernorm_backward(x, sx, g, sg, w, m, v, stochastic, *_sr(stochastic, noise, sr_key, x))


def int8_add_Ifp_Ig16_Ofp_Og(x1, x2, s_x2, QB, stochastic=False, *, noise=None, sr_key=None):
    """Jetfire/Nonlinear/add.py:164-211.  Returns (y1 fp32, y2 int8, s_y2 fp16)."""
    _qb(QB)
    return host().add(x1, x2, s_x2, False, False, stochastic, *_sr(stochastic, noise, sr_key, x1))


def int8_add_Ifp_Ig16_Ofp_Og_MeanVar(x1, x2, s_x2, QB):
    """Jetfire/Nonlinear/add_mean_var.py:179-231.  Returns (y1 fp32, y2 int8, s_y2 fp16, mean, rstd)."""
    _qb(QB)
    return host().add(x1, x2, s_x2, True, False, False, None, 0, 0)


def int8_add_out(x1, x2, s_x2, QB, out_dtype, mean_var=False, stochastic=False, *, sr_key=None):
    """The residual adds with y1 in `out_dtype` (fp32, or bf16 rounded once from the fp32 sum): int8_add_Ifp_Ig16_Ofp_Og or, with
    mean_var, int8_add_Ifp_Ig16_Ofp_Og_MeanVar, followed by y1.to(out_dtype) -- in one pass."""
    _qb(QB)
    if out_dtype not in (torch.float32, torch.bfloat16):
        raise TypeError("int8_add_out writes fp32 or bf16")
    if mean_var and stochastic:
        raise ValueError("the add with row statistics rounds to nearest")
    return host().add(x1, x2, s_x2, mean_var, out_dtype == torch.bfloat16, stochastic, *_sr(stochastic, None, sr_key, x1))
