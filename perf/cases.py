"""The work that a user of this package has it do, as cases that can be timed.

Four kinds of user are behind the list: one who trains a small model (the "tiny" configuration of the benchmark: 256 wide, 4 x 256
tokens), where a pass is launches and host work; one who trains GPT-2 124M (768 wide, 12 x 1024 tokens); one who trains at GPT-2 XL
widths (1600 wide: a multiple of 32 but not of 128, with token counts that fill no tile); and one who runs the block-quantised
linear layer alone at the large square of the GEMM sweep.  Each calls the operators of `Linear` and `Nonlinear` directly, or whole
training steps through `gpt2.QGPT` and `optim.ClipAdamW`.

A case is a dict: "op" names the operator (or "train_step"), the other entries are its sizes and options.
"""
import math

import torch

from jetfire_int8training_b200 import Linear, Nonlinear, rng as sr_rng
from jetfire_int8training_b200.gpt2 import GPTConfig, QGPT
from jetfire_int8training_b200.optim import ClipAdamW

QB = 32
DEV = "cuda"
DTYPES = {"fp32": torch.float32, "fp16": torch.float16, "bf16": torch.bfloat16}


def listed():
    return [
        # ---- a small model: latency of one call
        # LayerNorm before the projections of the tiny model
        {"name": "layernorm_fwd_tiny", "op": "layernorm", "rows": 1024, "cols": 256, "backward": False},
        # its QKV projection; the attention takes the dequantised fp16 product
        {"name": "linear_fwd_tiny", "op": "linear_forward", "tokens": 1024, "cin": 256, "cout": 768, "quantised": False},
        # ---- GPT-2 124M, micro-batch 12 x 1024
        # first MLP projection, INT8 in and out
        {"name": "linear_fwd_124m", "op": "linear_forward", "tokens": 12288, "cin": 768, "cout": 3072, "quantised": True},
        # both gradients of the QKV projection; the training harness takes fp32 weight gradients
        {"name": "linear_bwd_124m", "op": "linear_backward", "tokens": 12288, "cin": 768, "cout": 2304, "quantised": True, "wgrad": "fp32"},
        # the fp16 gradient that leaves the attention enters the INT8 stream
        {"name": "quantize_sr_124m", "op": "quantize", "rows": 12288, "cols": 2304, "dtype": "fp16", "stochastic": True},
        {"name": "gelu_bwd_124m", "op": "gelu", "rows": 12288, "cols": 3072, "backward": True},
        # ---- GPT-2 XL widths
        {"name": "layernorm_bwd_xl", "op": "layernorm", "rows": 8192, "cols": 1600, "backward": True},
        # residual add of an odd number of sequences, with the statistics of the next LayerNorm
        {"name": "add_meanvar_xl_ragged", "op": "add", "rows": 3104, "cols": 1600, "dtype": "bf16", "meanvar": True},
        # attention output projection on a batch that fills no tile: dequantised dX, fp16 dW (the reference's output types)
        {"name": "linear_bwd_xl_ragged", "op": "linear_backward", "tokens": 7392, "cin": 1600, "cout": 1600, "quantised": False, "wgrad": "fp16"},
        # ---- the largest square that the linear-layer benchmark times
        {"name": "linear_fwd_8192", "op": "linear_forward", "tokens": 8192, "cin": 8192, "cout": 8192, "quantised": True},
        # ---- whole training steps: forward, backward, clipping, AdamW
        {"name": "train_step_tiny", "op": "train_step", "layers": 2, "width": 256, "heads": 4, "batch": 4, "seq": 256, "vocab": 4096},
        {"name": "train_step_124m", "op": "train_step", "layers": 12, "width": 768, "heads": 12, "batch": 12, "seq": 1024, "vocab": 50304},
    ]


def _log(rng, lo, hi, step):
    """A multiple of `step`, spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, step * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)))


def draw(rng):
    op = rng.choice(["linear_forward", "linear_backward", "quantize", "gelu", "layernorm", "add", "train_step"])
    if op in ("linear_forward", "linear_backward"):
        while True:
            case = {"op": op, "tokens": _log(rng, 256, 16384, 32), "cin": _log(rng, 128, 8192, 32), "cout": _log(rng, 128, 8192, 32),
                    "quantised": rng.random() < 0.6}
            # no larger than a third (forward) / a tenth (backward: two GEMMs) of the 8192 cube, which also bounds the outputs
            if case["tokens"] * case["cin"] * case["cout"] <= 8192 ** 3 // (3 if op == "linear_forward" else 10):
                break
        if op == "linear_backward":
            case["wgrad"] = rng.choice(["fp32", "fp16"])
        return case
    if op == "train_step":
        heads = rng.randint(2, 12)
        return {"op": op, "layers": rng.randint(1, 4), "width": heads * rng.choice([32, 64]), "heads": heads, "batch": rng.randint(1, 8),
                "seq": _log(rng, 64, 1024, 32), "vocab": _log(rng, 512, 16384, 8)}
    case = {"op": op, "rows": _log(rng, 256, 16384, 32), "cols": _log(rng, 128, 6400, 32)}
    if op == "quantize":
        case.update(dtype=rng.choice(["fp16", "bf16", "fp32"]), stochastic=rng.random() < 0.5)
    elif op == "add":
        case.update(dtype=rng.choice(["bf16", "fp32"]), meanvar=rng.random() < 0.5)
    else:
        case["backward"] = rng.random() < 0.5
    return case


# ------------------------------------------------------------------------------------------------------------ inputs
def _activation(g, rows, cols):
    """N(0,1) with 0.5 % of the channels scaled by 30: the outlier channels of a transformer's activations."""
    x = torch.randn(rows, cols, generator=g, device=DEV)
    channels = torch.randperm(cols, generator=g, device=DEV)[:max(1, round(0.005 * cols))]
    x[:, channels] *= 30.0
    return x


def _quantised(x):
    return Nonlinear.int8_quantize(x.to(torch.bfloat16), QB)


def _sweep_operand(g, rows, cols):
    """The GEMM sweep's operands: payloads uniform in [-127, 127], scales uniform in [1e-3, 1e-1]."""
    q = torch.randint(-127, 128, (rows, cols), generator=g, device=DEV, dtype=torch.int8)
    return q, (torch.rand(rows // QB, cols // QB, generator=g, device=DEV) * 0.099 + 1e-3).half()


def prepare(case, seed):
    op = case["op"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    key = (seed, 1)           # the key of this state's stochastic rounding
    s = {"case": case, "key": key}
    if op == "train_step":
        torch.manual_seed(seed)
        sr_rng.manual_seed(seed)
        cfg = GPTConfig(block_size=case["seq"], vocab_size=case["vocab"], n_layer=case["layers"], n_head=case["heads"], n_embd=case["width"])
        with torch.device(DEV):
            model = QGPT(cfg)
        params = list(model.parameters())
        s["model"] = model
        s["opt"] = ClipAdamW([([p for p in params if p.dim() >= 2], 0.1), ([p for p in params if p.dim() < 2], 0.0)], lr=6e-4,
                             betas=(0.9, 0.95), max_norm=1.0, loss_scale=2.0 ** 16)
        ids = torch.randint(0, cfg.vocab_size, (case["batch"], cfg.block_size + 1), generator=g, device=DEV)
        s["x"], s["y"] = ids[:, :-1].contiguous(), ids[:, 1:].contiguous()
        return s
    if op in ("linear_forward", "linear_backward"):
        tokens, cin, cout = case["tokens"], case["cin"], case["cout"]
        if min(tokens, cin, cout) >= 8192:
            s["x"], s["w"] = _sweep_operand(g, tokens, cin), _sweep_operand(g, cout, cin)
        else:
            s["x"], s["w"] = _quantised(_activation(g, tokens, cin)), _quantised(0.02 * torch.randn(cout, cin, generator=g, device=DEV))
        if op == "linear_backward":
            s["g"] = _quantised(1e-2 * torch.randn(tokens, cout, generator=g, device=DEV))
        return s
    rows, cols = case["rows"], case["cols"]
    if op == "quantize":
        s["x"] = (1e-2 * torch.randn(rows, cols, generator=g, device=DEV) if case["stochastic"] else _activation(g, rows, cols)).to(DTYPES[case["dtype"]])
        return s
    if op == "add":
        # forward: residual stream + branch output; backward: residual gradient + INT8 gradient
        wide = _activation(g, rows, cols) if case["meanvar"] else 1e-2 * torch.randn(rows, cols, generator=g, device=DEV)
        s["x"] = wide.to(DTYPES[case["dtype"]])
        s["q"] = _quantised((1.0 if case["meanvar"] else 1e-2) * torch.randn(rows, cols, generator=g, device=DEV))
        return s
    x = _activation(g, rows, cols)
    s["x"] = _quantised(x)
    if op == "layernorm":
        s["gamma"] = 1.0 + 0.1 * torch.randn(cols, generator=g, device=DEV)
        s["mean"], s["rstd"] = x.mean(-1), 1.0 / x.var(-1).sqrt()
    if case["backward"]:
        s["g"] = _quantised(1e-2 * torch.randn(rows, cols, generator=g, device=DEV))
    return s


# ------------------------------------------------------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    op = case["op"]
    if op == "linear_forward":
        return Linear.int8_linear_forward(*s["x"], *s["w"], case["quantised"], QB)
    if op == "linear_backward":
        return Linear.int8_linear_backward(*s["x"], *s["g"], None, *s["w"], QB, stochastic=True, dgrad_quantize=case["quantised"],
                                           sr_key=s["key"], wgrad_out_dtype=DTYPES[case["wgrad"]])
    if op == "quantize":
        if case["stochastic"]:
            return Nonlinear.int8_quantize(s["x"], QB, stochastic=True, sr_key=s["key"])
        return Nonlinear.int8_quantize(s["x"], QB)
    if op == "gelu":
        if case["backward"]:
            return Nonlinear.int8_gelu_backward(*s["x"], *s["g"], QB, stochastic=True, sr_key=s["key"])
        return Nonlinear.int8_gelu_forward(*s["x"], QB)
    if op == "layernorm":
        if case["backward"]:
            return Nonlinear.int8_layernorm_backward(*s["x"], *s["g"], s["gamma"], QB, s["mean"], s["rstd"], stochastic=True, sr_key=s["key"])
        y, sy, _ = Nonlinear.int8_layernorm_forward(*s["x"], s["gamma"], s["mean"], s["rstd"], QB)
        return y, sy
    if op == "add":
        if case["meanvar"]:
            return Nonlinear.int8_add_Ifp_Ig16_Ofp_Og_MeanVar(s["x"], *s["q"], QB)
        return Nonlinear.int8_add_Ifp_Ig16_Ofp_Og(s["x"], *s["q"], QB, stochastic=True, sr_key=s["key"])
    opt = s["opt"]
    loss = s["model"](s["x"], s["y"])
    opt.scale_loss(loss).backward()
    norm = opt.step()
    opt.zero_grad(set_to_none=True)
    return {"loss": loss.detach(), "norm": norm, "params": opt.flat, "exp_avg": opt.exp_avg, "exp_avg_sq": opt.exp_avg_sq}


# ------------------------------------------------------------------------------------------------------------ what a pass cannot do without
def _int8(rows, cols):
    """Payload and fp16 block scales of one block-quantised tensor."""
    return rows * cols + 2 * (rows // QB) * (cols // QB)


def work(case):
    op = case["op"]
    if op == "train_step":
        C, V, T = case["width"], case["vocab"], case["batch"] * case["seq"]
        matrices = 12 * case["layers"] * C * C + V * C                     # linear layers and LM head: forward, dX, dW
        attention = 7 * case["layers"] * T * case["seq"] * C               # causal: two products forward, five backward, half of each
        params = matrices + case["seq"] * C + (2 * case["layers"] + 1) * C
        # parameters and both moments read and written, gradients written and read, the LM head's bf16 logits through memory once
        return {"bytes": 32 * params + 4 * T * V, "flops": 6 * T * matrices + attention}
    if op in ("linear_forward", "linear_backward"):
        T, I, O = case["tokens"], case["cin"], case["cout"]
        if op == "linear_forward":
            return {"bytes": _int8(T, I) + _int8(O, I) + (_int8(T, O) if case["quantised"] else 2 * T * O), "flops": 2 * T * I * O}
        dx = _int8(T, I) if case["quantised"] else 2 * T * I
        return {"bytes": _int8(T, I) + _int8(O, I) + _int8(T, O) + dx + (4 if case["wgrad"] == "fp32" else 2) * I * O, "flops": 4 * T * I * O}
    R, N = case["rows"], case["cols"]
    wide = {"fp32": 4, "fp16": 2, "bf16": 2}.get(case.get("dtype"), 0) * R * N
    if op == "quantize":
        return {"bytes": wide + _int8(R, N), "flops": 4 * R * N}
    if op == "add":
        return {"bytes": wide + 4 * R * N + 2 * _int8(R, N) + (8 * R if case["meanvar"] else 0), "flops": 8 * R * N}
    tensors = 3 if case["backward"] else 2
    if op == "layernorm":
        return {"bytes": tensors * _int8(R, N) + 8 * R + 4 * N * (2 if case["backward"] else 1), "flops": (20 if case["backward"] else 8) * R * N}
    return {"bytes": tensors * _int8(R, N), "flops": 8 * R * N}


def tolerance(case):
    op = case["op"]
    if op == "train_step":
        # bf16 LM head and fp16 attention (whose backward is not deterministic) feeding stochastic rounding
        return {"rel": 1e-2}
    if op == "linear_backward":
        # dW: fp32 sums over the tokens in another order; rounded to fp16 on request.  dX is exact
        return {"rel": 1e-5, "max": 1e-3} if case["wgrad"] == "fp32" else {"rel": 1e-4, "max": 2e-3}
    if op == "layernorm" and case["backward"]:
        return {"rel": 1e-5, "max": 1e-3, "differ": 1e-6}   # fp32 sums over rows and slabs
    if op == "add" and case["meanvar"]:
        return {"rel": 1e-5, "max": 1e-3}                   # fp32 row sums
    return "exact"      # block-quantised payloads and scales, and products of them
