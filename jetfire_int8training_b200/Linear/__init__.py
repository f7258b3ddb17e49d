"""The INT8 linear layer with the reference's function names and conventions
(Jetfire/Linear/linear_fwd.py:4-32 and linear_bwd.py:4-28 of thu-ml/Jetfire-INT8Training).

Differences that do not change results: scale tensors are read in their natural [rows/32, cols/32] layout (the
reference makes transposed copies), W and dY are read in place by the GEMMs (the `G8T` argument, the materialised
transpose of dY, is accepted and ignored), and the "dequantised output" variants are produced by the GEMM epilogue
instead of two torch kernels.  `operand_scratch` is accepted and has no effect: every GEMM reads its int8 operands in place.
"""
import torch

from .. import rng
from .._lib import host

__all__ = ["int8_linear_forward", "int8_linear_backward", "int8_linear_wgrad"]


def int8_linear_forward(X8_3D, SX16_3D, W8, SW16, output_quantized, B, *, operand_scratch=None):
    """Y = X W^T.  X8 int8 [..., K] with scales [..., K/32] (leading dims flattened), W8 int8 [N, K], SW16 [N/32, K/32].
    Returns (Y8, SY16) when output_quantized, else the dequantised fp16 tensor fp16(q) * scale."""
    if B != 32:
        raise ValueError("only the 32x32 quantisation block of the reference recipe is implemented")
    return host().linear_forward(X8_3D, SX16_3D, W8, SW16, output_quantized)


def int8_linear_wgrad(X8, SX, G8, SG, out_dtype=torch.float16, split_k=0, operand_scratch=None):
    """dW[Cout, Cin] = dY^T X with dY = G8 [T, Cout], X8 [T, Cin] (2-D, natural layouts, read in place)."""
    return host().linear_wgrad(X8, SX, G8, SG, out_dtype == torch.float16, split_k)


def int8_linear_backward(X8_3D, SX16_3D, G8_3D, SG16_3D, G8T, W8, SW16, B, stochastic=True, dgrad_quantize=True, *,
                         sr_key=None, noise=None, wgrad_split_k=0, wgrad_out_dtype=torch.float16, operand_scratch=None):
    """dX = dY W (block-quantised with stochastic rounding, or dequantised fp16 when dgrad_quantize is False) and
    dW = dY^T X (dense fp16).  Returns (GX8, GSX16, GW) or (GX16, GW), as the reference does.
    The reference ignores `stochastic` and always rounds stochastically; here stochastic=False rounds to nearest.
    `wgrad_out_dtype=torch.float32` (extra) returns dW in fp32 instead of the reference's fp16."""
    if B != 32:
        raise ValueError("only the 32x32 quantisation block of the reference recipe is implemented")
    seed = offset = 0
    if stochastic and noise is None:
        seed, offset = sr_key if sr_key is not None else rng.next_key()
    return host().linear_backward(X8_3D, SX16_3D, G8_3D, SG16_3D, W8, SW16, dgrad_quantize, wgrad_out_dtype == torch.float16, wgrad_split_k,
                                  stochastic, noise, seed, offset)
