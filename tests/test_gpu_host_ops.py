"""GPU: the operators' native host path (csrc/host_ops.cpp): ranks, non-contiguous inputs, float8 views of payloads, dtypes outside the
three native ones and refused arguments give what the contiguous 2-D call gives."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from jetfire_int8training_b200 import Linear, Nonlinear
    return Nonlinear, Linear


def _x(*shape, dtype=torch.bfloat16):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(sum(shape))).to(dtype).to(DEV)


@pytest.mark.parametrize("lead", [(96,), (3, 32), (2, 64), (1, 32), (2, 2, 32)])
def test_leading_dimensions(ops, lead):
    NL, L = ops
    x = _x(*lead, 160)
    flat = x.reshape(-1, 160)
    q2, s2 = NL.int8_quantize(flat, 32)
    q, s = NL.int8_quantize(x, 32)
    shape = (lambda r, c: (r, c)) if len(lead) == 1 else (lambda r, c: (lead[0], r // lead[0], c))
    assert q.shape == shape(flat.shape[0], 160) and s.shape == shape(flat.shape[0] // 32, 5)
    assert torch.equal(q.reshape(q2.shape), q2) and torch.equal(s.reshape(s2.shape), s2)
    w = torch.randint(-127, 128, (64, 160), device=DEV, dtype=torch.int8)
    sw = torch.full((2, 5), 0.01, device=DEV, dtype=torch.float16)
    y2, sy2 = L.int8_linear_forward(q2, s2, w, sw, True, 32)
    y, sy = L.int8_linear_forward(q, s, w, sw, True, 32)
    assert y.shape == (*q.shape[:-1], 64) and sy.shape == (*s.shape[:-1], 2)
    assert torch.equal(y.reshape(y2.shape), y2) and torch.equal(sy.reshape(sy2.shape), sy2)
    f8 = lambda t: t.view(torch.float8_e4m3fn)
    a = NL.int8_add_Ifp_Ig16_Ofp_Og_MeanVar(x, f8(q), s, 32)
    b = NL.int8_add_Ifp_Ig16_Ofp_Og_MeanVar(flat, q2, s2, 32)
    assert all(u.numel() == v.numel() and torch.equal(u.reshape(v.shape), v) for u, v in zip(a, b))
    assert a[3].shape == ((flat.shape[0],) if len(lead) == 1 else (lead[0], flat.shape[0] // lead[0]))


def test_non_contiguous_and_other_dtypes(ops):
    NL, _ = ops
    x = _x(160, 96).t()
    for a, b in zip(NL.int8_quantize(x, 32), NL.int8_quantize(x.contiguous(), 32)):
        assert torch.equal(a, b)
    d = _x(64, 96, dtype=torch.float64)
    for a, b in zip(NL.int8_quantize(d, 32), NL.int8_quantize(d.float(), 32)):
        assert torch.equal(a, b)


def test_refused_arguments(ops):
    NL, L = ops
    from jetfire_int8training_b200._lib import JetfireError
    x = _x(64, 96)
    q, s = NL.int8_quantize(x, 32)
    with pytest.raises(JetfireError):
        NL.int8_quantize(_x(48, 96), 32)
    with pytest.raises(RuntimeError):
        NL.int8_gelu_forward(q, s.cpu(), 32)
    with pytest.raises(RuntimeError):
        NL.int8_gelu_forward(x, s, 32)                    # not a payload
    with pytest.raises(AssertionError):
        NL.int8_add_Ifp_Ig16_Ofp_Og(_x(64, 64), q, s, 32)
    with pytest.raises(RuntimeError):
        L.int8_linear_backward(q, s, q, s, None, q, s, 32)   # dY's columns are not W's rows
    with pytest.raises(TypeError):
        NL.int8_quantize(None, 32)
