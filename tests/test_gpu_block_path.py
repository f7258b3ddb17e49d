"""GPU: what the GPT-2 caller's one-node-per-block pass is made of: the native calls around the INT8 stream, the quantisation of column
parts, the residual add with a bf16 output, and the attention, against autograd through torch's modules or the existing operators."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def H():
    from jetfire_int8training_b200._lib import host
    return host()


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


@pytest.mark.parametrize("B,T,P,C,V", [(1, 1, 1, 32, 2), (3, 5, 7, 32, 11), (4, 96, 128, 768, 1000)])
def test_embedding_and_final_norm_are_the_autograd_operators(H, B, T, P, C, V):
    """Bit for bit: the native calls against autograd through torch's modules, the head's bf16 gradient included."""
    g = _gen(C)
    wte = torch.randn(V, C, generator=g, device=DEV).requires_grad_()
    wpe = torch.randn(P, C, generator=g, device=DEV).requires_grad_()
    idx = torch.randint(0, V, (B, T), generator=g, device=DEV)
    want = F.embedding(idx, wte) + F.embedding(torch.arange(T, device=DEV), wpe)
    x, mean, rstd = H.embed_forward(idx, wte, wpe)
    assert torch.equal(x, want) and torch.equal(mean, want.mean(-1)) and torch.equal(rstd, 1.0 / want.var(-1).sqrt())
    gr = torch.randn(B, T, C, generator=g, device=DEV)
    head = torch.randn(V, C, generator=g, device=DEV).bfloat16()
    want.backward(gr)
    dwte, dwpe = H.embed_backward(idx, gr, head, V, P)
    assert torch.equal(dwte, wte.grad + head.float()) and torch.equal(dwpe, wpe.grad)
    for narrow in (False, True):
        h = want.detach().to(torch.bfloat16 if narrow else torch.float32).requires_grad_()
        w = (1 + 0.1 * torch.randn(C, generator=g, device=DEV)).requires_grad_()
        ref = F.layer_norm(h.float(), (C,), w, None, 1e-5).bfloat16()
        dy = torch.randn(B, T, C, generator=g, device=DEV).bfloat16()
        ref.backward(dy)
        y, xf, m, r = H.final_norm_forward(h, w, 1e-5)
        dx, dw = H.final_norm_backward(dy, xf, w, m, r, narrow)
        assert torch.equal(y, ref) and torch.equal(dx, h.grad) and torch.equal(dw, w.grad)
    with pytest.raises(ValueError):
        H.embed_forward(torch.zeros(1, P + 1, dtype=torch.int64, device=DEV), wte, wpe)


@pytest.mark.parametrize("parts,M,cols", [(1, 32, 32), (2, 64, 96), (3, 96, 160), (4, 32, 32), (3, 2048, 768)])
@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16, torch.float32])
def test_quantize_parts_equals_quantize_of_the_concatenation(parts, M, cols, dt):
    from jetfire_int8training_b200 import Nonlinear as NL
    g = _gen(parts + M)
    xs = [(1e-2 * torch.randn(M, cols, generator=g, device=DEV)).to(dt) for _ in range(parts)]
    for kw in ({}, {"stochastic": True, "sr_key": (7, 3)}):
        for a, b in zip(NL.int8_quantize_parts(xs, 32, **kw), NL.int8_quantize(torch.cat(xs, 1), 32, **kw)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dt", [torch.float32, torch.float16, torch.bfloat16])
def test_add_with_bf16_output(dt):
    from jetfire_int8training_b200 import Nonlinear as NL
    g = _gen(5)
    x = torch.randn(3, 64, 160, generator=g, device=DEV).to(dt)
    q, s = NL.int8_quantize(torch.randn(3, 64, 160, generator=g, device=DEV), 32)
    key = (5, 9)
    pairs = [(NL.int8_add_out(x, q, s, 32, torch.bfloat16, stochastic=True, sr_key=key), NL.int8_add_Ifp_Ig16_Ofp_Og(x, q, s, 32, stochastic=True, sr_key=key)),
             (NL.int8_add_out(x, q, s, 32, torch.bfloat16), NL.int8_add_Ifp_Ig16_Ofp_Og(x, q, s, 32)),
             (NL.int8_add_out(x, q, s, 32, torch.bfloat16, mean_var=True), NL.int8_add_Ifp_Ig16_Ofp_Og_MeanVar(x, q, s, 32))]
    for got, want in pairs:
        assert torch.equal(got[0], want[0].to(torch.bfloat16))
        assert all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))


@pytest.mark.parametrize("B,T,heads,hs", [(2, 64, 2, 32), (1, 96, 3, 64), (2, 33, 1, 64), (1, 32, 2, 128)])
def test_block_attention_matches_scaled_dot_product_attention(H, B, T, heads, hs):
    """The direct call of the fused operator (where the dispatcher picks it) against autograd through scaled_dot_product_attention."""
    from jetfire_int8training_b200.gpt2 import _attention
    g = _gen(T)
    qkv = torch.randn(B, T, 3 * heads * hs, generator=g, device=DEV).half()
    gy = torch.randn(B, T, heads * hs, generator=g, device=DEV).half()
    leaf = qkv.clone().requires_grad_()
    want = _attention(leaf, heads)
    want.backward(gy)
    fused = H.attention_forward(qkv, heads)
    if fused is None:
        pytest.skip("another backend is chosen at this shape")
    y, mq, mk, *att = fused
    torch.testing.assert_close(y, want.detach(), rtol=2e-3, atol=2e-3)
    grads = torch.cat(H.attention_backward(gy, qkv, heads, mq, mk, *att), -1)
    torch.testing.assert_close(grads, leaf.grad, rtol=1e-2, atol=1e-2)


def test_model_runs_through_another_attention_backend():
    """The block's fallback (an autograd graph of its own around the attention) gives the loss and gradients of the direct call."""
    from torch.nn.attention import SDPBackend, sdpa_kernel
    from jetfire_int8training_b200 import rng
    from jetfire_int8training_b200.gpt2 import GPTConfig, QGPT
    torch.manual_seed(0)
    model = QGPT(GPTConfig(block_size=64, vocab_size=512, n_layer=2, n_head=2, n_embd=128)).to(DEV)
    ids = torch.randint(0, 512, (2, 65), device=DEV)
    out = []
    for ctx in ([SDPBackend.MATH], [SDPBackend.CUDNN_ATTENTION, SDPBackend.FLASH_ATTENTION, SDPBackend.EFFICIENT_ATTENTION, SDPBackend.MATH]):
        rng.manual_seed(0)
        model.zero_grad(set_to_none=True)
        with sdpa_kernel(ctx):
            loss = model(ids[:, :-1], ids[:, 1:])
            (loss * 1024).backward()
        out.append((float(loss), {n: p.grad.clone() for n, p in model.named_parameters()}))
    assert abs(out[0][0] - out[1][0]) < 1e-3 * out[0][0]
    for n in out[0][1]:
        a, b = out[0][1][n].flatten(), out[1][1][n].flatten()
        assert float(torch.dot(a, b) / (a.norm() * b.norm())) > 0.99, n


@pytest.mark.parametrize("n", [8, 2040, 2048, 2056, 512 * 1000])
def test_add_widened(n):
    """Edges of a thread's eight elements and of a block's 2048."""
    from jetfire_int8training_b200._lib import lib
    g = _gen(n)
    a, b = torch.randn(n + 8, generator=g, device=DEV), torch.randn(n, generator=g, device=DEV).bfloat16()
    want = a.clone()
    want[:n] += b.float()
    assert lib().jf_add_widened(a.data_ptr(), b.data_ptr(), n, torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(a, want)
    assert lib().jf_add_widened(a.data_ptr(), b.data_ptr(), n + 1, None) == -2


@pytest.mark.parametrize("V", [8, 4088, 16376, 16384, 16392, 32776])
def test_lm_loss_at_the_unrolled_step(V):
    """Vocabularies around one and several steps of four 16-byte chunks per thread."""
    from jetfire_int8training_b200.lm_loss import lm_cross_entropy
    g = _gen(V)
    x = (3 * torch.randn(5, V, generator=g, device=DEV)).bfloat16()
    t = torch.tensor([0, V - 1, V // 2, -1, 1], device=DEV)
    want = F.cross_entropy(x.float(), t, ignore_index=-1)
    assert abs(float(lm_cross_entropy(x.clone(), t)) - float(want)) <= 1e-5 * abs(float(want))
