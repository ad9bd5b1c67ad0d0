"""Attention backward for head dim 256 at the edges of its 64-row tiles, key groups and windows, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,Hq,Hkv,window", [
    (1, 1, 2, 1, 0), (2, 31, 2, 2, 0), (1, 64, 3, 1, 0), (2, 65, 4, 2, 0), (1, 127, 8, 1, 0), (1, 129, 2, 2, 5), (2, 200, 4, 2, 64), (1, 515, 6, 2, 300),
])
def test_backward(B, S, Hq, Hkv, window):
    from ferrl_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(S * Hq + window)
    rnd = lambda h: torch.randn(B, S, h, 256, generator=gen, device="cuda").bfloat16()  # noqa: E731
    q, k, v, do = rnd(Hq), rnd(Hkv), rnd(Hkv), rnd(Hq)
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    o = ops.attention(*leaves, scale=1 / 16, causal=True, softmax_fp32=True, **({"window": window} if window else {}))
    got = torch.autograd.grad(o, leaves, do)
    ref = [t.double().requires_grad_() for t in (q, k, v)]
    far = torch.arange(S, device="cuda")[:, None] - torch.arange(S, device="cuda")[None, :]
    ok = (far >= 0) & ((far < window) if window else (far >= 0))
    qd = ref[0].transpose(1, 2).reshape(B, Hkv, -1, S, 256)
    p = torch.softmax((torch.einsum("bgrsd,btgd->bgrst", qd, ref[1]) / 16).masked_fill(~ok, float("-inf")), -1)
    od = torch.einsum("bgrst,btgd->bgrsd", p, ref[2]).reshape(B, Hq, S, 256).transpose(1, 2)
    want = torch.autograd.grad(od, ref, do.double())
    # probabilities and their gradients are 16-bit operands (2^-9 each), results are rounded once more
    for a, b in zip(got, want):
        assert float((a.double() - b).norm()) <= 1e-2 * float(b.norm()) + 1e-6
        assert float((a.double() - b).abs().max()) <= 2e-2 * float(b.abs().max()) + 1e-6


@pytest.mark.parametrize("Sq,Sk,off,causal,window", [
    (33, 97, 64, True, 0), (1, 77, 76, True, 0), (64, 200, 136, True, 50), (130, 195, 65, True, 0),      # queries behind cached keys
    (40, 130, 0, False, 0), (129, 63, 0, False, 0),                                                       # every key visible
])
def test_backward_of_unequal_lengths(Sq, Sk, off, causal, window):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(Sq * Sk)
    rnd = lambda n, h: torch.randn(2, n, h, 256, generator=gen, device="cuda").bfloat16()  # noqa: E731
    q, k, v, do = rnd(Sq, 4), rnd(Sk, 2), rnd(Sk, 2), rnd(Sq, 4)
    leaves = [t.clone().requires_grad_() for t in (q, k, v)]
    got = torch.autograd.grad(C.attention(*leaves, scale=1 / 16, causal=causal, window=window, q_offset=off), leaves, do)
    ref = [t.double().requires_grad_() for t in (q, k, v)]
    far = torch.arange(off, off + Sq, device="cuda")[:, None] - torch.arange(Sk, device="cuda")[None, :]
    ok = torch.ones_like(far, dtype=torch.bool) if not causal else (far >= 0) & ((far < window) if window else (far >= 0))
    p = torch.softmax((torch.einsum("bgrsd,btgd->bgrst", ref[0].transpose(1, 2).reshape(2, 2, 2, Sq, 256), ref[1]) / 16).masked_fill(~ok, float("-inf")), -1)
    want = torch.autograd.grad(torch.einsum("bgrst,btgd->bgrsd", p, ref[2]).reshape(2, 4, Sq, 256).transpose(1, 2), ref, do.double())
    # 16-bit operands and results as above
    for a, b in zip(got, want):
        assert float((a.double() - b).norm()) <= 1e-2 * float(b.norm()) + 1e-6
        assert float((a.double() - b).abs().max()) <= 2e-2 * float(b.abs().max()) + 1e-6
