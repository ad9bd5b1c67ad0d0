"""Attention backward at head dim 256 on tcgen05 (csrc/kernels/flash_bwd256_tc.cu) against fp32 autograd through the eager
attention.  Reference behaviour: the gated GQA core of crates/ferrl/src/qwen35.rs:1240-1313."""
import pytest
import torch

from _numerics import close

pytestmark = pytest.mark.gpu
D = 256


@pytest.mark.parametrize("B,S,Hq,Hkv,window", [
    (1, 16, 2, 2, 0), (3, 63, 2, 1, 0), (1, 64, 1, 1, 0), (2, 65, 3, 1, 0),      # one streamed tile, then a row of the next
    (1, 127, 4, 4, 0), (2, 128, 5, 1, 0), (2, 129, 8, 1, 0), (1, 193, 7, 1, 0),  # one row tile and its neighbours; uneven shares of the heads
    (2, 333, 8, 2, 0), (1, 1535, 16, 2, 0), (1, 1100, 6, 1, 0), (8, 700, 24, 4, 0),     # with and without shares
    (2, 300, 4, 2, 17), (1, 333, 8, 1, 64), (2, 700, 4, 2, 150), (1, 200, 4, 2, 4096),   # windows
])
def test_backward_at_head_dim_256(B, S, Hq, Hkv, window):
    from ferrl_b200.ops import cuda as C, eager
    g = torch.Generator(device="cuda").manual_seed(B * 31 + S + window)
    # rows as they lie in a fused projection: q, k, v side by side, with something else behind them
    n = (Hq + 2 * Hkv) * D
    wide = torch.randn(B, S, n + 64, device="cuda", generator=g).bfloat16()
    q, k, v = (t.unflatten(-1, (-1, D)) for t in wide[..., :n].split([Hq * D, Hkv * D, Hkv * D], -1))
    do = torch.randn(B, S, Hq, D, device="cuda", generator=g).bfloat16()
    scale = D ** -0.5
    o, lse = C.lib().flash_fwd(q, k, v, scale, True, window, 0, 0)
    run = lambda: C.lib().flash_bwd(q, k, v, o, lse, do, scale, True, window, 0, 0, None)  # noqa: E731
    got = run()
    refs = [t.float().requires_grad_() for t in (q, k, v)]
    eager.attention(*refs, scale=scale, causal=True, window=window).backward(do.float())
    warp = C.lib().flash_bwd(q, k, v, o, lse, do, scale, True, window, 0, 1, None)
    assert C.kernel_status() == 0
    # operands P and dS of 8 bits behind the leading one (2^-9 each, at random) and a 16-bit result (2^-9): 2e-2 of the largest
    # entry is what the warp-level kernels, which round the same operands, are held to
    for a, r, w in zip(got, refs, warp):
        close(a.float(), r.grad, 2e-2)
        rel = lambda x: float((x.float() - r.grad).norm() / r.grad.norm().clamp(min=1e-6))  # noqa: E731
        assert rel(a) <= 1.1 * rel(w) + 1e-3
    for a, b in zip(got, run()):
        assert torch.equal(a, b)        # fixed summation order


def test_a_single_token():
    """One key: its weight is one, so dV is the gradient of the output and dQ, dK vanish but for the 16-bit rounding of o."""
    from ferrl_b200.ops import cuda as C
    g = torch.Generator(device="cuda").manual_seed(3)
    q, k, v, do = (torch.randn(2, 1, 2, D, device="cuda", generator=g).bfloat16() for _ in range(4))
    o, lse = C.lib().flash_fwd(q, k, v, D ** -0.5, True, 0, 0, 0)
    dq, dk, dv = C.lib().flash_bwd(q, k, v, o, lse, do, D ** -0.5, True, 0, 0, 0, None)
    close(dv.float(), do.float(), 2e-3)
    # dS = dP - rowsum(o do) is a difference of 256 equal products in another order: 256 * 2^-24 of their absolute sum at most
    bound = 256 * 2 ** -24 * (v.float() * do.float()).abs().sum(-1, keepdim=True) * D ** -0.5
    assert (dq.float().abs() <= 1.1 * bound * k.float().abs() + 1e-6).all() and (dk.float().abs() <= 1.1 * bound * q.float().abs() + 1e-6).all()


def test_rows_of_another_sequence_do_not_enter():
    """Tiles reach past a sequence's end into the next one: what lies there, NaN even, stays out of the gradients."""
    from ferrl_b200.ops import cuda as C
    B, S, Hq, Hkv, scale = 3, 150, 4, 1, D ** -0.5
    g = torch.Generator(device="cuda").manual_seed(5)
    q, k, v, do = (torch.randn(B, S, h, D, device="cuda", generator=g).bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    o, lse = C.lib().flash_fwd(q, k, v, scale, True, 0, 0, 1)
    want = C.lib().flash_bwd(q, k, v, o, lse, do, scale, True, 0, 0, 0, None)
    for t in (q, k, v, o, do):
        t[1] = float("nan")
    lse[1] = float("nan")
    got = C.lib().flash_bwd(q, k, v, o, lse, do, scale, True, 0, 0, 0, None)
    for a, w in zip(got, want):
        assert torch.equal(a[::2], w[::2])
    assert C.kernel_status() == 0
