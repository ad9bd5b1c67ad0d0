"""RMSNorm kernels for short rows: widths around the lanes of a row, last rows of a CTA, gates inside a wider matrix."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,per,H,wide,off", [
    (1, 1, 8, 8, 0), (5, 13, 24, 400, 8), (64, 1, 32, 32, 0), (9, 7, 40, 283, 3), (3, 33, 64, 2200, 16),
    (257, 3, 128, 640, 128), (2, 48, 128, 6150, 6), (17, 2, 136, 300, 8), (31, 4, 256, 1024, 0), (2, 2, 264, 600, 8),
    (6, 3, 100, 391, 3),
])
def test_short_rows(n, per, H, wide, off):
    from ferrl_b200.ops import cuda as C, eager
    gen = torch.Generator(device="cuda").manual_seed(n * per * H)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    x, dy, w = rnd(n, per, H), rnd(n, per, H), (1 + 0.1 * rnd(H).float()).bfloat16()
    gate = rnd(n, wide)[:, off:off + per * H].unflatten(1, (per, H))
    xs, gs = x.clone().requires_grad_(), gate.detach().requires_grad_()
    y = C.rmsnorm_gated(xs, gs, w, 1e-6)
    with torch.no_grad():
        assert torch.equal(y, C.rmsnorm_gated(x, gate, w, 1e-6))
    y.backward(dy)
    xr, gr = x.double().requires_grad_(), gate.double().requires_grad_()
    xn = xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-6)
    yr = xn * w.double() * torch.nn.functional.silu(gr)
    yr.backward(dy.double())
    # one rounding to 16 bits each; dx is a difference of two terms of the size of its first
    assert bool(((y - yr).abs() <= 2 ** -8 * yr.abs() + 1e-6).all())
    first = (dy.double() * w.double() * torch.nn.functional.silu(gr)).abs() * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-6)
    assert bool(((xs.grad - xr.grad).abs() <= 2 ** -8 * xr.grad.abs() + 1e-5 * (first + first.mean(-1, keepdim=True))).all())
    assert bool(((gs.grad - gr.grad).abs() <= 2 ** -8 * gr.grad.abs() + 1e-5).all())
    for weight, zero in ((w, False), (w, True), (None, False)):
        xs = x.clone().requires_grad_()
        xr = x.double().requires_grad_()
        scale = 1.0 if weight is None else weight.double() + zero
        y, yr = C.rmsnorm(xs, weight, 1e-6, zero), xr * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-6) * scale
        y.backward(dy)
        yr.backward(dy.double())
        first = (dy.double() * scale).abs() * torch.rsqrt(xr.square().mean(-1, keepdim=True) + 1e-6)
        assert bool(((y - yr).abs() <= 2 ** -8 * yr.abs() + 1e-6).all())
        assert bool(((xs.grad - xr.grad).abs() <= 2 ** -8 * xr.grad.abs() + 1e-5 * (first + first.mean(-1, keepdim=True))).all())
