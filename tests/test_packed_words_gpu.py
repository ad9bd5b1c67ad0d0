"""Kernels that work on packed pairs of 16-bit values, against float64: QK norm with rotation, forward and backward, and the row
statistics of the attention backward where the output's rows start on 8 bytes only."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# whole and partial rotation, one head and odd numbers of heads, no norm, norms around one
@pytest.mark.parametrize("T,Hq,Hkv,D,rot,norm,zero", [(1, 1, 1, 128, 128, True, False), (37, 3, 1, 128, 64, True, True), (130, 5, 2, 256, 64, True, False),
                                                       (65, 2, 1, 256, 256, False, False), (2100, 8, 2, 128, 128, True, False)])
def test_qk_norm_and_rotation(T, Hq, Hkv, D, rot, norm, zero):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(T + D)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    q, k, dq, dk = rnd(1, T, Hq, D), rnd(1, T, Hkv, D), rnd(1, T, Hq, D), rnd(1, T, Hkv, D)
    w = [rnd(D), rnd(D)] if norm else [None, None]
    ang, pos = torch.rand(T, rot // 2, generator=gen, device="cuda") * 6, torch.arange(T, device="cuda")
    ins = [q.clone().requires_grad_(), k.clone().requires_grad_()]
    out = C.qk_norm_rope(*ins, *w, 1e-6, ang.cos(), ang.sin(), pos, zero)
    grads = torch.autograd.grad(out, ins, [dq, dk])
    co, si = (t.double()[None, :, None] for t in (ang.cos(), ang.sin()))

    def ref(x, wv):
        if wv is not None:
            x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * (wv.double() + (1 if zero else 0))
        a, b, rest = x[..., :rot // 2], x[..., rot // 2:rot], x[..., rot:]
        return torch.cat([a * co - b * si, b * co + a * si, rest], -1)
    for x, wv, y, g, gin in zip((q, k), w, out, (dq, dk), grads):
        x64 = x.double().requires_grad_()
        r = ref(x64, wv)
        r.backward(g.double())
        size = x64.detach().abs() if wv is None else (x64.detach() * torch.rsqrt(x64.detach().square().mean(-1, keepdim=True) + 1e-6) * (wv.double() + (1 if zero else 0))).abs()
        pair = torch.cat([size[..., :rot // 2] + size[..., rot // 2:rot]] * 2 + [size[..., rot:]], -1)
        # the normalised value rounds to 8 bits before it turns, the result once more
        assert bool(((y.double() - r).abs() <= 2 ** -8 * pair + 2 ** -8 * r.abs() + 1e-6).all())
        # 32-bit arithmetic on the way back, one rounding; the projection's sum of D terms cancels against a value of its size
        bound = 2 ** -8 * x64.grad.abs() + 2 ** -18 * x64.grad.abs().amax(-1, keepdim=True) + 1e-6
        assert bool(((gin.double() - x64.grad).abs() <= bound).all())


@pytest.mark.parametrize("B,S,Hq,Hkv", [(1, 1, 1, 1), (2, 129, 4, 2), (1, 700, 8, 2)])
def test_statistics_of_rows_on_8_bytes(B, S, Hq, Hkv):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(S)
    q, k, v, do = (torch.randn(B, S, h, 128, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    o, lse = C.lib().flash_fwd(q, k, v, 128 ** -0.5, True, 0, 0, 0)
    off = torch.cat([o.new_zeros(4), o.reshape(-1)])[4:].view(o.shape)
    assert off.data_ptr() % 16 == 8 and off.is_contiguous()
    run = lambda x: C.lib().flash_bwd(q, k, v, x, lse, do, 128 ** -0.5, True, 0, 0, 0)  # noqa: E731
    assert all(torch.equal(a, b) for a, b in zip(run(o), run(off)))
    assert C.kernel_status() == 0
