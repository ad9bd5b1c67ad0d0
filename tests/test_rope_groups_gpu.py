"""QK-norm and RoPE with many heads a warp (many tokens) against one head a warp (the same tokens in small calls), and embedding rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,Hq,Hkv,D,rot,weights,zero", [
    (9473, 3, 1, 128, 128, True, False), (7579, 4, 1, 128, 64, True, True), (6315, 5, 1, 256, 64, True, True), (5413, 5, 2, 256, 256, False, False),
])
def test_many_heads_a_warp(tokens, Hq, Hkv, D, rot, weights, zero):
    assert tokens * (Hq + Hkv) >= 148 * 64 * 4 > 512 * (Hq + Hkv)
    _same_as_in_small_calls(tokens, Hq, Hkv, D, rot, weights, zero, 512)


@pytest.mark.parametrize("tokens,Hq,Hkv,D,rot,weights,zero", [
    (751, 3, 1, 128, 128, True, False), (4001, 3, 1, 128, 64, True, True), (4737, 6, 2, 128, 128, True, False),      # 2, 4 and 8 heads a warp
    (753, 3, 1, 256, 64, True, True), (4003, 3, 1, 256, 64, False, False), (9473, 3, 1, 256, 256, True, True),       # 1, 2 and 4
    (1601, 9, 1, 128, 128, True, False), (3203, 4, 1, 256, 64, True, False),                                         # heads that do not fill them
])
def test_heads_a_warp(tokens, Hq, Hkv, D, rot, weights, zero):
    _same_as_in_small_calls(tokens, Hq, Hkv, D, rot, weights, zero, 128)


def _same_as_in_small_calls(tokens, Hq, Hkv, D, rot, weights, zero, small):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    p = rnd(1, tokens, (Hq + Hkv) * D + 8)
    q, k = p[..., :Hq * D].unflatten(-1, (Hq, D)), p[..., Hq * D:(Hq + Hkv) * D].unflatten(-1, (Hkv, D))
    qw, kw = (rnd(D), rnd(D)) if weights else (None, None)
    ang = torch.rand(tokens, rot // 2, generator=gen, device="cuda") * 6
    pos = torch.randperm(tokens, generator=gen, device="cuda")[None]
    dq, dk = rnd(1, tokens, Hq, D), rnd(1, tokens, Hkv, D)

    def run(at):
        leaves = [q[:, at].detach().requires_grad_(), k[:, at].detach().requires_grad_()]
        out = C.qk_norm_rope(*leaves, qw, kw, 1e-6, ang.cos(), ang.sin(), pos[:, at], zero)
        return [*out, *torch.autograd.grad(out, leaves, [dq[:, at], dk[:, at]])]
    whole = run(slice(None))
    for s in range(0, tokens, small):
        for a, b in zip(whole, run(slice(s, s + small))):
            # sums of squares in another order move a factor by 2^-24, which turns a rounding to 16 bits now and then
            d, b = (a[:, s:s + small].float() - b.float()).abs(), b.float()
            assert bool((d <= 2 ** -7 * b.abs() + 2 ** -8 * b.abs().amax(-1, keepdim=True)).all()) and float((d > 0).float().mean()) < 0.01


@pytest.mark.no_canary
def test_backward_of_few_heads_keeps_its_lanes_busy():
    """A quarter of the heads takes little more than a quarter of the time: 0.30 of it, 0.38 with eight heads a warp."""
    from ferrl_b200.ops import cuda as C
    L, co, pos = C.lib(), torch.rand(8192, 64, device="cuda"), torch.arange(8192, device="cuda")
    w = torch.ones(128, device="cuda", dtype=torch.bfloat16)

    def us(heads):
        sets = [[torch.randn(8192, h, 128, device="cuda").bfloat16() for h in (heads * 4, heads) * 3] for _ in range(3)]
        go = lambda: [L.qk_norm_rope_bwd(q, k, w, w, co, co, pos, 1, 1e-6, False, dq, dk, oq, ok) for q, k, dq, dk, oq, ok in sets]  # noqa: E731
        ts = []
        for _ in range(9):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            go()
            a.record()
            for _ in range(4):
                go()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b))
        return sorted(ts)[4]
    assert us(2) < 0.34 * us(8)


@pytest.mark.parametrize("H,off,dtype", [(4096, 0, torch.bfloat16), (6, 0, torch.bfloat16), (260, 0, torch.float32), (128, 1, torch.bfloat16), (8, 0, torch.float32)])
@pytest.mark.parametrize("scale", [1.0, 73.5])
def test_embedding_rows(H, off, dtype, scale):
    from ferrl_b200.ops import cuda as C
    table = torch.randn(777 * H + off, device="cuda").to(dtype)[off:].view(777, H)
    ids = torch.randint(0, 777, (3, 41), device="cuda")
    assert torch.equal(C.embedding(ids, table, scale), (table[ids].float() * scale).to(dtype))
