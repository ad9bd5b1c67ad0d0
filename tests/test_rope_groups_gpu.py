"""QK-norm and RoPE with many heads a warp (many tokens) against one head a warp (the same tokens in small calls), and embedding rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens,Hq,Hkv,D,rot,weights,zero", [
    (9473, 3, 1, 128, 128, True, False), (7579, 4, 1, 128, 64, True, True), (6315, 5, 1, 256, 64, True, True), (5413, 5, 2, 256, 256, False, False),
])
def test_many_heads_a_warp(tokens, Hq, Hkv, D, rot, weights, zero):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    assert tokens * (Hq + Hkv) >= 148 * 64 * 4 > 512 * (Hq + Hkv)
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
    for s in range(0, tokens, 512):
        for a, b in zip(whole, run(slice(s, s + 512))):
            # sums of squares in another order move a factor by 2^-24, which turns a rounding to 16 bits now and then
            d, b = (a[:, s:s + 512].float() - b.float()).abs(), b.float()
            assert bool((d <= 2 ** -7 * b.abs() + 2 ** -8 * b.abs().amax(-1, keepdim=True)).all()) and float((d > 0).float().mean()) < 0.01


@pytest.mark.parametrize("H,off,dtype", [(4096, 0, torch.bfloat16), (6, 0, torch.bfloat16), (260, 0, torch.float32), (128, 1, torch.bfloat16), (8, 0, torch.float32)])
@pytest.mark.parametrize("scale", [1.0, 73.5])
def test_embedding_rows(H, off, dtype, scale):
    from ferrl_b200.ops import cuda as C
    table = torch.randn(777 * H + off, device="cuda").to(dtype)[off:].view(777, H)
    ids = torch.randint(0, 777, (3, 41), device="cuda")
    assert torch.equal(C.embedding(ids, table, scale), (table[ids].float() * scale).to(dtype))
