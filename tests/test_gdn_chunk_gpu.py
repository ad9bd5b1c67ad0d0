"""Grad-free chunked delta rule at the edges of its chunks, slices of the state and rounds, against a float64 recurrence."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def recurrence(q, k, v, g, beta, S, l2norm):
    q, k, v, g, beta = (t.double() for t in (q, k, v, g, beta))
    if l2norm:
        q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    rep = v.shape[2] // k.shape[2]
    q, k = q.repeat_interleave(rep, 2) * 128 ** -0.5, k.repeat_interleave(rep, 2)
    S = v.new_zeros(v.shape[0], v.shape[2], 128, 128) if S is None else S.double()
    out = torch.empty_like(v)
    for t in range(v.shape[1]):
        S = S * g[:, t].exp()[..., None, None]
        d = (v[:, t] - torch.einsum("bhkv,bhk->bhv", S, k[:, t])) * beta[:, t, :, None]
        S = S + k[:, t, :, :, None] * d[:, :, None]
        out[:, t] = torch.einsum("bhkv,bhk->bhv", S, q[:, t])
    return out, S


@pytest.mark.parametrize("B,T,Hk,Hv,state,l2norm,wide", [
    (1, 1, 1, 1, True, True, 0), (1, 63, 1, 2, False, True, 8), (2, 65, 2, 6, True, True, 8), (1, 129, 1, 1, True, False, 4),
    (1, 191, 1, 37, True, True, 8), (1, 192, 2, 38, False, True, 8),      # 37 heads: the last that take narrow slices of the state
    (2, 5250, 32, 32, True, True, 8),                                      # more chunks than one round holds
])
def test_chunks_match_the_recurrence(B, T, Hk, Hv, state, l2norm, wide):
    from ferrl_b200.ops import cuda as Cc
    gen = torch.Generator(device="cuda").manual_seed(T * Hv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    mixed = rnd(B, T, (2 * Hk + Hv) * 128 + wide).bfloat16()[..., wide:] if wide else rnd(B, T, (2 * Hk + Hv) * 128).bfloat16()
    q, k, v = (t.reshape(B, T, -1, 128) if not wide else t.unflatten(-1, (-1, 128)) for t in mixed.split([Hk * 128, Hk * 128, Hv * 128], -1))
    if not l2norm:
        q, k = q * 0.125, k * 0.125
    g = -torch.rand(B, T, Hv, generator=gen, device="cuda") * torch.tensor([0.01, 1.0, 20.0], device="cuda")[torch.randint(0, 3, (Hv,), generator=gen, device="cuda")]
    beta = torch.rand(B, T, Hv, generator=gen, device="cuda")
    S0 = rnd(B, Hv, 128, 128) * 0.3 if state else None
    o, S = Cc.gdn_chunk_fwd(q, k, v, g, beta, S0, l2norm, 1e-6)
    ro, rS = recurrence(q, k, v, g, beta, S0, l2norm)
    # 32-bit sums over chunks of 64 x 128 terms: a few units of 2^-24 of the largest entry, ten times that allowed (the
    # exponential's argument alone rounds at 2^-24 of up to 20); outputs are rounded to 16 bits once
    assert float((S - rS).norm() / rS.norm()) < 5e-6 and float((S - rS).abs().max()) < 2e-5 * float(rS.abs().max())
    assert bool(((o - ro).abs() <= 2 ** -8 * ro.abs() + 2e-5 * ro.abs().max()).all())
    again = Cc.gdn_chunk_fwd(q, k, v, g, beta, S0, l2norm, 1e-6)
    assert torch.equal(again[0], o) and torch.equal(again[1], S)


def test_more_rows_than_a_grid_has_in_its_last_dimension():
    from ferrl_b200.ops import cuda as Cc
    B = 65536
    gen = torch.Generator(device="cuda").manual_seed(3)
    q, k, v = (torch.randn(B, 1, 1, 128, generator=gen, device="cuda").bfloat16() for _ in range(3))
    g, beta = -torch.rand(B, 1, 1, generator=gen, device="cuda"), torch.rand(B, 1, 1, generator=gen, device="cuda")
    o, S = Cc.gdn_chunk_fwd(q, k, v, g, beta, None, True, 1e-6)
    for at in (slice(0, 3), slice(B - 3, B)):
        ro, rS = recurrence(q[at], k[at], v[at], g[at], beta[at], None, True)
        assert float((S[at] - rS).norm() / rS.norm()) < 5e-6
        assert bool(((o[at] - ro).abs() <= 2 ** -8 * ro.abs() + 2e-5 * ro.abs().max()).all())


def test_scratch_is_guarded():
    """Canary mode keeps every buffer that kernels write until it is checked: the chunk factors' scratch is one of them."""
    from ferrl_b200.ops import cuda as Cc
    q, k, v = (torch.randn(1, 640, 4, 128, device="cuda").bfloat16() for _ in range(3))
    g, beta = -torch.rand(1, 640, 4, device="cuda"), torch.rand(1, 640, 4, device="cuda")
    before = torch.cuda.memory_allocated()
    out = Cc.gdn_chunk_fwd(q, k, v, g, beta, None, True, 1e-6)
    pieces = 10 * 4 * 6 * 64 * 64 * 2                                          # ten chunks of four heads, six 16-bit pieces each
    assert torch.cuda.memory_allocated() - before >= pieces + sum(t.numel() * t.element_size() for t in out)
