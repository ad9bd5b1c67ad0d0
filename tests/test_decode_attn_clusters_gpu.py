"""Decode attention whose splits merge inside a cluster, against float32: every number of splits, lengths about the split and tile
edges, empty and retired rows, windows, and the shared-prefix form that splits its private keys."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ref(q, k, v, lens, window=0):
    B, Hq, D = q.shape
    S, G = k.shape[1], Hq // k.shape[2]
    s = torch.einsum("bhgd,bshd->bhgs", q.float().view(B, -1, G, D), k.float()) * D ** -0.5
    j, n = torch.arange(S, device=q.device)[None, :], lens[:, None]
    ok = (j < n) & ((j >= n - window) if window else (j >= 0))
    p = torch.softmax(s.masked_fill(~ok[:, None, None], float("-inf")), -1).nan_to_num(0.0)
    return torch.einsum("bhgs,bshd->bhgd", p, v.float()).reshape(B, Hq, D)


def _close(got, ref):
    # 8-bit probabilities (2^-9 each, at random) and an output rounded to 8 bits
    assert torch.isfinite(got).all()
    assert (got.float() - ref).abs().max() <= 1.2e-2 * ref.abs().max() + 1e-6


@pytest.mark.parametrize("D,Hkv,rep", [(128, 2, 4), (128, 8, 2), (64, 2, 8), (256, 4, 6), (256, 2, 8)])
@pytest.mark.parametrize("splits", [0, 1, 2, 3, 5, 7, 8, 16])
@pytest.mark.parametrize("window", [0, 70])
def test_splits(D, Hkv, rep, splits, window):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(D + rep)
    lens = torch.tensor([0, 1, 31, 32, 33, 255, 256, 257, 700], dtype=torch.int32, device="cuda")
    B, S = len(lens), 700
    q = torch.randn(B, Hkv * rep, D, generator=gen, device="cuda").bfloat16()
    k, v = (torch.randn(B, S, Hkv, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    got = C.decode_attention(q, k, v, lens, scale=D ** -0.5, window=window, n_splits=splits)
    _close(got, _ref(q, k, v, lens, window))
    assert torch.equal(got, C.decode_attention(q, k, v, lens, scale=D ** -0.5, window=window, n_splits=splits))


@pytest.mark.parametrize("D,rep,G", [(128, 4, 8), (128, 4, 4), (128, 8, 2), (128, 2, 16), (64, 4, 8)])
@pytest.mark.parametrize("P,Hkv", [(1, 1), (1, 8), (3, 4), (13, 8)])
@pytest.mark.parametrize("prefix_splits", [0, 1, 2, 8])
def test_shared_prefix(D, rep, G, P, Hkv, prefix_splits):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(D + P)
    B, page, pages = P * G, 64, 8
    prefix = torch.tensor([[0, 64, 192][p % 3] for p in range(P)], dtype=torch.int32, device="cuda")
    lens = prefix.repeat_interleave(G) + torch.randint(1, 300, (B,), generator=gen, device="cuda", dtype=torch.int32)
    lens[1] = 0                                             # a retired row
    own = torch.arange(P * pages, (P + B) * pages, device="cuda").view(B, pages)
    shared = torch.arange(P * pages, device="cuda").view(P, pages).repeat_interleave(G, 0)
    table = torch.where(torch.arange(pages, device="cuda")[None] < prefix.repeat_interleave(G)[:, None] // page, shared, own).int().contiguous()
    k, v = (torch.randn((P + B) * pages, page, Hkv, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(B, Hkv * rep, D, generator=gen, device="cuda").bfloat16()
    got = C.decode_attention(q, k, v, lens, scale=D ** -0.5, block_table=table, prefix_len=prefix, group=G, prefix_splits=prefix_splits)
    _close(got, _ref(q, *(x[table.long()].reshape(B, -1, Hkv, D) for x in (k, v)), lens))
