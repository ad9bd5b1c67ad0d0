"""Grouped products on pairs of SMs (two row tiles of an expert at a time) against the one-SM form, which adds in the same order:
the same bits in every row that belongs to a token."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tokens of each expert: none, one row, a tile and its neighbours, odd and even numbers of tiles, the last expert empty or full
@pytest.mark.parametrize("counts", [
    [5], [128], [129], [0, 0, 300], [1, 127, 128, 129, 0, 255, 256, 257, 384, 385], [640, 0, 1], [130] * 40, [0, 900, 0, 17, 0],
])
@pytest.mark.parametrize("N,K,nn", [(256, 64, False), (264, 136, False), (320, 192, True), (776, 256, True), (1536, 512, False)])
def test_pairs_equal_single_tiles(counts, N, K, nn):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(N + len(counts))
    E = len(counts)
    tiles = [-(-c // 128) for c in counts]
    rows = (sum(tiles) + 3) * 128                      # unused tiles behind the last segment
    expert = torch.tensor([e for e, t in enumerate(tiles) for _ in range(t)] + [-1] * 3, dtype=torch.int32, device="cuda")
    token = torch.full((rows,), -1, dtype=torch.int32, device="cuda")
    at = 0
    for c, t in zip(counts, tiles):
        token[at:at + c] = torch.arange(c, dtype=torch.int32, device="cuda")
        at += t * 128
    xs = torch.randn(rows, K, generator=gen, device="cuda").bfloat16()
    W = torch.randn(E, *((K, N) if nn else (N, K)), generator=gen, device="cuda").bfloat16()
    for tok in (token, None):
        outs = []
        for form in (1, 2):
            out = torch.zeros(rows, N, device="cuda", dtype=torch.bfloat16)
            C.lib().moe_grouped_gemm(xs, W, expert, out, nn, tok, form)
            outs.append(out)
        assert C.kernel_status() == 0
        assert torch.equal(*outs)
    real = token >= 0
    ref = torch.cat([xs[i * 128:(i + 1) * 128].float() @ (W[e].float() if nn else W[e].float().T) for i, e in enumerate(expert.tolist()) if e >= 0])
    ref = ref[real[:ref.shape[0]]]
    # one rounding to 16 bits of a sum of K products in 32 bits
    assert (outs[1][real].float() - ref).abs().max() <= 2 ** -8 * ref.abs().max()


def test_too_many_row_tiles_are_refused():
    from ferrl_b200.ops import cuda as C
    xs = torch.zeros(4097 * 128, 64, device="cuda", dtype=torch.bfloat16)
    W = torch.zeros(1, 256, 64, device="cuda", dtype=torch.bfloat16)
    expert = torch.zeros(4097, dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="row tiles"):
        C.lib().moe_grouped_gemm(xs, W, expert, None, False, None, 2)
    C.lib().moe_grouped_gemm(xs, W, expert)
