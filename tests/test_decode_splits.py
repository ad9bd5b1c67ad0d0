"""How many splits a row of decode attention is cut into (a rule on sizes, checked on the CPU), and rows about the length up to which one
CTA of a cluster takes them alone."""
import pytest
import torch


def _splits(pairs, room, D=128, rep=4, **kw):
    from ferrl_b200.ops import cuda as C
    return C.lib().decode_attn_splits(pairs, rep, 1, D, room, **kw)


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("pairs", [1, 2, 8, 15, 16, 17, 33, 34, 66, 67, 111, 112, 148, 149, 200, 296, 297, 1024])
def test_splits_leave_work(D, pairs):
    for room in (1, 255, 256, 300, 511, 512, 1000, 1024, 2047, 2048, 4095, 4096, 8192, 100000):
        s = _splits(pairs, room, D)
        assert s in (1, 2, 4, 8, 16)
        # more than eight are merged by a second kernel, which only long splits pay for; a CTA never has less than a tile of 32 keys
        assert s <= 8 or room // s >= 256
        assert s == 1 or room // s >= 32
        assert s == 1 or pairs * s <= 4 * 148        # all at work at once
    assert _splits(pairs, 100000, D, window=300) == _splits(pairs, 300, D)
    assert _splits(pairs, 200, D, window=300) == _splits(pairs, 200, D)


def test_forms_without_tensor_cores_are_cut_finer():
    assert _splits(2, 900, rep=3) == 16 > _splits(2, 900, variant=1, window=200)
    assert _splits(2, 900, D=80) == _splits(2, 900, variant=2) == 16
    assert _splits(1000, 900, rep=3) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("D,Hkv,rep", [(128, 2, 4), (64, 4, 2), (256, 2, 8), (128, 2, 3)])
@pytest.mark.parametrize("S", [65, 300, 600])
@pytest.mark.parametrize("window", [0, 64, 66])
def test_short_rows(D, Hkv, rep, S, window):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    from test_decode_attn_clusters_gpu import _close, _ref
    gen = torch.Generator(device="cuda").manual_seed(D + S)
    lens = torch.tensor([0, 1, 63, 64, 65], dtype=torch.int32, device="cuda")
    q = torch.randn(5, Hkv * rep, D, generator=gen, device="cuda").bfloat16()
    k, v = (torch.randn(5, S, Hkv, D, generator=gen, device="cuda").bfloat16() for _ in range(2))
    for splits in (0, 4, 8):
        _close(C.decode_attention(q, k, v, lens, scale=D ** -0.5, window=window, n_splits=splits), _ref(q, k, v, lens, window))
