"""The form that a matrix product takes: which tile width and which split of k (host arithmetic, nothing is launched)."""
import os

import pytest

from ferrl_b200.ops import cuda as C

pytestmark = pytest.mark.skipif(not os.path.exists(C._SO), reason="the library is not built")
PAIRS = {(64, 2), (64, 4), (128, 2), (128, 4), (128, 8), (256, 2)}         # tile widths and clusters that are compiled


@pytest.mark.parametrize("M", [1, 64, 128, 200, 256, 257, 1000, 5000])
@pytest.mark.parametrize("N", [8, 16, 40, 64, 96, 512, 2048, 24576])
@pytest.mark.parametrize("K", [8, 64, 4096, 32768, 151936])
def test_only_forms_that_are_compiled(M, N, K):
    for nn in (False, True):
        bn, split, cluster = C.lib().gemm_plan(M, N, K, 0, 148, nn)
        assert bn in ((64, 128, 256) if nn else (32, 64, 128, 176, 256)) and (cluster == 1 or ((bn, cluster) in PAIRS and split == 1 and N % 16 == 0))
        assert split == 1 or (M <= 256 and split <= 16 and (K + 63) // 64 >= split)


@pytest.mark.parametrize("M,N,K,nn,ways", [
    (200, 2048, 32768, True, 4), (256, 4096, 32768, True, 2), (64, 64, 131072, True, 8),         # weights read as rows
    (1, 64, 131072, False, 8), (100, 96, 32768, False, 8), (256, 256, 32768, False, 8),           # one column of tiles, long k
    (128, 16, 17408, False, 4), (256, 48, 17408, False, 4), (300, 16, 17408, False, 4),           # narrow results, either side of 256 rows
])
def test_long_sums_are_split(M, N, K, nn, ways):
    _, split, cluster = C.lib().gemm_plan(M, N, K, 0, 148, nn)
    assert split * cluster >= ways


@pytest.mark.parametrize("M,N,K", [(100, 768, 64), (8, 1024, 64), (256, 4096, 64), (64, 768, 256)])
def test_short_sums_have_narrow_tiles_of_their_own(M, N, K):
    bn, split, cluster = C.lib().gemm_plan(M, N, K)
    assert bn <= 64 and split == cluster == 1
