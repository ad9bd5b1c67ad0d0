"""GEMM with the second operand stored [K, N]: same sums in the same order as the [N, K] form, so the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rnd(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").bfloat16()


@pytest.mark.parametrize("M,N,K,K2", [
    (1, 8, 64, 0), (5, 24, 72, 8), (129, 136, 200, 24),       # one tile, columns and k past its edges
    (257, 72, 1000, 0), (850, 48, 1536, 0), (130, 16, 512, 0),  # narrow results: cluster split of k
    (200, 2048, 32768, 0), (256, 1024, 16384, 8), (40, 64, 32768, 0),   # long k: split over clusters or memory
    (1023, 520, 136, 8), (1024, 512, 64, 16), (1025, 520, 136, 8), (2304, 4104, 192, 0),   # around the two-SM kernel's first shape
])
def test_matches_transposed_operand(M, N, K, K2):
    from ferrl_b200.ops import cuda as C
    a, b = _rnd(1, M, K), _rnd(2, K, N + 8)[:, :N]            # rows of a wider matrix
    a2, b2 = (_rnd(3, M, K2), _rnd(4, K2, N)) if K2 else (None, None)
    out = C.gemm_nn(a, b, a2, b2)
    ref = a.double() @ b.double() + (a2.double() @ b2.double() if K2 else 0)
    # float32 sums of K + K2 products of about unit size, one rounding to bf16
    assert bool(((out.double() - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -20 * (K + K2)).all())
    if not (N <= 128 and M > 256) and K < 16384:              # the two forms may split k differently there
        assert torch.equal(out, C.gemm(a, b.t().contiguous(), a2, None if b2 is None else b2.t().contiguous(), cluster_k=-1))
    assert C.kernel_status() == 0


@pytest.mark.parametrize("E,N,K,R", [(3, 64, 128, 256), (5, 136, 192, 640), (2, 768, 64, 256)])
def test_grouped(E, N, K, R):
    from ferrl_b200.ops import cuda as C
    x, w = _rnd(5, R, K), _rnd(6, E, K, N)
    expert = torch.arange(R // 128, dtype=torch.int32, device="cuda") % E
    expert[-1] = -1                                           # an unused tile is left alone
    out = C.lib().moe_grouped_gemm(x, w, expert, torch.zeros(R, N, dtype=torch.bfloat16, device="cuda"), True)
    ref = C.lib().moe_grouped_gemm(x, w.transpose(1, 2).contiguous(), expert, torch.zeros(R, N, dtype=torch.bfloat16, device="cuda"))
    assert torch.equal(out, ref) and not bool(out[-128:].any())


def test_refusals():
    from ferrl_b200.ops import cuda as C
    with pytest.raises(RuntimeError):
        C.gemm_nn(_rnd(1, 8, 64), _rnd(2, 64, 12))            # N not a multiple of 8
    with pytest.raises(RuntimeError):
        C.lib().moe_grouped_gemm(_rnd(1, 128, 72), _rnd(2, 2, 72, 64), torch.zeros(1, dtype=torch.int32, device="cuda"), None, True)
