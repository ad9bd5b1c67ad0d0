"""Stores of the GEMM epilogues that turn whole chunks of 64 columns around in shared memory: ragged rows and columns, residuals
and outputs whose rows do not start on 16 bytes (which keep the direct stores), against float32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [129, 160, 257, 1057])
@pytest.mark.parametrize("N", [64, 72, 120, 128, 200, 328, 1000])
@pytest.mark.parametrize("form", [(64, -1), (128, -1), (176, -1), (256, -1), (0, 128), (0, 256)])
@pytest.mark.parametrize("residual", [None, 0, 4])
def test_ragged_outputs(M, N, form, residual):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(M * N)
    K = 72
    x, w = (torch.randn(n, K, generator=gen, device="cuda").bfloat16() for n in (M, N))
    res = None if residual is None else torch.randn(M, N + residual, generator=gen, device="cuda").bfloat16()[:, :N]
    bn, two = form
    got = C.lib().gemm(x, w, None, None, res, False, bn, 0, two)
    assert C.kernel_status() == 0
    ref = x.float() @ w.float().T + (0 if res is None else res.float())
    # sums of 72 exact products in 32 bits, rounded once to 16: half a unit in the last place of 8 bits
    assert ((got.float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-4).all()
