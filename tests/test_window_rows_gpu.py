"""Windows of rows by one kernel: a gather and its gradient, windows that end inside, at and past the last row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,S,L,H,starts", [(1, 1, 1, 8, (0,)), (3, 17, 9, 264, (0, 8, 16)), (2, 130, 128, 4096, (1, 2)), (4, 33, 40, 72, (0, 5, 32, 200)),
                                            (2, 64, 0, 64, (0, 3)), (2, 9, 9, 60, (0, 4))])                 # the last keeps the gather
def test_rows_and_gradient(B, S, L, H, starts):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200 import ops
    gen = torch.Generator(device="cuda").manual_seed(S * H)
    x = torch.randn(B, S, H, generator=gen, device="cuda").bfloat16().requires_grad_()
    start = torch.tensor(starts, device="cuda")
    dy = torch.randn(B, L, H, generator=gen, device="cuda").bfloat16()
    out = ops.window_rows(x, start, L)
    idx = (start[:, None] + torch.arange(L, device="cuda")[None]).clamp(max=S - 1)[:, :, None].expand(B, L, H)
    assert torch.equal(out, torch.gather(x, 1, idx))
    out.backward(dy)
    ref = torch.zeros(B, S, H, dtype=torch.float64, device="cuda").scatter_add_(1, idx, dy.double())
    once = torch.zeros(B, S, H, dtype=torch.float64, device="cuda").scatter_add_(1, idx, torch.ones_like(dy).double()) <= 1
    assert torch.equal(x.grad[once].double(), ref[once])
    mag = torch.zeros_like(ref).scatter_add_(1, idx, dy.double().abs())
    # the last row's sum: 32 bits and one rounding (the gather's own gradient rounds at every term)
    assert H % 8 or bool(((x.grad - ref).abs() <= 2 ** -8 * ref.abs() + 2 ** -20 * mag).all())
