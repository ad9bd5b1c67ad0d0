"""Adapter gradients where the token ranges, their chains of sums and the column tiles end: against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one stage, whole chains and a stage more or less, ranges that are empty, more column tiles than run at once, ranks on either side
# of the tile's width
@pytest.mark.parametrize("M,R,C", [(1, 8, 8), (64, 64, 128), (1024, 16, 136), (1025, 24, 1000), (17 * 1024 - 1, 32, 56 * 1024),
                                   (2049, 48, 60000), (5000, 64, 4104), (5000, 72, 4104), (700, 128, 264), (300, 40, 128)])
def test_ranges_and_chains(M, R, C):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as Cc
    gen = torch.Generator(device="cuda").manual_seed(M + R)
    u = torch.randn(M, R + 8, generator=gen, device="cuda").bfloat16()[:, 8:] if R % 16 == 0 else torch.randn(M, R, generator=gen, device="cuda").bfloat16()
    x = torch.randn(M, C + 8, generator=gen, device="cuda").bfloat16()[:, :C]
    got = Cc.lib().lora_grad(u, x)
    ref = torch.cat([u.double().t() @ part.double() for part in x.split(8192, 1)], 1)
    # products are exact; a chain of 512 terms (of M above rank 64) adds with at most 2^-23 of its size a step of 16, the rest rounds once a sum
    steps = (min(M, 512) if R <= 64 else M) / 16 + 64
    bound = torch.cat([u.double().abs().t() @ part.double().abs() for part in x.split(8192, 1)], 1) * (steps * 2 ** -23)
    assert bool(((got - ref).abs() <= bound + 1e-12).all())
    assert torch.equal(got, Cc.lib().lora_grad(u, x))
