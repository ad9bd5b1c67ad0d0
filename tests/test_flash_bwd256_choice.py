"""Which kernels take the attention backward at head dim 256: many short rows go to the warp-level ones, everything else to tcgen05."""
import pytest
import torch


@pytest.mark.parametrize("B,S,Hq,Hkv,tc", [(1, 64, 8, 2, True), (8, 1, 8, 2, True), (16, 16, 16, 2, True), (8, 48, 24, 4, True), (4, 64, 32, 8, True),
                                           (4, 1, 32, 8, False), (8, 64, 32, 8, False), (16, 64, 24, 4, False), (16, 64, 32, 8, False),
                                           (16, 65, 32, 8, True), (64, 4096, 64, 8, True), (1, 1, 1, 1, True)])
def test_choice(B, S, Hq, Hkv, tc):
    from ferrl_b200.ops import cuda as C
    assert C.lib().flash_bwd256_tc_better(B, S, Hq, Hkv) == tc


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,Hq,Hkv", [(4, 3, 32, 8), (8, 64, 32, 8), (8, 65, 32, 8)])
def test_short_rows(B, S, Hq, Hkv):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C, eager
    gen = torch.Generator(device="cuda").manual_seed(S)
    q, k, v, do = (torch.randn(B, S, h, 256, generator=gen, device="cuda").bfloat16() for h in (Hq, Hkv, Hkv, Hq))
    o, lse = C.lib().flash_fwd(q, k, v, 0.0625, True, 0, 0, 0)
    run = lambda variant: C.lib().flash_bwd(q, k, v, o, lse, do, 0.0625, True, 0, 0, variant)  # noqa: E731
    refs = [t.float().requires_grad_() for t in (q, k, v)]
    eager.attention(*refs, scale=0.0625, causal=True).backward(do.float())
    for a, w, r in zip(run(0), run(1), refs):
        assert torch.equal(a, w) == (not C.lib().flash_bwd256_tc_better(B, S, Hq, Hkv))
        # 8-bit operands P and dS, 2^-9 each at random, and a 16-bit result
        assert float((a.float() - r.grad).abs().max()) <= 2e-2 * float(r.grad.abs().max())
    assert C.kernel_status() == 0
