"""The grad-free delta rule's scan over whole heads: remainders of a chunk, odd and even numbers of chunks, more heads than run
at once, and a sequence in two pieces with the state carried over."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,cut,Hk,Hv", [(1, 64, 0, 1, 1), (2, 128, 64, 1, 3), (1, 65, 64, 2, 2), (3, 190, 63, 2, 4), (1, 257, 192, 1, 2),
                                           (5, 97, 33, 16, 48)])
def test_scan_against_the_recurrence(B, T, cut, Hk, Hv):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    from test_gdn_chunk_gpu import recurrence
    gen = torch.Generator(device="cuda").manual_seed(T + Hv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    q, k, v = rnd(B, T, Hk, 128).bfloat16(), rnd(B, T, Hk, 128).bfloat16(), rnd(B, T, Hv, 128).bfloat16()
    g, beta = -torch.rand(B, T, Hv, generator=gen, device="cuda"), torch.rand(B, T, Hv, generator=gen, device="cuda")
    S = rnd(B, Hv, 128, 128) * 0.3
    ro, rS = recurrence(q, k, v, g, beta, S, True)
    outs = []
    for at in (slice(0, cut), slice(cut, T)):
        if at.stop > at.start:
            o, S = C.gdn_chunk_fwd(q[:, at], k[:, at], v[:, at], g[:, at], beta[:, at], S, True, 1e-6)
            outs.append(o)
    o = torch.cat(outs, 1)
    # sums of 64 and 128 terms in 32 bits, a few units of 2^-24 of the largest entry a chunk, ten times that allowed over up to
    # five chunks; outputs are rounded to 16 bits once
    assert float((S - rS).norm() / rS.norm()) < 5e-6 and float((S - rS).abs().max()) < 2e-5 * float(rS.abs().max())
    assert bool(((o - ro).abs() <= 2 ** -8 * ro.abs() + 2e-5 * ro.abs().max()).all())
    assert C.lib().kernel_status() == 0
