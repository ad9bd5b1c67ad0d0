"""Training delta rule between 16-bit activations: packing, padding and their derivatives against the tensor operations."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,T,Hk,Hv,wide,off", [(1, 1, 1, 1, 384, 0), (2, 63, 1, 3, 644, 4), (1, 64, 2, 2, 770, 2), (2, 130, 2, 6, 1288, 8), (3, 65, 4, 4, 1537, 1)])
def test_packed_matches_the_tensor_operations(B, T, Hk, Hv, wide, off):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(T * Hv + wide)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    y = rnd(B, T, wide).bfloat16()[..., off:off + (2 * Hk + Hv) * 128].requires_grad_()
    g, beta, S0 = -torch.rand(B, T, Hv, generator=gen, device="cuda"), torch.rand(B, T, Hv, generator=gen, device="cuda"), rnd(B, Hv, 128, 128) * 0.1
    do, ds = rnd(B, T, Hv, 128).bfloat16(), rnd(B, Hv, 128, 128)

    def grads(cast):
        leaf = y.detach().clone() if off % 4 else y.detach()
        leaves = [leaf.requires_grad_(), g.clone().requires_grad_(), beta.clone().requires_grad_(), S0.clone().requires_grad_()]
        q, k, v = (cast(t.unflatten(-1, (-1, 128))) for t in leaves[0].split([Hk * 128, Hk * 128, Hv * 128], -1))
        o, S = C.gdn_chunk_tc(q, k, v, *leaves[1:])
        return [o, S, *torch.autograd.grad([o, S], leaves, [do.to(o.dtype), ds])]

    # 32-bit inputs take the tensor operations around the same chunk kernels; what differs is the order of 32-bit sums in the
    # L2 norms, which the kernels' 10-bit operands (cut, not rounded) may turn into 2^-10 of a term, and one rounding to 16 bits
    for a, b in zip(grads(lambda t: t), grads(lambda t: t.float())):
        assert float((a.double() - b.double()).norm()) <= 4e-3 * float(b.double().norm()) + 1e-6
        assert float((a.double() - b.double()).abs().max()) <= 2e-2 * float(b.double().abs().max()) + 1e-6
