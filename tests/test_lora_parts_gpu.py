"""Fused projections from their adapters against the stacked operands built by tensor operations: same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,K,outs,adapted,r", [(1, 64, [64], [0], 8), (70, 128, [256, 64, 64], [0, 1, 2], 16), (333, 512, [128, 64, 40], [0, 2], 3),
                                                (129, 96, [24, 64, 8, 32], [1, 3], 5), (64, 256, [512, 512], [1], 32)])
def test_parts_equal_stacks(M, K, outs, adapted, r):
    from ferrl_b200.models.lora import FusedLoraLinear, LoraSpec
    from ferrl_b200 import ops
    torch.manual_seed(M + K)
    names = tuple("abcd"[:len(outs)])
    m = FusedLoraLinear(K, outs, names, tuple(i in adapted for i in range(len(outs))), LoraSpec(r, 2.5 * r), dtype=torch.bfloat16, device="cuda",
                        keep_transpose=M % 2 == 0)
    m.set_weight((torch.randn(sum(outs), K, device="cuda") * K ** -0.5).bfloat16())
    with torch.no_grad():
        for p in (*m.lora_A, *m.lora_B):
            p.copy_(torch.randn_like(p) * 0.1)
    x, res, dy = (torch.randn(M, n, device="cuda").bfloat16() for n in (K, sum(outs), sum(outs)))
    leaves = [*m.lora_A, *m.lora_B]

    def grads(f):
        xs, rs = x.clone().requires_grad_(), res.clone().requires_grad_()
        y = f(xs, rs)
        return [y, *torch.autograd.grad(y, [xs, rs, *leaves], dy)]
    stacked = grads(lambda a, b: ops.lora_linear(a, m.weight, *m._stacks(), wt=m.weight_t, residual=b))
    for one, two in zip(grads(m.forward), stacked):
        assert one.shape == two.shape and one.dtype == two.dtype and torch.equal(one, two)


def test_parts_inside_a_rematerialised_segment():
    """The forward runs twice and its saved operands are of the second time: same bits as without."""
    from ferrl_b200.models.lora import FusedLoraLinear, LoraSpec
    from ferrl_b200.remat import remat_segment
    torch.manual_seed(5)
    m = FusedLoraLinear(128, [256, 64], ("a", "b"), (True, True), LoraSpec(16, 32.0), dtype=torch.bfloat16, device="cuda")
    m.set_weight((torch.randn(320, 128, device="cuda") * 128 ** -0.5).bfloat16())
    with torch.no_grad():
        for p in (*m.lora_A, *m.lora_B):
            p.copy_(torch.randn_like(p) * 0.1)
    leaves = [*m.lora_A, *m.lora_B]
    x, dy = torch.randn(3, 50, 128, device="cuda").bfloat16(), torch.randn(3, 50, 320, device="cuda").bfloat16()

    def grads(f):
        xs = x.clone().requires_grad_()
        for p in leaves:
            p.grad = None
        y = f(xs)
        y.backward(dy)
        return [y, xs.grad, *(p.grad for p in leaves)]
    for one, two in zip(grads(m), grads(lambda t: remat_segment(m, t, leaves))):
        assert torch.equal(one, two)
