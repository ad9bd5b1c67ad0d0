"""The sigmoid gate on an attention's output, forward and backward, against float64 and on gates inside wider rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# one piece, rows that end inside a block, a row stride that is not the width; the last two keep the operators
@pytest.mark.parametrize("shape,wide,native", [((1, 1, 8), 0, True), ((2, 7, 264), 8, True), ((3, 129, 4096), 6144, True), ((0, 5, 64), 8, True),
                                               ((2, 3, 64), 4, False), ((2, 5, 60), 0, False)])
def test_gate(shape, wide, native):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(shape[-1])
    W = shape[-1]
    a = torch.randn(*shape, generator=gen, device="cuda").bfloat16().requires_grad_()
    rows = (torch.randn(*shape[:2], W + wide, generator=gen, device="cuda") * 3).bfloat16().requires_grad_()
    gate, dy = rows[..., wide:], torch.randn(*shape, generator=gen, device="cuda").bfloat16()
    out = C.gate_mul(a, gate)
    assert (out is not None) == native
    if not native:
        return
    out.backward(dy)
    a64, g64 = a.detach().double().requires_grad_(), gate.detach().double().requires_grad_()
    ref = a64 * torch.sigmoid(g64)
    ref.backward(dy.double())
    # the gate rounds to 8 bits and its product does; the gate's gradient rounds once after a few sums in 32 bits
    assert bool(((out - ref).abs() <= 2 ** -7 * ref.abs() + 1e-30).all())
    assert bool(((a.grad - a64.grad).abs() <= 2 ** -7 * a64.grad.abs() + 1e-30).all())
    assert bool(((rows.grad[..., wide:] - g64.grad).abs() <= 2 ** -8 * g64.grad.abs() + 2 ** -20 * (dy * a.detach()).abs()).all())
    assert not wide or not bool(rows.grad[..., :wide].any())
