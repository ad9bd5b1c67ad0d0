"""The gated shared expert in one kernel, forward and backward, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows on either side of a block's eight, widths on either side of a warp's 256, one piece
@pytest.mark.parametrize("T,H", [(1, 8), (7, 256), (9, 264), (128, 2048), (513, 1000), (33, 5120)])
def test_gated_sum_and_gradients(T, H):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.models.moe import add_shared
    gen = torch.Generator(device="cuda").manual_seed(T * H)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x, y, sh = (rnd(T, H).bfloat16().requires_grad_() for _ in range(3))
    w, dy = (rnd(1, H) * H ** -0.5).bfloat16(), rnd(T, H).bfloat16()
    out = add_shared(x, w, y, sh)
    out.backward(dy)
    x64, y64, sh64 = (t.detach().double().requires_grad_() for t in (x, y, sh))
    ref = y64 + torch.sigmoid(x64 @ w.double().t()) * sh64
    ref.backward(dy.double())
    # the logit, the gate, its product and the sum round to 8 bits each: the logit's rounding moves the gate by at most a quarter of it
    logit = (x64 @ w.double().t()).detach().abs()
    gate_err = 2 ** -9 + (logit * 2 ** -9 + 2 ** -20) / 4
    bound = gate_err * sh64.detach().abs() + 2 ** -8 * (sh64.detach().abs() + ref.detach().abs()) + 1e-6
    assert bool(((out - ref).abs() <= bound).all())
    assert torch.equal(y.grad, dy)
    assert bool(((sh.grad - sh64.grad).abs() <= gate_err * dy.double().abs() + 2 ** -8 * sh64.grad.abs() + 1e-6).all())
    dot = (dy.double() * sh64.detach()).sum(-1, keepdim=True).abs()
    slope = dot * gate_err + (dy.double() * sh64.detach()).abs().sum(-1, keepdim=True) * 2 ** -20
    assert bool(((x.grad - x64.grad).abs() <= slope * w.double().abs() + 2 ** -8 * x64.grad.abs() + 1e-6).all())


def test_a_trained_gate_keeps_its_gradient():
    from ferrl_b200.models.moe import add_shared
    x, y, sh = (torch.randn(5, 64, device="cuda").bfloat16() for _ in range(3))
    w = torch.randn(1, 64, device="cuda").bfloat16().requires_grad_()
    add_shared(x, w, y, sh).sum().backward()
    assert w.grad is not None and bool(w.grad.abs().sum() > 0)
