"""Gradients that arrive as packed views off a 16-byte boundary (out of a flat buffer, from a hook): the same bits as aligned ones."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _off(t):
    return torch.cat([t.new_zeros(1), t.reshape(-1)])[1:].view(t.shape)


@pytest.mark.parametrize("name", ["window_rows", "gate_mul", "moe_shared"])
def test_unaligned_gradient(name):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    if name == "window_rows":
        ins, start = [rnd(2, 9, 72)], torch.tensor([1, 6], device="cuda")
        f = lambda x: C.window_rows(x, start, 5)  # noqa: E731
    elif name == "gate_mul":
        ins, f = [rnd(3, 5, 72), rnd(3, 5, 72)], C.gate_mul
    else:
        ins, w = [rnd(15, 72) for _ in range(3)], rnd(1, 72)
        f = lambda x, y, sh: C.moe_shared(x, w, y, sh)  # noqa: E731
    got = []
    for move in (lambda t: t, _off):
        ins = [t.detach().requires_grad_() for t in ins]
        out = f(*ins)
        dy = move(torch.randn(out.shape, generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").bfloat16())
        assert dy.is_contiguous() and (dy.data_ptr() % 16 == 0) == (move is not _off)
        out.backward(dy)
        got.append([t.grad for t in ins])
    assert all(torch.equal(a, b) for a, b in zip(*got))
