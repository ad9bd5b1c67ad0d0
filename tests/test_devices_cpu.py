"""Operands on different devices: the fused kernels leave such a call to the operators, which refuse it."""
import torch


def test_mixed_devices_are_left_to_the_operators():
    from ferrl_b200.ops import cuda as C
    there = lambda *s: torch.zeros(*s, dtype=torch.bfloat16, device="meta")  # noqa: E731
    here = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)  # noqa: E731
    assert C.gate_mul(there(2, 8), here(2, 8)) is None and C.gate_mul(here(2, 8), there(2, 8)) is None
    assert C.window_rows(there(2, 4, 8), torch.zeros(2, dtype=torch.int64), 2) is None
    for i in range(1, 4):
        ts = [here(*s) if i == j else there(*s) for j, s in enumerate([(3, 8), (1, 8), (3, 8), (3, 8)])]
        assert C.moe_shared(*ts) is None
