"""Which gates of the gated RMSNorm go to the kernels where they lie, and which are copied first (the kernels are recorded, not run)."""
from types import SimpleNamespace

import pytest
import torch

from ferrl_b200.ops import cuda as C


@pytest.mark.parametrize("pitch,off,H,dtype,in_place", [
    (400, 0, 128, torch.bfloat16, True), (400, 8, 128, torch.bfloat16, True),     # rows on 16 bytes
    (390, 0, 128, torch.bfloat16, False), (404, 0, 128, torch.bfloat16, False),   # pitches off 16 bytes
    (400, 3, 128, torch.bfloat16, False), (400, 4, 128, torch.bfloat16, False),   # places off 16 bytes
    (391, 3, 100, torch.bfloat16, True), (391, 3, 128, torch.float32, True),      # entry by entry wherever they lie
    (384, 0, 128, torch.bfloat16, True),                                          # contiguous
])
@pytest.mark.parametrize("grad", [False, True])
def test_gates_off_16_bytes_are_copied(monkeypatch, pitch, off, H, dtype, in_place, grad):
    n, per = 5, 3
    base = torch.zeros(n * pitch + 64, dtype=dtype)
    base = base[-base.data_ptr() // base.element_size() % 16:]                    # starts on 16 bytes
    gate = base[off:off + n * pitch].as_strided((n, per, H), (pitch, H, 1), base.storage_offset() + off)
    x, w, seen = torch.ones(n, per, H, dtype=dtype, requires_grad=grad), torch.ones(H, dtype=dtype), []
    fake = SimpleNamespace(rmsnorm=lambda x, res, w, g, eps, zc: (seen.append(g) or torch.zeros_like(x), None),
                           rmsnorm_gated_bwd=lambda x, g, w, dy, eps: (seen.append(g) or torch.zeros_like(x), torch.zeros_like(x)))
    monkeypatch.setattr(C, "lib", lambda: fake)
    y = C.rmsnorm_gated(x, gate, w, 1e-6)
    if grad:
        y.backward(torch.ones_like(y))
    assert len(seen) == 1 + grad
    for g in seen:
        assert (g.data_ptr() == gate.data_ptr()) == in_place and (in_place or g.is_contiguous())
