"""Prompt rows into the paged pools by one kernel: the same bytes as by copies, gathers and indexed stores."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


# prompts shorter than a page, ends on page boundaries, padding past the pool's rows, rows of odd numbers of pieces, one row a group
@pytest.mark.parametrize("P,L,ppr,G,hkv,D,dtype", [(2, 70, 3, 4, 8, 128, torch.bfloat16), (3, 64, 1, 2, 1, 8, torch.bfloat16),
                                                    (1, 1, 2, 3, 2, 64, torch.bfloat16), (5, 129, 3, 1, 3, 72, torch.bfloat16),
                                                    (2, 200, 2, 2, 4, 32, torch.float32), (2, 131, 4, 7, 5, 256, torch.bfloat16),
                                                    (2, 40, 2, 2, 1, 4, torch.bfloat16)])                     # the last: half pieces
def test_pools_are_the_same_bytes(P, L, ppr, G, hkv, D, dtype):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.models.dense import DensePagedDecoder
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(L * D)
    page = DensePagedDecoder.PAGE
    lens = torch.randint(1, L + 1, (P,), generator=gen, device="cuda")
    lens[0] = L
    full = lens // page
    k = torch.randn(P, L, hkv, D, generator=gen, device="cuda").to(dtype)
    v = torch.randn(P, L, 3 * hkv * D, generator=gen, device="cuda").to(dtype)[..., 2 * hkv * D:].unflatten(-1, (hkv, D))
    pools = lambda: [torch.full((P * ppr * (1 + G), page, hkv, D), 7.0, dtype=dtype, device="cuda")]  # noqa: E731
    dec = lambda: types.SimpleNamespace(PAGE=page, pages_per_row=ppr, k=pools(), v=pools(), group=G, batch=P * G,  # noqa: E731
                                        shared_pages=P * ppr)
    a, b = dec(), dec()
    assert C.kv_prefill_paged(a.k[0], a.v[0], k, v, full, ppr, G) == (hkv * D * k.element_size() % 16 == 0)
    DensePagedDecoder._store(a, 0, k, v, full)
    from ferrl_b200 import ops
    native, ops.native = ops.native, lambda *t: False
    try:
        DensePagedDecoder._store(b, 0, k, v, full)
    finally:
        ops.native = native
    assert torch.equal(a.k[0], b.k[0]) and torch.equal(a.v[0], b.v[0])


def test_pools_without_pages_and_negative_lengths():
    """A layout without a page is refused before anything is written; a prompt whose length the device finds below zero gets NaNs."""
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    k, v = (torch.randn(2, 70, 2, 64, device="cuda").bfloat16() for _ in range(2))
    empty = torch.zeros(0, 64, 2, 64, device="cuda", dtype=torch.bfloat16)
    for ppr in (0, -1):
        with pytest.raises(RuntimeError, match="layout"):
            C.kv_prefill_paged(empty, empty.clone(), k, v, torch.tensor([1, 1], device="cuda"), ppr, 2)
    kc, vc = (torch.zeros(2 * 2 * 3, 64, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    assert C.kernel_status() == 0
    assert C.kv_prefill_paged(kc, vc, k, v, torch.tensor([1, -1], device="cuda"), 2, 2)
    try:
        assert C.kernel_status() == C.STATUS_BAD_INDEX
    finally:
        C.lib().reset_status()
    for pool, src in ((kc, k), (vc, v)):
        first = pool[4::2]                                  # first private pages of the four rows
        assert torch.equal(first[0, :6], src[0, 64:]) and torch.equal(first[0], first[1])
        assert first[2:].isnan().all() and not pool[:4].isnan().any()
