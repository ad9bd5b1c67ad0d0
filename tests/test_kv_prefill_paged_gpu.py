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
