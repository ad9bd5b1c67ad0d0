"""Routed experts with enough rows that the call itself puts the grouped products on pairs of SMs: plan with spare tiles, buffers that
nothing initialises, rows gathered sparsely, forward and backward, with the weights' transposes at hand or not; against float32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 256 rows an expert; 115, where only the blocks of 16 rows with a token are gathered; an expert without tokens
@pytest.mark.parametrize("E,T,k,empty", [(8, 2048, 2, False), (32, 1840, 2, False), (8, 2048, 2, True)])
@pytest.mark.parametrize("transposes", [False, True])
def test_against_float32(E, T, k, empty, transposes):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    H, I = 2048, 768
    gen = torch.Generator(device="cuda").manual_seed(E)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    gate_up, down = (rnd(E, 2 * I, H) * H ** -0.5).bfloat16(), (rnd(E, H, I) * I ** -0.5).bfloat16()
    x, sc, dy = rnd(T, H).bfloat16(), rnd(T, k).abs() + 0.1, rnd(T, H).bfloat16()
    pick = torch.rand(T, E, generator=gen, device="cuda")
    if empty:
        pick[:, 3] = -1
    idx = pick.topk(k, 1).indices.int()
    counts = torch.bincount(idx.flatten().long(), minlength=E).int()
    assert counts.sum() * 2 * I * H >= 6e9 and counts.sum() >= 112 * E
    t = [w.transpose(1, 2).contiguous() if transposes else None for w in (gate_up, down)]
    got = []
    xg, sg = x.clone().requires_grad_(), sc.clone().requires_grad_()
    # memory that the buffers are cut from holds NaNs: a row that is read without having been written shows
    junk = [torch.full((1 << 27,), float("nan"), device="cuda", dtype=torch.bfloat16) for _ in range(4)]
    del junk
    out = C.moe_experts(xg, sg, idx, counts, gate_up, down, "silu", *t)
    out.backward(dy)
    got = [out.detach(), xg.grad, sg.grad]
    xr, sr = x.float().requires_grad_(), sc.clone().requires_grad_()
    ref = torch.zeros(T, H, device="cuda")
    for e in range(E):
        at = (idx == e).nonzero()
        g, u = (xr[at[:, 0]] @ gate_up[e].float().T).chunk(2, -1)
        ref = ref.index_add(0, at[:, 0], (torch.nn.functional.silu(g) * u) @ down[e].float().T * sr[at[:, 0], at[:, 1], None])
    ref.backward(dy.float())
    assert C.kernel_status() == 0
    for a, r in zip(got, (ref.detach(), xr.grad, sr.grad)):
        # four to six roundings to 8 bits on the way, 2^-9 each at random, through matrices of norm about one
        assert torch.isfinite(a).all() and float((a.float() - r).norm() / r.norm()) < 1e-2
