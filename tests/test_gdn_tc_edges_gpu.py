"""Kernels of the training delta rule (csrc/kernels/gdn_tc.cu), each output row by row against float64: one chunk and several,
both widths of the scans, value heads that share a key head, decays from almost none to vanishing states."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D, C = 128, 64


def _chunked(q, k, v, g, beta, S):
    """float64 restatement by chunks; ``q, k`` normalised, heads as those of ``v``: outputs ``[B,T,H,D]`` and the last state."""
    q, k, v, g, beta = (t.transpose(1, 2) for t in (q, k, v, g, beta))
    outs = []
    for s in range(0, q.shape[2], C):
        qc, kc, vc, gc, bc = (t[:, :, s:s + C] for t in (q, k, v, g, beta))
        G = gc.cumsum(-1)
        low = torch.ones(C, C, dtype=torch.bool, device=q.device).tril()
        decay = (G[..., :, None] - G[..., None, :]).masked_fill(~low, float("-inf")).exp()
        M = torch.eye(C, dtype=q.dtype, device=q.device) + (kc @ kc.transpose(-1, -2) * decay).tril(-1) * bc[..., None]
        new = torch.linalg.solve_triangular(M, bc[..., None] * (vc - G.exp()[..., None] * (kc @ S)), upper=False)
        outs.append(G.exp()[..., None] * (qc @ S) + (qc @ kc.transpose(-1, -2) * decay) @ new)
        S = G[..., -1:, None].exp() * S + (kc * (G[..., -1:] - G).exp()[..., None]).transpose(-1, -2) @ new
    return torch.cat(outs, 2).transpose(1, 2), S


@pytest.mark.parametrize("B,n,Hk,Hv,rate,state", [
    (1, 1, 1, 1, 0.1, True), (1, 2, 1, 3, 0.0, False), (2, 5, 2, 2, 0.02, True), (1, 3, 37, 37, 0.3, True),      # 37 heads: the last of the narrow scans
    (1, 3, 19, 38, 0.3, True), (3, 2, 16, 48, 2.0, True),                                                       # the wide ones
])
def test_rows_against_float64(B, n, Hk, Hv, rate, state):
    from ferrl_b200.ops import cuda as O
    gen = torch.Generator(device="cuda").manual_seed(1000 * n + Hv)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    T = n * C
    q, k = (torch.nn.functional.normalize(rnd(B, T, Hk, D), dim=-1) for _ in range(2))
    q = q * D ** -0.5
    v, g = rnd(B, T, Hv, D), -torch.rand(B, T, Hv, generator=gen, device="cuda") * rate
    beta = torch.rand(B, T, Hv, generator=gen, device="cuda")
    S0 = rnd(B, Hv, D, D) * 0.1 if state else None
    dO, dS1 = rnd(B, T, Hv, D), (rnd(B, Hv, D, D) * 0.1 if state else None)
    out, S1, *saved = O.lib().gdn_tc_fwd(q, k, v, g, beta, S0)
    dq, dk, dv, dbeta, dG, dS0 = O.lib().gdn_tc_bwd(q, k, v, beta, *saved, dO, dS1)
    again = O.lib().gdn_tc_bwd(q, k, v, beta, *saved, dO, dS1)
    for a, b in zip((dq, dk, dv, dbeta, dG, dS0), again):
        assert torch.equal(a, b)            # fixed summation order

    leaves = [t.double().repeat_interleave(Hv // t.shape[2], 2).requires_grad_() for t in (q, k)] + \
        [t.double().requires_grad_() for t in (v, g, beta, S0 if state else torch.zeros(B, Hv, D, D, device="cuda"))]
    ro, rS = _chunked(*leaves)
    ((ro * dO).sum() + ((rS * dS1).sum() if state else 0)).backward()
    rq, rk, rv, rg, rb, rS0 = (t.grad for t in leaves)
    dg = dG.view(B, n, C, Hv).flip(2).cumsum(2).flip(2).reshape(B, T, Hv)
    # operands are read with 10 bits behind the leading one (2^-10, truncated): products of two are 2^-9 off at most, and what
    # reaches a gradient has passed four of them; rows are held against the typical row, sums of 64 signed ones more loosely
    for name, a, r, tol in (("out", out, ro, 8e-3), ("S", S1, rS, 8e-3), ("dq", dq, rq, 1.6e-2), ("dk", dk, rk, 1.6e-2), ("dv", dv, rv, 1.6e-2),
                            ("dS0", dS0, rS0, 1.6e-2)):
        err, size = (a.double() - r).norm(dim=-1), r.norm(dim=-1)
        assert torch.isfinite(a).all(), name
        assert (err <= tol * (size + size.square().mean().sqrt()) + 1e-6).all(), (name, float((err / (size + size.mean())).max()))
    for name, a, r in (("dg", dg, rg), ("dbeta", dbeta, rb)):
        assert (a.double() - r).abs().max() <= 2e-2 * float(r.square().mean().sqrt() + r.abs().max()), name
