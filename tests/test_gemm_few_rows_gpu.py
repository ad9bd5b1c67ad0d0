"""Products of at most 16 rows (csrc/gemm/few_rows.cu) against float32: ragged rows, columns and sums, tiles of
either height, residuals, the GLU epilogue, views, and the general entry point that chooses the kernel by itself."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _ok(got, ref):
    # sums in 32 bits of exact products of 16-bit values, rounded once to 16: half a unit of 8 bits
    assert torch.isfinite(got).all()
    assert ((got.float() - ref).abs() <= 2 ** -8 * ref.abs() + 1e-5 * ref.abs().max()).all()


@pytest.mark.parametrize("M", [1, 2, 7, 8, 9, 16])
@pytest.mark.parametrize("N", [1, 8, 15, 16, 17, 200, 4736, 4800])
@pytest.mark.parametrize("K", [8, 120, 128, 136, 1024, 1160, 2056])
@pytest.mark.parametrize("rows_of_w", [0, 8, 16])
def test_against_float32(M, N, K, rows_of_w):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(M * N + K)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    x, w, res = rnd(M, K + 8)[:, :K], rnd(N, K + 16)[:, :K], rnd(M, N + 3)[:, :N]
    ref = x.float() @ w.float().T
    _ok(C.lib().gemm_few_rows(x, w, None, -1, 0.0, 0.0, rows_of_w), ref)
    _ok(C.lib().gemm_few_rows(x, w, res, -1, 0.0, 0.0, rows_of_w), ref + res.float())


@pytest.mark.parametrize("M", [1, 5, 8, 13])
@pytest.mark.parametrize("N,K", [(16, 64), (48, 1032), (4752, 128), (6144, 512)])
@pytest.mark.parametrize("act", [0, 1, 2])
def test_gated(M, N, K, act):
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(N + act)
    x, w = torch.randn(M, K, generator=gen, device="cuda").bfloat16(), (torch.randn(N, K, generator=gen, device="cuda") * K ** -0.5).bfloat16()
    g, u = (x.float() @ w.float().T).view(M, N // 16, 2, 8).unbind(2)
    if act == 2:
        g, u = g.clamp(max=7.0), u.clamp(-7.0, 7.0)
        ref = g * torch.sigmoid(1.702 * g) * (u + 1)
    else:
        ref = (torch.nn.functional.silu(g) if act == 0 else torch.nn.functional.gelu(g, approximate="tanh")) * u
    ref = ref.reshape(M, N // 2)
    args = (1.702, 7.0) if act == 2 else (0.0, 0.0)
    _ok(C.lib().gemm_few_rows(x, w, None, act, *args), ref)
    _ok(C.lib().gemm_glu(x, w, act, True, *args), ref)


@pytest.mark.parametrize("M,N,K", [(1, 1536, 1024), (8, 1024, 3072), (16, 512, 256), (3, 33, 64)])
def test_chosen_in_a_graph_of_dependent_launches(M, N, K):
    """A chain whose activations change from replay to replay: nothing but the weights may be read early."""
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    n = max(N, K)
    ws = [(rnd(n, n) * n ** -0.5).bfloat16() for _ in range(6)]
    x = rnd(M, n).bfloat16()
    step = lambda y, w: C.lib().gemm(y, w, None, None, y, False, 0, 0, 0, None, 0, 0, True)  # noqa: E731

    def chain():
        y = x
        for w in ws:
            y = step(y, w)
        return y
    chain()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    for seed in range(3):
        x.copy_(torch.randn(M, n, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda"))
        graph.replay()
        torch.cuda.synchronize()
        y = x
        for w in ws:
            y = (y.float() @ w.float().T + y.float()).bfloat16()
        assert float((out.float() - y.float()).norm() / y.float().norm()) < 1e-2      # six roundings to 16 bits
