"""A chain of products of few rows as a decode step has them, narrow to wide and back with the weights' own sizes, so that tiles of
eight rows of the weight are launched early beside what runs (csrc/gemm/few_rows.cu): activations change from replay to replay."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of 8 early; tiles of 16 early and not; short sums; rows for two groups
@pytest.mark.parametrize("M,N,K", [(8, 1024, 3072), (1, 1032, 2048), (1, 1040, 2048), (5, 2064, 2048), (8, 2072, 2048), (16, 512, 2048), (3, 264, 72)])
def test_chain_of_a_weights_own_sizes(M, N, K):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as C
    gen = torch.Generator(device="cuda").manual_seed(N)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    down = [(rnd(N, K) * K ** -0.5).bfloat16() for _ in range(3)]
    up = [(rnd(K, N) * N ** -0.5).bfloat16() for _ in range(3)]
    x = rnd(M, K).bfloat16()
    step = lambda y, w: C.lib().gemm(y, w, None, None, None, False, 0, 0, 0, None, 0, 0, True)  # noqa: E731

    def chain():
        y = x
        for d, u in zip(down, up):
            y = step(step(y, d), u)
        return y
    chain()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    for seed in range(3):
        x.copy_(torch.randn(M, K, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda"))
        graph.replay()
        torch.cuda.synchronize()
        y = x
        for d, u in zip(down, up):
            y = (y.float() @ d.float().T).bfloat16()
            y = (y.float() @ u.float().T).bfloat16()
        # six roundings to 8 bits, at random 2^-9 of a value each, passed on by matrices of norm about one (two, at most)
        assert float((out.float() - y.float()).norm() / y.float().norm()) < 1e-2
