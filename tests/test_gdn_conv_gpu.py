"""Causal convolution kernels at the edges of their runs of tokens and groups of channels, against float64 autograd."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,C,K,wide,left", [
    (2, 31, 64, 4, 96, True), (1, 32, 64, 4, 64, False), (3, 33, 2048, 4, 2056, True),    # around a run of 32 tokens, strided rows
    (2, 129, 24, 3, 24, True), (1, 5, 8, 8, 16, True), (2, 70, 16, 1, 16, False),          # few channels, widest and narrowest kernel
    (1, 1, 8, 4, 8, True), (2, 37, 100, 4, 108, True), (2, 9, 20, 2, 21, False),           # one token; no whole groups of eight
    (1, 30, 4096, 4, 4096, True), (1, 100, 4096, 4, 4104, False), (4, 401, 1024, 4, 1024, True), (3, 1103, 512, 3, 520, True),   # runs of 1, 4, 16
    (2, 3005, 4096, 4, 4104, True), (1, 6001, 4000, 2, 4000, False),                       # groups of eight channels
])
def test_conv_at_run_and_group_edges(B, L, C, K, wide, left):
    from ferrl_b200.ops import cuda as Cc
    g = torch.Generator(device="cuda").manual_seed(L * C + K)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w, dy = rnd(B, L, wide)[..., :C], rnd(C, K), rnd(B, L, C)
    ctx = rnd(B, C, K - 1) if left else None
    xr = x.double().requires_grad_()
    pad = torch.cat([(ctx if left else x.new_zeros(B, C, K - 1)).double(), xr.transpose(1, 2)], -1)
    pre = sum(w.double()[:, j, None] * pad[..., j:j + L] for j in range(K)).transpose(1, 2)
    # the kernel rounds `pre` to bf16 once (2^-9 of it) and silu' is at most 1.1, silu'' at most 0.5; outputs are rounded once
    for act in (False, True):
        ref = torch.nn.functional.silu(pre) if act else pre
        y = Cc.lib().gdn_conv_fwd(x, w, ctx, act)
        assert bool(((y.double() - ref).abs() <= 2 ** -8 * ref.abs() + 1.2 * 2 ** -8 * pre.abs() + 1e-6).all())
        (dref,) = torch.autograd.grad(ref, xr, dy.double(), retain_graph=True)
        scale = sum(w.double()[:, j].abs() * torch.nn.functional.pad((dy.double().abs() * (1.1 + 0.5 * pre.detach().abs() if act else 1)),
                                                                    (0, 0, 0, K - 1))[:, K - 1 - j:K - 1 - j + L] for j in range(K))
        dx = Cc.lib().gdn_conv_bwd(x, w, ctx, dy, act)
        assert bool(((dx.double() - dref).abs() <= 2 ** -8 * dref.abs() + 2 ** -8 * scale + 1e-6).all())


@pytest.mark.no_canary
def test_short_inputs_take_little_more_than_a_launch():
    """40 tokens of 3072 channels: 3.1 us beside 2.4 for an empty pass in a chain; 5.1 with eight channels a thread."""
    from ferrl_b200.ops import cuda as Cc
    xs, w = [torch.randn(1, 40, 3072, device="cuda").bfloat16() for _ in range(8)], torch.randn(3072, 4, device="cuda").bfloat16()

    def us(f):
        for x in xs:
            f(x)
        g, ts = torch.cuda.CUDAGraph(), []
        with torch.cuda.graph(g):
            for _ in range(4):
                for x in xs:
                    f(x)
        for _ in range(9):
            a, b = torch.cuda.Event(True), torch.cuda.Event(True)
            a.record()
            g.replay()
            b.record()
            torch.cuda.synchronize()
            ts.append(a.elapsed_time(b) * 1e3 / 32)
        return sorted(ts)[4]
    assert us(lambda x: Cc.lib().gdn_conv_fwd(x, w, None, True)) < 1.6 * us(lambda x: Cc.lib().rmsnorm(x[:, :1], None, None, None, 1e-6, False))
