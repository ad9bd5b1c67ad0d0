"""The GatedDeltaNet convolution by words of four channels: the same bits as channel by channel."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# runs of 8, 16 and 32 tokens with a remainder, inputs shorter than the taps, rows that end inside a group of tokens
@pytest.mark.parametrize("B,L,C,K,left,act", [(1, 1031, 1028, 4, False, True), (2, 333, 8192, 4, True, True), (600, 2, 1024, 4, True, True),
                                              (5, 1, 262144, 3, False, True), (3, 129, 4096, 1, True, False),
                                              (2, 70, 8192, 7, True, True), (1, 2500, 8192, 4, True, True),
                                              (2, 259, 2052, 8, False, False), (4, 97, 4100, 2, True, True),
                                              (1, 260, 8192, 5, True, False), (1, 2049, 640, 6, False, True)])
def test_words_and_channels_agree(B, L, C, K, left, act):
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200.ops import cuda as Cc
    lib = Cc.lib()
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(L + C + K)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g).to(torch.bfloat16)
    wide = rnd(B, L, C + 8)
    w, dy = rnd(C, K), rnd(B, L, C)
    ctx = rnd(B, C, K - 1) if left else None
    x, odd = wide[..., 4:C + 4], torch.empty(B * L * (C + 8) + 1, device=dev, dtype=torch.bfloat16)[1:].view(B, L, C + 8)
    odd.copy_(wide)                                          # the same rows, two bytes off the boundary
    odd = odd[..., 4:C + 4]
    y, yo = lib.gdn_conv_fwd(x, w, ctx, act), lib.gdn_conv_fwd(odd, w, ctx, act)
    assert torch.equal(y.view(torch.int16), yo.view(torch.int16))
    d, do = lib.gdn_conv_bwd(x, w, ctx, dy, act), lib.gdn_conv_bwd(odd, w, ctx, dy, act)
    assert torch.equal(d.view(torch.int16), do.view(torch.int16))
    # taps that lie off a boundary
    wo = torch.empty(C * K + 1, device=dev, dtype=torch.bfloat16)[1:].view(C, K)
    wo.copy_(w)
    assert torch.equal(y.view(torch.int16), lib.gdn_conv_fwd(x, wo, ctx, act).view(torch.int16))
