"""A window that would start in front of its sequence is refused where its start is known on the host; on the device nothing that
could pass for a result comes out of it, and the status word says why."""
import pytest
import torch


def test_rollout_without_a_prompt_is_refused():
    from ferrl_b200.lm_policy import LmPolicy
    from ferrl_b200.models import DenseGradModel, DenseSpec, LoraSpec
    from ferrl_b200.policy import Rollout
    from ferrl_b200.sampler import GrpoSampler
    spec = DenseSpec(vocab_size=32, hidden_size=16, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, head_dim=8,
                     intermediate_size=32, max_position_embeddings=32)
    model = DenseGradModel(spec, LoraSpec(2, 4.0))
    model.init_random(0, 0.2)
    policy = LmPolicy(model, GrpoSampler(1, 1.0))
    toks = torch.arange(10).view(2, 5)
    for score in (policy.token_logprobs, policy.token_logprobs_detached):
        with pytest.raises(ValueError, match="empty prompt"):
            score([Rollout(toks, 2, [3, 3], None), Rollout(toks[:, :3], 0, [3, 3], None)])
    assert policy.token_logprobs([Rollout(toks, 1, [4, 4], None)]).shape == (2, 4)


@pytest.mark.gpu
def test_negative_start_on_the_device():
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA device")
    from ferrl_b200 import ops
    from ferrl_b200.ops import cuda as C
    assert C.kernel_status() == 0
    x = torch.randn(3, 9, 64, device="cuda").bfloat16().requires_grad_()
    out = ops.window_rows(x, torch.tensor([2, -1, 8], device="cuda"), 5)
    out.backward(torch.ones_like(out))
    try:
        assert C.kernel_status() == C.STATUS_BAD_INDEX and "below zero" in C.status_message(C.STATUS_BAD_INDEX)
    finally:
        C.lib().reset_status()
    bad = torch.tensor([False, True, False], device="cuda")
    for t in (out, x.grad):
        assert t[bad].isnan().all() and not t[~bad].isnan().any()
    assert torch.equal(out[0], x[0, 2:7]) and C.kernel_status() == 0
