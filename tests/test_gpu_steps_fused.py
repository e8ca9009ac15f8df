"""Edges of the kernels that do a whole step of the step-by-step evaluator (tests/test_gpu_step_evaluator.py holds them to the
upstream state) and of the ranker's int64 entry points."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("actions", [1, 8, 9, 17])
def test_seen_policy_for_any_number_of_actions(cuda_device, actions):
    """`p2b_steps_seen` takes eight children at a time: one parent with `actions` children against the one-for-one kernel."""
    from poker2_b200 import _lib, fused_cfr

    g = torch.Generator(device=cuda_device).manual_seed(actions)
    M, H = 1 + actions, 1326
    beliefs = torch.rand(M, 2, H, device=cuda_device, generator=g)
    policy = torch.rand(M, H, device=cuda_device, generator=g)
    one = lambda *v: torch.tensor(v, dtype=torch.int64, device=cuda_device)  # noqa: E731
    offsets, count, to_act, got = one(1), one(actions), one(1), torch.zeros(M, H, device=cuda_device)
    p = _lib.ptr
    _lib.call("p2b_steps_seen", p(beliefs), p(policy), p(to_act), p(offsets), p(count), p(got), 1, _lib.stream_ptr(cuda_device))
    marginal = (beliefs[0, 1] * policy[1:]).contiguous()
    parents = torch.zeros(actions, dtype=torch.int64, device=cuda_device)
    want = fused_cfr.unblocked_mass_ratio_indirect_triton(marginal, beliefs[:1, 1].contiguous(), parents)
    assert torch.equal(got[1:], want) and not got[0].any()


def test_compare_reads_int64_ids_like_int16(cuda_device):
    from poker2_b200 import rules

    g = torch.Generator(device=cuda_device).manual_seed(9)
    hands = torch.rand(1025, 52, device=cuda_device, generator=g).argsort(dim=1)[:, :14].reshape(1025, 2, 7)
    assert torch.equal(rules.compare_7_cards_single_batch(hands), rules.compare_7_cards_single_batch(hands.to(torch.int16)))
