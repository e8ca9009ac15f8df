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


def _busy(device):
    """Half a second or so of work on the current stream, and the event behind it."""
    torch.cuda.synchronize(device)
    torch.cuda._sleep(1 << 30)
    behind = torch.cuda.Event()
    behind.record()
    return behind


def test_an_iteration_does_not_wait_for_the_stream(cuda_device):
    """`TScalars.update` and a whole `cfr_iteration` only enqueue work: both return while what came before is still running."""
    from poker2_b200 import fused_cfr, step_evaluator, tree as ptree

    scalars = fused_cfr.TScalars(cuda_device)
    scalars.update(1, 1.5, 0.0, 1.0, 2.0)
    behind = _busy(cuda_device)
    scalars.update(3, 1.5, 0.5, 9.0, 16.0)
    assert not behind.query()

    trees = ptree.build_trees(ptree.root_states(torch.tensor([100]).numpy(), torch.tensor([400]).numpy()), [0.5, 1.0], 8, max_raises=2)
    ranges = torch.rand(1, 2, 1326, generator=torch.Generator().manual_seed(1))
    ev = step_evaluator.StepCFREvaluator(trees, torch.tensor([[0, 5, 17, 30, 51]]).numpy(), ranges, cuda_device, iterations=4)
    ev.initialize_policy_and_beliefs()
    ev.set_leaf_values(0)
    ev.compute_expected_values()
    for t in range(2):
        ev.cfr_iteration(t)  # every first-time set-up is behind
    behind = _busy(cuda_device)
    ev.cfr_iteration(2)
    assert not behind.query()


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("where", ["cuda", "cpu"])
@pytest.mark.parametrize("old,new", [(9.0, 16.0), (0.0, 1.0), (1.0, 0.0)])
def test_scalars_of_an_iteration(cuda_device, dtype, where, old, new):
    """Every field as its expression gives it in Python floats, rounded to the scalars' type; with no new weight the two
    quotients by it stay as they were."""
    from poker2_b200 import fused_cfr

    s = fused_cfr.TScalars(cuda_device if where == "cuda" else torch.device("cpu"), dtype)
    s.update(1, 1.0, 1.0, 3.0, 4.0)
    s.update(7, 1.5, -1.0, old, new)
    total = old + new
    want = dict(t_alpha_num=7 ** 1.5, t_beta_num=7 ** -1.0, t_alpha_den=7 ** 1.5 + 1.0, t_beta_den=7 ** -1.0 + 1.0, mix_old=old,
                mix_new=new, mix_total=total, mix_inv_total=1.0 / total,
                mix_onon=total / new if new else 7.0 / 4.0, mix_oon=old / new if new else 3.0 / 4.0)
    for name, value in want.items():
        assert torch.equal(getattr(s, name).cpu(), torch.tensor(value, dtype=dtype)), name
    assert s.t_tensor.item() == 7


@pytest.mark.parametrize("spoil", ["rows", "type", "strides"])
def test_state_arrays_of_another_form_are_refused(cuda_device, spoil):
    """Arrays that a caller hands to a step, or puts in place of the evaluator's own, reach the kernels as bare pointers: too few
    rows, another type or other strides are refused; what can be copied into place (a policy's or beliefs' strides) is."""
    from poker2_b200 import step_evaluator, tree as ptree

    trees = ptree.build_trees(ptree.root_states(torch.tensor([100]).numpy(), torch.tensor([400]).numpy()), [0.5, 1.0], 8, max_raises=2)
    ranges = torch.rand(1, 2, 1326, generator=torch.Generator().manual_seed(1))
    ev = step_evaluator.StepCFREvaluator(trees, torch.tensor([[0, 5, 17, 30, 51]]).numpy(), ranges, cuda_device, iterations=4)
    ev.evaluate_cfr()

    def spoilt(x):
        if spoil == "rows":
            return x[:-1].clone()
        if spoil == "type":
            return x.double()
        wide = torch.zeros(*x.shape[:-1], x.shape[-1] + 2, device=x.device)
        wide[..., :-2] = x
        return wide[..., :-2]

    if spoil == "strides":
        ev.compute_expected_values()
        want = ev.latest_values.clone()
        ev.compute_expected_values(policy=spoilt(ev.policy_probs), beliefs=spoilt(ev.beliefs))
        assert torch.equal(ev.latest_values, want)
    else:
        for kw in ({"policy": spoilt(ev.policy_probs)}, {"beliefs": spoilt(ev.beliefs)}):
            with pytest.raises(AssertionError):
                ev.compute_expected_values(**kw)
        with pytest.raises(AssertionError):
            ev.set_leaf_values(0, beliefs=spoilt(ev.beliefs))
    with pytest.raises((AssertionError, RuntimeError)):
        ev.compute_expected_values(values=spoilt(ev.latest_values))
    for name in ("latest_values", "beliefs", "self_reach", "self_reach_avg", "beliefs_avg", "policy_probs", "policy_probs_avg",
                 "cumulative_regrets", "regret_weight_sums", "uniform_policy"):
        own = getattr(ev, name)
        setattr(ev, name, spoilt(own))
        with pytest.raises((AssertionError, RuntimeError)):
            ev.cfr_iteration(3)
        setattr(ev, name, own)
    ev.cfr_iteration(3)
