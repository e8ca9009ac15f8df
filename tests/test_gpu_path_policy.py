"""The default choice of the kernels for the iteration passes of a one-call solve: the lean kernel from two subgames an SM on
unless some subgame may be too large for it, else the split kernels.  The names of the kernels that ran tell which; the
results must be the same bits under both policies, and the iteration timer works whichever it was."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kernels_of(fn):
    """Names of the kernels that fn launches."""
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        fn()
        torch.cuda.synchronize()
    return " ".join(e.name for e in prof.events() if "_kernel" in e.name)


def _ran(fn):
    """Which kernels ran the iteration passes: "lean" or "split"; checks that the timer recorded them."""
    from poker2_b200 import _lib

    _lib.call("p2b_cfr_iteration_timing", 1)
    try:
        names = _kernels_of(fn)
        ms = ctypes.c_float(0.0)
        assert _lib.lib().p2b_cfr_iteration_ms(ctypes.byref(ms)) == 0 and ms.value > 0.0
    finally:
        _lib.call("p2b_cfr_iteration_timing", 0)
    lean, split = "cfr_iter_kernel" in names, "split_rows_kernel" in names
    assert lean != split, names
    return "lean" if lean else "split"


@pytest.fixture
def auto_policy():
    from poker2_b200 import solver

    before = solver.set_path_policy("auto")
    yield
    solver.set_path_policy(before)


@pytest.mark.parametrize("twice_an_sm", [False, True])
def test_default_policy_by_batch_size(cuda_device, auto_policy, twice_an_sm):
    import bench
    from poker2_b200 import solver, tree as ptree

    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    boards, ranges, pot, stack = bench.make_inputs(2 * sms - (not twice_an_sm), 2)
    trees = ptree.build_trees(ptree.root_states(pot.numpy(), stack.numpy()), [0.5, 1.0], 8, max_raises=2)
    layout = solver.device_layout(trees, boards.numpy())
    rb = solver.pad_rows(ranges.to(cuda_device)).contiguous()
    scal = solver.iteration_scalars(4)
    sv = solver.SubgameSolver(layout, boards, cuda_device, exploitability=True)
    assert _ran(lambda: sv.solve(rb, scal)) == ("lean" if twice_an_sm else "split")
    got = [x.clone() for x in (sv.policy_avg, sv.regrets, sv.root_values, sv.exploitability)]
    solver.set_path_policy("lean")
    sv2 = solver.SubgameSolver(layout, boards, cuda_device, exploitability=True)
    assert _ran(lambda: sv2.solve(rb, scal)) == "lean"
    for a, b in zip(got, (sv2.policy_avg, sv2.regrets, sv2.root_values, sv2.exploitability)):
        assert torch.equal(a, b)


def test_default_policy_with_large_subgames(cuda_device, auto_policy):
    """A batch in which some subgame exceeds the lean kernel's node limit goes to the split kernels, however large it is; with
    the lean policy the general kernel takes the subgames that the lean kernel skips."""
    from poker2_b200 import solver, tree as ptree

    g = torch.Generator().manual_seed(3)
    B = 300  # more than two an SM
    pot = np.full(B, 100)
    stack = np.where(np.arange(B) % 5 == 0, 1000, 300)
    boards = torch.stack([torch.randperm(52, generator=g)[:5] for _ in range(B)])
    ranges = torch.empty(B, 2, 1326).exponential_(generator=g)
    ranges = ranges / ranges.sum(-1, keepdim=True)
    trees = ptree.build_trees(ptree.root_states(pot, stack, min_raise=2), [0.5, 1.0], 12, bb=2)
    assert np.bincount(trees.root_of).max() > 160
    layout = solver.device_layout(trees, boards.numpy())
    rb = solver.pad_rows(ranges.to(cuda_device)).contiguous()
    scal = solver.iteration_scalars(3)
    sv = solver.SubgameSolver(layout, boards, cuda_device)
    assert _ran(lambda: sv.solve(rb, scal)) == "split"
    got = [x.clone() for x in (sv.policy_avg, sv.regrets, sv.root_values)]
    solver.set_path_policy("lean")
    sv2 = solver.SubgameSolver(layout, boards, cuda_device)
    assert _ran(lambda: sv2.solve(rb, scal)) == "lean"
    for a, b in zip(got, (sv2.policy_avg, sv2.regrets, sv2.root_values)):
        assert torch.equal(a, b)
