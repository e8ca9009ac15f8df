"""The split kernels (a pass as one kernel over all nodes and one over all hands) against the general kernel, which walks
the tree: equal bits in every output, over the batch sizes at which the column kernel changes its shape, the widest
nodes and the solve options that change what a pass does."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def auto_policy(cuda_device):
    from poker2_b200 import solver

    before = solver.set_path_policy("auto")
    yield
    solver.set_path_policy(before)


def _both(cuda_device, B, *, bins=(0.5, 1.0), cap=2, iterations=5, cfr_type="discounted", deep=False, **kw):
    """The same solve with the full scratch area and with the minimal one, which keeps every pass in the general kernel."""
    import bench
    from poker2_b200 import solver, tree as ptree

    boards, ranges, pot, stack = bench.make_inputs(B, 11 + B)
    if deep:
        pot, stack = torch.full((B,), 60), torch.full((B,), 500)
    trees = ptree.build_trees(ptree.root_states(pot.numpy(), stack.numpy()), list(bins), 8, max_raises=cap)
    layout = solver.device_layout(trees, boards.numpy())
    rb = solver.pad_rows(ranges.to(cuda_device)).contiguous()
    scal = solver.iteration_scalars(iterations, cfr_type=cfr_type, dcfr_delay=1)
    out = []
    for lean in (True, False):
        sv = solver.SubgameSolver(layout, boards, cuda_device, exploitability=True, keep_policy=True, sampling=True,
                                  lean_iterations=lean)
        sv.set_sampling_schedule(torch.arange(B) % iterations + 1)
        r = sv.solve(rb, scal, check=True, **kw)
        out.append([x.clone() for x in (r.policy_avg, r.regrets, r.weight_sums, r.policy, r.policy_sample, r.root_values[..., :1326],
                                        r.values_avg[..., :1326], r.exploitability, r.br_values)] + [r.beliefs_last.clone()])
    return layout, out


@pytest.mark.parametrize("B", [1, 7, 8, 60])  # eight warps a slice of hands
def test_batch_sizes(cuda_device, B):
    for a, b in zip(*_both(cuda_device, B)[1]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("opts", [
    dict(bins=(0.5, 0.75, 1.0, 1.5, 2.0), cap=1),  # up to 8 actions at a node
    dict(cap=None, deep=True),  # more nodes than the lean kernel holds
    dict(cfr_type="linear", cfr_plus=True),
    dict(cfr_avg=True, enforce_zero_sum=True),
    dict(cfr_type="discounted_plus", iterations=1),
])
def test_options(cuda_device, opts):
    layout, out = _both(cuda_device, 5, **opts)
    if opts.get("deep"):
        assert np.asarray(layout.subgames["n_nodes"]).max() > 160
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("B", [160, 600])  # two warps a slice; more actions than the lean kernel takes
def test_wide_batches(cuda_device, B):
    for a, b in zip(*_both(cuda_device, B, bins=(0.5, 0.75, 1.0, 1.5, 2.0), cap=1, iterations=2)[1]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("L,W", [(1, 1344), (3, 1326), (257, 1344)])
def test_network_per_leaf_in_place(cuda_device, L, W):
    """The rows the feature kernel feeds a bf16 ValueMLP and the values written back, against the model called on the
    same beliefs: the same bits, padding untouched."""
    from poker2_b200 import leaf_eval

    g = torch.Generator(device=cuda_device).manual_seed(L)
    beliefs = torch.rand(L, 2, W, device=cuda_device, generator=g)
    boards = torch.rand(L, 52, device=cuda_device, generator=g).argsort(dim=1)[:, :5]
    boards[:, 3:] = -1
    ctx = torch.rand(L, 3, device=cuda_device, generator=g)
    model = leaf_eval.ValueMLP(64, 2, dtype=torch.bfloat16, seed=1).to(cuda_device)
    ev = leaf_eval.DirectLeafEvaluator(model, boards, ctx, cuda_device)
    want = model(beliefs[..., :1326].contiguous(), boards, ctx)
    out = torch.full((L, 2, W), 7.0, device=cuda_device)
    ev.evaluate_into(beliefs, out)
    assert torch.equal(out[..., :1326], want) and torch.equal(ev(beliefs), want)
    assert (out[..., 1326:] == 7.0).all()


@pytest.mark.parametrize("stepped", [False, True])
def test_refused_batch_stops_every_kernel(cuda_device, stepped):
    """Malformed records: the status word names the subgame and every split kernel leaves the outputs as they were."""
    import bench
    from poker2_b200 import solver, tree as ptree

    boards, ranges, pot, stack = bench.make_inputs(9, 5)
    trees = ptree.build_trees(ptree.root_states(pot.numpy(), stack.numpy()), [0.5, 1.0], 8, max_raises=2)
    layout = solver.device_layout(trees, boards.numpy())
    layout.nodes[int(layout.subgames[6]["node_begin"])]["n_children"] = 9
    cls = solver.SteppedSolver if stepped else solver.SubgameSolver
    sv = cls(layout, boards, cuda_device, exploitability=True)
    outputs = (sv.root_values, sv.values_avg, sv.regrets, sv.policy_avg, sv.exploitability)
    for x in outputs:
        x.fill_(-7.0)
    sv.solve(solver.pad_rows(ranges.to(cuda_device)).contiguous(), solver.iteration_scalars(4))
    assert sv.status() == 7
    assert all(bool((x == -7.0).all()) for x in outputs)


@pytest.mark.parametrize("rows,width", [(7, 1344), (3, 1344), (5, 1324)])
@pytest.mark.parametrize("what", ["beliefs", "out"])
def test_network_per_leaf_refuses_other_shapes(cuda_device, rows, width, what):
    """More or fewer leaves than the evaluator was made for, or rows that are too short, do not reach the kernels: the general
    path refuses them."""
    from poker2_b200 import leaf_eval

    L = 5
    g = torch.Generator(device=cuda_device).manual_seed(4)
    boards = torch.tensor([[0, 1, 2, -1, -1]], device=cuda_device).expand(L, 5)
    model = leaf_eval.ValueMLP(64, 2, dtype=torch.bfloat16, seed=1).to(cuda_device)
    ev = leaf_eval.DirectLeafEvaluator(model, boards, torch.rand(L, 3, device=cuda_device, generator=g), cuda_device)
    shapes = {"beliefs": (L, 2, 1344), "out": (L, 2, 1344)}
    shapes[what] = (rows, 2, width)
    beliefs = torch.rand(*shapes["beliefs"], device=cuda_device, generator=g)
    with pytest.raises((RuntimeError, ValueError)):
        ev.evaluate_into(beliefs, torch.zeros(*shapes["out"], device=cuda_device))
    if what == "beliefs":
        with pytest.raises((RuntimeError, ValueError)):
            ev(beliefs)


def _kernels_of(fn):
    torch.cuda.synchronize()
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
        fn()
        torch.cuda.synchronize()
    return " ".join(e.name for e in prof.events() if "_kernel" in e.name)


@pytest.mark.parametrize("B", [5, 160])  # the general kernel; the lean kernel where it covers the solve
@pytest.mark.parametrize("kind", ["plain", "eight actions", "cfr_avg", "warm"])
def test_smaller_scratch_areas(cuda_device, B, kind):
    """An area without room for the split kernels: the lean or the general kernel runs, with the same bits and without a write
    behind the area's end."""
    import bench
    from poker2_b200 import _lib, solver, tree as ptree

    boards, ranges, pot, stack = bench.make_inputs(B, 3)
    bins = (0.5, 0.75, 1.0, 1.5, 2.0) if kind == "eight actions" else (0.5, 1.0)
    trees = ptree.build_trees(ptree.root_states(pot.numpy(), stack.numpy()), list(bins), 8, max_raises=1)
    layout = solver.device_layout(trees, boards.numpy())
    rb = solver.pad_rows(ranges.to(cuda_device)).contiguous()
    kw = {"cfr_avg": True} if kind == "cfr_avg" else {}
    if kind == "warm":
        siblings = torch.from_numpy(trees.child_count[trees.parent_index.clip(min=0)]).clamp(min=1)
        kw = dict(start_policy=(1.0 / siblings.float())[:, None].expand(-1, 1326).contiguous(), warm_start_iterations=2,
                  warm_start_multiplier=3.0)
    scal = solver.iteration_scalars(5, warm_start_iterations=2 if kind == "warm" else 0)
    lib, args = _lib.lib(), (layout.max_internal, layout.max_children, min(B, 148), B, layout.rows)
    full = int(lib.p2b_cfr_solve_scratch_floats(*args))
    sizes = [full, int(lib.p2b_cfr_solve_block_scratch_floats(*args))]
    if kind != "warm":  # which needs rows handed from launch to launch
        sizes.append(int(lib.p2b_cfr_scratch_floats(layout.max_internal, min(B, 148))))
    assert sizes == sorted(sizes, reverse=True) and len(set(sizes)) == len(sizes)
    out = []
    for n in sizes:
        sv = solver.SubgameSolver(layout, boards, cuda_device, exploitability=True)
        assert sv.num_blocks == min(B, 148) and sv.scratch.numel() == full
        guarded = torch.full((n + (1 << 20),), float("nan"), device=cuda_device)
        guarded[n:] = 7.0
        sv.scratch = guarded[:n]
        names = _kernels_of(lambda: sv.solve(rb, scal, check=True, **kw))
        assert ("split_rows_kernel" in names) == (n == full)
        lean = n == sizes[1] and B > 148 and kind in ("plain", "warm")
        assert ("cfr_iter_kernel" in names) == lean, names
        assert bool((guarded[n:] == 7.0).all())
        out.append([x.clone() for x in (sv.policy_avg, sv.regrets, sv.weight_sums, sv.root_values[..., :1326], sv.exploitability)])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert torch.equal(a, b)


@pytest.mark.parametrize("stepped", [False, True])
def test_area_that_does_not_fit(cuda_device, stepped):
    """A process whose share of the card holds the state arrays but not the split kernels' area: the solver takes the smaller
    area, with the same results."""
    import bench
    from poker2_b200 import solver, tree as ptree

    B = 160
    boards, ranges, _, _ = bench.make_inputs(B, 4)
    trees = ptree.build_trees(ptree.root_states(np.full(B, 60), np.full(B, 500)), [0.5, 1.0], 8)
    layout = solver.device_layout(trees, boards.numpy())
    rb = solver.pad_rows(ranges.to(cuda_device)).contiguous()
    scal = solver.iteration_scalars(3)
    cls = solver.SteppedSolver if stepped else solver.SubgameSolver

    def solved(sv):
        sv.solve(rb, scal)
        assert sv.status() == 0
        return [x.cpu() for x in (sv.policy_avg, sv.regrets, sv.root_values[..., :1326])]

    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated(cuda_device)
    sv = cls(layout, boards, cuda_device)
    full, smallest = sv.scratch.numel(), sv._scratch_floats(True)[-1]
    assert full == sv._scratch_floats(True)[0] and 4 * (full - smallest) > 512 << 20
    state = torch.cuda.memory_allocated(cuda_device) - before - 4 * full
    want = solved(sv)
    del sv
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(cuda_device).total_memory
    share = torch.cuda.memory_reserved(cuda_device) + state + 4 * smallest + (256 << 20)
    torch.cuda.set_per_process_memory_fraction(share / total, cuda_device)
    try:
        sv = cls(layout, boards, cuda_device)
        assert sv.scratch.numel() == smallest
        got = solved(sv)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0, cuda_device)
    for a, b in zip(want, got):
        assert torch.equal(a, b)


def _small_trees(cuda_device, B):
    """A batch of small trees off the lean path, on the split kernels."""
    from poker2_b200 import _lib, device_tree, solver, tree as ptree

    boards = torch.rand(B, 52, generator=torch.Generator().manual_seed(B)).argsort(dim=1)[:, :5]
    layout = device_tree.build_device_layout(ptree.root_states(np.full(B, 100), 8 + np.arange(B) % 5), boards, [0.5, 1.0], 3,
                                             max_raises=1, device=cuda_device)
    layout.max_children = 8  # as if some node had so many actions
    sv = solver.SubgameSolver(layout, boards, cuda_device)
    assert sv.scratch.numel() == _lib.lib().p2b_cfr_solve_scratch_floats(layout.max_internal, 8, sv.num_blocks, B, layout.rows)
    ranges = torch.rand(B, 2, 1344, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(1))
    ranges[..., 1326:] = 0.0
    return sv, ranges, solver.iteration_scalars(2)


@pytest.mark.parametrize("B", [6143, 6144, 7001])  # below and from where the lists' beginnings are added up by one block
def test_work_lists_of_large_batches(cuda_device, B):
    from poker2_b200 import _lib

    sv, ranges, scal = _small_trees(cuda_device, B)
    outputs = (sv.policy_avg, sv.regrets, sv.root_values[..., :1326])
    names = _kernels_of(lambda: sv.solve(ranges, scal, check=True))
    assert "split_rows_kernel" in names and ("split_begin_kernel" in names) == (B >= 6144)
    got = [x.clone() for x in outputs]
    sv.scratch = torch.empty(int(_lib.lib().p2b_cfr_scratch_floats(sv.layout.max_internal, sv.num_blocks)), device=cuda_device)
    assert "split_rows_kernel" not in _kernels_of(lambda: sv.solve(ranges, scal, check=True))
    for a, b in zip(got, outputs):
        assert torch.equal(a, b)


def test_work_lists_take_time_in_proportion_to_the_batch(cuda_device):
    def microseconds(B):
        sv, ranges, scal = _small_trees(cuda_device, B)
        sv.solve(ranges, scal, check=True)
        times = []
        for _ in range(3):
            torch.cuda.synchronize()
            with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA], acc_events=True) as prof:
                sv.solve(ranges, scal)
                torch.cuda.synchronize()
            times.append(sum(e.device_time for e in prof.events() if "split_begin_kernel" in e.name or "split_items_kernel" in e.name))
        return min(times)

    few, many = microseconds(3072), microseconds(24576)
    assert 0.0 < many < 12.0 * few, (few, many)  # eight times the subgames; with 64 times the reads it was about 19 times as long


def test_a_wait_that_ran_out_is_reported_by_the_whole_solve(cuda_device):
    """The word a wait leaves when it runs out (put there by hand): every later call of the stepped solve reports it and leaves
    the outputs alone; the next start pass clears it."""
    import bench
    from poker2_b200 import solver, tree as ptree

    boards, ranges, pot, stack = bench.make_inputs(9, 5)
    trees = ptree.build_trees(ptree.root_states(pot.numpy(), stack.numpy()), [0.5, 1.0], 8, max_raises=2)
    sv = solver.SteppedSolver(solver.device_layout(trees, boards.numpy()), boards, cuda_device, exploitability=True)
    rb, scal = solver.pad_rows(ranges.to(cuda_device)).contiguous(), solver.iteration_scalars(4)
    sv.solve(rb, scal)
    outputs = (sv.policy_avg, sv.regrets, sv.root_values[..., :1326], sv.exploitability)
    want = [x.clone() for x in outputs]
    sv.work_counter[3] = 5
    for begin, end, phases in ((1, 1, 1), (1, 1, 2), (1, 2, 16), (4, 4, 3), (4, 4, 4)):
        assert sv.status() == 5
        sv._step(rb, sv._scalars, 4, 0, begin, end, phases)
        assert int(sv.work_counter[1]) == 5
    assert all(torch.equal(a, b) for a, b in zip(want, outputs))
    sv.solve(rb, scal)
    assert sv.status() == 0 and all(torch.equal(a, b) for a, b in zip(want, outputs))
    # a one-call solve begins anew each time
    one = solver.SubgameSolver(sv.layout, boards, cuda_device)
    one.work_counter[3] = 5
    one.solve(rb, scal, check=True)
    assert torch.equal(one.policy_avg, sv.policy_avg)


@pytest.mark.parametrize("spoil", ["actions", "orphans"])
def test_trees_beyond_the_sizes_named_are_refused(cuda_device, spoil):
    """Work space sized by the largest child count holds no node with more children and no node without a parent: the record
    check refuses such a subgame wherever the sizes matter, and the general kernel, where they do not, solves it."""
    import bench
    from poker2_b200 import solver, tree as ptree

    boards, ranges, pot, stack = bench.make_inputs(6, 8)
    trees = ptree.build_trees(ptree.root_states(pot.numpy(), stack.numpy()), [0.5, 1.0], 8, max_raises=2)
    layout = solver.device_layout(trees, boards.numpy())
    rb, scal = solver.pad_rows(ranges.to(cuda_device)).contiguous(), solver.iteration_scalars(3)
    sound = solver.SubgameSolver(layout, boards, cuda_device)
    sound.solve(rb, scal, check=True)
    assert layout.max_children == 5
    if spoil == "actions":
        layout.max_children = 4
    else:  # leaves behind the last subgame's own that no node has for a child
        extra = 310 - int(layout.subgames[5]["n_nodes"])
        leaf = layout.nodes[solver.node_kind(layout.nodes) == ptree.KIND_FOLD][-1]
        layout.nodes = np.concatenate([layout.nodes, np.repeat(leaf, extra)])
        layout.subgames[5]["n_nodes"] += extra
        assert 310 > int(layout.subgames[5]["n_internal"]) * layout.max_children + 1
    for policy in ("auto", "lean"):
        solver.set_path_policy(policy)
        for cls in (solver.SubgameSolver, solver.SteppedSolver):
            sv = cls(layout, boards, cuda_device)
            sv.root_values.fill_(-7.0)
            sv.regrets.fill_(-7.0)
            sv.solve(rb, scal)
            assert sv.status() > 0 and bool((sv.root_values == -7.0).all()) and bool((sv.regrets == -7.0).all())
    general = solver.SubgameSolver(layout, boards, cuda_device, lean_iterations=False)
    general.solve(rb, scal, check=True)
    rows = sound.regrets.shape[0]
    assert torch.equal(general.regrets[:rows], sound.regrets) and torch.equal(general.root_values, sound.root_values)
