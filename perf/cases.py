"""The work that users of poker2_b200 give it, as cases that can be timed.

A case is a dict of plain values; `kind` says which public entry points it goes through:

  compare    `rules.compare_7_cards_single_batch`: who wins at the showdowns of a batch of tables
  rank       `rules.rank_7_cards_single_batch`: scores of a batch of hands
  showdown   `showdown.BoardTables` and `showdown.showdown_values`
  river      a whole solve of river subgames: `solver.SubgameSolver.solve` on a prepared solver, or
             `solver.solve_subgames` from the roots on the host (`one_call`)
  turn       `solver.solve_subgames_with_model`: leaves valued by the network, averaged over the river cards
  generator  one turn of the data generator's loop: `evaluator.SubgameEvaluator.initialize_subgame`,
             `evaluate_cfr`, `training_data`
  steps      one `step_evaluator.StepCFREvaluator.cfr_iteration`, the form composed of the step kernels

Inputs are synthetic: uniform cards, Dirichlet(1) ranges over the combos that the board leaves, pots and stacks
uniform over the ranges of the benchmark, a value network with random weights in bf16.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from poker2_b200 import device_tree, evaluator, leaf_eval, rules, showdown, solver, step_evaluator, tree

HANDS = 1326
TWO_BETS = (0.5, 1.0)  # bet sizes of the production configuration
FIVE_BETS = (0.5, 0.75, 1.0, 1.5, 2.0)  # bet sizes of the configuration dataclasses: 8 actions a node
NET_WIDTH, NET_DEPTH = 1536, 4


def listed():
    return [
        # The environment's showdowns of one step: the production configuration plays 192 tables, cards are int64.
        {"name": "compare_192", "kind": "compare", "hands": 192, "dtype": "int64"},
        # The ranking half of the rules benchmark.
        {"name": "rank_67m", "kind": "rank", "hands": 1 << 26, "dtype": "int16"},
        # The showdown half of the rules benchmark: every board is new, so its tables are built each time.
        {"name": "showdown_4096", "kind": "showdown", "boards": 4096, "nodes": 1, "new_boards": True},
        # Showdown leaves of one CFR iteration: the boards' tables are kept, a river tree has 43 such leaves.
        {"name": "showdown_64x43", "kind": "showdown", "boards": 64, "nodes": 43, "new_boards": False},
        # A single river subgame for analysis, from its description to its strategy.
        {"name": "river_1", "kind": "river", "roots": 1, "iterations": 256, "cap": 2, "cfr_type": "discounted",
         "cfr_plus": False, "one_call": True},
        # A small ragged batch without a raise cap: an evaluation set, or what is left of a larger batch.
        {"name": "river_37_nocap", "kind": "river", "roots": 37, "iterations": 64, "cap": -1,
         "cfr_type": "discounted_plus", "cfr_plus": False, "one_call": False},
        # The headline batch, for a quarter of its iterations.
        {"name": "river_4096", "kind": "river", "roots": 4096, "iterations": 64, "cap": 2, "cfr_type": "discounted",
         "cfr_plus": False, "one_call": False},
        # Turn subgames whose leaves are averaged over the 48 river cards.
        {"name": "turn_128", "kind": "turn", "roots": 128, "iterations": 16, "cap": 2},
        # The data generator of the production configuration on flop roots: 192 environments, the largest trees.
        {"name": "flop_generator_192", "kind": "generator", "street": 1, "roots": 192, "iterations": 200,
         "settings": "production"},
        # The same on river roots, where most leaves end the hand.
        {"name": "river_generator_192", "kind": "generator", "street": 3, "roots": 192, "iterations": 200,
         "settings": "production"},
        # What the configuration dataclasses switch on by themselves, on turn roots.
        {"name": "turn_generator_64", "kind": "generator", "street": 2, "roots": 64, "iterations": 100,
         "settings": "defaults"},
        # One iteration of the transparent evaluator, as tools and tests that look between the steps run it.
        {"name": "steps_64", "kind": "steps", "roots": 64, "cap": 2},
    ]


def _spread(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["compare", "rank", "showdown", "river", "river", "turn", "generator", "generator", "steps"])
    if kind in ("compare", "rank"):
        dtype = rng.choice(["int16", "int64"])
        top = (1 << 26) // (8 if dtype == "int64" else 1) // (2 if kind == "compare" else 1)
        return {"kind": kind, "hands": _spread(rng, 1, top), "dtype": dtype}
    if kind == "showdown":
        new = rng.random() < 0.5
        nodes = 1 if new else rng.randint(1, 43)
        return {"kind": kind, "boards": _spread(rng, 1, 4096 if new else 16384 // nodes), "nodes": nodes, "new_boards": new}
    if kind == "river":
        cap = rng.choice([2, 2, -1])
        iterations = _spread(rng, 8, 256)
        most = (1 << 18) // iterations // (3 if cap < 0 else 1)
        return {"kind": kind, "roots": _spread(rng, 1, min(4096, most)), "iterations": iterations, "cap": cap,
                "cfr_type": rng.choice(["discounted", "discounted", "discounted_plus", "standard"]),
                "cfr_plus": rng.random() < 0.25, "one_call": rng.random() < 0.5}
    if kind == "turn":
        iterations = _spread(rng, 4, 64)
        return {"kind": kind, "roots": _spread(rng, 1, min(256, 2048 // iterations)), "iterations": iterations, "cap": 2}
    if kind == "generator":
        settings = rng.choice(["production", "production", "defaults"])
        most = 192 if settings == "production" else 64
        return {"kind": kind, "street": rng.choice([1, 2, 3]), "roots": _spread(rng, 4, most),
                "iterations": rng.randint(24, 200 if settings == "production" else 100), "settings": settings}
    return {"kind": kind, "roots": _spread(rng, 1, 256), "cap": 2}


# ---- inputs ---------------------------------------------------------------------------------------


def _deal(n, k, gen, dtype):
    """[n,k] distinct cards of a deck each, uniform: the first k cards of a Fisher-Yates shuffle, followed
    backwards through its swaps."""
    dev = gen.device
    swaps = [torch.randint(j, 52, (n,), generator=gen, device=dev, dtype=torch.uint8) for j in range(k)]
    out = torch.empty(n, k, device=dev, dtype=dtype)
    for j in range(k):
        at = swaps[j]
        for i in range(j - 1, -1, -1):
            at = torch.where(at == swaps[i], i, at)
        out[:, j] = at
    return out


def _ranges(boards, gen):
    """[n,2,1326] fp32: Dirichlet(1) over the combos that share no card with the board [n,L]."""
    dev = gen.device
    c1, c2 = (torch.from_numpy(c).to(dev) for c in np.triu_indices(52, k=1))
    hit = torch.zeros(boards.shape[0], 52, dtype=torch.bool, device=dev).scatter_(1, boards, True)
    r = torch.empty(boards.shape[0], 2, HANDS, device=dev).exponential_(generator=gen)
    r = r * ~(hit[:, c1] | hit[:, c2])[:, None, :]
    return r / r.sum(-1, keepdim=True)


def _pots(case):
    """Pot and effective stack of every root, on the host: the benchmark's ranges (larger pots without a raise cap, where
    the smallest would give trees of more nodes than a subgame can have), or for the generator hands of the
    production game, which start with 1000 chips a player. They set the sizes of the trees and so belong to the case."""
    n = case["roots"]
    g = np.random.default_rng(n)
    if case["kind"] == "generator":
        pot = g.integers(20, 900, n)
        return pot, 1000 - pot // 2
    if case["cap"] < 0:
        return g.integers(100, 201, n), g.integers(100, 1001, n)
    if n == 1 and case["kind"] == "river":
        return np.array([100]), np.array([400])
    return g.integers(20, 201, n), g.integers(100, 1001, n)


def _network(device, seed):
    return leaf_eval.ValueMLP(NET_WIDTH, NET_DEPTH, dtype=torch.bfloat16, seed=seed).to(device)


def prepare(case, seed):
    device = torch.device("cuda:0")
    gen = torch.Generator(device=device).manual_seed(seed)
    kind = case["kind"]
    state = {"case": case, "device": device, "seed": seed}
    if kind in ("compare", "rank"):
        dtype = getattr(torch, case["dtype"])
        if kind == "rank":
            state["cards"] = _deal(case["hands"], 7, gen, dtype)
        else:  # two hands that share the board: 9 cards of one deck
            nine = _deal(case["hands"], 9, gen, dtype)
            state["cards"] = torch.stack([nine[:, :7], torch.cat([nine[:, :5], nine[:, 7:]], dim=1)], dim=1).contiguous()
        return state
    if kind == "showdown":
        b, n = case["boards"], case["nodes"]
        boards = _deal(b, 5, gen, torch.int64)
        table = torch.arange(b, device=device, dtype=torch.int32).repeat_interleave(n)
        state["boards"] = boards
        state["beliefs"] = _ranges(boards[table.long()], gen).contiguous()
        pot = torch.randint(10, 500, (b * n, 2), generator=gen, device=device)
        state["potential"], state["scale"] = pot, torch.full((b * n,), 1000.0, device=device)
        state["table_of_row"] = None if n == 1 else table
        state["tables"] = None if case["new_boards"] else showdown.BoardTables(boards)
        return state
    street = {"turn": 2, "generator": case.get("street")}.get(kind, 3)
    boards = _deal(case["roots"], street + 2, gen, torch.int64)
    ranges = _ranges(boards, gen)
    pot, stack = _pots(case)
    boards5 = torch.full((case["roots"], 5), -1, dtype=torch.int64)
    boards5[:, : street + 2] = boards.cpu()
    cap = case.get("cap", -1)
    cap = None if cap < 0 else cap
    if kind == "generator":
        roots = tree.root_states(pot, stack, min_raise=10, street=street)
        state.update(env=evaluator.env_view(roots, boards5.numpy()), indices=torch.arange(case["roots"]), ranges=ranges,
                     model=_network(device, seed))
    elif kind == "turn":
        state.update(boards=boards5[:, :4].contiguous(), ranges=ranges, pot=torch.from_numpy(pot),
                     stack=torch.from_numpy(stack), cap=cap, model=_network(device, seed))
    elif kind == "steps":
        trees = tree.build_trees(tree.root_states(pot, stack), list(TWO_BETS), 8, max_raises=cap)
        ev = step_evaluator.StepCFREvaluator(trees, boards5.numpy(), ranges, device, iterations=16)
        ev.initialize_policy_and_beliefs()
        ev.set_leaf_values(0)
        ev.compute_expected_values()
        state["ev"] = ev
    elif case["one_call"]:
        state.update(boards=boards5, ranges=ranges, pot=torch.from_numpy(pot), stack=torch.from_numpy(stack), cap=cap)
    else:
        layout = device_tree.build_device_layout(tree.root_states(pot, stack), boards5, list(TWO_BETS), 8, max_raises=cap,
                                                 device=device)
        state["solver"] = solver.SubgameSolver(layout, boards5, device, exploitability=True)
        state["ranges"] = solver.pad_rows(ranges).contiguous()
        state["scalars"] = solver.iteration_scalars(case["iterations"], cfr_type=case["cfr_type"],
                                                    dcfr_delay=_delay(case))
    return state


def _delay(case):
    return case["iterations"] // 4 if case["cfr_type"] == "discounted_plus" else 0


# ---- one pass -------------------------------------------------------------------------------------


def _solved(res):
    """What a solve leaves for its caller: strategies and regrets of every node, values and exploitability."""
    return {"policy_avg": res.policy_avg[:, :HANDS], "regrets": res.regrets[:, :HANDS],
            "weight_sums": res.weight_sums[:, :HANDS], "root_values": res.root_values[..., :HANDS],
            "exploitability": res.exploitability, "br_values": res.br_values}


def _generator_settings(case):
    T = case["iterations"]
    ws = min(15, T - 1)
    if case["settings"] == "production":
        return dict(iterations=T, bet_bins=TWO_BETS, max_depth=5, bb=10, cfr_type="discounted_plus", alpha=2.0,
                    alpha_final=4.0, beta=-1.0, beta_final=-2.0, gamma=5.0, gamma_final=0.0, dcfr_delay=min(80, T // 2),
                    warm_start_iterations=ws, warm_start_multiplier=10.0, enforce_zero_sum=True, chance_average=False)
    return dict(iterations=T, bet_bins=FIVE_BETS, max_depth=2, bb=10, cfr_type="linear", cfr_plus=True, cfr_avg=True,
                running_values=True, warm_start_iterations=ws, warm_start_type="model_br", enforce_zero_sum=True,
                chance_average=False)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "compare":
        return rules.compare_7_cards_single_batch(state["cards"])
    if kind == "rank":
        return rules.rank_7_cards_single_batch(state["cards"])
    if kind == "showdown":
        tables = state["tables"] if state["tables"] is not None else showdown.BoardTables(state["boards"])
        return showdown.showdown_values(tables, state["beliefs"], state["potential"], state["scale"],
                                        table_of_row=state["table_of_row"])
    if kind == "river":
        if case["one_call"]:
            res, _ = solver.solve_subgames(state["boards"], state["ranges"], state["pot"], state["stack"],
                                           iterations=case["iterations"], bet_bins=TWO_BETS, max_raises=state["cap"],
                                           cfr_type=case["cfr_type"], dcfr_delay=_delay(case), cfr_plus=case["cfr_plus"],
                                           exploitability=True, device=state["device"])
        else:
            res = state["solver"].solve(state["ranges"], state["scalars"], cfr_plus=case["cfr_plus"])
        return _solved(res)
    if kind == "turn":
        res, _, _ = solver.solve_subgames_with_model(state["boards"], state["ranges"], state["pot"], state["stack"],
                                                     state["model"], street=2, iterations=case["iterations"],
                                                     bet_bins=TWO_BETS, max_raises=state["cap"], exploitability=True,
                                                     device_tree=True, device=state["device"])
        return _solved(res)
    if kind == "steps":
        ev = state["ev"]
        ev.cfr_iteration(3)
        return {"policy": ev.policy_probs, "policy_avg": ev.policy_probs_avg, "regrets": ev.cumulative_regrets,
                "weight_sums": ev.regret_weight_sums, "beliefs": ev.beliefs, "values": ev.latest_values}
    ev = evaluator.SubgameEvaluator(state["device"], model=state["model"],
                                    generator=torch.Generator(device=state["device"]).manual_seed(state["seed"]),
                                    **_generator_settings(case))
    ev.initialize_subgame(state["env"], state["indices"], state["ranges"])
    # The sampled next states are part of the call and not of the outputs: a draw turns a last bit of the bf16
    # network into another state, or into another number of states.
    ev.evaluate_cfr()
    out = {}
    for name, batch in zip(("value", "pre_chance", "policy"), ev.training_data()):
        if batch is not None:
            out[name] = {"beliefs": batch.beliefs, "legal": batch.legal_masks, "values": batch.value_targets,
                         "policy": batch.policy_targets}
    out["exploitability"], out["regrets"] = ev.stats["local_exploitability"], ev.cumulative_regrets
    return out


# ---- what a pass cannot do without, and how exact it is ---------------------------------------------


def _trees(case):
    """(all nodes, showdown leaves, leaves for the network) of the case's trees, a large batch scaled up from 64 roots."""
    n = min(case["roots"], 64)
    pot, stack = _pots(dict(case, roots=n))
    street = {"turn": 2, "generator": case.get("street")}.get(case["kind"], 3)
    bets, depth, bb, cap = TWO_BETS, 8, 2, case.get("cap", -1)
    if case["kind"] == "generator":
        depth, bb = 5, 10
        if case["settings"] == "defaults":
            bets, depth = FIVE_BETS, 2
    t = tree.build_trees(tree.root_states(pot, stack, min_raise=bb, street=street), list(bets), depth, bb=bb,
                         max_raises=None if cap < 0 else cap)
    leaf = t.child_count == 0
    down = leaf & (t.state.street == 4)
    model = leaf & ~down & ~t.state.done
    k = case["roots"] / n
    return t.total_nodes * k, down.sum() * k, model.sum() * k


def work(case):
    """Inputs and outputs once; operations by hand and node. A solve's state need not leave the chip between its
    iterations, so its bytes are the ranges read and the results written. An iteration costs about 40 operations a
    hand and node (reach, average, beliefs, regret, the next policy, the backup) and about 60 a hand and showdown leaf (sums
    over stronger and weaker hands and over the two cards)."""
    kind, f4 = case["kind"], 4
    if kind in ("compare", "rank"):
        hands = case["hands"] * (2 if kind == "compare" else 1)
        item = 8 if case["dtype"] == "int64" else 2
        return {"bytes": hands * 7 * item + case["hands"] * 4, "flops": 60.0 * hands}
    if kind == "showdown":
        rows = case["boards"] * case["nodes"]
        return {"bytes": rows * (2 * 2 * HANDS * f4 + 20) + case["boards"] * (40 if case["new_boards"] else 18592),
                "flops": 120.0 * HANDS * rows + (200.0 * HANDS * case["boards"] if case["new_boards"] else 0.0)}
    nodes, down, model = _trees(case)
    if kind == "steps":  # the state is in memory before and after: 3 rows read, 8 written a node
        return {"bytes": nodes * HANDS * f4 * 11, "flops": HANDS * (40.0 * nodes + 60.0 * down)}
    passes = case["iterations"] + 2
    if kind == "generator":
        passes -= min(15, case["iterations"] - 1)
    flops = HANDS * (40.0 * nodes + 60.0 * down) * passes
    net = 2.0 * (leaf_eval.ValueMLP.IN_FEATURES * NET_WIDTH + (NET_DEPTH - 1) * NET_WIDTH ** 2 + NET_WIDTH * 2 * HANDS)
    flops += net * model * passes * (48 if kind == "turn" else 1)
    rows_out = {"generator": 4}.get(kind, 3)
    return {"bytes": HANDS * f4 * (rows_out * nodes + 4 * case["roots"]), "flops": flops}


def tolerance(case):
    """Scores and winners are whole numbers. Everything else is fp32; where the network values the leaves its bf16
    layers set the precision."""
    kind = case["kind"]
    if kind in ("compare", "rank"):
        return "exact"
    if kind in ("turn", "generator"):
        return {"rel": 1e-2, "max": 0.5}
    return {"rel": 1e-5}
