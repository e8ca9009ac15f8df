"""What the short way through the leaf network must not lose: hooks on the network and on its layers fire, a layer whose output
a hook has kept is not overwritten by the activation behind it, a derived evaluator's own call is made, and one evaluator
serves several streams and threads."""
import pytest
import torch

from poker2_b200 import leaf_eval


def _model():
    return leaf_eval.ValueMLP(16, 2, dtype=torch.bfloat16, seed=1)


def _rows(n=3):
    return torch.rand(n, leaf_eval.ValueMLP.IN_PADDED, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)


def test_without_hooks_the_layers_give_the_network():
    model = _model()
    with torch.no_grad():
        assert torch.equal(model.layers(_rows()), model.net(_rows()))


@pytest.mark.parametrize("where", ["net", "linear", "gelu", "global"])
@pytest.mark.parametrize("pre", [False, True])
def test_hooks_on_the_network_fire(where, pre):
    model, seen = _model(), []
    target = {"net": model.net, "linear": model.net[0], "gelu": model.net[1]}.get(where)
    hook = (lambda m, args: seen.append(args[0])) if pre else (lambda m, args, out: seen.append(out))
    if where == "global":
        register = (torch.nn.modules.module.register_module_forward_pre_hook if pre
                    else torch.nn.modules.module.register_module_forward_hook)
        handle = register(hook)
    else:
        handle = (target.register_forward_pre_hook if pre else target.register_forward_hook)(hook)
    try:
        got = model.layers(_rows())
    finally:
        handle.remove()
    assert seen
    with torch.no_grad():
        assert torch.equal(got, model.net(_rows()))
        if where == "linear" and not pre:  # what the hook kept is the layer's output, not the activation's
            assert torch.equal(seen[0], model.net[0](_rows()))


@pytest.mark.parametrize("what", ["layer", "net"])
def test_a_replaced_forward_is_called(what):
    class Doubled(torch.nn.Module):
        def __init__(self, net):
            super().__init__()
            self.inner = net

        def forward(self, x):
            return self.inner(x) * 2.0

    model = _model()
    if what == "layer":
        model.net[1].forward = lambda x: torch.zeros_like(x)
    else:
        model.net = Doubled(model.net)
    with torch.no_grad():
        assert torch.equal(model.layers(_rows()), model.net(_rows()))


class _Halved(leaf_eval.DirectLeafEvaluator):
    def __call__(self, leaf_beliefs):
        return super().__call__(leaf_beliefs) * 0.5


class _HalvedInPlace(leaf_eval.DirectLeafEvaluator):
    def evaluate_into(self, leaf_beliefs, out):
        super().evaluate_into(leaf_beliefs, out)
        out.mul_(0.5)


def test_a_subclass_with_a_call_of_its_own_is_called():
    """The solver writes values in place only where `evaluate_into` is not behind another `__call__`."""
    from types import SimpleNamespace

    from poker2_b200 import solver

    L = 3
    beliefs = torch.rand(L, 2, 1344, generator=torch.Generator().manual_seed(5))
    boards, ctx = torch.tensor([[0, 1, 2, -1, -1]]).expand(L, 5), torch.rand(L, 3)
    plain, half, in_place = (c(_model(), boards, ctx, torch.device("cpu")) for c in (leaf_eval.DirectLeafEvaluator, _Halved, _HalvedInPlace))
    want = plain(beliefs)
    for fn, factor in ((plain, 1.0), (half, 0.5), (in_place, 0.5), (lambda b: plain(b) * 0.25, 0.25)):
        state = SimpleNamespace(leaf_beliefs=beliefs, leaf_values=torch.zeros(L, 2, 1344))
        solver.SteppedSolver._value_leaves(state, fn, L)
        assert torch.equal(state.leaf_values[..., :1326], want * factor)


@pytest.mark.gpu
@pytest.mark.parametrize("evaluate", ["call", "into"])
def test_hooks_on_the_model_of_a_leaf_evaluator_fire(cuda_device, evaluate):
    model, L, seen = _model().to(cuda_device), 5, []
    g = torch.Generator(device=cuda_device).manual_seed(3)
    beliefs = torch.rand(L, 2, 1344, device=cuda_device, generator=g)
    boards = torch.tensor([[0, 1, 2, -1, -1]], device=cuda_device).expand(L, 5)
    ev = leaf_eval.DirectLeafEvaluator(model, boards, torch.rand(L, 3, device=cuda_device, generator=g), cuda_device)
    want = ev(beliefs).clone()
    handle = model.register_forward_hook(lambda m, args, out: (seen.append(out), out * 2.0)[1])
    if evaluate == "call":
        got = ev(beliefs)
    else:
        got = torch.zeros(L, 2, 1344, device=cuda_device)
        ev.evaluate_into(beliefs, got)
    handle.remove()
    assert len(seen) == 1 and torch.equal(got[..., :1326], want * 2.0)
    assert torch.equal(ev(beliefs), want)


def _two_calls(cuda_device):
    L = 6
    g = torch.Generator(device=cuda_device).manual_seed(9)
    boards = torch.tensor([[0, 1, 2, -1, -1]], device=cuda_device).expand(L, 5)
    ev = leaf_eval.DirectLeafEvaluator(_model().to(cuda_device), boards, torch.rand(L, 3, device=cuda_device, generator=g), cuda_device)
    beliefs = [torch.rand(L, 2, 1344, device=cuda_device, generator=g) for _ in range(2)]
    want = [ev(b) for b in beliefs]
    torch.cuda.synchronize()
    assert not torch.equal(*want)
    return ev, beliefs, want


@pytest.mark.gpu
def test_one_evaluator_on_two_streams(cuda_device, monkeypatch):
    """A call on another stream while this one's is between its input and its layers."""
    ev, beliefs, want = _two_calls(cuda_device)
    other = torch.cuda.Stream(cuda_device)
    with torch.cuda.stream(other):  # its memory and handles are there: nothing makes the second call wait for the first
        for _ in range(2):
            ev(beliefs[1])
    torch.cuda.synchronize()
    layers, slow = leaf_eval.ValueMLP.layers, [False, True]  # the first call's layers begin late

    def delayed(self, x):
        if slow.pop():
            torch.cuda._sleep(1 << 27)
        return layers(self, x)

    monkeypatch.setattr(leaf_eval.ValueMLP, "layers", delayed)
    first = ev(beliefs[0])
    with torch.cuda.stream(other):
        second = ev(beliefs[1])
    torch.cuda.synchronize()
    assert torch.equal(second, want[1]) and torch.equal(first, want[0])


@pytest.mark.gpu
def test_an_evaluator_can_be_copied(cuda_device):
    import copy
    import pickle

    ev, beliefs, want = _two_calls(cuda_device)
    for other in (copy.deepcopy(ev), pickle.loads(pickle.dumps(ev))):
        assert torch.equal(other(beliefs[0]), want[0]) and torch.equal(other(beliefs[1]), want[1])


@pytest.mark.gpu
def test_one_evaluator_in_two_threads(cuda_device, monkeypatch):
    """A second thread's call while the first is between the launches of its input and of its layers."""
    import threading
    import time

    ev, beliefs, want = _two_calls(cuda_device)
    layers, entered = leaf_eval.ValueMLP.layers, threading.Event()

    def delayed(self, x):
        if not entered.is_set():
            entered.set()
            time.sleep(0.2)
        return layers(self, x)

    monkeypatch.setattr(leaf_eval.ValueMLP, "layers", delayed)
    got = [None, None]
    threads = [threading.Thread(target=lambda i=i: got.__setitem__(i, ev(beliefs[i]))) for i in range(2)]
    threads[0].start()
    assert entered.wait(5.0)
    threads[1].start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
