"""Leaf evaluators for subgames that end before the river: the callables a `SteppedSolver`
invokes between the two sweeps of every pass.

Upstream, the leaves at the start of the next street are valued by the value network
(`set_leaf_values`, p2/search/cfr_evaluator.py:1025-1047), and the value of such a
pre-chance state is the expectation over the next public card of the network's values on
the post-card beliefs (`ChanceNodeHelper.single_card_chance_values`,
p2/search/chance_node_helper.py:359-479).  `ChanceLeafEvaluator` computes that expectation
explicitly: the expansion over the next card and the per-leaf averaging are this library's
kernels (`chance.expand_next_card`, `chance.indexed_add_rows`); the network's GEMMs are
torch / cuBLAS.
"""
from __future__ import annotations

import threading

import numpy as np
import torch

from . import _lib, chance

NUM_HANDS = 1326


class ValueMLP(torch.nn.Module):
    """Value network stand-in with the shape of the benchmark configuration: input = two
    1326-combo ranges + 52-d board one-hot + 3 pot/stack scalars, `depth` hidden layers of
    `width` GELU units, output = 2 x 1326 hand values.  Random initialisation."""

    IN_FEATURES = 2 * NUM_HANDS + 52 + 3  # 2707
    IN_PADDED = 2720  # GEMM operands want rows that are multiples of 16 bytes; the extra columns are zero
    OUT_PADDED = 2656

    def __init__(self, width: int = 1536, depth: int = 4, *, dtype=torch.bfloat16, seed: int = 0):
        super().__init__()
        g = torch.Generator().manual_seed(seed)
        dims = [self.IN_FEATURES] + [width] * depth + [2 * NUM_HANDS]
        padded = [self.IN_PADDED] + [width] * depth + [self.OUT_PADDED]
        layers = []
        for i in range(len(dims) - 1):
            lin = torch.nn.Linear(padded[i], padded[i + 1])
            with torch.no_grad():
                lin.weight.zero_()
                lin.weight[: dims[i + 1], : dims[i]] = torch.randn(dims[i + 1], dims[i], generator=g) / dims[i] ** 0.5
                lin.bias.zero_()
            layers.append(lin)
            if i < len(dims) - 2:
                layers.append(torch.nn.GELU())
        self.net = torch.nn.Sequential(*layers).to(dtype)
        self.dtype = dtype

    @torch.no_grad()
    def forward(self, beliefs: torch.Tensor, boards: torch.Tensor, context: torch.Tensor) -> torch.Tensor:
        """beliefs [S,2,1326] fp32, boards [S,L] int64 (-1 = empty), context [S,3] fp32
        -> values [S,2,1326] fp32."""
        S = beliefs.shape[0]
        x = torch.zeros(S, self.IN_PADDED, device=beliefs.device, dtype=self.dtype)
        x[:, : 2 * NUM_HANDS] = beliefs.reshape(S, 2 * NUM_HANDS)
        onehot = torch.zeros(S, 53, device=beliefs.device, dtype=self.dtype)
        onehot.scatter_(1, torch.where(boards >= 0, boards, torch.full_like(boards, 52)), 1.0)
        x[:, 2 * NUM_HANDS: 2 * NUM_HANDS + 52] = onehot[:, :52]
        x[:, 2 * NUM_HANDS + 52: self.IN_FEATURES] = context
        y = self.net(x)[:, : 2 * NUM_HANDS]
        return y.to(torch.float32).view(S, 2, NUM_HANDS)

    @torch.no_grad()
    def layers(self, x: torch.Tensor) -> torch.Tensor:
        """`self.net` on input rows x, activations in place (half the memory traffic and footprint of a GELU, same bits) and
        linear layers without the module's wrapper: a pass over few leaves lasts as long as the host takes to launch it.
        A network that someone listens to (hooks) or has changed goes through its modules instead."""
        net = self.net
        if type(net) is not torch.nn.Sequential or not _bare(net, *net._modules.values()):
            return net(x)
        for layer in net._modules.values():
            if type(layer) is torch.nn.GELU and layer.approximate == "none":
                x = torch.ops.aten.gelu_(x)
            elif type(layer) is torch.nn.Linear:
                x = torch.nn.functional.linear(x, layer.weight, layer.bias)
            else:
                x = layer(x)
        return x


_module_hooks = torch.nn.modules.module


def _bare(*modules: torch.nn.Module) -> bool:
    """Nothing but the modules' own `forward` would run if they were called: no forward hooks, on them or on all modules, no
    `forward` put in place of the class's, not compiled.  (By their dictionaries: asked once a pass, for nine modules.)"""
    if _module_hooks._global_forward_hooks or _module_hooks._global_forward_pre_hooks:
        return False
    for m in modules:
        own = m.__dict__
        if own["_forward_hooks"] or own["_forward_pre_hooks"] or "forward" in own or own.get("_compiled_call_impl") is not None:
            return False
    return True


def leaf_context(trees, node_index) -> torch.Tensor:
    """[L,3] fp32 context of the tree nodes `node_index` (upstream numbering): pot and both
    stacks as fractions of the two starting stacks together."""
    st = trees.state
    idx = np.asarray(node_index, dtype=np.int64)
    total = np.maximum(st.starting_stacks[idx].astype(np.float32).sum(axis=1), np.float32(1.0))
    f32 = lambda a: a.astype(np.float32)  # noqa: E731  (fp32 division, as the upstream encoder does)
    ctx = np.stack([f32(st.pot[idx]) / total, f32(st.stacks[idx, 0]) / total, f32(st.stacks[idx, 1]) / total], axis=1)
    return torch.from_numpy(np.ascontiguousarray(ctx, dtype=np.float32))


class ChanceLeafEvaluator:
    """values(leaf) = mean over the next public card of model(post-card beliefs).

    boards: [L,W] int64 public cards of each leaf with -1 in the empty slots (at least one);
    context: [L,3] fp32; model(beliefs [S,2,1326], boards [S,W], context [S,3]) -> [S,2,1326].
    Leaves are processed `chunk` at a time (a chunk expands to about 48 x chunk samples)."""

    def __init__(self, model, boards: torch.Tensor, context: torch.Tensor, device: torch.device, *, chunk: int = 2048):
        self.model = model
        self.boards = boards.to(device=device, dtype=torch.int64).contiguous()
        self.context = context.to(device=device, dtype=torch.float32).contiguous()
        self.chunk = int(chunk)
        self.samples_per_call = int((52 - (self.boards >= 0).sum(dim=1)).sum().item())
        self.calls = 0
        # a bf16 `ValueMLP` takes the fused path: the network input is written directly by the
        # expansion kernel and its bf16 output is averaged per leaf without an fp32 copy
        self.fused = isinstance(model, ValueMLP) and model.dtype == torch.bfloat16
        self._chunks = []
        for a in range(0, self.boards.shape[0], self.chunk):
            b = min(a + self.chunk, self.boards.shape[0])
            off = chance.sample_offsets_of(self.boards[a:b])
            self._chunks.append((a, b, off, int(off[-1].item())))

    def evaluate_into(self, leaf_beliefs: torch.Tensor, out: torch.Tensor) -> None:
        """Values of all leaves into out[..., :1326] (fp32 [L,2,W])."""
        if not self.fused:
            out[..., :NUM_HANDS].copy_(self(leaf_beliefs))
            return
        for a, b, off, n_samples in self._chunks:
            x = chance.expand_features_bf16(leaf_beliefs[a:b], self.boards[a:b], off, n_samples, self.context[a:b],
                                            self.model.IN_PADDED)
            y = self.model.layers(x)
            chance.indexed_mean_bf16(y, off, out[a:b])
        self.calls += 1

    def __call__(self, leaf_beliefs: torch.Tensor) -> torch.Tensor:
        L = leaf_beliefs.shape[0]
        if self.fused:
            out = torch.zeros(L, 2, leaf_beliefs.shape[2], device=leaf_beliefs.device, dtype=torch.float32)
            self.evaluate_into(leaf_beliefs, out)
            return out
        out = torch.empty(L, 2, NUM_HANDS, device=leaf_beliefs.device, dtype=torch.float32)
        for a in range(0, L, self.chunk):
            b = min(a + self.chunk, L)
            pre = leaf_beliefs[a:b, :, :NUM_HANDS].contiguous()
            ctx = self.context[a:b]
            out[a:b] = chance.single_card_chance_values(
                pre, self.boards[a:b], lambda post, samples, lookup: self.model(post, samples, ctx[lookup]))
        self.calls += 1
        return out


class DirectLeafEvaluator:
    """values(leaf) = model(beliefs at the leaf): the network is trained to predict the
    pre-chance value itself, which is how the upstream CFR loop calls it."""

    def __init__(self, model, boards: torch.Tensor, context: torch.Tensor, device: torch.device):
        self.model = model
        self.boards = boards.to(device=device, dtype=torch.int64).contiguous()
        self.context = context.to(device=device, dtype=torch.float32).contiguous()

        # a bf16 `ValueMLP` reads rows that the feature kernel writes: the columns that no pass changes (board
        # one-hot, context, padding) are filled in once
        self._rows = None
        self._rows_lock = threading.RLock()
        if type(model) is ValueMLP and model.dtype == torch.bfloat16 and self.boards.is_cuda and self.boards.shape[0] > 0:
            L, first = self.boards.shape[0], 2 * NUM_HANDS
            x = torch.zeros(L, ValueMLP.IN_PADDED, device=device, dtype=torch.bfloat16)
            card = torch.arange(52, device=device)
            x[:, first: first + 52] = (self.boards[:, :, None] == card).any(dim=1)
            x[:, first + 52: ValueMLP.IN_FEATURES] = self.context
            self._rows = x
            self._rows_stream = _lib.stream_ptr(x.device)  # where the rows are at home

    def evaluate_into(self, leaf_beliefs: torch.Tensor, out: torch.Tensor) -> None:
        """Values of all leaves into out[..., :1326] (fp32 [L,2,W])."""
        if not (self._direct() and _paired_rows(leaf_beliefs, self._rows) and _paired_rows(out, self._rows)):
            out[..., :NUM_HANDS].copy_(self.model(leaf_beliefs[..., :NUM_HANDS].contiguous(), self.boards, self.context))
            return
        p, L = _lib.ptr, leaf_beliefs.shape[0]
        # calls from several threads take the rows in turn, calls on another stream (or recorded for later) a copy of them
        with _lib.on(out.device), torch.no_grad(), self._rows_lock:
            stream, rows = _lib.stream_ptr(out.device), self._rows
            if stream != self._rows_stream:
                rows = rows.clone()
                if not torch.cuda.is_current_stream_capturing():
                    self._rows.record_stream(torch.cuda.current_stream(out.device))
            _lib.call("p2b_leaf_features_bf16", p(leaf_beliefs), leaf_beliefs.stride(1), L, p(rows), rows.stride(0), stream)
            y = self.model.layers(rows)
            _lib.call("p2b_leaf_values_bf16", p(y), y.stride(0), L, p(out), out.stride(1), stream)

    def __getstate__(self):  # (a lock is neither copied nor pickled)
        return {k: v for k, v in self.__dict__.items() if k != "_rows_lock"}

    def __setstate__(self, state):
        self.__dict__.update(state, _rows_lock=threading.RLock())

    def _direct(self) -> bool:
        """The model's layers may be called on rows kept here instead of the model itself."""
        return self._rows is not None and type(self.model) is ValueMLP and _bare(self.model)

    def __call__(self, leaf_beliefs: torch.Tensor) -> torch.Tensor:
        if not self._direct():
            return self.model(leaf_beliefs[..., :NUM_HANDS].contiguous(), self.boards, self.context)
        out = torch.empty(leaf_beliefs.shape[0], 2, NUM_HANDS, device=leaf_beliefs.device, dtype=torch.float32)
        self.evaluate_into(leaf_beliefs, out)
        return out


def _paired_rows(t: torch.Tensor, network_rows: torch.Tensor) -> bool:
    """[L,2,W] fp32, rows of whole pairs of hands one after the other, as many leaves as there are network rows."""
    if t.dim() != 3 or t.dtype != torch.float32 or t.device != network_rows.device:
        return False
    leaves, players, width = t.shape
    per_leaf, per_player, per_hand = t.stride()
    return (leaves == network_rows.shape[0] and players == 2 and width >= NUM_HANDS and per_hand == 1
            and per_leaf == 2 * per_player and per_player % 2 == 0 and t.data_ptr() % 8 == 0)
