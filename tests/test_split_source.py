"""The kernels of cfr_split.cu may start before the kernel ahead of them has ended, and that one may still set the status word.
So no thread may leave a kernel by what it alone read there: the others of its block would wait for it at a barrier.  The
event itself (a wait that ran out in one block while the next kernel starts) cannot be staged; this holds the source to the rule."""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "poker2_b200", "csrc", "cfr_split.cu")


def _body(text, start):
    open_at = text.index("{", start)
    depth = 0
    for i in range(open_at, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[open_at:i]
    raise AssertionError("unbalanced braces")


def test_a_block_leaves_a_kernel_as_a_whole():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    kernels = [m.start() for m in re.finditer(r"__global__", text)]
    assert len(kernels) >= 7
    for at in kernels:
        body = _body(text, text.index(")", text.index("_kernel(", at)))
        name = re.search(r"(\w+_kernel)\(", text[at:]).group(1)
        check = body.find("block_stops(p)")
        assert check >= 0, f"{name}: the status word is not asked by the block as a whole"
        for early in ("return", "bar.sync", "__shfl", "previous_done()", "launch_next()", "level_wait("):
            assert body.find(early) < 0 or body.find(early) > check, f"{name}: {early} before the block has agreed to go on"
    helper = _body(text, text.index("bool block_stops("))
    assert "__syncthreads_or(" in helper and "threadIdx.x == 0" in helper
    reads = re.findall(r"work_counter(?:\[1\]| \+ 1)", text.replace(helper, "").replace("atomicMax(p.work_counter + 1", ""))
    assert not reads, "the status word is read outside block_stops"
