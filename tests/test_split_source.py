"""The two kernels of a pass (cfr_split.cu) may start before the kernel ahead of them has ended.  Were the status word written
meanwhile, threads of one block could read different words, and the ones that stay would wait at a barrier for the others.
So a kernel that can be ahead of such a one never writes the word (a wait that runs out has a word of its own), and in every
other kernel a block reads it once and leaves as a whole.  The event itself cannot be staged; this holds the source to the rule."""
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


def test_blocks_leave_a_kernel_as_a_whole():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    bodies = {}
    for m in re.finditer(r"__global__", text):
        name = re.search(r"(\w+_kernel)\(", text[m.start():]).group(1)
        bodies[name] = _body(text, text.index(")", text.index("_kernel(", m.start())))
    assert len(bodies) >= 8
    overlapped = {n for n, b in bodies.items() if "previous_done()" in b}
    launched_early = set(re.findall(r"launch_pass_kernel\((\w+_kernel)", text))
    assert overlapped == launched_early == {"split_rows_kernel", "split_up_kernel"}
    for name, body in bodies.items():
        check = "if (refused(p)) return;" if name in overlapped else "if (block_refused(p))"
        at = body.find(check)
        assert at >= 0, f"{name}: leaves by another rule"
        for early in ("return", "bar.sync", "__shfl", "previous_done()", "launch_next()", "level_wait(", "__syncwarp"):
            found = body.find(early)
            assert found < 0 or found >= at, f"{name}: {early} before the status word has been asked"
        if name in overlapped:  # a kernel that another may overlap leaves the word alone
            assert "work_counter" not in body and "report_gave_up" not in body, f"{name} writes the status word"
    block = _body(text, text.index("bool block_refused("))
    assert "__syncthreads_or(threadIdx.x == 0 &&" in block
    # nothing else in the file reads the word
    assert len(re.findall(r"work_counter(?:\[1\]| \+ 1)", text.replace("atomicMax(p.work_counter + 1", ""))) == 2
