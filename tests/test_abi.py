"""The C-ABI library loads and exports every symbol the public header declares."""
import ctypes
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "poker2_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(p2b_[a-z0-9_]+)\s*\(", text)))


def test_library_builds_and_exports_declared_symbols():
    from poker2_b200 import _lib, build

    path = build.build()
    handle = ctypes.CDLL(path)
    declared = _declared_symbols()
    assert len(declared) >= 5
    for name in declared:
        assert hasattr(handle, name), f"{name} is declared in the header but not exported"
    # the Python binding table covers the same set
    assert sorted(_lib.exported_symbols()) == declared
    assert handle.p2b_version() >= 1


def test_product_does_not_import_oracle():
    pkg = os.path.join(ROOT, "poker2_b200")
    for dirpath, _, files in os.walk(pkg):
        for f in files:
            if f.endswith((".py", ".cu", ".cuh", ".h")):
                src = open(os.path.join(dirpath, f)).read()
                assert "import oracle" not in src and "from oracle" not in src, f


def test_tree_builder_rejects_bad_arguments_without_a_gpu():
    """Argument checks come before any CUDA call: status code and message, no launch."""
    from poker2_b200 import _lib, build

    build.build()
    handle = _lib.lib()
    bins = (ctypes.c_float * 16)(*([0.5] * 16))
    dummy = (ctypes.c_int32 * 64)()
    p = ctypes.cast(dummy, ctypes.c_void_p)
    assert handle.p2b_tree_count(p, 1, bins, 14, 4, -1, p, p, None) == -1  # too many bet bins
    assert b"bet bins" in handle.p2b_last_error()
    assert handle.p2b_tree_count(p, 1, bins, 2, 64, -1, p, p, None) == -1  # depth beyond the limit
    assert b"max_depth" in handle.p2b_last_error()
    assert handle.p2b_tree_count(None, 1, bins, 2, 4, -1, p, p, None) == -1  # null roots
    assert handle.p2b_tree_records(p, None, 5, 1, bins, 2, 4, -1, p, p, p, p, p, p, None, None, None) == -1
    assert handle.p2b_tree_count(p, 0, bins, 2, 4, -1, p, p, None) == 0  # empty batch: nothing to do


def test_whole_step_entry_points_reject_bad_arguments_without_a_gpu():
    """`p2b_steps_*`: null and misaligned arrays, negative sizes and a prior inside the beliefs are refused before any launch."""
    from poker2_b200 import _lib, build

    build.build()
    handle = _lib.lib()
    array = (ctypes.c_int64 * 64)()
    p = ctypes.addressof(array)
    good = {
        "p2b_steps_regrets": [p] * 10 + [1, 1, 1, 0, None],
        "p2b_steps_reach": [p, p, p, p, 1, p, p, p, p + 2 * 1326 * 4, 1, None],
        "p2b_steps_average": [p] * 10 + [1, None],
        "p2b_steps_seen": [p] * 6 + [1, None],
    }
    sizes = {"p2b_steps_regrets": (10, 11), "p2b_steps_reach": (4, 9), "p2b_steps_average": (10,), "p2b_steps_seen": (6,)}
    arrays = {"p2b_steps_regrets": range(10), "p2b_steps_reach": (0, 1, 2, 3, 5, 6, 7), "p2b_steps_average": range(10),
              "p2b_steps_seen": range(6)}

    def refused(name, args):
        rc = getattr(handle, name)(*args)
        return rc == -1 and name.encode() in handle.p2b_last_error()

    for name, args in good.items():
        for i in arrays[name]:
            assert refused(name, args[:i] + [None] + args[i + 1:]), (name, i, "null")
            if (name, i) != ("p2b_steps_reach", 1):  # one byte a hand: any address is aligned
                assert refused(name, args[:i] + [args[i] + 1] + args[i + 1:]), (name, i, "misaligned")
        for i in sizes[name]:
            assert refused(name, args[:i] + [-1] + args[i + 1:]), (name, i, "negative")
        nothing = [0 if i in sizes[name] else None if i in arrays[name] else a for i, a in enumerate(args)]
        assert getattr(handle, name)(*nothing) == 0, name  # an empty call: nothing to do
    reach = good["p2b_steps_reach"]
    for beliefs in (p, p + 4, p - 4):
        assert refused("p2b_steps_reach", reach[:8] + [beliefs] + reach[9:]), "overlap"


def test_solves_without_iterations_are_refused_without_a_gpu():
    """No pass of a solve can go without a table of iterations: zero iterations are refused before anything is launched (an empty
    batch has nothing to do whatever it says)."""
    from poker2_b200 import _lib, build

    build.build()
    handle = _lib.lib()
    area = (ctypes.c_char * 4096)()
    p = (ctypes.addressof(area) + 63) // 64 * 64

    def solve(subgames, iterations, scalars):
        return handle.p2b_cfr_solve(p, p, subgames, 8, 5, 2, p, p, p, p, p, p, p, None, None, None, None, p, 1 << 30, scalars,
                                    iterations, 0, 2, p, 1, None, None, None, None, None, 0.0, None)

    def noalloc(subgames, iterations, scalars):
        return handle.p2b_cfr_solve_noalloc(p, p, subgames, 8, 5, 2, p, p, p, p, p, p, p, None, None, None, None, scalars,
                                            iterations, 0, 2, None)

    for call in (solve, noalloc):
        for scalars in (None, p):
            assert call(1, 0, scalars) == -1 and b"at least one iteration" in handle.p2b_last_error()
            assert call(0, 0, scalars) == 0
        assert call(1, 1, None) == -1 and b"null" in handle.p2b_last_error()
