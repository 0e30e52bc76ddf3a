"""The autotuner where its Jacobi candidates are one kernel: on a small firm
graph FP64 and FP32 storage are the same column solve, which is timed once; on
a dense one every candidate is solved."""

import pytest

from device_trace import kernels, resolve_kernels
from fevc_b200 import abi
from fevc_b200.panel import generate_panel

pytestmark = pytest.mark.gpu


def run(lib, tmp_path, spec, preconditioner, precision):
    """(result, tuning, 64-column solves of the first solve and of a resolve)"""
    e = abi.Engine(lib)
    e.prepare(generate_panel(periods=5, pareto_shape=1.3, seed=21, **spec))
    e.device_options(64, preconditioner, precision)
    q = e.default_request()
    q.probes = 64

    def solves(launched):
        wide = ("k_pcg_flex<64", "k_pcg_persistent<64")
        return sum(name.startswith(wide) or (name.startswith("k_pcg_columns") and grid[0] == 64)
                   for name, grid, _ in launched)

    first = solves(kernels(lambda: e.solve(q), tmp_path))
    res, tuning = e.result(), e.tuning()
    assert solves(resolve_kernels(e, tmp_path)) == 3  # one leverage block, two target blocks
    assert e.result() == res
    e.release()
    return res, tuning, first


def test_equal_candidates_are_solved_once(lib, tmp_path):
    spec = dict(workers=6_000, firms=600, move_p=0.3)
    want, _, _ = run(lib, tmp_path, spec, 1, 0)
    got, t, first = run(lib, tmp_path, spec, 1, 2)
    assert [(c["precision"], c["preconditioner"]) for c in t["candidates"]] == [(0, 1), (1, 1)]
    assert t["candidates"][0]["ms"] == t["candidates"][1]["ms"] > 0.0
    assert t["chosen"] == 0 and first == 3  # its solve serves the first block
    assert got == want
    got, t, first = run(lib, tmp_path, spec, 4, 2)
    assert [(c["precision"], c["preconditioner"]) for c in t["candidates"]] == [(0, 1), (1, 1), (1, 4)]
    assert t["candidates"][0]["ms"] == t["candidates"][1]["ms"] > 0.0 and t["candidates"][2]["ms"] > 0.0
    assert t["chosen"] in (0, 2) and first == (4 if t["chosen"] == 2 else 5)


def test_different_candidates_are_each_solved(lib, tmp_path):
    spec = dict(workers=95_000, firms=1_900, move_p=0.15)
    _, t, first = run(lib, tmp_path, spec, 4, 2)
    assert len(t["candidates"]) == 3 and all(c["ms"] > 0.0 for c in t["candidates"])
    assert first == (5 if t["chosen"] == 2 else 6)
