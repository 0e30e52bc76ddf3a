"""Which solve a block takes on firm graphs of at most 2,048 vertices: one thread
block per column while the graph has few entries, the cooperative kernels on
dense graphs, and the same components either way."""

import numpy as np
import pytest

from device_trace import count, resolve_kernels
from fevc_b200 import abi
from fevc_b200.panel import generate_panel

pytestmark = pytest.mark.gpu

# entries + 16 vertices: 15,000 (every width takes the column form), 51,000
# (all but FP64 Jacobi at 32 columns), 108,000 (the fit alone), 357,000 (none)
SPARSE = dict(workers=6_000, firms=600, move_p=0.3)
MIDDLE = dict(workers=50_000, firms=1_000, move_p=0.15)
DENSE = dict(workers=75_000, firms=1_500, move_p=0.15)
DENSEST = dict(workers=380_000, firms=1_900, move_p=0.15)


def run(lib, tmp_path, spec, block, preconditioner, precision, probes):
    e = abi.Engine(lib)
    e.prepare(generate_panel(periods=5, pareto_shape=1.3, seed=spec["firms"], **spec))
    e.device_options(block, preconditioner, precision)
    q = e.default_request_v5()
    q.v4.v3.v2.algorithm = 2
    q.v4.v3.v2.v1.probes = probes
    q.v4.v3.v2.v1.pcg_tolerance = 1e-12
    e.solve_v5(q)
    res, t = e.result(), e.timings()
    launched = resolve_kernels(e, tmp_path)
    e.release()
    return res, t, launched


# (panel, block width, precision, preconditioner): the column form at one
# column (the fit) and at the block's width
RULE = [(SPARSE, 2, 0, 1, True, True), (SPARSE, 8, 0, 1, True, True), (SPARSE, 16, 0, 1, True, True),
        (SPARSE, 32, 0, 1, True, True), (SPARSE, 32, 1, 4, True, True), (SPARSE, 64, 0, 1, True, True),
        (MIDDLE, 8, 0, 1, True, True), (MIDDLE, 32, 0, 1, True, False), (MIDDLE, 32, 1, 1, True, True),
        (MIDDLE, 64, 0, 4, True, True), (DENSE, 2, 0, 1, True, False), (DENSE, 8, 0, 1, True, False),
        (DENSE, 64, 0, 1, True, False), (DENSE, 64, 1, 4, True, False), (DENSEST, 8, 0, 1, False, False),
        (DENSEST, 64, 0, 1, False, False), (DENSEST, 64, 1, 1, False, False)]


@pytest.mark.parametrize("spec,block,precision,preconditioner,one,wide", RULE)
def test_solve_form_follows_the_graph(lib, tmp_path, spec, block, precision, preconditioner, one, wide):
    probes = min(block, 37)
    got, t, launched = run(lib, tmp_path, spec, block, preconditioner, precision, probes)
    n, entries = t["vertices"], 2 * t["edges"]
    cost = entries + 16 * n
    lo, hi = {600: (0, 46_000), 1_000: (46_000, 62_000), 1_500: (90_000, 125_000), 1_900: (125_000, 1e9)}[
        spec["firms"]]
    assert n <= 2048 and lo < cost < hi, (n, entries)
    columns = [grid[0] for name, grid, _ in launched if name.startswith("k_pcg_columns")]
    cooperative = count(launched, "k_pcg_persistent") + count(launched, "k_pcg_flex")
    # one launch a block: the fit's first, then the probe blocks'
    assert (1 in columns) == one, columns
    assert (block in columns) == wide, columns
    assert (cooperative == 0) == (one and wide), launched
    want, _, _ = run(lib, tmp_path, spec, block, 2, 0, probes)
    # components are quadratic in solutions that meet 1e-12: the suite's 1e-8
    for key in ("plugin", "correction", "corrected", "numerical_mcse"):
        a, b = np.array(got[key]), np.array(want[key])
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), key
