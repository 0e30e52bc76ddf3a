"""The multigrid form at every block width: blocks of 32 and 64 columns take one
warp per segment, narrower ones a lane group; both give the Jacobi solve's
components and, column by column, the same iteration counts."""

import numpy as np
import pytest

from fevc_b200 import abi
from fevc_b200.panel import generate_panel

pytestmark = pytest.mark.gpu

# a hub firm's row spans hundreds of segments (Pareto 1.1), the rest a few entries
PANEL = dict(workers=6000, firms=400, periods=5, move_p=0.25, pareto_shape=1.1, seed=17)


def solve(lib, block, preconditioner, probes):
    e = abi.Engine(lib)
    e.prepare(generate_panel(**PANEL))
    e.device_options(block, preconditioner, 0)
    q = e.default_request_v5()
    q.v4.v3.v2.algorithm = 2
    q.v4.v3.v2.v1.probes = probes
    q.v4.v3.v2.v1.pcg_tolerance = 1e-12
    e.solve_v5(q)
    res, receipts = e.result(), e.rhs_receipts(1 + 3 * probes)
    e.release()
    return res, [r["iterations"] for r in receipts]


@pytest.mark.parametrize("block,probes", [(2, 5), (8, 13), (16, 33), (32, 33), (64, 65)])
def test_multigrid_widths_agree(lib, block, probes):
    got, its = solve(lib, block, 2, probes)
    want, _ = solve(lib, 64, 1, probes)
    narrow, its8 = solve(lib, 8, 2, probes)
    # both solves meet a 1e-12 reduced residual; the components are quadratic
    # in the solutions, so two solvers agree to the suite's 1e-8
    for key in ("plugin", "correction", "corrected", "numerical_mcse"):
        a, b = np.array(got[key]), np.array(want[key])
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), (key, a, b)
    # the widths differ by summation order alone: a column may cross its
    # tolerance one iteration apart, no more
    assert len(its) == len(its8)
    assert max(abs(a - b) for a, b in zip(its, its8)) <= 1
