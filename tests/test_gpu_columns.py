"""The one-block-per-column solve on Laplacians around its size limits (thread
counts at 64 and 256 vertices, two vertices a thread above 1,024, the matrix in
shared memory up to about 1,150, the cooperative kernels above 2,048): Jacobi
and the degree-1 stage against the multigrid solve of the same columns."""

import numpy as np
import pytest

from fevc_b200 import abi
from fevc_b200.panel import generate_panel

pytestmark = pytest.mark.gpu


def solve(lib, panel, probes, block, preconditioner, precision):
    e = abi.Engine(lib)
    e.prepare(panel)
    e.device_options(block, preconditioner, precision)
    q = e.default_request_v5()
    q.v4.v3.v2.algorithm = 2
    q.v4.v3.v2.v1.probes = probes
    q.v4.v3.v2.v1.pcg_tolerance = 1e-12
    q.v4.v3.v2.v1.maximum_iterations = 20000
    e.solve_v5(q)
    res, vertices = e.result(), e.timings()["vertices"]
    worst = max(r["complete_residual"] for r in e.rhs_receipts(1 + 3 * probes))
    e.release()
    return res, vertices, worst


@pytest.mark.parametrize("firms", [12, 68, 262, 1010, 1040, 1200, 2030, 2090])
@pytest.mark.parametrize("block,probes", [(2, 3), (64, 37)])
def test_column_solve_matches_the_multigrid_solve(lib, firms, block, probes):
    panel = generate_panel(12 * firms, firms, 5, move_p=0.3, pareto_shape=1.3, seed=firms)
    want, n, _ = solve(lib, panel, probes, block, 2, 0)
    assert 0.85 * firms <= n <= firms
    for preconditioner, precision in ((1, 0), (4, 0), (4, 1)):
        got, _, worst = solve(lib, panel, probes, block, preconditioner, precision)
        assert worst <= 1e-11  # ten times the reduced tolerance, the solver's own gate
        # components are quadratic in solutions that meet 1e-12: the suite's 1e-8
        for key in ("plugin", "correction", "corrected", "numerical_mcse"):
            a, b = np.array(got[key]), np.array(want[key])
            assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), (key, preconditioner, precision)
