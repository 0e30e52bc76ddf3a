"""Panels whose largest firms span from a few to thousands of 32-cell segments
(the hub rows one block sums), at every block width: the components equal the
oracle's, whose sums run firm by firm."""

import numpy as np
import pytest

from fevc_b200 import abi
from fevc_b200.panel import generate_panel
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block", [2, 8, 16, 32, 64])
@pytest.mark.parametrize("workers,firms,pareto", [(2500, 4, 1.5), (9000, 60, 0.6), (12000, 2500, 0.7)])
def test_hub_firms_match_the_oracle(lib, block, workers, firms, pareto):
    e = abi.Engine(lib)
    e.prepare(generate_panel(workers, firms, 5, move_p=0.4, pareto_shape=pareto, seed=31))
    e.device_options(block, 1, 0)
    q = e.default_request()
    q.probes = 9
    q.pcg_tolerance = 1e-12
    e.solve(q)
    got = e.result()
    want = oracle.run(oracle.problem_view(lib, e.generation), probes=9)
    e.release()
    for key, okey in (("plugin", "plugin"), ("corrected", "corrected"), ("numerical_mcse", "mcse")):
        a, b = np.array(got[key]), want[okey]
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), key  # the suite's component tolerance
