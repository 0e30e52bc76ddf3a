"""How a block's solve ends other than by convergence, in the column form and in
the cooperative kernels: the capped learned solve that falls back to the
multigrid form, the iteration limit and a nonpositive curvature."""

import numpy as np
import pytest

from device_trace import count, resolve_kernels
from fevc_b200 import abi, learned
from fevc_b200.panel import Panel, generate_panel

pytestmark = pytest.mark.gpu

PCG_CURVATURE_BREAKDOWN, PCG_MAX_ITERATIONS, FULL_RESIDUAL_FAILED = 60, 63, 64
LEARNED_CAP = 300


def ring_panel(firms, seed=1):
    """Two to four workers between each firm and the next, around a ring: a
    solve takes about as many iterations as there are firms."""
    rng = np.random.default_rng(seed)
    a = np.repeat(np.arange(firms), rng.integers(2, 5, firms))
    n = a.size
    w = np.repeat(np.arange(n), 2)
    f = np.stack([a, (a + 1) % firms], 1).reshape(-1)
    y = rng.normal(0, 0.3, n)[w] + rng.normal(0, 0.2, firms)[f] + rng.normal(0, 0.25, 2 * n)
    ones = np.ones(2 * n)
    return Panel(w + 1.0, f + 1.0, np.arange(1.0, 2 * n + 1), y, ones, ones.copy())


def solve(lib, panel, block, preconditioner, precision, probes=37, tolerance=1e-12, limit=20000):
    if preconditioner == 3:
        learned.install(lib, learned.load_params())
    e = abi.Engine(lib)
    e.prepare(panel)
    e.device_options(block, preconditioner, precision)
    q = e.default_request()
    q.probes = probes
    q.pcg_tolerance = tolerance
    q.maximum_iterations = limit
    try:
        e.solve(q)
    except abi.EngineError:
        e.release()
        raise
    return e


@pytest.mark.parametrize("block,precision", [(32, 0), (64, 0), (64, 1)])
@pytest.mark.parametrize("firms,kernel", [(700, "k_pcg_columns<true, 1"), (1300, "k_pcg_columns<true, 2"),
                                          (2400, "k_pcg_flex")])
def test_capped_learned_solve_falls_back_to_multigrid(lib, tmp_path, firms, kernel, block, precision):
    probes = 37
    panel = ring_panel(firms)
    e = solve(lib, panel, block, 3, precision, probes)
    got, t, receipts = e.result(), e.timings(), e.rhs_receipts(1 + 3 * probes)
    launched = resolve_kernels(e, tmp_path)
    again, t2 = e.result(), e.timings()
    e.release()
    assert t["vertices"] == firms
    # every block of probe columns was capped, and went on where it stood; the
    # fit's single column has no learned form and no cap
    blocks = -(-probes // block) + -(-2 * probes // block)
    assert count(launched, kernel) == count(launched, "k_reactivate") == blocks == t["fallbacks"] == t2["fallbacks"]
    iterations = [r["iterations"] for r in receipts[1:]]
    assert LEARNED_CAP < max(iterations) < LEARNED_CAP + 200 and min(iterations) >= 1
    assert max(r["complete_residual"] for r in receipts) <= 1e-11  # ten times the tolerance, the solver's gate
    assert again == got
    e = solve(lib, panel, block, 2, 0, probes)
    want = e.result()
    e.release()
    # components are quadratic in solutions that meet 1e-12: the suite's 1e-8
    for key in ("plugin", "correction", "corrected", "numerical_mcse"):
        a, b = np.array(got[key]), np.array(want[key])
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), key


FORMS = [(64, 1, 0), (64, 1, 1), (64, 4, 0), (64, 3, 1), (32, 1, 0), (32, 4, 1), (8, 1, 0), (2, 1, 0)]


@pytest.mark.parametrize("block,preconditioner,precision", FORMS)
@pytest.mark.parametrize("firms", [100, 1400, 2600])
def test_iteration_limit_is_reported(lib, firms, block, preconditioner, precision):
    panel = generate_panel(6 * firms, firms, 5, move_p=0.3, pareto_shape=2.0, seed=3)
    with pytest.raises(abi.EngineError) as caught:
        solve(lib, panel, block, preconditioner, precision, limit=4)
    assert caught.value.code == PCG_MAX_ITERATIONS, str(caught.value)
    # a limit that just suffices
    e = solve(lib, panel, block, preconditioner, precision, probes=9)
    most = max(r["iterations"] for r in e.rhs_receipts(1 + 3 * 9))
    want = e.result()
    e.release()
    e = solve(lib, panel, block, preconditioner, precision, probes=9, limit=most)
    assert e.result() == want
    e.release()
    with pytest.raises(abi.EngineError) as caught:
        solve(lib, panel, block, preconditioner, precision, probes=9, limit=most - 1)
    assert caught.value.code == PCG_MAX_ITERATIONS, str(caught.value)


@pytest.mark.parametrize("block,preconditioner,precision", FORMS)
@pytest.mark.parametrize("firms", [100, 2600])
def test_overflowing_outcomes_break_down(lib, firms, block, preconditioner, precision):
    panel = generate_panel(6 * firms, firms, 5, move_p=0.3, pareto_shape=2.0, seed=3)
    panel.outcome = panel.outcome * 1e160
    with pytest.raises(abi.EngineError) as caught:
        solve(lib, panel, block, preconditioner, precision)
    assert caught.value.code == PCG_CURVATURE_BREAKDOWN, str(caught.value)


@pytest.mark.parametrize("block,preconditioner", [(64, 1), (64, 4), (8, 1)])
def test_unreachable_tolerance_is_reported(lib, block, preconditioner):
    """A long ring at a tolerance below what its conditioning allows: the
    column form's probe blocks stop on a nonpositive curvature, at the iteration
    limit or after the refinement steps, whichever rounding brings first."""
    with pytest.raises(abi.EngineError) as caught:
        solve(lib, ring_panel(1600), block, preconditioner, 0, probes=33, tolerance=1e-12)
    assert caught.value.code in (PCG_CURVATURE_BREAKDOWN, PCG_MAX_ITERATIONS, FULL_RESIDUAL_FAILED), str(caught.value)
