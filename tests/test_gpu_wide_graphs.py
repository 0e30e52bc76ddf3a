"""The cooperative solve kernels on a firm graph too large for the column solve
(more than 2,048 vertices), each form at every width it has, against the oracle."""

import numpy as np
import pytest

from device_trace import resolve_kernels
from fevc_b200 import abi, learned
from fevc_b200.panel import generate_panel
from oracle import oracle

pytestmark = pytest.mark.gpu

PROBES = 37


def prepared(lib):
    e = abi.Engine(lib)
    e.prepare(generate_panel(15_000, 2_600, 5, move_p=0.3, pareto_shape=1.5, seed=3))
    return e


@pytest.fixture(scope="module")
def want(lib):
    e = prepared(lib)
    res = oracle.run(oracle.problem_view(lib, e.generation), probes=PROBES)
    e.release()
    return res


# (block width, preconditioner, precision): the kernel that solves full blocks.
# FP64 Jacobi blocks of two columns and more; FP32 storage, the uniform and the
# learned degree-1 stage in both storages.
FORMS = [(2, 1, 0, "k_pcg_persistent<2,"), (8, 1, 0, "k_pcg_persistent<8,"), (16, 1, 0, "k_pcg_persistent<16,"),
         (32, 1, 0, "k_pcg_persistent_cg<32,"), (64, 1, 0, "k_pcg_persistent<64,")]
FORMS += [(k, pre, prec, f"k_pcg_flex<{k}, {'float' if prec else 'double'}, {'false' if pre == 1 else 'true'}>")
          for k in (32, 64) for pre, prec in ((1, 1), (4, 0), (4, 1), (3, 0), (3, 1))]


@pytest.mark.parametrize("block,preconditioner,precision,kernel", FORMS)
def test_cooperative_forms_match_the_oracle(lib, tmp_path, want, block, preconditioner, precision, kernel):
    if preconditioner == 3:
        learned.install(lib, learned.load_params())
    e = prepared(lib)
    e.device_options(block, preconditioner, precision)
    q = e.default_request()
    q.probes = PROBES
    q.pcg_tolerance = 1e-12
    q.maximum_iterations = 20000
    e.solve(q)
    got, t = e.result(), e.timings()
    receipts = e.rhs_receipts(1 + 3 * PROBES)
    names = [name for name, _, _ in resolve_kernels(e, tmp_path)]
    e.release()
    assert t["vertices"] > 2048 and t["fallbacks"] == 0
    assert any(name.startswith(kernel) for name in names), sorted(set(names))
    assert not any(name.startswith("k_pcg_columns") for name in names)
    assert max(r["complete_residual"] for r in receipts) <= 1e-11  # ten times the tolerance, the solver's gate
    for key, okey in (("plugin", "plugin"), ("corrected", "corrected"), ("numerical_mcse", "mcse")):
        a, b = np.array(got[key]), want[okey]
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), key  # the suite's component tolerance


@pytest.mark.parametrize("preconditioner,precision", [(1, 1), (4, 0), (3, 1)])
def test_exact_leverages_agree_between_the_forms(lib, preconditioner, precision):
    """The exact estimator above the column solve's size: every form's blocks
    give the FP64 Jacobi form's components."""
    if preconditioner == 3:
        learned.install(lib, learned.load_params())
    out = []
    for pre, prec in ((1, 0), (preconditioner, precision)):
        e = abi.Engine(lib)
        e.prepare(generate_panel(6_000, 2_600, 6, move_p=0.3, pareto_shape=2.5, seed=1))
        e.device_options(64, pre, prec)
        e.exact_ceiling(1_000_000)
        e.solve_v5(e.exact_request_v5())
        assert e.timings()["vertices"] > 2048
        out.append(e.result())
        e.release()
    for key in ("plugin", "correction", "corrected"):
        a, b = np.array(out[1][key]), np.array(out[0][key])
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), key  # the suite's component tolerance
