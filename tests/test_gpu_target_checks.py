"""Target right-hand sides that cannot be balanced: weights whose total has no
finite reciprocal.  Every solver form reports the balance check ahead of
anything its solve of them runs into."""

import numpy as np
import pytest

from fevc_b200 import abi, learned
from fevc_b200.panel import generate_panel

pytestmark = pytest.mark.gpu

TARGET_CENTERING_FAILED = 77


@pytest.mark.parametrize("workers,firms", [(1_000, 100), (15_000, 2_600)])
@pytest.mark.parametrize("block,preconditioner,precision", [(64, 1, 0), (64, 1, 1), (64, 3, 1), (64, 4, 0), (64, 2, 0),
                                                           (8, 1, 0), (8, 2, 0), (2, 1, 0)])
def test_unbalanced_targets_are_refused(lib, workers, firms, block, preconditioner, precision):
    panel = generate_panel(workers, firms, 5, move_p=0.3, pareto_shape=1.5, seed=3)
    if preconditioner == 3:
        learned.install(lib, learned.load_params())
    total = 4e-309  # 1 / total overflows
    panel.target_weight = np.full(panel.rows, total / panel.rows)
    e = abi.Engine(lib)
    e.prepare(panel)
    e.device_options(block, preconditioner, precision)
    q = e.default_request()
    q.probes = 33
    with pytest.raises(abi.EngineError) as caught:
        e.solve(q)
    vertices = e.receipt()["firms"]
    e.release()
    assert (vertices > 2048) == (firms > 2048)
    assert caught.value.code == TARGET_CENTERING_FAILED, str(caught.value)
    # the generation's next call is unaffected
    e = abi.Engine(lib)
    panel.target_weight = np.ones(panel.rows)
    e.prepare(panel)
    e.device_options(block, preconditioner, precision)
    e.solve(q)
    assert np.all(np.isfinite(e.result()["corrected"]))
    e.release()
