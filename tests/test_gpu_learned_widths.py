"""The training pass's gradient against the oracle at every number of training
pairs (24, 48, 96 and 192: one to six columns a lane), on graphs with fewer and
more vertices than a grid has blocks, hub rows among them."""

import numpy as np
import pytest

from fevc_b200 import learned
from fevc_b200.panel import generate_panel
from oracle import gnn_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("columns", [8, 16, 32, 64])
@pytest.mark.parametrize("workers,firms", [(300, 40), (4000, 700), (6000, 1300)])
def test_gradient_at_every_pair_count(lib, columns, workers, firms):
    with learned.Trainer(lib, seed=4) as t:
        t.add_panel(generate_panel(workers, firms, 5, move_p=0.3, pareto_shape=1.1, seed=9), columns=columns, seed=5)
        params = t.params
        rng = np.random.default_rng(columns)
        params += 0.05 * rng.standard_normal(params.size).astype(np.float32)
        t.params = params
        loss, grad = t.gradient(0)
        ref_loss, ref = gnn_oracle.loss_and_grad(t.dump(0), params)
    # the bounds of the suite's gradient check: FP32 activations and products
    # against the oracle's float64
    assert abs(loss - ref_loss) <= 1e-4 * abs(ref_loss)
    assert np.linalg.norm(grad - ref) < 2e-3 * np.linalg.norm(ref)
