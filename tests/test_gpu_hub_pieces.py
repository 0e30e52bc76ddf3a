"""A firm of so many workers that its cells' segments are summed in several
pieces (1,024 segments of 32 cells each): piece boundaries, ragged last pieces
and segments, and many pieces, at every kind of block width."""

import numpy as np
import pytest

from device_trace import resolve_kernels
from fevc_b200 import abi
from fevc_b200.panel import Panel
from oracle import oracle

pytestmark = pytest.mark.gpu

PIECE_CELLS = 1024 * 32


def star_panel(workers, firms=300):
    """Every worker holds one job at the hub and one at one of the other firms:
    nothing is pruned, and the hub has one cell a worker."""
    rng = np.random.default_rng(workers)
    w = np.repeat(np.arange(workers), 2)
    f = np.zeros(2 * workers, np.int64)
    f[1::2] = 1 + np.concatenate([np.arange(2 * firms) % firms, rng.integers(0, firms, workers - 2 * firms)])
    y = rng.normal(0, 0.3, workers)[w] + rng.normal(0, 0.2, firms + 1)[f] + rng.normal(0, 0.25, 2 * workers)
    ones = np.ones(2 * workers)
    return Panel(w + 1.0, f + 1.0, np.arange(1.0, 2 * workers + 1), y, ones, ones.copy())


CASES = [(cells, block) for cells in (PIECE_CELLS, PIECE_CELLS + 1, 2 * PIECE_CELLS + 33) for block in (2, 8, 32, 64)]


@pytest.mark.parametrize("cells,block", CASES + [(12 * PIECE_CELLS, 8), (12 * PIECE_CELLS, 64)])
def test_hub_pieces_match_the_oracle(lib, tmp_path, cells, block):
    probes = 5 if cells > 3 * PIECE_CELLS else 9
    e = abi.Engine(lib)
    e.prepare(star_panel(cells))
    e.device_options(block, 1, 0)
    q = e.default_request()
    q.probes = probes
    q.pcg_tolerance = 1e-12
    e.solve(q)
    got = e.result()
    launched = resolve_kernels(e, tmp_path)
    want = oracle.run(oracle.problem_view(lib, e.generation), probes=probes)
    e.release()
    for key, okey in (("plugin", "plugin"), ("corrected", "corrected"), ("numerical_mcse", "mcse")):
        a, b = np.array(got[key]), want[okey]
        assert np.max(np.abs(a - b)) < 1e-8 * np.max(np.abs(b)), key  # the suite's component tolerance
    # the hub's segments, and those of other firms of more than 32 segments,
    # in blocks of at most 1,024
    segments = -(-cells // 32)
    grids = {grid[0] for name, grid, _ in launched if name.startswith("k_hub_rows")}
    assert len(grids) == 1 and min(grids) >= -(-segments // 1024)
