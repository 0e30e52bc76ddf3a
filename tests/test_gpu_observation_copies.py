"""Leave-observation-out rows of one copy whose numbers inside their class run
past 32 and 64 (identical rows), and rows of many copies: the one-copy form of
the atom pass against blocks of two columns, half of which start off a multiple
of four and draw the copies one range at a time."""

import numpy as np
import pytest

from fevc_b200 import abi
from fevc_b200.panel import Panel, generate_panel

pytestmark = pytest.mark.gpu


def copies_panel(repeats, frequency):
    p = generate_panel(600, 40, 5, move_p=0.4, year_controls=True, seed=23)
    pick = np.arange(0, p.rows, 97)
    again = np.repeat(pick, repeats)
    freq = np.concatenate([p.frequency, np.full(again.size, float(frequency))])
    cat = lambda a: np.concatenate([a, a[again]])  # noqa: E731
    return Panel(cat(p.worker), cat(p.firm), np.arange(1.0, freq.size + 1), cat(p.outcome), freq, freq.copy(),
                 [cat(c) for c in p.controls])


@pytest.mark.parametrize("repeats,frequency", [(1, 1), (31, 1), (33, 1), (70, 1), (2, 40)])
def test_copies_across_word_halves(lib, repeats, frequency):
    out = {}
    for block in (2, 8, 64):
        e = abi.Engine(lib)
        e.prepare(copies_panel(repeats, frequency), deletion_mode=2)
        e.device_options(block, 1, 0)
        q = e.default_request_v5(2)
        q.v4.v3.v2.algorithm = 2
        q.v4.v3.engine = 2
        q.v4.v3.v2.v1.probes = 70
        q.v4.v3.v2.v1.pcg_tolerance = 1e-12
        e.solve_v5(q, 4)
        out[block] = e.result()
        e.release()
    for block in (8, 64):
        for key in ("plugin", "correction", "corrected", "numerical_mcse"):
            a, b = np.array(out[block][key]), np.array(out[2][key])
            # the same draws and systems, solved to 1e-12 at another width
            assert np.max(np.abs(a - b)) < 1e-9 * np.max(np.abs(b)), (block, key, a, b)


@pytest.mark.parametrize("repeats,frequency", [(7, 1), (9, 2), (1, 16), (2, 17), (1, 18), (3, 34)])
def test_copies_across_update_groups(lib, repeats, frequency):
    """Eight rows and sixteen further copies of a row are updated together in the
    moment pass: counts on both sides of those."""
    out = {}
    for block in (2, 8, 64):
        e = abi.Engine(lib)
        e.prepare(copies_panel(repeats, frequency), deletion_mode=2)
        e.device_options(block, 1, 0)
        q = e.default_request_v5(2)
        q.v4.v3.v2.algorithm = 2
        q.v4.v3.engine = 2
        q.v4.v3.v2.v1.probes = 70
        q.v4.v3.v2.v1.pcg_tolerance = 1e-12
        e.solve_v5(q, 4)
        out[block] = e.result()
        e.release()
    for block in (8, 64):
        for key in ("plugin", "correction", "corrected", "numerical_mcse"):
            a, b = np.array(out[block][key]), np.array(out[2][key])
            # the same draws and systems, solved to 1e-12 at another width
            assert np.max(np.abs(a - b)) < 1e-9 * np.max(np.abs(b)), (block, key, a, b)
