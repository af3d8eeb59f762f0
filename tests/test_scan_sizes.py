"""Prefix sums at the sizes where their form changes: one block, one cluster, and the
two-launch form with full and ragged rows.  The cell starts of a frame are the scan of
its cell counts, so grids of chosen sizes exercise each; integers, compared exactly.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# cells per axis spanned by the particles (the grid adds its margin around them)
@pytest.mark.parametrize("cells", [(1, 1, 1), (9, 8, 10), (11, 11, 9), (45, 44, 44), (45, 46, 45), (77, 61, 52), (300, 90, 41)])
def test_cell_starts_are_the_scan_of_the_counts(pms_lib, tmp_config, cells):
    from postmps_gb300 import synth
    cs, n = 0.015, 3001
    pos = np.stack([synth.uniform(5, k, n) * cells[k] * cs for k in range(3)], 1).astype(np.float32)
    pos[0], pos[1] = 0.0, np.asarray(cells, np.float32) * np.float32(cs)
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        size = ctx.grid().sp_size
        keys, start, end = (ctx.debug(k) for k in ("keys_sorted", "cell_start", "cell_end"))
    count = np.bincount(keys, minlength=size)
    first = np.concatenate([[0], np.cumsum(count)[:-1]])
    np.testing.assert_array_equal(start, np.where(count > 0, first, 0))
    np.testing.assert_array_equal(end, np.where(count > 0, first + count, 0))
    np.testing.assert_array_equal(keys, np.sort(keys))
