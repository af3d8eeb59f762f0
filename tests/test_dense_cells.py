"""Cells holding many particles: the order inside a cell is the input's (a stable sort by
key) up to the most particles a cell may hold; one more is refused.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_cell", [1, 63, 64, 65, 1000, 4096])
def test_cell_order_is_the_input_order(pms_lib, tmp_config, per_cell):
    from postmps_gb300 import synth
    n = 3 * per_cell
    # three cells in a row of the grid, particles dealt to them in turn
    pos = np.stack([synth.uniform(3, k, n) * 0.002 for k in range(3)], 1).astype(np.float32)
    pos[:, 0] += np.float32(0.015) * (np.arange(n) % 3).astype(np.float32)
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        keys, perm, out = (ctx.debug(k) for k in ("keys_sorted", "perm", "pos_sorted"))
    np.testing.assert_array_equal(out, pos[perm])
    np.testing.assert_array_equal(np.sort(perm), np.arange(n))
    same = keys[1:] == keys[:-1]
    assert np.all(keys[1:] >= keys[:-1]) and np.all(perm[1:][same] > perm[:-1][same])


def test_overfull_cell_is_refused(pms_lib, tmp_config):
    from postmps_gb300 import synth
    pos = np.stack([synth.uniform(3, k, 4097) * 0.002 for k in range(3)], 1).astype(np.float32)
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        with pytest.raises(pms_lib.PmsError):
            ctx.surface()
