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


@pytest.mark.parametrize("per_cell", [4, 9, 120, 400])
def test_crowded_blocks_match_oracle(pms_lib, oracle, tmp_config, per_cell):
    """Frames past the warp form's size whose blocks of cells hold from less than 32 to thousands of
    particles, with densities near the surface only (all are made for the download): the float64
    densities to 1e-5 and the rounding of a float sum of as many terms as 27 cells hold, and the
    frame's field that of the stages one by one."""
    from postmps_gb300 import synth
    n = 70000
    side = int(round((n / per_cell) ** (1 / 3)))
    cell = np.random.default_rng(per_cell).integers(0, side, (n, 3)).astype(np.float32)
    at = np.stack([synth.uniform(7, k, n) for k in range(3)], 1).astype(np.float32)
    pos = ((cell + at) * np.float32(0.015)).astype(np.float32)
    text = synth.config_text()
    p = oracle.derive_params(oracle.config_from_keys(oracle.parse_ini(text)))
    g = oracle.grid_from_positions(p, pos)
    r = oracle.run_surface(p, pos, g)
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos)
        ctx.run_frame()
        field, density, perm = ctx.debug("field"), ctx.debug("density"), ctx.debug("perm")
        np.testing.assert_array_equal(perm, r.perm)
        terms = 27 * int(np.bincount(r.keys_sorted).max())
        assert float((np.abs(density - r.rho) / r.rho).max()) < 1e-5 + terms * 2.0 ** -24
        for stage in ("build_grid", "anisotropy", "band", "field"):
            getattr(ctx, stage)()
        np.testing.assert_array_equal(ctx.debug("density"), density)
        np.testing.assert_array_equal(ctx.debug("field"), field)
