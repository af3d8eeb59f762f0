"""The band marking at the edges of its tiles (32 x 4 x 8 vertices, a row per lane): grids
whose sides are not multiples of a tile's, boxes wider than a tile's rows, flagged and
unflagged particles.  Bit for bit against the oracle's band test on the GPU's own normals
and flags.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,jitter,ratio,sc", [
    ((1, 1, 2), 0.002, 2, 2), ((3, 2, 1), 0.002, 1, 1), ((13, 3, 7), 0.004, 2, 1), ((12, 5, 9), 0.002, 2, 2),
    ((25, 24, 2), 0.001, 2, 2), ((7, 9, 10), 0.003, 4, 3), ((15, 6, 16), 0.005, 3, 2)])
def test_band_matches_oracle(pms_lib, oracle, tmp_config, dims, jitter, ratio, sc):
    from postmps_gb300 import synth
    text = synth.config_text(**{"surface.smoothingradiusratio": ratio, "domain.sclargridsizescale": sc})
    pos = synth.lattice(*dims, 0.01, jitter, seed=77, origin=(-0.37, 1.91, 0.05))
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        ctx.anisotropy()
        ctx.band()
        perm, slist, normal, flag = (ctx.debug(k) for k in ("perm", "surf_list", "normal", "flag"))
        bitmap, band = ctx.debug("band_bitmap"), ctx.debug("band_list")
    p = oracle.derive_params(oracle.config_from_keys(oracle.parse_ini(text)))
    g = oracle.grid_from_positions(p, pos)
    want_bitmap, want = oracle.band_bitmap(g, p.h, np.ascontiguousarray(pos[perm]), slist, normal, flag)
    np.testing.assert_array_equal(band, want)
    np.testing.assert_array_equal(bitmap, want_bitmap[: len(bitmap)])
