"""The field's tile kernel at the edges of its tiles: grids whose sides are not
multiples of a tile's, bands of a few vertices, kernels wider and narrower than
the default, every vertex count per lane.

Against the float64 oracle: 1e-5 of max(|f|, iso) below the early-exit threshold
(the field's tolerance everywhere in these tests: float sums of up to a few
hundred terms), both past it otherwise.  Between the tile shapes: bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,ratio,sc", [
    ((1, 1, 2), 2, 2), ((3, 2, 1), 1, 1), ((7, 5, 3), 2, 1), ((9, 4, 11), 2, 2), ((6, 13, 5), 3, 2), ((10, 9, 8), 2, 3),
    ((8, 7, 9), 4, 2)])
def test_tiles_match_oracle_and_each_other(pms_lib, oracle, tmp_config, dims, ratio, sc):
    from postmps_gb300 import synth
    text = synth.config_text(**{"surface.smoothingradiusratio": ratio, "domain.sclargridsizescale": sc})
    pos = synth.lattice(*dims, 0.01, 0.002, seed=31)
    got = []
    for vpt in (2, 1, 4):
        for threads in (64, 128, 256):
            with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
                ctx.set_tune({"field_threads": threads, "field_waves": 1, "density_threads": 128, "moments_threads": 128,
                              "field_vpt": vpt})
                ctx.upload(pos)
                ctx.run_frame()
                got.append((ctx.debug("band_list"), ctx.debug("field"), ctx.mesh()[0]))
    for other in got[1:]:
        for a, b in zip(got[0], other):
            np.testing.assert_array_equal(a, b)
    band, field = got[0][0], got[0][1].astype(np.float64)
    p = oracle.derive_params(oracle.config_from_keys(oracle.parse_ini(text)))
    g = oracle.grid_from_positions(p, pos)
    r = oracle.run_surface(p, pos, g)
    ref = np.zeros(len(band))
    if len(band):
        import ctypes as C
        sp = np.ascontiguousarray(pos[r.perm])
        oracle.lib().orc_field(C.byref(p), C.byref(g), sp.reshape(-1), len(pos), r.rho, r.cell_start, r.cell_end,
                               r.surf_count, r.surf_scan, np.ascontiguousarray(r.G.reshape(-1)),
                               np.ascontiguousarray(r.maxv), band, len(band), ref)
    thr = 2 * p.iso_value
    below = (ref < thr * 0.999) & (field < thr * 0.999)
    err = np.abs(field - ref) / np.maximum(np.abs(ref), p.iso_value)
    assert float(err[below].max(initial=0.0)) < 1e-5
    past = ~((ref < thr * 1.001) & (field < thr * 1.001))
    assert np.all((ref[past] > thr * 0.99) & (field[past] > thr * 0.99))
