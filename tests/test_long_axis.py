"""A body and a stray particle far from it: grids of more cells along one axis than float32 cell
positions resolve to 0.01 cells, where the walks' margin has to grow with the axis.  A thin sheet
with supports of 2.5 h, so that particles reach past the windows; below the margin's line, above
it, and where a fixed margin cut contributions (2 % of the field).

Keys, density and field against the oracle as everywhere (exact; 1e-5; 1e-5 of max(|f|, iso)
below the early exit).  Not the mesh: its vertices are float32 lattice positions counted from the
grid's far end, so they carry that end's rounding.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from test_gpu_surface import oracle_setup, run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [20000, 30000, 262144])
def test_field_matches_oracle(pms_lib, oracle, tmp_config, cells):
    from postmps_gb300 import synth
    sheet = synth.lattice(20, 6, 1, 0.01, 0.001, seed=1)
    pos = np.concatenate([sheet, np.array([[-cells * 0.015, 0.01, 0.01]], np.float32)])
    text = synth.config_text(**{"surface.smoothingradiusratio": 4, "domain.sclargridsizescale": 1})
    p, g = oracle_setup(oracle, text, pos)
    r = oracle.run_surface(p, pos, g)
    assert cells <= max(g.spres) < cells + 100 and r.maxv.max() > 2.5
    out = run_gpu(pms_lib, tmp_config(text), pos)
    np.testing.assert_array_equal(out["keys_sorted"], r.keys_sorted)
    assert float((np.abs(out["density"] - r.rho) / r.rho).max()) < 1e-5
    spos = np.ascontiguousarray(pos[r.perm])
    _, band = oracle.band_bitmap(g, p.h, spos, r.surf_list, out["normal"], out["flag"])
    np.testing.assert_array_equal(out["band_list"], band)
    want = np.zeros(len(band))
    oracle.lib().orc_field(C.byref(p), C.byref(g), spos.reshape(-1), len(pos), r.rho, r.cell_start, r.cell_end, r.surf_count,
                           r.surf_scan, np.ascontiguousarray(r.G.reshape(-1)), np.ascontiguousarray(r.maxv), band, len(band), want)
    got, thr = out["field"].astype(np.float64), 2 * p.iso_value
    below = (want < thr * 0.999) & (got < thr * 0.999)
    err = np.abs(got - want) / np.maximum(np.abs(want), p.iso_value)
    assert float(err[below].max()) < 1e-5
