"""Welded meshes whose edges lie evenly over the words of the edge bitmap (a lane makes a word's) and in
few words (the lanes of a warp share them): blocks, a sheet across the words, isolated particles.  Every
edge is used once, positions do not depend on the normals being asked for, every soup vertex is its
triangle's welded vertex up to the rounding of the interpolation direction (two roundings at the size
of the coordinates), and so are the normals (but for a vertex in ten thousand, where the two ends'
normals nearly cancel).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(kind):
    from postmps_gb300 import synth
    if kind == "isolated":
        return (np.random.default_rng(5).random((3000, 3)) * 0.8).astype(np.float32)
    return synth.lattice(*{"3": (3, 3, 3), "30": (30, 30, 30), "58": (58, 58, 58), "sheet": (90, 80, 2)}[kind], 0.01, 0.001, seed=3)


@pytest.mark.parametrize("kind", ["3", "30", "58", "sheet", "isolated"])
def test_weld_forms(pms_lib, tmp_config, kind):
    from postmps_gb300 import synth
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(scene(kind))
        ctx.run_frame()
        soup, soup_n = ctx.mesh()
        plain, _, plain_idx = ctx.weld(normals=False)
        pos, nrm, idx = ctx.weld(normals=True)
        cs = float(ctx.grid().sc_grid_size)
    assert len(soup) > 0
    np.testing.assert_array_equal(pos, plain)
    np.testing.assert_array_equal(idx, plain_idx)
    at = idx.reshape(-1)
    assert len(np.unique(at)) == len(pos) and at.max() < len(pos)
    assert float(np.abs(pos[at] - soup).max()) <= 2.0 ** -22 * float(np.abs(soup).max()) + 1e-5 * cs
    assert np.mean(np.abs(nrm[at] - soup_n).max(axis=1) < 1e-3) > 0.9999
