"""Welded meshes on both sides of the line where a mesh with normals changes its kernel: positions are
those of the weld without normals bit for bit (a form of its own below the line), and the normals the
soup's up to the rounding of the interpolation direction (but for a vertex in ten thousand, where the
two ends' normals nearly cancel).
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,low,high", [(3, 1, 10000), (30, 100000, 400000), (58, 400000, 1 << 24)])
def test_weld_forms(pms_lib, tmp_config, side, low, high):
    from postmps_gb300 import synth
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(synth.lattice(side, side, side, 0.01, 0.001, seed=3))
        ctx.run_frame()
        soup, soup_n = ctx.mesh()
        plain, _, plain_idx = ctx.weld(normals=False)
        pos, nrm, idx = ctx.weld(normals=True)
    assert low <= len(soup) < high
    np.testing.assert_array_equal(pos, plain)
    np.testing.assert_array_equal(idx, plain_idx)
    at = idx.reshape(-1)
    assert len(np.unique(at)) == len(pos) and at.max() < len(pos)
    assert np.mean(np.abs(nrm[at] - soup_n).max(axis=1) < 1e-3) > 0.9999
