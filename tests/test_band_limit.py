"""The most band vertices a field is made for, 2^29: more are refused by the field and by a frame,
not by the band alone; a batch, whose graph does not look at the count, refuses every frame whose
scalar grid is that large, and a single frame of such a grid with a small band runs.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_band_above_the_limit(pms_lib, tmp_config):
    from postmps_gb300 import synth
    text = synth.config_text(**{"surface.smoothingradiusratio": 4, "domain.sclargridsizescale": 32})
    pos = synth.lattice(24, 24, 24, 0.01, 0.001, seed=1)
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        ctx.anisotropy()
        ctx.band()
        assert 1 << 29 <= ctx.counts().n_band_vertices < 1 << 30
        with pytest.raises(pms_lib.PmsError, match="2\\^29"):
            ctx.field()
        with pytest.raises(pms_lib.PmsError, match="2\\^29"):
            ctx.surface()


@pytest.mark.parametrize("band", ["plain", "certified"])
def test_batch_of_a_grid_above_the_limit(pms_lib, tmp_config, band):
    from postmps_gb300 import synth
    corner = synth.lattice(5, 5, 5, 0.01, 0.001, seed=1)
    frames = [(np.concatenate([corner, corner + np.float32(d)]), None, None) for d in (0.5, 4.05)]
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        with pytest.raises(pms_lib.PmsError, match="2\\^29"):
            ctx.run_batch(frames, learned=band)
        ctx.run_batch(frames[:1], learned=band)
        small = ctx.batch_mesh(0)
        ctx.upload(frames[1][0])
        ctx.build_grid()
        assert ctx.grid().sc_size >= 1 << 29
        ctx.surface()
        assert len(small) > 0 and len(ctx.mesh(False)[0]) > 0
