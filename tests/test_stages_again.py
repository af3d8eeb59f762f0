"""A stage called again on the same upload: building the grid a second time starts its counters
again, but the stages after it still give what they give on one grid, bit for bit.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene():
    from postmps_gb300 import synth
    pos = synth.lattice(23, 19, 14, 0.005, 0.0008, seed=9)
    vel = np.random.default_rng(3).normal(0, 3.0, pos.shape).astype(np.float32)
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "true", "config.issurfacereconstruct": "true"})
    return pos, vel, text


@pytest.mark.parametrize("before", ["surface", "anisotropy", None])
def test_diffuse_after_a_second_grid(pms_lib, tmp_config, before):
    pos, vel, text = scene()
    results = []
    for again in (False, True):
        with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
            frames = []
            for _ in range(2):                                  # the second frame carries particles
                ctx.upload(pos, vel)
                ctx.build_grid()
                if before:
                    getattr(ctx, before)()
                if again:
                    ctx.build_grid()
                ctx.diffuse()
                c = ctx.counts()
                frames.append([ctx.debug("diffuse_potential"), ctx.debug("diffuse_count"), *(
                    v for _, v in sorted(ctx.diffuse_particles(-1).items())), np.array([c.n_free_surface, c.n_spawning])])
            results.append(frames)
    assert results[0][0][0][:, 0].max() > 0 and results[0][0][1].max() > 0        # wave crests, spawned particles
    for one, two in zip(*results):
        for a, b in zip(one, two, strict=True):
            np.testing.assert_array_equal(a, b)
