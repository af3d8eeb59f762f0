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


@pytest.mark.parametrize("band", ["band", "band_learned"])
@pytest.mark.parametrize("first", ["band", "field", "marching_cubes"])
def test_surface_after_a_second_grid(pms_lib, tmp_config, band, first):
    """The surface stages from `first` on run after a second grid, on what the stages before left."""
    pos, vel, text = scene()
    once = ["anisotropy", "band", "field", "marching_cubes"] if band == "band" else ["anisotropy", band, "marching_cubes"]
    then = once[1:] if first == "band" else ["field", "marching_cubes"] if first == "field" else ["marching_cubes"]
    results = []
    for again in (False, True):
        with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
            ctx.set_band_mode("certified")                      # (read by band_learned alone)
            ctx.upload(pos, vel)
            for stage in ["build_grid"] + once + (["build_grid"] + then if again else []):
                getattr(ctx, stage)()
            results.append([ctx.mesh(False)[0], ctx.weld(False)])
            if first != "marching_cubes":
                results[-1] += [ctx.debug("band_list"), ctx.debug("surf_list")]
                if band == "band":
                    results[-1].append(ctx.debug("field"))
    assert len(results[0][0]) > 0
    for a, b in zip(*results, strict=True):
        for x, y in zip(a, b, strict=True) if isinstance(a, tuple) else [(a, b)]:
            np.testing.assert_array_equal(x, y)


def test_autotune_after_a_second_grid(pms_lib, tmp_config):
    pos, vel, text = scene()
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos, vel)
        ctx.build_grid()
        ctx.surface()
        mesh, field = ctx.mesh(False)[0], ctx.debug("field")
        ctx.build_grid()
        assert ctx.autotune()["field_ms"] > 0
        ctx.marching_cubes()
        np.testing.assert_array_equal(ctx.mesh(False)[0], mesh)
        np.testing.assert_array_equal(ctx.debug("field"), field)


def test_normals_after_a_second_grid(pms_lib, tmp_config):
    """The colour-gradient normals that a frame left out are still made after a second grid."""
    pos, vel, text = scene()
    vel[len(vel) // 20:] = 0.0                                  # few particles that can spawn
    normals = []
    for again in (False, True):
        with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
            ctx.upload(pos, vel)
            ctx.run_frame()
            if again:
                ctx.build_grid()
            normals.append(ctx.debug("free_normal"))
    assert np.any(normals[0] != 0)
    np.testing.assert_array_equal(normals[1], normals[0])


def test_results_on_demand_after_a_second_grid(pms_lib, tmp_config):
    """A mesh made before the second grid: its normals, welded mesh and scalar values."""
    pos, vel, text = scene()
    results = []
    for again in (False, True):
        with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
            ctx.upload(pos, vel)
            ctx.run_frame()
            if again:
                ctx.build_grid()
            results.append([*ctx.mesh(True), *ctx.weld(True), *(v for _, v in sorted(ctx.scalar_values().items())),
                            ctx.debug("band_list"), ctx.debug("field"), np.array(ctx.counts().n_mesh_vertices)])
    assert len(results[0][0]) > 0
    for a, b in zip(*results, strict=True):
        np.testing.assert_array_equal(a, b)
