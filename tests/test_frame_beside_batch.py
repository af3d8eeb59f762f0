"""A batch leaves the context's frame alone: what the frame made, and what is made from it on
demand, is bit for bit the same before and after batches of smaller and larger frames, also
where the batch is refused; and the batch's meshes are those of a context without a frame.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAGES = ("anisotropy", "band", "field", "marching_cubes")


def batch_frames(kind):
    from postmps_gb300 import synth
    sides = {"smaller": (13, 11, 9), "larger": (55, 40, 42), "refused": (13, 11, 9)}[kind]
    frames = [(synth.lattice(*sides, 0.005, 0.0005, seed=k), None, None) for k in range(5)]
    if kind == "refused":
        frames[3][0][7, 1] = np.nan
    return frames


def run_batch(pms, ctx, frames, kind):
    if kind == "refused":
        with pytest.raises(pms.PmsError):
            ctx.run_batch(frames)
        return []
    ctx.run_batch(frames)
    return [ctx.batch_mesh(f) for f in range(len(frames))]


@pytest.mark.parametrize("kind", ["smaller", "larger", "refused"])
def test_frame_results_after_a_batch(pms_lib, tmp_config, kind):
    from postmps_gb300 import synth
    pos = synth.lattice(43, 41, 40, 0.005, 0.0008, seed=4)             # enough to leave far densities out
    vel = np.random.default_rng(3).normal(0, 3.0, pos.shape).astype(np.float32)
    vel[len(vel) // 20:] = 0.0
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "true", "config.issurfacereconstruct": "true"})
    frames = batch_frames(kind)

    def results(ctx):
        yield from ctx.mesh(True)
        yield from ctx.weld(True)
        yield from (v for _, v in sorted(ctx.scalar_values().items()))
        for name in ("density", "band_list", "field", "cube_case", "cube_nvert", "free_normal", "surf_list", "G"):
            yield ctx.debug(name)
        yield np.array(ctx.learn_prepare())
        for s in STAGES:
            getattr(ctx, s)()
        yield ctx.mesh(False)[0]
        yield ctx.debug("field")

    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        alone = run_batch(pms_lib, ctx, frames, kind)
    got = []
    for batches in (0, 2):
        with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
            ctx.upload(pos, vel)
            ctx.run_frame()
            for k in range(batches):
                meshes = run_batch(pms_lib, ctx, frames, kind)
                for a, b in zip(meshes, alone, strict=True):
                    np.testing.assert_array_equal(a, b)
                if k == 1 and kind != "refused":
                    assert ctx.batch_info()["captures"] == 1
            got.append(list(results(ctx)))
    assert len(got[0][0]) > 0
    for a, b in zip(*got, strict=True):
        np.testing.assert_array_equal(a, b)


def test_batch_frame_batch(pms_lib, tmp_config):
    """A context whose first work is a batch (it is a lane itself then), a frame and batches again."""
    from postmps_gb300 import synth
    pos = synth.lattice(31, 27, 22, 0.005, 0.0008, seed=4)
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "false", "config.issurfacereconstruct": "true"})
    frames = batch_frames("smaller")
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos)
        ctx.run_frame()
        want = [*ctx.mesh(True), ctx.debug("field")]
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        first = run_batch(pms_lib, ctx, frames, "smaller")
        ctx.upload(pos)
        ctx.run_frame()
        for _ in range(2):
            for a, b in zip(run_batch(pms_lib, ctx, frames, "smaller"), first, strict=True):
                np.testing.assert_array_equal(a, b)
            for a, b in zip([*ctx.mesh(True), ctx.debug("field")], want, strict=True):
                np.testing.assert_array_equal(a, b)
