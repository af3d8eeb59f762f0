"""Densities inside a surface reconstruction: blocks of cells far from the surface are left out
until all densities are asked for.  The frame's mesh, normals, welded mesh and scalar values, and
the densities handed out afterwards, are bit for bit those of the stages called one by one (which
make every density), over supports of 2, 4 and 5 spacings, scalar grids above and below the limit,
a hollow body (a surface inside) and a frame after a frame.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def scene(kind: str) -> np.ndarray:
    from postmps_gb300 import synth
    if kind == "small":
        return synth.lattice(40, 40, 40, 0.01, 0.001, seed=5)              # below the limit of the rule
    pos = synth.lattice(61, 53, 47, 0.01, 0.001, seed=5, origin=(-0.2, 0.7, 0.1))
    if kind == "hollow":
        centre = pos.mean(axis=0)
        pos = pos[np.linalg.norm(pos - centre, axis=1) > 0.06]
    if kind == "stray":
        pos = np.concatenate([pos, np.array([[2.0, 1.0, 0.3], [-0.9, 0.5, 0.2]], np.float32)])
    return pos


@pytest.mark.parametrize("kind,ratio,sc", [("small", 2, 2), ("block", 2, 1), ("block", 2, 3), ("block", 4, 1),
                                           ("block", 1, 1), ("block", 5, 2), ("hollow", 2, 2), ("stray", 2, 1)])
def test_frame_matches_stages(pms_lib, tmp_config, kind, ratio, sc):
    from postmps_gb300 import synth
    text = synth.config_text(**{"surface.smoothingradiusratio": ratio, "domain.sclargridsizescale": sc})
    pos = scene(kind)

    def results(ctx):
        return [*ctx.mesh(True), *ctx.weld(True), *[v for _, v in sorted(ctx.scalar_values().items())],
                ctx.debug("field"), ctx.debug("density"), ctx.debug("G")]

    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos)
        for stage in ("build_grid", "anisotropy", "band", "field", "marching_cubes"):
            getattr(ctx, stage)()
        want = results(ctx)
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        for _ in range(2):
            ctx.upload(pos)
            ctx.run_frame()
            for a, b in zip(results(ctx), want, strict=True):
                np.testing.assert_array_equal(a, b)
            np.testing.assert_array_equal(ctx.debug("density"), want[-2])


def test_download_after_a_batch(pms_lib, tmp_config):
    """A batch runs its frames in the context's own arrays, also when its graph is only launched again:
    a frame before it leaves nothing that a download could still make.  The frame run after it gives
    its own."""
    from postmps_gb300 import synth
    pos = scene("block")
    frames = [(synth.lattice(30, 20, 25, 0.01, 0.001, seed=k), None, None) for k in range(2)]
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.run_batch(frames)
        ctx.upload(pos)
        ctx.run_frame()
        want = ctx.debug("density")
        ctx.upload(pos)
        ctx.run_frame()
        names = ("density", "band_list", "field", "cube_case", "cube_nvert")
        before = [ctx.debug(k) for k in names]
        ctx.run_batch(frames)
        assert [len(ctx.debug(k)) for k in names] == [len(b) for b in before]
        ctx.upload(pos)
        ctx.run_frame()
        for k, b in zip(names, before):
            np.testing.assert_array_equal(ctx.debug(k), b)
        np.testing.assert_array_equal(ctx.debug("density"), want)
