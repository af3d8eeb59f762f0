"""The field's own choice of vertices per lane: bands below and above each line of the rule, dense
bodies and droplets.  The dense field is bit for bit that of every fixed choice.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def droplets(n: int) -> np.ndarray:
    rng = np.random.default_rng(6)
    centre = rng.uniform(0, 1.5, (n // 200, 3))
    p = np.repeat(centre, 200, axis=0) + rng.normal(0, 0.02, (n // 200 * 200, 3))
    return p.astype(np.float32)


# expected: the number of band vertices against the rule's lines
@pytest.mark.parametrize("kind,ratio,sc,low,high", [
    ("block", 2, 2, 1, 160000), ("block", 2, 2, 160000, 500000), ("block", 2, 3, 1, 500000), ("block", 2, 3, 500000, 1 << 29),
    ("block", 4, 2, 160000, 1000000), ("block", 4, 2, 1000000, 1 << 29), ("droplets", 3, 2, 1000000, 1 << 29),
    ("droplets", 2, 1, 1, 1000000)])
def test_choice_keeps_the_field(pms_lib, tmp_config, kind, ratio, sc, low, high):
    from postmps_gb300 import synth
    sides = {160000: 12, 500000: 30 if sc == 2 else 22, 1000000: 40}
    side = sides.get(high, 70 if ratio == 4 else 40)
    pos = synth.lattice(side, side, side, 0.01, 0.001, seed=2) if kind == "block" else droplets(24000 if sc == 2 else 6000)
    text = synth.config_text(**{"surface.smoothingradiusratio": ratio, "domain.sclargridsizescale": sc})
    fields = []
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        for vpt in (0, 1, 2, 4):
            if vpt:
                ctx.set_tune({"field_threads": 128, "field_waves": 8, "density_threads": 128, "moments_threads": 128,
                              "field_vpt": vpt})
            ctx.upload(pos)
            ctx.run_frame()
            fields.append(ctx.debug("field"))
        n = ctx.counts().n_band_vertices
    assert low <= n < high, n
    for f in fields[1:]:
        np.testing.assert_array_equal(fields[0], f)


def test_saved_shape_restores_the_choice(pms_lib, tmp_config):
    """What get_tune reports before a tuning brings the frame's own choice back, and keeps it."""
    from postmps_gb300 import synth
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        saved = ctx.get_tune()
        ctx.upload(synth.lattice(12, 12, 12, 0.01, 0.001, seed=2))
        ctx.run_frame()
        field = ctx.debug("field")
        assert ctx.autotune()["field_vpt"] in (1, 2, 4)
        ctx.set_tune(saved)
        assert ctx.get_tune()["field_vpt"] == saved["field_vpt"] == 0
        ctx.run_frame()
        np.testing.assert_array_equal(ctx.debug("field"), field)
        with pytest.raises(pms_lib.PmsError):
            ctx.set_tune({**saved, "field_vpt": 3})
