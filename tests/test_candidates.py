"""The learned band's candidates and network where their tiles end: grids smaller than a tile's 16
coarse cells along x or 8 along z, and sides of either parity.  Candidates and features exact, logits
1e-4 (float sums of 64 products in another order), against the oracle.  And a batch's captured graph
follows the context's model: the model's last layer is part of the launches.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_learned_band import LO

pytestmark = pytest.mark.gpu


def random_model(pms, threshold: float):
    p = np.random.default_rng(11).normal(0, 0.2, LO.N_PARAMS).astype(np.float32)
    t = pms.Trainer(0, 1)
    t.set_params(p)
    m = t.model(threshold)
    t.close()
    return p, m


@pytest.mark.parametrize("dims,ratio,sc", [((1, 1, 1), 1, 1), ((2, 3, 1), 2, 1), ((9, 4, 5), 1, 2), ((24, 3, 2), 2, 1),
                                           ((25, 2, 14), 1, 1), ((3, 17, 15), 2, 2), ((30, 12, 9), 2, 3)])
def test_candidates_and_logits(pms_lib, tmp_config, dims, ratio, sc):
    from postmps_gb300 import synth
    text = synth.config_text(**{"surface.smoothingradiusratio": ratio, "domain.sclargridsizescale": sc})
    cfg = pms_lib.load_config(tmp_config(text))
    p, model = random_model(pms_lib, 0.0)
    with pms_lib.Context(cfg, 0) as ctx:
        ctx.upload(synth.lattice(*dims, 0.01, 0.002, seed=3))
        ctx.build_grid()
        ctx.surface()
        ctx.learn_prepare()
        ctx.set_band_model(model)
        got = ctx.learn_candidates(logits=True)
        g = ctx.grid()
        counts = LO.coarse_counts(ctx.debug("pos_sorted"), list(g.scmin_pos), g.sc_grid_size, list(g.scres))
        inv = LO.inv_expected(g.sc_grid_size, pms_lib.derive_params(cfg).particle_spacing)
        cand = LO.candidates(counts, list(g.scres), inv)
        np.testing.assert_array_equal(got["cube"], cand)
        x = LO.features(counts, list(g.scres), inv, cand)
        np.testing.assert_array_equal(ctx.learn_features(cand), LO.bf16_bits(x))
    z = LO.forward(p.astype(np.float64), x)[0]
    assert np.allclose(got["logit"], z, rtol=1e-4, atol=1e-4 * np.abs(z).max())


def test_batch_follows_the_model(pms_lib, tmp_config):
    from postmps_gb300 import synth
    pos = synth.lattice(14, 13, 12, 0.01, 0.002, seed=3)
    frames = [(pos, np.zeros_like(pos), None)] * 2
    _, most = random_model(pms_lib, -1e30)
    _, none = random_model(pms_lib, 1e30)
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        predicted = []
        for m in (most, most, none, most):
            ctx.set_band_model(m)
            ctx.run_batch(frames, learned=True)
            predicted.append([ctx.batch_frame(f)[0].n_band_predicted for f in range(2)])
    assert predicted[0][0] > 0 and predicted[0][0] == predicted[0][1]
    assert predicted == [predicted[0], predicted[0], [0, 0], predicted[0]]
