"""The training pass over batches that fill its blocks of 128 samples, end in one, or are smaller
than one: the gradient against the float64 oracle with the tolerances of the BF16 backward (dh, h
and dz rounded to 8 bits of mantissa: 5e-3 in norm, loss 1e-4), and a training step, whose
samples the kernel gathers from a frame by itself, against the frame's candidates.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_learned_band import LO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 31, 127, 128, 129, 640, 4097])
def test_gradient(pms_lib, batch):
    rng = np.random.default_rng(batch)
    x = LO.bf16_round(rng.uniform(0, 2, (batch, 64)).astype(np.float32))
    y = (rng.uniform(size=batch) < 0.3).astype(np.uint8)
    p = rng.normal(0, 0.15, LO.N_PARAMS).astype(np.float32)
    t = pms_lib.Trainer(0, 5)
    t.set_params(p)
    g, loss = t.grad(LO.bf16_bits(x).reshape(batch, 64), y, 4.0)
    t.close()
    lo, go = LO.loss_and_grad(p.astype(np.float64), x, y.astype(np.float64), 4.0)
    assert abs(loss - lo) <= 1e-4 * max(1.0, abs(lo))
    assert np.linalg.norm(g - go) / np.linalg.norm(go) < 5e-3


def test_step_gathers_its_samples(pms_lib, tmp_config):
    """A step over one sample has that candidate's loss: every seed's is the oracle's for one of the
    frame's candidates (their features and labels as handed out), spread by random weights."""
    from postmps_gb300 import synth
    p = np.random.default_rng(1).normal(0, 0.3, LO.N_PARAMS).astype(np.float32)
    t = pms_lib.Trainer(0, 5)
    t.set_params(p)
    with pms_lib.Context(pms_lib.load_config(tmp_config(synth.config_text())), 0) as ctx:
        ctx.upload(synth.lattice(9, 8, 7, 0.01, 0.002, seed=2))
        ctx.run_frame()
        ctx.learn_prepare()
        losses = np.array([t.step(ctx, 1, seed, 0.0, 4.0) for seed in range(12)])
        cand = ctx.learn_candidates(logits=False)
        x = LO.bf16_value(ctx.learn_features(cand["cube"]))
    t.close()
    each = np.array([LO.loss_and_grad(p.astype(np.float64), x[i:i + 1], cand["label"][i:i + 1].astype(np.float64), 4.0)[0]
                     for i in range(len(x))])
    assert np.ptp(losses) > 0.01
    for v in losses:
        assert np.abs(each - v).min() <= 1e-4 * max(1.0, v)
