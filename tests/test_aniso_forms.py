"""Density and moments in each of their forms: a warp per particle, a warp per block of
cells, a thread per particle.  Against the float64 oracle with the anisotropy's tolerances
(density 1e-5 relative, G 1e-4 of its largest entry, neighbour counts exact but for pairs at
the support's edge): float sums of a few hundred terms.
"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,ratio", [
    ((5, 4, 3), 2),          # a block of cells with few particles, warp forms
    ((25, 25, 25), 2),       # just below the density's warp limit
    ((33, 31, 17), 2),       # above it: blocks of cells, partly filled
    ((33, 31, 17), 3),       # a window that ends where the support does: a thread per particle
    ((131, 127, 2), 2),      # more surface particles than take a warp each
    ((17, 16, 15), 4)])
def test_forms_match_oracle(pms_lib, oracle, tmp_config, dims, ratio):
    from postmps_gb300 import synth
    text = synth.config_text(**{"surface.smoothingradiusratio": ratio})
    pos = synth.lattice(*dims, 0.01, 0.001, seed=9)
    with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
        ctx.upload(pos)
        ctx.build_grid()
        ctx.anisotropy()
        density, G, nnb = ctx.debug("density"), ctx.debug("G"), ctx.debug("neighbors")
    p = oracle.derive_params(oracle.config_from_keys(oracle.parse_ini(text)))
    r = oracle.run_surface(p, pos, oracle.grid_from_positions(p, pos))
    assert float((np.abs(density - r.rho) / r.rho).max()) < 1e-5
    scale = np.abs(r.G).max(axis=1, keepdims=True)
    assert float((np.abs(G[:, :9] - r.G) / scale).max()) < 1e-4
    assert np.mean(nnb == r.nnb) > 0.999
