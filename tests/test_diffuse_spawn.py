"""Spawning where the count around a parent decides its children's type: lattices of several
spacings put 0 to more than 20 particles within the diffuse radius, and large multipliers give a
parent more children than a warp has lanes.  Everything the spawning writes is exact against the
oracle but the velocities (1e-5), as in the diffuse frames' own tests.
"""
from __future__ import annotations

import numpy as np
import pytest

from test_diffuse import check_gpu_frames, run_gpu_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread,multiplier", [(0.55, 40), (0.8, 4000), (1.0, 800), (1.3, 30000), (1.9, 800)])
def test_spawned_types(pms_lib, oracle, tmp_config, spread, multiplier):
    from postmps_gb300 import synth
    pos = synth.lattice(12, 9, 7, 0.005 * spread, 0.0008, seed=3)
    vel = np.random.default_rng(4).normal(0, 1.5, pos.shape).astype(np.float32)
    rho = np.full(len(pos), 1000, np.float32)
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "true",
                                                    "diffuse.diffusetrappedairmultiplier": multiplier})
    d = {"config": text, "seed": 11, "f0_pos": pos, "f0_vel": vel, "f0_rho": rho}
    gpu = run_gpu_frames(pms_lib, tmp_config, d, frames=(0,))
    if multiplier >= 4000:
        assert gpu[0]["num"].max() > 32
    check_gpu_frames(oracle, d, gpu, reference=False)


@pytest.mark.parametrize("n", [1, 2, 31, 33, 255, 257, 1000])
@pytest.mark.parametrize("moving", [0.0, 0.4, 1.0])
def test_listed_particles(pms_lib, oracle, tmp_config, n, moving):
    """Frames in which none, some and all of the particles move fast enough to spawn: the walks'
    lists end at every place in a warp, and are empty."""
    from postmps_gb300 import synth
    rng = np.random.default_rng(n)
    pos = synth.lattice(10, 10, 10, 0.005, 0.0005, seed=8)[rng.permutation(1000)[:n]]
    vel = rng.normal(0, 2.0, pos.shape).astype(np.float32)
    vel[rng.random(n) >= moving] = 0.0
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "true"})
    d = {"config": text, "seed": 5}
    for f in (0, 1):
        d.update({f"f{f}_pos": pos, f"f{f}_vel": vel, f"f{f}_rho": np.full(n, 1000, np.float32)})
    check_gpu_frames(oracle, d, run_gpu_frames(pms_lib, tmp_config, d), reference=False)


@pytest.mark.parametrize("moving", [0.0, 0.02, 1.0])
@pytest.mark.parametrize("surface", ["true", "false"])
def test_normals_do_not_depend_on_who_moves(pms_lib, tmp_config, moving, surface):
    """Normals are made only where a particle that can spawn may read them; a download makes the rest,
    bit for bit those of a frame in which every particle moves."""
    from postmps_gb300 import synth
    pos = synth.lattice(31, 27, 14, 0.005, 0.0008, seed=9)
    rho = np.full(len(pos), 1000, np.float32)
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "true", "config.issurfacereconstruct": surface})
    normals = []
    for share in (1.0, moving):
        rng = np.random.default_rng(3)
        vel = rng.normal(0, 3.0, pos.shape).astype(np.float32)
        vel[rng.random(len(pos)) >= share] = 0.0
        with pms_lib.Context(pms_lib.load_config(tmp_config(text)), 0) as ctx:
            ctx.upload(pos, vel, rho)
            ctx.run_frame()
            normals.append((ctx.debug("free_normal"), ctx.debug("free_normal")))
    assert np.any(normals[0][0] != 0)
    for n in normals[1]:
        np.testing.assert_array_equal(n, normals[0][0])


@pytest.mark.parametrize("moving", [0.3, 0.15, 0.08, 0.04, 0.02, 0.01])
def test_short_lists(pms_lib, oracle, tmp_config, moving):
    """Few particles that can spawn, in crowded cells: the walks' lists are spread over 2 to 32 lanes each."""
    from postmps_gb300 import synth
    pos = synth.lattice(13, 13, 13, 0.003, 0.0003, seed=8)
    rng = np.random.default_rng(5)
    vel = rng.normal(0, 3.0, pos.shape).astype(np.float32)
    vel[rng.random(len(pos)) >= moving] = 0.0
    text = synth.config_text(**synth.CROWN_KEYS, **{"config.isdiffusegeneration": "true"})
    d = {"config": text, "seed": 5, "f0_pos": pos, "f0_vel": vel, "f0_rho": np.full(len(pos), 1000, np.float32)}
    check_gpu_frames(oracle, d, run_gpu_frames(pms_lib, tmp_config, d, frames=(0,)), reference=False)
