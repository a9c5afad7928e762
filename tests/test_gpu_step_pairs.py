"""Pairs of substeps in the step of one groom (step_pairs): frames equal the
oracle's bit for bit on both sides of each line of the rule (points, spheres,
substeps), with a last tile that is not full."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("substeps", [1, 2, 3, 8])
@pytest.mark.parametrize("n,spheres", [(21, 1), (20, 2), (21, 2), (32, 9), (20, 16), (9, 17), (16, 17), (32, 32), (33, 0),
                                       (48, 0), (49, 0), (64, 0), (33, 1), (64, 32)])
def test_rule_edges(n, spheres, substeps):
    from barbu_gb300 import hairsim
    frames = 2
    roots, normals = random_roots_on_sphere(77, n)
    rng = np.random.default_rng(n * 100 + spheres)
    d = rng.standard_normal((spheres, 3))
    around = np.concatenate([d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3, np.full((spheres, 1), 0.35)], 1)
    around = around.astype(np.float32)
    sp = abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5)
    sim = abi.sim_params_dftl(substeps=substeps, damping=0.9, root_mode=abi.HS_ROOT_RIGID)
    with hairsim.Context() as ctx:
        g = ctx.groom(roots, normals, sp, sim)
        g.set_mapping(abi.HS_MAPPING_THREAD)
        g.set_spheres(around)
        p, v = g.readback(), g.readback_velocities()
        rest = p[:, 0, :3].copy()
        for f in range(frames):
            m = scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)
            g.set_root_transform(m)
            g.update(DT)
            oracle.frame(p, v, sim, DT, seed=5, spheres=around, root_targets=oracle.rigid_targets(rest, m, np.float32))
        assert_bit_equal(g.readback(), p, "positions")
        assert_bit_equal(g.readback_velocities(), v, "velocities")


@pytest.mark.parametrize("n", [48, 49])
@pytest.mark.parametrize("spheres", [8, 9])
def test_more_than_a_wave(n, spheres):
    """More strands than the SMs hold at once, against the lane groups."""
    from barbu_gb300 import hairsim
    roots, normals = random_roots_on_sphere(39000, n)
    rng = np.random.default_rng(spheres)
    d = rng.standard_normal((spheres, 3))
    around = np.concatenate([d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3, np.full((spheres, 1), 0.35)], 1)
    sim = abi.sim_params_dftl(substeps=7, damping=0.9, root_mode=abi.HS_ROOT_RIGID)
    got = []
    for mapping in (abi.HS_MAPPING_THREAD, abi.HS_MAPPING_LANES):
        with hairsim.Context() as ctx:
            g = ctx.groom(roots, normals, abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5), sim)
            g.set_mapping(mapping)
            g.set_spheres(around.astype(np.float32))
            for f in range(2):
                g.set_root_transform(scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5))
                g.update(DT)
            got.append((g.readback(), g.readback_velocities()))
    assert_bit_equal(got[0][0], got[1][0], "positions")
    assert_bit_equal(got[0][1], got[1][1], "velocities")
