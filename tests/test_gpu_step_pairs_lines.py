"""The lines of step_pairs (points, spheres, substeps, contract, strands):
frames of one groom equal the oracle's bit for bit, FAST ones the lane groups'."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def spheres_around(count):
    d = np.random.default_rng(count).standard_normal((count, 3))
    xyz = d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3
    return np.concatenate([xyz, np.full((count, 1), 0.35)], 1).astype(np.float32)


def motion(f):
    return scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)


@pytest.mark.parametrize("substeps", [2, 3, 8])
@pytest.mark.parametrize("n,spheres", [(19, 5), (20, 3), (20, 4), (20, 5), (20, 6), (20, 10), (20, 11), (20, 16), (20, 17),
                                       (11, 25), (12, 25), (16, 25), (15, 24), (16, 20), (16, 21), (33, 2), (33, 8),
                                       (33, 9), (33, 12), (33, 13), (33, 24), (33, 25), (48, 0), (49, 0), (48, 13), (49, 13)])
def test_points_and_spheres(n, spheres, substeps):
    from barbu_gb300 import hairsim
    roots, normals = random_roots_on_sphere(77, n)
    sp = abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5)
    around = spheres_around(spheres)
    with hairsim.Context() as ctx:
        for contract in (abi.HS_CONTRACT_EXACT, abi.HS_CONTRACT_FAST):
            sim = abi.sim_params_dftl(substeps=substeps, damping=0.9, root_mode=abi.HS_ROOT_RIGID, contract=contract)
            g, lanes = (ctx.groom(roots, normals, sp, sim) for _ in range(2))
            p, v = g.readback(), g.readback_velocities()
            rest = p[:, 0, :3].copy()
            for q, mapping in ((g, abi.HS_MAPPING_THREAD), (lanes, abi.HS_MAPPING_LANES)):
                q.set_mapping(mapping)
                q.set_spheres(around)
            for f in range(2):
                for q in (g, lanes):
                    q.set_root_transform(motion(f))
                    q.update(DT)
                if contract == abi.HS_CONTRACT_EXACT:
                    oracle.frame(p, v, sim, DT, seed=5, spheres=around,
                                 root_targets=oracle.rigid_targets(rest, motion(f), np.float32))
            if contract == abi.HS_CONTRACT_FAST:
                p, v = lanes.readback(), lanes.readback_velocities()
            assert_bit_equal(g.readback(), p, "positions")
            assert_bit_equal(g.readback_velocities(), v, "velocities")


@pytest.mark.parametrize("n,spheres,per_sm", [(20, 17, 8), (20, 5, 12), (12, 32, 16), (49, 4, 8)])
def test_strands(n, spheres, per_sm):
    """A tile on either side of half a wave, of three quarters and of a wave."""
    import torch
    from barbu_gb300 import hairsim
    tiles = per_sm * torch.cuda.get_device_properties(0).multi_processor_count
    sim = abi.sim_params_dftl(substeps=4, damping=0.9, root_mode=abi.HS_ROOT_RIGID)
    for ns in (32 * tiles, 32 * tiles + 1):
        roots, normals = random_roots_on_sphere(ns, n)
        got = []
        for mapping in (abi.HS_MAPPING_THREAD, abi.HS_MAPPING_LANES):
            with hairsim.Context() as ctx:
                g = ctx.groom(roots, normals, abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5), sim)
                g.set_mapping(mapping)
                g.set_spheres(spheres_around(spheres))
                for f in range(2):
                    g.set_root_transform(motion(f))
                    g.update(DT)
                got.append((g.readback(), g.readback_velocities()))
        assert_bit_equal(got[0][0], got[1][0], "positions")
        assert_bit_equal(got[0][1], got[1][1], "velocities")
