"""Batched lane groups on both sides of the line between few and many spheres,
in one bucket, for every group size, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("points", [9, 16, 64])
@pytest.mark.parametrize("warps,substeps", [(2, 2), (4, 3), (8, 8), (16, 12)])
def test_few_and_many_in_one_bucket(warps, substeps, points):
    from barbu_gb300 import hairsim
    sim = abi.sim_params_dftl(substeps=substeps, damping=0.9, root_mode=abi.HS_ROOT_RIGID)
    counts = (8, 9, 32, 0)
    with hairsim.Context() as ctx:
        ctx.tune_override(points, abi.HS_MODE_DFTL, abi.HS_VARIANT_LANES, warps, 1)
        grooms, states = [], []
        for k, count in enumerate(counts):
            roots, normals = random_roots_on_sphere(40 + 11 * k, points + k)
            g = ctx.groom(roots, normals, abi.strand_params(points, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5), sim)
            d = np.random.default_rng(count).standard_normal((count, 3))
            s = np.concatenate([d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3, np.full((count, 1), 0.35)], 1)
            p, v = g.readback(), g.readback_velocities()
            grooms.append(g)
            states.append((p, v, p[:, 0, :3].copy(), s.astype(np.float32)))
            g.set_spheres(states[-1][3])
        for f in range(2):
            m = scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)
            for g, (p, v, rest, s) in zip(grooms, states):
                g.set_root_transform(m)
                oracle.frame(p, v, sim, DT, seed=5, spheres=s, root_targets=oracle.rigid_targets(rest, m, np.float32))
            ctx.update_many(grooms, DT)
        for g, (p, v, _, _), count in zip(grooms, states, counts):
            assert_bit_equal(g.readback(), p, f"positions among {count} spheres")
            assert_bit_equal(g.readback_velocities(), v, f"velocities among {count} spheres")
