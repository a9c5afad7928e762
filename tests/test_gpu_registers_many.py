"""Strands in registers (up to 8 points) on both sides of the line between few
and many spheres, one groom and batched, against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("iterations", [1, 2])
@pytest.mark.parametrize("spheres", [8, 9, 32])
@pytest.mark.parametrize("points", [2, 4, 5, 8])
def test_line(points, spheres, iterations):
    from barbu_gb300 import hairsim
    roots, normals = random_roots_on_sphere(70, points)
    d = np.random.default_rng(spheres).standard_normal((spheres, 3))
    around = np.concatenate([d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3, np.full((spheres, 1), 0.4)], 1)
    around = around.astype(np.float32)
    sp = abi.strand_params(points, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5)
    sim = abi.sim_params_dftl(substeps=3, damping=0.9, root_mode=abi.HS_ROOT_RIGID, iterations=iterations)
    with hairsim.Context() as ctx:
        sets = []
        for variant in (None, abi.HS_VARIANT_REGISTERS, abi.HS_VARIANT_REGISTERS_SHARED):
            g = ctx.groom(roots, normals, sp, sim)
            g.set_mapping(abi.HS_MAPPING_THREAD)
            g.set_spheres(around)
            sets.append((variant, g))
        p, v = g.readback(), g.readback_velocities()
        rest = p[:, 0, :3].copy()
        for f in range(3):
            m = scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)
            oracle.frame(p, v, sim, DT, seed=5, spheres=around, root_targets=oracle.rigid_targets(rest, m, np.float32))
            for variant, g in sets:
                g.set_root_transform(m)
                if variant is None:
                    g.update(DT)
                else:
                    ctx.tune_override(points, abi.HS_MODE_DFTL, variant, 2, 1)
                    ctx.update_many([g], DT)
        for variant, g in sets:
            assert_bit_equal(g.readback(), p, f"positions, variant {variant}")
            assert_bit_equal(g.readback_velocities(), v, f"velocities, variant {variant}")
