"""The AUTO mapping of a groom's step: lane groups below its line and a thread
per strand above it, which the substeps, the points and the spheres move; the
frames are the same bit for bit as under either mapping."""
from __future__ import annotations

import numpy as np
import pytest

from barbu_gb300 import abi, scenarios
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("n,substeps,spheres,few,many", [
    (16, 4, 0, 5000, 15000), (16, 4, 1, 12000, 20000), (16, 4, 7, 20000, 26000), (16, 4, 16, 24000, 32000),
    (64, 2, 7, 12000, 16000), (8, 8, 0, 7000, 12000), (64, 16, 32, 9000, 30000), (3, 2, 2, 8000, 40000)])
def test_line(n, substeps, spheres, few, many):
    from barbu_gb300 import hairsim
    rng = np.random.default_rng(n + spheres)
    d = rng.standard_normal((spheres, 3))
    around = np.concatenate([d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3, np.full((spheres, 1), 0.35)], 1)
    sim = abi.sim_params_dftl(substeps=substeps, damping=0.9, root_mode=abi.HS_ROOT_RIGID)
    for ns, mapping in ((few, abi.HS_MAPPING_LANES), (many, abi.HS_MAPPING_THREAD)):
        roots, normals = random_roots_on_sphere(ns, n)
        with hairsim.Context() as ctx:
            got = []
            for m in (abi.HS_MAPPING_AUTO, abi.HS_MAPPING_THREAD, abi.HS_MAPPING_LANES):
                g = ctx.groom(roots, normals, abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5), sim)
                g.set_spheres(around.astype(np.float32))
                g.set_mapping(m)
                if m == abi.HS_MAPPING_AUTO:
                    assert g.mapping() == mapping
                for f in range(2):
                    g.set_root_transform(scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5))
                    g.update(DT)
                got.append((g.readback(), g.readback_velocities()))
                g.destroy()
        for p, v in got[1:]:
            assert_bit_equal(p, got[0][0], "positions")
            assert_bit_equal(v, got[0][1], "velocities")
