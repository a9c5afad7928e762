"""Several substeps at once (WavePass): frames equal the oracle's bit for bit
at the edges of the sweeps (the fewest points they take, odd substeps left
over, sweeps of two and of four) with moving roots and spheres, and the
batched kernels with and without it give the same frames."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from .util import SIDE_SPHERES, assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def run(ctx, grooms, frames, batched):
    for f in range(frames):
        m = scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)
        for g in grooms:
            g.set_root_transform(m)
        if batched:
            ctx.update_many(grooms, DT)
        else:
            for g in grooms:
                g.update(DT)


@pytest.mark.parametrize("substeps", [1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("n", [7, 8, 9, 16, 17, 32, 33, 63, 64])
def test_sweep_edges(n, substeps):
    from barbu_gb300 import hairsim
    frames = 3
    roots, normals = random_roots_on_sphere(70, n)
    sp = abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5)
    with hairsim.Context() as ctx:
        for contract in (abi.HS_CONTRACT_EXACT, abi.HS_CONTRACT_FAST):
            sim = abi.sim_params_dftl(substeps=substeps, damping=0.9, wind_jitter=0.2, root_mode=abi.HS_ROOT_RIGID,
                                      contract=contract)
            got = []
            for batched in (False, True):
                g = ctx.groom(roots, normals, sp, sim)
                g.set_mapping(abi.HS_MAPPING_THREAD)
                g.set_spheres(SIDE_SPHERES)
                p, v = g.readback(), g.readback_velocities()
                rest = p[:, 0, :3].copy()
                run(ctx, [g], frames, batched)
                got.append((g.readback(), g.readback_velocities()))
                g.destroy()
            if contract == abi.HS_CONTRACT_EXACT:
                for f in range(frames):
                    m = scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)
                    oracle.frame(p, v, sim, DT, seed=5, spheres=SIDE_SPHERES,
                                 root_targets=oracle.rigid_targets(rest, m, np.float32))
                want = (p, v)
            else:
                want = got[0]
            for name, (q, u) in zip(("plain", "batched"), got):
                assert_bit_equal(q, want[0], f"{name} positions")
                assert_bit_equal(u, want[1], f"{name} velocities")


def test_busy_bucket_equals_small_ones():
    """80,000 strands (more tiles than an SM's warps: one substep at a time)
    against the same grooms in buckets of their own (two at a time)."""
    from barbu_gb300 import hairsim
    with hairsim.Context() as ctx:
        sim = abi.sim_params_dftl(substeps=4, damping=0.9, root_mode=abi.HS_ROOT_RIGID)
        sets = []
        for together in (True, False):
            grooms = []
            for k, n in enumerate((9, 16, 24, 12)):
                roots, normals = random_roots_on_sphere(20000 + k, k)
                g = ctx.groom(roots, normals, abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.6, 0.0, k), sim)
                g.set_spheres(SIDE_SPHERES)
                grooms.append(g)
            if together:
                run(ctx, grooms, 3, True)
            else:
                for g in grooms:
                    run(ctx, [g], 3, True)
            sets.append([(g.readback(), g.readback_velocities()) for g in grooms])
            for g in grooms:
                g.destroy()
        for (p, v), (q, u) in zip(*sets):
            assert_bit_equal(p, q, "positions")
            assert_bit_equal(v, u, "velocities")
