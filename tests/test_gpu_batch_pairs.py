"""Pairs of substeps in the batched step (bucket_pairs): buckets with and
without them, spheres that come and go between frames, substeps left over,
against the oracle bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def spheres_around(count, seed):
    d = np.random.default_rng(seed).standard_normal((count, 3))
    xyz = d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3
    return np.concatenate([xyz, np.full((count, 1), 0.35)], 1).astype(np.float32)


def check(shapes, substeps, frames=3, contract=abi.HS_CONTRACT_EXACT):
    """shapes: (strands, points, spheres of each frame)."""
    from barbu_gb300 import hairsim
    sim = abi.sim_params_dftl(substeps=substeps, damping=0.9, wind_jitter=0.2, root_mode=abi.HS_ROOT_RIGID,
                              contract=contract)
    with hairsim.Context() as ctx:
        grooms, alone, states = [], [], []
        for k, (ns, n, _) in enumerate(shapes):
            roots, normals = random_roots_on_sphere(ns, 100 * n + k)
            sp = abi.strand_params(n, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5)
            grooms.append(ctx.groom(roots, normals, sp, sim))
            if contract == abi.HS_CONTRACT_EXACT:
                p, v = grooms[-1].readback(), grooms[-1].readback_velocities()
                states.append((p, v, p[:, 0, :3].copy()))
            else:
                alone.append(ctx.groom(roots, normals, sp, sim))
                alone[-1].set_mapping(abi.HS_MAPPING_LANES)
        for f in range(frames):
            m = scenarios.rigid_motion((f + 1) * DT, np.array([0.6, 0.0, 0.8]), 30.0, 0.2, 0.5)
            for k, (ns, n, counts) in enumerate(shapes):
                s = spheres_around(counts[f % len(counts)], 7 * k + f)
                for g in [grooms[k]] + alone[k:k + 1]:
                    g.set_root_transform(m)
                    g.set_spheres(s)
                if states:
                    p, v, rest = states[k]
                    oracle.frame(p, v, sim, DT, seed=5, spheres=s, root_targets=oracle.rigid_targets(rest, m, np.float32))
            ctx.update_many(grooms, DT)
            for g in alone:
                g.update(DT)
        for k, g in enumerate(grooms):
            p, v = states[k][:2] if states else (alone[k].readback(), alone[k].readback_velocities())
            assert_bit_equal(g.readback(), p, f"positions of groom {k}")
            assert_bit_equal(g.readback_velocities(), v, f"velocities of groom {k}")


@pytest.mark.parametrize("substeps", [1, 2, 3, 4, 5, 7, 8])
def test_short_strands_in_a_bucket_with_pairs(substeps):
    """Points from below the fewest a sweep takes (8) to 32, one bucket."""
    check([(40, n, (k,)) for n, k in ((7, 16), (8, 16), (9, 16), (11, 15), (12, 15), (12, 14), (16, 9), (16, 1),
                                      (21, 4), (20, 4), (24, 0), (32, 32))], substeps)


@pytest.mark.parametrize("substeps", [2, 5])
@pytest.mark.parametrize("slowest", [(12, 10), (12, 11), (12, 25), (13, 3), (13, 4), (13, 12), (13, 13)])
def test_lines_of_the_rule(slowest, substeps):
    n, k = slowest
    check([(40, n, (k,)), (33, 10, (1,)), (31, 8, (0,)), (5, 4, (2,))], substeps, frames=2)


@pytest.mark.parametrize("substeps", [2, 3, 4, 5, 8])
def test_spheres_come_and_go(substeps):
    check([(70, 24, (0, 16, 3)), (33, 16, (0, 9, 1)), (64, 12, (0, 8, 32)), (50, 40, (0, 17, 1)), (65, 64, (9, 0, 32))],
          substeps, frames=4)


@pytest.mark.parametrize("substeps", [2, 3, 4])
def test_more_tiles_than_a_wave(substeps):
    """More than 8 tiles an SM of 33 points: pairs by substeps and spheres."""
    check([(20000, 33, (8,)), (20000, 36, (17, 0)), (77, 33, (9,))], substeps, frames=2)


@pytest.mark.parametrize("substeps", [2, 5, 8])
def test_fast_contract(substeps):
    check([(70, 24, (0, 16, 3)), (33, 16, (9, 0, 1)), (64, 21, (4,)), (50, 40, (0, 17, 1))], substeps,
          contract=abi.HS_CONTRACT_FAST)
