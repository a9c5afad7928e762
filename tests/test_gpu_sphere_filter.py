"""The DFTL passes' sphere filter on the GPU: frames equal the oracle's bit
for bit (EXACT) whatever the number of spheres a strand reaches (the edges
of the filter's slots: 2, 4, 8, and more than 8), far from the origin, and
with strands that rest on spheres, a thread per strand, a lane group per
strand and batched; every form gives the same FAST frames."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def cluster(k: int, seed: int, offset: float) -> np.ndarray:
    """k overlapping spheres under the roots, where the strands come to rest."""
    rng = np.random.default_rng(seed)
    s = np.zeros((k, 4), np.float32)
    s[:, :3] = rng.uniform(-0.6, 0.6, (k, 3)) + [offset, offset - 1.0, offset]
    s[:, 3] = rng.uniform(0.1, 0.35, k)
    return s


@pytest.mark.parametrize("offset", [0.0, 50.0, 5000.0])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 8, 9, 32])
@pytest.mark.parametrize("n", [5, 16, 40])
def test_frames_equal_the_oracle(k, n, offset):
    from barbu_gb300 import hairsim
    roots, normals = random_roots_on_sphere(77, 100 * k + n)
    roots = (roots + np.float32(offset)).astype(np.float32)
    spheres = cluster(k, k, offset)
    sp = abi.strand_params(n, abi.HS_LENGTH_TOTAL, 1.2, 0.0, 3)
    frames = 8
    with hairsim.Context() as ctx:
        for contract in (abi.HS_CONTRACT_EXACT, abi.HS_CONTRACT_FAST):
            sim = abi.sim_params_dftl(substeps=4, damping=0.9, contract=contract)
            got = {}
            for form in ("thread", "lanes", "batched", "noalloc"):
                g = ctx.groom(roots, normals, sp, sim)
                g.set_spheres(spheres)
                if form in ("thread", "lanes"):
                    g.set_mapping(abi.HS_MAPPING_THREAD if form == "thread" else abi.HS_MAPPING_LANES)
                p, v = g.readback(), g.readback_velocities()
                for _ in range(frames):
                    if form == "batched":
                        ctx.update_many([g], DT)
                    elif form == "noalloc":
                        ctx.update_many_noalloc([g], DT)
                    else:
                        g.update(DT)
                got[form] = (g.readback(), g.readback_velocities())
                g.destroy()
            if contract == abi.HS_CONTRACT_EXACT:
                for _ in range(frames):
                    oracle.frame(p, v, sim, DT, seed=3, spheres=spheres)
                want = (p, v)
            else:
                want = got["thread"]
            for form, (q, u) in got.items():
                assert_bit_equal(q, want[0], f"{form} positions")
                assert_bit_equal(u, want[1], f"{form} velocities")
