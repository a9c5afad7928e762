"""The plan of a groom set (tiles, directory, launch shape) is kept from frame
to frame: a groom made anew with other strands, on the address of one that was
destroyed, is another set, and every strand of it advances."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi
from .util import SIDE_SPHERES, assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0
N = 12
MORE = [33, 64, 100, 161, 290, 515, 1000, 2049]


def sim():
    return abi.sim_params_dftl(substeps=2, damping=0.9)


@pytest.mark.parametrize("sizes", [MORE, MORE[::-1]], ids=["more strands", "fewer strands"])
def test_groom_made_anew(sizes):
    from barbu_gb300 import hairsim
    seen, again = set(), 0
    with hairsim.Context() as ctx:
        for ns in sizes:
            roots, normals = random_roots_on_sphere(ns, ns)
            g = ctx.groom(roots, normals, abi.strand_params(N, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5), sim())
            again += g.h.value in seen
            seen.add(g.h.value)
            g.set_spheres(SIDE_SPHERES)
            p, v = g.readback(), g.readback_velocities()
            for _ in range(2):
                ctx.update_many([g], DT)
                oracle.frame(p, v, sim(), DT, seed=5, spheres=SIDE_SPHERES)
            assert_bit_equal(g.readback(), p, f"positions of {ns} strands")
            assert_bit_equal(g.readback_velocities(), v, f"velocities of {ns} strands")
            g.destroy()
    assert again, "no address came back: the test has tested nothing"


def test_served_groom_after_another():
    """One groom at a time through a server: no frame comes between them."""
    from barbu_gb300 import hairsim
    with hairsim.Context() as ctx, hairsim.Server(ctx, budget_bytes=1 << 24) as srv:
        for ns in MORE:
            roots, normals = random_roots_on_sphere(ns, ns)
            sp = abi.strand_params(N, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5)
            t = srv.submit(roots, normals, sp, sim(), 2, spheres=SIDE_SPHERES, keep=True)
            for _ in range(8):
                srv.tick(DT)
                if srv.poll(t)[0] == abi.HS_REQ_DONE:
                    break
            q, _ = srv.collect(t)
            p, v = oracle.init(roots, normals, sp, dtype=np.float32)
            for _ in range(2):
                oracle.frame(p, v, sim(), DT, seed=5, spheres=SIDE_SPHERES)
            assert_bit_equal(q, p, f"positions of {ns} strands")
