"""Reference mode's iterations that leave no velocities (all but a substep's
last): one, two, three and eight iterations, one and several substeps, in the
register and the streaming forms, plain and batched, bit for bit against the
oracle, among spheres that push the strands."""
from __future__ import annotations

import pytest

import oracle
from barbu_gb300 import abi
from .util import SIDE_SPHERES, assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


@pytest.mark.parametrize("iterations,substeps", [(1, 1), (2, 1), (3, 2), (8, 1), (8, 3)])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 9, 17, 32, 33, 64])
def test_iterations_match_the_oracle(n, iterations, substeps):
    from barbu_gb300 import hairsim
    roots, normals = random_roots_on_sphere(101, n)
    sp = abi.strand_params(n, abi.HS_LENGTH_REFERENCE, 0.5, 0.1, 5)
    sim = abi.sim_params_reference(1.45)
    sim.iterations, sim.substeps = iterations, substeps
    with hairsim.Context() as ctx:
        for batched in (False, True):
            g = ctx.groom(roots, normals, sp, sim)
            g.set_spheres(SIDE_SPHERES)
            p, v = g.readback(), g.readback_velocities()
            for _ in range(3):
                if batched:
                    ctx.update_many([g], DT)
                else:
                    g.update(DT)
                oracle.frame(p, v, sim, DT, seed=5, spheres=SIDE_SPHERES)
            assert_bit_equal(g.readback(), p, f"positions, batched {batched}")
            assert_bit_equal(g.readback_velocities(), v, f"velocities, batched {batched}")
            g.destroy()
