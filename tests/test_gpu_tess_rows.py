"""The tessellation pass's staging rows and copies at their edges: the fewest
and the most subsegments, lines and instances, and line counts that leave
threads of the last block without a line; bit for bit against the oracle."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from barbu_gb300 import abi, scenarios
from tests import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("params", [(1, 1, 1, 1.0), (16, 16, 1, 1.0), (1, 3, 2, 0.7), (5, 1, 15, 1.45), (16, 16, 16, 1.45)])
@pytest.mark.parametrize("n,nfaces", [(2, 1), (3, 43), (64, 5)])
def test_rows_match_the_oracle(n, nfaces, params):
    from barbu_gb300 import hairsim
    rng = np.random.default_rng(n + nfaces)
    ns = 50
    spec = scenarios.plain(ns=ns, npoints=n)
    faces = rng.integers(0, ns, (nfaces, 3)).astype(np.uint32)
    tangents = rng.uniform(-0.1, 0.1, (ns, n, 4)).astype(np.float32)
    rand = rng.random(abi.HS_TESS_RANDOM_SIZE).astype(np.float32)
    with hairsim.Context() as ctx:
        g = ctx.groom(spec.roots, spec.normals, spec.strand, spec.sim)
        g.tess_setup(faces, tangents, rand)
        for _ in range(2):  # the second pass rewrites the same buffer
            count = g.tess_stream(abi.TessParams(*params))
        got, pos = g.tess_readback(), g.readback()
    want = oracle.tess(pos, tangents, faces, rand, *params)
    assert count == want.shape[0]
    util.assert_bit_equal(got, want, "vertices")
