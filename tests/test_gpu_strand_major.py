"""Strand-major exports and readbacks against the device buffer's own layout:
point counts on both sides of the tiles' remainders, strand counts that leave
lanes without a strand, four floats and three a point."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from barbu_gb300 import abi
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [1, 31, 32, 33, 97, 1000])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 8, 12, 23, 24, 31, 32, 33, 48, 63, 64])
def test_strand_major_equals_the_device_buffer(n, ns):
    from barbu_gb300 import hairsim
    rng = np.random.default_rng(64 * ns + n)
    pos = rng.uniform(-1, 1, (ns, n, 4)).astype(np.float32)
    vel = rng.uniform(-1, 1, (ns, n, 4)).astype(np.float32)
    with hairsim.Context() as ctx:
        g = ctx.groom_from_state(pos, vel, abi.sim_params_dftl())
        want, wvel = g.readback(), g.readback_velocities()
        assert_bit_equal(want[..., :3], pos[..., :3], "readback")
        assert_bit_equal(g.readback_xyz(), pos[..., :3], "readback_xyz")
        out = torch.full((ns * n * 4 + 64,), -7.0, device="cuda")
        for field, ref in ((abi.HS_FIELD_POSITIONS, want), (abi.HS_FIELD_VELOCITIES, wvel)):
            g.export(out.data_ptr(), ns * n * 4, abi.HS_EXPORT_STRAND_MAJOR, field)
            ctx.sync()
            got = out.cpu().numpy()
            assert_bit_equal(got[:ns * n * 4].reshape(ns, n, 4), ref, "export")
            assert (got[ns * n * 4:] == -7.0).all()
            g.export(out.data_ptr(), ns * n * 4, abi.HS_EXPORT_POINT_MAJOR, field)
            ctx.sync()
            got = out.cpu().numpy()[:ns * n * 4].reshape(n, ns, 4)
            assert_bit_equal(got.transpose(1, 0, 2), ref, "point-major export")
        g.destroy()
