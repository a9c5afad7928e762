"""Tuned shapes of the batched step: a bucket of less than a wave of tiles and
one of more, of the same power of two, run different kernels and keep shapes of
their own; every form of a pinned shape is checked when it is pinned."""
from __future__ import annotations

import numpy as np
import pytest

from barbu_gb300 import abi
from .util import assert_bit_equal, random_roots_on_sphere

pytestmark = pytest.mark.gpu

DT = 1.0 / 60.0


def test_sides_of_a_wave_are_tuned_apart():
    import torch
    from barbu_gb300 import hairsim
    wave = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    sim = abi.sim_params_dftl(substeps=2, damping=0.9)
    with hairsim.Context() as ctx:
        entries = []
        for tiles in (wave - 1, wave + 1):
            roots, normals = random_roots_on_sphere(32 * tiles, tiles)
            g = ctx.groom(roots, normals, abi.strand_params(9, abi.HS_LENGTH_TOTAL, 0.5, 0.0, 3), sim)
            before = g.readback()
            ctx.autotune([g], DT)
            assert_bit_equal(g.readback(), before, "state after autotune")
            ctx.update_many([g], DT)
            entries.append(ctx.tune_entries())
            g.destroy()
        assert len(entries[0]) == 1 and len(entries[1]) == 2
        assert len({e["tiles_log2"] for e in entries[1]}) == 1


@pytest.mark.parametrize("points", [16, 32, 64])
@pytest.mark.parametrize("warps", [4, 8])
def test_pinned_tensor_memory_shape_runs_in_both_forms(points, warps):
    """A small set without spheres, then with many: the two kernels of the pin."""
    from barbu_gb300 import hairsim
    sim = abi.sim_params_dftl(substeps=4, damping=0.9)
    roots, normals = random_roots_on_sphere(70, points)
    d = np.random.default_rng(points).standard_normal((32, 3))
    around = np.concatenate([d / np.linalg.norm(d, axis=1, keepdims=True) * 1.3, np.full((32, 1), 0.3)], 1)
    with hairsim.Context() as ctx:
        g, alone = (ctx.groom(roots, normals, abi.strand_params(points, abi.HS_LENGTH_TOTAL, 0.9, 0.0, 5), sim)
                    for _ in range(2))
        ctx.tune_override(points, abi.HS_MODE_DFTL, abi.HS_VARIANT_STREAM_TMEM, warps, 1)
        for spheres in (around[:0], around):
            for q in (g, alone):
                q.set_spheres(spheres.astype(np.float32))
            ctx.update_many([g], DT)
            alone.update(DT)
            assert_bit_equal(g.readback(), alone.readback(), "positions")
            assert_bit_equal(g.readback_velocities(), alone.readback_velocities(), "velocities")
