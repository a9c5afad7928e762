"""The arithmetic of the DFTL passes' sphere filter (hs_stream.cuh,
filter_spheres and flagged) restated in numpy float32: whatever point the
exact FP32 test finds inside a sphere, the filter flags, for points at and
about the surface, at many scales and distances from the origin. A filter
without its margin misses some, so the points reach the rounding in
question."""
from __future__ import annotations

import numpy as np

F = np.float32


def fma(a, b, c):
    """a * b + c rounded once (the product is exact in 64 bits)."""
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(F)


def dot(p):
    return fma(p[:, 2], p[:, 2], fma(p[:, 1], p[:, 1], p[:, 0] * p[:, 0]))


def missed(margin: float, seed: int = 1, n: int = 400_000) -> int:
    rng = np.random.default_rng(seed)
    scale = 10.0 ** rng.uniform(-3, 4, n)
    c = (rng.normal(size=(n, 3)) * scale[:, None]).astype(F)
    r = (scale * 10.0 ** rng.uniform(-3, 0.5, n)).astype(F)
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    near = 1.0 - np.abs(rng.normal(size=n)) * 10.0 ** rng.uniform(-8, -3, n)
    p = (c + d * (r * near)[:, None]).astype(F)
    pt = p - c
    r2 = r * r
    inside = dot(pt) < r2
    c2 = c[:, 0] * c[:, 0] + c[:, 1] * c[:, 1] + c[:, 2] * c[:, 2]
    far = (np.linalg.norm(p.astype(np.float64), axis=1)).astype(F)  # the least the kernel's bound can be
    big = far + np.sqrt(c2)
    size = big * big + r2
    k = (c2 - r2) - (F(margin) * size + F(1e-30))
    v = fma(F(-2) * c[:, 0], p[:, 0], fma(F(-2) * c[:, 1], p[:, 1], fma(F(-2) * c[:, 2], p[:, 2], k)))
    flagged = v <= -dot(p)
    assert inside.sum() > n // 4
    return int((inside & ~flagged).sum())


def test_filter_flags_every_point_inside():
    for seed in range(4):
        assert missed(1.25e-6, seed) == 0


def test_margin_is_needed():
    assert missed(0.0) > 0
