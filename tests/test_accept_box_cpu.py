"""The accept box of a triangle of any conditioning (bary.cuh: cull_box, its
margin scaled by the triangle's squared double area over its longest edges'
product), emulated in single precision: every pixel centre that escapes the
fast reject lies inside it."""

import numpy as np

from .test_exactness_cpu import _cull_box, _dot2, _numerators, _setup, _triangles, _with_small_threshold, f32


def _scaled_box(g, p):
    """cull_box's tighter box; None when it is open."""
    if _cull_box(g, p) is None and g["dd"] > f32(2.0 ** -20):
        return None
    ext = max(f32(p[:, 0].max() - p[:, 0].min()), f32(p[:, 1].max() - p[:, 1].min()))
    e23 = (p[2] - p[1]).astype(f32)
    l = g["d1212"], g["d1313"], _dot2(*e23, *e23)
    worst = max(f32(l[0] * l[1]), f32(l[0] * l[2]), f32(l[1] * l[2]))
    small = g["dd"] <= f32(2.0 ** -20)
    area = f32(g["dd"] - f32(1e-8)) if small else g["dd"]
    if min(l) < f32(2.0 ** -50) or not area >= f32(f32(1e-4) * worst) or (small and not area >= f32(1e-13)):
        return None
    # A quotient two ulps low (the kernel's is approximate) gives the smaller box.
    c = f32(f32(2.5e-5) * worst) / area * f32(1 - 2.0 ** -22)
    m = min(f32(f32(1.0) + f32(f32(1e-3) * ext)), f32(f32(0.0625) + f32(c * ext)))
    return (f32(p[:, 0].min() - m), f32(p[:, 0].max() + m), f32(p[:, 1].min() - m), f32(p[:, 1].max() + m)), float(c)


def test_scaled_accept_box_holds_every_pixel_that_escapes_the_fast_reject():
    rng = np.random.default_rng(5)
    shapes = list(_triangles(rng, 600))
    for _ in range(6000):
        c, size = rng.uniform(0, rng.choice([50, 4000]), 2), 10 ** rng.uniform(-2, 1.3)
        d = rng.normal(0, 1, 2)
        d /= np.linalg.norm(d)
        n = np.array([-d[1], d[0]])
        thin = 10 ** rng.uniform(-2.3, 0.2)
        if rng.random() < 0.5:  # along a row or a column, a corner near a pixel centre
            d, n = np.eye(2)[rng.permutation(2)]
            c = np.floor(c) + 0.5 + rng.normal(0, 0.06, 2)
        shapes.append((c + size * np.array([0 * d, d, rng.uniform(-0.3, 1.3) * d + thin * n])).astype(f32))
    boxed = tight = near = 0
    for p in shapes:
        g = _with_small_threshold(_setup(p[0], p[1], p[2]))
        found = _scaled_box(g, p)
        if found is None:
            continue
        box, c = found
        boxed += 1
        tight += c < 0.01
        lo, hi = np.floor(p.min(0)).astype(int) - 3, np.floor(p.max(0)).astype(int) + 4
        if (hi - lo).max() > 80:
            continue
        px, py = (a.ravel().astype(f32) + f32(0.5) for a in np.meshgrid(np.arange(lo[0], hi[0]), np.arange(lo[1], hi[1])))
        un, vn, wn = _numerators(g, px, py)
        escapes = ~((un < g["thr"]) | (vn < g["thr"]) | (wn < g["thr"]))
        inside = (px >= box[0]) & (px <= box[1]) & (py >= box[2]) & (py <= box[3])
        assert not (escapes & ~inside).any(), p
        near += int((inside & ~escapes).any())
    assert boxed > 4000 and tight > 1500 and near > 1500
