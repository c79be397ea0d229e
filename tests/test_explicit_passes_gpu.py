"""The explicit mode's kernels at the sizes where their split can go wrong:
first hits where a thread's own triangle and the pixels share the work (lists
longer than a chunk, tiles of partial warps, slivers, huge and sub-pixel
triangles) against the oracle, bit for bit; and the one-pass shading against
``interpolate`` + ``composite``, bit for bit forward, and within 1e-5 of the
largest gradient (the order of atomic sums)."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import triangle_rasterization as tr
from oracle import oracle

from .test_rasterization_gpu import _adversarial_triangles

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [(16, 16), (8, 4), (10, 10), (1, 33), (20, 29), (32, 32)])
@pytest.mark.parametrize("kind", ["mixed", "fine", "large"])
def test_first_hits_match_oracle(cuda_device, tile, kind):
    rng = np.random.default_rng(sum(tile))
    h, w, s = 61, 75, 3
    xy, faces = _adversarial_triangles(rng, 2500, h, w)
    if kind != "mixed":
        n = faces.shape[0]
        centre = rng.uniform([0, 0], [w, h], (n, 1, 2))
        xy = (centre + rng.normal(0, 0.8 if kind == "fine" else 15.0, (n, 3, 2))).reshape(-1, 2).astype(np.float32)
    t = -(-h // tile[0]) * -(-w // tile[1])
    # Any list is a valid one: long ones, short ones, an empty one.
    sizes = rng.integers(0, 3 * tile[0] * tile[1] // 2 + 40, (s, t))
    sizes[0, 0] = 0
    ends = np.cumsum(sizes.ravel()).reshape(1, s, t)
    bounds = np.stack((ends - sizes, ends), -1).astype(np.int64)
    tri = rng.integers(0, faces.shape[0], int(sizes.sum())).astype(np.int32)
    d = cuda_device
    grid = tr.TileGrid(tile, (h, w), 1, s)
    got = tr.intersect(torch.from_numpy(xy[None]).to(d), torch.from_numpy(faces).to(d), torch.from_numpy(tri).to(d),
                       torch.from_numpy(bounds).to(d), grid, None)
    uv, index = oracle.intersect(xy[None], faces, tri, bounds, s, tile, (h, w))
    np.testing.assert_array_equal(got.index.cpu().numpy(), index)
    np.testing.assert_array_equal(got.uv.cpu().numpy(), uv)
    assert (index >= 0).any()


@pytest.mark.parametrize("b,s,h,w", [(1, 1, 1, 1), (2, 3, 5, 7), (1, 8, 33, 20), (3, 64, 9, 11)])
@pytest.mark.parametrize("mode", ["reference", "exact"])
@pytest.mark.parametrize("blend", [False, True])
def test_shading_in_one_pass(cuda_device, b, s, h, w, mode, blend):
    rng = np.random.default_rng(s)
    v, f, d = 50, 80, cuda_device

    def t(a, grad=False):
        return torch.from_numpy(np.ascontiguousarray(a)).to(d).requires_grad_(grad)

    index = rng.integers(0, f, (b, s, h, w)).astype(np.int32)
    index[rng.random(index.shape) < 0.4] = -1
    uv = (rng.random((b, s, h, w, 2)) * 0.5).astype(np.float32)
    faces = rng.integers(0, v, (f, 3)).astype(np.int32)
    uv, index, faces = t(uv), t(index), t(faces)
    sdf = t(rng.normal(0, 0.03, v).astype(np.float32), True)
    colors = t(rng.random((b, v, 3)).astype(np.float32), True)
    sharp = torch.tensor(40.0, device=d, requires_grad=True)
    background = t(np.array([0.2, 0.5, 0.9], np.float32))
    g_rgb, g_t = t(rng.normal(size=(b * h * w, 3)).astype(np.float32)), t(rng.normal(size=b * h * w).astype(np.float32))

    i_sdf, i_col = tr.interpolate(uv, index, faces, sdf, colors)
    rgb, trans = tr.Composite.apply(i_sdf.permute(0, 2, 3, 1).reshape(-1, s), i_col.permute(0, 2, 3, 1, 4).reshape(-1, s, 3),
                                    (index != -1).permute(0, 2, 3, 1).reshape(-1, s), sharp, mode)
    if blend:
        want = (rgb + background * trans[:, None],)
        got = (tr.ShadeShells.apply(uv, index, faces, sdf, colors, sharp, background, mode),)
        grads = (g_rgb,)
    else:
        want = (rgb, trans)
        got = tr.ShadeShells.apply(uv, index, faces, sdf, colors, sharp, None, mode)
        grads = (g_rgb, g_t)
    for a, x in zip(got, want):
        assert torch.equal(a, x)
    wants = torch.autograd.grad(want, (sdf, colors, sharp), grads)
    gots = torch.autograd.grad(got, (sdf, colors, sharp), grads)
    for a, x in zip(gots, wants):
        assert float((a - x).abs().max()) <= 1e-5 * max(float(x.abs().max()), 1e-30)
