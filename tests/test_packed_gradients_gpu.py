"""The compositing adjoint's packed gradients (colour and signed distance of a
(camera, vertex) in 16 bytes) equal the separate ones, through every entry
point's path: unpacked for callers of the stage, read in place by the SH
adjoints. Within 1e-5 of the largest gradient: the order of atomic sums."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import _native as nt
from meshtryoshka_gb300 import triangle_rasterization as tr
from tests.scenes import make_scene

pytestmark = pytest.mark.gpu


def _close(got, want):
    assert float((got - want).abs().max()) <= 1e-5 * max(float(want.abs().max()), 1e-30)


@pytest.mark.parametrize("b,v", [(1, 1), (1, 2), (3, 257), (5, 1000)])
def test_unpacking_and_rows_in_place(cuda_device, b, v):
    rows = torch.randn((b, v, 4), device=cuda_device)
    packed = tr._PackedGradients(b, v, cuda_device)
    packed.rows.copy_(rows)
    colors, sdf = packed.split(False)
    assert torch.equal(colors, rows[..., :3]) and colors.is_contiguous()
    _close(sdf, rows[..., 3].sum(0))
    view, _ = packed.split(True)
    found, in_place = nt.colour_gradient_rows(view)
    assert in_place == (v > 1) and torch.equal(found, rows[..., :3])
    # Other strides of the same shape are copied.
    for other in (rows[..., 1:], torch.randn((v, b, 4), device=cuda_device).transpose(0, 1)[..., :3],
                  torch.randn((b, 2 * v, 4), device=cuda_device)[:, ::2, :3]):
        found, in_place = nt.colour_gradient_rows(other)
        assert torch.equal(found, other) and (not in_place or other.stride()[1:] == (4, 1))


@pytest.mark.parametrize("mode", ["reference", "exact"])
@pytest.mark.parametrize("tile", [(16, 16, 128), (8, 8, 256), (12, 20, 512)])
def test_stage_and_render_gradients(cuda_device, mode, tile):
    sc = make_scene(sh_degree=2, levels=(0.03, 0.0, -0.03))
    d = cuda_device

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(d)

    vertices, faces, sfb = t(sc.vertices), t(sc.faces), t(sc.face_boundaries)
    ext, intr = t(sc.extrinsics), t(sc.intrinsics)
    sdf, sh = t(sc.sdf).requires_grad_(True), t(sc.sh).requires_grad_(True)
    b, s = ext.shape[0], sfb.shape[0]
    grid = tr.TileGrid(tile, tuple(sc.image_shape), b, s)
    kd = tr.create_key_defines(("camera", 6), ("tile", 20), ("depth", 32), ("shell", 6))
    xy, depths = tr.project_vertices(vertices, ext, intr)
    bounds = tr.bound_triangles(xy, depths, faces, grid, 0.2)
    keys = tr.sort_keys(tr.generate_keys(depths, faces, sfb, bounds.tile_minima, bounds.tile_maxima,
                                         bounds.num_tiles_overlapped, grid, kd))
    ranges = tr.delineate_tiles(keys, grid, kd, False).view(b, -1, 2)
    colors = tr.evaluate_spherical_harmonics(vertices, sh, ext, sc.sh_degree).detach().requires_grad_(True)
    raw = tr.intersect_and_composite(xy, colors, sdf, faces, float(sc.sharpness), keys.keys, keys.triangle_indices,
                                     ranges, s, grid, kd, mode)
    g = torch.randn(raw.shape, device=d)
    got_colors, got_sdf = torch.autograd.grad(raw, (colors, sdf), g)
    assert got_colors.is_contiguous()
    # The separate gradients of the same kernel.
    want_colors, want_sdf = torch.zeros_like(colors), torch.zeros_like(sdf)
    sharp, gsharp = torch.tensor(float(sc.sharpness), device=d), torch.zeros((), device=d)
    masks = torch.empty_like(keys.triangle_indices)
    counter = torch.empty(1, dtype=torch.int64, device=d)
    out = torch.empty_like(raw)
    h, w = grid.image_shape
    rows, cols = grid.grid_shape
    c, f = colors.detach(), sdf.detach()
    head = (nt.ptr(xy), nt.ptr(c), nt.ptr(f), xy.shape[1], nt.ptr(faces), nt.ptr(sharp), nt.ptr(keys.keys),
            nt.ptr(keys.triangle_indices), keys.num_keys)
    shape = (nt.ptr(ranges), b, s, rows, cols, *grid.tile_shape, h, w, tr._layout(kd), None, grid.camera_tiles)
    nt.call("mt_intersect_and_composite_forward", *head, None, *shape, nt.ptr(masks), nt.ptr(counter), nt.ptr(out), None,
            None, 0.0, None, None, 0, None, 0, grid.cta_threads, nt.stream(d))
    nt.call("mt_intersect_and_composite_backward", *head, *shape, nt.ptr(masks), nt.ptr(counter), nt.ptr(out),
            nt.ptr(g), None, None, 0.0, None, 1, nt.ptr(want_colors), nt.ptr(want_sdf), nt.ptr(gsharp),
            int(mode == "exact"), None, 0, None, 0, None, 0, grid.cta_threads, nt.stream(d))
    _close(got_colors, want_colors)
    _close(got_sdf, want_sdf)
    # A render's SH gradient (rows read in place) against the stages' one.
    background = torch.zeros(3, device=d)
    image = tr.render_fused(ext, intr, sc.image_shape, vertices, faces, sfb, sdf, sh, sc.sh_degree,
                            float(sc.sharpness), background, tile_shape=tile, gradient_mode=mode)
    gi = torch.randn(image.shape, device=d)
    got = torch.autograd.grad(image, (sdf, sh), gi)
    chained = tr.intersect_and_composite(xy, tr.evaluate_spherical_harmonics(vertices, sh, ext, sc.sh_degree), sdf, faces,
                                         float(sc.sharpness), keys.keys, keys.triangle_indices, ranges, s, grid, kd, mode)
    want = torch.autograd.grad((chained[:, :3] + chained[:, 3:] * background[:, None, None]).clip(0, 1), (sdf, sh), gi)
    for a, x in zip(got, want):
        _close(a, x)


@pytest.mark.parametrize("call", ["fused", "explicit", "cameras", "loss"])
@pytest.mark.parametrize("shape", ["column", "longer"])
def test_gradients_have_the_inputs_shapes(cuda_device, call, shape):
    """Signed distances as a column, or in a buffer longer than the vertices."""
    sc = make_scene(n=32, sh_degree=1, image_shape=(48, 40))
    d = cuda_device
    ext, intr, vertices, faces, sfb, sh, background = (
        torch.from_numpy(np.ascontiguousarray(x)).to(d)
        for x in (sc.extrinsics, sc.intrinsics, sc.vertices, sc.faces, sc.face_boundaries, sc.sh, sc.background))
    plain = torch.from_numpy(sc.sdf).to(d)
    other = plain[:, None] if shape == "column" else torch.cat((plain, plain.new_full((37,), 5.0)))
    target = torch.zeros((1, 3, *sc.image_shape), device=d)

    def gradients(sdf):
        sdf, rows = sdf.clone().requires_grad_(True), sh.clone().requires_grad_(True)
        mesh = (vertices, faces, sfb, sdf, rows, sc.sh_degree, 40.0, background)
        if call == "loss":
            loss = tr.render_fused_loss(ext, intr, sc.image_shape, *mesh, target)
        elif call == "cameras":
            loss = sum((x ** 2).mean() for x in tr.render_cameras(ext, intr, [sc.image_shape], *mesh))
        else:
            loss = (tr.render(ext, intr, sc.image_shape, *mesh, mode=call) ** 2).mean()
        return torch.autograd.grad(loss, (sdf, rows))

    want, want_sh = gradients(plain)
    got, got_sh = gradients(other)
    assert got.shape == other.shape
    _close(got.view(-1)[:len(plain)], want)
    _close(got_sh, want_sh)
    assert not got.view(-1)[len(plain):].any()


def test_gradient_of_longer_colours(cuda_device):
    grad = torch.randn((1, 5, 3), device=cuda_device)
    assert torch.equal(tr._flat_like(grad, torch.empty((1, 7, 3), device=cuda_device))[:, :5], grad)
    assert tr._flat_like(grad, grad) is grad


@pytest.mark.parametrize("tile", [(16, 16), (8, 8)])
def test_hits_of_a_warp_are_summed_first(cuda_device, monkeypatch, tile):
    """Two shells of eight triangles that fill the image, added to rows that hold
    2^24, where floats lie 2 apart: a hit's own contribution (below 1) would leave
    a row as it is, the sum over a warp's block of 8x4 pixels does not. Every
    addition rounds by at most 1, so a row misses 2^24 and its sum by at most the
    additions to it: one for every block and triangle around its vertex with six
    pixels or more in common, else one for each pixel."""
    d, size, start = cuda_device, 512, 2.0**24
    inner_init = tr._PackedGradients.__init__

    def init(self, *args):
        inner_init(self, *args)
        self.rows.fill_(start)

    monkeypatch.setattr(tr._PackedGradients, "__init__", init)
    at = torch.linspace(-8, size + 8, 3, device=d)
    xy = torch.stack(torch.meshgrid(at, at, indexing="xy"), -1).reshape(-1, 2)
    xy[4] += torch.tensor([37.0, -21.0], device=d)  # the vertex inside
    first = torch.tensor([0, 1, 3, 4], dtype=torch.int32, device=d)[:, None]
    corners = torch.tensor([[0, 3, 1], [1, 3, 4]], dtype=torch.int32, device=d)
    one = (first + corners.view(1, -1)).view(-1, 3)
    v, shells = xy.shape[0], 2
    faces = torch.cat((one, one + v))
    levels, sharpness = (0.01, -0.01), 40.0
    sdf = torch.tensor(levels, device=d).repeat_interleave(v)
    positions = xy.repeat(shells, 1)[None].contiguous()
    depths = torch.tensor([1.0, 2.0], device=d).repeat_interleave(v)[None].contiguous()
    grid = tr.TileGrid(tile, (size, size), 1, shells)
    kd = tr.create_key_defines(("camera", 6), ("tile", 20), ("depth", 32), ("shell", 6))
    ends = torch.tensor([8, 16], dtype=torch.int32, device=d)
    rect = tr.bound_triangles(positions, depths, faces, grid, 0.2)
    if not rect.num_tiles_overlapped.any():  # seen from behind
        faces = faces.flip(1).contiguous()
        rect = tr.bound_triangles(positions, depths, faces, grid, 0.2)
    keys = tr.sort_keys(tr.generate_keys(depths, faces, ends, rect.tile_minima, rect.tile_maxima,
                                         rect.num_tiles_overlapped, grid, kd))
    ranges = tr.delineate_tiles(keys, grid, kd, False).view(1, -1, 2)
    colors = torch.rand((1, shells * v, 3), generator=torch.Generator(d).manual_seed(1), device=d).requires_grad_(True)
    upstream = torch.full((1, 4, size, size), 2.0, device=d)
    upstream[:, 3] = 0
    raw = tr.intersect_and_composite(positions, colors, sdf, faces, sharpness, keys.keys, keys.triangle_indices, ranges,
                                     shells, grid, kd, "exact")
    (got,) = torch.autograd.grad(raw, colors, upstream)

    pixels = torch.arange(size, device=d, dtype=torch.float64) + 0.5
    points = torch.stack(torch.meshgrid(pixels, pixels, indexing="xy"), -1).view(-1, 2)
    sums, additions = (torch.zeros(v, dtype=torch.float64, device=d) for _ in range(2))
    free = torch.ones(len(points), dtype=torch.bool, device=d)

    def cross(p, q, r):
        return (q - p)[0] * (r - p)[..., 1] - (q - p)[1] * (r - p)[..., 0]

    for corner in one.tolist():
        p = xy[corner].double()
        weights = torch.stack([cross(p[(q + 1) % 3], p[(q + 2) % 3], points) for q in range(3)], -1)
        weights /= cross(p[0], p[1], p[2])
        # Pixels of the blocks that are the triangle's, and that rounding may make so.
        sure, most = ((weights >= x).all(-1).view(size // 4, 4, size // 8, 8).sum((1, 3)) for x in (1e-3, -1e-3))
        additions[corner] += torch.where(sure >= 6, most.clamp(max=1), most).sum()
        inside = (weights >= 0).all(-1) & free  # weights agree where two triangles meet
        free &= ~inside
        sums[corner] += weights[inside].sum(0)
    assert not free.any()
    outer, light = 1.0, 1.0
    for shell, level in enumerate(levels):
        inner = 1.0 / (1.0 + np.exp(-float(np.float32(level)) * sharpness))
        alpha = min(max((outer - inner + 1e-5) / (outer + 1e-5), 0.0), 1.0)
        want = 2.0 * light * alpha * sums
        assert 2.0 * light * alpha < 1.0 and float((want / additions).min()) > 1.5  # the test tells the two apart
        light, outer = light * (1.0 - alpha), inner
        off = (got[0, shell * v:(shell + 1) * v].double() - start - want[:, None]).abs()
        assert float((off / additions[:, None]).max()) <= 1.0
