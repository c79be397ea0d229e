"""The keys of a render without a capacity (bounds, count read back, keys from
the records of the faces that touch a tile) equal bound_triangles ->
generate_keys: at a chunk's edges, with cameras that share a chunk, few and many
faces that touch a tile, faces past a live count and out-of-range vertices."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import triangle_rasterization as tr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,f", [(1, 1), (1, 1023), (1, 1024), (3, 1025), (70, 7), (2, 30_000)])
@pytest.mark.parametrize("spread", [0.3, 1.0, 6.0])
@pytest.mark.parametrize("ragged", [False, True])
def test_equal_the_chain(cuda_device, b, f, spread, ragged):
    rng = np.random.default_rng(b + f)
    d = cuda_device
    v, h, w = max(3, f // 2), 75, 131
    xy = (rng.normal(0.5, spread, (b, v, 2)) * (w, h)).astype(np.float32)
    depth = rng.uniform(0.0, 3.0, (b, v)).astype(np.float32)
    faces = rng.integers(0, v, (f, 3)).astype(np.int32)
    faces[:: 97] = (0, v, 1)  # names a vertex that does not exist
    near = np.minimum(faces, v - 1)
    # Small triangles: the second and third corners close to the first.
    for q in (1, 2):
        xy[:, near[:, q]] = xy[:, near[:, 0]] + rng.normal(0, 9, (b, f, 2)).astype(np.float32)
    bounds = np.sort(rng.integers(0, f + 1, 4)).astype(np.int32)
    bounds[-1] = f
    if ragged:
        grid = tr.TileGrid.for_cameras((16, 8), [(int(x), int(y)) for x, y in rng.integers(9, 140, (b, 2))], 4)
    else:
        grid = tr.TileGrid((16, 8), (h, w), b, 4)
    kd = tr.create_key_defines(("camera", 7), ("tile", 19), ("depth", 32), ("shell", 6))
    t = [torch.from_numpy(x).to(d) for x in (xy, depth, faces, bounds)]
    for live in (None, torch.tensor(f // 2 + 1, dtype=torch.int32, device=d)):
        got = tr._keys(t[0], t[1], t[2], t[3], grid, 0.2, live, kd, None)
        rect = tr.bound_triangles(t[0], t[1], t[2], grid, 0.2, live)
        want = tr.generate_keys(t[1], t[2], t[3], rect.tile_minima, rect.tile_maxima, rect.num_tiles_overlapped, grid, kd)
        assert torch.equal(got.keys, want.keys)
        assert torch.equal(got.triangle_indices, want.triangle_indices)


@pytest.mark.parametrize("b,f", [(1, 1 << 24), (1, (1 << 24) + 1), (3, 5_600_017), (2, (5 << 22) // 2 + 1024)])
def test_many_chunks(cuda_device, b, f):
    """Counts scanned by one CTA at most, and by one to each group of chunks: at
    the line between them, a group's edge and within one. Also by capacity."""
    d = cuda_device
    rng = torch.Generator(d).manual_seed(f)
    v, h, w = 4096, 64, 96
    xy = torch.rand((b, v, 2), generator=rng, device=d) * 40 * w
    depth = torch.rand((b, v), generator=rng, device=d) + 0.5
    first = torch.randint(0, v - 2, (f, 1), generator=rng, device=d, dtype=torch.int32)
    faces = (first + torch.arange(3, dtype=torch.int32, device=d)).contiguous()
    xy[:, 1::2] = xy[:, ::2] + torch.rand((b, v // 2, 2), generator=rng, device=d) * 9
    faces[f // 2:, 1:] = faces[f // 2:, 1:].flip(1)
    bounds = torch.tensor([f // 3, f // 2, f], dtype=torch.int32, device=d)
    grid = tr.TileGrid((16, 8), (h, w), b, 3)
    kd = tr.create_key_defines(("camera", 7), ("tile", 19), ("depth", 32), ("shell", 6))
    rect = tr.bound_triangles(xy, depth, faces, grid, 0.2)
    want = tr.generate_keys(depth, faces, bounds, rect.tile_minima, rect.tile_maxima, rect.num_tiles_overlapped, grid, kd)
    assert want.keys.numel() > 0
    got = tr._keys(xy, depth, faces, bounds, grid, 0.2, None, kd, None)
    assert torch.equal(got.keys, want.keys) and torch.equal(got.triangle_indices, want.triangle_indices)
    n = want.keys.numel() - 1  # one key too few
    got = tr._keys(xy, depth, faces, bounds, grid, 0.2, None, kd, n)
    assert int(got.count) == n + 1
    assert torch.equal(got.keys, want.keys[:n]) and torch.equal(got.triangle_indices, want.triangle_indices[:n])
