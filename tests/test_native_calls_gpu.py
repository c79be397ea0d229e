"""Calls of the C entries that the Python functions never make, and that a C
program may: optional pointers left out, buffers at their least alignment."""

import pytest
import torch

from meshtryoshka_gb300 import _native as nt
from meshtryoshka_gb300 import triangle_rasterization as tr

pytestmark = pytest.mark.gpu


def _entries(g, device):
    """Signed distances and lower corners [4, g] of entries with absent corners."""
    lower = torch.arange(g, dtype=torch.int32, device=device).repeat(4, 1)
    lower[1:] = (lower[1:] + 1) % g
    lower[2, ::3] = -64
    return torch.linspace(-1, 1, g, device=device), lower


@pytest.mark.parametrize("g", [1, 255, 1000])
def test_no_level_sets_and_no_offsets(cuda_device, g):
    """Without level sets there are no vertices: empty lists, zero gradients."""
    sdf, lower = _entries(g, cuda_device)
    kw = dict(device=cuda_device)
    inverse = torch.empty((4, g), dtype=torch.int32, **kw)
    offsets = torch.full((g + 1,), 7, dtype=torch.int32, **kw)
    need = int(nt.library().mt_build_vertex_grad_list_workspace_bytes(g))
    scratch = torch.zeros((need,), dtype=torch.uint8, **kw)
    nt.call("mt_build_vertex_grad_list", sdf.data_ptr(), lower.data_ptr(), g, None, 0, None, 0, inverse.data_ptr(),
            offsets.data_ptr(), None, scratch.data_ptr(), need, nt.stream(cuda_device))
    assert not offsets.any()

    need = int(nt.library().mt_create_triangle_vertices_backward_workspace_bytes(g, 0))
    scratch = torch.zeros((need,), dtype=torch.uint8, **kw)
    for workspace in (scratch.data_ptr(), None):  # lists, and the single pass
        grads = [torch.full(shape, 7.0, **kw) for shape in ((g,), (4, g, 3))]
        nt.call("mt_create_triangle_vertices_backward", sdf.data_ptr(), 4, lower.data_ptr(), g, None, 0, None, None,
                None, None, 0, inverse.data_ptr(), None, grads[0].data_ptr(), grads[1].data_ptr(), workspace,
                need if workspace else 0, nt.stream(cuda_device))
        assert not any(x.any() for x in grads)


@pytest.mark.parametrize("tile", [(16, 16), (9, 7), (20, 29)])
def test_first_hits_into_an_unaligned_buffer(cuda_device, tile):
    """out_uv at a 4-byte boundary: hits, misses and tiles without triangles."""
    d, (h, w) = cuda_device, (45, 70)
    rng = torch.Generator(d).manual_seed(3)
    f = 40
    xy = torch.rand((1, f, 1, 2), generator=rng, device=d) * 40 + torch.rand((1, f, 3, 2), generator=rng, device=d) * 9
    xy = xy.view(1, 3 * f, 2).contiguous()
    depths = torch.rand((1, 3 * f), generator=rng, device=d) + 1
    faces = torch.arange(3 * f, dtype=torch.int32, device=d).view(f, 3)
    faces = torch.cat((faces, faces.flip(1))).contiguous()  # one of the two faces the camera
    ends = torch.tensor([f, 2 * f], dtype=torch.int32, device=d)
    grid = tr.TileGrid(tile, (h, w), 1, 2)
    kd = tr.create_key_defines(("camera", 6), ("shell", 6), ("tile", 20), ("depth", 32))
    rect = tr.bound_triangles(xy, depths, faces, grid, 0.2)
    keys = tr.sort_keys(tr.generate_keys(depths, faces, ends, rect.tile_minima, rect.tile_maxima,
                                         rect.num_tiles_overlapped, grid, kd))
    ranges = tr.delineate_tiles(keys, grid, kd, True).contiguous()
    want = tr.intersect(xy, faces, keys.triangle_indices, ranges, grid, kd)
    assert 0 < int((want.index >= 0).sum()) < want.index.numel()
    rows, cols = grid.grid_shape
    uv = torch.full((want.uv.numel() + 1,), 7.0, device=d)
    index = torch.empty_like(want.index)
    nt.call("mt_intersect", xy.data_ptr(), xy.shape[1], faces.data_ptr(), keys.triangle_indices.data_ptr(),
            ranges.data_ptr(), 1, 2, rows, cols, *tile, h, w, uv.data_ptr() + 4, index.data_ptr(), nt.stream(d))
    assert torch.equal(uv[1:].view(want.uv.shape), want.uv) and torch.equal(index, want.index)
    assert float(uv[0]) == 7.0


@pytest.mark.parametrize("n", [1, 64, 5003])
def test_first_equal_keys_by_sorting(cuda_device, n):
    """Point keys and their numbers, a stable sort and its runs' heads give what
    the hash table gives; the numbers may be left out."""
    d = cuda_device
    rng = torch.Generator(d).manual_seed(n)
    quantized = torch.randint(-4, 5, (n, 3), generator=rng, device=d)
    keys, same = (torch.empty((n,), dtype=torch.int64, device=d) for _ in range(2))
    numbers, iota, order, got, want = (torch.empty((n,), dtype=torch.int32, device=d) for _ in range(5))
    nt.call("mt_pack_point_keys", quantized.data_ptr(), n, 4, keys.data_ptr(), numbers.data_ptr(), nt.stream(d))
    nt.call("mt_pack_point_keys", quantized.data_ptr(), n, 4, same.data_ptr(), None, nt.stream(d))
    nt.call("mt_iota_i32", n, iota.data_ptr(), nt.stream(d))
    assert torch.equal(same, keys) and torch.equal(iota, numbers)
    scratch, need = nt.workspace(d).get(nt.library().mt_sort_pairs_workspace_bytes(n))
    nt.call("mt_sort_pairs_i64_i32", keys.data_ptr(), iota.data_ptr(), same.data_ptr(), order.data_ptr(), n, None, 0,
            64, scratch, need, nt.stream(d))
    nt.call("mt_index_sorted_runs", same.data_ptr(), order.data_ptr(), n, got.data_ptr(), nt.stream(d))
    need = int(nt.library().mt_index_keys_workspace_bytes(n))
    table = torch.empty((need,), dtype=torch.uint8, device=d)
    nt.call("mt_index_keys", keys.data_ptr(), n, want.data_ptr(), table.data_ptr(), need, nt.stream(d))
    assert torch.equal(got, want)
