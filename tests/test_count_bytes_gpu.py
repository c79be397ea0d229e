"""The byte forms of the tessellation's counts: the scan of bytes (values and set
bits) around its vectors, warps and tiles, and the offsets and faces that the
crossings give, equal to those of the separate stages."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import pipeline
from meshtryoshka_gb300 import triangle_extraction as te

pytestmark = pytest.mark.gpu

TILE = 256 * 48


@pytest.mark.parametrize("n", [0, 1, 3, 4, 5, 127, 128, 1535, 1536, 1537, TILE - 1, TILE, TILE + 1, 7 * TILE, 40 * TILE + 77])
@pytest.mark.parametrize("set_bits", [False, True])
@pytest.mark.parametrize("most", [8, 256])
def test_scan_of_bytes(cuda_device, n, set_bits, most):
    values = np.random.default_rng(n).integers(0, most, n).astype(np.uint8)
    counts = np.unpackbits(values[:, None], axis=1).sum(1) if set_bits else values
    want = np.concatenate([[0], np.cumsum(counts, dtype=np.int64)])
    got = te._scan_bytes(torch.from_numpy(values).to(cuda_device), set_bits)
    np.testing.assert_array_equal(got.cpu().numpy(), want)


@pytest.mark.parametrize("side, shells", [(2, 1), (8, 1), (33, 5), (40, 24), (64, 6)])  # the last: 8 items a thread
@pytest.mark.parametrize("nans", [False, True])
def test_offsets_and_faces(cuda_device, side, shells, nans):
    rng = np.random.default_rng(side)
    voxels = te.extract_voxels(te.pack_occupancy(torch.from_numpy(rng.random((side, side, 64)) < 0.4).to(cuda_device)))
    sdf = torch.from_numpy(rng.normal(0.0, 0.05, voxels.num_vertices).astype(np.float32)).to(cuda_device)
    if nans:
        sdf[::7] = float("nan")
    levels = torch.linspace(0.05, -0.05, shells, device=cuda_device)
    sh = torch.zeros((1, voxels.num_vertices, 3), device=cuda_device)

    voff = te.count_triangle_vertices(sdf, voxels.lower_corners, levels)
    te.compute_exclusive_cumsum(voff)
    foff, codes = te.count_triangle_faces(sdf, voxels.lower_corners, voxels.upper_corners, levels)
    te.compute_exclusive_cumsum(foff)
    types = te.create_triangle_vertices(voxels.vertices, sdf, sh, voxels.lower_corners, levels, voff)[3]

    got_voff, crossings = te._vertex_offsets(sdf, voxels.lower_corners, levels)
    got_foff, got_codes = te._face_offsets(sdf, voxels.lower_corners, voxels.upper_corners, levels)
    assert torch.equal(got_voff, voff) and torch.equal(got_foff, foff) and torch.equal(got_codes, codes)
    v, f = int(voff[-1]), int(foff[-1]) // 3
    for vertices, faces in ((v, f), (v // 2, f // 2), (v + 100, f + 100)):  # also capacities
        common = (sdf, voxels.neighbors, voxels.indices, voff)
        rows = torch.cat([types, types.new_full((100,), 255)])[:vertices]
        want = te._create_triangle_faces("mt_create_triangle_faces", *common, rows, vertices, codes, levels, foff, faces,
                                         None)
        got = te._create_triangle_faces("mt_create_triangle_faces_by_crossings", *common, crossings, vertices, codes,
                                        levels, foff, faces, None)
        live = min(faces, f)
        assert torch.equal(got.faces[:live], want.faces[:live])
        assert torch.equal(got.voxel_indices[:live], want.voxel_indices[:live])


@pytest.mark.parametrize("counted", [False, True])
def test_no_level_sets_are_refused(cuda_device, counted):
    w = pipeline.build_workload("small", cuda_device)
    v = w.voxels
    args = (w.grid_sdf.detach(), v.vertices, w.grid_sh.detach(), v.neighbors, v.lower_corners, v.upper_corners,
            v.indices, w.level_sets[:0])
    with pytest.raises(RuntimeError, match="invalid argument"):
        te.tessellate_voxels_counted(*args, 10, 10) if counted else te.tessellate_voxels(*args)
