"""Subdivision reads each vertex's parameters from its canonical duplicate in
place: bit for bit what copying them first gives, also where rows of more
vertices follow, in every coefficient count and with spans of words that hold
few and many vertices."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import subdivision
from meshtryoshka_gb300 import triangle_extraction as te

from oracle import oracle

from . import semantics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 4, 5, 9, 16, 18, 33])
@pytest.mark.parametrize("density,tol,more", [(0.01, 1e-6, 0), (0.2, 0.08, 0), (1.0, 0.08, 7)])
def test_canonical_rows_in_place(cuda_device, c, density, tol, more):
    rng = np.random.default_rng(c)
    occ = semantics.pack(rng.random((9, 14, 64)) < density)
    occ = torch.from_numpy(np.ascontiguousarray(occ)).to(cuda_device)
    vox = te.extract_voxels(occ)
    v, nv = vox.num_vertices, vox.num_voxels
    sdf = torch.from_numpy(rng.normal(size=v + more).astype(np.float32)).to(cuda_device)
    sh = torch.from_numpy(rng.normal(size=(c, v + more, 3)).astype(np.float32)).to(cuda_device)
    marked = vox.indices[:: max(1, nv // 20)]
    target = (13, 14, 96)
    got = subdivision.subdivide(vox, sdf, sh, occ, marked, target, dilation=2, tol=tol)
    canonical = te.index_vertices(vox.vertices, tol).long()
    assert (tol < 1e-3) or (canonical != torch.arange(v, device=cuda_device)).any()
    mask = te.dilate_occupancy(te.write_occupancy(marked, tuple(occ.shape), 0, 1), 2)
    want = te.upscale_parameters(sdf[canonical], sh[:, canonical], occ, mask, target)
    assert got.signed_distances.numel() > 0
    for a, b in zip(got, want):
        assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("c", [1, 5, 16, 18])
def test_infinities_and_nan_stay_where_they_are(cuda_device, c):
    """Absent corners add nothing, not even a zero times an infinity."""
    rng = np.random.default_rng(c)
    occ = semantics.pack(rng.random((7, 9, 64)) < 0.3)
    vox = oracle.extract_voxels(occ)
    v = vox.vertices.shape[0]
    sdf = rng.normal(size=v).astype(np.float32)
    sh = rng.normal(size=(c, v, 3)).astype(np.float32)
    for value in (np.inf, -np.inf, np.nan, 3e38):
        sh.reshape(-1)[rng.integers(0, sh.size, 40)] = value
    everything = np.full_like(occ, -1)
    with np.errstate(all="ignore"):
        want = oracle.upscale_parameters(sdf, sh, occ, everything, (12, 11, 96))
    got = te.upscale_parameters(*(torch.from_numpy(x).to(cuda_device) for x in (sdf, sh, occ, everything)), (12, 11, 96))
    np.testing.assert_array_equal(got.signed_distances.cpu().numpy(), want[0])
    np.testing.assert_array_equal(got.spherical_harmonics.cpu().numpy(), want[1])
    assert np.isfinite(want[1]).any() and not np.isfinite(want[1]).all()


def test_too_few_rows_are_refused(cuda_device):
    occ = torch.from_numpy(semantics.pack(np.ones((3, 4, 32), bool))).to(cuda_device)
    vox = te.extract_voxels(occ)
    sh = torch.zeros((1, vox.num_vertices, 3), device=cuda_device)
    with pytest.raises(IndexError):
        subdivision.subdivide(vox, sh.new_zeros(vox.num_vertices - 1), sh, occ, vox.indices, (6, 8, 64))


def test_rows_past_the_last_canonical_vertex_are_not_needed(cuda_device):
    """With a tolerance that merges the last vertices into earlier ones."""
    rng = np.random.default_rng(0)
    occ = torch.from_numpy(semantics.pack(np.ones((3, 4, 32), bool))).to(cuda_device)
    vox = te.extract_voxels(occ)
    tol = 0.9
    rows = int(te.index_vertices(vox.vertices, tol).max()) + 1
    assert rows < vox.num_vertices
    sdf = torch.from_numpy(rng.normal(size=vox.num_vertices).astype(np.float32)).to(cuda_device)
    sh = torch.from_numpy(rng.normal(size=(4, vox.num_vertices, 3)).astype(np.float32)).to(cuda_device)
    want = subdivision.subdivide(vox, sdf, sh, occ, vox.indices, (6, 8, 64), tol=tol)
    got = subdivision.subdivide(vox, sdf[:rows], sh[:, :rows], occ, vox.indices, (6, 8, 64), tol=tol)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    with pytest.raises(IndexError):
        subdivision.subdivide(vox, sdf[:rows - 1], sh, occ, vox.indices, (6, 8, 64), tol=tol)
