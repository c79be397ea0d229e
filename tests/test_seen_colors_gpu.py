"""Colours formed only for the vertices of the keys' triangles: the marks, and a
fused loss and its gradients with and without them (cameras that see a part of
the scene; a camera that sees nothing)."""

import pytest
import torch

from meshtryoshka_gb300 import pipeline
from meshtryoshka_gb300 import triangle_extraction as te
from meshtryoshka_gb300 import triangle_rasterization as tr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("live", [None, 0, 5, 64])
def test_marks(cuda_device, live):
    faces = torch.tensor([[0, 1, 2], [2, 3, 9], [4, -1, 40], [5, 6, 7]] + [[8, 8, 8]] * 60, dtype=torch.int32, device=cuda_device)
    keys = [0, 0, 1, 1, 1, 2, 70, -3] + [3] * 56
    triangles = torch.tensor(keys, dtype=torch.int32, device=cuda_device)
    deferred = te.DeferredSH(torch.empty((1, 10_000_000, 3), device="meta"))
    deferred.vertex_sources = torch.empty((3, 10), dtype=torch.int32, device=cuda_device)
    count = None if live is None else torch.tensor(live, dtype=torch.int64, device=cuda_device)
    seen = deferred.seen_vertices(triangles, count, faces, 0)
    want = {v for f in keys[:live] if 0 <= f < 64 for v in faces[f].tolist() if 0 <= v < 10}
    assert set(seen.nonzero()[:, 0].tolist()) == want and int(seen.max()) <= 1


@pytest.mark.parametrize("shift", [0.0, 0.6, 50.0])
def test_same_loss_and_gradients(cuda_device, monkeypatch, shift):
    w = pipeline.build_workload("small", cuda_device)
    rows = torch.randn((16, w.voxels.num_vertices, 3), generator=torch.Generator().manual_seed(0)).to(cuda_device) * 0.3
    results, marked = [], []
    inner = te.DeferredSH.seen_vertices
    monkeypatch.setattr(te.DeferredSH, "seen_vertices", lambda *a: marked.append(inner(*a)) or marked[-1])
    for limit in (1 << 40, -1):
        monkeypatch.setattr(te, "SEEN_COLOURS_BYTES", limit)
        torch.manual_seed(0)
        sdf = w.grid_sdf.detach().clone().requires_grad_(True)
        sh = rows.clone().requires_grad_(True)
        tri = te.tessellate_voxels(sdf, w.voxels.vertices, sh, w.voxels.neighbors, w.voxels.lower_corners,
                                   w.voxels.upper_corners, w.voxels.indices, w.level_sets, defer_sh=True)
        extrinsics = w.extrinsics.clone()
        extrinsics[:, 0, 3] += shift
        b, (h, wd) = extrinsics.shape[0], w.image_shape
        image = tr.render_fused(extrinsics, w.intrinsics, w.image_shape, pipeline.uncontract_stand_in(tri.vertices), tri.faces,
                                tri.face_boundaries, tri.signed_distances, tri.spherical_harmonics, 3, 40.0,
                                torch.zeros(3, device=cuda_device), tile_shape=(8, 8))
        weight = torch.rand((b, 3, h, wd), device=cuda_device)
        (image * weight).sum().backward()
        results.append((image.detach(), sdf.grad, sh.grad))
    assert marked[0] is None and marked[1] is not None
    (image0, d0, h0), (image1, d1, h1) = results
    assert torch.equal(image0, image1)
    for x, y in ((d0, d1), (h0, h1)):  # the atomic sums' order
        assert bool(torch.isfinite(y).all())
        assert float((x - y).abs().max()) <= 1e-4 * max(float(x.abs().max()), 1e-12)


@pytest.mark.parametrize("call", ["fused", "cameras", "loss"])
def test_unseen_colours_are_not_read(cuda_device, monkeypatch, call):
    """NaN in the place of every colour that was not formed changes nothing."""
    w = pipeline.build_workload("small", cuda_device)
    d, b = cuda_device, w.extrinsics.shape[0]
    h, wd = w.image_shape
    extrinsics = w.extrinsics.clone()
    extrinsics[:, 0, 3] += 0.6  # a part of the scene outside the image
    rows = torch.randn((16, w.voxels.num_vertices, 3), generator=torch.Generator().manual_seed(0)).to(d) * 0.3
    target = torch.rand((b, 3, h, wd), generator=torch.Generator().manual_seed(1)).to(d)
    poisoned = []

    def evaluate(self, vertices, extrinsics, sh_degree, seen=None):
        colors = inner(self, vertices, extrinsics, sh_degree, seen)
        if seen is not None:
            colors.data[:, seen == 0] = float("nan")
            poisoned.append(int((seen == 0).sum()))
        return colors

    inner = te.DeferredSH.evaluate
    monkeypatch.setattr(te.DeferredSH, "evaluate", evaluate)
    results = []
    for limit in (1 << 40, -1):
        monkeypatch.setattr(te, "SEEN_COLOURS_BYTES", limit)
        sdf, sh = w.grid_sdf.detach().clone().requires_grad_(True), rows.clone().requires_grad_(True)
        tri = te.tessellate_voxels(sdf, w.voxels.vertices, sh, w.voxels.neighbors, w.voxels.lower_corners,
                                   w.voxels.upper_corners, w.voxels.indices, w.level_sets, defer_sh=True)
        mesh = (pipeline.uncontract_stand_in(tri.vertices), tri.faces, tri.face_boundaries, tri.signed_distances,
                tri.spherical_harmonics, 3, 40.0, torch.zeros(3, device=d))
        if call == "loss":
            loss = tr.render_fused_loss(extrinsics, w.intrinsics, (h, wd), *mesh, target)
        elif call == "cameras":
            images = tr.render_cameras(extrinsics, w.intrinsics, [(h, wd)] * b, *mesh)
            loss = ((torch.stack(images) - target) ** 2).mean()
        else:
            loss = ((tr.render_fused(extrinsics, w.intrinsics, (h, wd), *mesh) - target) ** 2).mean()
        loss.backward()
        results.append((loss.detach(), sdf.grad, sh.grad))
    assert len(poisoned) == 1 and poisoned[0] > 0
    for x, y in zip(*results):  # the atomic sums' order
        assert bool(torch.isfinite(y).all())
        assert float((x - y).abs().max()) <= 1e-4 * max(float(x.abs().max()), 1e-12)
