"""Several threads on one stream: every thread's results are those of a call by
itself, though all share the stream's workspace, which grows on the way."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import _native as nt
from meshtryoshka_gb300 import pipeline
from meshtryoshka_gb300 import triangle_extraction as te
from meshtryoshka_gb300 import triangle_rasterization as tr
from tests.scenes import make_scene

pytestmark = pytest.mark.gpu


def _together(work, count):
    results, errors = [None] * count, []

    def run(i):
        try:
            results[i] = work(i)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=run, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors
    return results


@pytest.mark.parametrize("mode", ["fused", "explicit"])
def test_renders(cuda_device, mode):
    cameras = ((0.0, 0.0, 2.0), (1.2, 0.8, 1.3), (-1.5, -0.3, 1.1))
    sc = make_scene(cameras=cameras, image_shape=(96, 120), sh_degree=1)
    ext, intr, vertices, faces, sfb, sdf, sh, background = (
        torch.from_numpy(np.ascontiguousarray(x)).to(cuda_device)
        for x in (sc.extrinsics, sc.intrinsics, sc.vertices, sc.faces, sc.face_boundaries, sc.sdf, sc.sh, sc.background))

    def render(i):
        n, size = 1 + i % 3, (40 + 9 * i, 120 - 5 * i)
        for _ in range(4):
            image = tr.render(ext[:n], intr[:n], size, vertices, faces, sfb, sdf, sh, 1, 40.0, background, mode=mode)
        return image

    want = [render(i) for i in range(6)]
    torch.cuda.synchronize()
    nt._workspaces.clear()  # to grow again
    for got, image in zip(_together(render, 6), want):
        assert torch.equal(got, image)


def test_tessellations_and_their_gradients(cuda_device):
    w = pipeline.build_workload("small", cuda_device)
    v = w.voxels

    def tessellate(i):
        levels = w.level_sets[: 1 + i % w.level_sets.numel()]
        for _ in range(4):
            sdf, sh = (x.detach().clone().requires_grad_(True) for x in (w.grid_sdf, w.grid_sh))
            tri = te.tessellate_voxels(sdf, v.vertices, sh, v.neighbors, v.lower_corners, v.upper_corners, v.indices,
                                       levels)
            grads = torch.autograd.grad((tri.signed_distances.sum() + (tri.spherical_harmonics ** 2).sum()), (sdf, sh))
        return tri.vertices, tri.faces, *grads

    want = [tessellate(i) for i in range(6)]
    torch.cuda.synchronize()
    nt._workspaces.clear()
    for got, alone in zip(_together(tessellate, 6), want):
        for a, b in zip(got, alone):
            assert torch.equal(a, b)
