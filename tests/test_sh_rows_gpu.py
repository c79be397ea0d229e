"""Per-vertex SH rows and their gradient at the sizes where the kernels' tiles
can go wrong: fewer entries than a tile and ragged ones, one shell to more than
a warp's lanes of them, every split of the coefficient rows. Rows equal the
oracle's bit for bit; the list form of the gradient equals the single-pass
form, which enumerates the same contributions in the same order, bit for bit."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import _native as nt
from meshtryoshka_gb300 import triangle_extraction as te
from oracle import oracle

from . import semantics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("c", [1, 4, 5, 9, 16, 18])
@pytest.mark.parametrize("shape,shells", [((1, 2, 32), 1), ((5, 4, 64), 3), ((9, 11, 64), 21), ((9, 11, 32), 40)])
def test_rows_and_gradients(cuda_device, c, shape, shells):
    rng = np.random.default_rng(c)
    d = cuda_device
    occ = semantics.pack(rng.random(shape) < 0.5)
    vox = oracle.extract_voxels(occ)
    g = vox.vertices.shape[0]
    sdf = rng.normal(0, 0.05, g).astype(np.float32)
    sh = rng.normal(0, 1, (c, g, 3)).astype(np.float32)
    ls = np.linspace(0.06, -0.06, shells).astype(np.float32)
    t = {k: torch.from_numpy(np.ascontiguousarray(getattr(vox, k))).to(d)
         for k in ("vertices", "neighbors", "lower_corners", "upper_corners", "indices")}
    sdf_t = torch.from_numpy(sdf).to(d).requires_grad_(True)
    sh_t = torch.from_numpy(sh).to(d).requires_grad_(True)
    v_t = t["vertices"].requires_grad_(True)
    ls_t = torch.from_numpy(ls).to(d)
    tri = te.tessellate_voxels(sdf_t, v_t, sh_t, t["neighbors"], t["lower_corners"], t["upper_corners"], t["indices"],
                               ls_t)
    want = oracle.tessellate_voxels(sdf, vox.vertices, sh, vox.neighbors, vox.lower_corners, vox.upper_corners,
                                    vox.indices, ls)
    np.testing.assert_array_equal(tri.spherical_harmonics.detach().cpu().numpy(), want.spherical_harmonics)
    v = tri.vertices.shape[0]
    assert v > 0
    grads = [torch.from_numpy(rng.normal(0, 1, x.shape).astype(np.float32)).to(d)
             for x in (tri.vertices, tri.signed_distances, tri.spherical_harmonics)]
    got = torch.autograd.grad((tri.vertices, tri.signed_distances, tri.spherical_harmonics), (v_t, sdf_t, sh_t), grads)
    offsets = te.count_triangle_vertices(sdf_t.detach(), t["lower_corners"], ls_t)
    te.compute_exclusive_cumsum(offsets)
    single = [torch.empty_like(x) for x in (v_t, sdf_t, sh_t)]
    inverse = torch.empty((4, g), dtype=torch.int32, device=d)
    nt.call("mt_create_triangle_vertices_backward", sdf_t.data_ptr(), c, t["lower_corners"].data_ptr(), g,
            ls_t.data_ptr(), shells, offsets.data_ptr(), *(x.data_ptr() for x in grads), v, inverse.data_ptr(),
            *(x.data_ptr() for x in single), None, 0, nt.stream(d))
    for a, b in zip(got, single):
        assert torch.equal(a, b)
