"""Calls of the C entries that the Python functions never make, and that a C
program may: optional pointers left out, buffers at their least alignment."""

import pytest
import torch

from meshtryoshka_gb300 import _native as nt

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
