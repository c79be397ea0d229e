"""Projection with four vertices to a thread: the same positions and depths as by
small calls, around the size where it begins, and into an output that is not
8-byte aligned."""

import pytest
import torch

from meshtryoshka_gb300 import _native as nt
from meshtryoshka_gb300 import triangle_rasterization as tr

pytestmark = pytest.mark.gpu

LINE = 2 * 152 * 4 * 256


@pytest.mark.parametrize("v", [LINE - 1, LINE, LINE + 1, LINE + 1023, LINE + 1025])
@pytest.mark.parametrize("b", [1, 3])
def test_as_by_small_calls(cuda_device, v, b):
    gen = torch.Generator(device=cuda_device).manual_seed(v)
    vertices = torch.randn((v, 3), generator=gen, device=cuda_device)
    extrinsics = torch.randn((b, 4, 4), generator=gen, device=cuda_device)
    intrinsics = torch.randn((b, 3, 3), generator=gen, device=cuda_device)
    parts = [tr.project_vertices(p, extrinsics, intrinsics) for p in vertices.split(100_000)]
    want_xy = torch.cat([p.positions for p in parts], 1)
    want_depth = torch.cat([p.depths for p in parts], 1)
    got = tr.project_vertices(vertices, extrinsics, intrinsics)
    assert torch.equal(got.positions, want_xy) and torch.equal(got.depths, want_depth)

    odd = torch.full((2 * b * v + 1,), 7.0, device=cuda_device)[1:].view(b, v, 2)
    depths = torch.empty((b, v), device=cuda_device)
    nt.call("mt_project_vertices", nt.ptr(vertices), v, nt.ptr(extrinsics), nt.ptr(intrinsics), b, odd.data_ptr(),
            nt.ptr(depths), nt.stream(cuda_device))
    assert torch.equal(odd, want_xy) and torch.equal(depths, want_depth)
