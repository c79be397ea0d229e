"""create_voxels deals the vertices of 32 consecutive grid words out to a warp:
grids whose rows are shorter, as long as and longer than such a span, with
spans from a single vertex to 1024 of them, equal the oracle's tables."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import triangle_extraction as te
from oracle import oracle

from . import semantics

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1, 1, 32), (2, 3, 32 * 31), (1, 2, 32 * 32), (3, 1, 32 * 70), (37, 5, 32)])
@pytest.mark.parametrize("density", [0.002, 0.5, 1.0])
def test_spans_match_oracle(cuda_device, shape, density):
    rng = np.random.default_rng(shape[2])
    occupied = rng.random(shape) < density
    occupied[-1, -1, -1] = True  # the last word's bit 31
    occ = semantics.pack(occupied)
    want = oracle.extract_voxels(occ)
    got = te.extract_voxels(torch.from_numpy(np.ascontiguousarray(occ)).to(cuda_device))
    for field in ("vertices", "neighbors", "lower_corners", "upper_corners", "indices"):
        np.testing.assert_array_equal(getattr(got, field).cpu().numpy(), getattr(want, field), err_msg=field)
