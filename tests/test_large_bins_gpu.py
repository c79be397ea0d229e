"""Tiles of more keys than one CTA sorts: their chunks are sorted side by side
and every key placed by its rank in each. Sizes at the chunk's edges, equal
depths (ties by original index), several such tiles beside small ones."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import triangle_rasterization as tr

pytestmark = pytest.mark.gpu

FUSED = (("camera", 6), ("tile", 20), ("depth", 32), ("shell", 6))


@pytest.mark.parametrize("sizes", [(4096,), (4097,), (4095, 4097, 1), (8192, 3), (8193, 0, 600, 4100),
                                   (12289, 200, 1024, 1025, 4096, 20000), (70001,)])
@pytest.mark.parametrize("depths", [3, 5000])
def test_sorted_as_one(cuda_device, sizes, depths):
    rng = np.random.default_rng(len(sizes) + sizes[0])
    tiles = len(sizes)
    kd = tr.create_key_defines(*FUSED)
    d = dict(kd)
    tile = np.repeat(np.arange(tiles, dtype=np.uint64), sizes)
    rng.shuffle(tile)
    depth = rng.choice(rng.uniform(0.5, 4.0, depths).astype(np.float32), tile.size).view(np.uint32).astype(np.uint64)
    shell = rng.integers(0, 4, tile.size).astype(np.uint64)
    keys = ((tile << np.uint64(d["TILE_BIT_OFFSET"])) | (depth << np.uint64(d["DEPTH_BIT_OFFSET"]))
            | (shell << np.uint64(d["SHELL_BIT_OFFSET"]))).view(np.int64)
    order = np.argsort(keys, kind="stable")
    paired = tr.PairedKeys(torch.from_numpy(keys).to(cuda_device),
                           torch.arange(keys.size, dtype=torch.int32, device=cuda_device), None)
    got, bounds = tr._sort_and_delineate(paired, tr.TileGrid((16, 16), (16, 16 * tiles), 1, 4), kd, False)
    np.testing.assert_array_equal(got.keys.cpu().numpy(), keys[order])
    np.testing.assert_array_equal(got.triangle_indices.cpu().numpy(), order)
    ends = np.cumsum(sizes)
    want = np.stack((ends - sizes, ends), -1) * (np.array(sizes) > 0)[:, None]
    np.testing.assert_array_equal(bounds.cpu().numpy().reshape(-1, 2), want)
