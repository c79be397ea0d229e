"""index_keys by its hash table: every table size's edge, keys of any bits (all
set among them), from all alike to all different, keys that differ in high bits
only."""

import numpy as np
import pytest
import torch

from meshtryoshka_gb300 import triangle_extraction as te

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 65, 4096, 100_003])
@pytest.mark.parametrize("kind", ["alike", "few", "half", "different", "high", "odd"])
def test_first_equal_key(cuda_device, n, kind):
    rng = np.random.default_rng(n)
    if kind == "odd":
        pool = np.array([-1, 0, 1, -2, np.iinfo(np.int64).min, np.iinfo(np.int64).max], np.int64)
        keys = rng.choice(pool, n)
    elif kind == "high":
        keys = rng.integers(-(1 << 20), 1 << 20, n) << 43
    else:
        many = {"alike": 1, "few": 7, "half": max(1, n // 2), "different": 1 << 62}[kind]
        keys = rng.integers(0, many, n) - (many // 2)
    _, first, inverse = np.unique(keys, return_index=True, return_inverse=True)
    got = te.index_keys(torch.from_numpy(keys.astype(np.int64)).to(cuda_device))
    np.testing.assert_array_equal(got.cpu().numpy(), first[inverse])
