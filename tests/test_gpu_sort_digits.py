"""Radix passes over digits that are spread (a warp's lanes of one digit found by shared atomics)
and concentrated (by ballots), around the share of one digit that decides between them, with
whole and partial partitions: the stable order in each, and passes of both kinds in one sort."""
import numpy as np
import pytest

import torpedo_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [12289, 40960, 131073, 600001])
@pytest.mark.parametrize("share", [0.0, 1 / 24.5, 1 / 23.5, 0.5, 1.0])
def test_sort_of_shared_digits(cuda, n, share):
    torch = cuda
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 45, size=n, dtype=np.uint64)
    for shift in (0, 16, 24, 40):  # the bytes between stay spread
        digit = np.full(n, 7, np.uint64) << np.uint64(shift)
        mask = np.uint64(0xFF << shift)
        took = np.zeros(n, bool)
        took[rng.permutation(n)[:round(n * share)]] = True
        keys = np.where(took, (keys & ~mask) | digit, keys)
    keys &= np.uint64((1 << 45) - 1)
    vals = np.arange(n, dtype=np.uint32)
    order = np.argsort(keys, kind="stable")
    k, v = T.sort_pairs(torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals.view(np.int32)).cuda(), 45)
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys[order])
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])
