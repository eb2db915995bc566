"""The one-launch sort of few pairs, where it can go wrong: sizes around its CTAs' 32 keys, its
staging rounds of 4096 and the size past which the radix passes take over, key widths on both
sides of 32 bits, ties, and the largest keys; and frames whose depth sort takes it (single and
several views, culled Gaussians, equal depths)."""
import numpy as np
import pytest

import torpedo_gb300 as T
from tests import gpu_helpers as H
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 8, 32, 33, 45, 64])
@pytest.mark.parametrize("n", [1, 31, 33, 1025, 4096, 4097, 8192, 8193, 12287, 12288, 12289])
def test_sort_pairs(cuda, n, bits):
    torch = cuda
    rng = np.random.default_rng(n * 64 + bits)
    keys = rng.integers(0, 1 << 64, size=n, dtype=np.uint64)
    keys[rng.random(n) < 0.3] = rng.integers(0, 1 << 64, dtype=np.uint64)        # ties
    keys[rng.random(n) < 0.1] = np.uint64(0xFFFFFFFFFFFFFFFF)                     # as the padding
    keys = (keys & ~np.uint64(0xFF00)) | np.uint64(0x4200)                        # eight equal bits
    vals = rng.integers(0, 1 << 32, size=n, dtype=np.uint64).astype(np.uint32)
    low = keys & np.uint64((1 << bits) - 1)
    order = np.argsort(low, kind="stable")
    k, v = T.sort_pairs(torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals.view(np.int32)).cuda(), bits)
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys[order])
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("n", [1 << 17, (1 << 17) + 1, 1 << 19, (1 << 19) + 1])
def test_sort_pairs_where_the_partitions_grow(cuda, n):
    """Sizes at which a radix pass takes more keys per thread."""
    torch = cuda
    rng = np.random.default_rng(n)
    keys = rng.integers(0, 1 << 45, size=n, dtype=np.uint64)
    keys[rng.random(n) < 0.5] &= np.uint64(0xFF)
    vals = np.arange(n, dtype=np.uint32)
    order = np.argsort(keys, kind="stable")
    k, v = T.sort_pairs(torch.from_numpy(keys.view(np.int64)).cuda(), torch.from_numpy(vals.view(np.int32)).cuda(), 45)
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), keys[order])
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), vals[order])


@pytest.mark.parametrize("n,views", [(1, 1), (1025, 1), (12288, 1), (12289, 1), (3072, 4), (2000, 5)])
def test_frames(cuda, n, views):
    rec = configs.scene("cfg0", n).records.copy()
    rec[::7, 2] = 0.25  # equal depths in a view along z
    cams = [T.Camera.orbit(e, 96, 64) for e in ((0, 0, -5.0), (0, 0, 5.0), (4.0, 1.0, 0), (0, 0.5, -1.0), (-2, 1, 3.0))]
    eng, stats = H.render(rec, cams[:views])
    got = H.gpu_state(eng, stats)
    eng.close()
    at = base = 0
    for v, cam in enumerate(cams[:views]):
        want = H.oracle_frame(rec, cam, f64=False)
        sl = slice(at, at + want["K"])
        np.testing.assert_array_equal(got["keys"][sl], want["keys"] + (np.uint64(base) << np.uint64(32)))
        np.testing.assert_array_equal(got["vals"][sl], want["vals"])
        at += want["K"]
        base += ((cam.width + 15) // 16) * ((cam.height + 15) // 16)
    assert at == got["K"]
