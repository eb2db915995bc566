"""The standalone scan at the edges of its chunks of 32, warps of 512 and partitions of 4096 splats."""
import numpy as np
import pytest

import torpedo_gb300 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 33, 511, 513, 4095, 4096, 4097, 65 * 4096, 65 * 4096 + 1, 1_000_003])
def test_scan_tiles(cuda, n):
    torch = cuda
    rng = np.random.default_rng(n)
    sp = rng.integers(0, 1 << 32, size=(n, 12), dtype=np.uint64).astype(np.uint32)
    sp[:, 3] = rng.integers(0, 2000, size=n)
    offs, total = T.scan_tiles(torch.from_numpy(sp.view(np.int32)).cuda())
    want = np.cumsum(sp[:, 3], dtype=np.uint64)
    np.testing.assert_array_equal(offs.cpu().numpy().view(np.uint32), (want - sp[:, 3]).astype(np.uint32))
    assert int(total.item()) == int(want[-1])
