"""Key duplication split by key slots: sorted keys, values and tile ranges bit-exact
against the oracle where a 4096-slot partition holds one Gaussian or thousands, and
around the sizes at which the counted passes' offsets take another level (one chunk
of 32 partitions, 131072 keys; one group of 32 chunks, 4M keys)."""
import numpy as np
import pytest

import torpedo_gb300 as T
from tests import gpu_helpers as H
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu


def _scene(n, scale):
    rec = configs.scene("cfg0", n).records.copy()
    rec[:, 0:3] *= 0.3
    rec[:, 8:11] = scale
    return rec


@pytest.mark.parametrize("lookback", [False, True])
@pytest.mark.parametrize("n,scale,width,height", [
    (1, 2.0, 40, 40),           # one Gaussian, a few keys
    (5000, 1e-4, 640, 480),     # thousands of small Gaussians in a partition
    (33, 3.0, 1008, 1040),      # 33 x 63 x 65 keys: 33 partitions, one past a chunk
    (32, 3.0, 1024, 1024),      # 32 x 4096 keys: exactly one chunk of whole partitions
    (1024, 3.0, 1024, 1024),    # 4M keys: exactly one group
    (1025, 3.0, 1024, 1024),    # one partition past a group
])
def test_keys_at_partition_edges(cuda, lookback, n, scale, width, height):
    rec = _scene(n, scale)
    cam = T.Camera.orbit((0.0, 0.0, -5.0), width, height)
    eng, stats = H.render(rec, [cam], key_sort_lookback=lookback)
    got = H.gpu_state(eng, stats)
    eng.close()
    want = H.oracle_frame(rec, cam, f64=False)
    assert got["K"] == want["K"]
    kept = int((want["s32"][:, 3] > 0).sum())
    np.testing.assert_array_equal(got["offsets"][:kept], want["depth_offsets"][:kept])
    np.testing.assert_array_equal(got["keys"], want["keys"])
    np.testing.assert_array_equal(got["vals"], want["vals"])
    np.testing.assert_array_equal(got["ranges"], want["ranges"])
