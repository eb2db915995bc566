"""The key sort by column strips (one view, up to 256 x 256 tiles, more than 4096): offsets,
sorted keys, values and tile ranges bit-exact against the oracle at the edges of the column
and row digits (128 and 256 of each), where one strip holds one key or 256, around a chunk of
32 partitions of strips or keys, with few keys to a column and several columns to a partition,
and after the buffers have grown; and its look-back gives up as the keys' does."""
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


@pytest.mark.parametrize("n,scale,width,height", [
    (1, 3.0, 1040, 1024),        # one Gaussian over 65 x 64 tiles
    (3000, 1e-4, 1040, 1024),    # strips of one key or two
    (3000, 0.02, 2048, 513),     # 128 columns
    (3000, 0.02, 2049, 513),     # 129
    (3000, 0.02, 513, 2048),     # 128 rows
    (3000, 0.02, 513, 2049),     # 129
    (600, 3.0, 4081, 260),       # 256 columns, 33 + partitions of strips
    (300, 3.0, 260, 4096),       # 256 rows: strips of 256 keys
    (40, 3.0, 4096, 4096),       # both: 65536 tiles
    (500, 0.1, 4097, 260),       # 257 columns: sorted as keys
    (32, 3.0, 1039, 1020),       # 32 x 4160 keys
])
def test_strips_equal_the_oracle(cuda, n, scale, width, height):
    rec = _scene(n, scale)
    cam = T.Camera.orbit((0.0, 0.0, -5.0), width, height)
    eng, stats = H.render(rec, [cam], initial_key_capacity=5000)
    got = H.gpu_state(eng, stats)
    eng.close()
    want = H.oracle_frame(rec, cam, f64=False)
    assert got["K"] == want["K"]
    kept = int((want["s32"][:, 3] > 0).sum())
    np.testing.assert_array_equal(got["offsets"][:kept], want["depth_offsets"][:kept])
    np.testing.assert_array_equal(got["keys"], want["keys"])
    np.testing.assert_array_equal(got["vals"], want["vals"])
    np.testing.assert_array_equal(got["ranges"], want["ranges"])


@pytest.mark.parametrize("width,height", [(1920, 1080), (3840, 2160)])
def test_strips_equal_the_sorted_keys(cuda, width, height):
    rec = configs.scene("cfg0", 60000).records
    cam = T.Camera.orbit((0.5, 0.3, -4.0), width, height)
    states = []
    for ctas in (0, 2):  # 2: the keys themselves are sorted
        eng, stats = H.render(rec, [cam], sort_ctas_per_sm=ctas)
        states.append(H.gpu_state(eng, stats))
        eng.close()
    for field in ("offsets", "keys", "vals", "ranges", "n_contrib"):
        np.testing.assert_array_equal(states[0][field], states[1][field])
    np.testing.assert_array_equal(states[0]["images"][0], states[1]["images"][0])


def test_strip_scan_gives_up(cuda):
    eng = T.GaussianEngine(test_never_publish=True, spin_limit=2000, use_graph=False)
    eng.compile(configs.scene("cfg0", 20000).records)
    eng.set_camera(T.Camera.orbit((0.5, 0.3, -4.0), 1920, 1080))
    with pytest.raises(T.TpdError):
        eng.raster_frame()
    eng.close()
