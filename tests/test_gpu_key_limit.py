"""A frame of 2^32 keys and a few more: the 32-bit key offsets come round to a
small count, which must not pass for the frame's. Every form of the key
duplication (column strips, keys of several views, the look-back form) ends with
TPD_ERR_CAPACITY, and the engine renders the next scene as a new one does."""
import numpy as np
import pytest

import torpedo_gb300 as T
from torpedo_gb300 import _lib as L
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu

W, H = 3840, 2160
TILES = (W // 16) * (H // 16)


@pytest.mark.parametrize("views,settings", [(1, {}), (2, {}), (1, {"key_sort_lookback": True})])
def test_more_keys_than_the_offsets_hold(cuda, views, settings):
    n = (1 << 32) // (TILES * views) + 1
    wrapped = n * TILES * views - (1 << 32)
    assert 0 < wrapped < 1 << 20  # within the smallest key buffers
    rng = np.random.default_rng(5)
    recs = configs.scene("cfg0", n).records.copy()
    recs[:, 0:3] = rng.normal(0.0, 0.1, (n, 3))
    recs[:, 4:8] = [0.0, 0.0, 0.0, 1.0]
    recs[:, 8:11] = 50.0  # every Gaussian covers the image
    cams = [T.Camera.orbit((0.0, 0.0, -5.0 - 0.01 * v), W, H) for v in range(views)]
    small = configs.scene("cfg0", 2000).records

    def frame(eng):
        eng.compile(small)
        eng.set_camera(cams[0])
        stats = eng.raster_frame()
        return stats["keys"], eng.read_image()[0]

    eng = T.GaussianEngine(**settings)
    eng.compile(recs)
    eng.set_views(cams)
    with pytest.raises(T.TpdError) as ei:
        eng.raster_frame()
    assert ei.value.code == L.TPD_ERR_CAPACITY
    keys, img = frame(eng)
    eng.close()
    ref = T.GaussianEngine(**settings)
    ref_keys, ref_img = frame(ref)
    ref.close()
    assert keys == ref_keys
    np.testing.assert_array_equal(img, ref_img)
