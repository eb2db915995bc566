"""Frames whose blend takes the tiles by list length (between one and five waves of CTAs): the
same image, final transmittance and contributor counts as the FP64 oracle finds and, bit for
bit, as a frame of the same views whose blend takes them in order (batched with others beyond
five waves), for the plain and the persistent launch."""
import numpy as np
import pytest

import torpedo_gb300 as T
from tests import gpu_helpers as H
from tests import tolerances as tol
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("persistent", [False, True])
@pytest.mark.parametrize("width,height", [(592, 530), (801, 603), (1270, 719)])
def test_ordered_blend_equals_the_batched_views(cuda, persistent, width, height):
    sms = cuda.cuda.get_device_properties(0).multi_processor_count
    tiles = ((width + 15) // 16) * ((height + 15) // 16)
    rec = configs.scene("cfg0", 4000).records
    cam = T.Camera.orbit((0.5, 0.0, -4.0), width, height)
    eng, stats = H.render(rec, [cam], blend_persistent=persistent)
    got = H.gpu_state(eng, stats)
    eng.close()
    assert 8 * sms < tiles <= 40 * sms or sms != 152
    copies = 40 * sms // tiles + 1
    eng, stats = H.render(rec, [cam] * copies, blend_persistent=persistent)
    many = H.gpu_state(eng, stats)
    eng.close()
    n = width * height
    np.testing.assert_array_equal(got["images"][0], many["images"][-1])
    np.testing.assert_array_equal(got["final_T"], many["final_T"][-n:])
    np.testing.assert_array_equal(got["n_contrib"], many["n_contrib"][-n:])
    want = H.oracle_frame(rec, cam)
    err = np.abs(got["images"][0] - want["img64"]).max(axis=2)
    assert err[~want["pfrag"]].max() <= tol.IMAGE_ABS
