"""The blend's one comparison per pair at its ends: a Gaussian whose conic is not a number (the
determinant of its covariance overflows: every pixel of its tiles takes alpha 0.99, as neither
skip test holds), one that is flat over the image (alpha is the opacity), and opacities that
never blend."""
import numpy as np
import pytest

import torpedo_gb300 as T
from tests import gpu_helpers as H
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("overflows,opacity,alpha", [(True, 0.5, 0.99), (True, 0.02, 0.99), (True, 0.003, 0.0),
                                                     (True, 0.0, 0.0), (False, 0.5, 0.5), (False, 1.0, 0.99),
                                                     (False, 0.003, 0.0), (False, -1.0, 0.0)])
def test_alpha_at_the_limits(cuda, overflows, opacity, alpha):
    rec = np.array(configs.scene("cfg0", 1).records)
    rec[0, :3], rec[0, 3], rec[0, 11] = 0.0, opacity, 1.0
    rec[0, 4:8] = 0.0, 0.0, np.sin(np.pi / 8), np.cos(np.pi / 8)  # long axis along x = y
    rec[0, 8:11] = (1e13, 1e9, 1e9) if overflows else 1e5
    eng, stats = H.render(rec, [T.Camera.orbit((0.0, 0.0, -4.0), 75, 50)])
    got = H.gpu_state(eng, stats)
    eng.close()
    splat = got["splats"].view(np.float32)[0]
    assert np.isnan(splat[8:11]).any() == overflows
    seen = np.zeros((50, 75), bool)
    for t, (lo, hi) in enumerate(got["ranges"]):
        seen[16 * (t // 5):16 * (t // 5) + 16, 16 * (t % 5):16 * (t % 5) + 16] = hi > lo
    assert seen.any()
    want = np.where(seen, np.float32(alpha), np.float32(0.0))
    np.testing.assert_allclose(got["images"][0], want[..., None] * splat[:3], rtol=1e-6, atol=0)
    np.testing.assert_array_equal(got["n_contrib"].reshape(50, 75), (want > 0).astype(np.uint32))
