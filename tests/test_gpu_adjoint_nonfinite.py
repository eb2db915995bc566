"""An infinite, undefined or huge gradient of one pixel reaches the Gaussians that the pixel
counts and no other: the rest get what they get with that pixel's gradient at 0."""
import numpy as np
import pytest

import torpedo_gb300 as T
from tests import tolerances as tol
from torpedo_gb300 import _lib as L
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu

N, W, H = 1500, 96, 80
PIXEL = (40, 48)


@pytest.mark.parametrize("round_", [32, 64, 128])
@pytest.mark.parametrize("value,channels", [(np.inf, [0, 1, 2]), (-np.inf, [1]), (np.nan, [2]), (1e38, [0, 1, 2])])
def test_one_pixels_gradient_stays_with_its_entries(cuda, value, channels, round_):
    torch = cuda
    sc = configs.scene("cfg2", N)
    params = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
              for a in (sc.means, sc.log_scales, sc.quats, sc.opacity_logits, sc.sh)]
    eng = T.GaussianEngine(blend_backward_round=round_)
    eng.compile_params(*params)
    eng.set_camera(T.Camera.orbit((0.0, 0.0, -5.0), W, H))
    eng.raster_frame()

    def gradients(dimg):
        g = [t.cpu().numpy().reshape(N, -1) for t in eng.backward(torch.from_numpy(dimg).cuda().reshape(-1))]
        return g + [eng.read_buffer(L.TPD_BUF_G2D, np.float32, N * 12).reshape(N, 12)[:, :9]]

    one = np.zeros((H, W, 3), np.float32)
    one[PIXEL] = 1.0
    counted = gradients(one)[-1][:, 6] > 0.0  # the pixel's weights
    assert 0 < counted.sum() < N
    dimg = np.random.default_rng(3).normal(size=(H, W, 3)).astype(np.float32)
    dimg[PIXEL] = 0.0
    want = gradients(dimg)
    dimg[PIXEL + (channels,)] = value
    got = gradients(dimg)
    eng.close()
    for a, b in zip(got, want):
        assert np.linalg.norm((a - b)[~counted]) <= tol.GRAD_REL * np.linalg.norm(b[~counted])
    if not np.isfinite(value):
        assert not np.isfinite(got[-1][counted][:, [6 + c for c in channels]]).any()


def test_an_infinite_colour_stays_with_pixels_that_meet_it(cuda):
    """A Gaussian of infinite colour makes the gradient undefined at the pixels whose block meets
    it. An entry that such a pixel does not count takes nothing from it: with the gradient 0
    outside those pixels, the geometry of every Gaussian that they do not count gets exactly 0."""
    torch = cuda
    sc = configs.scene("cfg2", N)
    sh = np.ascontiguousarray(sc.sh).copy()
    sh[5, :3] = np.inf
    params = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
              for a in (sc.means, sc.log_scales, sc.quats, sc.opacity_logits, sh)]
    eng = T.GaussianEngine()
    eng.compile_params(*params)
    eng.set_camera(T.Camera.orbit((0.0, 0.0, -5.0), W, H))
    eng.raster_frame()
    bad = ~np.isfinite(eng.read_image()[0]).all(-1)
    assert 0 < bad.sum() < bad.size

    def records(dimg):
        eng.backward(torch.from_numpy(dimg).cuda().reshape(-1))
        return eng.read_buffer(L.TPD_BUF_G2D, np.float32, N * 12).reshape(N, 12)[:, :9]

    dimg = np.where(bad[..., None], np.float32(1.0), np.float32(0.0)) * np.ones((1, 1, 3), np.float32)
    got = records(dimg)
    eng.close()
    counted = got[:, 6] > 0.0  # weights of those pixels
    assert 0 < counted.sum() < N
    assert not np.any(got[~counted])
