"""The blend adjoint where its blocks, rounds and lists are ragged: images cut inside a
tile's 8x4 blocks, lists of a round's length and one more, and every round setting,
against the FP64 oracle's analytic gradient."""
import numpy as np
import pytest

import torpedo_gb300 as T
from oracle import oracle as O
from tests import gpu_helpers as H
from tests import tolerances as tol
from torpedo_gb300 import configs
from torpedo_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("round_", [32, 64, 128])
@pytest.mark.parametrize("n,width,height", [(1, 1, 1), (32, 9, 5), (33, 17, 4), (64, 16, 16), (65, 31, 13),
                                            (129, 8, 33), (700, 47, 30)])
def test_adjoint_on_ragged_blocks(cuda, n, width, height, round_):
    torch = cuda
    sc = configs.scene("cfg2", n)
    means = sc.means * 0.2  # all Gaussians in front of the camera, on few tiles
    cam = T.Camera.orbit((0.0, 0.0, -3.0), width, height)
    params = [torch.from_numpy(np.ascontiguousarray(a)).cuda()
              for a in (means, sc.log_scales + 2.0, sc.quats, sc.opacity_logits, sc.sh)]
    dimg = np.random.default_rng(n).normal(size=(height, width, 3)).astype(np.float32)
    eng = T.GaussianEngine(blend_backward_round=round_)
    eng.compile_params(*params)
    eng.set_camera(cam)
    stats = eng.raster_frame()
    got = [t.cpu().numpy() for t in eng.backward(torch.from_numpy(dimg).cuda().reshape(-1))]
    vals = eng.read_buffer(L.TPD_BUF_VALUES, np.uint32, stats["keys"])
    rng = eng.read_buffer(L.TPD_BUF_RANGES, np.uint32, stats["tiles"] * 2).reshape(-1, 2)
    eng.close()
    p64 = [a.cpu().numpy().astype(np.float64) for a in params]
    want, _ = O.backward_f64(p64, H.ocam(cam), vals, rng, dimg.astype(np.float64))
    for name, a, b in zip(("means", "log_scales", "quats", "logits", "sh"), got, want):
        b = np.asarray(b, np.float64)
        assert np.linalg.norm(a.reshape(b.shape) - b) <= tol.GRAD_REL * np.linalg.norm(b), name
