"""Records built on the device from raw parameters: aligned and unaligned inputs, sizes around
a launch block's 256 16-byte pieces; and scenes compiled again on one engine."""
import numpy as np
import pytest

import torpedo_gb300 as T
from torpedo_gb300 import configs
from torpedo_gb300 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 17, 18, 257, 5003])
def test_records_of_raw_parameters(cuda, n, shift):
    torch = cuda
    sc = configs.scene("cfg2", n)
    raw = (sc.means, sc.log_scales, sc.quats, sc.opacity_logits, sc.sh)
    params = []
    for a in raw:  # shift: 4 bytes past the allocation's alignment
        flat = torch.empty(a.size + shift, dtype=torch.float32, device="cuda")
        flat[shift:] = torch.from_numpy(np.ascontiguousarray(a)).cuda().reshape(-1)
        params.append(flat[shift:].view(a.shape))
    eng = T.GaussianEngine()
    eng.compile_params(*params)
    eng.set_camera(T.Camera.orbit((0.0, 0.0, -5.0), 32, 32))
    got = eng.read_buffer(L.TPD_BUF_RECORDS, np.float32).reshape(n, 60)
    eng.close()
    for cols, want in ((slice(0, 3), sc.means), (slice(4, 8), sc.quats), (slice(12, 60), sc.sh)):
        np.testing.assert_array_equal(got[:, cols], want)
    np.testing.assert_array_equal(got[:, 11], 1.0)
    # expf is within 2 ulp, the sigmoid's sum and quotient add half an ulp each
    np.testing.assert_allclose(got[:, 8:11], np.exp(sc.log_scales.astype(np.float64)), rtol=1e-6)
    np.testing.assert_allclose(got[:, 3], 1 / (1 + np.exp(-sc.opacity_logits.astype(np.float64))), rtol=1e-6)


def test_scene_compiled_again_equals_a_fresh_engine(cuda):
    """One engine through scenes of the same size, another size, entities with transforms and
    back: each frame equals a fresh engine's (buffers and the captured frame may be kept)."""
    torch = cuda
    cam = T.Camera.orbit((0.0, 0.5, -5.0), 200, 120)
    model = np.eye(4, dtype=np.float32)
    model[0, 3] = 0.4

    def frames(eng, kind, n, seed):
        sc = T.synthetic_scene(seed, n)
        if kind == "params":
            eng.compile_params(*[torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in
                                 (sc.means, sc.log_scales, sc.quats, sc.opacity_logits, sc.sh)])
        else:
            ids = (np.arange(n) % 2).astype(np.uint32) if kind == "entities" else None
            eng.compile(sc.records, ids, 2 if kind == "entities" else 1)
            if kind == "entities":
                eng.transform_host.transform(1, model)
        eng.set_camera(cam)
        out = []
        for _ in range(3):  # the first frame, then replays
            eng.raster_frame()
            out.append(eng.read_image()[0])
        return out

    one = T.GaussianEngine()
    for kind, n, seed in (("params", 3000, 1), ("params", 3000, 2), ("params", 2500, 3), ("records", 2500, 4),
                          ("entities", 2500, 5), ("params", 2500, 6), ("params", 9000, 7), ("params", 10, 8),
                          ("params", 0, 9), ("params", 3000, 1)):
        fresh = T.GaussianEngine()
        want = frames(fresh, kind, n, seed)
        fresh.close()
        for a, b in zip(frames(one, kind, n, seed), want):
            np.testing.assert_array_equal(a, b)
    one.close()
