"""A training step whose keys outgrow the buffers, on an engine that has never
blended with the adjoint's inputs: its walk lengths are whatever the memory held
(here 0xFF bytes, where the allocator hands such memory out again). The step ends
with TPD_ERR_CAPACITY, and after a synchronous frame the next step's gradients are
those of an engine that saw only the second camera."""
import numpy as np
import pytest

import torpedo_gb300 as T
from torpedo_gb300 import _lib as L
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu

N, W, H = 3000, 96, 80


def test_step_overflows_before_any_state_was_kept(cuda):
    torch = cuda
    dev = torch.device("cuda")
    sc = configs.scene("cfg2", N)
    params = [torch.from_numpy(np.ascontiguousarray(a)).to(dev) for a in
              (sc.means, sc.log_scales, sc.quats, sc.opacity_logits, sc.sh)]
    inside, outside = T.Camera.orbit((0.0, 0.0, -0.5), W, H), T.Camera.orbit((0.0, 0.0, -5.0), W, H)  # few and many keys
    dimg = torch.from_numpy(np.random.default_rng(6).normal(size=H * W * 3).astype(np.float32)).to(dev)

    def step(eng):
        grads = [torch.empty_like(p) for p in params]
        eng.step_async(dimg, grads, 1)
        eng.sync()
        return [g.cpu().numpy() for g in grads]

    ones = torch.full((1 << 30,), 0xFF, dtype=torch.uint8, device=dev)
    del ones
    torch.cuda.empty_cache()
    eng = T.GaussianEngine(initial_key_capacity=1000)
    eng.compile_params(*params)
    eng.set_camera(inside)
    eng.raster_frame()
    eng.set_camera(outside)
    with pytest.raises(T.TpdError) as ei:
        step(eng)
    assert ei.value.code == L.TPD_ERR_CAPACITY
    eng.raster_frame()
    got = step(eng)
    eng.close()
    ref = T.GaussianEngine()
    ref.compile_params(*params)
    ref.set_camera(outside)
    ref.raster_frame()
    want = step(ref)
    ref.close()
    for a, b in zip(got, want):  # (equal up to the order of the adjoint's float atomic additions)
        np.testing.assert_allclose(a, b, rtol=1e-5, atol=1e-6 * float(np.abs(b).max(initial=0.0)))
