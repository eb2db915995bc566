"""One engine taken through frames whose sorts and blends have different forms, in an order that
goes back and forth between them: few items (sorted in one launch) and many, one large view
(column strips), several views and small ones (keys of 8 or 9 bits a pass), tiles in list order
or not, scenes that shrink, key buffers that overflow. Every frame's keys, values, ranges and
image are those of an engine made for that frame alone, bit for bit."""
import numpy as np
import pytest

import torpedo_gb300 as T
from tests import gpu_helpers as H
from torpedo_gb300 import configs

pytestmark = pytest.mark.gpu

# (Gaussians, views, width, height)
FRAMES = {
    "few": (3000, 1, 201, 151),
    "strips": (40_000, 1, 1920, 1080),
    "views": (15_000, 3, 640, 360),
    "list order": (20_000, 1, 801, 603),
    "strips of few": (9000, 1, 1600, 900),
}
ORDER = ["strips", "views", "strips", "few", "list order", "strips of few", "views", "few", "strips"]


def _cams(views, w, h):
    return [T.Camera.orbit((0.3 * v, 0.1, -4.0), w, h) for v in range(views)]


def _frame(eng, name):
    n, views, w, h = FRAMES[name]
    eng.compile(configs.scene("cfg2", n).records)
    cams = _cams(views, w, h)
    if views == 1:
        eng.set_camera(cams[0])
    else:
        eng.set_views(cams)
    eng.raster_frame()  # (eager after a change, and where the keys overflow)
    stats = eng.raster_frame()  # a graph replay
    return H.gpu_state(eng, stats)


@pytest.mark.parametrize("settings", [{}, {"initial_key_capacity": 5000}, {"key_sort_lookback": True}])
def test_one_engine_through_all_forms(cuda, settings):
    want = {}
    for name in FRAMES:
        eng = T.GaussianEngine()
        want[name] = _frame(eng, name)
        eng.close()
    eng = T.GaussianEngine(**settings)
    for name in ORDER:
        got = _frame(eng, name)
        for what in ("keys", "vals", "ranges"):
            np.testing.assert_array_equal(got[what], want[name][what], err_msg=f"{name}: {what}")
        for a, b in zip(got["images"], want[name]["images"]):
            np.testing.assert_array_equal(a.view(np.uint32), b.view(np.uint32), err_msg=name)
    eng.close()
