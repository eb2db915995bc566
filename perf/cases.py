"""The calls that programs make of this package, as measurable cases.

Kinds of case, each through the package's public entry points:
  frame   a viewer's frame: set_camera, raster_frame, read the image (RGBA8 in
          host memory, or float RGB on the device)
  stream  a camera path rendered with two frames in flight into pinned host
          images (render_async / wait_render)
  train   one optimisation step's forward and gradients through torch.autograd
          (rasterize): parameters change every step, so they are taken anew
  step    the batched multi-view forward + backward (step_async) on parameters
          that the engine holds
  sort    the standalone radix sort of (tile | depth) keys
  scan    the standalone scan of tile counts

Scenes have the distributions of torpedo_gb300.configs: log-scales N(-4, .5),
unit quaternions, opacity sigmoid(N(0, 1)), SH coefficients N(0, .2); means
N(0, 1)^3 ("ball") or uniform in a box of half-width `box`. Cameras look at the
origin from a sphere of radius 5, field of view 60 degrees.
"""
import math

import numpy as np
import torch

import torpedo_gb300 as T
from torpedo_gb300.autograd import rasterize

SIZES_3 = ((640, 480), (1280, 720), (1920, 1080))  # the sizes of a mixed training batch
NEAR, FAR, FOV = 0.2, 100.0, 60.0


def listed():
    return [
        # a preview: few Gaussians, where launches and the host's waits count
        {"name": "frame preview", "kind": "frame", "n": 10_000, "width": 256, "height": 256, "box": 0.0, "degree": 3,
         "entities": 1, "host": True},
        # a mid-sized window of odd size over a scene of three moved entities, SH degree 2
        {"name": "frame odd entities", "kind": "frame", "n": 120_001, "width": 801, "height": 603, "box": 0.0,
         "degree": 2, "entities": 3, "host": False},
        # the headline frame: a million Gaussians at 1080p
        {"name": "frame 1080p", "kind": "frame", "n": 1_000_000, "width": 1920, "height": 1080, "box": 3.0, "degree": 3,
         "entities": 1, "host": False},
        # a 4K frame of a large scene
        {"name": "frame 4k", "kind": "frame", "n": 3_000_000, "width": 3840, "height": 2160, "box": 3.0, "degree": 3,
         "entities": 1, "host": False},
        # a recorded camera path: eight frames, two in flight, RGBA8 into pinned host memory
        {"name": "stream 1080p", "kind": "stream", "n": 1_000_000, "width": 1920, "height": 1080, "box": 3.0,
         "degree": 3, "frames": 8},
        # the first steps of an optimisation: a sparse initial cloud, small images of odd size
        {"name": "train small", "kind": "train", "n": 5_003, "width": 201, "height": 151, "box": 0.0, "degree": 1,
         "views": 1},
        # an optimisation step at the usual size of object scenes
        {"name": "train 800", "kind": "train", "n": 200_000, "width": 800, "height": 800, "box": 0.0, "degree": 3,
         "views": 1},
        # a batch of training views of mixed sizes, as one step
        {"name": "step 16 views", "kind": "step", "n": 500_000, "width": 0, "height": 0, "box": 0.0, "degree": 3,
         "views": 16},
        # the largest: 4K views from inside a large scene
        {"name": "step 4k inside", "kind": "step", "n": 6_000_000, "width": 3840, "height": 2160, "box": 10.0,
         "degree": 3, "views": 8},
        # the stages by themselves, for a caller's own pipeline
        {"name": "sort small", "kind": "sort", "n": 5_003, "bits": 40},
        {"name": "sort 9M", "kind": "sort", "n": 9_000_000, "bits": 45},
        {"name": "scan 1M", "kind": "scan", "n": 1_000_000},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tiles_per_gaussian(height, box):
    """About how many 16x16 tiles a Gaussian touches in a view of that height."""
    radius = (0.0145 if box <= 3.0 else 0.04) * height + 2.0
    return (2.0 * radius / 16.0 + 1.0) ** 2


def draw(rng):
    kind = rng.choice(("frame", "frame", "stream", "train", "train", "step", "step", "sort", "scan"))
    if kind == "sort":
        return {"kind": kind, "n": _log_uniform(rng, 100, 20_000_000), "bits": rng.randint(33, 50)}
    if kind == "scan":
        return {"kind": kind, "n": _log_uniform(rng, 1_000, 20_000_000)}
    height = _log_uniform(rng, 100, 2160)
    width = int(height * rng.choice((1.0, 4 / 3, 16 / 9)))
    case = {"kind": kind, "n": 0, "width": width, "height": height, "box": rng.choice((0.0, 3.0)),
            "degree": rng.choice((0, 1, 2, 3, 3, 3))}
    count, keys, most = 1, 60e6, 4_000_000
    if kind == "frame":
        case.update(entities=rng.choice((1, 1, 4)), host=rng.random() < 0.3)
    elif kind == "stream":
        case.update(frames=rng.randint(3, 10))
        count, keys, most = case["frames"], 100e6, 2_000_000
    elif kind == "train":
        case.update(views=rng.choice((1, 1, 2, 4)))
        count, keys, most = case["views"], 60e6, 1_000_000
    else:
        case.update(views=_log_uniform(rng, 2, 24))
        count, keys, most = case["views"], 120e6, 4_000_000
    # sizes whose keys stay below those of the largest listed case
    most = min(most, keys / count / _tiles_per_gaussian(height, case["box"]))
    case["n"] = _log_uniform(rng, 2_000, max(4_000, most))
    return case


# ---------------------------------------------------------------- inputs


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 7919 + 13)


def _params(case, seed):
    """Raw parameters (means, log-scales, quaternions, opacity logits, SH) on the GPU."""
    g, n = _gen(seed), case["n"]
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")  # noqa: E731
    if case["box"] > 0:
        means = (torch.rand((n, 3), generator=g, device="cuda") * 2 - 1) * case["box"]
    else:
        means = normal(n, 3)
    log_scales = normal(n, 3) * 0.5 - 4.0
    quats = torch.nn.functional.normalize(normal(n, 4))
    return [means, log_scales, quats, normal(n), normal(n, 48) * 0.2]


def _records(params):
    """The 240-byte records a scene file holds: activated opacity and scale, modifier 1."""
    means, log_scales, quats, logits, sh = params
    one = torch.ones_like(logits)[:, None]
    return torch.cat([means, torch.sigmoid(logits)[:, None], quats, torch.exp(log_scales), one, sh], 1)


def _entities(case, seed):
    """Per-record entity numbers and the entities' model matrices (small rigid moves)."""
    k = case.get("entities", 1)
    if k == 1:
        return None, []
    rng = np.random.default_rng(seed)
    ids = rng.integers(0, k, size=case["n"]).astype(np.uint32)
    mats = []
    for _ in range(k):
        a, t = rng.uniform(-0.3, 0.3), rng.uniform(-0.4, 0.4, 3)
        m = np.eye(4)
        m[0, 0] = m[2, 2] = math.cos(a)
        m[0, 2], m[2, 0] = math.sin(a), -math.sin(a)
        m[:3, 3] = t
        mats.append(m.astype(np.float32))
    return ids, mats


def _camera(rng, width, height):
    """A camera on the sphere, from its pose and intrinsics as a program reads them from a capture."""
    phi, y = rng.uniform(0.0, 2.0 * math.pi), rng.uniform(-0.7, 0.7)
    r = math.sqrt(1.0 - y * y)
    eye = 5.0 * np.array([r * math.cos(phi), y, r * math.sin(phi)])
    z = -eye / np.linalg.norm(eye)
    x = np.cross(z, (0.0, -1.0, 0.0))
    x /= np.linalg.norm(x)
    view = np.eye(4)
    for i, axis in enumerate((x, np.cross(z, x), z)):
        view[i, :3], view[i, 3] = axis, -axis @ eye
    fy = 1.0 / math.tan(math.radians(FOV) / 2)
    proj = np.zeros((4, 4))
    proj[0, 0], proj[1, 1] = fy * height / width, fy
    proj[2, 2], proj[2, 3], proj[3, 2] = NEAR / (NEAR - FAR), NEAR * FAR / (FAR - NEAR), 1.0
    return T.Camera(view.astype(np.float32), proj.astype(np.float32), width, height)


def _cameras(case, seed):
    rng = np.random.default_rng(1_000_003 + seed)
    count = case.get("views", case.get("frames", 1))
    sizes = [(case["width"], case["height"])] * count
    if not case["width"]:
        sizes = [SIZES_3[(seed + i) % 3] for i in range(count)]
    return [_camera(rng, w, h) for w, h in sizes]


def _pixel_gradient(pixels, seed):
    return torch.randn(pixels * 3, generator=_gen(seed + 1), device="cuda")


def prepare(case, seed):
    kind = case["kind"]
    if kind == "sort":
        g, n = _gen(seed), case["n"]
        tiles = torch.randint(0, 1 << (case["bits"] - 32), (n,), generator=g, device="cuda")
        depth = (torch.rand((n,), generator=g, device="cuda") * 6.0 + 2.0).view(torch.int32).long()
        keys, vals = tiles << 32 | depth, torch.arange(n, dtype=torch.int32, device="cuda")
        return {"case": case, "keys": keys, "vals": vals, "k": torch.empty_like(keys), "v": torch.empty_like(vals)}
    if kind == "scan":
        g, n = _gen(seed), case["n"]
        splats = torch.randint(0, 1 << 30, (n, 12), generator=g, device="cuda", dtype=torch.int32)
        counts = torch.randn((n,), generator=g, device="cuda").exp().mul(5).int()
        splats[:, 3] = torch.where(torch.rand((n,), generator=g, device="cuda") < 0.1, 0, counts)  # some culled
        return {"case": case, "splats": splats}

    params, cams = _params(case, seed), _cameras(case, seed)
    engine = T.GaussianEngine(sh_degree=case["degree"])
    state = {"case": case, "engine": engine, "cams": cams}
    pixels = sum(c.width * c.height for c in cams)
    if kind in ("frame", "stream"):
        ids, mats = _entities(case, seed)
        engine.compile(_records(params).cpu().numpy(), ids, max(1, len(mats)))
        for e, m in enumerate(mats):
            engine.get_transform_host().transform(e, m)
        if kind == "frame":
            state["image"] = torch.empty(pixels * 3, device="cuda")
        else:
            state["images"] = [torch.empty((c.height, c.width, 4), dtype=torch.uint8, pin_memory=True) for c in cams]
            engine.set_camera(cams[0])
            engine.raster_frame()  # sizes the key buffers before the pipelined frames
    elif kind == "train":
        state["params"] = [p.requires_grad_(True) for p in params]
        state["dimage"] = _pixel_gradient(pixels, seed)
    else:
        engine.compile_params(*params)
        engine.set_views(cams)
        engine.raster_frame()
        state["grads"] = [torch.empty_like(p) for p in params]
        state["dimage"] = _pixel_gradient(pixels, seed)
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "sort":
        # the sort works in place: the caller's pipeline writes fresh keys into these buffers each time
        state["k"].copy_(state["keys"])
        state["v"].copy_(state["vals"])
        return T.sort_pairs(state["k"], state["v"], case["bits"])
    if kind == "scan":
        return T.scan_tiles(state["splats"])
    engine, cams = state["engine"], state["cams"]
    if kind == "frame":
        engine.set_camera(cams[0])
        engine.raster_frame()
        if case["host"]:
            return engine.read_image(rgba8=True)
        engine.read_image_device(state["image"])
        return state["image"]
    if kind == "stream":
        images = state["images"]
        for i, cam in enumerate(cams):
            if i >= 2:
                engine.wait_render()
            engine.set_camera(cam)
            engine.render_async(images[i])
        for _ in range(min(2, len(cams))):
            engine.wait_render()
        return images
    if kind == "train":
        image = rasterize(*state["params"], engine, cams)
        return [image.detach(), *torch.autograd.grad(image, state["params"], state["dimage"])]
    engine.step_async(state["dimage"], state["grads"])
    engine.sync()
    return state["grads"]


# ---------------------------------------------------------------- work


def work(case):
    """Bytes: the inputs read once and the outputs written once. Operations: about 600 for each projected
    Gaussian and view, and 20 for each of about 64 blended entries of a pixel (three times both with the
    gradients); for the stages by themselves, one for each key and digit or count."""
    kind, n = case["kind"], case["n"]
    if kind == "sort":
        return {"bytes": 24 * n, "flops": n * math.ceil(case["bits"] / 8)}
    if kind == "scan":
        return {"bytes": 8 * n, "flops": n}
    count = case.get("views", case.get("frames", 1))
    if case["width"]:
        pixels = count * case["width"] * case["height"]
    else:
        pixels = sum(SIZES_3[i % 3][0] * SIZES_3[i % 3][1] for i in range(count))
    flops = 600 * n * count + 20 * 64 * pixels
    if kind == "frame":
        return {"bytes": 236 * n + (4 if case["host"] else 12) * pixels, "flops": flops}
    if kind == "stream":
        return {"bytes": 236 * n * count + 4 * pixels, "flops": flops}
    return {"bytes": 2 * 236 * n + (24 if kind == "train" else 12) * pixels, "flops": 3 * flops}


# ---------------------------------------------------------------- the same in 64 bits

_C1 = 0.4886025119029199
_C2 = (1.0925484305920792, -1.0925484305920792, 0.31539156525252005, -1.0925484305920792, 0.5462742152960396)
_C3 = (-0.5900435899266435, 2.890611442640554, -0.4570457994644658, 0.3731763325901154, -0.4570457994644658,
       1.445305721320277, -0.5900435899266435)


def _colour(degree, sh, d):
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    basis = [-_C1 * y, _C1 * z, -_C1 * x,
             _C2[0] * x * y, _C2[1] * y * z, _C2[2] * (2 * zz - xx - yy), _C2[3] * z * x, _C2[4] * (xx - yy),
             _C3[0] * y * (3 * xx - yy), _C3[1] * x * y * z, _C3[2] * y * (4 * zz - xx - yy),
             _C3[3] * z * (2 * zz - 3 * xx - 3 * yy), _C3[4] * x * (4 * zz - xx - yy), _C3[5] * z * (xx - yy),
             _C3[6] * x * (xx - 3 * yy)][:(0, 3, 8, 15)[degree]]
    out = 0.28209479177387814 * sh[:, :3]
    rest = sh[:, 3:].reshape(-1, 3, 15)
    for k, b in enumerate(basis):
        # the twelfth term is added, not multiplied: the default band-3 form
        out = out + (b[:, None] + rest[:, :, k] if k == 11 else b[:, None] * rest[:, :, k])
    return torch.clamp(out + 0.5, min=0.0)


def _project(means, opacity, quats, scales, sh, cam, degree, models, ids):
    """Splat tensors of the visible Gaussians in depth order, their tile rectangles and numbers."""
    view, proj = (torch.tensor(np.asarray(m, np.float64), device="cuda") for m in (cam.view, cam.proj))
    h = torch.cat([means, torch.ones_like(means[:, :1])], 1)
    if models:
        m = torch.tensor(np.asarray(models, np.float64), device="cuda")[torch.from_numpy(ids.astype(np.int64)).cuda()]
        h = (m @ h[:, :, None])[:, :, 0]
    v, c = h @ view.T, h @ (proj @ view).T
    w = c[:, 3]
    keep = (v[:, 2] > 0) & (c[:, 0].abs() <= 1.3 * w) & (c[:, 1].abs() <= 1.3 * w) & (c[:, 2] >= 0) & (c[:, 2] <= w)
    at = keep.nonzero()[:, 0]
    at = at[torch.argsort(v[at, 2].detach().float(), stable=True)]
    v, c, quats, scales, opacity = v[at], c[at], quats[at], scales[at], opacity[at]
    x, y, z, w = quats.unbind(1)
    rot = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                       2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                       2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    m = rot * scales[:, None, :]
    fx, fy = 0.5 * cam.width * proj[0, 0], 0.5 * cam.height * proj[1, 1]
    zero = torch.zeros_like(v[:, 0])
    jac = torch.stack([fx / v[:, 2], zero, -fx * v[:, 0] / v[:, 2] ** 2,
                       zero, fy / v[:, 2], -fy * v[:, 1] / v[:, 2] ** 2], 1).reshape(-1, 2, 3)
    tm = jac @ view[:3, :3] @ m
    cov = tm @ tm.transpose(1, 2)
    a, b, d = cov[:, 0, 0] + 0.3, cov[:, 1, 0], cov[:, 1, 1] + 0.3
    det = a * d - b * b
    conic = torch.stack([d / det, -b / det, a / det], 1)
    mid = 0.5 * (a + d)
    radius = torch.ceil(3 * torch.sqrt(mid + torch.sqrt(torch.clamp(mid * mid - det, min=0.1)))).detach()
    px = ((c[:, 0] / c[:, 3] + 1) * cam.width - 1) * 0.5
    py = ((c[:, 1] / c[:, 3] + 1) * cam.height - 1) * 0.5
    gx, gy = (cam.width + 15) // 16, (cam.height + 15) // 16
    bound = lambda p, most: torch.trunc(p.detach() / 16).clamp(0, most).long()  # noqa: E731
    rect = torch.stack([bound(px - radius, gx), bound(py - radius, gy), bound(px + radius + 15, gx),
                        bound(py + radius + 15, gy)], 1)
    eye = -(view[:3, :3].T @ view[:3, 3])
    direction = torch.nn.functional.normalize(means[at] - eye)
    return torch.cat([px[:, None], py[:, None], conic, opacity[:, None], _colour(degree, sh[at], direction)], 1), rect


def _tile(splats, xs, ys):
    """Colours of a tile's pixels from its depth-ordered splats (list x 9)."""
    px, py, ca, cb, cc, o, colour = *splats[:, :6].split(1, 1), splats[:, 6:]
    dx, dy = px - xs, py - ys
    power = -0.5 * (ca * dx * dx + cc * dy * dy) - cb * dx * dy
    alpha = torch.clamp(o * torch.exp(torch.clamp(power, max=0.0)), max=0.99)
    alpha = alpha * ((power <= 0) & (alpha >= 1 / 255)).detach()
    behind = torch.cumsum(torch.log1p(-alpha), 0)
    front = torch.exp(behind - torch.log1p(-alpha))
    weight = alpha * front * (torch.exp(behind) >= 1e-4).detach()
    return weight.T @ colour


def _render(splats, rect, cam, dimage=None):
    """The image, and the gradient of sum(dimage * image) to the splats where dimage is given."""
    image = torch.zeros((cam.height, cam.width, 3), dtype=torch.float64, device="cuda")
    leaf, grad = splats.detach(), None if dimage is None else torch.zeros_like(splats)
    gx, gy = (cam.width + 15) // 16, (cam.height + 15) // 16
    wide, high = (rect[:, 2] - rect[:, 0]).clamp(min=0), (rect[:, 3] - rect[:, 1]).clamp(min=0)
    count = wide * high
    owner = torch.repeat_interleave(torch.arange(len(rect), device="cuda"), count)
    local = torch.arange(len(owner), device="cuda") - (torch.cumsum(count, 0) - count)[owner]
    tile = (rect[owner, 1] + local // wide[owner]) * gx + rect[owner, 0] + local % wide[owner]
    tile, by = torch.sort(tile, stable=True)
    owner = owner[by]
    ends = torch.searchsorted(tile, torch.arange(gx * gy, device="cuda"), right=True).tolist()
    for t in range(gx * gy):
        start, end = ends[t - 1] if t else 0, ends[t]
        if start == end:
            continue
        x0, y0 = t % gx * 16, t // gx * 16
        x1, y1 = min(x0 + 16, cam.width), min(y0 + 16, cam.height)
        ys, xs = torch.meshgrid(torch.arange(y0, y1, device="cuda", dtype=torch.float64),
                                torch.arange(x0, x1, device="cuda", dtype=torch.float64), indexing="ij")
        own = leaf[owner[start:end]].requires_grad_(grad is not None)
        out = _tile(own, xs.reshape(1, -1), ys.reshape(1, -1))
        image[y0:y1, x0:x1] = out.detach().reshape(y1 - y0, x1 - x0, 3)
        if grad is not None:
            given = dimage[y0:y1, x0:x1].reshape(-1, 3)
            grad.index_add_(0, owner[start:end], torch.autograd.grad(out, own, given)[0])
    return image, grad


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("frame", "train") or case.get("host"):
        return None  # whole numbers, or (step) a frame too large for this
    count = case.get("views", 1)
    if count * case["n"] * _tiles_per_gaussian(case["height"], case["box"]) > (12e6 if kind == "frame" else 3e6):
        return None
    cams = _cameras(case, seed)
    params = _params(case, seed)
    if kind == "frame":
        rec = _records(params).double()
        ids, models = _entities(case, seed)
        splats, rect = _project(rec[:, :3], rec[:, 3], rec[:, 4:8], rec[:, 8:11], rec[:, 12:], cams[0], case["degree"],
                                models, ids)
        return _render(splats, rect, cams[0])[0].reshape(-1)
    raw = [p.double().requires_grad_(True) for p in params]
    dimage = _pixel_gradient(sum(c.width * c.height for c in cams), seed).double()
    images, at = [], 0
    for cam in cams:
        splats, rect = _project(raw[0], torch.sigmoid(raw[3]), raw[2], torch.exp(raw[1]), raw[4], cam, case["degree"],
                                None, None)
        size = cam.width * cam.height * 3
        image, grad = _render(splats, rect, cam, dimage[at:at + size].reshape(cam.height, cam.width, 3))
        splats.backward(grad)
        images.append(image.reshape(-1))
        at += size
    return [torch.cat(images), *(p.grad for p in raw)]
