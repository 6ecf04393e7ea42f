"""The work this library is measured on: what a program has it do, through its public
entry points, from the smallest calls to the largest.

Scenes have the distributions of athenea_b200/scenes.py (means uniform in a cube or from
eight clusters, log scales N(-4.5, 0.5), opacities sigmoid(N(0, 1)), SH N(0, 0.3)), drawn on
the GPU; cameras stand on a circle of radius 3 around them with a vertical field of view of
60 degrees. Kinds of case:

  frame   TileRasterizer.render of packed clouds: one view, colour and depth, and with
          "extra" the P layer and Cryptomatte layers ("matte") or the splats' weights in
          the frame ("weights")
  train   one differentiable frame of FP32 parameters, its L2 loss and its backward
  step    BatchTrainer.step: many views of a mixed-precision cloud, forward, loss, backward
  views   BatchTrainer.render: many views' colour and depth
  sort    ath_sorter_sort: (64-bit key, 32-bit value) pairs
  decode  CloudLoader.upload: 3DGS records to the packed cloud
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import athenea_b200 as A
from athenea_b200 import _native as N

REST = (0, 3, 8, 15)   # SH coefficients a colour after the constant, by degree
MIXED = ((320, 180), (640, 360), (960, 540), (1280, 720), (1920, 1080))
SH0 = 0.28209479177387814
FAINT = 1.0 / 255.0
TILE = 16


def listed():
    return [
        # an interactive preview or a thumbnail: a few thousand splats, the program waits for each frame
        dict(name="frame_5k_160x120", kind="frame", count=4999, clustered=True, degree=0, width=160, height=120,
             clouds=1, extra="none", threshold=False, wait=True),
        # an ordinary plain frame, spread evenly (workload 0 of scenes.py)
        dict(name="frame_100k_960x540", kind="frame", count=100_000, clustered=False, degree=3, width=960, height=540,
             clouds=1, extra="none", threshold=False, wait=False),
        # a trained capture at full HD (workload 1)
        dict(name="frame_1500k_1920x1080", kind="frame", count=1_500_000, clustered=True, degree=3, width=1920,
             height=1080, clouds=1, extra="none", threshold=False, wait=False),
        # a large capture at 4K, the sizes workload 4 is drawn at
        dict(name="frame_6000k_3840x2160", kind="frame", count=6_000_000, clustered=True, degree=3, width=3840,
             height=2160, clouds=1, extra="none", threshold=False, wait=False),
        # a composited shot: several clouds placed in one scene, the P layer and a Cryptomatte, odd sizes,
        # the depth layer in its threshold mode
        dict(name="frame_sections_matte", kind="frame", count=200_003, clustered=True, degree=1, width=1279, height=717,
             clouds=3, extra="matte", threshold=True, wait=False),
        # fitting a small object from a crop: odd sizes, a depth loss beside the colour's
        dict(name="train_20k_333x251", kind="train", count=20_011, clustered=True, degree=2, width=333, height=251,
             depth_loss=True),
        # one view a step in FP32 (workload 2)
        dict(name="train_500k_1280x720", kind="train", count=500_000, clustered=True, degree=3, width=1280, height=720,
             depth_loss=False),
        # the batched training step at its benchmark's size (workload 1, eight views)
        dict(name="step_1500k_8x1920x1080", kind="step", count=1_500_000, clustered=True, degree=3, views=8, width=1920,
             height=1080, tile=32, batch=256),
        # a batch of photographs of mixed sizes, as workload 3 has them, with the untuned defaults
        dict(name="step_250k_16_mixed", kind="step", count=250_007, clustered=True, degree=3, views=16, width=0,
             height=0, tile=0, batch=0),
        # evaluating a trained cloud from many cameras
        dict(name="views_500k_8x1280x720", kind="views", count=500_000, clustered=True, degree=3, views=8, width=1280,
             height=720, tile=32, batch=256),
        # the sorter on its own: keys of a 1080p frame's width (24 depth bits, 16 tile bits)
        dict(name="sort_8m_40bits", kind="sort", count=8_000_000, bits=40),
        # loading a trained capture, some of its records faint or broken
        dict(name="decode_1500k", kind="decode", count=1_500_000, degree=3),
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm, odd and even alike."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, most):
    """An image size: a standard one, or a ragged one of up to `most` pixels."""
    if rng.random() < 0.4:
        sizes = [s for s in MIXED + ((3840, 2160),) if s[0] * s[1] <= most]
        return rng.choice(sizes)
    pixels = _between(rng, 160 * 120, most)
    width = max(48, int(math.sqrt(pixels * rng.uniform(0.8, 2.2))))
    return width, max(32, min(pixels // width, most // width))


def draw(rng):
    kind = rng.choice(("frame", "frame", "frame", "train", "train", "step", "step", "views", "sort", "decode"))
    clustered, degree = rng.random() < 0.7, rng.choice((0, 1, 2, 3, 3))
    if kind == "frame":
        width, height = _size(rng, 3840 * 2160)
        return dict(kind=kind, count=_between(rng, 2000, 4_000_000), clustered=clustered, degree=degree, width=width,
                    height=height, clouds=rng.choice((1, 1, 1, 2, 5)),
                    extra=rng.choice(("none", "none", "matte", "weights")), threshold=rng.random() < 0.3,
                    wait=rng.random() < 0.3)
    if kind == "train":
        width, height = _size(rng, 1920 * 1080)
        return dict(kind=kind, count=_between(rng, 2000, 1_000_000), clustered=clustered, degree=degree, width=width,
                    height=height, depth_loss=rng.random() < 0.4)
    if kind in ("step", "views"):
        views = _between(rng, 1, 16)
        width, height = (0, 0) if rng.random() < 0.3 else _size(rng, 1280 * 720)
        return dict(kind=kind, count=_between(rng, 2000, 600_000), clustered=clustered, degree=degree, views=views,
                    width=width, height=height, tile=rng.choice((0, 16, 32, 32)), batch=rng.choice((128, 256)))
    if kind == "sort":
        return dict(kind=kind, count=_between(rng, 500, 10_000_000), bits=rng.choice((24, 32, 37, 40, 45, 64)))
    return dict(kind=kind, count=_between(rng, 2000, 1_500_000), degree=degree)


# ---- inputs ----------------------------------------------------------------------

def _gaussians(count, clustered, degree, seed):
    """The Gaussians of a scene, FP32 on the GPU (scenes.gaussians' distributions)."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 7919 + 20261203)
    normal = lambda *shape: torch.randn(shape, generator=gen, device="cuda")  # noqa: E731
    uniform = lambda *shape: torch.rand(shape, generator=gen, device="cuda") * 2.0 - 1.0  # noqa: E731
    if clustered:
        centres = uniform(8, 3)
        means = centres[torch.randint(0, 8, (count,), generator=gen, device="cuda")] + normal(count, 3) * 0.3
    else:
        means = uniform(count, 3)
    sh = normal(count, 3 + 3 * REST[degree]) * 0.3
    sh[:, 0:3] += 0.5
    quats = normal(count, 4)
    return dict(means=means, logits=normal(count), log_scales=normal(count, 3) * 0.5 - 4.5,
                quats=quats / quats.norm(dim=1, keepdim=True), sh=sh, degree=degree)


def _records(g):
    """3DGS records (x y z, normal, f_dc, f_rest colour-outer, opacity, scales, rotation), one a Gaussian."""
    count, rest = g["means"].shape[0], REST[g["degree"]]
    enc = A.encoding_3dgs(rest)
    out = torch.zeros((count, enc["stride"]), device="cuda")
    out[:, 0:3] = g["means"]
    out[:, 6:9] = g["sh"][:, 0:3]
    out[:, 9:9 + 3 * rest] = g["sh"][:, 3:].reshape(count, rest, 3).transpose(1, 2).reshape(count, 3 * rest)
    out[:, enc["opacity"]] = g["logits"]
    out[:, enc["scale0"]:enc["scale0"] + 3] = g["log_scales"]
    out[:, enc["rot_w"]:enc["rot_w"] + 4] = g["quats"]
    return out, enc


def _training(g):
    """The Gaussians as ath_params: means with the logit fourth, padded log scales."""
    means = torch.cat([g["means"], g["logits"][:, None]], 1).contiguous()
    scales = torch.cat([g["log_scales"], torch.zeros_like(g["logits"])[:, None]], 1).contiguous()
    return A.Params(means, scales, g["quats"].contiguous(), g["sh"].contiguous(), g["degree"])


def _eye(view, views, seed):
    t = 2.0 * math.pi * (view + 0.37 * (seed % 7)) / max(views, 1)
    return 3.0 * math.sin(t), 0.2, 3.0 * math.cos(t)


def _views(case, seed):
    """(projection, width, height) of each view of a batch (the mixed sizes are the case's own, whatever the seed)."""
    rng = np.random.default_rng(case["count"] + case["views"])
    found = []
    for v in range(case["views"]):
        w, h = (case["width"], case["height"]) if case["width"] else MIXED[rng.integers(0, len(MIXED))]
        cam = A.pinhole_for_vertical_fov(_eye(v, case["views"], seed), (0, 0, 0), w, h, 60.0)
        found.append((cam.projection_for(w, h), w, h))
    return found


def _sections(case):
    """Each cloud's Gaussian count and object_to_world: the clouds stand side by side, turned a little."""
    k, found = case["clouds"], []
    for c in range(k):
        t = 0.3 * c
        m = np.eye(4)
        m[0, 0], m[0, 2], m[2, 0], m[2, 2] = math.cos(t), math.sin(t), -math.sin(t), math.cos(t)
        m[:3, 3] = (0.5 * (c - 0.5 * (k - 1)), 0.1 * c, 0.0)
        found.append((case["count"] * (c + 1) // k - case["count"] * c // k, m))
    return found


def _random(shape, seed, scale=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed * 104729 + 5)
    return torch.rand(shape, generator=gen, device="cuda") * scale


def _sort_keys(case, seed):
    """Pairs as a frame emits them: a splat's depth with each of a run of neighbouring tiles (or random
    keys where the width is not a frame's)."""
    gen = torch.Generator(device="cuda").manual_seed(seed * 31 + 11)
    n, bits = case["count"], case["bits"]
    if 32 <= bits <= 45:
        splats = n // 7 + 1
        depth = (torch.randn(splats, generator=gen, device="cuda") * 0.4 + 3.0).clamp(0.5, 6.0)
        key = (depth.view(torch.int32).long() >> 7)
        first = torch.randint(0, 1 << (bits - 24), (splats,), generator=gen, device="cuda")
        at = torch.arange(n, device="cuda")
        tile = (first[at // 7] + at % 7) & ((1 << (bits - 24)) - 1)
        return (tile << 24) | key[at // 7], torch.arange(n, device="cuda", dtype=torch.int32)
    hi = torch.randint(0, 1 << 32, (n,), generator=gen, device="cuda")
    lo = torch.randint(0, 1 << 32, (n,), generator=gen, device="cuda")
    return (hi << 32) | lo, torch.arange(n, device="cuda", dtype=torch.int32)


class _Sorter:
    """An ath_sorter that is destroyed with its owner."""

    def __init__(self):
        self.lib, self.handle = N.lib(), ctypes.c_void_p()
        N.check(self.lib.ath_sorter_create(ctypes.byref(self.handle)))

    def __del__(self):
        self.lib.ath_sorter_destroy(self.handle)


def prepare(case, seed):
    kind, s = case["kind"], dict(case=case)
    if kind == "frame":
        w, h = case["width"], case["height"]
        s["instances"] = []
        for c, (count, placed) in enumerate(_sections(case)):
            records, enc = _records(_gaussians(count, case["clustered"], case["degree"], seed + 1000 * c))
            s["instances"].append(A.SplatInstance(A.CloudLoader.upload(records, enc), placed))
        s["camera"] = A.pinhole_for_vertical_fov(_eye(0, 7, seed), (0, 0, 0), w, h, 60.0)
        s["targets"] = A.RenderTargets.make(w, h, position=case["extra"] == "matte")
        s["settings"] = A.RenderSettings(width=w, height=h, depth_mode=1 if case["threshold"] else 0)
        if case["extra"] == "matte":
            gen = torch.Generator(device="cuda").manual_seed(seed + 3)
            s["settings"].crypto_ids = torch.randint(1, 24, (case["count"],), generator=gen, device="cuda",
                                                     dtype=torch.int32)
            s["settings"].crypto = torch.zeros((3, w * h, 4), device="cuda")
        elif case["extra"] == "weights":
            s["settings"].contribution_mode = 1
            s["settings"].contribution = torch.zeros(case["count"], dtype=torch.int32, device="cuda")
        s["raster"] = A.TileRasterizer.create()
    elif kind == "train":
        w, h = case["width"], case["height"]
        s["params"] = _training(_gaussians(case["count"], case["clustered"], case["degree"], seed))
        s["grads"] = s["params"].zeros_like()
        s["camera"] = A.pinhole_for_vertical_fov(_eye(0, 7, seed), (0, 0, 0), w, h, 60.0).projection_for(w, h)
        s["settings"], s["targets"] = A.RenderSettings(width=w, height=h), A.RenderTargets.make(w, h)
        s["target"] = _random((w * h, 3), seed)
        s["dcolour"], s["loss"] = torch.empty((w * h, 4), device="cuda"), torch.zeros(1, device="cuda")
        s["ddepth"] = _random((w * h,), seed + 1, 1.0 / (w * h)) if case["depth_loss"] else None
        s["raster"] = A.TileRasterizer.create()
    elif kind in ("step", "views"):
        g = _gaussians(case["count"], case["clustered"], case["degree"], seed)
        s["params"] = A.MixedParams.from_params(_training(g))
        s["trainer"] = A.BatchTrainer()
        s["trainer"].set_views(_views(case, seed))
        if case["tile"]:
            s["trainer"].set_tuning(case["tile"], case["batch"])
        pixels = s["trainer"].pixels
        s["colour"] = torch.empty((pixels, 4), device="cuda")
        if kind == "step":
            like = s["params"]
            s["target"], s["loss"] = _random((pixels, 3), seed), torch.zeros(1, device="cuda")
            s["grads"] = A.Params(torch.zeros_like(like.means), torch.zeros_like(like.scales),
                                  torch.zeros_like(like.quats), torch.zeros((case["count"], 48), device="cuda"))
        else:
            s["depth"] = torch.empty(pixels, device="cuda")
    elif kind == "sort":
        s["keys"], s["values"] = _sort_keys(case, seed)
        s["work"] = [torch.empty_like(s["keys"]), torch.empty_like(s["values"]), torch.empty_like(s["keys"]),
                     torch.empty_like(s["values"])]
        s["sorter"] = _Sorter()
    else:
        s["records"], s["encoding"] = _records(_file(case, seed))
    return s


def _file(case, seed):
    """A capture's Gaussians as its file has them: one in 50 too faint to keep, one in 5000 broken."""
    g = _gaussians(case["count"], True, case["degree"], seed)
    at = torch.arange(case["count"], device="cuda")
    g["logits"][at % 50 == 7] = -7.5
    g["means"][at % 5000 == 13, 1] = float("nan")
    return g


# ---- one pass ---------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "frame":
        settings, targets = s["settings"], s["targets"]
        if settings.contribution is not None:
            settings.contribution.zero_()
        s["raster"].render(s["camera"], s["instances"], settings, targets, do_check=case["wait"])
        out = dict(colour=targets.colour, depth=targets.depth)
        if case["extra"] == "matte":
            out["position"] = targets.position
            # a layer's four words are (id, coverage, id, coverage), the ids' bits as floats
            out["ids"] = settings.crypto.view(torch.int32)[..., 0::2]
            out["coverage"] = settings.crypto[..., 1::2]
        elif case["extra"] == "weights":
            out["weights"] = settings.contribution
        return out
    if kind == "train":
        g = s["grads"]
        for t in (g.means, g.scales, g.quats, g.sh, s["loss"]):
            t.zero_()
        s["raster"].render_params(s["camera"], s["params"], s["settings"], s["targets"], do_check=False)
        A.l2_loss(s["targets"].colour, s["target"], s["dcolour"], s["loss"])
        s["raster"].backward(s["dcolour"], g, s["ddepth"])
        return dict(colour=s["targets"].colour, depth=s["targets"].depth, loss=s["loss"], means=g.means,
                    scales=g.scales, quats=g.quats, sh=g.sh)
    if kind == "step":
        g = s["grads"]
        s["trainer"].step(s["params"], s["target"], s["colour"], s["loss"], g)
        return dict(colour=s["colour"], loss=s["loss"], means=g.means, scales=g.scales, quats=g.quats, sh=g.sh)
    if kind == "views":
        s["trainer"].render(s["params"], s["colour"], s["depth"])
        return dict(colour=s["colour"], depth=s["depth"])
    if kind == "sort":
        keys, values, more_keys, more_values = s["work"]
        keys.copy_(s["keys"])   # the sort is in place: each pass sorts the pairs as they were emitted
        values.copy_(s["values"])
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
        N.check(N.lib().ath_sorter_sort(s["sorter"].handle, ptr(keys), ptr(values), ptr(more_keys), ptr(more_values),
                                        case["count"], case["bits"],
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return dict(keys=keys, values=values)
    cloud = A.CloudLoader.upload(s["records"], s["encoding"])
    return dict(count=cloud.count, positions=cloud.positions, shape=cloud.shape, sh=cloud.sh)


# ---- what a pass cannot do without --------------------------------------------------

def _blended(case, width, height):
    """About how many splats a pixel blends: the footprints' area over the picture's, up to the ~40 after
    which a pixel of these scenes is opaque."""
    sigma = math.exp(-4.5) * (height * 0.5 / math.tan(math.radians(30.0))) / 3.0
    area = math.pi * 7.0 * (sigma * sigma + 0.3)
    spread = 0.35 if case["clustered"] else 0.25   # the share of the picture the scene covers
    return min(40.0, case["count"] * area / (width * height * spread)) * spread


def work(case):
    kind, n = case["kind"], case["count"]
    if kind == "sort":
        return {"bytes": 24 * n, "flops": 0}
    rest = REST[case["degree"]]
    packed = 32 + 4 * max(1, (3 * rest + 1) // 2)
    if kind == "decode":
        return {"bytes": n * (4 * (17 + 3 * rest) + packed), "flops": 60 * n}
    if kind in ("frame", "train"):
        w, h = case["width"], case["height"]
        sizes = [(w, h)]
    else:
        sizes = [(w, h) for _, w, h in _views(case, 0)]
    pixels = sum(w * h for w, h in sizes)
    blended = sum(_blended(case, w, h) * w * h for w, h in sizes)
    project = 400 * n * len(sizes)
    if kind == "frame":
        more = {"none": 0, "matte": 16 + 48, "weights": 0}[case["extra"]] * pixels
        return {"bytes": packed * n + 20 * pixels + more, "flops": project + 20 * blended}
    if kind == "views":
        return {"bytes": 112 * n + 20 * pixels, "flops": project + 20 * blended}
    cloud = 4 * (12 + 3 + 3 * rest) if kind == "train" else 112
    grads = 4 * (12 + 3 + 3 * rest) if kind == "train" else 240
    return {"bytes": (cloud + grads) * n + (16 + 12 + (24 if kind == "train" else 0)) * pixels,
            "flops": 2 * project + 65 * blended}


# ---- the same in 64 bits, in plain torch ----------------------------------------------

def _decoded(g):
    """A cloud as the packed layout holds it (half log scales, colours and SH, a smallest-three quaternion of ten
    bits a component), widened to 64 bits."""
    half = lambda t: t.clamp(-65000.0, 65000.0).half().double()  # noqa: E731
    q = torch.cat([g["quats"][:, 1:], g["quats"][:, :1]], 1)   # x y z w
    q = q / (((q[:, 0] * q[:, 0] + q[:, 1] * q[:, 1]) + q[:, 2] * q[:, 2]) + q[:, 3] * q[:, 3]).sqrt()[:, None]
    largest = q.abs().argmax(1, keepdim=True)
    q = torch.where(q.gather(1, largest) < 0, -q, q)
    unit = ((q / 0.70710678) * 0.5 + 0.5).clamp(0.0, 1.0) * 1023.0
    kept = ((torch.floor(unit + 0.5).double() / 1023.0) * 2.0 - 1.0) * math.sqrt(0.5)
    kept.scatter_(1, largest, 0.0)
    kept.scatter_(1, largest, (1.0 - kept.square().sum(1, keepdim=True)).clamp(min=0.0).sqrt())
    return dict(means=g["means"].double(), opacity=torch.sigmoid(g["logits"].double()),
                scales=half(g["log_scales"]).exp(), quats=kept, base=half(0.5 + SH0 * g["sh"][:, :3]),
                rest=half(g["sh"][:, 3:]).reshape(g["sh"].shape[0], REST[g["degree"]], 3))


def _trained(means, scales, quats, sh):
    """Training parameters (64 bits) as the projection reads them."""
    q = quats / quats.norm(dim=1, keepdim=True)
    return dict(means=means[:, :3], opacity=torch.sigmoid(means[:, 3]), scales=scales[:, :3].exp(),
                quats=torch.cat([q[:, 1:], q[:, :1]], 1), base=0.5 + SH0 * sh[:, :3],
                rest=sh[:, 3:].reshape(sh.shape[0], (sh.shape[1] - 3) // 3, 3))


def _sh_basis(d):
    x, y, z = d.unbind(1)
    xx, yy, zz = x * x, y * y, z * z
    c1, c2, c3 = 0.4886025119029199, 1.0925484305920792, -0.4570457994644658
    return torch.stack([
        -c1 * y, c1 * z, -c1 * x,
        c2 * x * y, -c2 * y * z, 0.31539156525252005 * (2 * zz - xx - yy), -c2 * x * z, 0.5462742152960396 * (xx - yy),
        -0.5900435899266435 * y * (3 * xx - yy), 2.890611442640554 * x * y * z, c3 * y * (4 * zz - xx - yy),
        0.3731763325901154 * z * (2 * zz - 3 * xx - 3 * yy), c3 * x * (4 * zz - xx - yy),
        1.445305721320277 * z * (xx - yy), -0.5900435899266435 * x * (xx - 3 * yy)], 1)


def _matrix(values):
    return np.array(list(values), np.float64).reshape(4, 4)


def _project(c, proj, width, height, placed):
    """The splats' screen records: (cx, cy, z, conic a b c, alpha, r g b) a splat and the cutoff power (below zero
    for one that is not drawn)."""
    # the frame's constants are handed over as 32-bit numbers
    m = torch.from_numpy((_matrix(proj.world_to_view) @ placed).astype(np.float32).astype(np.float64)).cuda()
    eye = np.append(np.array(list(proj.eye_world)), 1.0)
    eye = torch.from_numpy((np.linalg.inv(placed) @ eye)[:3].astype(np.float32).astype(np.float64)).cuda()
    fx, fy, cx0, cy0, near, far = (float(np.float32(v)) for v in (proj.focal_x, proj.focal_y, proj.centre_x,
                                                                  proj.centre_y, proj.near_z, proj.far_z))
    t = c["means"] @ m[:3, :3].T + m[:3, 3]
    z = t[:, 2]
    seen = (z > near) & (z <= far)
    zs = torch.where(seen, z, torch.ones_like(z))
    x, y, zz, w = c["quats"].unbind(1)
    r = torch.stack([1 - 2 * (y * y + zz * zz), 2 * (x * y - w * zz), 2 * (x * zz + w * y),
                     2 * (x * y + w * zz), 1 - 2 * (x * x + zz * zz), 2 * (y * zz - w * x),
                     2 * (x * zz - w * y), 2 * (y * zz + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(-1, 3, 3)
    shape = r * c["scales"][:, None, :]
    ux = (t[:, 0] / zs).clamp((-0.15 * width - cx0) / fx, (1.15 * width - cx0) / fx)
    uy = (t[:, 1] / zs).clamp((-0.15 * height - cy0) / fy, (1.15 * height - cy0) / fy)
    jx = (fx / zs)[:, None] * (m[0, :3] - ux[:, None] * m[2, :3])
    jy = (fy / zs)[:, None] * (m[1, :3] - uy[:, None] * m[2, :3])
    ax, ay = torch.einsum("ni,nij->nj", jx, shape), torch.einsum("ni,nij->nj", jy, shape)
    a, b, cc = (ax * ax).sum(1), (ax * ay).sum(1), (ay * ay).sum(1)
    before, det = a * cc - b * b, (a + 0.3) * (cc + 0.3) - b * b
    paid = (before.clamp(min=1e-30) / det).sqrt()
    spread = paid * c["opacity"]
    alpha = torch.where(spread >= FAINT, spread + (1.0 - paid) * FAINT, spread)
    drawn = seen & (det > 1e-12) & (alpha >= FAINT)
    direction = c["means"] - eye
    direction = direction / direction.norm(dim=1, keepdim=True)
    colour = c["base"]
    k = c["rest"].shape[1]
    if k:
        colour = colour + torch.einsum("nk,nkc->nc", _sh_basis(direction)[:, :k], c["rest"])
    colour = colour.clamp(min=0.0)
    colour = torch.where(colour <= 0.04045, colour / 12.92, ((colour.clamp(min=0.01) + 0.055) / 1.055) ** 2.4)
    rec = torch.cat([torch.stack([fx * t[:, 0] / zs + cx0, fy * t[:, 1] / zs + cy0, z, (cc + 0.3) / det, -b / det,
                                  (a + 0.3) / det, alpha], 1), colour], 1)
    cutoff = (2.0 * (255.0 * alpha).clamp(min=1.0001).log()).clamp(max=9.0)
    return rec, torch.where(drawn, cutoff, torch.full_like(cutoff, -1.0))


def _bin(rec, cutoff, width, height):
    """The splats of each tile in the order they are blended, (splat of a pair, first, last) a tile. Drawn order is
    by the depth's 24 most significant bits as a 32-bit float, ties in the splats' order."""
    det = rec[:, 3] * rec[:, 5] - rec[:, 4] ** 2
    power = cutoff.clamp(min=0.0)
    ex, ey = (power * rec[:, 5] / det).sqrt(), (power * rec[:, 3] / det).sqrt()
    lo_x, hi_x, lo_y, hi_y = rec[:, 0] - ex, rec[:, 0] + ex, rec[:, 1] - ey, rec[:, 1] + ey
    on = (cutoff >= 0) & (hi_x >= 0) & (hi_y >= 0) & (lo_x < width) & (lo_y < height)
    which = on.nonzero().squeeze(1)
    tiles_x, tiles_y = -(-width // TILE), -(-height // TILE)
    at = lambda v, most: (v[which].clamp(0, most) / TILE).long()  # noqa: E731
    x0, x1, y0, y1 = at(lo_x, width - 1), at(hi_x, width - 1), at(lo_y, height - 1), at(hi_y, height - 1)
    across = x1 - x0 + 1
    area = across * (y1 - y0 + 1)
    owner = torch.repeat_interleave(torch.arange(which.numel(), device=rec.device), area)
    local = torch.arange(owner.numel(), device=rec.device) - (area.cumsum(0) - area)[owner]
    tile = (y0[owner] + local // across[owner]) * tiles_x + x0[owner] + local % across[owner]
    depth = rec[which, 2].float().view(torch.int32).long() >> 7
    key, order = torch.sort((tile << 24) | depth[owner], stable=True)
    edges = torch.searchsorted(key, torch.arange(tiles_x * tiles_y + 1, device=rec.device) << 24)
    return which[owner[order]], edges[:-1], edges[1:]


def _chunk(rows, power_limit, xy, light):
    """One run of a tile's splats over its pixels: what they add (r g b, depth), the light left after them, and which
    of them crosses a coverage of a half."""
    dx, dy = xy[:, None, :, 0] - rows[:, :, 0, None], xy[:, None, :, 1] - rows[:, :, 1, None]
    power = rows[:, :, 3, None] * dx * dx + 2.0 * rows[:, :, 4, None] * dx * dy + rows[:, :, 5, None] * dy * dy
    alpha = (rows[:, :, 6, None] * (-0.5 * power).exp()).clamp(max=0.99)
    alpha = torch.where((power <= power_limit[:, :, None]) & (alpha >= FAINT), alpha, torch.zeros_like(alpha))
    through = torch.cat([light[:, None], light[:, None] * (1.0 - alpha).cumprod(1)], 1)
    alpha = torch.where(through[:, :-1] >= 1e-4, alpha, torch.zeros_like(alpha))
    weight = through[:, :-1] * alpha
    added = torch.einsum("gkp,gkc->gpc", weight, rows[:, :, [7, 8, 9, 2]])
    return added, light * (1.0 - alpha).prod(1), weight, through


def _walk(rec, cutoff, width, height, adjoint=None, threshold=False, tiles_at_once=768, run=32):
    """Blends a view: (colour, depth), and with `adjoint` (colour, depth -> dL/dcolour, dL/ddepth; depth in its mean
    mode) also dL/drec."""
    pairs, first, last = _bin(rec, cutoff, width, height)
    tiles_x = -(-width // TILE)
    colour = torch.zeros((width * height, 4), dtype=torch.float64, device=rec.device)
    depth = torch.zeros(width * height, dtype=torch.float64, device=rec.device)
    kept = []
    inner = torch.arange(TILE * TILE, device=rec.device)
    order = torch.argsort(last - first)
    for block in order.split(tiles_at_once):
        px = (block % tiles_x)[:, None] * TILE + inner % TILE
        py = (block // tiles_x)[:, None] * TILE + inner // TILE
        inside = (px < width) & (py < height)
        xy = torch.stack([px + 0.5, py + 0.5], 2).double()
        total = torch.zeros((*px.shape, 4), dtype=torch.float64, device=rec.device)
        light = inside.double()
        light = torch.where(inside, light, torch.zeros_like(light))
        crossed = torch.full_like(light, -1.0)
        active, k = torch.arange(block.numel(), device=rec.device), 0
        steps = []
        while True:
            active = active[((last - first)[block[active]] > k) & (light[active].amax(1) >= 1e-4)]
            if not active.numel():
                break
            at = first[block[active]][:, None] + k + torch.arange(run, device=rec.device)
            real = at < last[block[active]][:, None]
            which = pairs[at.clamp(max=pairs.numel() - 1)]
            limit = torch.where(real, cutoff[which], torch.full_like(cutoff[which], -1.0))
            began = light[active]
            added, after, weight, through = _chunk(rec[which], limit, xy[active], began)
            if threshold:
                reached = (weight > 0) & (1.0 - through[:, 1:] >= 0.5)
                z = torch.where(reached.any(1), rec[which][:, :, 2].gather(1, reached.double().argmax(1)),
                                torch.full_like(began, -1.0))
                crossed[active] = torch.where(crossed[active] < 0, z, crossed[active])
            total[active] += added
            light[active] = after
            if adjoint is not None:
                steps.append((active, which, limit, began))
            k += run
        pixel = (py * width + px)[inside]
        cover = torch.where(inside, 1.0 - light, torch.zeros_like(light))
        colour[pixel] = torch.cat([total[..., :3], cover[..., None]], 2)[inside]
        mean = torch.where(cover > 1e-6, total[..., 3] / cover.clamp(min=1e-6), torch.zeros_like(cover))
        depth[pixel] = (crossed.clamp(min=0.0) if threshold else mean)[inside]
        if adjoint is not None:
            kept.append((steps, xy, inside, (py * width + px).clamp(max=width * height - 1), cover, mean))
    if adjoint is None:
        return colour, depth
    d_colour, d_depth = adjoint(colour, depth)
    d_rec = torch.zeros_like(rec)
    for steps, xy, inside, pixel, cover, mean in kept:
        ok = inside & (cover > 1e-6)
        d_sum = torch.where(ok, d_depth[pixel] / cover.clamp(min=1e-6), torch.zeros_like(cover))
        d_added = torch.cat([d_colour[pixel][..., :3] * inside[..., None], d_sum[..., None]], 2)
        d_light = torch.where(inside, -d_colour[pixel][..., 3], torch.zeros_like(cover)) + d_sum * mean
        for active, which, limit, began in reversed(steps):
            with torch.enable_grad():
                rows, light = rec[which].requires_grad_(), began.clone().requires_grad_()
                added, after = _chunk(rows, limit, xy[active], light)[:2]
                f = (added * d_added[active]).sum() + (after * d_light[active]).sum()
                d_rows, d_began = torch.autograd.grad(f, (rows, light))
            d_rec.index_add_(0, which.reshape(-1), d_rows.reshape(-1, rec.shape[1]))
            d_light[active] = d_began
    return colour, depth, d_rec


def _world(depth, proj, width, height):
    """The P layer: each pixel's world position from its depth."""
    at = torch.arange(width * height, device=depth.device)
    x, y = (at % width).double() + 0.5, (at // width).double() + 0.5
    f = [float(np.float32(v)) for v in (proj.centre_x, proj.focal_x, proj.centre_y, proj.focal_y)]
    v = torch.stack([(x - f[0]) / f[1] * depth, (y - f[2]) / f[3] * depth, depth, torch.ones_like(depth)], 1)
    m = torch.from_numpy(np.linalg.inv(_matrix(proj.world_to_view)).astype(np.float32).astype(np.float64)).cuda()
    return torch.where((depth > 0)[:, None], v @ m.T, torch.zeros_like(v))


def _l2(colour, target):
    error = colour[:, :3] - target
    scale = 1.0 / (3.0 * colour.shape[0])
    return error.square().sum() * scale, torch.cat([2.0 * scale * error, torch.zeros_like(error[:, :1])], 1)


def _exact_view(leaves, proj, w, h, target, d_depth):
    """One view's colour, depth, loss and gradients with respect to `leaves` (means, scales, quats, sh)."""
    with torch.enable_grad():
        rec, cutoff = _project(_trained(*leaves), proj, w, h, np.eye(4))
    said = {}

    def adjoint(colour, depth):
        said["loss"], d = _l2(colour, target)
        return d, d_depth if d_depth is not None else torch.zeros_like(depth)

    colour, depth, d_rec = _walk(rec.detach(), cutoff.detach(), w, h, adjoint)
    drawn = (cutoff.detach() >= 0)[:, None]
    grads = torch.autograd.grad(rec, leaves, torch.where(drawn, d_rec, torch.zeros_like(d_rec)))
    return colour, depth, said["loss"], grads


@torch.no_grad()
def exact(case, seed):
    kind = case["kind"]
    if kind == "sort":
        return None   # nothing computed: the pairs' order is whole or wrong
    if kind == "decode":
        g = _file(case, seed)
        good = ~torch.isnan(g["means"]).any(1) & (g["logits"] > -7.0)
        positions = torch.cat([g["means"].double(), torch.sigmoid(g["logits"].double())[:, None]], 1)[good]
        return dict(count=None, positions=positions, shape=None, sh=None)
    if kind == "frame":
        w, h = case["width"], case["height"]
        proj = A.pinhole_for_vertical_fov(_eye(0, 7, seed), (0, 0, 0), w, h, 60.0).projection_for(w, h)
        parts = []
        for c, (count, placed) in enumerate(_sections(case)):
            cloud = _decoded(_gaussians(count, case["clustered"], case["degree"], seed + 1000 * c))
            parts.append(_project(cloud, proj, w, h, placed))
        rec, cutoff = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        colour, depth = _walk(rec, cutoff, w, h, threshold=case["threshold"])
        out = dict(colour=colour, depth=depth)
        if case["extra"] == "matte":
            out.update(position=_world(depth, proj, w, h), ids=None, coverage=None)
        elif case["extra"] == "weights":
            out["weights"] = None
        return out
    g = _gaussians(case["count"], case["clustered"], case["degree"], seed)
    p = _training(g)
    if kind == "train":
        w, h = case["width"], case["height"]
        proj = A.pinhole_for_vertical_fov(_eye(0, 7, seed), (0, 0, 0), w, h, 60.0).projection_for(w, h)
        leaves = [t.double().requires_grad_() for t in (p.means, p.scales, p.quats, p.sh)]
        d_depth = _random((w * h,), seed + 1, 1.0 / (w * h)).double() if case["depth_loss"] else None
        colour, depth, loss, grads = _exact_view(leaves, proj, w, h, _random((w * h, 3), seed).double(), d_depth)
        return dict(colour=colour, depth=depth, loss=loss.reshape(1), means=grads[0], scales=grads[1], quats=grads[2],
                    sh=grads[3])
    # the mixed layout: SH DC and band 1 in BF16, bands 2 and 3 in e4m3 over a scale a Gaussian
    sh = torch.zeros((case["count"], 48), device="cuda")
    sh[:, :p.sh.shape[1]] = p.sh
    scale = sh[:, 12:].abs().amax(1, keepdim=True) / 448.0
    scale = torch.where(scale > 0, scale, torch.ones_like(scale))
    high = (sh[:, 12:] * (1.0 / scale)).to(torch.float8_e4m3fn).float() * scale
    sh = torch.cat([sh[:, :12].bfloat16().float(), high], 1)[:, :p.sh.shape[1]]
    views = _views(case, seed)
    leaves = [t.double() for t in (p.means, p.scales, p.quats, sh)]
    if kind == "views":
        cloud = _trained(*leaves)
        drawn = [_walk(*_project(cloud, proj, w, h, np.eye(4)), w, h) for proj, w, h in views]
        return dict(colour=torch.cat([d[0] for d in drawn]), depth=torch.cat([d[1] for d in drawn]))
    leaves = [t.requires_grad_() for t in leaves]
    target = _random((sum(w * h for _, w, h in views), 3), seed).double()
    colours, loss, sums, first = [], 0.0, None, 0
    for proj, w, h in views:
        colour, _, one, grads = _exact_view(leaves, proj, w, h, target[first:first + w * h], None)
        first += w * h
        colours.append(colour)
        loss = loss + one
        sums = grads if sums is None else [a + b for a, b in zip(sums, grads)]
    d_sh = torch.zeros((case["count"], 48), dtype=torch.float64, device="cuda")
    d_sh[:, :sums[3].shape[1]] = sums[3]
    return dict(colour=torch.cat(colours), loss=loss.reshape(1), means=sums[0], scales=sums[1], quats=sums[2], sh=d_sh)
