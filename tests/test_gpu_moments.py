"""The adjoints' sums over a footprint's pixels, held to 64 bits axis by axis. The Gaussians stand apart, a pixel or
so wide, anywhere against the pixels and the boxes a warp sums: their moments in x and in y are the same sums of the
same terms, so they are to be equally exact, whatever rows or columns a kernel takes them over. Half as much again
is allowed for chance (some 400 Gaussians and more, each a term)."""
import ctypes as C

import numpy as np
import pytest
import torch

import athenea_b200 as A
from athenea_b200 import _native as N
from athenea_b200.raster import BatchTrainer, MixedParams
from perf import cases
from tests.gpu_helpers import fetch

pytestmark = pytest.mark.gpu

FAINT = 1.0 / 255.0


def _apart(W, H, sigma, seed, exact=False):
    """Gaussians of `sigma` pixels on a grid 16 pixels apart, each moved by up to 8; `exact`: by 16ths of a pixel,
    before a camera of powers of two, whose projection rounds no centre."""
    away, focal = (4.0, 256.0) if exact else (3.0, None)
    cam = A.pinhole_for_vertical_fov((0, 0, away), (0, 0, 0), W, H, 60.0).projection_for(W, H)
    if exact:
        cam.focal_x = cam.focal_y = focal
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rand = lambda *s: torch.rand(s, generator=gen, device="cuda")  # noqa: E731
    x, y = torch.meshgrid(torch.arange(16, W - 15, 16, device="cuda"), torch.arange(16, H - 15, 16, device="cuda"),
                          indexing="ij")
    at = torch.stack([x.reshape(-1) - W / 2, y.reshape(-1) - H / 2], 1) + 8.0 * rand(x.numel(), 2)
    if exact:
        at = (at * 16.0).round() / 16.0
    n = at.shape[0]
    unit = away / cam.focal_x
    means = torch.cat([at * unit, torch.zeros((n, 1), device="cuda"), 2.0 * rand(n, 1) - 0.5], 1).contiguous()
    scales = torch.full((n, 4), float(np.log(sigma * unit)), device="cuda")
    quats = torch.zeros((n, 4), device="cuda")
    quats[:, 0] = 1.0
    sh = (rand(n, 3) * 2.0).bfloat16().float()   # as the mixed layout holds it
    return cam, A.Params(means, scales, quats, sh, 0)


# boxes of one pixel a lane and of two (from 2368 tiles on 148 SMs)
@pytest.mark.parametrize("size", [(320, 320), (1184, 528)])
def test_record_gradients_are_as_exact_in_y_as_in_x(native, size):
    W, H = size
    cam, P = _apart(W, H, 0.02, 7)   # the frame widens each to 0.55 pixels
    raster, t = A.TileRasterizer.create(), A.RenderTargets.make(W, H)
    raster.render_params(cam, P, A.RenderSettings(width=W, height=H, antialias=False), t)
    dl = torch.randn((W * H, 4), generator=torch.Generator(device="cuda").manual_seed(9), device="cuda")
    raster.backward(dl, P.zeros_like())
    b = N.FrameBuffers()
    N.check(N.lib().ath_raster_frame_buffers(raster._h, C.byref(b)))
    got = fetch(b.grads, (b.slots, 10), np.float32).astype(np.float64)
    rec = fetch(b.records, (b.slots, 12), np.float32).astype(np.float64)
    up = dl.cpu().numpy().astype(np.float64).reshape(H, W, 4)
    errors = {k: [] for k in ("cx", "cy", "a", "c")}
    for r, g in zip(rec, got):
        cx, cy, _, cutoff, a, b2, c, opacity = r[:8]
        x = np.arange(max(0, int(cx) - 8), min(W, int(cx) + 9))
        y = np.arange(max(0, int(cy) - 8), min(H, int(cy) + 9))
        dx, dy = np.meshgrid(x + 0.5 - cx, y + 0.5 - cy)
        power = a * dx * dx + 2.0 * b2 * dx * dy + c * dy * dy
        alpha = opacity * np.exp(-0.5 * power)
        if np.any(np.abs(power - cutoff) < 1e-4) or np.any(np.abs(alpha - FAINT) < 1e-6):
            continue   # a pixel at the footprint's edge
        on = (power <= cutoff) & (alpha >= FAINT)
        d = up[y[0]:y[-1] + 1, x[0]:x[-1] + 1]
        # nothing else is in these pixels: dL/dalpha is the colour's change over the background of zeros
        term = np.where(on, alpha * (d[..., :3] @ r[8:11] + d[..., 3]), 0.0)
        for name, word, weight in (("cx", 0, a * dx + b2 * dy), ("cy", 1, b2 * dx + c * dy), ("a", 2, -0.5 * dx * dx),
                                   ("c", 4, -0.5 * dy * dy)):
            terms = term * weight
            errors[name].append((g[word] - terms.sum()) / np.abs(terms).sum())
    rms = {k: float(np.sqrt(np.mean(np.square(v)))) for k, v in errors.items()}
    print(size, len(errors["a"]), rms)
    assert len(errors["a"]) > 300
    assert rms["c"] <= 1.5 * rms["a"] and rms["cy"] <= 1.5 * rms["cx"], rms


@pytest.mark.parametrize("tile", [8, 16, 32])
def test_batched_gradients_are_as_exact_in_y_as_in_x(native, tile):
    W = H = 496
    cam, P = _apart(W, H, 0.45, 11, exact=True)   # 0.71 pixels as drawn
    M = MixedParams.from_params(P)
    b = BatchTrainer()
    b.set_views([(cam, W, H)])
    b.set_tuning(tile, 128)
    target = torch.rand((W * H, 3), generator=torch.Generator(device="cuda").manual_seed(13), device="cuda")
    grads = A.Params(*[torch.zeros_like(v) for v in (P.means, P.scales, P.quats)],
                     torch.zeros((P.count, 48), device="cuda"))
    b.step(M, target, torch.empty((W * H, 4), device="cuda"), torch.zeros(1, device="cuda"), grads)
    leaves = [v.double().requires_grad_() for v in (P.means, P.scales, P.quats, P.sh)]
    want = cases._exact_view(leaves, cam, W, H, target.double(), None)[3]
    # four Gaussians of five, so that the few with a pixel at the footprint's edge, in or out of the sum, do not count
    spread = lambda got, exact, k: float(((got[:, k] - exact[:, k]).abs() / exact[:, k].square().mean().sqrt()).quantile(0.8))  # noqa: E731
    found = [(name, *[spread(g.double(), w, k) for k in (0, 1)]) for name, g, w in (("means", grads.means, want[0]),
                                                                                    ("scales", grads.scales, want[1]))]
    print(tile, P.count, found)
    for name, x, y in found:
        assert y <= 1.5 * x, (name, x, y)
