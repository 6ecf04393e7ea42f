"""The paths a call takes by its sizes, alignment and options, at the sizes where they
change or leave remainders: boxes of one and of two pixels a lane, rects too large for a
mask, sorts in one block and in small and large tiles, decodes through shared memory and
not, gradient rows moved by 16 bytes and by values."""
import ctypes as C

import numpy as np
import pytest
import torch

import athenea_b200 as A
from athenea_b200 import _native as N
from athenea_b200 import scenes
from perf import cases
from tests.fixtures import CloudBuilder, random_cloud
from tests.gpu_helpers import frame_buffers, oracle_projection, upload
from tests.test_gpu_parity import _compare, _decode, _settings

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def raster(native):
    return A.TileRasterizer.create()


# On 148 SMs a frame takes boxes of one pixel a lane below 4736 tiles: (1184, 1008) is the last of them here,
# (1184, 1024) is past it; (1279, 719) leaves part of a box in both directions; (16, 16) is one tile, (3, 5) less than a box
@pytest.mark.parametrize("size", [(3, 5), (16, 16), (250, 190), (1279, 719), (1184, 1008), (1184, 1024)])
@pytest.mark.parametrize("threshold", [0, 1])
@pytest.mark.parametrize("opacity", [1.0, 6.0])
def test_frames_equal_the_restatement_to_the_bit(oracle, native, raster, size, opacity, threshold):
    """Footprints from a pixel to the whole image (rects of more than 64 tiles), with opacities over 1 (the harder
    kernel) by an edit, over a background, the depth layer in both modes."""
    W, H = size
    packed = _decode(oracle, random_cloud(900, 17 + W, min_size=0.002, max_size=1.5))
    cam = A.pinhole_for_vertical_fov((0.3, 0.2, 4.0), (0, 0, 0), W, H, 60.0)
    s = _settings(W, H, background=(0.1, 0.3, 0.2, 0.4), depth_mode=threshold)
    edit = A.SplatEdit(active=True, mode=2, size=(1.0, 2.0, 2.0), opacity=opacity) if opacity != 1.0 else None
    got, want = _compare(oracle, None, raster, [packed], [np.eye(4)], cam.projection_for(W, H), s, edit=edit)
    np.testing.assert_array_equal(got["colour"], want["colour"])
    np.testing.assert_array_equal(got["depth"], want["depth"])


# boxes of one pixel a lane and of two
@pytest.mark.parametrize("size", [(1184, 1008), (1185, 1025)])
@pytest.mark.parametrize("threshold", [0, 1])
def test_frames_over_a_layer_equal_the_restatement_to_the_bit(oracle, native, size, threshold):
    W, H = size
    packed = _decode(oracle, random_cloud(900, 5, min_size=0.002, max_size=1.5))
    cam = A.pinhole_for_vertical_fov((0.3, 0.2, 4.0), (0, 0, 0), W, H, 60.0).projection_for(W, H)
    s = _settings(W, H, background=(0.1, 0.3, 0.2, 0.4), depth_mode=threshold)
    drawn = oracle.render([(*packed, np.eye(4), 0)], oracle_projection(oracle, cam), W, H, bg=s.background, depth_mode=threshold)
    gen = torch.Generator().manual_seed(W)
    depth = 2.0 + torch.rand(W * H, generator=gen) * 5.0   # among the splats, from 2 to 6.5
    depth[torch.rand(W * H, generator=gen) < 0.2] = 0.0
    under, t = A.RenderTargets.make(W, H), A.RenderTargets.make(W, H)
    under.colour.copy_(torch.rand((W * H, 4), generator=gen).cuda())
    under.depth.copy_(depth.cuda())
    A.TileRasterizer.create().render(cam, [A.SplatInstance(upload(packed))], s, t, under=under)
    want = oracle.blend_over(drawn["frame"], drawn["binned"], drawn["proj"], under.colour.cpu().numpy(), depth.numpy())
    np.testing.assert_array_equal(t.colour.cpu().numpy(), want["colour"])
    np.testing.assert_array_equal(t.depth.cpu().numpy(), want["depth"])


def test_the_last_capacity_of_one_block_sorts_and_the_next_agree(oracle, native):
    """After release_scratch a frame's pairs have room for a seventh more than they are: 7168 pairs for 8192, which one
    block sorts, 7169 for 8193, which tiles do. The same frame by both, each splat inside a tile of its own."""
    W, H = 160, 128
    cam = A.pinhole_for_vertical_fov((0, 0, 3), (0, 0, 0), W, H, 60.0).projection_for(W, H)
    rng, b = np.random.default_rng(8), CloudBuilder()
    for _ in range(7169):
        z = rng.uniform(-0.3, 0.3)
        at = 16 * rng.integers(0, (W // 16, H // 16)) + 8 + rng.uniform(-3, 3, 2) - (W / 2, H / 2)
        x, y = at * (3.0 - z) / cam.focal_x
        b.add(x, y, z, 0.05, 1e-3, 1e-3, 1e-3, (1, 0, 0, 0), rng.uniform(0, 1, 3))
    more = _decode(oracle, b)
    less = tuple(a[:7168] for a in more[:3]) + more[3:]
    found = []
    for first, pairs in ((less, 7168), (more, 7169)):
        r, t = A.TileRasterizer.create(), A.RenderTargets.make(W, H)
        r.release_scratch()
        settings = A.RenderSettings(width=W, height=H, antialias=False)
        assert r.render(cam, [A.SplatInstance(upload(first))], settings, t).pairs == pairs
        r.render(cam, [A.SplatInstance(upload(less))], settings, t)
        found.append((t.colour.cpu().numpy(), t.depth.cpu().numpy(), frame_buffers(r)))
    for k in range(2):
        np.testing.assert_array_equal(found[0][k], found[1][k])
    for name in ("pair_keys", "pair_splats", "ranges"):
        np.testing.assert_array_equal(found[0][2][name], found[1][2][name], err_msg=name)


# one block up to 8192; 2048-key tiles up to 606,208; then tiles of 6144 (pairs)
@pytest.mark.parametrize("count", [2, 511, 513, 8191, 8192, 8193, 10_240, 606_208, 606_209, 700_001])
@pytest.mark.parametrize("bits", [1, 9, 12, 24, 37, 38, 45, 64])
def test_sorts_are_stable_at_every_tile_size(native, count, bits):
    gen = torch.Generator(device="cuda").manual_seed(count + bits)
    keys = (torch.randint(0, 1 << 32, (count,), generator=gen, device="cuda") << 32) | \
        torch.randint(0, 1 << 32, (count,), generator=gen, device="cuda")
    keys[::3] = keys[0].clone()   # ties
    values = torch.arange(count, dtype=torch.int32, device="cuda")
    k, v, k2, v2 = keys.clone(), values.clone(), torch.empty_like(keys), torch.empty_like(values)
    sorter = cases._Sorter()
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    N.check(N.lib().ath_sorter_sort(sorter.handle, ptr(k), ptr(v), ptr(k2), ptr(v2), count, bits,
                                    C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    N.check(N.lib().ath_sorter_check(sorter.handle))
    host = keys.cpu().numpy().view(np.uint64)
    order = np.argsort(host & np.uint64((1 << bits) - 1), kind="stable")   # the low bits alone
    np.testing.assert_array_equal(v.cpu().numpy().view(np.uint32), order.astype(np.uint32))
    np.testing.assert_array_equal(k.cpu().numpy().view(np.uint64), host[order])


# strides whose records' 16-byte pieces end in the middle, that fill shared memory, and that do not fit it;
# counts around a warp and a block
@pytest.mark.parametrize("pad,shift", [(0, 1), (1, 0), (2, 3), (330, 0), (600, 0)])
@pytest.mark.parametrize("count", [1, 31, 33, 128, 1291])
def test_decode_takes_any_stride_and_base(native, count, pad, shift):
    records, enc = cases._records(cases._file(dict(count=count, degree=3), 3))
    want = A.CloudLoader.upload(records, enc)
    stride = enc["stride"] + pad
    flat = torch.full((count * stride + shift,), 7.0, device="cuda")
    flat[shift:].view(count, stride)[:, :enc["stride"]] = records
    got = A.CloudLoader.upload(flat[shift:], dict(enc, stride=stride))
    assert got.count == want.count
    for name in ("positions", "shape", "sh"):
        assert torch.equal(getattr(got, name)[:want.count], getattr(want, name)[:want.count]), name


# A pixel whose walk takes a decision near its threshold (about 1 in 500) may take it the other way in 64 bits: a
# splat of alpha 1/255 in or out. Images then agree to 1/255 / sqrt(500) = 2e-4 of their norm, gradients, which such a
# splat's are few of but whole, to 1e-2.
@pytest.mark.parametrize("case", [
    dict(kind="train", count=3001, clustered=True, degree=0, width=97, height=61, depth_loss=True),
    dict(kind="train", count=2500, clustered=False, degree=1, width=480, height=480, depth_loss=False),
    dict(kind="train", count=4003, clustered=True, degree=2, width=640, height=361, depth_loss=True),
    dict(kind="train", count=4003, clustered=True, degree=3, width=1281, height=483, depth_loss=True),
    dict(kind="step", count=2000, clustered=True, degree=3, views=3, width=131, height=77, tile=8, batch=64),
    dict(kind="step", count=3000, clustered=True, degree=1, views=2, width=320, height=201, tile=16, batch=512),
    dict(kind="step", count=3000, clustered=True, degree=2, views=5, width=161, height=120, tile=32, batch=128),
    dict(kind="views", count=3000, clustered=False, degree=3, views=2, width=333, height=251, tile=32, batch=512),
    dict(kind="frame", count=3000, clustered=True, degree=2, width=801, height=433, clouds=5, extra="matte",
         threshold=False, wait=True),
], ids=lambda c: f"{c['kind']}-{c['width']}x{c['height']}-{c['degree']}")
def test_calls_agree_with_64_bits(native, case):
    got = cases.run(cases.prepare(case, 5))
    want = cases.exact(case, 5)
    for name, value in want.items():
        if value is None:
            continue
        g, w = got[name].double().reshape(-1), value.double().reshape(-1)
        rel = float((g - w).norm() / w.norm())
        assert rel <= (1e-3 if name in ("colour", "loss") else 1e-2), (name, rel)


# SH rows that are not whole 16-byte pieces (a stride of 49, a base 4 bytes off) take the values one at a time: the
# same gradients, to the order of the atomic sums
@pytest.mark.parametrize("stride,shift", [(48, 0), (49, 0), (48, 1), (52, 0)])
def test_gradients_do_not_depend_on_the_rows_layout(native, stride, shift):
    W, H, n = 320, 200, 5003
    p = scenes.params(n, True, 7, 3)
    base = A.Params(*[torch.from_numpy(np.ascontiguousarray(p[k])).cuda() for k in ("means", "scales", "quats", "sh")], 3)

    def rows(values):
        flat = torch.zeros(n * stride + shift, device="cuda")
        out = flat[shift:].view(n, stride)
        out[:, :48] = values
        return out

    def step(params, grads):
        r, t = A.TileRasterizer.create(), A.RenderTargets.make(W, H)
        cam = A.pinhole_for_vertical_fov((0, 0, 3), (0, 0, 0), W, H, 60.0).projection_for(W, H)
        r.render_params(cam, params, A.RenderSettings(width=W, height=H), t)
        r.backward(torch.ones_like(t.colour), grads)
        return t.colour

    want = base.zeros_like()
    image = step(base, want)
    mine = A.Params(base.means, base.scales, base.quats, rows(base.sh), 3)
    grads = A.Params(torch.zeros_like(base.means), torch.zeros_like(base.scales), torch.zeros_like(base.quats),
                     rows(torch.full((n, 48), 0.25, device="cuda")), 3)
    assert torch.equal(step(mine, grads), image)
    assert torch.allclose(grads.sh[:, :48] - 0.25, want.sh, rtol=1e-4, atol=1e-5 * float(want.sh.abs().max()))
    assert torch.equal(grads.sh[:, 48:], torch.zeros_like(grads.sh[:, 48:]))
    for name in ("means", "scales", "quats"):
        a, b = getattr(grads, name), getattr(want, name)
        assert torch.allclose(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max())), name


# less than a block, a block and a cluster of blocks with remainders, and past one pixel a thread of the whole grid
@pytest.mark.parametrize("pixels", [1, 255, 257, 2048, 2049, 303_104, 303_105, 921_600])
def test_the_l2_loss_at_every_size(native, pixels):
    """148 additions of 32 bits at most into the loss: 3e-7 of it where they round at random, 1e-6 allowed."""
    gen = torch.Generator(device="cuda").manual_seed(pixels)
    colour = torch.rand((pixels, 4), generator=gen, device="cuda")
    target = torch.rand((pixels, 3), generator=gen, device="cuda")
    dl, loss = torch.full_like(colour, 7.0), torch.full((1,), 0.5, device="cuda")
    A.l2_loss(colour, target, dl, loss)
    error = colour[:, :3].double() - target.double()
    want = 0.5 + float(error.square().mean())
    assert abs(loss.item() - want) <= 1e-6 * want
    assert float((dl[:, :3].double() - 2.0 * error / (3.0 * pixels)).abs().max()) <= 1e-6 / (3.0 * pixels)
    assert not bool(dl[:, 3].any())


# depth sorts in one block, in small tiles and in large ones; none, one and some of the slots in sight
@pytest.mark.parametrize("slots", [5000, 20_011, 700_003])
@pytest.mark.parametrize("seen", [0, 1, 257, 4000])
def test_a_cloud_mostly_out_of_sight_draws_as_what_is_in_sight(native, slots, seen):
    p = scenes.params(seen + 1, True, 21, 3)
    few = A.Params(*[torch.from_numpy(np.ascontiguousarray(p[k][:seen])).cuda() for k in ("means", "scales", "quats", "sh")], 3)
    gen = torch.Generator(device="cuda").manual_seed(slots)
    at = torch.randperm(slots, generator=gen, device="cuda")[:seen].sort().values   # in order: ties in depth keep it
    means = torch.zeros((slots, 4), device="cuda")
    means[:, 2] = 10.0   # behind the camera
    scales, quats = torch.full_like(means, -4.0), torch.ones_like(means)
    sh = torch.zeros((slots, few.sh.shape[1]), device="cuda")
    for whole, part in ((means, few.means), (scales, few.scales), (quats, few.quats), (sh, few.sh)):
        whole[at] = part
    W, H = 320, 200
    cam = A.pinhole_for_vertical_fov((0, 0, 3), (0, 0, 0), W, H, 60.0).projection_for(W, H)
    images, slot_of = [], []
    for cloud in (A.Params(means, scales, quats, sh, 3), few):
        r, t = A.TileRasterizer.create(), A.RenderTargets.make(W, H)
        for _ in range(2):   # sized by its own pairs, then as any later frame
            stats = r.render_params(cam, cloud, A.RenderSettings(width=W, height=H), t)
        images.append((t.colour.cpu(), t.depth.cpu()))
        slot_of.append(torch.from_numpy(frame_buffers(r)["pair_splats"].astype(np.int64)))
        assert stats.visible <= seen
    assert torch.equal(images[0][0], images[1][0]) and torch.equal(images[0][1], images[1][1])
    assert torch.equal(slot_of[0], at.cpu()[slot_of[1]])
