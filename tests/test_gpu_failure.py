"""Failure detection without a GPU fault: the device-memory budget (the
reference's ATHENEA_GPU_BUDGET, modules/gpu/src/Device.cpp:434-449) turning an
allocation into OutOfMemory on the host side, and the library's bounded
device-side wait running out on a flag nothing sets, with the context usable
after both."""
import functools

import numpy as np
import pytest
import torch

import athenea_b200 as A
from tests.fixtures import ENC_BUILDER, CloudBuilder, product_encoding
from tests.gpu_helpers import frame_buffers

pytestmark = pytest.mark.gpu


@functools.lru_cache
def _cloud(count=200, size=0.05):
    b = CloudBuilder()
    rng = np.random.default_rng(5)
    for _ in range(count):
        x, y, z = rng.uniform(-1, 1, 3)
        b.add(x, y, z, 0.8, size, size, size, (1, 0, 0, 0), tuple(rng.uniform(0, 1, 3)))
    recs = torch.from_numpy(b.records().reshape(-1)).cuda()
    return A.CloudLoader.upload(recs, product_encoding(ENC_BUILDER), 3)


def _frame(raster, cloud, W=256, H=192):
    s = A.RenderSettings(width=W, height=H)
    t = A.RenderTargets.make(W, H)
    raster.render(A.Camera.looking_at((0.0, 0.0, 4.0), (0, 0, 0)), [A.SplatInstance(cloud)], s, t)
    torch.cuda.synchronize()
    return t.colour.cpu().numpy()


def test_a_budget_turns_scratch_into_out_of_memory_and_release_gives_it_back(native):
    cloud = _cloud()
    want = _frame(A.TileRasterizer.create(), cloud)
    raster = A.TileRasterizer.create()
    import gc
    gc.collect()                                    # what earlier tests left is freed now, not mid-test
    held_before, _ = A.memory_held()
    try:
        A.set_memory_budget(1)                      # room for no new buffer, whatever is held
        assert A.memory_held()[1] == 1
        with pytest.raises(A.AtheneaError) as e:
            _frame(raster, cloud)
        assert e.value.code == 9                    # OutOfMemory
        A.set_memory_budget(0)
        got = _frame(raster, cloud)                 # the same rasteriser, usable again
        np.testing.assert_array_equal(got, want)
        held_after, budget = A.memory_held()
        assert budget == 0 and held_after > 0
        raster.release_scratch()
        assert A.memory_held()[0] < held_after
    finally:
        A.set_memory_budget(0)


# The budget admits a part of what a larger frame of the handle asks for, so that some of its buffers have grown when
# one cannot: the next frame, small enough for what the handle had, asks for all of them again.
@pytest.mark.parametrize("part", [0.02, 0.2, 0.5, 0.6, 0.75, 0.9])
def test_a_growth_that_fails_part_way_leaves_a_handle_that_draws(native, part):
    import gc
    small, large = _cloud(), _cloud(60_000, 0.02)
    want = _frame(A.TileRasterizer.create(), small)
    raster, other = A.TileRasterizer.create(), A.TileRasterizer.create()
    np.testing.assert_array_equal(_frame(raster, small), want)
    gc.collect()
    before = A.memory_held()[0]
    whole = _frame(other, large, 640, 480)
    need = A.memory_held()[0] - before
    del other
    gc.collect()
    try:
        A.set_memory_budget(A.memory_held()[0] + int(part * need))
        with pytest.raises(A.AtheneaError) as e:
            _frame(raster, large, 640, 480)
        assert e.value.code == 9                    # OutOfMemory
        A.set_memory_budget(0)
        np.testing.assert_array_equal(_frame(raster, small), want)
        np.testing.assert_array_equal(_frame(raster, large, 640, 480), whole)
    finally:
        A.set_memory_budget(0)


def test_a_failed_frame_leaves_nothing_to_inspect(native):
    small, large = _cloud(), _cloud(60_000, 0.02)
    raster = A.TileRasterizer.create()
    _frame(raster, small)
    want = frame_buffers(raster)
    try:
        A.set_memory_budget(1)
        with pytest.raises(A.AtheneaError) as e:
            _frame(raster, large, 640, 480)
        assert e.value.code == 9                    # OutOfMemory
        with pytest.raises(A.AtheneaError) as e:
            frame_buffers(raster)
        assert e.value.code == 2                    # NotFound
    finally:
        A.set_memory_budget(0)
    _frame(raster, small)
    for name, value in frame_buffers(raster).items():
        np.testing.assert_array_equal(value, want[name], err_msg=name)


def test_a_wait_on_a_flag_nothing_sets_gives_up_with_timeout(native):
    with pytest.raises(A.AtheneaError) as e:
        A.check_bounded_wait(0, 1000)
    assert e.value.code == 12                       # Timeout
    assert A.check_bounded_wait(1, 1000) == 0       # a set flag: no spin at all
    with pytest.raises(A.AtheneaError) as e:
        A.check_bounded_wait(1, 0)                  # a limit of none is refused
    assert e.value.code == 3
    # the context is still usable: a frame renders after the timeout
    assert _frame(A.TileRasterizer.create(), _cloud())[:, 3].max() > 0
