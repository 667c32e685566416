"""Frames beyond the bounds of the unchecked arithmetic at every lane count, alone
and beside others in a batch (GB300 only)."""
import pytest

from meteoros_gb300 import abi, scenes
from tests.gpu_util import assert_bits_equal
from tests.test_gpu_march_paths import scene
from tests.test_gpu_parity import gpu_render

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

STORAGES = [abi.MT_STORAGE_U8, abi.MT_STORAGE_F16, abi.MT_STORAGE_BF16]
# rays that take 32, 16, 8, 4, 2 and 1 lanes each when the choice is left open
SIZES = [(64, 36), (130, 100), (250, 200), (400, 300), (600, 500), (700, 650)]


@pytest.fixture(scope="module")
def ctx(lib):
    from meteoros_gb300.renderer import Context

    c = Context(0)
    c.generate_volumes(7)
    yield c
    c.close()


@pytest.fixture(autouse=True)
def tuning(ctx):
    yield
    ctx.set_tuning(march_lanes=0, batch_lanes=0, batch_tile=(16, 8), batch_direct=False)


def counts(st):
    return st.primary_samples, st.light_samples, st.marched_rays, st.pixels


@pytest.mark.parametrize("lanes", [1, 4, 8, 16])
@pytest.mark.parametrize("name", ["storm", "jitter", "beyond"])
def test_asked_lanes_equal_oracle(ctx, oracle, vol7, name, lanes):
    cam, tm, params = scene(name)
    _, want, cnt = oracle.render(vol7, cam, cam, tm, params, None, 64, 36, abi.MT_RENDER_FULL)
    ctx.set_tuning(march_lanes=lanes)
    _, got, st = gpu_render(ctx, cam, cam, tm, params, None, 64, 36, abi.MT_RENDER_FULL)
    assert_bits_equal(got, want, name)
    assert counts(st)[:3] == tuple(int(c) for c in cnt[:3])


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("size", SIZES)
def test_lanes_by_size_give_one_frame(ctx, size, storage):
    w, h = size
    cam, tm, params = scene("storm")
    params.storage, params.fp64_shells = storage, int(storage != abi.MT_STORAGE_U8)
    frames = []
    for lanes in (1, 0):
        ctx.set_tuning(march_lanes=lanes)
        frames.append(gpu_render(ctx, cam, cam, tm, params, None, w, h, abi.MT_RENDER_FULL))
    (a, am, sa), (b, bm, sb) = frames
    assert_bits_equal(b, a, "rgba")
    assert_bits_equal(bm, am, "mask")
    assert counts(sa) == counts(sb)


@pytest.mark.parametrize("storage", STORAGES)
@pytest.mark.parametrize("names", [("storm",), ("config", "jitter", "config")])
@pytest.mark.parametrize("size", SIZES)
def test_batches_with_general_frames_equal_renders(ctx, size, names, storage):
    """One such view takes a whole batch to the checked kernels."""
    w, h = size[0], (size[1] + len(names) - 1) // len(names)
    views, images = [], []
    for i, name in enumerate(names):
        cam, tm, params = scene(name)
        params.storage, params.fp64_shells = storage, int(storage != abi.MT_STORAGE_U8)
        want = torch.full((h, w, 4), float("nan"), device="cuda")
        got = torch.full_like(want, float("nan"))
        flags = abi.MT_RENDER_FULL | abi.MT_RENDER_COUNT
        ctx.render(cam, cam, tm, params, None, want, None, flags)
        views.append(scenes.make_view(cam, cam, tm, params, got, None, None, flags))
        images.append((want, got))
    a = ctx.stats(reset=True)
    for tuning in ({}, {"batch_lanes": 4}, {"batch_lanes": 16, "batch_direct": True}):
        ctx.set_tuning(**tuning)
        for _, got in images:
            got.fill_(float("nan"))
        ctx.render_batch(views)
        b = ctx.stats(reset=True)
        for want, got in images:
            assert_bits_equal(got.cpu().numpy(), want.cpu().numpy(), f"{names} {tuning}")
        assert counts(a) == counts(b)
