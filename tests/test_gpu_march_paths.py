"""The raymarch's shortcuts against the oracle, where they can go wrong (GB300 only)."""
import numpy as np
import pytest

from meteoros_gb300 import abi, scenes
from tests.gpu_util import assert_bits_equal
from tests.test_gpu_parity import gpu_render

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

W, H = 64, 36


@pytest.fixture(scope="module")
def ctx(lib):
    from meteoros_gb300.renderer import Context

    c = Context(0)
    c.generate_volumes(7)
    yield c
    c.close()


def check_density(oracle, vol, ctx, params, cam, tm):
    """The density path alone: god-ray values bit for bit, counters exact."""
    _, want, cnt = oracle.render(vol, cam, cam, tm, params, None, W, H, abi.MT_RENDER_FULL)
    _, got, st = gpu_render(ctx, cam, cam, tm, params, None, W, H, abi.MT_RENDER_FULL)
    assert_bits_equal(got, want, "mask")
    assert (st.primary_samples, st.light_samples, st.marched_rays) == tuple(int(c) for c in cnt[:3])


@pytest.mark.parametrize("height_gradient", [0, 1])
@pytest.mark.parametrize("coverage", [-0.25, 0.0, 0.3, 0.6, 0.999, 1.0, 1.5])
def test_empty_step_rules_constant_coverage(ctx, oracle, vol7, coverage, height_gradient):
    """Steps are empty where the height gradient does not exceed the coverage
    threshold; thresholds at and beyond the ends of [0, 1] keep the shader's outcome."""
    cam, tm, params, _ = scenes.config_view(3, W, H)
    params.coverage_mode, params.coverage, params.height_gradient = 0, coverage, height_gradient
    check_density(oracle, vol7, ctx, params, cam, tm)


@pytest.mark.parametrize("kind", ["clear", "overcast", "binary", "faint"])
def test_empty_step_rules_weather_extremes(ctx, oracle, volumes_seed7, kind):
    """Weather maps whose thresholds are 0, 1 or a rounding away from 1."""
    w = np.array(volumes_seed7["weather"])
    rng = np.random.default_rng(5)
    if kind == "binary":
        w[..., 0] = rng.integers(0, 2, w.shape[:2]) * 255
    elif kind == "faint":
        w[..., 0] = rng.integers(0, 50, w.shape[:2]) == 0
    else:
        w[..., 0] = 255 if kind == "overcast" else 0
    ctx.upload_weather(9, w)
    v = volumes_seed7
    vol = oracle.Volumes(v["base"], v["detail"], v["curl"], w)
    cam, tm, params, _ = scenes.config_view(4, W, H)
    params.weather_slot = 9
    check_density(oracle, vol, ctx, params, cam, tm)


@pytest.fixture(scope="module")
def trace_buffer():
    return torch.zeros((H, W, 4), dtype=torch.int32, device="cuda")


def scene(name):
    cam, tm, params, _ = scenes.config_view(3, W, H)
    if name == "reference":
        cam, tm, params = scenes.reference_frame(W, H, 9.0, 3, 1.0)
    elif name == "axis":  # rays in the x = 0 plane: quotients of exact zeros
        cam = scenes.look((0.0, 100.0, 0.0), 0.0, 20.0, 60.0, W, H)
        for seq in (tm.halton_seq1, tm.halton_seq2, tm.halton_seq3, tm.halton_seq4):
            seq[:] = [0.0] * 4
    elif name == "far eye":  # just inside the bound on lengths, and beyond it
        cam.eye[0], cam.eye[2] = 0.9e9, 0.3e9
    elif name == "beyond":
        cam.eye[0] = 4.0e9
    elif name == "small scales":
        params.noise_period, params.weather_scale = 2.0 ** -19, 2.0 ** -19
    elif name == "still air":
        params.wind_speed, params.cloud_top_offset = 0.0, 0.0
    elif name == "storm":  # beyond the bound on the wind's offset
        params.wind_speed, tm.time[1] = 1.0e9, 1.0e3
    elif name == "jitter":  # beyond the bound on the steps' jitter
        tm.halton_seq1[0], tm.halton_seq2[1] = 6.0, -6.0
    return cam, tm, params


SCENES = ["config", "reference", "axis", "far eye", "beyond", "small scales", "still air", "storm", "jitter"]


@pytest.mark.parametrize("storage", [abi.MT_STORAGE_U8, abi.MT_STORAGE_F16, abi.MT_STORAGE_BF16])
@pytest.mark.parametrize("name", SCENES)
def test_unchecked_quotients_equal_checked(ctx, trace_buffer, name, storage):
    """Frames whose scene bounds every quotient march without range checks;
    a traced render always checks.  Both give the same bits, on either side
    of the bounds, one view at a time and in a batch."""
    cam, tm, params = scene(name)
    params.storage, params.fp64_shells = storage, int(storage != abi.MT_STORAGE_U8)
    frames = []
    for lanes, traced in ((1, True), (1, False), (4, True), (4, False)):
        cur = torch.full((H, W, 4), float("nan"), device="cuda")
        mask = torch.full((H, W), float("nan"), device="cuda")
        ctx.set_tuning(march_lanes=lanes)
        ctx.set_sample_trace(trace_buffer if traced else None)
        ctx.render(cam, cam, tm, params, None, cur, mask, abi.MT_RENDER_FULL)
        frames.append((cur, mask))
    ctx.set_sample_trace(None)
    ctx.set_tuning(march_lanes=0)
    cur, mask = torch.zeros((H, W, 4), device="cuda"), torch.zeros((H, W), device="cuda")
    ctx.render_batch([scenes.make_view(cam, cam, tm, params, cur, None, mask, abi.MT_RENDER_FULL)])
    frames.append((cur, mask))
    torch.cuda.synchronize()
    for cur, mask in frames[1:]:
        assert_bits_equal(cur.cpu().numpy(), frames[0][0].cpu().numpy(), name)
        assert_bits_equal(mask.cpu().numpy(), frames[0][1].cpu().numpy(), name)


@pytest.mark.parametrize("name", ["axis", "still air", "small scales", "jitter"])
def test_quotient_edges_equal_oracle(ctx, oracle, vol7, name):
    cam, tm, params = scene(name)
    check_density(oracle, vol7, ctx, params, cam, tm)


@pytest.mark.parametrize("size", [(16, 8), (90, 91), (91, 91), (167, 168), (300, 300), (300, 301), (458, 459), (670, 672),
                                  (671, 671)])
def test_lane_counts_by_size_give_one_frame(ctx, size):
    """The lanes per ray follow the ray count; each line's two sides, marched
    as chosen and at one lane, counters included."""
    w, h = size
    cam, tm, params, _ = scenes.config_view(5, w, h)
    frames = []
    for lanes in (0, 1):
        ctx.set_tuning(march_lanes=lanes)
        frames.append(gpu_render(ctx, cam, cam, tm, params, None, w, h, abi.MT_RENDER_FULL))
    ctx.set_tuning(march_lanes=0)
    (a, am, sa), (b, bm, sb) = frames
    assert_bits_equal(a, b, "rgba")
    assert_bits_equal(am, bm, "mask")
    assert (sa.primary_samples, sa.light_samples, sa.marched_rays, sa.pixels) == \
        (sb.primary_samples, sb.light_samples, sb.marched_rays, sb.pixels)


@pytest.mark.parametrize("limit", [0.99, 0.3, 0.0, -1.0])
@pytest.mark.parametrize("lanes", [0, 1, 4, 8, 16])
def test_early_exit_at_every_limit(ctx, oracle, vol7, lanes, limit):
    """A limit at or below 0 ends a ray after its first step, in cloud or not."""
    cam, tm, params, _ = scenes.config_view(3, W, H)
    params.accum_limit = limit
    ctx.set_tuning(march_lanes=lanes)
    check_density(oracle, vol7, ctx, params, cam, tm)
    ctx.set_tuning(march_lanes=0)


@pytest.mark.parametrize("coverage", [2.0**-29, 2.0**-31, 1.0 - 2.0**-24, 2.0**29, 2.0**31, -2.0**20])
def test_coverage_bounds_equal_oracle(ctx, oracle, vol7, coverage):
    """Constant coverages on either side of the bounds under which the density
    path drops its special cases."""
    cam, tm, params, _ = scenes.config_view(3, W, H)
    params.coverage_mode, params.coverage, params.height_gradient = 0, coverage, 1
    check_density(oracle, vol7, ctx, params, cam, tm)


@pytest.mark.parametrize("size", [(1, 1), (7, 3), (8, 4), (9, 5), (65, 37), (130, 18)])
def test_warp_tiles_march_every_ray_once(ctx, oracle, vol7, size):
    """One-lane warps take 8x4 rays: grids smaller than a tile, whole tiles and one
    ray more, either row order, every CTA size, full and checkerboard, against the
    oracle's god-ray values and counters."""
    w, h = size
    cam, tm, params, _ = scenes.config_view(5, w, h)
    prev = np.random.default_rng(w).random((h, w, 4), dtype=np.float32)
    for flags in (abi.MT_RENDER_FULL, 0):
        _, want, cnt = oracle.render(vol7, cam, cam, tm, params, prev, w, h, flags)
        for order, block in ((0, 0), (1, 128), (0, 32)):
            ctx.set_tuning(march_lanes=1, march_order=order, march_block=block)
            try:
                _, got, st = gpu_render(ctx, cam, cam, tm, params, prev, w, h, flags)
            finally:
                ctx.set_tuning(march_lanes=0, march_order=0, march_block=0)
            assert_bits_equal(got, want, f"{size} flags {flags} order {order} block {block}")
            assert (st.primary_samples, st.light_samples, st.marched_rays) == tuple(int(c) for c in cnt[:3])
