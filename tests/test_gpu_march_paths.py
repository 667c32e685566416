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
