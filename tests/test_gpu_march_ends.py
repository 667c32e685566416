"""Rays whose march ends before it begins, against the oracle (GB300 only)."""
import pytest

from meteoros_gb300 import abi, scenes
from tests.gpu_util import assert_bits_equal
from tests.test_gpu_parity import gpu_render

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

W, H = 64, 36


@pytest.mark.parametrize("lanes", [0, 1, 4, 8, 16])
@pytest.mark.parametrize("steps", [1, 3, 8, 17, 33])
@pytest.mark.parametrize("eye_x", [-4.0e5, 4.0e5])
@pytest.mark.parametrize("preset", ["config", "reference"])
def test_rays_toward_the_origin(lib, oracle, vol7, preset, eye_x, steps, lanes):
    """The march's bounds are distances from the origin, not from the eye: for an
    eye far to the side, rays toward the origin end nearer than they begin and
    march no step, however many lanes look ahead along them."""
    from meteoros_gb300.renderer import Context

    _, tm, params, _ = scenes.config_view(3, W, H)
    if preset == "reference":
        params = abi.params_reference()
    params.steps_min = params.steps_max = steps
    cam = scenes.look((eye_x, 100.0, 0.0), 90.0, 25.0, 60.0, W, H)
    _, want, cnt = oracle.render(vol7, cam, cam, tm, params, None, W, H, abi.MT_RENDER_FULL)
    with Context(0) as ctx:
        ctx.generate_volumes(7)
        ctx.set_tuning(march_lanes=lanes)
        _, got, st = gpu_render(ctx, cam, cam, tm, params, None, W, H, abi.MT_RENDER_FULL)
    assert_bits_equal(got, want, "mask")
    assert (st.primary_samples, st.light_samples, st.marched_rays) == tuple(int(c) for c in cnt[:3])
    reversed_rays = eye_x * params.eye_sign < 0  # the view looks along +x
    assert (st.primary_samples == 0) == reversed_rays
