"""The downstream and temporal passes' size-dependent forms against the oracle (GB300 only)."""
import numpy as np
import pytest

from meteoros_gb300 import abi, scenes
from tests.gpu_util import assert_bits_equal, to_dev
from tests.test_gpu_post import check_tonemap

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx(lib):
    from meteoros_gb300.renderer import Context

    c = Context(0)
    yield c
    c.close()


# The blur takes 1, 2 or 4 rows a thread by the image's size, and a loop without
# border checks where every tap lies inside: both sides of the size lines, images
# smaller than a tile, and suns at and beyond each edge.
@pytest.mark.parametrize("size", [(1, 1), (2, 3), (31, 5), (33, 17), (130, 67), (448, 446), (447, 448), (1700, 1058),
                                  (1700, 1059)])
@pytest.mark.parametrize("light", [(1.0, 1.0, 0.57, 1.0), (0.25, 0.75, 0.5, 1.0)])
def test_godray_forms_bit_exact(ctx, oracle, size, light):
    w, h = size
    rng = np.random.default_rng(w * 31 + h)
    mask = rng.random((h, w), dtype=np.float32) - np.float32(0.25)
    img = rng.random((h, w, 4), dtype=np.float32)
    for yaw, pitch in ((0.0, 10.0), (40.0, 60.0), (-75.0, 5.0)):
        cam = scenes.look((0.0, 0.0, 2.0), yaw, pitch, 45.0, w, h)
        out = torch.empty((h, w, 4), device="cuda")
        ctx.godrays(cam, light, to_dev(mask, torch), to_dev(img, torch), out)
        want = oracle.godrays(cam, np.array(light, np.float32), mask, img)
        assert_bits_equal(out.cpu().numpy(), want, f"{size} yaw {yaw}")
        same = to_dev(img, torch)  # in place
        ctx.godrays(cam, light, to_dev(mask, torch), same, same)
        assert_bits_equal(same.cpu().numpy(), want, f"{size} yaw {yaw} in place")


# The previous camera's uv checks three denominators instead of eleven quotients
# and takes the checked routine where one is out of range: cameras that look
# across and away from the shell hits, fields of view inside and outside the
# range, images without an interior for the history's filter.
@pytest.mark.parametrize("size", [(1, 1), (2, 2), (5, 3), (66, 37)])
@pytest.mark.parametrize("case", ["turned", "across", "away", "up", "narrow", "narrowest", "wide", "widest"])
def test_previous_uv_forms_bit_exact(vctx, oracle, vol7, size, case):
    w, h = size
    yaw, pitch, tan = {"turned": (1.5, 15.0, None), "across": (90.0, 0.0, None), "away": (180.0, -15.0, None),
                       "up": (0.0, 89.9, None), "narrow": (0.5, 15.0, 2.0**-29), "narrowest": (0.5, 15.0, 2.0**-31),
                       "wide": (0.5, 15.0, 2.0**29), "widest": (0.5, 15.0, 2.0**31)}[case]
    cam = scenes.look((0.0, 100.0, 0.0), 0.0, 15.0, 60.0, w, h)
    old = scenes.look((0.0, 100.0, 0.0), yaw, pitch, 60.0, w, h)
    if tan is not None:
        cam.tan_fov_by_2[0], cam.tan_fov_by_2[1] = tan, tan
    _, tm, params, _ = scenes.config_view(2, w, h)
    tm.frame_count_mod16 = 7
    rng = np.random.default_rng(w + h)
    prev, hist = (rng.random((h, w, 4), dtype=np.float32) for _ in range(2))
    want, wmask, _ = oracle.render(vol7, cam, old, tm, params, prev, w, h, 0)
    cur = torch.zeros((h, w, 4), device="cuda")
    vctx.render(cam, old, tm, params, to_dev(prev, torch), cur)
    repro = np.isnan(wmask)  # not marched
    got = cur.cpu().numpy()
    assert_bits_equal(got[repro], want[repro], "reprojected")
    out = torch.zeros((h, w, 4), device="cuda")
    vctx.txaa(cam, old, tm, params, cur, to_dev(hist, torch), out)
    assert_bits_equal(out.cpu().numpy(), oracle.txaa(cam, old, tm, params, got, hist), "txaa")
    frame, resolved = torch.zeros_like(cur), torch.zeros_like(cur)
    vctx.render_frame(cam, old, tm, params, to_dev(prev, torch), frame, to_dev(hist, torch), resolved)
    assert_bits_equal(frame.cpu().numpy(), got, "frame")
    assert_bits_equal(resolved.cpu().numpy(), out.cpu().numpy(), "resolved")


@pytest.fixture(scope="module")
def vctx(lib):
    from meteoros_gb300.renderer import Context

    c = Context(0)
    c.generate_volumes(7)
    yield c
    c.close()


# The tone map takes 1, 2 or 4 rows a thread by the image's size, their columns and
# rows looked up apart: both sides of the size lines, images smaller than a tile.
@pytest.mark.parametrize("size", [(1, 1), (3, 70), (33, 17), (448, 446), (447, 448), (1700, 1058), (1700, 1059)])
def test_tonemap_forms_vs_oracle(ctx, oracle, size):
    w, h = size
    rng = np.random.default_rng(w * 31 + h)
    img = rng.random((h, w, 4), dtype=np.float32) * np.float32(3.0)
    tm = abi.time_init()
    tm.time[1] = 2.5
    check_tonemap(ctx, oracle, tm, img, f"{size}")
