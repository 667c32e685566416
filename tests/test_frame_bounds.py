"""Scenes just inside and just beyond each bound under which the raymarch drops the
special cases of its arithmetic: on which side the host puts each one (CPU), and that
the frames are the oracle's and the checked kernel's bits on both sides (GB300)."""
import ctypes as C
import math
import subprocess

import pytest

from meteoros_gb300 import abi, build, scenes
from tests.gpu_util import assert_bits_equal

W, H = 64, 36
FAR = 2.0**30

SOURCE = r"""
#include "mt_kernels.h"
using namespace mt;
extern "C" __attribute__((visibility("default"))) int frame_tame(const mt_params* p, const mt_camera_ubo* cam,
                                                                 const mt_time_ubo* tm) {
    float jitter[16][3];
    make_march_jitter(jitter, *tm);
    Frame f;
    make_march_frame(&f, *p, *cam, *tm, jitter);
    return f.tame;
}
"""


@pytest.fixture(scope="module")
def frame_tame(tmp_path_factory):
    folder = tmp_path_factory.mktemp("frame_bounds")
    (folder / "tame.cpp").write_text(SOURCE)
    lib = folder / "tame.so"
    subprocess.run([build.nvcc(), *build.COMMON, *build.UNITS["mt_consts.cpp"], f"-I{build.CSRC}", "-shared", "-o",
                    str(lib), str(folder / "tame.cpp"), str(build.CSRC / "mt_consts.cpp")], check=True, capture_output=True)
    return C.CDLL(str(lib)).frame_tame


def set_eye(cam, params, x, y, z):
    cam.eye[0], cam.eye[1], cam.eye[2] = (params.eye_sign * v for v in (x, y, z))


def planet(params, r, inner, outer):
    params.earth_radius, params.shell_inner_radius, params.shell_outer_radius = r, inner, outer


# name: (inside, beyond) the bound
BOUNDS = {
    "eye to the side": (6.14e6, 6.23e6),
    "eye to the far corner": (4.34e6, 4.41e6),
    "planet": (7.62e6, 7.63e6),
    "small planet": (2.0**-9, 0.9 * 2.0**-10),
    "thin shell": (0.0015, 0.0007),
    "eye below ground": (-0.499, -0.501),
    "wind": (0.999 * FAR, 1.001 * FAR),
    "cloud top": (0.999 * FAR, 1.001 * FAR),
    "jitter": (3.74, 3.76),
    "fine noise": (1.01 * 2.0**-20, 0.99 * 2.0**-20),
    "coarse noise": (0.999 * FAR, 1.001 * FAR),
    "fine weather": (1.01 * 2.0**-20, 0.99 * 2.0**-20),
    "coarse weather": (0.999 * FAR, 1.001 * FAR),
    "little coverage": (2.0**-29, 2.0**-31),
    "much coverage": (2.0**29, 2.0**31),
}


def scene(name, preset, value):
    cam, tm, params, _ = scenes.config_view(3, W, H)
    if preset == "reference":
        cam, tm, params = scenes.reference_frame(W, H, 25.0, 3, 1.0)
    if name == "eye to the side":
        set_eye(cam, params, value, 100.0, 0.0)
    elif name == "eye to the far corner":
        set_eye(cam, params, value, 100.0, value)
    elif name == "planet":
        planet(params, value, value + 1500.0, value + 4000.0)
    elif name == "small planet":
        planet(params, value, value + 0.5, value + 0.6)
    elif name == "thin shell":
        planet(params, 1.0, 1.25, 1.25 + value)
        set_eye(cam, params, 0.0, 0.1, 0.0)
    elif name == "eye below ground":
        set_eye(cam, params, 0.0, value * params.earth_radius, 0.0)
    elif name == "wind":
        params.wind_dir[0], params.wind_dir[1], params.wind_dir[2] = 0.0, 0.6, 0.8
        params.wind_speed, tm.time[1] = value, 1.0
    elif name == "cloud top":
        params.skew_dir[0], params.skew_dir[1], params.skew_dir[2] = 0.6, 0.0, 0.8
        params.cloud_top_offset = value
    elif name == "jitter":
        tm.halton_seq1[0], tm.halton_seq2[0] = value, -value
    elif name.endswith("noise"):
        params.noise_period = value
    elif name.endswith("weather"):
        params.coverage_mode, params.weather_scale = 1, value
    elif name.endswith("coverage"):
        params.coverage_mode, params.coverage = 0, value
    return cam, tm, params


CASES = [(name, preset, side) for name in BOUNDS for preset in ("config", "reference") for side in (0, 1)]


@pytest.mark.parametrize("name,preset,side", CASES)
def test_side_of_the_bound(frame_tame, name, preset, side):
    cam, tm, params = scene(name, preset, BOUNDS[name][side])
    assert frame_tame(C.byref(params), C.byref(cam), C.byref(tm)) == 1 - side


@pytest.mark.parametrize("field", ["wind_speed", "cloud_top_offset", "noise_period", "weather_scale", "eye"])
@pytest.mark.parametrize("value", [math.nan, math.inf])
def test_values_out_of_every_bound(frame_tame, field, value):
    cam, tm, params, _ = scenes.config_view(3, W, H)
    tm.time[1] = 1.0
    if field == "eye":
        cam.eye[2] = value
    else:
        setattr(params, field, value)
    assert frame_tame(C.byref(params), C.byref(cam), C.byref(tm)) == 0


@pytest.fixture(scope="module")
def ctx(lib):
    from meteoros_gb300.renderer import Context

    c = Context(0)
    c.generate_volumes(7)
    yield c
    c.close()


@pytest.mark.gpu
@pytest.mark.parametrize("name,preset,side", CASES)
def test_density_equals_oracle(ctx, oracle, vol7, name, preset, side):
    from tests.test_gpu_parity import gpu_render

    cam, tm, params = scene(name, preset, BOUNDS[name][side])
    _, want, cnt = oracle.render(vol7, cam, cam, tm, params, None, W, H, abi.MT_RENDER_FULL)
    _, got, st = gpu_render(ctx, cam, cam, tm, params, None, W, H, abi.MT_RENDER_FULL)
    assert_bits_equal(got, want, name)
    assert (st.primary_samples, st.light_samples, st.marched_rays) == tuple(int(c) for c in cnt[:3])


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [abi.MT_STORAGE_U8, abi.MT_STORAGE_F16, abi.MT_STORAGE_BF16])
@pytest.mark.parametrize("name,preset,side", CASES)
def test_unchecked_equals_checked(ctx, name, preset, side, storage):
    """The traced march always checks."""
    import torch

    cam, tm, params = scene(name, preset, BOUNDS[name][side])
    params.storage, params.fp64_shells = storage, int(storage != abi.MT_STORAGE_U8)
    trace = torch.zeros((H, W, 4), dtype=torch.int32, device="cuda")
    frames = []
    try:
        for lanes, traced in ((4, True), (1, False), (4, False), (0, False)):
            cur = torch.full((H, W, 4), float("nan"), device="cuda")
            mask = torch.full((H, W), float("nan"), device="cuda")
            ctx.set_tuning(march_lanes=lanes)
            ctx.set_sample_trace(trace if traced else None)
            ctx.render(cam, cam, tm, params, None, cur, mask, abi.MT_RENDER_FULL)
            frames.append((cur.cpu().numpy(), mask.cpu().numpy()))
    finally:
        ctx.set_sample_trace(None)
        ctx.set_tuning(march_lanes=0)
    for cur, mask in frames[1:]:
        assert_bits_equal(cur, frames[0][0], name)
        assert_bits_equal(mask, frames[0][1], name)
