"""The lanes and tile a batch is marched with: as asked for, or by its rays."""
import subprocess

import pytest

from meteoros_gb300 import abi, build, scenes
from tests.gpu_util import assert_bits_equal

MAIN = r"""
#include <cstdio>
#include "mt_batch.h"
int main() {
    int lanes, w, h, texels16;
    long long rays;
    while (scanf("%d %d %d %lld %d", &lanes, &w, &h, &rays, &texels16) == 5) {
        const mt::BatchShape s = mt::batch_shape(lanes, w, h, mt::auto_lanes(rays, texels16 != 0));
        printf("%d %d %d\n", s.lanes, s.tile_w, s.tile_h);
    }
}
"""


def test_shape_rule(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "shape"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.CSRC}", str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    lines = {0: {32: 8192, 16: 28000, 8: 90000, 4: 210000, 2: 450000}, 1: {32: 7500, 16: 22000, 8: 90000, 4: 210000, 2: 450000}}
    rays = {t: [0, 1, 900, 10**9] + [n + d for n in lines[t].values() for d in (0, 1)] for t in lines}
    tiles = [(1, 1), (16, 8), (7, 5), (32, 8), (16, 16), (1, 4096), (4096, 1), (64, 64)]
    asked = [(lanes, w, h, n, t) for lanes in (0, 1, 4, 8, 16) for w, h in tiles for t in lines for n in rays[t]]
    text = "\n".join(" ".join(map(str, a)) for a in asked)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    for (lanes, w, h, n, t), line in zip(asked, out, strict=True):
        got, gw, gh = map(int, line.split())
        if lanes or n > 450000:  # an explicit count and its tile are kept, one lane too
            assert (got, gw, gh) == (lanes or 1, w, h)
        else:
            assert got == max(g for g in lines[t] if n <= lines[t][g])
            assert 1 <= gw <= w and 1 <= gh <= h and gw * gh <= 128 // got
            assert (gw, gh) == (w, h) or gw * gh * 4 > 128 // got  # no smaller than it has to be


@pytest.mark.gpu
def test_lanes_that_can_be_asked_for(lib):
    import torch

    from meteoros_gb300.renderer import Context

    w, h = 150, 87
    cam, tm, params, _ = scenes.config_view(3, w, h)
    with Context(0) as ctx:
        ctx.generate_volumes(7)
        assert ctx.set_tuning().batch_lanes == 0
        want, got = torch.zeros((h, w, 4), device="cuda"), torch.zeros((h, w, 4), device="cuda")
        ctx.render(cam, cam, tm, params, None, want, None, abi.MT_RENDER_FULL)
        for lanes in (0, 1, 4, 8, 16):
            assert ctx.set_tuning(batch_lanes=lanes).batch_lanes == lanes
            got.zero_()
            ctx.render_batch([scenes.make_view(cam, cam, tm, params, got, None, None, abi.MT_RENDER_FULL)])
            assert_bits_equal(got.cpu().numpy(), want.cpu().numpy(), f"{lanes} lanes")
        for lanes in (-1, 2, 3, 32, 64):
            with pytest.raises(abi.MeteorosError):
                ctx.set_tuning(batch_lanes=lanes)


@pytest.mark.gpu
@pytest.mark.parametrize("storage", [abi.MT_STORAGE_F16, abi.MT_STORAGE_BF16])
@pytest.mark.parametrize("size", [(75, 100), (76, 100), (200, 110), (201, 110), (300, 300), (301, 300), (671, 670), (671, 671)])
def test_16_bit_lines_give_one_frame(lib, size, storage):
    """Either side of the 16-bit forms' lines, marched as chosen and at one lane."""
    from meteoros_gb300.renderer import Context
    from tests.test_gpu_parity import gpu_render

    w, h = size
    cam, tm, params, _ = scenes.config_view(5, w, h)
    params.storage, params.fp64_shells = storage, 1
    with Context(0) as ctx:
        ctx.generate_volumes(7)
        frames = []
        for lanes in (0, 1):
            ctx.set_tuning(march_lanes=lanes)
            frames.append(gpu_render(ctx, cam, cam, tm, params, None, w, h, abi.MT_RENDER_FULL))
    (a, am, sa), (b, bm, sb) = frames
    assert_bits_equal(a, b, "rgba")
    assert_bits_equal(am, bm, "mask")
    assert (sa.primary_samples, sa.light_samples, sa.marched_rays) == (sb.primary_samples, sb.light_samples, sb.marched_rays)
