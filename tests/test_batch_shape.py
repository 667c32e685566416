"""The lanes and tile a batch is marched with: as asked for, or by its rays."""
import subprocess

import pytest

from meteoros_gb300 import abi, build, scenes
from tests.gpu_util import assert_bits_equal

MAIN = r"""
#include <cstdio>
#include "mt_batch.h"
int main() {
    int lanes, w, h;
    long long rays;
    while (scanf("%d %d %d %lld", &lanes, &w, &h, &rays) == 4) {
        const mt::BatchShape s = mt::batch_shape(lanes, w, h, rays);
        printf("%d %d %d\n", s.lanes, s.tile_w, s.tile_h);
    }
}
"""


def test_shape_rule(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "shape"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.CSRC}", str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    rays = [0, 1, 900, 8192, 8193, 28000, 28001, 90000, 90001, 210000, 210001, 450000, 450001, 10**9]
    tiles = [(1, 1), (16, 8), (7, 5), (32, 8), (16, 16), (1, 4096), (4096, 1), (64, 64)]
    asked = [(lanes, w, h, n) for lanes in (0, 1, 4, 8, 16) for w, h in tiles for n in rays]
    text = "\n".join(" ".join(map(str, a)) for a in asked)
    out = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.splitlines()
    for (lanes, w, h, n), line in zip(asked, out, strict=True):
        got, gw, gh = map(int, line.split())
        if lanes or n > 450000:  # an explicit count and its tile are kept, one lane too
            assert (got, gw, gh) == (lanes or 1, w, h)
        else:
            assert got in (2, 4, 8, 16, 32)
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
