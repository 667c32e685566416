"""Batches whose views share images: which reprojections may run side by side."""
import itertools
import subprocess

import pytest

from meteoros_gb300 import abi, build, scenes
from tests.gpu_util import assert_bits_equal

MAIN = r"""
#include <cstdio>
#include "mt_batch.h"
int main() {
    unsigned n;
    while (scanf("%u", &n) == 1) {
        std::vector<mt::ImageBytes> v(n);
        for (auto& i : v) {
            unsigned long long at, bytes, written;
            if (scanf("%llu %llu %llu", &at, &bytes, &written) != 3) return 1;
            i = mt::image_bytes((const void*)at, bytes, written != 0);
        }
        printf("%d\n", mt::written_overlap(v) ? 1 : 0);
    }
}
"""


def test_overlap_rule_equals_every_pair(tmp_path):
    """The sweep against a look at every pair, over all arrangements of three and
    many random ones of up to nine images, in any order."""
    import random

    (tmp_path / "main.cpp").write_text(MAIN)
    exe = tmp_path / "overlap"
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{build.CSRC}", str(tmp_path / "main.cpp"), "-o", str(exe)], check=True)
    kinds = [(at, n, w) for at in (1, 2, 4) for n in (1, 2, 4) for w in (0, 1)]
    lists = [list(c) for c in itertools.product(kinds, repeat=3)]
    rng = random.Random(1)
    for _ in range(4000):
        lists.append([(rng.randrange(1, 40), rng.randrange(1, 9), rng.randrange(2)) for _ in range(rng.randrange(10))])
    text = "\n".join(" ".join([str(len(c))] + [f"{a} {n} {w}" for a, n, w in c]) for c in lists)
    got = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
    want = [int(any((a[2] or b[2]) and a[0] < b[0] + b[1] and b[0] < a[0] + a[1] for a, b in itertools.combinations(c, 2)))
            for c in lists]
    assert [int(g) for g in got] == want
    assert 0 < sum(want) < len(want)


@pytest.mark.gpu
@pytest.mark.parametrize("order", ["read first", "written first"])
@pytest.mark.parametrize("n_views", [2, 6, 11])
def test_views_that_share_images(lib, n_views, order):
    """A chain of views, each one's frame the image that the view before it (or
    after it) reprojects from: the graph, the direct and the allocation-free form
    agree, and where each image is read before it is written they equal one render
    per view."""
    import torch

    from meteoros_gb300.renderer import Context

    w, h = 331, 187
    gen = torch.Generator(device="cuda").manual_seed(n_views)
    first = [torch.rand((h, w, 4), device="cuda", generator=gen) for _ in range(n_views + 1)]
    views = []
    for i in range(n_views):
        cam, tm, params, _ = scenes.config_view(30 + i, w, h, steps=64)
        tm.frame_count_mod16 = 5 * i % 16
        views.append((cam, tm, params))

    with Context(0) as ctx:
        ctx.generate_volumes(7)

        def run(form):
            images = [t.clone() for t in first]
            if order == "read first":  # view i reads image i, view i + 1 overwrites it
                prev, cur = images[:-1], [images[-1]] + images[:-2]
            else:  # view i overwrites the image that view i + 1 reads
                prev, cur = images[:-1], images[1:]
            batch = [scenes.make_view(c, c, t, p, cur[i], prev[i], None, abi.MT_RENDER_CHECKERBOARD)
                     for i, (c, t, p) in enumerate(views)]
            if form == "each":
                for i, (c, t, p) in enumerate(views):
                    ctx.render(c, c, t, p, prev[i], cur[i], None, abi.MT_RENDER_CHECKERBOARD)
            elif form == "noalloc":
                arr = (abi.View * n_views)(*batch)
                assert ctx.lib.mt_render_batch_noalloc(ctx.handle, arr, n_views,
                                                       torch.cuda.current_stream().cuda_stream) == abi.MT_OK
            else:
                ctx.set_tuning(batch_direct=form == "direct")
                ctx.render_batch(batch)
            torch.cuda.synchronize()
            return [t.cpu().numpy() for t in images]

        want = run("each" if order == "read first" else "direct")
        for form in ("graph", "direct", "noalloc", "graph"):
            for i, (got, ref) in enumerate(zip(run(form), want)):
                assert_bits_equal(got, ref, f"{form}, image {i}")
