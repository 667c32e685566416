"""Batches whose rays are too few for one lane each, against one render per view (GB300 only)."""
import pytest

from meteoros_gb300 import abi, scenes
from tests.gpu_util import assert_bits_equal

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module")
def ctx(lib):
    from meteoros_gb300.renderer import Context

    c = Context(0)
    c.generate_volumes(7)
    yield c
    c.close()


# Rays on either side of each line of the lane rule, in one, two and six views;
# odd tiles too, which shrink to a pass.
@pytest.mark.parametrize("sizes", [((128, 64),), ((128, 64), (1, 1)), ((150, 186), (10, 10)), ((150, 187),),
                                   ((299, 300), (30, 10)), ((300, 300), (1, 1)), ((447, 448), (97, 100)),
                                   ((670, 671),), ((670, 671), (43, 11)), ((64, 36), (65, 37), (7, 3), (1, 9), (33, 5), (160, 90))])
@pytest.mark.parametrize("tile", [(16, 8), (7, 5)])
def test_small_batches_equal_renders(ctx, sizes, tile):
    views, images = [], []
    for i, (w, h) in enumerate(sizes):
        cam, tm, params, _ = scenes.config_view(20 + i, w, h, steps=64)
        checkerboard = i % 2 == 1
        tm.frame_count_mod16 = 3 * i % 16
        prev = torch.rand((h, w, 4), device="cuda") if checkerboard else None
        want = torch.full((h, w, 4), float("nan"), device="cuda")
        got, mask = torch.full_like(want, float("nan")), torch.zeros((h, w), device="cuda")
        flags = abi.MT_RENDER_COUNT | (abi.MT_RENDER_CHECKERBOARD if checkerboard else abi.MT_RENDER_FULL)
        ctx.render(cam, cam, tm, params, prev, want, None, flags)
        views.append(scenes.make_view(cam, cam, tm, params, got, prev, mask, flags))
        images.append((prev, want, got, mask))
    a = ctx.stats(reset=True)
    for direct in (False, True):
        for _, _, got, _ in images:
            got.fill_(float("nan"))
        ctx.set_tuning(batch_tile=tile, batch_direct=direct)
        ctx.render_batch(views)
        b = ctx.stats(reset=True)
        for i, (_, want, got, _) in enumerate(images):
            assert_bits_equal(got.cpu().numpy(), want.cpu().numpy(), f"view {i}")
        assert (a.primary_samples, a.light_samples, a.marched_rays, a.pixels) == \
            (b.primary_samples, b.light_samples, b.marched_rays, b.pixels)
    ctx.set_tuning(batch_tile=(16, 8), batch_direct=False)
