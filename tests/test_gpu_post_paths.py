"""The downstream and temporal passes' size-dependent forms against the oracle (GB300 only)."""
import numpy as np
import pytest

from meteoros_gb300 import scenes
from tests.gpu_util import assert_bits_equal, to_dev

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
