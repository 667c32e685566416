"""The blur's small-image form and the image that passes unblurred, against the oracle (GB300 only)."""
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


# Either side of the lines between the forms, single rows and columns, a tile and
# one more; the sun in the image, at its edges and corners, and behind the camera,
# where the image passes as it is (with the pixels that no fragment stores to).
SIZES = [(1, 1), (1, 40), (64, 1), (3, 2), (32, 4), (33, 5), (160, 90), (300, 240), (301, 240), (447, 448), (500, 401)]
SUNS = ["ahead", "left", "right", "above", "corner", "behind"]


@pytest.mark.parametrize("size,sun", [(size, sun) for size in SIZES for sun in SUNS] + [((1700, 1060), "behind")])
@pytest.mark.parametrize("light", [(1.0, 1.0, 0.57, 1.0), (0.25, 0.75, 0.5, 1.0)])
def test_godrays_bit_exact(ctx, oracle, size, sun, light):
    w, h = size
    eye, yaw, pitch = {"ahead": ((0.0, 0.0, 2.0), 0.0, 20.0), "left": ((0.0, 0.0, 2.0), 50.0, 25.0),
                       "right": ((0.0, 0.0, 2.0), -50.0, 25.0), "above": ((0.0, 0.0, 2.0), 0.0, -20.0),
                       "corner": ((0.0, 0.0, 2.0), 40.0, -10.0), "behind": ((0.0, 100.0, 0.0), 30.0, 10.0)}[sun]
    rng = np.random.default_rng(w * 31 + h)
    mask = rng.random((h, w), dtype=np.float32) - np.float32(0.25)
    img = rng.random((h, w, 4), dtype=np.float32)
    cam = scenes.look(eye, yaw, pitch, 45.0, w, h)
    want = oracle.godrays(cam, np.array(light, np.float32), mask, img)
    assert (sun == "behind") == np.array_equal(want, img)
    out = torch.full((h, w, 4), float("nan"), device="cuda")
    ctx.godrays(cam, light, to_dev(mask, torch), to_dev(img, torch), out)
    assert_bits_equal(out.cpu().numpy(), want, f"{size} {sun}")
    same = to_dev(img, torch)
    ctx.godrays(cam, light, to_dev(mask, torch), same, same)
    assert_bits_equal(same.cpu().numpy(), want, f"{size} {sun} in place")
