"""The volumes' generator and sampler layouts against the CPU generator and
against whole uploads (GB300 only)."""
import numpy as np
import pytest

from meteoros_gb300 import abi, scenes
from tests.gpu_util import assert_bits_equal

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

KEYS = ("base", "detail", "curl", "weather")


@pytest.fixture(scope="module")
def context(lib):
    from meteoros_gb300.renderer import Context

    return Context


@pytest.mark.parametrize("seed", [0, 1, 2**32 - 1, 2**63 + 12345])
def test_generator_bit_exact_over_seeds(context, oracle, seed):
    want = oracle.generate_volumes(seed)
    with context(0) as ctx:
        ctx.generate_volumes(seed)
        got = ctx.download_volumes()
        half, bf = ctx.download_volumes_16(abi.MT_STORAGE_F16), ctx.download_volumes_16(abi.MT_STORAGE_BF16)
        for k in KEYS:
            assert np.array_equal(got[k], want[k]), k
            assert np.array_equal(half[k], want[k + "_h16"]), k
            assert np.array_equal(bf[k], want[k + "_b16"]), k


@pytest.mark.parametrize("changed", [("base",), ("detail",), ("curl",), ("weather",), ("detail", "curl"), KEYS])
def test_layouts_follow_each_change(context, changed):
    """Uploading some volumes over generated ones gives the frames of a context
    that was given all of them, in every storage, and a generated volume's
    layouts are its own."""
    rng = np.random.default_rng(11)
    with context(0) as a, context(0) as b:
        a.generate_volumes(3)
        vols = a.download_volumes()
        new = dict(vols)
        for k in changed:
            new[k] = rng.integers(0, 256, vols[k].shape, dtype=np.uint8)
        a.upload_volumes(**vols)  # bytes for all: the 16-bit texels are the bytes' too
        a.upload_volumes(**{k: new[k] for k in changed})
        b.upload_volumes(**new)
        cam, tm, params, _ = scenes.config_view(6, 64, 36)
        for storage in (abi.MT_STORAGE_U8, abi.MT_STORAGE_F16, abi.MT_STORAGE_BF16):
            params.storage = storage
            frames = []
            for ctx in (a, b):
                cur = torch.zeros((36, 64, 4), device="cuda")
                ctx.render(cam, cam, tm, params, None, cur, None, abi.MT_RENDER_FULL)
                frames.append(cur.cpu().numpy())
                got = ctx.download_volumes()
                assert all(np.array_equal(got[k], new[k]) for k in KEYS)
            assert_bits_equal(frames[0], frames[1], f"storage {storage}")
            if storage:
                got = a.download_volumes_16(storage)
                for k in KEYS:
                    c = torch.from_numpy(new[k].astype(np.float32)) / 255.0
                    want = c.half() if storage == abi.MT_STORAGE_F16 else c.bfloat16()
                    assert np.array_equal(got[k], want.view(torch.int16).numpy().view(np.uint16)), k


@pytest.mark.parametrize("kind", ["literal", "runs", "mixed", "single", "truncated"])
def test_tga_packet_shapes(context, oracle, kind):
    """Packets of 128, of 1 and of every length between, literal and run, files
    cut off at every kind of byte, sizes that are no multiple of 16."""
    import ctypes as C

    n = abi.MT_DETAIL_N
    rng = np.random.default_rng(5)
    files = []
    for z in range(n):
        head = bytearray([z % 3, 0, 10, 0, 0, 0, 0, 0, 0, 0, 0, 0, n, 0, n, 0, 32 if z % 2 else 24, 32 * (z % 4 == 1)])
        body, left = bytearray(rng.integers(0, 256, z % 3, dtype=np.uint8).tobytes()), n * n
        while left > 0:
            length = {"literal": 128, "runs": 128, "single": 1}.get(kind, int(rng.integers(1, 129)))
            run = kind == "runs" or (kind != "literal" and rng.random() < 0.5)
            px = 1 if run else length
            body.append((128 if run else 0) | (length - 1))
            body += rng.integers(0, 256, px * (4 if z % 2 else 3), dtype=np.uint8).tobytes()
            left -= length
        data = bytes(head + body)
        files.append(data[:18 + z * 61 % (len(data) - 18)] if kind == "truncated" else data)
    want = np.stack([oracle.decode_tga(f) for f in files])
    arr = (C.c_void_p * n)(*[C.cast(C.c_char_p(f), C.c_void_p) for f in files])
    sizes = (C.c_size_t * n)(*[len(f) for f in files])
    with context(0) as ctx:
        ctx.generate_volumes(1)
        assert ctx.lib.mt_decode_tga_volume(ctx.handle, abi.MT_VOLUME_DETAIL, arr, sizes, n, None) == abi.MT_OK
        assert np.array_equal(ctx.download_volumes()["detail"], want)
