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
