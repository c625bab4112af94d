"""Device Z-Sobol at the edges of its 32-bit form: the Morton index and the
sample index of a frame fit 32 bits up to 16 base-4 digits, wider frames take
the 64-bit form; both equal the oracle's sampler bit for bit."""
import numpy as np
import pytest

from oracle import pyoracle as O
from tests.test_gpu_render import device_zsobol

pytestmark = pytest.mark.gpu

# (spp, resolution): no digits at all, one odd bit, odd and even sample bits,
# exactly 32 index bits, the first frames beyond, a far wider one
FRAMES = [(1, (1, 1)), (2, (1, 1)), (8, (1, 3)), (1024, (2048, 2048)), (512, (2048, 1100)), (2048, (2048, 2048)),
          (256, (4096, 2160)), (512, (4096, 4096)), (64, (30000, 20000))]


@pytest.mark.parametrize("spp,res", FRAMES)
@pytest.mark.parametrize("seed", [1234, 0, (7 << 40) + 9])
def test_sampler_bits_at_index_widths(spp, res, seed):
    rng = np.random.default_rng(spp + res[0])
    n = 777  # not a whole number of blocks or warps
    px, py, idx = (rng.integers(0, m, n) for m in (res[0], res[1], spp))
    px[:4], py[:4], idx[:4] = [0, 0, res[0] - 1, res[0] - 1], [0, res[1] - 1, 0, res[1] - 1], [0, spp - 1, 0, spp - 1]
    kinds = [2, 2] + [1, 2, 3, 3, 1] * 12
    ours = device_zsobol(spp, res[0], res[1], px, py, idx, kinds, seed=seed)
    ref = O.zsobol_batch(spp, res[0], res[1], px, py, idx, kinds, seed=seed)
    assert ours.tobytes() == ref.tobytes()


def test_nibble_tables_of_many_dimensions():
    """The tables that the device fills from the matrices: 192 dimensions, all
    eight groups of index bits."""
    rng = np.random.default_rng(5)
    px, py, idx = (rng.integers(0, m, 512) for m in (2048, 2048, 1024))
    for k in range(0, 64, 16):  # every draw of a path takes the next dimensions
        kinds = [1] * k + [3] * (64 - k)
        ours = device_zsobol(1024, 2048, 2048, px, py, idx, kinds)
        assert ours.tobytes() == O.zsobol_batch(1024, 2048, 2048, px, py, idx, kinds).tobytes()
