"""The tiled noise kernels at the edges of their tiles and column lengths: every byte equals the oracle's."""
import numpy as np
import pytest

from gpu_util import noise_fill

pytestmark = pytest.mark.gpu

# 3D: column lengths 1, 2, 4 and 8 change at 28, 40 and 64; tiles are 32 x 2 texels; a small side has more
# cells in reach than the tables hold.  2D: the curl's blocks are 8 x 8 texels.
CASES = [(0, n, n, n, 4) for n in (1, 2, 27, 28, 39, 40, 63, 65, 97, 130)] + \
        [(1, n, n, n, 4) for n in (1, 3, 27, 33, 41, 64, 66)] + \
        [(2, w, h, 1, 2) for w, h in ((1, 1), (7, 9), (33, 100), (200, 3))] + \
        [(3, w, h, 1, 4) for w, h in ((1, 1), (31, 65), (300, 7))]


@pytest.mark.parametrize("kind,w,h,d,ch", CASES)
@pytest.mark.parametrize("seed", [0, 0xFFFFFFFF])
def test_noise_tiles_match_oracle(cuda, mmlib, orc, kind, w, h, d, ch, seed):
    got = noise_fill(cuda, mmlib, kind, seed, w, h, d).reshape(d, h, w, ch)
    assert np.array_equal(got, orc.noise(kind, seed, w, h, d, ch).reshape(d, h, w, ch))
