"""Training whose kernels follow each other without a gap (no loss history) gives the parameters of training that
synchronizes after every step (with one), bit for bit: all sums are taken in a fixed order."""
import ctypes as C

import numpy as np
import pytest

from gpu_util import stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [1, 2, 303, 304, 305, 1024])
def test_overlapped_steps_equal_synchronized_ones(cuda, mmlib, tiles):
    steps, batch = 24, 128 * tiles
    n = 2 * batch + 128  # the batches wrap around
    rng = np.random.default_rng(tiles)
    x = cuda.from_numpy(rng.normal(0, 1, (n, 16)).astype(np.float32)).to(cuda.bfloat16).cuda()
    t = cuda.from_numpy(rng.uniform(0.05, 0.95, n).astype(np.float32)).cuda()
    got = []
    for synchronized in (True, False, False):
        h = C.c_void_p()
        assert mmlib.mm_mlp_create(11, C.byref(h)) == 0
        try:
            losses = np.zeros(steps, np.float32)
            for _ in range(2):  # the second run starts behind the first one's last kernel
                assert mmlib.mm_mlp_train(h, C.c_void_p(x.data_ptr()), C.c_void_p(t.data_ptr()), n, batch, steps, 1e-3,
                                          losses.ctypes.data if synchronized else None, stream_ptr(cuda)) == 0
            p = np.zeros(mmlib.mm_mlp_param_count(), np.float32)
            assert mmlib.mm_mlp_get_params(h, p.ctypes.data, p.size) == 0
            got.append(p)
        finally:
            mmlib.mm_mlp_destroy(h)
    assert np.isfinite(got[0]).all()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
