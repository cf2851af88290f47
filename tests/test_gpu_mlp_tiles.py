"""The training kernel at the edges of its 128-sample tiles: one CTA with a padded tile, a launch of one
tile per CTA, CTAs with one tile more than others, several tiles per CTA (gradients summed in tensor memory,
the operand tiles used in turn)."""
import ctypes as C

import numpy as np
import pytest

import mlp_ref
from gpu_util import stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles,extra", [(0, 1), (0, 127), (1, 1), (2, 0), (304, 0), (304, 1), (911, 5), (1216, 77)])
def test_gradients_at_tile_edges(cuda, mmlib, tiles, extra):
    # Per layer within 1e-3 of the float64 reference with the same BF16 rounding points: a BF16 value that
    # FP32 sums round the other way is off by 2^-9 in one of 64 inputs.
    n = 128 * tiles + extra
    h = C.c_void_p()
    assert mmlib.mm_mlp_create(11, C.byref(h)) == 0
    try:
        k = mmlib.mm_mlp_param_count()
        p = np.zeros(k, np.float32)
        assert mmlib.mm_mlp_get_params(h, p.ctypes.data, k) == 0
        rng = np.random.default_rng(n)
        x = rng.normal(0, 1, (n, 16)).astype(np.float32)
        t = rng.uniform(0.05, 0.95, n).astype(np.float32)
        dx, dt = cuda.from_numpy(x).to(cuda.bfloat16).cuda(), cuda.from_numpy(t).cuda()
        ref, ref_loss = mlp_ref.gradients(p, x, t.astype(np.float64))
        for _ in range(2):  # a second launch starts from the first one's leftovers
            g = cuda.full((k,), 7.0, device="cuda")
            loss = C.c_float()
            assert mmlib.mm_mlp_gradients(h, C.c_void_p(dx.data_ptr()), C.c_void_p(dt.data_ptr()), n,
                                          C.c_void_p(g.data_ptr()), C.byref(loss), stream_ptr(cuda)) == 0
            got = g.cpu().numpy().astype(np.float64)
            assert abs(loss.value - ref_loss) < 1e-3 * ref_loss + 1e-6
            o = 0
            for name, shape in mlp_ref.SIZES:
                m = int(np.prod(shape))
                rel = np.linalg.norm(got[o:o + m] - ref[o:o + m]) / max(np.linalg.norm(ref[o:o + m]), 1e-12)
                assert rel < 1e-3, (name, rel)
                o += m
    finally:
        mmlib.mm_mlp_destroy(h)
