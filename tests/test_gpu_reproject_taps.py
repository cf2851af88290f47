"""The production reprojection's two tap paths (all taps inside the image, or clamped) against the exact
kernel, on a smooth source: a tap may take the neighbouring texel, no more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (31, 5), (33, 4), (257, 129), (641, 363)])
@pytest.mark.parametrize("turn", [0.0, 0.3, 20.0, 75.0])
def test_reproject_taps(cuda, mmlib, w, h, turn):
    import marshmallow as mm
    import marshmallow.lib as L
    r = mm.render.Renderer()
    try:
        u = mm.scene.uniforms(w, h, yaw=30.0, pitch=15.0)
        before = mm.scene.uniforms(w, h, yaw=30.0 - turn, pitch=15.0 + 0.1 * turn)
        u.camera_prev.view = before.camera.view
        y, x = np.mgrid[0:h, 0:w].astype(np.float32)
        src = np.stack([np.sin(0.05 * x) + 2, np.cos(0.04 * y) + 2, 0.001 * (x + y), np.sin(0.03 * (x - y)) + 2], -1)
        dep = 1000.0 + 0.01 * x + 0.02 * y
        src, dep = cuda.from_numpy(src.astype(np.float32)).cuda(), cuda.from_numpy(dep.astype(np.float32)).cuda()
        out = []
        for math in (L.MATH_FAST, L.MATH_EXACT):
            dst = (cuda.zeros((h, w, 4), device="cuda"), cuda.zeros((h, w), device="cuda"))
            r.reproject(u, (src, dep), dst, math=math)
            cuda.cuda.synchronize()
            out.append([t.cpu().numpy() for t in dst])
        # every tap within one texel of the exact kernel's: the mean moves by at most the largest step
        # between diagonal neighbours, 0.05 + 0.04 of the steepest channels, plus float rounding
        assert np.abs(out[0][0] - out[1][0]).max() <= 0.09 + 1e-5
        assert np.abs(out[0][1] - out[1][1]).max() <= 0.03 + 1e-3
    finally:
        r.close()
