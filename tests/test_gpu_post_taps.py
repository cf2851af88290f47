"""The single post passes' production taps, inside the image and clamped, against the exact passes: the sun in
the view, at its edge and outside it, on images down to one pixel."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(1, 1), (2, 3), (33, 9), (257, 129), (640, 361)])
@pytest.mark.parametrize("yaw,pitch,sun", [(0.0, 15.0, 20.0), (40.0, 10.0, 30.0), (170.0, 20.0, 45.0), (5.0, 20.0, 21.0)])
def test_passes_match_exact(cuda, mmlib, w, h, yaw, pitch, sun):
    import marshmallow as mm
    import marshmallow.lib as L
    r = mm.render.Renderer()
    try:
        u = mm.scene.uniforms(w, h, yaw=yaw, pitch=pitch, sun_elevation=sun)
        rng = np.random.default_rng(w + 1000 * h)
        src = cuda.from_numpy(rng.uniform(0, 1, (h, w, 4)).astype(np.float32)).cuda()
        got = {}
        for math in (L.MATH_FAST, L.MATH_EXACT):
            a, b = cuda.zeros_like(src), cuda.zeros_like(src)
            r.god_rays(u, src, a, math=math)
            r.radial_blur(u, src, b, math=math)
            cuda.cuda.synchronize()
            got[math] = a.cpu().numpy(), b.cpu().numpy()
        # a tap's position is off by a few roundings of numbers up to max(w, h): its weights move by that much
        # of a texel, its value by as much of the range 1; the blur is scaled by colour * intensity * 1.1
        k = max(1.1 * u.sun.color[c] * u.sun.intensity for c in range(3))
        tol = 16 * max(w, h, 8) * 2.0 ** -23
        far = max(1.0, abs(_sun(u)[0]), abs(_sun(u)[1]))  # taps towards a sun far outside start from larger numbers
        assert np.abs(got[0][0] - got[1][0]).max() <= tol * far
        assert np.abs(got[0][1] - got[1][1]).max() <= tol * far * max(k, 1.0) + 1e-6
    finally:
        r.close()


def _sun(u):
    p, v = (np.array(list(m), np.float64).reshape(4, 4).T for m in (u.camera.proj, u.camera.view))
    q = p @ v @ np.array(list(u.sun.location), np.float64)
    return q[0] / q[3], q[1] / q[3]
