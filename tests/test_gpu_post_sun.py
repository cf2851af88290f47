"""The single post passes with the sun exactly on a fragment: there the radial blur divides 0 by 0, as its shader
does, and production arithmetic gives that pixel what the exact pass gives it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F = np.float32


@pytest.mark.parametrize("w,h", [(3, 3), (33, 9), (257, 129), (641, 361)])
@pytest.mark.parametrize("where", ["centre", "corner", "beside", "edge", "inner"])
def test_sun_on_a_fragment(cuda, mmlib, w, h, where):
    import marshmallow as mm
    import marshmallow.lib as L

    def at(i, n):
        return F(F(F(F(i) + F(0.5)) / F(n)) * F(2.0) - F(1.0))

    i, j = {"centre": (w // 2, h // 2), "corner": (0, h - 1), "beside": (w // 2, h // 2), "edge": (w - 1, h // 3),
            "inner": (w // 3, h // 4)}[where]
    sx, sy = at(i, w), at(j, h)
    if where == "beside":
        sx = sx + F(1e-6)
    r = mm.render.Renderer()
    try:
        u = mm.scene.uniforms(w, h, sun_elevation=20.0)
        for m in (u.camera.proj, u.camera.view):  # the sun's position is its place in the image
            for k in range(16):
                m[k] = 1.0 if k % 5 == 0 else 0.0
        for k, value in enumerate((sx, sy, 0.0, 1.0)):
            u.sun.location[k] = float(value)
        src = cuda.from_numpy(np.random.default_rng(w + h).uniform(0, 1, (h, w, 4)).astype(F)).cuda()
        got = {}
        for math in (L.MATH_FAST, L.MATH_EXACT):
            a, b = cuda.zeros_like(src), cuda.zeros_like(src)
            r.god_rays(u, src, a, math=math)
            r.radial_blur(u, src, b, math=math)
            cuda.cuda.synchronize()
            got[math] = a.cpu().numpy(), b.cpu().numpy()
        assert np.isnan(got[L.MATH_EXACT][1][j, i, :3]).all() == (where != "beside")
        # as for the passes with the sun elsewhere: a tap's position is off by a few roundings of numbers up to
        # max(w, h), the blur is scaled by colour * intensity * 1.1
        k = max(1.1 * u.sun.color[c] * u.sun.intensity for c in range(3))
        tol = 16 * max(w, h, 8) * 2.0 ** -23
        assert np.abs(got[L.MATH_FAST][0] - got[L.MATH_EXACT][0]).max() <= tol
        fast, exact = got[L.MATH_FAST][1], got[L.MATH_EXACT][1]
        assert np.array_equal(np.isnan(fast), np.isnan(exact))
        assert np.nanmax(np.abs(fast - exact)) <= tol * max(k, 1.0) + 1e-6
    finally:
        r.close()
