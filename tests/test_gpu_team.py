"""The team march (launches with little work next to their longest rays): the three team sizes and the pooled
kernel at the edges of their ranges, in exact arithmetic against the oracle, bit for bit, work counts included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# odd sides at all team sizes; a small image; the pooled kernel's first
SIZES = [(5, 3), (263, 266), (301, 299), (301, 300), (479, 501), (481, 500), (509, 513), (517, 509), (775, 773),
         (777, 773)]


@pytest.fixture(scope="module")
def env(cuda, mmlib):
    import marshmallow as mm
    t = mm.render.Textures(seed=0)
    r = mm.render.Renderer()
    yield t, r
    r.close()
    t.close()


def _roll(u, degrees):
    """Turns the camera about its view direction: right and up (rows 0 and 1 of the view matrix)."""
    c, s = np.cos(np.radians(degrees)), np.sin(np.radians(degrees))
    for k in range(3):
        right, up = u.camera.view[4 * k], u.camera.view[4 * k + 1]
        u.camera.view[4 * k], u.camera.view[4 * k + 1] = float(c * right + s * up), float(c * up - s * right)


def _check(cuda, orc, oracle_textures, env, w, h, u):
    import marshmallow.lib as L
    tex, r = env
    rgba, dep = cuda.zeros((h, w, 4), device="cuda"), cuda.zeros((h, w), device="cuda")
    cnt = cuda.zeros(4, dtype=cuda.int64, device="cuda")
    want, wd, wc = orc.march(u, oracle_textures, w, h)
    for counters in (cnt, None):  # the counting launch and the other one resolve their rounds differently
        r.march(u, tex, rgba, dep, math=L.MATH_EXACT, sampler=L.SAMPLER_SOFTWARE, counters=counters)
        cuda.cuda.synchronize()
        assert np.array_equal(rgba.cpu().numpy().view(np.uint32), want.view(np.uint32))
        assert np.array_equal(dep.cpu().numpy().view(np.uint32), wd.view(np.uint32))
    assert np.array_equal(cnt.cpu().numpy().astype(np.uint64), wc)


# just below and above each line of the dispatch (work 30,000, 90,000, 212,000): (pitch, width in degrees, w, h)
LINES = [(6.0, 60.0, 313, 311), (6.0, 60.0, 317, 315), (6.0, 60.0, 545, 539), (6.0, 60.0, 549, 541),
         (6.0, 60.0, 835, 831), (6.0, 60.0, 839, 831), (80.0, 60.0, 189, 187), (80.0, 60.0, 195, 193),
         (3.0, 8.0, 331, 331), (3.0, 8.0, 337, 335), (3.0, 8.0, 513, 515), (3.0, 8.0, 517, 515),
         (-20.0, 60.0, 333, 331), (-60.0, 60.0, 195, 193), (90.0, 60.0, 129, 7)]


@pytest.mark.parametrize("pitch,fov,w,h", LINES)
def test_dispatch_lines_exact(cuda, orc, oracle_textures, env, pitch, fov, w, h):
    import marshmallow as mm
    u = mm.scene.uniforms(w, h, yaw=70.0, pitch=pitch, fov=fov, time=0.7)
    _check(cuda, orc, oracle_textures, env, w, h, u)


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("roll,pitch,sun", [(0.0, 6.0, 30.0), (25.0, 12.0, 8.0)])
def test_team_sizes_exact(cuda, orc, oracle_textures, env, w, h, roll, pitch, sun):
    import marshmallow as mm
    u = mm.scene.uniforms(w, h, yaw=70.0, pitch=pitch, sun_elevation=sun, time=0.7)
    if roll:
        _roll(u, roll)
    _check(cuda, orc, oracle_textures, env, w, h, u)
