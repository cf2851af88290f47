"""The march's dispatch at the lines of exact arithmetic and the software sampler: just below and above the work at
which teams of 8, 4 and 2 lanes and the pooled kernel take over, bit for bit, work counts included."""
import numpy as np
import pytest

from gpu_util import render, render_counted

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(cuda, mmlib):
    import marshmallow as mm
    t = mm.render.Textures(seed=0)
    r = mm.render.Renderer()
    yield t, r
    r.close()
    t.close()


# software sampler: work 30,000, 40,000 and 55,000 at (pitch, width in degrees, w, h)
@pytest.mark.parametrize("pitch,fov,w,h", [(6.0, 60.0, 313, 311), (6.0, 60.0, 317, 315), (6.0, 60.0, 359, 357),
                                           (6.0, 60.0, 365, 361), (6.0, 60.0, 421, 421), (6.0, 60.0, 427, 425),
                                           (-20.0, 60.0, 577, 575), (-20.0, 60.0, 587, 577), (80.0, 60.0, 233, 229)])
def test_software_sampler_equals_oracle(cuda, orc, oracle_textures, env, pitch, fov, w, h):
    import marshmallow as mm
    import marshmallow.lib as L
    tex, r = env
    u = mm.scene.uniforms(w, h, yaw=70.0, pitch=pitch, fov=fov, time=0.7)
    want, wd, wc = orc.march(u, oracle_textures, w, h)
    kw = dict(math=L.MATH_EXACT, sampler=L.SAMPLER_SOFTWARE)
    got, gd, gc = render_counted(cuda, r, u, tex, w, h, **kw)
    plain, pd = render(cuda, r, u, tex, w, h, **kw)
    for c, d in ((got, gd), (plain, pd)):
        assert np.array_equal(c.view(np.uint32), want.view(np.uint32))
        assert np.array_equal(d.view(np.uint32), wd.view(np.uint32))
    assert np.array_equal(gc, wc)


# texture unit: work 30,000, 50,000 and 100,000; the persistent schedule is the same arithmetic ray by ray
@pytest.mark.parametrize("pitch,fov,w,h", [(6.0, 60.0, 313, 311), (6.0, 60.0, 317, 315), (6.0, 60.0, 403, 401),
                                           (6.0, 60.0, 409, 405), (6.0, 60.0, 571, 569), (6.0, 60.0, 577, 573),
                                           (3.0, 8.0, 331, 329), (3.0, 8.0, 389, 387)])
def test_texture_unit_equals_persistent(cuda, env, pitch, fov, w, h):
    import marshmallow as mm
    import marshmallow.lib as L
    tex, r = env
    u = mm.scene.uniforms(w, h, yaw=70.0, pitch=pitch, fov=fov, time=0.7)
    want, wd, wc = render_counted(cuda, r, u, tex, w, h, math=L.MATH_EXACT, schedule=L.SCHEDULE_PERSISTENT)
    got, gd, gc = render_counted(cuda, r, u, tex, w, h, math=L.MATH_EXACT)
    plain, pd = render(cuda, r, u, tex, w, h, math=L.MATH_EXACT)
    for c, d in ((got, gd), (plain, pd)):
        assert np.array_equal(c.view(np.uint32), want.view(np.uint32))
        assert np.array_equal(d.view(np.uint32), wd.view(np.uint32))
    assert np.array_equal(gc, wc)


# production arithmetic with the software sampler: teams of 8 up to work 110,000, then the pooled kernel
@pytest.mark.parametrize("w,h", [(601, 595), (613, 599), (5, 3), (333, 331)])
def test_production_software_sampler(cuda, orc, oracle_textures, env, w, h):
    import marshmallow as mm
    import marshmallow.lib as L
    tex, r = env
    u = mm.scene.uniforms(w, h, yaw=70.0, pitch=6.0, time=0.7)
    got, gd = render(cuda, r, u, tex, w, h, sampler=L.SAMPLER_SOFTWARE)
    want, wd, _ = orc.march(u, oracle_textures, w, h, precision=64)
    e = mm.metrics.frame_errors(got, want, gd, wd)
    # the bounds that production arithmetic with the software sampler has against FP64 elsewhere
    assert e["nan"] == 0 and e["rmse_255"] <= 1.0 and e["p999_255"] <= 4.0 and e["frac_over_4"] <= 2e-3, e
