"""One pixel in 16 by the pooled kernel, which keeps its background in the image while the reprojection writes the
other pixels of the same image on a second stream."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env(cuda, mmlib):
    import marshmallow as mm
    t = mm.render.Textures(seed=0)
    r = mm.render.Renderer()
    yield t, r
    r.close()
    t.close()


def _frame(mm, w, h, phase):
    u = mm.scene.uniforms(w, h, yaw=30.0, pitch=20.0, time=1.0)
    u.camera_prev = mm.scene.uniforms(w, h, yaw=29.0, pitch=20.0).camera_prev
    u.sun.color[3] = float(phase)
    rng = np.random.default_rng(phase)
    return u, rng.uniform(0, 20, (h, w, 4)).astype(np.float32), rng.uniform(1e3, 3e5, (h, w)).astype(np.float32)


@pytest.mark.parametrize("phase", [0, 9])
def test_exact_frame_equals_oracle(cuda, orc, oracle_textures, env, phase):
    # 2881x1621: 293,000 marched rays, work above the exact software march's last line
    import marshmallow as mm
    import marshmallow.lib as L
    tex, r = env
    w, h = 2881, 1621
    u, src, sd = _frame(mm, w, h, phase)
    prev = cuda.from_numpy(src).cuda(), cuda.from_numpy(sd).cuda()
    out = cuda.zeros_like(prev[0]), cuda.zeros_like(prev[1])
    r.frame(u, tex, prev, out, math=L.MATH_EXACT, sampler=L.SAMPLER_SOFTWARE)
    cuda.cuda.synchronize()
    want, wd = orc.reproject(u, src, sd)
    mw, md, _ = orc.march(u, oracle_textures, w, h, pixel_mode=1)
    at = np.s_[phase // 4::4, phase % 4::4]
    want[at], wd[at] = mw[at], md[at]
    assert np.array_equal(out[0].cpu().numpy().view(np.uint32), want.view(np.uint32))
    assert np.array_equal(out[1].cpu().numpy(), wd)


@pytest.mark.parametrize("phase", [3, 14])
def test_production_frame_equals_its_passes(cuda, env, phase):
    # 4203x2403: 632,000 marched rays, work above production's last line; the same kernels one after the other
    import marshmallow as mm
    tex, r = env
    w, h = 4203, 2403
    u, src, sd = _frame(mm, w, h, phase)
    prev = cuda.from_numpy(src).cuda(), cuda.from_numpy(sd).cuda()
    want = cuda.zeros_like(prev[0]), cuda.zeros_like(prev[1])
    r.reproject(u, prev, want)
    r.march(u, tex, *want, pixel_mode=1)
    cuda.cuda.synchronize()
    for _ in range(3):
        out = cuda.full_like(prev[0], -7.0), cuda.full_like(prev[1], -7.0)
        r.frame(u, tex, prev, out)
        cuda.cuda.synchronize()
        assert cuda.equal(out[0], want[0]) and cuda.equal(out[1], want[1])
