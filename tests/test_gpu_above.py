"""Cameras above and inside the cloud layer through the pooled kernel: warps none of whose rays take a sample, warps
some of whose rays do."""
import numpy as np
import pytest

from gpu_util import render, render_counted

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("height", [30000.0, 23010.0, 22950.0, 12000.0])
@pytest.mark.parametrize("pitch", [3.0, -28.0, 40.0])
def test_rays_without_a_sample(cuda, orc, oracle_textures, mmlib, height, pitch):
    import marshmallow as mm
    import marshmallow.lib as L
    tex, r = mm.render.Textures(seed=0), mm.render.Renderer()
    try:
        w, h = 701, 399
        u = mm.scene.uniforms(w, h, eye=(0.0, height, 0.0), yaw=70.0, pitch=pitch, time=0.7)
        want, wd, wc = orc.march(u, oracle_textures, w, h)
        kw = dict(math=L.MATH_EXACT, sampler=L.SAMPLER_SOFTWARE)
        got, gd, gc = render_counted(cuda, r, u, tex, w, h, **kw)
        plain, pd = render(cuda, r, u, tex, w, h, **kw)
        for c, d in ((got, gd), (plain, pd)):
            assert np.array_equal(c.view(np.uint32), want.view(np.uint32))
            assert np.array_equal(d.view(np.uint32), wd.view(np.uint32))
        assert np.array_equal(gc, wc)
    finally:
        r.close()
        tex.close()
