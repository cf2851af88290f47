"""The erosion bound is reduced for generated hi-res volumes and for textures made from texels; a march that erodes
with a generated low-res volume, which has none, gives the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(120, 80), (700, 500), (1101, 701)])
def test_march_with_and_without_the_bound(cuda, mmlib, w, h):
    import marshmallow as mm
    made = mm.render.Textures(seed=4)
    arrays = made.host_all()
    arrays["hi_res"] = arrays["low_res"]
    uploaded, r = mm.render.Textures.from_arrays(arrays), mm.render.Renderer()
    try:
        u = mm.scene.uniforms(w, h, yaw=50.0, pitch=12.0)
        got = []
        for t, hi in ((made, "low_res"), (uploaded, "hi_res")):
            s = t.scene()
            s.hi_res = t.handles[hi]
            rgba, dep = cuda.zeros((h, w, 4), device="cuda"), cuda.zeros((h, w), device="cuda")
            r.march(u, s, rgba, dep)
            cuda.cuda.synchronize()
            got.append((rgba.cpu().numpy(), dep.cpu().numpy()))
        assert np.isfinite(got[0][1]).any()
        assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    finally:
        r.close()
        made.close()
        uploaded.close()
