"""Where production rays end: past relative height 0.9 the cloud layer is empty, so the samples a ray
leaves out there (march_kernel.cuh, shell_end) are all zero."""
import numpy as np
import pytest

F = np.float32


@pytest.mark.parametrize("x,y,z", [(0.0, 10.0, 0.0), (1.0e6, 10.0, -1.0e6), (3.0e4, 9000.0, -7.0e5), (0.0, 22900.0, 0.0),
                                   (-1.0e6, -9.0e5, 1.0e6)])
def test_samples_past_the_end_are_empty(x, y, z):
    # The sample's height in float32, operation by operation as geo_at forms it (a rsqrt off by 2^-22
    # either way), for rays of every elevation and distances from the end to 400 km beyond it.
    rng = np.random.default_rng(7)
    n = 200000
    el = np.concatenate([np.geomspace(1e-7, np.pi / 2, n // 2), rng.uniform(0, np.pi / 2, n // 2)])
    az = rng.uniform(0, 2 * np.pi, n)
    rd = np.stack([np.cos(el) * np.cos(az), np.sin(el), np.cos(el) * np.sin(az)], 1).astype(F)
    cam, centre = np.array([x, y, z], F), np.array([x, -995000.0, z], F)
    h, re = float(F(y)) + 995000.0, 1.0e6 + 0.9 * 20000.0 + 40.0
    assert h < re
    end_h, end_c = F(h), F(re * re - h * h)
    b = end_h * rd[:, 1]
    t_end = np.sqrt(b * b + end_c) - b
    for past in (0.0, 1.0, 300.0, 1000.0, 4.0e5):
        t = (t_end + F(past)).astype(F)
        d = (cam + t[:, None] * rd).astype(F) - centre
        dd = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
        for err in (-1.0, 1.0):
            rs = (1.0 / np.sqrt(dd.astype(np.float64)) * (1 + err * 2.0 ** -22)).astype(F)
            rh = np.clip(np.abs(dd * rs - F(1.0e6)) * F(1.0 / 20000.0), 0, 1)
            assert (rh > F(0.9)).all(), (past, float(rh.min()))
            cumulus = np.maximum(rh * (F(22.5) - F(25.0) * rh), 0)
            assert (cumulus < 1e-4).all()  # the other two profiles end at 0.7 and 0.3


@pytest.mark.gpu
@pytest.mark.parametrize("w,h,eye,pitch,sun", [(331, 173, (0.0, 10.0, 0.0), 4.0, 30.0), (1280, 720, (0.0, 10.0, 0.0), 25.0, 5.0),
                                               (512, 200, (3.0e4, 9000.0, -7.0e5), 5.0, 60.0),
                                               (640, 420, (0.0, 24000.0, 0.0), 3.0, 30.0),
                                               (200, 100, (2.0e6, 10.0, 0.0), 10.0, 30.0)])
def test_ended_rays_equal_counted_ones(w, h, eye, pitch, sun):
    # A launch that counts the shader's samples runs them all; without counters the rays end early.
    # Same depth, and colours equal up to the rounding of two builds of the same expressions.
    import torch
    import marshmallow as mm
    tex, r = mm.render.Textures(seed=3), mm.render.Renderer()
    try:
        u = mm.scene.uniforms(w, h, eye=eye, yaw=40.0, pitch=pitch, sun_elevation=sun, time=1.0)
        out = []
        for counters in (None, torch.zeros(4, dtype=torch.int64, device="cuda")):
            rgba, dep = torch.zeros((h, w, 4), device="cuda"), torch.zeros((h, w), device="cuda")
            r.march(u, tex, rgba, dep, counters=counters)
            torch.cuda.synchronize()
            out.append((rgba.cpu().numpy(), dep.cpu().numpy()))
        assert np.array_equal(out[0][1], out[1][1])
        np.testing.assert_allclose(out[0][0], out[1][0], rtol=1e-5, atol=1e-6)
    finally:
        r.close()
        tex.close()
