"""The rounding of production god rays: every step, lerp and sum of god-ray.frag:56-75 one fused multiply-add, whether
a pixel's taps are clamped or not.  Later passes round to 8 bits, where a rounding more or less shows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

F, D = np.float32, np.float64


def _fma(a, b, c):
    # the product of two floats is exact in a double; the sum's second rounding shows about once in 2^29
    return (D(a) * D(b) + D(c)).astype(F)


def _sun(u):
    """(proj * view) * location / w as the host evaluates it: the matrices first, then pairwise sums."""
    p, v, loc = np.array(list(u.camera.proj), F), np.array(list(u.camera.view), F), np.array(list(u.sun.location), F)
    q = []
    for r in range(4):
        row = []
        for c in range(4):
            s = F(p[r] * v[4 * c])
            for k in range(1, 4):
                s = F(s + F(p[4 * k + r] * v[4 * c + k]))
            row.append(F(s * loc[c]))
        q.append(F(F(row[0] + row[1]) + F(row[2] + row[3])))
    return F(q[0] / q[3]), F(q[1] / q[3])


def _god_rays(alpha, sx, sy):
    h, w = alpha.shape
    x, y = np.meshgrid(np.arange(w, dtype=F), np.arange(h, dtype=F))
    px, py = ((x + F(0.5)) / F(w)) * F(2) - F(1), ((y + F(0.5)) / F(h)) * F(2) - F(1)
    lx, ly = -(px - sx), -(py - sy)

    def lerp(a, b, t):
        return _fma(a, F(1) - t, b * t)

    total, decay = alpha * F(0.5), F(1)
    for _ in range(8):
        px, py = _fma(lx, F(0.09375), px), _fma(ly, F(0.09375), py)
        tx, ty = _fma(_fma(px, F(0.5), F(0.5)), F(w), F(-0.5)), _fma(_fma(py, F(0.5), F(0.5)), F(h), F(-0.5))
        fx, fy = np.floor(tx), np.floor(ty)
        i, j = np.clip(fx, -1, w).astype(int), np.clip(fy, -1, h).astype(int)
        x0, x1 = np.clip(i, 0, w - 1), np.clip(i + 1, 0, w - 1)
        y0, y1 = np.clip(j, 0, h - 1), np.clip(j + 1, 0, h - 1)
        t = lerp(lerp(alpha[y0, x0], alpha[y0, x1], tx - fx), lerp(alpha[y1, x0], alpha[y1, x1], tx - fx), ty - fy)
        total = _fma(t * F(0.5), F(0.125) * decay, total)
        decay = F(decay * F(0.99))
    return total * F(0.9)


@pytest.mark.parametrize("w,h,yaw", [(257, 129, 7.0), (641, 361, -20.0), (33, 9, 12.0), (640, 360, 90.0)])
def test_production_god_rays_round_as_fused_steps(cuda, mmlib, w, h, yaw):
    import marshmallow as mm
    r = mm.render.Renderer()
    try:
        u = mm.scene.uniforms(w, h, yaw=yaw, pitch=15.0, sun_elevation=21.0)
        src = np.random.default_rng(5).uniform(0, 1, (h, w, 4)).astype(F)
        dev = cuda.from_numpy(src).cuda()
        out = cuda.zeros_like(dev)
        r.god_rays(u, dev, out)
        cuda.cuda.synchronize()
        differ = (out.cpu().numpy()[..., 3] != _god_rays(src[..., 3], *_sun(u))).mean()
        assert differ <= 1e-3, differ  # two contractions of one step differ in a fifth of the pixels
    finally:
        r.close()
