"""Thin samples (march_kernel.cuh, thin_density): production launches skip the erosion fetches of samples that
are eroded to nothing whatever they return."""
import numpy as np
import pytest

F = np.float32


def _formats(texel):
    """The three storages of texel / 255: UNORM8, FP16, BF16 (rounded to nearest even)."""
    v = (texel.astype(F) / F(255.0)).astype(F)
    b = v.view(np.uint32)
    bf = ((b + 0x7FFF + ((b >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(F)
    return v, v.astype(np.float16).astype(F), bf


@pytest.mark.parametrize("lo,hi", [(0, 255), (0, 0), (255, 255), (100, 235), (250, 255), (0, 3)])
def test_thin_samples_are_eroded_away(lo, hi):
    # Any convex mix of eight texels (8-bit weights summing to 256, or float weights) in each storage, with
    # the result rounded as the texture unit rounds it, then the production arithmetic of hires_finish with
    # and without contraction: a density below the bound gives less than 1e-4 at every height from 0.1 up.
    rng = np.random.default_rng(hi * 256 + lo)
    n = 20000
    texel = rng.integers(lo, hi + 1, (n, 8, 3))
    texel[: n // 4] = texel[: n // 4, :1]  # flat neighbourhoods reach the ends of the range
    texel[0] = hi
    erosion_max = F((texel.reshape(-1, 3).astype(F) @ np.array([0.625, 0.25, 0.125], F)).max() * F(1.0 / 255.0))
    thin = F(1.0) - erosion_max * F(257.0 / 256.0) - F(0.001)
    whole = rng.multinomial(256, np.full(8, 0.125), n) / 256.0
    weights = np.where(rng.random((n, 1)) < 0.5, whole, rng.dirichlet(np.full(8, 0.3), n)).astype(F)
    rh = np.where(rng.random(n) < 0.3, F(0.1), rng.uniform(0.1, 1.0, n).astype(F)).astype(F)
    if not thin > 0:
        return
    orig = np.nextafter(thin, F(0)) * np.where(rng.random(n) < 0.5, F(1), rng.random(n).astype(F)).astype(F)
    for store in _formats(texel):
        mixed = np.einsum("nkc,nk->nc", store.astype(np.float64), weights.astype(np.float64))
        for dn in (mixed.astype(F), (np.round(mixed * 65535) / 65535).astype(F), mixed.astype(np.float16).astype(F)):
            for wide in (F, np.float64):  # every product rounded; products kept (as contraction keeps them)
                d = dn.astype(wide)
                e = (wide(0.625) * d[:, 0] + wide(0.25) * d[:, 1] + wide(0.125) * d[:, 2]).astype(F)
                s = np.clip(rh * F(10.0), 0, 1)
                e2 = (e.astype(wide) + (wide(1) - wide(2) * e.astype(wide)) * s.astype(wide)).astype(F)
                with np.errstate(divide="ignore", invalid="ignore"):
                    got = (orig - e2) * (F(1) / (F(1) - e2))
                assert (orig < e2).all() and not (got >= 1e-4).any()


@pytest.mark.gpu
@pytest.mark.parametrize("hi", ["generated", "zeros", "full", "one_texel"])
@pytest.mark.parametrize("fmt", [0, 1, 2])
@pytest.mark.parametrize("w,h", [(403, 200), (311, 333), (700, 411), (1001, 701)])
def test_thin_samples_move_no_ray(cuda, mmlib, hi, fmt, w, h):
    # A launch with work counters runs every sample.  The depth image (where each ray first accumulates)
    # agrees bit for bit, for hi-res textures at the ends of the erosion's range and in every format.
    import marshmallow as mm
    seeded, r = mm.render.Textures(seed=2), mm.render.Renderer()
    arrays = seeded.host_all()
    if hi != "generated":
        arrays["hi_res"] = np.full_like(arrays["hi_res"], 255 if hi == "full" else 0)
    if hi == "one_texel":
        arrays["hi_res"][5, 6, 7] = 255
    tex = mm.render.Textures.from_arrays(arrays)
    tex.set_density_format(fmt)
    try:
        u = mm.scene.uniforms(w, h, yaw=10.0, pitch=12.0, time=0.4)
        out = []
        for counters in (None, cuda.zeros(4, dtype=cuda.int64, device="cuda")):
            rgba, dep = cuda.zeros((h, w, 4), device="cuda"), cuda.zeros((h, w), device="cuda")
            r.march(u, tex, rgba, dep, counters=counters, density_format=fmt)
            cuda.cuda.synchronize()
            out.append(dep.cpu().numpy())
        assert np.array_equal(out[0], out[1])
        assert hi == "zeros" or np.isfinite(out[0]).any()
    finally:
        r.close()
        tex.close()
        seeded.close()
