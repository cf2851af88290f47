/*
 * post_taps.h - the single post passes' taps and the tests that let production arithmetic take them without
 * clamps, for the kernels (post_kernel.cuh) and, compiled by a host compiler, for the tests.
 */
#ifndef MM_POST_TAPS_H_
#define MM_POST_TAPS_H_

#if defined(__CUDACC__)
#define MM_TAPS_HD __host__ __device__ __forceinline__
#else
#define MM_TAPS_HD inline
#endif

#if !defined(__CUDA_ARCH__)
#include <math.h>
#endif

namespace mm {
namespace post {

MM_TAPS_HD void frag(int x, int y, int w, int h, float* px, float* py, float* u, float* v) {
    *u = ((float)x + 0.5f) / (float)w;
    *v = ((float)y + 0.5f) / (float)h;
    *px = *u * 2.0f - 1.0f;
    *py = *v * 2.0f - 1.0f;
}

// god-ray.frag:56-75 for the fragment at NDC (px, py) with centre alpha ca.
template <class Taps>
MM_TAPS_HD float god_ray_term(float sun_x, float sun_y, const Taps& alpha, float px, float py, float ca) {
    const float weight_density = 1.0f / 8.0f * 0.75f;  // SAMPLE_WEIGHT * DENSITY
    const float dx = (px - sun_x) * weight_density, dy = (py - sun_y) * weight_density;
    float accum = ca * 0.5f;
    float decay = 1.0f;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 8; ++i) {
        px = px - dx;
        py = py - dy;
        float amt = alpha(px * 0.5f + 0.5f, py * 0.5f + 0.5f) * 0.5f;
        amt = amt * (1.0f / 8.0f * decay);
        accum = accum + amt;
        decay = decay * 0.99f;
    }
    return accum * 0.9f;
}

// radialBlur.frag:51-60: the mean of ten taps of the god-ray term along the line to the sun.
template <class Taps>
MM_TAPS_HD float radial_term(float sun_x, float sun_y, const Taps& g, float px, float py) {
    float lx = sun_x - px, ly = sun_y - py;
    const float dist = sqrtf(lx * lx + ly * ly);
    lx = lx / dist;
    ly = ly / dist;
    const float taps[10] = {-0.08f, -0.05f, -0.03f, -0.02f, -0.01f, 0.01f, 0.02f, 0.03f, 0.05f, 0.08f};
    float accum = 0.0f;
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (int i = 0; i < 10; ++i) {
        const float ox = taps[i] * lx * 1.5f * dist, oy = taps[i] * ly * 1.5f * dist;
        accum = accum + g((px + ox) * 0.5f + 0.5f, (py + oy) * 0.5f + 0.5f) * 1.1f;
    }
    return accum / 10.0f;
}

// The part of a w x h image where a bilinear tap has its four texels inside.  The ends of a line are tested here
// and the taps on it computed elsewhere, in more steps and contracted as the compiler likes: eight subtractions
// of positions up to 1 and a step off by 2^-23 of its size put a tap up to 8 * 2^-23 from where the end says, half
// of that in (u, v), and two roundings more make the texel position: less than 6 * 2^-23 of the image's side.
// The margin is 8 * 2^-23 of it.
constexpr float kTapMargin = 1.0f / 1048576.0f;
struct TapArea {
    float w, h;
    // Whether a tap at (u, v) has its four texels inside by the margin; taps between two such taps of a line have
    // them inside too.  False for NaN.
    MM_TAPS_HD bool holds(float u, float v) const {
        const float x = u * w - 0.5f, y = v * h - 0.5f, mx = kTapMargin * w, my = kTapMargin * h;
        return x >= mx && x < w - 1.0f - mx && y >= my && y < h - 1.0f - my;
    }
};

// a - b, apart from any other use of the two: where the test below shared the taps' own differences and steps, the
// compiler contracted those anew and a quarter of the pixels came out a rounding off.
MM_TAPS_HD float minus_apart(float a, float b) {
#if defined(__CUDA_ARCH__)
    return __fsub_rn(a, b);
#else
    return a - b;
#endif
}

// Whether all taps of god_ray_term at (px, py) have their four texels inside: the first and the eighth, 3/32 and
// 3/4 of the way to the sun.
MM_TAPS_HD bool god_ray_inside(const TapArea& a, float sun_x, float sun_y, float px, float py) {
    const float lx = minus_apart(sun_x, px), ly = minus_apart(sun_y, py);
    return a.holds((px + lx * 0.09375f) * 0.5f + 0.5f, (py + ly * 0.09375f) * 0.5f + 0.5f) &&
           a.holds((px + lx * 0.75f) * 0.5f + 0.5f, (py + ly * 0.75f) * 0.5f + 0.5f);
}

// Whether all taps of radial_term at (px, py) have their four texels inside.  On the sun radial_term divides 0
// by 0 (as the shader does), and next to it a square could be flushed to zero: its taps are then NaN, which only
// the clamped ones take.  The outermost taps lie 0.12 of the way to the sun on either side; a little further
// out here, since the division and the products after it round in proportion to the way.
MM_TAPS_HD bool radial_inside(const TapArea& a, float sun_x, float sun_y, float px, float py) {
    const float lx = sun_x - px, ly = sun_y - py;
    if (!(fabsf(lx) + fabsf(ly) > 1.0e-12f)) return false;
    const float ox = lx * 0.1201f, oy = ly * 0.1201f;
    return a.holds((px - ox) * 0.5f + 0.5f, (py - oy) * 0.5f + 0.5f) &&
           a.holds((px + ox) * 0.5f + 0.5f, (py + oy) * 0.5f + 0.5f);
}

}  // namespace post
}  // namespace mm

#endif  // MM_POST_TAPS_H_
