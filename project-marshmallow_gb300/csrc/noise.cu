// noise.cu - GPU generators for the cloud textures (mm_noise_generate / mm_noise_fill).
//
// Built with -fmad=false so every float operation rounds exactly as the sequential definition
// in the CPU oracle does: the integer hash and lattice stages are exact by construction and the
// 8-bit texels come out identical.
//
// Generator definition (the reference ships these textures pre-baked, README.md:68, so the
// seeded generators below are this library's own):
//   hash32     lowbias32 integer mixer; hash3(x,y,z,s) = hash32(x + hash32(y + hash32(z + s)))
//   stream     s = hash32(seed ^ hash32(0x9E3779B9 * (1 + 64 kind + 8 channel + octave)))
//   lattice    texel centre i of n at frequency f: ((2i+1) f) / (2n)
//   Worley     inverted F1 (1 - min(F1, 1)), one feature point per cell, period f on each axis
//   WorleyFBM  0.625 W(f) + 0.25 W(2f) + 0.125 W(4f)
//   Perlin     gradient noise, 12 edge gradients, quintic fade, period f
//   low-res    R = remap(PerlinFBM01(4, 3 oct), WorleyFBM(4) - 1, 1, 0, 1) * 1.64 - 0.593,
//              G/B/A = WorleyFBM(4/8/16) * 0.866 + 0.271              (128^3 RGBA8)
//   hi-res     R/G/B = WorleyFBM(2/4/8) * 0.866 + 0.271, A = 0          (32^3 RGBA8)
//   curl       psi = 2D Perlin FBM (4 cells, 5 octaves); (dpsi/dy, -dpsi/dx) by central
//              differences a quarter texel apart, stored as 0.5 + 0.03 curl  (128^2 RG8)
//   weather    R = value-noise FBM (8 cells, 4 oct), G = 0, B = value-noise FBM (4 cells,
//              4 oct), A = 255                                          (512^2 RGBA8)
// The affine output maps give the channels the mean/deviation of the shipped Nubis textures.
//
// The reference-compatible curl (MM_NOISE_REF_CURL) restates ImageUtils.cpp:7-222 with the
// reference's float/double typing and a correctly rounded sinf (mmx::mm_sinf_cr).
#include <cuda_runtime.h>
#include <stdint.h>

#include "mm_internal.h"
#include "mm_math.h"

namespace mm {
namespace noise {

__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

__device__ __forceinline__ uint32_t hash3(int x, int y, int z, uint32_t s) {
    return hash32((uint32_t)x + hash32((uint32_t)y + hash32((uint32_t)z + s)));
}

__device__ __forceinline__ float rand01(uint32_t h) { return (float)(h >> 8) * 0x1p-24f; }

__device__ __forceinline__ uint32_t stream_seed(uint32_t seed, int kind, int ch, int oct) {
    return hash32(seed ^ hash32(0x9E3779B9u * (uint32_t)(1 + kind * 64 + ch * 8 + oct)));
}

// c modulo f; every frequency of the generators is a power of two
__device__ __forceinline__ int wrapi(int c, int f) { return c & (f - 1); }

__device__ __forceinline__ float lattice(int i, int n, int f) {
    return __fdiv_rn((float)((2 * i + 1) * f), (float)(2 * n));
}

__device__ __forceinline__ uint8_t quantize(float v) {
    v = fminf(fmaxf(v, 0.0f), 1.0f);
    return (uint8_t)(int)floorf(v * 255.0f + 0.5f);
}

__device__ float worley3(float qx, float qy, float qz, int f, uint32_t s) {
    const int cx = (int)floorf(qx), cy = (int)floorf(qy), cz = (int)floorf(qz);
    const float fx = qx - (float)cx, fy = qy - (float)cy, fz = qz - (float)cz;
    float best = 4.0f;
#pragma unroll 1
    for (int dz = -1; dz <= 1; ++dz) {
        const uint32_t hz = (uint32_t)wrapi(cz + dz, f) + s;
        const uint32_t hz2 = hash32(hz);
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy) {
            const uint32_t hy = hash32((uint32_t)wrapi(cy + dy, f) + hz2);
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                const uint32_t h = hash32((uint32_t)wrapi(cx + dx, f) + hy);
                const float px = (float)dx + rand01(h);
                const float py = (float)dy + rand01(hash32(h + 0x9E3779B9u));
                const float pz = (float)dz + rand01(hash32(h + 0x3C6EF372u));
                const float ex = px - fx, ey = py - fy, ez = pz - fz;
                const float d2 = (ex * ex + ey * ey) + ez * ez;
                best = fminf(best, d2);
            }
        }
    }
    return 1.0f - fminf(__fsqrt_rn(best), 1.0f);
}

__device__ __forceinline__ float fade(float t) { return t * t * t * (t * (t * 6.0f - 15.0f) + 10.0f); }
__device__ __forceinline__ float lerpf(float a, float b, float t) { return a + t * (b - a); }

// 12 edge gradients (+-1,+-1,0), (+-1,0,+-1), (0,+-1,+-1) in the oracle's table order.
__device__ __forceinline__ float grad3(uint32_t h, float x, float y, float z) {
    const int g = (int)(h % 12u);
    float gx, gy, gz;
    if (g < 4) {
        gx = (g & 1) ? -1.0f : 1.0f;
        gy = (g & 2) ? -1.0f : 1.0f;
        gz = 0.0f;
    } else if (g < 8) {
        gx = (g & 1) ? -1.0f : 1.0f;
        gy = 0.0f;
        gz = (g & 2) ? -1.0f : 1.0f;
    } else {
        gx = 0.0f;
        gy = (g & 1) ? -1.0f : 1.0f;
        gz = (g & 2) ? -1.0f : 1.0f;
    }
    return (gx * x + gy * y) + gz * z;
}

__device__ float perlin3(float qx, float qy, float qz, int f, uint32_t s) {
    const int cx = (int)floorf(qx), cy = (int)floorf(qy), cz = (int)floorf(qz);
    const float x = qx - (float)cx, y = qy - (float)cy, z = qz - (float)cz;
    const int x0 = wrapi(cx, f), x1 = wrapi(cx + 1, f);
    const int y0 = wrapi(cy, f), y1 = wrapi(cy + 1, f);
    const int z0 = wrapi(cz, f), z1 = wrapi(cz + 1, f);
    const float n000 = grad3(hash3(x0, y0, z0, s), x, y, z);
    const float n100 = grad3(hash3(x1, y0, z0, s), x - 1.0f, y, z);
    const float n010 = grad3(hash3(x0, y1, z0, s), x, y - 1.0f, z);
    const float n110 = grad3(hash3(x1, y1, z0, s), x - 1.0f, y - 1.0f, z);
    const float n001 = grad3(hash3(x0, y0, z1, s), x, y, z - 1.0f);
    const float n101 = grad3(hash3(x1, y0, z1, s), x - 1.0f, y, z - 1.0f);
    const float n011 = grad3(hash3(x0, y1, z1, s), x, y - 1.0f, z - 1.0f);
    const float n111 = grad3(hash3(x1, y1, z1, s), x - 1.0f, y - 1.0f, z - 1.0f);
    const float u = fade(x), v = fade(y), w = fade(z);
    const float n00 = lerpf(n000, n100, u), n10 = lerpf(n010, n110, u);
    const float n01 = lerpf(n001, n101, u), n11 = lerpf(n011, n111, u);
    return lerpf(lerpf(n00, n10, v), lerpf(n01, n11, v), w);
}

// 8 gradients (+-1,+-1), (+-1,0), (0,+-1) in the oracle's table order.
__device__ __forceinline__ float grad2(uint32_t h, float x, float y) {
    const int g = (int)(h & 7u);
    float gx, gy;
    if (g < 4) {
        gx = (g & 1) ? -1.0f : 1.0f;
        gy = (g & 2) ? -1.0f : 1.0f;
    } else if (g < 6) {
        gx = (g & 1) ? -1.0f : 1.0f;
        gy = 0.0f;
    } else {
        gx = 0.0f;
        gy = (g & 1) ? -1.0f : 1.0f;
    }
    return gx * x + gy * y;
}

__device__ float perlin2(float qx, float qy, int f, uint32_t s) {
    const int cx = (int)floorf(qx), cy = (int)floorf(qy);
    const float x = qx - (float)cx, y = qy - (float)cy;
    const int x0 = wrapi(cx, f), x1 = wrapi(cx + 1, f), y0 = wrapi(cy, f), y1 = wrapi(cy + 1, f);
    const float n00 = grad2(hash3(x0, y0, 0, s), x, y), n10 = grad2(hash3(x1, y0, 0, s), x - 1.0f, y);
    const float n01 = grad2(hash3(x0, y1, 0, s), x, y - 1.0f), n11 = grad2(hash3(x1, y1, 0, s), x - 1.0f, y - 1.0f);
    const float u = fade(x), v = fade(y);
    return lerpf(lerpf(n00, n10, u), lerpf(n01, n11, u), v);
}

__device__ float value2(float qx, float qy, int f, uint32_t s) {
    const int cx = (int)floorf(qx), cy = (int)floorf(qy);
    const float x = qx - (float)cx, y = qy - (float)cy;
    const int x0 = wrapi(cx, f), x1 = wrapi(cx + 1, f), y0 = wrapi(cy, f), y1 = wrapi(cy + 1, f);
    const float v00 = rand01(hash3(x0, y0, 0, s)), v10 = rand01(hash3(x1, y0, 0, s));
    const float v01 = rand01(hash3(x0, y1, 0, s)), v11 = rand01(hash3(x1, y1, 0, s));
    const float u = x * x * (3.0f - 2.0f * x), v = y * y * (3.0f - 2.0f * y);
    return lerpf(lerpf(v00, v10, u), lerpf(v01, v11, u), v);
}

// ---------------------------------------------------------------- 3D density volumes
//
// A block makes a tile of 32 x 2 x kRun texels (x, y, z).  Its work is split into units of two warps (one
// lane a column of kRun texels): one unit per Worley channel and, for the low-res volume, one for the
// Perlin octaves.  For each octave a unit first hashes the cells its tile can reach into shared memory,
// once per cell instead of 27 times per texel, then every lane takes its 27 neighbours from there.  The
// texels of a column that lie in the same cell along z (8 at a time, 4, 2, or 1: the same for every lane) go
// through a neighbour together: its x and y distances are theirs in common, which leaves a subtraction,
// a product, a sum and a minimum each.  Every float operation is worley3's own, so the texels are the same
// bytes.  Where an octave has more cells in reach than the table holds (more than about half a cell per
// texel), its texels are computed one by one as before.
// Bound by FP32 issue: 27 distances x 12 octaves a texel.  us hashing every cell -> with the tables -> with packed FP32
// operations -> 8 texels at a time: low-res 128^3 1229 -> 226 -> 201 -> 183, 64^3 164 -> 56 -> 52; hi-res 32^3
// 27 -> 11, 64^3 109 -> 27 -> 25 -> 23.
// (Passing over rows of cells no closer than the distance found so far costs what it saves: 232 -> 240.)
constexpr int kCells = 680;         // table entries of a Worley unit: 32 x 2 x 8 texels at 0.55 cells a texel
constexpr int kPerlinCells = 256;   // of the Perlin unit, whose octaves are the coarse ones

// Two floats in one register pair; the packed operations round each half as the scalar ones do.
__device__ __forceinline__ unsigned long long pair(float a, float b) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpair(unsigned long long v, float& a, float& b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// The square, rounded by itself: a packed product followed by a packed sum is contracted by the assembler
// even at -fmad=false, a product already fused with + 0 is not.
__device__ __forceinline__ unsigned long long square2(unsigned long long a) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(r) : "l"(a), "l"(0ull));
    return r;
}

// Minimum squared distance (at most 1) to the 27 neighbours for M texels that share their cell; the
// texels' fractions are (fx, fy, fz[m]) and `at` is the table entry of neighbour (-1, -1, -1).  The
// distances along x and y, and those of two texels along z, go through packed FP32 operations.
template <int M>
__device__ __forceinline__ void nearest(const float* at, int cells, int nx, int nxy, float fx, float fy, const float* fz,
                                        float* best) {
    unsigned long long nz[M / 2 + 1];
#pragma unroll
    for (int m = 0; m < M; ++m) best[m] = 1.0f;
#pragma unroll
    for (int m = 0; m + 1 < M; m += 2) nz[m / 2] = pair(-fz[m], -fz[m + 1]);
    const unsigned long long nfxy = pair(-fx, -fy);
#pragma unroll 1
    for (int dz = 0; dz < 3; ++dz) {
        const float oz = (float)(dz - 1);
#pragma unroll
        for (int dy = 0; dy < 3; ++dy) {
            const float* row = at + dy * nx;
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                unsigned long long e = add2(pair(row[dx], row[cells + dx]), pair((float)(dx - 1), (float)(dy - 1)));
                e = add2(e, nfxy);
                e = square2(e);
                float ex, ey;
                unpair(e, ex, ey);
                const float exy = ex + ey;
                const float pz = oz + row[2 * cells + dx];
                if (M == 1) {
                    const float ez = pz - fz[0];
                    best[0] = fminf(best[0], exy + ez * ez);
                } else {
                    const unsigned long long pz2 = pair(pz, pz), exy2 = pair(exy, exy);
#pragma unroll
                    for (int m = 0; m + 1 < M; m += 2) {
                        unsigned long long ez = add2(pz2, nz[m / 2]);
                        ez = add2(exy2, square2(ez));
                        float d0, d1;
                        unpair(ez, d0, d1);
                        best[m] = fminf(best[m], d0);
                        best[m + 1] = fminf(best[m + 1], d1);
                    }
                }
            }
        }
        at += nxy;
    }
}

// Barrier of a unit's two warps: units take their octaves at their own pace.
__device__ __forceinline__ void unit_sync(int unit) { asm volatile("bar.sync %0, 64;" ::"r"(unit + 1) : "memory"); }

template <int kRun>
__global__ void __launch_bounds__(320) volume_kernel(int kind, uint32_t seed, int n, uchar4* out) {
    constexpr unsigned full = 0xffffffffu;
    __shared__ float s_table[4 * 3 * kCells + 3 * kPerlinCells];
    __shared__ float s_sum[kRun][320];  // each thread's own octave sums, and the Perlin unit's for unit 0
    __shared__ __align__(4) uint8_t s_out[kRun][64][4];
    const bool low = kind == MM_NOISE_LOWRES_PERLIN_WORLEY;
    const int worleys = low ? 4 : 3;
    const int unit = threadIdx.x >> 6, t = threadIdx.x & 63, lane = t & 31;
    const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 2, k0 = blockIdx.z * kRun;
    const int i = min(i0 + lane, n - 1);  // columns outside: a neighbour's
    const bool perlin = unit == worleys;
    const int cap = perlin ? kPerlinCells : kCells;
    float* const table = s_table + unit * 3 * kCells;
    // first octave of the unit's channel: low-res R (and the Perlin octaves) 4, G/B/A 4/8/16; hi-res 2/4/8
    const int f0 = low ? (unit == 0 || perlin ? 4 : 4 << (unit - 1)) : 2 << unit;
    float amp = 1.0f, norm = 0.0f;
#pragma unroll 1
    for (int o = 0; o < 3; ++o) {
        const int f = f0 << o;
        const uint32_t s = stream_seed(seed, kind, perlin ? 0 : unit, perlin ? 4 + o : o);
        // lattice points: this lane's x, the tile's two y and (lane r) its z
        const float qx = lattice(i, n, f), qy0 = lattice(j0, n, f), qy1 = lattice(min(j0 + 1, n - 1), n, f);
        const float ql = lattice(min(k0 + min(lane, kRun - 1), n - 1), n, f);
        const float qy = t < 32 ? qy0 : qy1;
        const float fx = qx - floorf(qx), fy = qy - floorf(qy), fl = ql - floorf(ql);
        const int cx = (int)floorf(qx), cy = (int)floorf(qy), cl = (int)floorf(ql);
        // cells in reach of the tile: x0 .. x0 + nx - 1 and so on
        const int x0 = __shfl_sync(full, cx, 0) - 1, nx = __shfl_sync(full, cx, 31) - x0 + 2;
        const int y0 = (int)floorf(qy0) - 1, ny = (int)floorf(qy1) - y0 + 2;
        const int z0 = __shfl_sync(full, cl, 0) - 1, nz = __shfl_sync(full, cl, 31) - z0 + 2;
        const int nxy = nx * ny, cells = nxy * nz;
        const bool tabled = cells <= cap;
        if (o) unit_sync(unit);  // the last octave's entries are read
        if (tabled) {
            // c / nxy and q / nx by multiplication: exact for entries below 2^16
            const uint32_t by_xy = 0xffffffffu / (uint32_t)nxy + 1u, by_x = 0xffffffffu / (uint32_t)nx + 1u;
            for (int c = t; c < cells; c += 64) {
                const int z = (int)__umulhi((uint32_t)c, by_xy), q = c - z * nxy;
                const int y = (int)__umulhi((uint32_t)q, by_x), x = q - y * nx;
                const uint32_t h = hash3(wrapi(x0 + x, f), wrapi(y0 + y, f), wrapi(z0 + z, f), s);
                if (perlin) {  // the gradient of lattice point (x, y, z)
                    table[c] = grad3(h, 1.0f, 0.0f, 0.0f);
                    table[cap + c] = grad3(h, 0.0f, 1.0f, 0.0f);
                    table[2 * cap + c] = grad3(h, 0.0f, 0.0f, 1.0f);
                } else {  // the feature point of cell (x, y, z)
                    table[c] = rand01(h);
                    table[cap + c] = rand01(hash32(h + 0x9E3779B9u));
                    table[2 * cap + c] = rand01(hash32(h + 0x3C6EF372u));
                }
            }
        }
        unit_sync(unit);
        const float* const column = table + (cy - 1 - y0) * nx + (cx - 1 - x0);  // neighbour (-1, -1), plane z0
        const float weight = o == 0 ? 0.625f : (o == 1 ? 0.25f : 0.125f);
        if (perlin) {
            const float u = fade(fx), v = fade(fy);
#pragma unroll 1
            for (int r = 0; r < kRun; ++r) {
                const float fz = __shfl_sync(full, fl, r);
                float p;
                if (tabled) {
                    const float* at = column + (__shfl_sync(full, cl, r) - z0) * nxy + nx + 1;
                    float g[8];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float* e = at + (c & 1) + (c & 2 ? nx : 0) + (c & 4 ? nxy : 0);
                        const float x = c & 1 ? fx - 1.0f : fx, y = c & 2 ? fy - 1.0f : fy, z = c & 4 ? fz - 1.0f : fz;
                        g[c] = (e[0] * x + e[kPerlinCells] * y) + e[2 * kPerlinCells] * z;
                    }
                    const float w = fade(fz);
                    p = lerpf(lerpf(lerpf(g[0], g[1], u), lerpf(g[2], g[3], u), v),
                              lerpf(lerpf(g[4], g[5], u), lerpf(g[6], g[7], u), v), w);
                } else {
                    p = perlin3(qx, qy, __shfl_sync(full, ql, r), f, s);
                }
                s_sum[r][threadIdx.x] = (o ? s_sum[r][threadIdx.x] : 0.0f) + amp * p;
            }
            norm += amp;
            amp *= 0.5f;
        } else if (tabled) {
            auto add = [&](int r, float best) {
                const float w = weight * (1.0f - fminf(__fsqrt_rn(best), 1.0f));
                s_sum[r][threadIdx.x] = o ? s_sum[r][threadIdx.x] + w : w;
            };
#pragma unroll 1
            for (int r = 0; r < kRun;) {  // the next 8, 4, 2 or 1 texels of the column that share a cell
                const int c = __shfl_sync(full, cl, r);
                const bool two = r + 1 < kRun && __shfl_sync(full, cl, r + 1) == c;
                const bool four = r + 3 < kRun && __shfl_sync(full, cl, r + 3) == c;
                const float* at = column + (c - 1 - z0) * nxy;
                if constexpr (kRun == 8) {
                    if (r == 0 && __shfl_sync(full, cl, 7) == c) {
                        float fz[8], best[8];
#pragma unroll
                        for (int m = 0; m < 8; ++m) fz[m] = __shfl_sync(full, fl, m);
                        nearest<8>(at, kCells, nx, nxy, fx, fy, fz, best);
#pragma unroll
                        for (int m = 0; m < 8; ++m) add(m, best[m]);
                        break;
                    }
                }
                float fz[4], best[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) fz[m] = __shfl_sync(full, fl, r + m);
                if (four) {
                    nearest<4>(at, kCells, nx, nxy, fx, fy, fz, best);
#pragma unroll
                    for (int m = 0; m < 4; ++m) add(r + m, best[m]);
                    r += 4;
                } else if (two) {
                    nearest<2>(at, kCells, nx, nxy, fx, fy, fz, best);
                    add(r, best[0]);
                    add(r + 1, best[1]);
                    r += 2;
                } else {
                    nearest<1>(at, kCells, nx, nxy, fx, fy, fz, best);
                    add(r, best[0]);
                    r += 1;
                }
            }
        } else {
#pragma unroll 1
            for (int r = 0; r < kRun; ++r) {
                const float w = weight * worley3(qx, qy, __shfl_sync(full, ql, r), f, s);
                s_sum[r][threadIdx.x] = o ? s_sum[r][threadIdx.x] + w : w;
            }
        }
    }
    // ---- texels: R of the low-res volume needs the Perlin unit's sums
    if (perlin) {
#pragma unroll 1
        for (int r = 0; r < kRun; ++r)
            s_sum[r][threadIdx.x] = __fdiv_rn(s_sum[r][threadIdx.x], norm) * 0.5f + 0.5f;
    }
    __syncthreads();
    if (!perlin) {
#pragma unroll 1
        for (int r = 0; r < kRun; ++r) {
            const float wf = s_sum[r][threadIdx.x];
            if (low && unit == 0) {
                const float pw = __fdiv_rn(s_sum[r][4 * 64 + t] - (wf - 1.0f), 1.0f - (wf - 1.0f));
                s_out[r][t][0] = quantize(1.64f * pw + -0.593f);
            } else {
                s_out[r][t][unit] = quantize(0.866f * wf + 0.271f);
            }
            if (!low && unit == 0) s_out[r][t][3] = 0;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kRun * 64; e += blockDim.x) {
        const int x = i0 + (e & 31), y = j0 + ((e >> 5) & 1), z = k0 + (e >> 6);
        if (x < n && y < n && z < n)
            out[((size_t)z * n + y) * n + x] = *reinterpret_cast<const uchar4*>(s_out[e >> 6][e & 63]);
    }
}

__device__ float curl_potential(float qx, float qy, uint32_t seed) {
    float sum = 0.0f, amp = 1.0f, norm = 0.0f;
#pragma unroll 1
    for (int o = 0; o < 5; ++o) {
        const int fo = 4 << o;
        sum += amp * perlin2(qx * (float)fo, qy * (float)fo, fo, stream_seed(seed, MM_NOISE_CURL2D, 0, o));
        norm += amp;
        amp *= 0.5f;
    }
    return __fdiv_rn(sum, norm);
}

// Four lanes a texel, one potential each: 128^2 texels are too few to fill the GPU with one thread each
// (12.5 -> 6.4 us).
__global__ void __launch_bounds__(256) curl_kernel(uint32_t seed, int w, int h, uchar2* out) {
    const int part = threadIdx.x & 3;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 2);
    const int j = blockIdx.y * 8 + threadIdx.y;
    const int ic = min(i, w - 1), jc = min(j, h - 1);
    // x + a quarter texel, x - a quarter, y + a quarter, y - a quarter
    const float x = part == 0   ? __fdiv_rn((float)(4 * ic + 3), (float)(4 * w))
                    : part == 1 ? __fdiv_rn((float)(4 * ic + 1), (float)(4 * w))
                                : __fdiv_rn((float)(2 * ic + 1), (float)(2 * w));
    const float y = part == 2   ? __fdiv_rn((float)(4 * jc + 3), (float)(4 * h))
                    : part == 3 ? __fdiv_rn((float)(4 * jc + 1), (float)(4 * h))
                                : __fdiv_rn((float)(2 * jc + 1), (float)(2 * h));
    const float p = curl_potential(x, y, seed);
    const float other = __shfl_xor_sync(0xffffffffu, p, 1);
    const float d = (p - other) * (float)(part == 0 ? 2 * w : 2 * h);  // lanes 0 and 2: dp/dx, dp/dy
    const float dpy = __shfl_down_sync(0xffffffffu, d, 2);
    if (part == 0 && i < w && j < h)
        out[(size_t)j * w + i] = make_uchar2(quantize(0.5f + 0.03f * dpy), quantize(0.5f - 0.03f * d));
}

__global__ void __launch_bounds__(256) weather_kernel(uint32_t seed, int w, int h, uchar4* out) {
    const int i = blockIdx.x * 32 + threadIdx.x;
    const int j = blockIdx.y * 8 + threadIdx.y;
    if (i >= w || j >= h) return;
    float ch[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int f = c == 0 ? 8 : 4;
        float sum = 0.0f, amp = 1.0f, norm = 0.0f;
#pragma unroll 1
        for (int o = 0; o < 4; ++o) {
            const int fo = f << o;
            sum += amp * value2(lattice(i, w, fo), lattice(j, h, fo), fo, stream_seed(seed, MM_NOISE_WEATHER, c, o));
            norm += amp;
            amp *= 0.5f;
        }
        ch[c] = __fdiv_rn(sum, norm);
    }
    out[(size_t)j * w + i] = make_uchar4(quantize(ch[0]), 0, quantize(ch[1]), 255);
}

// ---------------------------------------------------------------- reference-compatible curl

__constant__ float kRefBasis[12][3] = {
    {0.7071f, 0.7071f, 0.f},  {0.7071f, -0.7071f, 0.f},  {-0.7071f, 0.7071f, 0.f},
    {-0.7071f, -0.7071f, 0.f}, {0.7071f, 0.f, 0.7071f},  {0.7071f, 0.f, -0.7071f},
    {-0.7071f, 0.f, 0.7071f},  {-0.7071f, 0.f, -0.7071f}, {0.f, 0.7071f, 0.7071f},
    {0.f, 0.7071f, -0.7071f},  {0.f, -0.7071f, 0.7071f},  {0.f, -0.7071f, -0.7071f},
};

__device__ __forceinline__ int ref_index(float x, float y, float z) {  // ImageUtils.cpp:25-34
    float d = x * 12.9898f + y * 78.233f;
    d = d + z * 47.387f;
    float n = mmx::mm_sinf_cr(d) * 43758.5453f;
    n = n - floorf(n);
    return (int)floorf(12.f * n);
}

__device__ __forceinline__ float ref_dot(int g, float rx, float ry, float rz) {
    float a = kRefBasis[g][0] * rx + kRefBasis[g][1] * ry;
    return a + kRefBasis[g][2] * rz;
}

__device__ __forceinline__ float ref_lerp(float a, float b, float t) {  // ImageUtils.cpp:36-38
    return (float)((1.0 - (double)t) * (double)a + (double)(t * b));
}

__device__ float ref_perlin(float px, float py, float pz, float freq) {  // ImageUtils.cpp:41-73
    px *= freq;
    py *= freq;
    pz *= freq;
    const float fx = floorf(px), fy = floorf(py), fz = floorf(pz);
    const float rx = px - fx, ry = py - fy, rz = pz - fz;
    const float ux = rx * rx * rx * (rx * (rx * 6.0f - 15.0f) + 10.0f);
    const float uy = ry * ry * ry * (ry * (ry * 6.0f - 15.0f) + 10.0f);
    const float uz = rz * rz * rz * (rz * (rz * 6.0f - 15.0f) + 10.0f);
    float f1x = fx + 1.f, f1y = fy + 1.f, f1z = fz + 1.f;
    if (fabsf(f1x - freq) < 0.001f) f1x = freq;
    if (fabsf(f1y - freq) < 0.001f) f1y = freq;
    if (fabsf(f1z - freq) < 0.001f) f1z = freq;
    const float nnn = ref_dot(ref_index(fx, fy, fz), rx, ry, rz);
    const float nnp = ref_dot(ref_index(fx, fy, f1z), rx, ry, rz - 1.f);
    const float npn = ref_dot(ref_index(fx, f1y, fz), rx, ry - 1.f, rz);
    const float npp = ref_dot(ref_index(fx, f1y, f1z), rx, ry - 1.f, rz - 1.f);
    const float pnn = ref_dot(ref_index(f1x, fy, fz), rx - 1.f, ry, rz);
    const float pnp = ref_dot(ref_index(f1x, fy, f1z), rx - 1.f, ry, rz - 1.f);
    const float ppn = ref_dot(ref_index(f1x, f1y, fz), rx - 1.f, ry - 1.f, rz);
    const float ppp = ref_dot(ref_index(f1x, f1y, f1z), rx - 1.f, ry - 1.f, rz - 1.f);
    const float nn = ref_lerp(nnn, pnn, ux), np = ref_lerp(nnp, pnp, ux);
    const float pn = ref_lerp(npn, ppn, ux), pp = ref_lerp(npp, ppp, ux);
    const float n = ref_lerp(nn, pn, uy), q = ref_lerp(np, pp, uy);
    return ref_lerp(n, q, uz);
}

__device__ float ref_fbm(float x, float y, float z, float freq) {  // ImageUtils.cpp:75-87, 4 octaves
    float noise = 0.0f, weight = 1.0f, total = 0.0f;
#pragma unroll 1
    for (int i = 0; i < 4; i++) {
        total += weight;
        noise += weight * ref_perlin(x, y, z, freq);
        freq *= 2.0f;
        weight *= 0.4f;
    }
    return __fdiv_rn(noise, total);
}

__device__ __forceinline__ float ref_quot(float fa, float fb) {
    const double EPS = 0.0005;
    return (float)((double)(fb - fa) / (double)(2.f * EPS));
}

// One thread per texel: the curl vector of ImageUtils.cpp:130-169 at (col/128, row/128).
__global__ void __launch_bounds__(128) ref_curl_vectors(float* curls) {
    const int col = threadIdx.x, row = blockIdx.x;
    const double EPS = 0.0005;
    const float px = __fdiv_rn((float)col, 128.0f), py = __fdiv_rn((float)row, 128.0f);
    const float xm = (float)((double)px - EPS), xp = (float)((double)px + EPS);
    const float ym = (float)((double)py - EPS), yp = (float)((double)py + EPS);
    const float F = 3.f;
    const float dydx = ref_quot(ref_fbm(xm, py, 0.5f, F), ref_fbm(xp, py, 0.5f, F));
    const float dxdy = ref_quot(ref_fbm(px, ym, 0.5f, F), ref_fbm(px, yp, 0.5f, F));
    const float dxdz = ref_quot(ref_fbm(px, 0.5f, ym, F), ref_fbm(px, 0.5f, yp, F));
    const float dzdx = ref_quot(ref_fbm(xm, 0.5f, py, F), ref_fbm(xp, 0.5f, py, F));
    const float dzdy = ref_quot(ref_fbm(0.5f, ym, px, F), ref_fbm(0.5f, yp, px, F));
    const float dydz = ref_quot(ref_fbm(0.5f, py, xm, F), ref_fbm(0.5f, py, xp, F));
    float* c = curls + 3 * ((size_t)row * 128 + col);
    c[0] = dzdy - dydz;
    c[1] = dxdz - dzdx;
    c[2] = dydx - dxdy;
}

// One block: per-channel min/max over the 128x128 vectors (ImageUtils.cpp:179-198), then the
// remap to [0,1] and 8-bit rounding (ImageUtils.cpp:200-219).
__global__ void __launch_bounds__(1024) ref_curl_normalize(const float* curls, float* bounds, uchar4* out) {
    __shared__ float s_lo[3][32], s_hi[3][32];
    float lo[3] = {3.402823466e+38f, 3.402823466e+38f, 3.402823466e+38f};
    float hi[3] = {-3.402823466e+38f, -3.402823466e+38f, -3.402823466e+38f};
    for (int i = threadIdx.x; i < 128 * 128; i += blockDim.x)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            lo[k] = fminf(lo[k], curls[3 * i + k]);
            hi[k] = fmaxf(hi[k], curls[3 * i + k]);
        }
#pragma unroll
    for (int k = 0; k < 3; ++k)
        for (int o = 16; o > 0; o >>= 1) {
            lo[k] = fminf(lo[k], __shfl_xor_sync(0xffffffffu, lo[k], o));
            hi[k] = fmaxf(hi[k], __shfl_xor_sync(0xffffffffu, hi[k], o));
        }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
        for (int k = 0; k < 3; ++k) {
            s_lo[k][warp] = lo[k];
            s_hi[k][warp] = hi[k];
        }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int k = threadIdx.x;
        float a = s_lo[k][0], b = s_hi[k][0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
            a = fminf(a, s_lo[k][w]);
            b = fmaxf(b, s_hi[k][w]);
        }
        bounds[k] = a;
        bounds[3 + k] = b;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 128 * 128; i += blockDim.x) {
        unsigned char b[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float m = 0.f + (__fdiv_rn(curls[3 * i + k] - bounds[k], bounds[3 + k] - bounds[k]) * (1.f - 0.f));
            b[k] = (unsigned char)(int)roundf(m * 255.f);
        }
        out[i] = make_uchar4(b[0], b[1], b[2], 255);
    }
}

__global__ void hash3_kernel(const int* xyz, uint32_t s, size_t n, uint32_t* out) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = hash3(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], s);
}

__global__ void ref_hash_kernel(const float* xyz, size_t n, float* out) {
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float d = xyz[3 * i] * 12.9898f + xyz[3 * i + 1] * 78.233f;
    d = d + xyz[3 * i + 2] * 47.387f;
    float v = mmx::mm_sinf_cr(d) * 43758.5453f;
    out[i] = v - floorf(v);
}

}  // namespace noise

int launch_hash_stage(int which, const void* in, uint32_t seed, size_t n, void* out, cudaStream_t s) {
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (which == 0)
        noise::hash3_kernel<<<blocks, 256, 0, s>>>((const int*)in, seed, n, (uint32_t*)out);
    else
        noise::ref_hash_kernel<<<blocks, 256, 0, s>>>((const float*)in, n, (float*)out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "hash stage launch");
    count_launch();
    return MM_OK;
}

int launch_noise(int kind, uint32_t seed, int w, int h, int d, uint8_t* out, cudaStream_t s) {
    using namespace noise;
    switch (kind) {
        case MM_NOISE_LOWRES_PERLIN_WORLEY:
        case MM_NOISE_HIRES_WORLEY: {
            const int threads = kind == MM_NOISE_LOWRES_PERLIN_WORLEY ? 320 : 192;
            uchar4* texels = reinterpret_cast<uchar4*>(out);
            // Texels of a column: longer columns hash fewer cells a texel, shorter ones make more blocks.
            // 8 / 4 / 2 / 1 texels, us: low-res 128^3 224 / 261 / 388 / -, 64^3 64 / 58 / 62 / -, 40^3 - / 35 /
            // 39 / 47, 24^3 - / 23 / 15 / 15; hi-res 64^3 27 / 29 / 37 / -, 48^3 - / 21 / 27 / 37, 32^3 - / 17 /
            // 11 / 13, 16^3 - / 18 / 13 / 9.
            const int run = w >= 64 ? 8 : (w >= 40 ? 4 : (w >= 28 ? 2 : 1));
            const dim3 grid((w + 31) / 32, (h + 1) / 2, (d + run - 1) / run);
            switch (run) {
                case 8: volume_kernel<8><<<grid, threads, 0, s>>>(kind, seed, w, texels); break;
                case 4: volume_kernel<4><<<grid, threads, 0, s>>>(kind, seed, w, texels); break;
                case 2: volume_kernel<2><<<grid, threads, 0, s>>>(kind, seed, w, texels); break;
                default: volume_kernel<1><<<grid, threads, 0, s>>>(kind, seed, w, texels); break;
            }
            break;
        }
        case MM_NOISE_CURL2D:
            curl_kernel<<<dim3((w + 7) / 8, (h + 7) / 8), dim3(32, 8), 0, s>>>(seed, w, h, reinterpret_cast<uchar2*>(out));
            break;
        case MM_NOISE_WEATHER:
            weather_kernel<<<dim3((w + 31) / 32, (h + 7) / 8), dim3(32, 8), 0, s>>>(seed, w, h,
                                                                                    reinterpret_cast<uchar4*>(out));
            break;
        default:
            return fail(MM_ERR_INVALID_ARGUMENT, "launch_noise: kind %d", kind);
    }
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "noise kernel launch");
    count_launch();
    return MM_OK;
}

int launch_ref_curl(uint8_t* out_rgba, float* scratch_curl, float* scratch_bounds, cudaStream_t s) {
    noise::ref_curl_vectors<<<128, 128, 0, s>>>(scratch_curl);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "ref_curl_vectors launch");
    noise::ref_curl_normalize<<<1, 1024, 0, s>>>(scratch_curl, scratch_bounds, reinterpret_cast<uchar4*>(out_rgba));
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "ref_curl_normalize launch");
    count_launch(2);
    return MM_OK;
}

}  // namespace mm
