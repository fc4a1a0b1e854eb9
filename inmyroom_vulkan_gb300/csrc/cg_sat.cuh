// A filter for the 15-axis box test of cg_device.cuh (sat): for each axis it
// decides, from FP32 values with a rounding bound, what the reference's own
// FP32 expression (overlap_on) must answer, or that it cannot tell; only the
// axes left open are evaluated with the reference's expression. The verdict
// is therefore the reference's, bit for bit.
//
// The reference builds each axis L = x * y (a cross product) and projects
// both boxes' centres and half-extents on it: about 60 instructions an axis,
// 900 a box pair without FMA contraction. All those projections are triple
// products of the boxes' edge vectors, and the same few occur on several
// axes: with the boxes' face normals N_k, M_k (cross products of their edges),
//   face axis N_i:    |x_i . N_i| + sum_j |y_j . N_i|           against |d . N_i|
//   edge x_i x y_j:   sum_{m != i} |y_j . N_m| + sum_{m != j} |x_i . M_m|
//                                                              against |y_j . (d x x_i)|
// (d the difference of the centres), so a box pair takes 9 cross products
// and 35 dot products, with FMA: about 280 instructions. No orthogonality of
// the boxes' edges is assumed. The traversal of 10,000 uneven queries (36 M
// box pairs) took 2,268 us without the filter and 1,474 with it.
//
// Bound. Let u = 2^-24, |.| the 1-norm and W the sum of the 1-norms of both
// centres and all six edges. For an axis L = x * y every component of the
// reference's rounded L is within 2u (|x_p y_q| + |x_q y_p|) of the exact one,
// each of its dot products within 3u of its terms' magnitudes, the extents'
// sums, the interval ends and their comparison add 3u of W's share: the
// margin it compares, (sum of extents) - |difference of centre projections|,
// is within 8u W |x||y| of the exact margin (second-order terms included).
// The filter's own margin, three chained roundings per triple product, a
// rounded d and four sums, is within 9u W |x||y| of it. kSatK = 32u covers the
// two together with room for the bound's own rounding; the added constant
// covers products that underflow. A NaN makes every comparison with the bound
// false: the axis stays open. An infinity does not (the bound is a 2^-19th of
// products that the margin is a sum of, and may be finite beside it), so from
// W = 1e12 on, NaN included, all axes stay open: below it no product, sum or
// interval end of either side exceeds 8 W^3 = 8e36.
#pragma once

#include <cstdint>

#include "cg_device.cuh"

namespace cg {

// Axis k (0..14) of the SAT in the reference's order: a's face normals
// (v x w, u x w, u x v), b's, then a_i x b_j; true when the boxes overlap on
// it. The SAT verdict is the conjunction over k, whatever lanes compute it.
__device__ __forceinline__ bool sat_axis(const Box& a, const Box& b, uint32_t k) {
    float3 x, y;
    if (k < 6u) {
        const bool onA = k < 3u;
        const uint32_t f = onA ? k : k - 3u;
        const float3 u = onA ? a.u : b.u, v = onA ? a.v : b.v, w = onA ? a.w : b.w;
        x = f == 0u ? v : u;
        y = f == 2u ? v : w;
    } else {
        const uint32_t i = (k - 6u) / 3u, j = (k - 6u) % 3u;
        x = i == 0u ? a.u : (i == 1u ? a.v : a.w);
        y = j == 0u ? b.u : (j == 1u ? b.v : b.w);
    }
    return overlap_on(a, b, cross3(x, y));
}

constexpr float kSatK = 32.0f * 0x1p-24f;
constexpr float kSatTiny = 0x1p-120f;
constexpr float kSatMax = 1e12f;
constexpr float kSurfaceTiny = 0x1p-70f, kSurfaceMax = 1e18f;

__device__ __forceinline__ float norm1_3(float3 p) { return (fabsf(p.x) + fabsf(p.y)) + fabsf(p.z); }
__device__ __forceinline__ float fdot(float3 a, float3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ float3 fcross(float3 a, float3 b) {
    return make_float3(fmaf(a.y, b.z, -(b.y * a.z)), fmaf(a.z, b.x, -(b.z * a.x)), fmaf(a.x, b.y, -(b.x * a.y)));
}

// |p| with the hardware's approximate square root (2^-23 relative).
__device__ __forceinline__ float norm_approx(float3 p) {
    float r;
#ifdef __CUDA_ARCH__
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(fdot(p, p)));
#else
    r = sqrtf(fdot(p, p));
#endif
    return r;
}

// A box with what the filter needs of it: its face normals (v x w, u x w,
// u x v), its volume |u . (v x w)|, its edges' 1-norms, its share of W.
struct SatBox {
    Box b;
    float3 nu, nv, nw;
    float vol, lu, lv, lw, W;
};

__device__ __forceinline__ SatBox sat_box(const Box& b) {
    SatBox s;
    s.b = b;
    s.nu = fcross(b.v, b.w);
    s.nv = fcross(b.u, b.w);
    s.nw = fcross(b.u, b.v);
    s.vol = fabsf(fdot(b.u, s.nu));
    s.lu = norm1_3(b.u);
    s.lv = norm1_3(b.v);
    s.lw = norm1_3(b.w);
    s.W = norm1_3(b.c) + ((s.lu + s.lv) + s.lw);
    return s;
}

// Paralgram::GetSurface of the box (cg::surface) from its normals, and how far
// that can be from the reference's FP32 value: each normal's components are
// within 2u, as the reference's are, of exact ones bounded by its edges'
// 1-norms; the norms and their sum add at most 8u. Squares that underflow put
// a squared norm off by up to 2^-148 and its root by 2^-74: six roots, the
// reference's among them, doubled, by less than kSurfaceTiny. Where squares
// may overflow (the products of 1-norms bound the normals) the error has no
// limit: one side's sum may be finite beside an infinite one.
__device__ __forceinline__ float sat_surface(const SatBox& s, float& err) {
    const float q = norm_approx(s.nu) + norm_approx(s.nv) + norm_approx(s.nw);
    const float l = fmaf(s.lu, s.lv, fmaf(s.lu, s.lw, s.lv * s.lw));
    err = l < kSurfaceMax ? fmaf(kSatK, l, kSurfaceTiny) : HUGE_VALF;
    return 2.0f * q;
}

// The filter over all 15 axes. Returns true when some axis certainly
// separates the boxes; else `open` has bit k set for each axis k (in the
// reference's order with a = x, b = y, the numbering of sat_axis) that the
// filter could not decide, and every other axis certainly overlaps.
__device__ __forceinline__ bool sat_filter(const SatBox& x, const SatBox& y, unsigned& open) {
    const float3 d = make_float3(y.b.c.x - x.b.c.x, y.b.c.y - x.b.c.y, y.b.c.z - x.b.c.z);
    const float W = x.W + y.W;
    const float K = kSatK * W, T = fmaf(kSatTiny, W, kSatTiny);
    bool sep = false;
    unsigned m = 0;
    auto axis = [&](int k, float extents, float dist, float bound) {
        const float s = extents - fabsf(dist);
        sep = sep || s < -bound;
        if (!(s > bound)) m |= 1u << k;
    };
    // |y_j . N_i| of x's normals, |x_i . M_j| of y's
    const float3 xe[3] = {x.b.u, x.b.v, x.b.w}, ye[3] = {y.b.u, y.b.v, y.b.w};
    const float3 N[3] = {x.nu, x.nv, x.nw}, M[3] = {y.nu, y.nv, y.nw};
    const float xl[3] = {x.lu, x.lv, x.lw}, yl[3] = {y.lu, y.lv, y.lw};
    float g[3][3], h[3][3];  // g[i][j] = |N_i . y_j|, h[i][j] = |x_i . M_j|
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            g[i][j] = fabsf(fdot(N[i], ye[j]));
            h[i][j] = fabsf(fdot(xe[i], M[j]));
        }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int p = i == 0 ? 1 : 0, q = i == 2 ? 1 : 2;  // the edges that span the face
        axis(i, x.vol + ((g[i][0] + g[i][1]) + g[i][2]), fdot(d, N[i]), fmaf(K * xl[p], xl[q], T));
        axis(3 + i, y.vol + ((h[0][i] + h[1][i]) + h[2][i]), fdot(d, M[i]), fmaf(K * yl[p], yl[q], T));
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const float3 e = fcross(d, xe[i]);
        const float ki = K * xl[i];
        const int i1 = i == 0 ? 1 : 0, i2 = i == 2 ? 1 : 2;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const int j1 = j == 0 ? 1 : 0, j2 = j == 2 ? 1 : 2;
            axis(6 + 3 * i + j, (g[i1][j] + g[i2][j]) + (h[i][j1] + h[i][j2]), fdot(ye[j], e), fmaf(ki, yl[j], T));
        }
    }
    const bool sane = W < kSatMax;
    open = sane ? m : 0x7fffu;
    return sane && sep;
}

}  // namespace cg
