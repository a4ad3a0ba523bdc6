/*
 * composite_common.cuh - pixel blocking and the splat reach test shared by
 * the forward and backward compositors.
 */
#pragma once

#include "splat_common.cuh"

namespace lumen {

/* Pairs of floats in a 64-bit register and the packed FP32 operations of
 * sm_100: one instruction for two operations, each rounded on its own. The
 * product is written mul.rn: a fused multiply-add with a constant -0 addend
 * is simplified to a product and then contracted with a following sum. */
using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f32x2 splat2(float v) { return pack2(v, v); }
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

/* A tile as 4x4 blocks of 4x4 pixels. */
constexpr int kBlocks = 16;

/* Bit 4 * row + column set when the splat may reach the blend threshold at
 * some pixel centre of that 4x4-pixel block of the tile; *finite tells that
 * no power formed at the tile's pixels overflows or is NaN.
 *
 * A pixel is blended only if power <= 4.5 and opacity * exp(-power) >= 1/255
 * (compositor.mojo:62-89, :33-35), i.e. q(x, y) = a x^2 + 2 b x y + c y^2 <=
 * 2 min(4.5, ln(255 opacity)) around the splat's centre. thr is that bound
 * with a 0.1% + 0.01 margin and one for the rounding of the blend's power and
 * of the steps below: each is within a few units in the last place of the sum
 * of the absolute terms, |a| x^2 + 2 |b x y| + |c| y^2 <= S (x^2 + y^2) with S
 * = |a| + |c| + 2 |b|, so 4e-6 S R^2 (R^2 bounding x^2 + y^2 over the tile's
 * pixel centres, about 64 float ulps) covers them. It matters only for
 * needle-like splats, whose terms cancel. Culling therefore never removes a
 * splat that the per-pixel loop would blend.
 *
 * Each band of four pixel rows gets the x interval that the ellipse q = thr
 * covers within it: the right edge x+(y) = -(b/a) y + sqrt(thr/a - (det/a^2)
 * y^2) is concave with its maximum at y_r = -b sqrt(thr / (det c)), so its
 * maximum over the band is at y_r clamped to the band, and likewise the left
 * edge's minimum at -y_r clamped. Outside the ellipse the square root is NaN,
 * which the clamps below turn into an empty interval. The interval is widened
 * by 0.2% of the ellipse's half width: an error of d in y_r moves the edge by
 * about (d^2 / 2) (a c / det) of the half width, and d <= 2^-24 a c / det,
 * which is below 0.2% for a c <= 1e4 det.
 * Splats beyond that (needles), and those whose numbers leave the range in
 * which the formulas hold, get every block. 16 blocks cost about 150
 * instructions, where the minima of q over 8 blocks of 8x4 cost about 200. */
__device__ __forceinline__ unsigned int reach_blocks(float4 geo, float4 con, float tile_x0, float tile_y0,
                                                     bool* finite) {
    const float a = con.x, b = con.y, c = con.z, op = geo.w;
    const float x0 = tile_x0 + 0.5f - geo.x, x1 = x0 + (float)(kTile - 1);
    const float y0 = tile_y0 + 0.5f - geo.y, y1 = y0 + (float)(kTile - 1);
    const float r2 = fmaxf(x0 * x0, x1 * x1) + fmaxf(y0 * y0, y1 * y1);
    const float spread = (fabsf(a) + fabsf(c) + 2.0f * fabsf(b)) * r2;
    *finite = spread < 1e30f && op < 1e30f;
    const float ac = a * c, det = __fmaf_rn(-b, b, ac);
    if (!(fminf(a, c) > 1e-15f && fmaxf(a, c) < 1e15f && det > 1e-4f * ac && spread < 1e15f)) return 0xFFFFu;
    const float pcut = fminf(4.5f, __logf(op * 255.0f) + 0.01f);
    if (pcut < 0.0f) return 0u;
    const float thr = 2.002f * pcut + 1e-3f + 4e-6f * spread;
    float ra, rc, rdet, xm;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ra) : "f"(a));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rc) : "f"(c));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rdet) : "f"(det));
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(xm) : "f"(thr * c * rdet));   /* the half width */
    const float boa = b * ra, qa = thr * ra, da = det * ra * ra;
    const float yr = -(b * rc) * xm;
    const float e = 2e-3f * xm + 1e-3f;
    /* columns k of the band: X0 + 4 k <= right edge, X0 + 4 k + 3 >= left
     * edge; rounded by the 1.5 * 2^23 addition, a tie at most adds a column */
    const float hi_c = (e - x0) * 0.25f + 0.501f, lo_c = (-e - x0 - 3.0f) * 0.25f + 0.499f;
    unsigned int m = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float b0 = y0 + (float)(4 * k), b1 = b0 + 3.0f;
        const float ur = fminf(fmaxf(yr, b0), b1), ul = fminf(fmaxf(-yr, b0), b1);
        float sr, sl;
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sr) : "f"(__fmaf_rn(-da * ur, ur, qa)));
        asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(sl) : "f"(__fmaf_rn(-da * ul, ul, qa)));
        const float hi = __fmaf_rn(__fmaf_rn(-boa, ur, sr), 0.25f, hi_c);
        const float lo = __fmaf_rn(__fmaf_rn(-boa, ul, -sl), 0.25f, lo_c);
        const unsigned int kh = __float_as_uint(fminf(fmaxf(hi, -0.499f), 4.4f) + 12582912.0f);
        const unsigned int kl = __float_as_uint(fminf(fmaxf(lo, 0.0f), 4.4f) + 12582912.0f);
        /* columns [kl, kh): the low five bits hold the rounded values */
        m |= ((((1u << (kh & 31u)) - 1u) & ~((1u << (kl & 31u)) - 1u)) & 15u) << (4 * k);
    }
    return m;
}

}  // namespace lumen
