/*
 * backward.cu - the adjoint of the forward pipeline (no reference
 * counterpart: the reference has no analytic backward; its gradient code
 * only stores buffers, src/optim/gradients.mojo:11-106).
 *
 * K6 composite_backward_kernel: per 16x16 tile, per pixel, one front-to-
 * back sweep over the splats the forward blended, up to the pixel's
 * last-visited instance (the forward's last_idx output, so the sweep stops
 * on the splat where the forward stopped). Per splat j, with the
 * transmittance T_j before it and w_j = alpha_j T_j:
 *   dL/dc = G_rgb w, dL/dz = G_depth w,
 *   dL/dalpha = T_j (G . col_j) - (G . C - G . P_j - g_tail) / (1 - alpha),
 * where G . C is the upstream gradient dotted with the forward's blended
 * colour and depth, G . P_j the same dot product of the running sum up to
 * and including j (so G . (C - P_j) is what is blended behind j) and g_tail
 * = (G_alpha - [white] sum_ch G_ch) T_final; then through
 * alpha = min(op exp(-power), 0.99) (no gradient when clamped) and power =
 * 0.5 (a dx^2 + 2 b dx dy + c dy^2) to the centre, the conic and the
 * opacity. Gradient arithmetic uses fused multiply-adds and the hardware
 * exponential and reciprocal; the decisions the forward took (power above
 * 4.5, alpha below 1/255, the 0.99 clamp) are taken exactly as the forward
 * took them: the power is formed with separately rounded operations in the
 * forward's order, and an alpha near a threshold is recomputed with the
 * shared exponential. A power that rounds below 0 (or is, of a conic that is
 * not positive definite) is a constant 0 in the forward: the centre and the
 * conic get nothing from that pixel.
 *
 * The work is split as in the compositor: two pixels per lane in packed FP32,
 * groups of 8 lanes with a 4x4 block and a splat list of their own. A splat's
 * 10 gradients are sums over the block's pixels of two scalars, s =
 * -dL/dopacity and w = alpha T: s times the opacity is dL/dpower, which goes
 * with dx^2, dx dy, dy^2 to the conic and with the power's derivatives to the
 * centre; w goes with the pixel's upstream gradient to colour and depth. So a
 * lane only forms s and w for its pixels and leaves them in shared memory;
 * after eight list steps every lane takes one of the warp's 32 (splat, block)
 * entries, reads its 16 pixels, forms the sums, with dx per column and dy per
 * row, and adds them to the warp's sums for the splat. At a chunk's end a
 * thread per splat adds the four warps' sums and sends the tile's to the
 * Gaussian with three vector atomics.
 *
 * A Gaussian's gradients are thus sums over tiles of sums that do not depend
 * on the order of the warps. Sent block by block, the running sums took 16
 * times as many additions, and their error went into the rotations of needles
 * (the conic's way back to the covariance cancels three to four digits): over
 * 500 k Gaussians at 1080p single quaternion gradients then scattered by 8e-4
 * of the typical one where they now do by 2.5e-4, and a splat over the whole
 * screen could lose 2e-3 of its colour's gradient.
 *
 * Bound by what shared memory delivers, so staged splats are read as 10 words
 * and the rows lie without bank conflicts, and by the four CTAs per SM that its
 * sums leave room for. Measured on a B200 at 500 k Gaussians and 1080p: 0.425
 * ms with one pixel per thread, 10 values per pixel summed over the warp by a
 * transpose and over the CTA by shared atomics; 0.300 ms in this form (0.230
 * with an atomic per block and six CTAs; the warps' sums by shared atomics,
 * which need a quarter of the room: 0.343).
 *
 * K7 project_backward_kernel: per Gaussian, the chain rule through the
 * conic inverse, the EWA product T Sigma T^T with T = J W, the projective
 * Jacobian, the screen projection, Sigma = M M^T with M = R(q) S, the
 * quaternion normalisation, the SH colour (clamped channels get none) and
 * the view direction, and the exp / sigmoid activations.
 *
 * K8 l1_loss_kernel: compute_l1_loss (src/optim/loss.mojo:11-35).
 *
 * This file is compiled with fused multiply-add contraction; the few
 * operations that must round as the forward's do are written with
 * explicitly rounded intrinsics.
 */
#include "composite_common.cuh"

namespace lumen {

/* floats per Gaussian in splat2d: cx, cy, ic00, ic01, ic11, opacity, r, g, b,
 * depth and two of padding, so that rows take 16-byte vector atomics */
constexpr int kGrad2DStride = 12;
constexpr int kBwdThreads = 128;
constexpr int kBwdChunk = 128;        /* instances staged per round */
constexpr int kBwdSteps = 8;          /* list entries per group and batch: 4 groups x 8 = one entry per lane */

/* A batch's rows: entry (step u, group g) has 16 values of s and, kRowsW
 * 16-byte units further, 16 of w (the group's pixels), at unit row_unit(u, g).
 * The units are placed so that the two groups of a half-warp write different
 * banks and eight lanes reading their own rows read different ones. */
__host__ __device__ constexpr int row_unit(int u, int g) { return 18 * u + (g & 1) * 4 + (g >> 1) * 9; }
constexpr int kRowsW = 18 * kBwdSteps;

template <bool kDepth>
struct BackwardSmem {
    static constexpr int kChannels = kDepth ? 4 : 3;
    float4 geo[kBwdChunk + 1];    /* cx, -cy, -0.5 ic00, ic01; slot kBwdChunk: the padding splat */
    float4 con[kBwdChunk + 1];    /* 0.5 ic11, opacity, -(power cutoff), r */
    float4 col[kBwdChunk + 1];    /* g, b, depth, - */
    __align__(16) unsigned short mask[kBwdChunk];
    unsigned short list[kBlocks][kBwdChunk + 8];   /* byte offsets (16 x slot), as in the forward */
    ulonglong2 rows[kBwdThreads / 32][2 * kRowsW];
    /* per warp and slot: the sums over the warp's pixels, in the order of splat2d */
    float4 acc0[kBwdThreads / 32][kBwdChunk], acc1[kBwdThreads / 32][kBwdChunk];
    float2 acc2[kBwdThreads / 32][kBwdChunk];
    /* per group and channel: dL/d(r, g, b, depth) of its pixels, 16 values in 4 units */
    ulonglong2 grad[kBwdThreads / 32][4][4 * kChannels + 1];
    int tile_last;
    int special;
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

/* Stage chunk [cs, min(cs + kBwdChunk, end)) of the tile's sorted
 * instances: records, reach masks, Gaussian ids. Returns (to the whole CTA)
 * whether a staged splat's opacity can reach the 0.99 clamp. */
template <bool kDepth>
__device__ __forceinline__ bool stage_chunk(BackwardSmem<kDepth>& s, const LumenSplatRecord* __restrict__ records,
                                            const unsigned int* __restrict__ vals, unsigned int& next,
                                            const unsigned int* __restrict__ visible_ids, unsigned int& gid,
                                            unsigned int n_visible,
                                            Control* ctrl, int cs, int end, float tile_x0, float tile_y0) {
    static_assert(kBwdChunk == kBwdThreads, "one slot per thread");
    int high = 0;
    {
        const int slot = threadIdx.x, i = cs + slot;
        unsigned int m = 0;
        if (i < end) {
            const unsigned int v = next;
            next = i + kBwdChunk < end ? vals[i + kBwdChunk] : 0u;   /* the next chunk's, read ahead */
            if (v >= n_visible) {
                atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
            } else {
                const float4* r4 = reinterpret_cast<const float4*>(records + v);
                const float4 geo = __ldg(r4), con = __ldg(r4 + 1), col = __ldg(r4 + 2);
                /* a pixel blends only if power <= 4.5 (compositor.mojo:80-82)
                 * and alpha = opacity * exp(-power) reaches 1/255 (:33-35),
                 * that is power <= ln(opacity / (1/255)) = faint. The margins
                 * of 1e-3 are far above the rounding of the exponential and
                 * the logarithm: beyond the cutoff faint + 1e-3 the exact test
                 * fails, up to 2e-3 before it the test holds, and it is taken
                 * in between (also below 4.5, where it is not needed) */
                const float faint = logf(geo.w / min_alpha());
                s.geo[slot] = make_float4(geo.x, -geo.y, -0.5f * con.x, con.y);
                s.con[slot] = make_float4(0.5f * con.z, geo.w, -fminf(4.5f, faint + 1e-3f), col.x);
                s.col[slot] = make_float4(col.y, col.z, geo.z, 0.0f);
                gid = visible_ids[v];
                bool finite;
                m = reach_blocks(geo, con, tile_x0, tile_y0, &finite);
                finite = finite && fabsf(col.x) + fabsf(col.y) + fabsf(col.z) + fabsf(geo.z) < 1e15f;
                if (!finite) s.special = 1;   /* for the rest of the tile */
                high |= geo.w > 0.9899f;
            }
        }
        s.mask[slot] = (unsigned short)m;
    }
    return __syncthreads_or(high) != 0;
}

/* The lists of the warp's four groups, as build_lists in the compositor, of
 * the slots up to each group's limit (the last one that any of its pixels
 * visited, or less than 0), padded to a multiple of kBwdSteps. */
template <bool kDepth>
__device__ __forceinline__ int build_backward_lists(BackwardSmem<kDepth>& s, int warp, int lane, const int limit[4]) {
    constexpr int kPer = kBwdChunk / 32;
    static_assert(kPer == 4, "four masks per lane in one 8-byte load");
    const int shift = 8 * (warp >> 1) + 2 * (warp & 1);
    const uint2 w = reinterpret_cast<const uint2*>(s.mask)[lane];
    const unsigned int raw[kPer] = {w.x >> shift, w.x >> (16 + shift), w.y >> shift, w.y >> (16 + shift)};
    unsigned int m[kPer], c01 = 0u, c23 = 0u;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const int slot = lane * kPer + i;
        m[i] = raw[i] & ((slot <= limit[0] ? 1u : 0u) | (slot <= limit[1] ? 2u : 0u) | (slot <= limit[2] ? 16u : 0u) |
                         (slot <= limit[3] ? 32u : 0u));
        c01 += ((m[i] & 3u) * 0x8001u) & 0x10001u;
        c23 += ((m[i] >> 4) * 0x8001u) & 0x10001u;
    }
    unsigned int i01 = c01, i23 = c23;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y01 = __shfl_up_sync(0xffffffffu, i01, o), y23 = __shfl_up_sync(0xffffffffu, i23, o);
        if (lane >= o) {
            i01 += y01;
            i23 += y23;
        }
    }
    const unsigned int n01 = __shfl_sync(0xffffffffu, i01, 31), n23 = __shfl_sync(0xffffffffu, i23, 31);
    const unsigned int e01 = i01 - c01, e23 = i23 - c23;
    const int n[4] = {(int)(n01 & 0xFFFFu), (int)(n01 >> 16), (int)(n23 & 0xFFFFu), (int)(n23 >> 16)};
    unsigned short* at[4] = {s.list[4 * warp] + (e01 & 0xFFFFu), s.list[4 * warp + 1] + (e01 >> 16),
                             s.list[4 * warp + 2] + (e23 & 0xFFFFu), s.list[4 * warp + 3] + (e23 >> 16)};
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const unsigned short off = (unsigned short)(16 * (lane * kPer + i));
        if (m[i] & 1u) *at[0]++ = off;
        if (m[i] & 2u) *at[1]++ = off;
        if (m[i] & 16u) *at[2]++ = off;
        if (m[i] & 32u) *at[3]++ = off;
    }
    const int longest = max(max(n[0], n[1]), max(n[2], n[3]));
    const int padded = (longest + kBwdSteps - 1) & ~(kBwdSteps - 1);
#pragma unroll
    for (int g = 0; g < 4; ++g)
        for (int k = n[g] + lane; k < padded; k += 32) s.list[4 * warp + g][k] = (unsigned short)(16 * kBwdChunk);
    __syncwarp();
    return padded;
}

/* The hardware exponential of x (x in [-4.5, 0]): within a few parts per
 * million of lumen_expf_core(x). */
__device__ __forceinline__ float fast_exp(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.44269504088896341f));
    return r;
}

__device__ __forceinline__ float fast_rcp(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

/* A lane's two pixels: the transmittance, R = G . C - g_tail, the running
 * -G . P and the negated upstream gradient, as packed pairs; end: 16 x the
 * chunk slot of the last splat each pixel visited. */
struct GradPair {
    f32x2 T, R, nP, nr, ng, nb, nd;
    int end[2];
};

/* Marks in a batch's w (which is never negative itself), read by the marked
 * form of backward_flush: -w where the forward clamped a power below 0 to 0, so
 * that the pixel's s belongs to the opacity only; -0 where the pixel did not
 * blend the splat, so that an upstream gradient that is not finite stays out
 * of its colour. */
__device__ __forceinline__ float marked(float w) { return __uint_as_float(__float_as_uint(w) | 0x80000000u); }
__device__ __forceinline__ bool is_marked(float w) { return (__float_as_uint(w) & 0x80000000u) != 0u; }

/* One list entry for the lane's two pixels: s = -dL/dopacity and w = alpha T
 * of each, zero where the pixel did not blend the splat. Every staged value and
 * upstream gradient is finite. Returns whether a w is marked. */
template <bool kClamp, bool kDepth>
__device__ __forceinline__ bool backward_step(const BackwardSmem<kDepth>& sm, unsigned int off, float pxc, f32x2 pyc,
                                              f32x2 minus_one, GradPair& p, f32x2& s_out, f32x2& w_out) {
    /* 10 words per lane (12 with the depth): the kernel is bound by what
     * shared memory delivers */
    const float4 g = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(sm.geo) + off);
    const float4 c = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(sm.con) + off);
    const char* at_col = reinterpret_cast<const char*>(sm.col) + off;
    const float2 k = *reinterpret_cast<const float2*>(at_col);
    const float op = c.y, skip = c.z;
    /* the forward's power (negated), operation by operation */
    const float dx = __fsub_rn(pxc, g.x);
    const f32x2 dy = add2(pyc, splat2(g.y));
    const f32x2 q = fma2(mul2(mul2(splat2(c.x), dy), dy), minus_one,
                         fma2(mul2(splat2(__fmul_rn(g.w, dx)), dy), minus_one,
                              splat2(__fmul_rn(__fmul_rn(g.z, dx), dx))));
    float q0, q1;
    unpack2(q, q0, q1);
    const float x0 = fminf(q0, 0.0f), x1 = fminf(q1, 0.0f);
    const int at = (int)off;
    bool b0 = !(x0 < skip) && at <= p.end[0];
    bool b1 = !(x1 < skip) && at <= p.end[1];
    const float sure = skip + 2e-3f;
    const bool unsure0 = b0 && x0 < sure, unsure1 = b1 && x1 < sure;
    if (unsure0 || unsure1) {
        /* near the 1/255 skip the decision is taken with the forward's exponential */
        if (unsure0) b0 = !(__fmul_rn(op, lumen_expf_core(x0)) < min_alpha());
        if (unsure1) b1 = !(__fmul_rn(op, lumen_expf_core(x1)) < min_alpha());
    }
    float e0 = fast_exp(x0), e1 = fast_exp(x1);
    if (kClamp) {
        /* near the 0.99 clamp likewise */
        if (fabsf(__fmul_rn(op, e0) - (float)0.99) <= 4e-6f) e0 = lumen_expf_core(x0);
        if (fabsf(__fmul_rn(op, e1) - (float)0.99) <= 4e-6f) e1 = lumen_expf_core(x1);
    }
    const f32x2 e = pack2(b0 ? e0 : 0.0f, b1 ? e1 : 0.0f);
    f32x2 alpha = mul2(splat2(op), e);
    bool c0 = false, c1 = false;
    if (kClamp) {
        /* a clamped alpha passes no gradient on */
        float a0, a1;
        unpack2(alpha, a0, a1);
        c0 = a0 > (float)0.99;
        c1 = a1 > (float)0.99;
        alpha = pack2(fminf(a0, (float)0.99), fminf(a1, (float)0.99));
    }
    const f32x2 w = mul2(alpha, p.T);
    f32x2 ngcol = fma2(splat2(k.y), p.nb, fma2(splat2(c.w), p.nr, mul2(splat2(k.x), p.ng)));
    if (kDepth) ngcol = fma2(splat2(*reinterpret_cast<const float*>(at_col + 8)), p.nd, ngcol);
    p.nP = fma2(w, ngcol, p.nP);
    const f32x2 om = fma2(alpha, splat2(-1.0f), splat2(1.0f));
    float o0, o1;
    unpack2(om, o0, o1);
    const f32x2 ndalpha = fma2(p.T, ngcol, mul2(add2(p.R, p.nP), pack2(fast_rcp(o0), fast_rcp(o1))));
    f32x2 sv = mul2(ndalpha, e);
    if (kClamp) {
        float s0, s1;
        unpack2(sv, s0, s1);
        sv = pack2(c0 ? 0.0f : s0, c1 ? 0.0f : s1);
    }
    p.T = mul2(p.T, om);
    s_out = sv;
    w_out = w;
    const bool below0 = q0 > 0.0f && b0, below1 = q1 > 0.0f && b1;
    if (!(below0 || below1)) return false;
    float w0, w1;
    unpack2(w, w0, w1);
    w_out = pack2(below0 ? marked(w0) : w0, below1 ? marked(w1) : w1);
    return true;
}

/* The same for a tile with a value that is not finite: one pixel at a time,
 * nothing computed for a pixel that skips (its w is marked). */
template <bool kDepth>
__device__ __forceinline__ void backward_step_general(const BackwardSmem<kDepth>& sm, unsigned int off, float pxc,
                                                      float pyc0, GradPair& p, f32x2& s_out, f32x2& w_out) {
    const unsigned int j = off >> 4;
    const float4 g = sm.geo[j], c = sm.con[j], k = sm.col[j];
    const float op = c.y;
    float T[2], R[2], nP[2], nr[2], ng[2], nb[2], nd[2], s[2] = {0.0f, 0.0f}, w[2] = {-0.0f, -0.0f};
    unpack2(p.T, T[0], T[1]);
    unpack2(p.R, R[0], R[1]);
    unpack2(p.nP, nP[0], nP[1]);
    unpack2(p.nr, nr[0], nr[1]);
    unpack2(p.ng, ng[0], ng[1]);
    unpack2(p.nb, nb[0], nb[1]);
    unpack2(p.nd, nd[0], nd[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if ((int)off > p.end[h]) continue;
        const float dx = __fsub_rn(pxc, g.x), dy = __fadd_rn(pyc0 + (float)h, g.y);
        float x = __fsub_rn(__fsub_rn(__fmul_rn(__fmul_rn(g.z, dx), dx), __fmul_rn(__fmul_rn(g.w, dx), dy)),
                            __fmul_rn(__fmul_rn(c.x, dy), dy));
        const bool below = x > 0.0f;
        if (below) x = 0.0f;
        if (x < c.z) continue;
        float e = fast_exp(x), alpha = __fmul_rn(op, e);
        if (fabsf(alpha - min_alpha()) <= 4e-6f * min_alpha() || fabsf(alpha - (float)0.99) <= 4e-6f) {
            e = lumen_expf_core(x);
            alpha = __fmul_rn(op, e);
        }
        const bool clamped = alpha > (float)0.99;
        if (clamped) alpha = (float)0.99;
        if (alpha < min_alpha()) continue;
        const float wh = alpha * T[h];
        float ngcol = __fmaf_rn(k.y, nb[h], __fmaf_rn(c.w, nr[h], __fmul_rn(k.x, ng[h])));
        if (kDepth) ngcol = __fmaf_rn(k.z, nd[h], ngcol);
        nP[h] = __fmaf_rn(wh, ngcol, nP[h]);
        const float om = 1.0f - alpha;
        const float ndalpha = __fmaf_rn(T[h], ngcol, __fmul_rn(__fadd_rn(R[h], nP[h]), fast_rcp(om)));
        if (!clamped) s[h] = __fmul_rn(ndalpha, e);
        T[h] *= om;
        w[h] = below ? marked(wh) : wh;
    }
    p.T = pack2(T[0], T[1]);
    p.nP = pack2(nP[0], nP[1]);
    s_out = pack2(s[0], s[1]);
    w_out = pack2(w[0], w[1]);
}

/* The sums of a batch: lane e takes entry e (list position t0 + e / 4 of
 * group e % 4), reads the group's 16 values of s and w from its row and adds
 * its 10 gradients to the warp's sums for the splat, group by group (a group's
 * entries are different splats, so no two lanes add to one). Rows hold the
 * pixels in the order (row pair, column, row within the pair), so the packed
 * halves are the two rows of a pair. kMarked: some w of the batch is marked. */
template <bool kDepth, bool kMarked>
__device__ __forceinline__ void backward_flush(BackwardSmem<kDepth>& sm, int warp, int lane, int t0, float quad_x,
                                               float quad_y) {
    const int g = lane & 3, u = lane >> 2;
    const unsigned int off = sm.list[4 * warp + g][t0 + u];
    const float4 geo = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(sm.geo) + off);
    const float2 con = *reinterpret_cast<const float2*>(reinterpret_cast<const char*>(sm.con) + off);
    const ulonglong2* row = sm.rows[warp] + row_unit(u, g);
    const ulonglong2* gr = sm.grad[warp][g];
    const float bx = quad_x + (float)(4 * (g & 1)), by = quad_y + (float)(4 * (g >> 1));
    float dx[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) dx[x] = (bx + (float)x) - geo.x;
    constexpr int kCh = BackwardSmem<kDepth>::kChannels;
    const f32x2 zero = splat2(0.0f);
    f32x2 So = zero, Gx = zero, Gy = zero, Sxx = zero, Sxy = zero, Syy = zero, c[kCh];
#pragma unroll
    for (int ch = 0; ch < kCh; ++ch) c[ch] = zero;
    const f32x2 op = splat2(con.y), na = splat2(2.0f * geo.z), nb = splat2(-geo.w), nc = splat2(-2.0f * con.x);
#pragma unroll
    for (int yp = 0; yp < 2; ++yp) {
        const f32x2 dy = add2(pack2(by + (float)(2 * yp), by + (float)(2 * yp + 1)), splat2(geo.y));
        const f32x2 nbdy = mul2(nb, dy), ncdy = mul2(nc, dy);
        f32x2 r0 = zero, r1 = zero;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            ulonglong2 s2 = row[2 * yp + q], w2 = row[kRowsW + 2 * yp + q];
            So = add2(So, add2(s2.x, s2.y));
            bool skip[4] = {false, false, false, false};
            if (kMarked) {
                float s[4], w[4];
                unpack2(s2.x, s[0], s[1]);
                unpack2(s2.y, s[2], s[3]);
                unpack2(w2.x, w[0], w[1]);
                unpack2(w2.y, w[2], w[3]);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (!is_marked(w[i])) continue;
                    w[i] = -w[i];
                    skip[i] = w[i] == 0.0f;
                    s[i] = 0.0f;
                }
                s2 = make_ulonglong2(pack2(s[0], s[1]), pack2(s[2], s[3]));
                w2 = make_ulonglong2(pack2(w[0], w[1]), pack2(w[2], w[3]));
            }
            s2 = make_ulonglong2(mul2(s2.x, op), mul2(s2.y, op));   /* dL/dpower */
            const f32x2 d0 = splat2(dx[2 * q]), d1 = splat2(dx[2 * q + 1]);
            Gx = fma2(fma2(na, d0, nbdy), s2.x, fma2(fma2(na, d1, nbdy), s2.y, Gx));
            Gy = fma2(fma2(nb, d0, ncdy), s2.x, fma2(fma2(nb, d1, ncdy), s2.y, Gy));
            r0 = add2(r0, add2(s2.x, s2.y));
            const f32x2 e0 = mul2(s2.x, d0), e1 = mul2(s2.y, d1);
            r1 = add2(r1, add2(e0, e1));
            Sxx = fma2(e0, d0, fma2(e1, d1, Sxx));
#pragma unroll
            for (int ch = 0; ch < kCh; ++ch) {
                ulonglong2 G = gr[4 * ch + 2 * yp + q];
                if (kMarked) {
                    float G0[4];
                    unpack2(G.x, G0[0], G0[1]);
                    unpack2(G.y, G0[2], G0[3]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) G0[i] = skip[i] ? 0.0f : G0[i];
                    G = make_ulonglong2(pack2(G0[0], G0[1]), pack2(G0[2], G0[3]));
                }
                c[ch] = fma2(w2.x, G.x, fma2(w2.y, G.y, c[ch]));
            }
        }
        Sxy = fma2(r1, dy, Sxy);
        Syy = fma2(r0, mul2(dy, dy), Syy);
    }
    auto both = [](f32x2 v) {
        float a, b;
        unpack2(v, a, b);
        return a + b;
    };
    const unsigned int slot = off >> 4;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (g == k && slot < (unsigned int)kBwdChunk) {   /* not a padding entry */
            float4 a = sm.acc0[warp][slot], b = sm.acc1[warp][slot];
            float2 d = sm.acc2[warp][slot];
            a.x += both(Gx);
            a.y += both(Gy);
            a.z += 0.5f * both(Sxx);
            a.w += both(Sxy);
            b.x += 0.5f * both(Syy);
            b.y -= both(So);
            b.z += both(c[0]);
            b.w += both(c[1]);
            d.x += both(c[2]);
            if (kDepth) d.y += both(c[kCh - 1]);
            sm.acc0[warp][slot] = a;
            sm.acc1[warp][slot] = b;
            sm.acc2[warp][slot] = d;
        }
        __syncwarp();
    }
}

/* The lists' n entries of one staged chunk, kBwdSteps at a time. */
template <int kWay, bool kDepth>   /* kWay 0: general, 1: no clamp, 2: clamp */
__device__ __forceinline__ void backward_walk(BackwardSmem<kDepth>& sm, int warp, int lane, int n, float pxc,
                                              float pyc, f32x2 minus_one, float quad_x, float quad_y, GradPair& p) {
    const int group = lane >> 3;
    const unsigned short* lst = sm.list[4 * warp + group];
    const f32x2 pyc2 = pack2(pyc, pyc + 1.0f);
    f32x2* row = reinterpret_cast<f32x2*>(sm.rows[warp] + row_unit(0, group)) + (lane & 7);
    for (int t0 = 0; t0 < n; t0 += kBwdSteps) {
        bool any_marked = kWay == 0;
#pragma unroll 2
        for (int u = 0; u < kBwdSteps; ++u) {
            f32x2 s, w;
            const unsigned int off = lst[t0 + u];
            if (kWay == 0) backward_step_general<kDepth>(sm, off, pxc, pyc, p, s, w);
            else any_marked |= backward_step<kWay == 2, kDepth>(sm, off, pxc, pyc2, minus_one, p, s, w);
            row[2 * row_unit(u, 0)] = s;
            row[2 * (row_unit(u, 0) + kRowsW)] = w;
        }
        __syncwarp();
        if (__any_sync(0xffffffffu, any_marked)) backward_flush<kDepth, true>(sm, warp, lane, t0, quad_x, quad_y);
        else backward_flush<kDepth, false>(sm, warp, lane, t0, quad_x, quad_y);
    }
}

/* 4 CTAs per SM (128 registers, 53 KB of shared memory). kDepth: there is an
 * upstream depth gradient. */
template <bool kDepth>
__global__ void __launch_bounds__(kBwdThreads, 4)
composite_backward_kernel(const LumenSplatRecord* __restrict__ records, LumenGpuFrame f, Control* ctrl,
                          int width, int height, int tiles_x, LumenRenderOptions opt,
                          const float* __restrict__ out_rgb, const float* __restrict__ out_depth,
                          const float* __restrict__ out_alpha, const int* __restrict__ out_last,
                          const float* __restrict__ grad_rgb, const float* __restrict__ grad_depth,
                          const float* __restrict__ grad_alpha, float* __restrict__ grad2d, float minus_one) {
    chain_begin();
    extern __shared__ float4 bwd_smem[];
    BackwardSmem<kDepth>& s = *reinterpret_cast<BackwardSmem<kDepth>*>(bwd_smem);
    const int tile = (int)tile_in_line(ctrl, blockIdx.x);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tile % tiles_x, ty = tile / tiles_x;
    /* the compositor's pixels: a lane's two are one above the other */
    const int group = lane >> 3;
    const int px = tx * kTile + 8 * (warp & 1) + 4 * (group & 1) + (lane & 3);
    const int py = ty * kTile + 8 * (warp >> 1) + 4 * (group >> 1) + 2 * ((lane >> 2) & 1);
    const long long cap = f.instance_capacity;
    const long long K = (long long)ctrl->n_instances < cap ? (long long)ctrl->n_instances : cap;
    if (K == 0) return;
    const int rs = f.ranges[2 * tile], re = f.ranges[2 * tile + 1];
    if (rs == -1 || rs >= re) return;
    if (rs < 0 || (long long)re > K) {
        if (tid == 0) atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
        return;
    }
    const unsigned int n_visible = ctrl->n_visible;
    const unsigned int* __restrict__ vals = ctrl->list_buffer ? f.vals[1] : f.vals[0];
    const float tile_x0 = (float)(tx * kTile), tile_y0 = (float)(ty * kTile);

    if (tid == 0) {
        s.tile_last = -1;
        s.special = 0;
        s.geo[kBwdChunk] = make_float4(0.0f, 0.0f, -1e30f, 0.0f);   /* out of every pixel's reach */
        s.con[kBwdChunk] = make_float4(1e30f, 0.0f, -4.5f, 0.0f);
        s.col[kBwdChunk] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int w = 0; w < kBwdThreads / 32; ++w) {
        s.acc0[w][tid] = s.acc1[w][tid] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        s.acc2[w][tid] = make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    /* the pixels' upstream gradients and the forward's outputs */
    GradPair p;
    int last[2] = {-1, -1};
    {
        float R[2] = {0.0f, 0.0f}, nr[2] = {0.0f, 0.0f}, ng[2] = {0.0f, 0.0f}, nb[2] = {0.0f, 0.0f},
              nd[2] = {0.0f, 0.0f};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (px >= width || py + h >= height) continue;
            const long long pix = (long long)(py + h) * width + px;
            last[h] = out_last[pix];
            if (last[h] >= re) {   /* self-check: a last-visited instance beyond the tile's range */
                atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
                last[h] = re - 1;
            }
            const float g_r = grad_rgb[pix * 3 + 0], g_g = grad_rgb[pix * 3 + 1], g_b = grad_rgb[pix * 3 + 2];
            float g_d = 0.0f, C_z = 0.0f;
            if (kDepth) {
                g_d = grad_depth[pix];
                C_z = out_depth[pix];
            }
            const float g_a = grad_alpha ? grad_alpha[pix] : 0.0f;
            const float T_final = 1.0f - out_alpha[pix];
            const float bg = opt.white_background ? T_final : 0.0f;
            /* terms of dL/dalpha_j that scale with 1 / (1 - alpha_j) and do not
             * change along the sweep: G . C - g_tail */
            const float g_tail = (g_a - (opt.white_background ? (g_r + g_g + g_b) : 0.0f)) * T_final;
            R[h] = g_r * (out_rgb[pix * 3 + 0] - bg) + g_g * (out_rgb[pix * 3 + 1] - bg) +
                   g_b * (out_rgb[pix * 3 + 2] - bg) + g_d * C_z - g_tail;
            nr[h] = -g_r;
            ng[h] = -g_g;
            nb[h] = -g_b;
            nd[h] = -g_d;
            if (!(fabsf(g_r) + fabsf(g_g) + fabsf(g_b) + fabsf(g_d) < 1e15f && fabsf(R[h]) < 1e20f)) s.special = 1;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            float* at = reinterpret_cast<float*>(s.grad[warp][group]) + 2 * (lane & 7) + h;
            at[0] = -nr[h];
            at[16] = -ng[h];
            at[32] = -nb[h];
            if (kDepth) at[48] = -nd[h];
        }
        p.T = splat2(1.0f);
        p.R = pack2(R[0], R[1]);
        p.nP = splat2(0.0f);
        p.nr = pack2(nr[0], nr[1]);
        p.ng = pack2(ng[0], ng[1]);
        p.nb = pack2(nb[0], nb[1]);
        p.nd = pack2(nd[0], nd[1]);
    }
    /* the last instance that any pixel visited, per group and for the tile,
     * where the sweep ends */
    int group_last = max(last[0], last[1]);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) group_last = max(group_last, __shfl_xor_sync(0xffffffffu, group_last, o));
    int ends[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) ends[g] = __shfl_sync(0xffffffffu, group_last, 8 * g);
    const int warp_last = max(max(ends[0], ends[1]), max(ends[2], ends[3]));
    if (lane == 0 && warp_last >= rs) atomicMax(&s.tile_last, warp_last);
    __syncthreads();
    const int end = s.tile_last + 1;   /* <= re */
    if (end <= rs) return;

    const float pxc = (float)px + 0.5f, pyc = (float)py + 0.5f;
    const float quad_x = tile_x0 + (float)(8 * (warp & 1)) + 0.5f, quad_y = tile_y0 + (float)(8 * (warp >> 1)) + 0.5f;
    unsigned int next = rs + tid < end ? vals[rs + tid] : 0u, gid = 0u;
    for (int cs = rs; cs < end; cs += kBwdChunk) {
        const bool clamp = stage_chunk<kDepth>(s, records, vals, next, f.visible_ids, gid, n_visible, ctrl, cs, end,
                                               tile_x0, tile_y0);
        if (warp_last >= cs) {
            const int limit[4] = {ends[0] - cs, ends[1] - cs, ends[2] - cs, ends[3] - cs};
            const int n = build_backward_lists<kDepth>(s, warp, lane, limit);
            p.end[0] = 16 * min(last[0] - cs, kBwdChunk);
            p.end[1] = 16 * min(last[1] - cs, kBwdChunk);
            if (last[0] < cs) p.end[0] = -1;
            if (last[1] < cs) p.end[1] = -1;
            if (s.special) backward_walk<0, kDepth>(s, warp, lane, n, pxc, pyc, splat2(minus_one), quad_x, quad_y, p);
            else if (clamp) backward_walk<2, kDepth>(s, warp, lane, n, pxc, pyc, splat2(minus_one), quad_x, quad_y, p);
            else backward_walk<1, kDepth>(s, warp, lane, n, pxc, pyc, splat2(minus_one), quad_x, quad_y, p);
        }
        __syncthreads();
        /* thread t: the tile's sums of the chunk's splat t, over the warps */
        float4 a = s.acc0[0][tid], b = s.acc1[0][tid];
        float2 d = s.acc2[0][tid];
#pragma unroll
        for (int w = 1; w < kBwdThreads / 32; ++w) {
            const float4 a1 = s.acc0[w][tid], b1 = s.acc1[w][tid];
            const float2 d1 = s.acc2[w][tid];
            a = make_float4(a.x + a1.x, a.y + a1.y, a.z + a1.z, a.w + a1.w);
            b = make_float4(b.x + b1.x, b.y + b1.y, b.z + b1.z, b.w + b1.w);
            d = make_float2(d.x + d1.x, d.y + d1.y);
        }
        float* dst = grad2d + (size_t)gid * kGrad2DStride;
        if (a.x != 0.0f || a.y != 0.0f || a.z != 0.0f || a.w != 0.0f) atomicAdd(reinterpret_cast<float4*>(dst), a);
        if (b.x != 0.0f || b.y != 0.0f || b.z != 0.0f || b.w != 0.0f) atomicAdd(reinterpret_cast<float4*>(dst + 4), b);
        if (d.x != 0.0f || d.y != 0.0f) atomicAdd(reinterpret_cast<float2*>(dst + 8), d);
        if (cs + kBwdChunk >= end) break;
#pragma unroll
        for (int w = 0; w < kBwdThreads / 32; ++w) {
            s.acc0[w][tid] = s.acc1[w][tid] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            s.acc2[w][tid] = make_float2(0.0f, 0.0f);
        }
    }
}

/* ---------------------------------------------------------------- K7 -- */

__device__ __forceinline__ void rot_from_quat(float w, float x, float y, float z, float R[9]) {
    R[0] = 1.0f - 2.0f * (y * y + z * z); R[1] = 2.0f * (x * y - w * z); R[2] = 2.0f * (x * z + w * y);
    R[3] = 2.0f * (x * y + w * z); R[4] = 1.0f - 2.0f * (x * x + z * z); R[5] = 2.0f * (y * z - w * x);
    R[6] = 2.0f * (x * z - w * y); R[7] = 2.0f * (y * z + w * x); R[8] = 1.0f - 2.0f * (x * x + y * y);
}

/* SH basis function k and its gradient with respect to the (unit)
 * direction components, for the constants of spherical_harmonics.mojo:17-26
 * (k is a compile-time constant after unrolling). */
__device__ __forceinline__ void sh_term(int k, float x, float y, float z, float& Y, float& dX, float& dY,
                                        float& dZ) {
    const float C0 = (float)0.28209479177387814, C1 = (float)0.4886025119029199;
    const float C2_0 = (float)1.0925484305920792, C2_1 = (float)0.31539156525252005;
    const float C2_2 = (float)0.5462742152960396, C3_0 = (float)0.5900435899266435;
    const float C3_1 = (float)2.890611442640554, C3_2 = (float)0.4570457994644658;
    const float C3_3 = (float)0.3731763325901154, C3_4 = (float)1.445305721320277;
    const float xx = x * x, yy = y * y, zz = z * z;
    switch (k) {
        case 0: Y = C0; dX = 0.0f; dY = 0.0f; dZ = 0.0f; break;
        case 1: Y = -C1 * y; dX = 0.0f; dY = -C1; dZ = 0.0f; break;
        case 2: Y = C1 * z; dX = 0.0f; dY = 0.0f; dZ = C1; break;
        case 3: Y = -C1 * x; dX = -C1; dY = 0.0f; dZ = 0.0f; break;
        case 4: Y = C2_0 * x * y; dX = C2_0 * y; dY = C2_0 * x; dZ = 0.0f; break;
        case 5: Y = -C2_0 * y * z; dX = 0.0f; dY = -C2_0 * z; dZ = -C2_0 * y; break;
        case 6: Y = C2_1 * (2.0f * zz - xx - yy); dX = -2.0f * C2_1 * x; dY = -2.0f * C2_1 * y; dZ = 4.0f * C2_1 * z;
            break;
        case 7: Y = -C2_0 * x * z; dX = -C2_0 * z; dY = 0.0f; dZ = -C2_0 * x; break;
        case 8: Y = C2_2 * (xx - yy); dX = 2.0f * C2_2 * x; dY = -2.0f * C2_2 * y; dZ = 0.0f; break;
        case 9: Y = -C3_0 * y * (3.0f * xx - yy); dX = -6.0f * C3_0 * x * y; dY = -3.0f * C3_0 * (xx - yy);
            dZ = 0.0f; break;
        case 10: Y = C3_1 * x * y * z; dX = C3_1 * y * z; dY = C3_1 * x * z; dZ = C3_1 * x * y; break;
        case 11: Y = -C3_2 * y * (4.0f * zz - xx - yy); dX = 2.0f * C3_2 * x * y;
            dY = -C3_2 * (4.0f * zz - xx - 3.0f * yy); dZ = -8.0f * C3_2 * y * z; break;
        case 12: Y = C3_3 * z * (2.0f * zz - 3.0f * xx - 3.0f * yy); dX = -6.0f * C3_3 * x * z;
            dY = -6.0f * C3_3 * y * z; dZ = C3_3 * (6.0f * zz - 3.0f * xx - 3.0f * yy); break;
        case 13: Y = -C3_2 * x * (4.0f * zz - xx - yy); dX = -C3_2 * (4.0f * zz - 3.0f * xx - yy);
            dY = 2.0f * C3_2 * x * y; dZ = -8.0f * C3_2 * x * z; break;
        case 14: Y = C3_4 * z * (xx - yy); dX = 2.0f * C3_4 * x * z; dY = -2.0f * C3_4 * y * z;
            dZ = C3_4 * (xx - yy); break;
        default: Y = -C3_0 * x * (xx - 3.0f * yy); dX = -3.0f * C3_0 * (xx - yy); dY = 6.0f * C3_0 * x * y;
            dZ = 0.0f; break;
    }
}

constexpr int kProjBwdThreads = 128;
constexpr size_t kProjBwdStageBytes = (size_t)kProjBwdThreads * 48 * sizeof(float);

/* One visible Gaussian's gradients. row: its 48 SH coefficients staged in
 * shared memory (chunk q at q ^ swz), overwritten with dL/dsh. */
__device__ __forceinline__ void project_backward_gaussian(const LumenGpuGaussians& g, const DevCamera& cam,
                                                          const LumenRenderOptions& opt, long long i,
                                                          const float* __restrict__ grad2d,
                                                          const LumenGpuGradients& out, float4* row, int swz) {
    float* gm = out.means + i * 3;
    float* gs = out.scales + i * 3;
    float* gq = out.quats + i * 4;
    const float4 G0 = reinterpret_cast<const float4*>(grad2d + i * kGrad2DStride)[0];
    const float4 G1 = reinterpret_cast<const float4*>(grad2d + i * kGrad2DStride)[1];
    const float2 G2 = reinterpret_cast<const float2*>(grad2d + i * kGrad2DStride)[4];
    const float g_cx = G0.x, g_cy = G0.y, g_a = G0.z, g_b = G0.w, g_c = G1.x, g_op = G1.y;
    const float g_col[3] = {G1.z, G1.w, G2.x};
    const float g_z = G2.y;

    /* parameters and activations */
    const float mx = g.means[i * 3], my = g.means[i * 3 + 1], mz = g.means[i * 3 + 2];
    float s3[3] = {g.scales[i * 3], g.scales[i * 3 + 1], g.scales[i * 3 + 2]};
    float op = g.opacities[i];
    if (opt.params_are_logits) {
        for (int k = 0; k < 3; ++k) s3[k] = lumen_expf(s3[k]);
        op = 1.0f / (1.0f + lumen_expf(-op));
    }
    const float4 q4 = reinterpret_cast<const float4*>(g.quats)[i];
    const float qn2 = q4.x * q4.x + q4.y * q4.y + q4.z * q4.z + q4.w * q4.w;
    const float qlen = sqrtf(qn2);
    const bool qok = qlen > (float)0.000001;
    const float qw = qok ? q4.x / qlen : 1.0f, qx = qok ? q4.y / qlen : 0.0f;
    const float qy = qok ? q4.z / qlen : 0.0f, qz = qok ? q4.w / qlen : 0.0f;
    float R[9];
    rot_from_quat(qw, qx, qy, qz, R);
    float sc[3];
    bool sclamp[3];
    for (int k = 0; k < 3; ++k) {
        sclamp[k] = s3[k] < (float)0.00001;
        sc[k] = sclamp[k] ? (float)0.00001 : s3[k];
    }
    float M[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) M[r * 3 + c] = R[r * 3 + c] * sc[c];
    float S[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) S[r * 3 + c] = M[r * 3] * M[c * 3] + M[r * 3 + 1] * M[c * 3 + 1] + M[r * 3 + 2] * M[c * 3 + 2];
    /* camera space (the Hamilton-product transform equals W (mu - position)) */
    const float* W = cam.W;
    const float vx = mx - cam.px, vy = my - cam.py, vz = mz - cam.pz;
    const float x = W[0] * vx + W[1] * vy + W[2] * vz;
    const float y = W[3] * vx + W[4] * vy + W[5] * vz;
    float z = W[6] * vx + W[7] * vy + W[8] * vz;
    const bool zclamp = z < (float)0.0001;
    const float zj = zclamp ? (float)0.0001 : z;
    const float iz = 1.0f / zj, iz2 = iz * iz, iz3 = iz2 * iz;
    const float fx = cam.fx, fy = cam.fy;
    const float j00 = fx * iz, j02 = -fx * x * iz2, j11 = fy * iz, j12 = -fy * y * iz2;
    float t0[3], t1[3];
    for (int k = 0; k < 3; ++k) {
        t0[k] = j00 * W[k] + j02 * W[6 + k];
        t1[k] = j11 * W[3 + k] + j12 * W[6 + k];
    }
    float St0[3], St1[3];
    for (int r = 0; r < 3; ++r) {
        St0[r] = S[r * 3] * t0[0] + S[r * 3 + 1] * t0[1] + S[r * 3 + 2] * t0[2];
        St1[r] = S[r * 3] * t1[0] + S[r * 3 + 1] * t1[1] + S[r * 3 + 2] * t1[2];
    }
    const float A = t0[0] * St0[0] + t0[1] * St0[1] + t0[2] * St0[2] + opt.lowpass;
    const float B = t0[0] * St1[0] + t0[1] * St1[1] + t0[2] * St1[2];
    const float Cc = t1[0] * St1[0] + t1[1] * St1[1] + t1[2] * St1[2] + opt.lowpass;
    const float det = A * Cc - B * B;

    /* conic -> Sigma2D (A, B, C) */
    float gA = 0.0f, gB = 0.0f, gC = 0.0f;
    if (!(det > (float)-0.0000001 && det < (float)0.0000001)) {
        const float id2 = 1.0f / (det * det);
        gA = (-Cc * Cc * g_a + B * Cc * g_b - B * B * g_c) * id2;
        gB = (2.0f * B * Cc * g_a - (det + 2.0f * B * B) * g_b + 2.0f * A * B * g_c) * id2;
        gC = (-B * B * g_a + A * B * g_b - A * A * g_c) * id2;
    }
    /* Sigma2D = T Sigma T^T (+ low pass) -> rows of T and Sigma */
    float dt0[3], dt1[3];
    for (int k = 0; k < 3; ++k) {
        dt0[k] = 2.0f * gA * St0[k] + gB * St1[k];
        dt1[k] = gB * St0[k] + 2.0f * gC * St1[k];
    }
    float Gs[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) Gs[r * 3 + c] = gA * t0[r] * t0[c] + gB * t0[r] * t1[c] + gC * t1[r] * t1[c];
    /* T = J W -> Jacobian entries */
    const float gj00 = dt0[0] * W[0] + dt0[1] * W[1] + dt0[2] * W[2];
    const float gj02 = dt0[0] * W[6] + dt0[1] * W[7] + dt0[2] * W[8];
    const float gj11 = dt1[0] * W[3] + dt1[1] * W[4] + dt1[2] * W[5];
    const float gj12 = dt1[0] * W[6] + dt1[1] * W[7] + dt1[2] * W[8];
    /* camera-space point: screen centre (camera.mojo:73-79), Jacobian, depth */
    const float iz_s = 1.0f / z, iz2_s = iz_s * iz_s;
    float gx = g_cx * fx * iz_s;
    float gy = g_cy * fy * iz_s;
    float gzc = -(g_cx * fx * x + g_cy * fy * y) * iz2_s + g_z;
    gx += gj02 * (-fx * iz2);
    gy += gj12 * (-fy * iz2);
    if (!zclamp) gzc += gj00 * (-fx * iz2) + gj02 * (2.0f * fx * x * iz3) + gj11 * (-fy * iz2) + gj12 * (2.0f * fy * y * iz3);
    float gmu[3];
    for (int k = 0; k < 3; ++k) gmu[k] = W[k] * gx + W[3 + k] * gy + W[6 + k] * gzc;

    /* colour: clamp(0.5 + sum sh_k Y_k(d)), d = normalize(mu - position) */
    {
        const float len = sqrtf(vx * vx + vy * vy + vz * vz);
        const bool dok = len > (float)0.000001;
        const float dx_ = dok ? vx / len : 0.0f, dy_ = dok ? vy / len : 0.0f, dz_ = dok ? vz / len : 0.0f;
        const int n = opt.sh_degree == 0 ? 1 : opt.sh_degree == 1 ? 4 : opt.sh_degree == 2 ? 9 : 16;
        /* two streaming passes over the coefficients, 4 at a time (12 floats
         * = 3 float4): the colour before the clamp (which channels pass a
         * gradient), then the direction gradient and dL/dsh */
        float v0 = 0.5f, v1 = 0.5f, v2 = 0.5f;
#pragma unroll
        for (int grp = 0; grp < 4; ++grp) {
            if (4 * grp >= n) break;
            const float4 a = row[(3 * grp) ^ swz], b = row[(3 * grp + 1) ^ swz], c = row[(3 * grp + 2) ^ swz];
            const float e[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const int k = 4 * grp + kk;
                if (k < n) {
                    float Y, dX, dY, dZ;
                    sh_term(k, dx_, dy_, dz_, Y, dX, dY, dZ);
                    v0 += e[3 * kk] * Y;
                    v1 += e[3 * kk + 1] * Y;
                    v2 += e[3 * kk + 2] * Y;
                }
            }
        }
        const float gc0 = (v0 < 0.0f || v0 > 1.0f) ? 0.0f : g_col[0];
        const float gc1 = (v1 < 0.0f || v1 > 1.0f) ? 0.0f : g_col[1];
        const float gc2 = (v2 < 0.0f || v2 > 1.0f) ? 0.0f : g_col[2];
        float gd0 = 0.0f, gd1 = 0.0f, gd2 = 0.0f;
#pragma unroll
        for (int grp = 0; grp < 4; ++grp) {
            float o[12];
            if (4 * grp < n) {
                const float4 a = row[(3 * grp) ^ swz], b = row[(3 * grp + 1) ^ swz], c = row[(3 * grp + 2) ^ swz];
                const float e[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const int k = 4 * grp + kk;
                    float Y = 0.0f, dX = 0.0f, dY = 0.0f, dZ = 0.0f;
                    if (k < n) sh_term(k, dx_, dy_, dz_, Y, dX, dY, dZ);
                    const float s3 = gc0 * e[3 * kk] + gc1 * e[3 * kk + 1] + gc2 * e[3 * kk + 2];
                    gd0 += s3 * dX;
                    gd1 += s3 * dY;
                    gd2 += s3 * dZ;
                    /* dL/dsh[k][ch] = gcol[ch] Y_k */
                    o[3 * kk] = gc0 * Y;
                    o[3 * kk + 1] = gc1 * Y;
                    o[3 * kk + 2] = gc2 * Y;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 12; ++q) o[q] = 0.0f;
            }
            row[(3 * grp) ^ swz] = make_float4(o[0], o[1], o[2], o[3]);
            row[(3 * grp + 1) ^ swz] = make_float4(o[4], o[5], o[6], o[7]);
            row[(3 * grp + 2) ^ swz] = make_float4(o[8], o[9], o[10], o[11]);
        }
        if (dok) {
            const float dot = gd0 * dx_ + gd1 * dy_ + gd2 * dz_;
            gmu[0] += (gd0 - dx_ * dot) / len;
            gmu[1] += (gd1 - dy_ * dot) / len;
            gmu[2] += (gd2 - dz_ * dot) / len;
        }
    }
    gm[0] = gmu[0]; gm[1] = gmu[1]; gm[2] = gmu[2];

    /* Sigma = M M^T, M = R diag(s) */
    float gM[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) {
            float a = 0.0f;
            for (int k = 0; k < 3; ++k) a += (Gs[r * 3 + k] + Gs[k * 3 + r]) * M[k * 3 + c];
            gM[r * 3 + c] = a;
        }
    float gsc[3];
    for (int c = 0; c < 3; ++c) {
        float a = 0.0f;
        for (int r = 0; r < 3; ++r) a += gM[r * 3 + c] * R[r * 3 + c];
        gsc[c] = sclamp[c] ? 0.0f : a;
    }
    float gR[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) gR[r * 3 + c] = gM[r * 3 + c] * sc[c];
    /* R(q) for the unit quaternion (w, x, y, z) */
    float gqw = 2.0f * (-qz * gR[1] + qy * gR[2] + qz * gR[3] - qx * gR[5] - qy * gR[6] + qx * gR[7]);
    float gqx = 2.0f * (qy * gR[1] + qz * gR[2] + qy * gR[3] - 2.0f * qx * gR[4] - qw * gR[5] + qz * gR[6] +
                        qw * gR[7] - 2.0f * qx * gR[8]);
    float gqy = 2.0f * (-2.0f * qy * gR[0] + qx * gR[1] + qw * gR[2] + qx * gR[3] + qz * gR[5] - qw * gR[6] +
                        qz * gR[7] - 2.0f * qy * gR[8]);
    float gqz = 2.0f * (-2.0f * qz * gR[0] - qw * gR[1] + qx * gR[2] + qw * gR[3] - 2.0f * qz * gR[4] + qy * gR[5] +
                        qx * gR[6] + qy * gR[7]);
    if (qok) {   /* through q / |q| */
        const float dot = gqw * qw + gqx * qx + gqy * qy + gqz * qz;
        gq[0] = (gqw - qw * dot) / qlen;
        gq[1] = (gqx - qx * dot) / qlen;
        gq[2] = (gqy - qy * dot) / qlen;
        gq[3] = (gqz - qz * dot) / qlen;
    } else {
        gq[0] = gq[1] = gq[2] = gq[3] = 0.0f;
    }
    if (opt.params_are_logits) {
        for (int k = 0; k < 3; ++k) gs[k] = gsc[k] * s3[k];
        out.opacities[i] = g_op * op * (1.0f - op);
    } else {
        for (int k = 0; k < 3; ++k) gs[k] = gsc[k];
        out.opacities[i] = g_op;
    }
}

/* Per block of 128 Gaussians: the SH rows come in with coalesced
 * asynchronous 16-byte copies (swizzled rows, see sh_swizzle), each thread
 * forms its Gaussian's gradients (its dL/dsh in place of its row), and the
 * rows go out with coalesced 16-byte stores. Culled Gaussians get zeros. */
__global__ void __launch_bounds__(kProjBwdThreads, 8)
project_backward_kernel(LumenGpuGaussians g, LumenViewCamera camera, LumenRenderOptions opt,
                        const int* __restrict__ radii, const float* __restrict__ grad2d, LumenGpuGradients out) {
    chain_begin();
    __shared__ DevCamera cam_s;
    extern __shared__ float4 sh_rows[];   /* kProjBwdThreads x 12 chunks */
    const int tid = threadIdx.x;
    const long long i0 = (long long)blockIdx.x * kProjBwdThreads;
    const int nblk = (int)(g.count - i0 < kProjBwdThreads ? g.count - i0 : kProjBwdThreads);
    {
        const float4* src = reinterpret_cast<const float4*>(g.sh + i0 * 48);
        for (int c = tid; c < nblk * 12; c += kProjBwdThreads) {
            const int t = c / 12, q = c - 12 * t;
            cp_async16(sh_rows + 12 * t + (q ^ sh_swizzle(t)), src + c);
        }
        cp_async_commit();
    }
    if (tid == 0) setup_camera(camera, cam_s);
    const long long i = i0 + tid;
    const bool visible = tid < nblk && radii[i] > 0;
    cp_async_wait_all();
    __syncthreads();
    float4* row = sh_rows + tid * 12;
    const int swz = sh_swizzle(tid);
    if (visible) {
        project_backward_gaussian(g, cam_s, opt, i, grad2d, out, row, swz);
    } else if (tid < nblk) {
        float* gm = out.means + i * 3;
        float* gs = out.scales + i * 3;
        float* gq = out.quats + i * 4;
        gm[0] = gm[1] = gm[2] = 0.0f;
        gs[0] = gs[1] = gs[2] = 0.0f;
        gq[0] = gq[1] = gq[2] = gq[3] = 0.0f;
        out.opacities[i] = 0.0f;
#pragma unroll
        for (int k = 0; k < 12; ++k) row[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    float4* dst = reinterpret_cast<float4*>(out.sh + i0 * 48);
    for (int c = tid; c < nblk * 12; c += kProjBwdThreads) {
        const int t = c / 12, q = c - 12 * t;
        dst[c] = sh_rows[12 * t + (q ^ sh_swizzle(t))];
    }
}

/* ---------------------------------------------------------------- K8 -- */

constexpr int kL1Blocks = 1024;

__global__ void __launch_bounds__(256)
l1_loss_kernel(const float* __restrict__ pred, const float* __restrict__ target, long long n,
               float* __restrict__ grad, float* __restrict__ partial) {
    chain_begin();
    __shared__ float ws[8];
    const float inv_n = 1.0f / (float)n;
    float sum = 0.0f;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float diff = pred[i] - target[i];
        /* loss.mojo:27-33: the diff >= 0 branch takes +1/n */
        if (diff >= 0.0f) { sum += diff; grad[i] = inv_n; }
        else { sum -= diff; grad[i] = -inv_n; }
    }
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < 8; ++w) t += ws[w];
        partial[blockIdx.x] = t;
    }
}

__global__ void l1_finish_kernel(const float* __restrict__ partial, long long n, float* loss) {
    chain_begin();
    __shared__ float ws[32];
    float t = 0.0f;
    for (int b = threadIdx.x; b < kL1Blocks; b += blockDim.x) t += partial[b];
    t = warp_sum(t);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        float a = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) a += ws[w];
        *loss = n > 0 ? a * (1.0f / (float)n) : 0.0f;
    }
}

}  // namespace lumen

using namespace lumen;

namespace lumen {

/* Six 33 KB CTAs of the compositing adjoint per SM need the largest
 * shared-memory carveout; set per device by configure_once. */
void configure_backward_kernels() {
    auto allow = [](auto kernel, size_t smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
    };
    allow(composite_backward_kernel<false>, sizeof(BackwardSmem<false>));
    allow(composite_backward_kernel<true>, sizeof(BackwardSmem<true>));
}

void configure_once();
LumenStatus check_inputs(const LumenGpuGaussians* g, const LumenViewCamera* cam, const LumenRenderOptions* opt);
LumenStatus map_cuda(cudaError_t e);
cudaEvent_t* stage_timer_take(LumenGpuStageTimer* t);

/* timer: a stage timer whose next frame receives five events (start,
 * after the compositing adjoint, then three after the projection adjoint),
 * taken once the arguments are valid; or nullptr. */
static LumenStatus backward_impl(const LumenGpuGaussians* g, const LumenViewCamera* cam,
                                 const LumenRenderOptions* opt, const LumenGpuFrame* f,
                                 const LumenGpuImage* fwd, const float* grad_rgb, const float* grad_depth,
                                 const float* grad_alpha, LumenGpuGradients* out, LumenGpuStageTimer* timer,
                                 void* stream) {
    LumenStatus st = check_inputs(g, cam, opt);
    if (st != LUMEN_SUCCESS) return st;
    if (!f || !f->scratch || !grad_rgb || !out || !fwd || !fwd->rgb || !fwd->alpha || !fwd->last_idx)
        return LUMEN_ERROR_INVALID_ARGUMENT;
    if (grad_depth && opt->compute_depth && !fwd->depth) return LUMEN_ERROR_INVALID_ARGUMENT;
    if (g->count > 0 &&
        (!out->means || !out->scales || !out->quats || !out->opacities || !out->sh || !out->splat2d ||
         !f->records || !f->visible_ids || !f->radii || !f->ranges || !f->vals[0] || !f->vals[1] ||
         ((uintptr_t)out->splat2d & 15u) != 0))
        return LUMEN_ERROR_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    configure_once();
    cudaEvent_t* ev = nullptr;
    if (timer && !(ev = stage_timer_take(timer))) return LUMEN_ERROR_INVALID_ARGUMENT;
    if (g->count == 0) {
        if (ev)
            for (int k = 0; k < 5; ++k) cudaEventRecord(ev[k], s);
        return LUMEN_SUCCESS;
    }
    Control* ctrl = (Control*)f->scratch;
    if (ev) cudaEventRecord(ev[0], s);
    cudaError_t e = cudaMemsetAsync(out->splat2d, 0, (size_t)g->count * kGrad2DStride * sizeof(float), s);
    if (e != cudaSuccess) return map_cuda(e);
    const int tiles_x = (cam->width + kTile - 1) / kTile;
    const int tiles = tiles_x * ((cam->height + kTile - 1) / kTile);
    /* without an upstream depth gradient the sweep and its sums leave the depth out */
    const bool depth = grad_depth && opt->compute_depth;
    launch_chained(depth ? composite_backward_kernel<true> : composite_backward_kernel<false>, dim3(tiles),
                   dim3(kBwdThreads), depth ? sizeof(BackwardSmem<true>) : sizeof(BackwardSmem<false>), s,
                   (const LumenSplatRecord*)f->records, *f, ctrl, cam->width, cam->height, tiles_x, *opt,
                   (const float*)fwd->rgb, (const float*)fwd->depth, (const float*)fwd->alpha,
                   (const int*)fwd->last_idx, grad_rgb, grad_depth, grad_alpha, out->splat2d, -1.0f);
    if (ev) cudaEventRecord(ev[1], s);
    const long long nb = (g->count + kProjBwdThreads - 1) / kProjBwdThreads;
    launch_chained(project_backward_kernel, dim3((unsigned int)nb), dim3(kProjBwdThreads), kProjBwdStageBytes, s,
                   *g, *cam, *opt, (const int*)f->radii, (const float*)out->splat2d, *out);
    if (ev)
        for (int k = 2; k < 5; ++k) cudaEventRecord(ev[k], s);
    return map_cuda(cudaGetLastError());
}
}  // namespace lumen

extern "C" {

LumenStatus lumen_gpu_render_backward(const LumenGpuGaussians* g, const LumenViewCamera* cam,
                                      const LumenRenderOptions* opt, const LumenGpuFrame* f,
                                      const LumenGpuImage* fwd, const float* grad_rgb, const float* grad_depth,
                                      const float* grad_alpha, LumenGpuGradients* out, void* stream) {
    return backward_impl(g, cam, opt, f, fwd, grad_rgb, grad_depth, grad_alpha, out, nullptr, stream);
}

LumenStatus lumen_gpu_render_backward_timed(const LumenGpuGaussians* g, const LumenViewCamera* cam,
                                            const LumenRenderOptions* opt, const LumenGpuFrame* f,
                                            const LumenGpuImage* fwd, const float* grad_rgb, const float* grad_depth,
                                            const float* grad_alpha, LumenGpuGradients* out,
                                            LumenGpuStageTimer* timer, void* stream) {
    if (!timer) return LUMEN_ERROR_INVALID_ARGUMENT;
    return backward_impl(g, cam, opt, f, fwd, grad_rgb, grad_depth, grad_alpha, out, timer, stream);
}

size_t lumen_gpu_l1_loss_scratch_bytes(void) { return (size_t)kL1Blocks * sizeof(float); }

LumenStatus lumen_gpu_l1_loss(const float* pred, const float* target, int64_t n, float* grad, float* loss,
                              void* scratch, void* stream) {
    if (n < 0 || !loss || !scratch || (n > 0 && (!pred || !target || !grad))) return LUMEN_ERROR_INVALID_ARGUMENT;
    cudaStream_t s = (cudaStream_t)stream;
    float* partial = (float*)scratch;
    if (n > 0) {
        launch_chained(l1_loss_kernel, dim3(kL1Blocks), dim3(256), 0, s, pred, target, (long long)n, grad, partial);
    } else {
        cudaMemsetAsync(partial, 0, lumen_gpu_l1_loss_scratch_bytes(), s);
    }
    launch_chained(l1_finish_kernel, dim3(1), dim3(256), 0, s, (const float*)partial, (long long)n, loss);
    return map_cuda(cudaGetLastError());
}

}  // extern "C"
