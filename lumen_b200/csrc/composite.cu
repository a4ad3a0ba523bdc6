/*
 * composite.cu - K5: per-tile front-to-back alpha compositing.
 *
 * Reference: the per-tile pixel loop of rasterize_scene,
 * src/raster/pipeline.mojo:172-229, with compute_gaussian_pixel_alpha and
 * PixelAccumulator.blend/finalize, src/raster/compositor.mojo:10-89.
 *
 * One CTA of 128 threads per 16x16 tile. A group of 8 lanes shades a 4x4
 * block of pixels, a lane two pixels one above the other, so a warp holds
 * four blocks (an 8x8 quadrant) that walk four lists of their own in step.
 * The tile's sorted instances are processed in chunks of 128, 256 or 512 (a
 * launch parameter the autotuner picks): the threads gather the chunk's 48-byte records (through the sorted
 * visible index) into shared memory and compute which blocks each splat can
 * reach at all (reach_blocks); each warp then builds its four lists and walks
 * them in sorted order, so each pixel blends exactly the reference's
 * sequence. A pixel stops after the blend that saturates it; a warp leaves
 * the chunk once all its pixels stopped, and the CTA stops loading chunks
 * once all 256 pixels stopped.
 *
 * Built with --fmad=false: power, alpha, weights and transmittance round as
 * in the reference, so contributor counts match the CPU restatement bit for
 * bit. The exponential is lumen_expf (shared with the restatement).
 *
 * Why this split: the kernel is bound by the FMA and ALU pipes and by issue
 * (58%, 58% and 74% busy; DRAM 3%), so what counts is the work per blended
 * pixel. Two pixels per lane let the packed FP32 instructions carry two
 * roundings each in one issue slot (the pipe still takes two cycles) and
 * share dx and its products. 4x4 blocks instead of 8x4 keep small splats
 * from occupying lanes they do not reach: of a block's 16 pixels 10 blend an
 * entry (7 for the 720p orbit views), against 16 (9) of 32 before. Four
 * independent lists per warp cost 20 to 30% of their steps in waiting for
 * the longest, less than the shared list of 32 pixels lost.
 * Measured on a B200, one pixel per thread with 8x4 lists -> this form: 1 M
 * Gaussians at 1080p 0.220 -> 0.152 ms (189 -> 121 M warp instructions), 2 M
 * at 4K 0.424 -> 0.279, 64 views of 300 k at 720p 4.79 -> 2.99, 9 mixed
 * views 0.577 -> 0.362.
 */
#include <cmath>
#include <cstring>

#include "composite_common.cuh"

namespace lumen {

/* (uint8)(clamp(c, 0, 1) * 255), truncating (c_api/src/lumen_c.c:541-543). */
__device__ __forceinline__ unsigned char to_byte(float c) {
    if (c < 0.0f) c = 0.0f;
    if (c > 1.0f) c = 1.0f;
    return (unsigned char)(c * 255.0f);
}

/* A chunk of kChunk sorted instances is staged at a time; the warps walk their
 * lists of the chunk's splats kVoteGroup at a time. */
constexpr int kVoteGroup = 4;
constexpr int kCompositeThreads = 128;

template <int kChunk>
struct CompositeSmem {
    float4 geo[kChunk + 1];             /* cx, -cy, depth, opacity; slot kChunk: the padding splat */
    float4 con[kChunk + 1];             /* -0.5 ic00, ic01, 0.5 ic11, - */
    float4 col[kChunk + 1];             /* r, g, b, - */
    __align__(16) unsigned short mask[kChunk];   /* bit 4 row + column: the splat can reach that 4x4 block */
    /* per pixel group: byte offsets (16 x slot) of the splats that can reach it */
    unsigned short list[kBlocks][kChunk + 8];
    unsigned int ticket;
    int special;                        /* some staged value is not finite, or a power may overflow */
};

/* The lists of a warp's groups are padded to one length with slot kChunk, a
 * splat of opacity 0 whose power is above 4.5 away from (0, 0) (conic 1e30):
 * it is skipped like any out-of-reach splat and changes nothing. */
template <int kChunk>
__device__ __forceinline__ void init_padding_splat(CompositeSmem<kChunk>& s) {
    if (threadIdx.x == 0) {
        s.geo[kChunk] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        s.con[kChunk] = make_float4(-1e30f, 0.0f, 1e30f, 0.0f);
        s.col[kChunk] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
}

/* The front-to-back state of a lane's two pixels (PixelAccumulator,
 * compositor.mojo:10-59), one above the other, as packed pairs: the
 * transmittance and the negated sums. cut: the
 * argument of the exponential below which the pixel skips a splat, -4.5
 * while the pixel is open and kClosed (every argument is <= 0) once it has
 * stopped or when it lies outside the image. */
constexpr float kOpen = -4.5f, kClosed = 1.0f;

struct PixelPair {
    f32x2 T, ncr, ncg, ncb, ndep;
    float cut[2];
    unsigned int count[2];
    int last[2];
    __device__ __forceinline__ bool open() const { return cut[0] < 0.0f || cut[1] < 0.0f; }
};

/* lumen_expf_core of both halves of x, operation by operation. */
__device__ __forceinline__ f32x2 expf_core2(f32x2 x) {
    const f32x2 shifter = splat2(12582912.0f);
    const f32x2 t = fma2(x, splat2(1.44269504088896341f), shifter);
    const f32x2 k = add2(t, splat2(-12582912.0f));
    f32x2 r = fma2(k, splat2(-0.693145751953125f), x);
    r = fma2(k, splat2(-1.42860682030941723e-6f), r);
    f32x2 p = splat2(1.98412698412698413e-4f);
    p = fma2(p, r, splat2(1.38888888888888889e-3f));
    p = fma2(p, r, splat2(8.33333333333333333e-3f));
    p = fma2(p, r, splat2(4.16666666666666667e-2f));
    p = fma2(p, r, splat2(1.66666666666666667e-1f));
    p = fma2(p, r, splat2(0.5f));
    p = fma2(p, r, splat2(1.0f));
    p = fma2(p, r, splat2(1.0f));
    float t0, t1;
    unpack2(t, t0, t1);
    return mul2(p, pack2(__uint_as_float(__float_as_uint(t0) * 8388608u + 0x3F800000u),
                         __uint_as_float(__float_as_uint(t1) * 8388608u + 0x3F800000u)));
}

/* n entries (a multiple of kVoteGroup) of the lane's group's list, in sorted
 * order, for the lane's two pixels; every staged value is finite and no
 * power overflows. A pixel stops after the blend that brings T to t_stop.
 * kClamp: some staged splat has opacity above 0.99, so the 0.99 alpha clamp
 * can apply (exp(-power) <= 1). kTrack: count the blended splats and note
 * where a pixel stopped (the byte offset of its slot; only when the view's
 * image asks for contributor counts or last-visited offsets). The arithmetic is the reference's, operation by
 * operation, with signs flipped where that saves one (exact) and a pixel that
 * does not blend the splat given alpha 0, which leaves its sums and its
 * transmittance as they are.
 *
 * minus_one holds (-1, -1) in a form the compiler cannot see (a kernel
 * argument): every sum of a product is written fma2(product, minus_one, sum),
 * a subtraction rounded once like the reference's sum. Written add2, it was
 * contracted with the product into one fused multiply-add, against the
 * explicit rounding of both and --fmad=false. */
template <int kChunk, bool kClamp, bool kTrack>
__device__ __forceinline__ void blend_list(const CompositeSmem<kChunk>& s, const unsigned short* lst, int n,
                                           float pxc, f32x2 pyc, float t_stop, f32x2 minus_one, PixelPair& p) {
    const f32x2 one = splat2(1.0f);
    for (int t0 = 0; t0 < n; t0 += kVoteGroup) {
#pragma unroll
        for (int u = 0; u < kVoteGroup; ++u) {
            const unsigned int off = lst[t0 + u];
            const float4 g = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(s.geo) + off);
            const float4 c = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(s.con) + off);
            const float4 k = *reinterpret_cast<const float4*>(reinterpret_cast<const char*>(s.col) + off);
            /* compute_gaussian_pixel_alpha, compositor.mojo:62-89 */
            const float dx = pxc - g.x;
            const f32x2 dy = add2(pyc, splat2(g.y));
            const f32x2 q = fma2(mul2(mul2(splat2(c.z), dy), dy), minus_one,
                                 fma2(mul2(splat2(c.y * dx), dy), minus_one, splat2(c.x * dx * dx)));
            float x0, x1;
            unpack2(q, x0, x1);
            x0 = fminf(x0, 0.0f);
            x1 = fminf(x1, 0.0f);
            const f32x2 raw = mul2(splat2(g.w), expf_core2(pack2(x0, x1)));
            float a0, a1;
            unpack2(raw, a0, a1);
            /* PixelAccumulator.blend, compositor.mojo:25-53 */
            const bool b0 = !(x0 < p.cut[0]) && !(a0 < min_alpha());
            const bool b1 = !(x1 < p.cut[1]) && !(a1 < min_alpha());
            a0 = b0 ? (kClamp ? fminf(a0, (float)0.99) : a0) : 0.0f;
            a1 = b1 ? (kClamp ? fminf(a1, (float)0.99) : a1) : 0.0f;
            const f32x2 alpha = pack2(a0, a1);
            const f32x2 w = mul2(alpha, p.T);
            p.ncr = fma2(mul2(splat2(k.x), w), minus_one, p.ncr);
            p.ncg = fma2(mul2(splat2(k.y), w), minus_one, p.ncg);
            p.ncb = fma2(mul2(splat2(k.z), w), minus_one, p.ncb);
            p.ndep = fma2(mul2(splat2(g.z), w), minus_one, p.ndep);
            p.T = mul2(p.T, fma2(alpha, minus_one, one));
            float v0, v1;
            unpack2(p.T, v0, v1);
            const bool stop0 = b0 && v0 <= t_stop, stop1 = b1 && v1 <= t_stop;
            if (stop0) p.cut[0] = kClosed;
            if (stop1) p.cut[1] = kClosed;
            if (kTrack) {
                p.count[0] += b0;
                p.count[1] += b1;
                if (stop0) p.last[0] = (int)off;
                if (stop1) p.last[1] = (int)off;
            }
        }
        if (__all_sync(0xffffffffu, !p.open())) break;
    }
}

/* The same for a chunk with a value that is not finite or a power that may
 * overflow: one pixel at a time, nothing computed for a pixel that skips. */
template <int kChunk>
__device__ __forceinline__ void blend_list_general(const CompositeSmem<kChunk>& s, const unsigned short* lst, int n,
                                                   float pxc, float pyc0, float t_stop, PixelPair& p) {
    float T[2], cr[2], cg[2], cb[2], dep[2];
    unpack2(p.T, T[0], T[1]);
    unpack2(p.ncr, cr[0], cr[1]);
    unpack2(p.ncg, cg[0], cg[1]);
    unpack2(p.ncb, cb[0], cb[1]);
    unpack2(p.ndep, dep[0], dep[1]);
#pragma unroll 1
    for (int t = 0; t < n; ++t) {
        const unsigned int j = lst[t] >> 4;
        const float4 g = s.geo[j], c = s.con[j], k = s.col[j];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (p.cut[h] > 0.0f) continue;
            const float dx = pxc - g.x, dy = (pyc0 + (float)h) + g.y;
            float x = c.x * dx * dx - c.y * dx * dy - c.z * dy * dy;
            if (x > 0.0f) x = 0.0f;
            else if (x < kOpen) continue;
            float alpha = g.w * lumen_expf_core(x);
            if (alpha > (float)0.99) alpha = (float)0.99;
            if (alpha < min_alpha()) continue;
            const float w = alpha * T[h];
            cr[h] -= k.x * w;
            cg[h] -= k.y * w;
            cb[h] -= k.z * w;
            dep[h] -= g.z * w;
            T[h] *= (1.0f - alpha);
            ++p.count[h];
            if (T[h] <= t_stop) {
                p.cut[h] = kClosed;
                p.last[h] = 16 * (int)j;
            }
        }
    }
    p.T = pack2(T[0], T[1]);
    p.ncr = pack2(cr[0], cr[1]);
    p.ncg = pack2(cg[0], cg[1]);
    p.ncb = pack2(cb[0], cb[1]);
    p.ndep = pack2(dep[0], dep[1]);
}

/* The lists of the warp's four groups from the chunk's masks: each lane
 * takes kChunk / 32 consecutive slots, the four counts are scanned over the
 * warp as 16-bit fields of two words, and every lane then appends its slots
 * to the lists in order. open: the bits (0, 1, 4, 5) of the groups that
 * still have an open pixel; the others get no entries. Returns the common
 * padded length. */
template <int kChunk>
__device__ __forceinline__ int build_lists(CompositeSmem<kChunk>& s, int warp, int lane, unsigned int open) {
    constexpr int kPer = kChunk / 32;
    const int shift = 8 * (warp >> 1) + 2 * (warp & 1);   /* the warp's 2x2 blocks in the 4x4 of the mask */
    unsigned int m[kPer];
    unsigned int c01 = 0u, c23 = 0u;
#pragma unroll
    for (int q = 0; q < kPer / 2; ++q) {
        const unsigned int two = reinterpret_cast<const unsigned int*>(s.mask)[lane * (kPer / 2) + q];
        m[2 * q] = (two >> shift) & open;
        m[2 * q + 1] = (two >> (16 + shift)) & open;
    }
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
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
    const int padded = (longest + kVoteGroup - 1) & ~(kVoteGroup - 1);
#pragma unroll
    for (int g = 0; g < 4; ++g)
        for (int k = n[g] + lane; k < padded; k += 32) s.list[4 * warp + g][k] = (unsigned short)(16 * kChunk);
    __syncwarp();
    return padded;
}

/* finalize, compositor.mojo:55-59, and the store of one pixel */
__device__ __forceinline__ void store_pixel(const ViewDesc& vd, const LumenRenderOptions& opt, bool background, int px,
                                            int py, float T, float cr, float cg, float cb, float dep,
                                            unsigned int count, int last) {
    if (px >= vd.cam.width || py >= vd.cam.height) return;
    const LumenGpuImage& img = vd.img;
    const long long pix = (long long)py * vd.cam.width + px;
    const float acc = 1.0f - T;   /* the value the reference's blend leaves (compositor.mojo:51) */
    /* last visited instance as an offset within the view's instances
     * (positions are below 2^30) */
    if (last >= 0) last -= (int)vd.inst_begin;
    if (background) { cr += T; cg += T; cb += T; }
    if (img.rgb) {
        img.rgb[pix * 3 + 0] = cr;
        img.rgb[pix * 3 + 1] = cg;
        img.rgb[pix * 3 + 2] = cb;
    }
    if (img.rgb8) {
        img.rgb8[pix * 3 + 0] = to_byte(cr);
        img.rgb8[pix * 3 + 1] = to_byte(cg);
        img.rgb8[pix * 3 + 2] = to_byte(cb);
    }
    if (img.depth) img.depth[pix] = opt.compute_depth ? dep : 0.0f;
    if (img.alpha) img.alpha[pix] = acc;
    if (img.n_contrib) img.n_contrib[pix] = count;
    if (img.last_idx) img.last_idx[pix] = last;
}

/* One tile of the batch (batch-wide id gtile, owned by the last view whose
 * tile_begin <= gtile). */
template <int kChunk, bool kTrack>
__device__ __forceinline__ void composite_tile(CompositeSmem<kChunk>& s, const ViewTable* __restrict__ vt,
                                               const LumenSplatRecord* __restrict__ records, const LumenGpuFrame& f,
                                               long long capacity, Control* __restrict__ ctrl,
                                               const LumenRenderOptions& opt, float t_stop, f32x2 minus_one,
                                               int n_views, long long gtile) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    /* everything that depends on the tile's number alone is read first, so
     * that these reads, the view's and the first indices' overlap */
    int rs = f.ranges[2 * gtile], re = f.ranges[2 * gtile + 1];
    const long long n_instances = (long long)ctrl->n_instances;
    const unsigned int n_visible = ctrl->n_visible;
    const unsigned int* __restrict__ vals = ctrl->list_buffer ? f.vals[1] : f.vals[0];
    const long long K = n_instances < capacity ? n_instances : capacity;
    bool listed = rs != -1 && rs < re;
    if (listed && (rs < 0 || (long long)re > K)) {
        /* self-check: a range outside the sorted instances */
        if (tid == 0) atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
        listed = false;
    }
    constexpr int kRounds = kChunk / kCompositeThreads;
    unsigned int next[kRounds];   /* the next chunk's visible indices, read ahead */
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
        const int i = rs + r * kCompositeThreads + tid;
        next[r] = listed && i < re ? vals[i] : 0u;
    }
    const int view = n_views == 1 ? 0 : find_view_by_tile_warp(vt, n_views, gtile);
    const ViewDesc& vd = vt->view[view];
    const int tile = (int)(gtile - vd.tile_begin);
    const int tx = tile % vd.tiles_x, ty = tile / vd.tiles_x;
    /* a warp shades an 8x8 quadrant, a group of 8 lanes a 4x4 block of it,
     * a lane two pixels one above the other */
    const int group = lane >> 3;
    const int px = tx * kTile + 8 * (warp & 1) + 4 * (group & 1) + (lane & 3);
    const int py = ty * kTile + 8 * (warp >> 1) + 4 * (group >> 1) + 2 * ((lane >> 2) & 1);
    const bool column = px < vd.cam.width;

    PixelPair p;
    p.T = splat2(1.0f);
    p.ncr = p.ncg = p.ncb = p.ndep = splat2(-0.0f);
    p.cut[0] = column && py < vd.cam.height ? kOpen : kClosed;
    p.cut[1] = column && py + 1 < vd.cam.height ? kOpen : kClosed;
    p.count[0] = p.count[1] = 0u;
    p.last[0] = p.last[1] = -1;
    bool background = opt.white_background != 0;

    if (vd.inst_begin < 0) {
        /* pipeline.mojo:162-163: no instances in the view, the output stays zero */
        background = false;
    } else {
        if (listed) {
            const float pxc = (float)px + 0.5f, pyc = (float)py + 0.5f;
            const f32x2 pyc2 = pack2(pyc, pyc + 1.0f);
            const float tile_x0 = (float)(tx * kTile), tile_y0 = (float)(ty * kTile);
            if (tid == 0) s.special = 0;
            for (int cs = rs; cs < re; cs += kChunk) {
                if (__syncthreads_count(p.open()) == 0) break;
                int high = 0;
#pragma unroll
                for (int r = 0; r < kRounds; ++r) {
                    const int slot = r * kCompositeThreads + tid;
                    const int i = cs + slot;
                    unsigned int m = 0;
                    if (i < re) {
                        const unsigned int v = next[r];
                        next[r] = i + kChunk < re ? vals[i + kChunk] : 0u;
                        if (v >= n_visible) {   /* self-check: an index beyond the visible records */
                            atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
                        } else {
                            const float4* r4 = reinterpret_cast<const float4*>(records + v);
                            const float4 geo = __ldg(r4), con = __ldg(r4 + 1), col = __ldg(r4 + 2);
                            s.geo[slot] = make_float4(geo.x, -geo.y, geo.z, geo.w);
                            /* 0.5 folded into the conic: scaling by a power of two commutes
                             * with rounding, and so does the sign, so the argument of the
                             * exponential below equals the reference's
                             * -0.5 * (a dx dx + 2 b dx dy + c dy dy) bit for bit */
                            s.con[slot] = make_float4(-0.5f * con.x, con.y, 0.5f * con.z, 0.0f);
                            s.col[slot] = col;
                            bool finite;
                            m = reach_blocks(geo, con, tile_x0, tile_y0, &finite);
                            finite = finite && fabsf(col.x) + fabsf(col.y) + fabsf(col.z) + fabsf(geo.z) < 1e30f;
                            if (!finite) s.special = 1;   /* for the rest of the tile */
                            high |= geo.w > (float)0.99;
                        }
                    }
                    s.mask[slot] = (unsigned short)m;
                }
                const bool clamp = __syncthreads_or(high) != 0;
                const unsigned int b = __ballot_sync(0xffffffffu, p.open());
                if (b == 0u) continue;
                const unsigned int open = ((b & 0xFFu) ? 1u : 0u) | ((b & 0xFF00u) ? 2u : 0u) |
                                          ((b & 0xFF0000u) ? 16u : 0u) | ((b & 0xFF000000u) ? 32u : 0u);
                const int n = build_lists<kChunk>(s, warp, lane, open);
                const unsigned short* lst = s.list[4 * warp + group];
                const bool open0 = p.cut[0] < 0.0f, open1 = p.cut[1] < 0.0f;
                if (s.special) blend_list_general<kChunk>(s, lst, n, pxc, pyc, t_stop, p);
                else if (clamp) blend_list<kChunk, true, kTrack>(s, lst, n, pxc, pyc2, t_stop, minus_one, p);
                else blend_list<kChunk, false, kTrack>(s, lst, n, pxc, pyc2, t_stop, minus_one, p);
                if (open0 && p.cut[0] > 0.0f) p.last[0] = cs + (p.last[0] >> 4);
                if (open1 && p.cut[1] > 0.0f) p.last[1] = cs + (p.last[1] >> 4);
            }
            /* a pixel that never saturated visited the whole range */
            if (p.cut[0] < 0.0f) p.last[0] = re - 1;
            if (p.cut[1] < 0.0f) p.last[1] = re - 1;
        }
    }
    float T[2], cr[2], cg[2], cb[2], dep[2];
    unpack2(p.T, T[0], T[1]);
    unpack2(p.ncr, cr[0], cr[1]);
    unpack2(p.ncg, cg[0], cg[1]);
    unpack2(p.ncb, cb[0], cb[1]);
    unpack2(p.ndep, dep[0], dep[1]);
#pragma unroll
    for (int h = 0; h < 2; ++h)
        store_pixel(vd, opt, background, px, py + h, T[h], -cr[h], -cg[h], -cb[h], -dep[h], p.count[h], p.last[h]);
}

/* One CTA per tile of the batch. kTrack: keep contributor counts and
 * last-visited offsets (some view's image asks for them). */
template <int kChunk, bool kTrack>
__global__ void __launch_bounds__(kCompositeThreads, kCompositeBlocksPerSm)
composite_kernel(const ViewTable* __restrict__ vt, int n_views, const LumenSplatRecord* __restrict__ records,
                 LumenGpuFrame f, long long capacity, Control* __restrict__ ctrl, LumenRenderOptions opt,
                 long long tile_offset, bool in_line, float t_stop, float minus_one) {
    chain_begin();
    __shared__ CompositeSmem<kChunk> s;
    init_padding_splat(s);
    composite_tile<kChunk, kTrack>(s, vt, records, f, capacity, ctrl, opt, t_stop, splat2(minus_one), n_views,
                                   in_line ? tile_in_line(ctrl, blockIdx.x) : tile_offset + blockIdx.x);
}

/* The transmittance at or below which a blend stops its pixel. Termination
 * mode 0 compares T with the threshold itself (compositor.mojo:53); mode 1
 * stops when 1 - T, rounded, reaches the threshold, which holds for every T
 * up to the largest float for which it holds. */
static float stop_transmittance(const LumenRenderOptions& opt) {
    const float thr = opt.term_threshold;
    if (opt.term_mode != 1) return thr;
    if (!(1.0f >= thr)) return -1.0f;      /* never (T >= 0) */
    if (0.0f >= thr) return INFINITY;      /* after the first blend */
    unsigned int lo = 0u, hi = 0x3F800000u;   /* bits of 0 (holds) and of 1 (does not) */
    while (hi - lo > 1u) {
        const unsigned int mid = lo + (hi - lo) / 2u;
        float t;
        std::memcpy(&t, &mid, sizeof(t));
        if (1.0f - t >= thr) lo = mid;
        else hi = mid;
    }
    float t;
    std::memcpy(&t, &lo, sizeof(t));
    return t;
}

template <int kChunk, bool kTrack>
static void launch_composite_chunk(const ViewTable* vt, int n_views, const LumenGpuFrame& f, Control* ctrl,
                                   const LumenRenderOptions& opt, long long tile_offset, long long n_tiles, bool whole, cudaStream_t st) {
    launch_chained(composite_kernel<kChunk, kTrack>, dim3((unsigned int)n_tiles), dim3(kCompositeThreads), 0, st, vt,
                   n_views, (const LumenSplatRecord*)f.records, f, (long long)f.instance_capacity, ctrl, opt,
                   tile_offset, whole, stop_transmittance(opt), -1.0f);
}

template <int kChunk>
static void launch_composite_track(const ViewTable* vt, int n_views, const LumenGpuFrame& f, Control* ctrl,
                                   const LumenRenderOptions& opt, long long tile_offset, long long n_tiles, bool whole,
                                   bool track, cudaStream_t st) {
    if (track)
        launch_composite_chunk<kChunk, true>(vt, n_views, f, ctrl, opt, tile_offset, n_tiles, whole, st);
    else
        launch_composite_chunk<kChunk, false>(vt, n_views, f, ctrl, opt, tile_offset, n_tiles, whole, st);
}

/* Shades tiles [tile_offset, tile_offset + n_tiles) of the batch. whole: these
 * are all its tiles, so they may go longest list first. chunk: instances
 * staged per round, one of kCompositeChunks. track: some view's image asks for
 * contributor counts or last-visited offsets. */
void launch_composite(const ViewTable* vt, int n_views, const LumenGpuFrame& f, Control* ctrl,
                      const LumenRenderOptions& opt, long long tile_offset, long long n_tiles, bool whole,
                      int chunk, bool track, cudaStream_t st) {
    if (n_tiles <= 0) return;
    /* Not chained: blocks that are resident before the list kernel ends are
     * placed where that leaves room, so the first (longest) tiles crowd on a
     * few SMs. Launched after it, they spread over all: 100 k splats at
     * 999x563 74 -> 58 us without an order, 79 -> 40 with one; 50 k at 640x480
     * the whole frame 110 -> 98.5 us. */
    ChainedLaunches chained(false);
    switch (chunk) {
        case 128:
            launch_composite_track<128>(vt, n_views, f, ctrl, opt, tile_offset, n_tiles, whole, track, st);
            break;
        case 512:
            launch_composite_track<512>(vt, n_views, f, ctrl, opt, tile_offset, n_tiles, whole, track, st);
            break;
        default:
            launch_composite_track<256>(vt, n_views, f, ctrl, opt, tile_offset, n_tiles, whole, track, st);
            break;
    }
}

}  // namespace lumen
