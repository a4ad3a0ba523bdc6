/*
 * project.cu - K1 (projection with the compacting scan) and K2 (emission
 * of the splats' cells in depth order).
 *
 * Reference: the geometry-and-culling loop of rasterize_scene,
 * src/raster/pipeline.mojo:84-157. There, visible splats get consecutive
 * indices in Gaussian order (pipeline.mojo:141-149) and each appends one
 * key per covered tile (:152-157); the keys are then stably sorted (:166).
 *
 * K1, for one view of few Gaussians (below for the rest): a block of 128
 * threads projects 128 consecutive Gaussians (their SH coefficients staged in
 * shared memory by asynchronous copies) and scans their visibility flags; the global offset comes from a decoupled look-back
 * over blocks taken in ticket order, so visible indices are exactly the
 * reference's sequential ones. Each visible splat writes its 48-byte record,
 * its Gaussian index, its tile rectangle and its depth key.
 *
 * K2 (after the visible splats were stably sorted by depth key): a block
 * takes 256 consecutive splats of the depth order, scans their cell counts
 * (decoupled look-back again; a cell is 4x4 tiles), and writes one (cell and
 * tile mask, visible index) pair per touched cell, cooperatively, so
 * consecutive threads write consecutive pairs. A stable sort of these pairs by
 * cell and a stable split of each cell's list over its tiles (lists.cu) yield
 * the reference's permutation: in both, a tile's instances are ordered by
 * (depth key, visible index).
 *
 * Memory: K1 reads 236 B per Gaussian once and writes 68 B per visible
 * splat + 4 B per Gaussian; K2 reads 12 B per visible splat and writes 8 B
 * per pair (about two pairs per splat where there are seven instances).
 */
#include "splat_common.cuh"

namespace lumen {

struct ProjSmem {
    LumenGpuGaussians g;         /* the view's */
    DevCamera cam;
    unsigned int blk;
    unsigned int warp_tot[kProjThreads / 32];
    unsigned long long vis_base;
    unsigned long long key_or, key_or_not;
};

constexpr int kCamWords = (int)(sizeof(DevCamera) / 4);
constexpr int kGaussiansWords = (int)(sizeof(LumenGpuGaussians) / 4);
static_assert(sizeof(DevCamera) % 4 == 0 && kCamWords <= kProjThreads, "camera copy layout");
static_assert(sizeof(LumenGpuGaussians) % 4 == 0 && kGaussiansWords <= 32, "scene copy layout");

__device__ __forceinline__ void copy_camera(DevCamera& dst, const DevCamera& src) {
    const int tid = threadIdx.x;
    if (tid < kCamWords) reinterpret_cast<unsigned int*>(&dst)[tid] = reinterpret_cast<const unsigned int*>(&src)[tid];
}

/* The projection of one view of few Gaussians (kOnePassBlocks): each CTA takes
 * a 128-Gaussian block by ticket, and visible indices run over the blocks in
 * order. One launch, but the look-back is a chain: the resident CTAs start
 * together, and sums travel 32 blocks per step of about 0.45 us. */
__global__ void __launch_bounds__(kProjThreads)
project_kernel(const ViewTable* __restrict__ vt, LumenRenderOptions opt, LumenGpuFrame f, Control* ctrl,
               unsigned long long* lb) {
    chain_begin();
    __shared__ ProjSmem s;
    extern __shared__ float4 sh_stage[];   /* kProjThreads x 12: the block's SH coefficients */
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long total_blocks = vt->hdr.total_blocks;
    copy_camera(s.cam, vt->view[0].dcam);
    if (tid >= kProjThreads - kGaussiansWords) {
        const int w = tid - (kProjThreads - kGaussiansWords);
        reinterpret_cast<unsigned int*>(&s.g)[w] = reinterpret_cast<const unsigned int*>(&vt->view[0].g)[w];
    }
    if (tid == 0) {
        s.blk = atomicAdd(&ctrl->proj_ticket, 1u);
        s.key_or = 0ull;
        s.key_or_not = 0ull;
    }
    __syncthreads();
    const int blk = (int)s.blk;
    if ((long long)blk >= total_blocks) return;
    const long long i0 = (long long)blk * kProjThreads, i = i0 + tid;
    const long long count = s.g.count;
    /* the block's SH rows (192 B per Gaussian, contiguous) go to shared
     * memory with coalesced 16-byte asynchronous copies, overlapped with
     * the loads of the other parameters */
    {
        const int nblk = (int)(count - i0 < kProjThreads ? count - i0 : kProjThreads);
        const float4* src = reinterpret_cast<const float4*>(s.g.sh + i0 * 48);
        for (int c = tid; c < nblk * 12; c += kProjThreads) {
            const int t = c / 12, q = c - 12 * t;
            cp_async16(sh_stage + 12 * t + (q ^ sh_swizzle(t)), src + c);
        }
        cp_async_commit();
    }
    float mx = 0.0f, my = 0.0f, mz = 0.0f, sx = 0.0f, sy = 0.0f, sz = 0.0f, op = 0.0f;
    float4 q = make_float4(1.0f, 0.0f, 0.0f, 0.0f);
    if (i < count) {
        const LumenGpuGaussians& g = s.g;
        const float* m = g.means + i * 3;
        const float* sc = g.scales + i * 3;
        q = __ldg(reinterpret_cast<const float4*>(g.quats) + i);
        mx = __ldg(m); my = __ldg(m + 1); mz = __ldg(m + 2);
        sx = __ldg(sc); sy = __ldg(sc + 1); sz = __ldg(sc + 2);
        op = __ldg(g.opacities + i);
    }
    cp_async_wait_all();
    __syncthreads();

    Projected p;
    p.visible = false;
    p.radius = 0;
    if (i < count) {
        p = project_gaussian(s.cam, mx, my, mz, sx, sy, sz, Quat{q.x, q.y, q.z, q.w}, op,
                             reinterpret_cast<const float*>(sh_stage + tid * 12), opt, sh_swizzle(tid));
        if (f.radii) f.radii[i] = p.visible ? p.radius : 0;
    }
    unsigned int block_vis = 0;
    const unsigned int vis_local = block_exclusive_scan<kProjThreads>(p.visible ? 1u : 0u, s.warp_tot, &block_vis);
    if (tid == 0) st_volatile_u64(lb + blk, (blk == 0 ? kDescIncl64 : kDescAgg64) | block_vis);
    if (warp == 0) {
        const unsigned long long e = blk > 0 ? lookback64(lb, blk, &ctrl->error_flags) : 0ull;
        if (lane == 0) {
            s.vis_base = e;
            if (blk > 0) st_volatile_u64(lb + blk, kDescIncl64 | (e + block_vis));
        }
    }
    __syncthreads();
    const unsigned long long vis_base = s.vis_base;
    unsigned long long kor = 0ull, knot = 0ull;
    if (p.visible) {
        const unsigned long long vid = vis_base + vis_local;
        float4* dst = reinterpret_cast<float4*>(f.records + vid);
        dst[0] = make_float4(p.cx, p.cy, p.z, p.op);
        dst[1] = make_float4(p.ic00, p.ic01, p.ic11, 0.0f);
        dst[2] = make_float4(p.r, p.g, p.b, 0.0f);
        f.visible_ids[vid] = (unsigned int)i;
        f.rects[vid] = pack_rect(p.min_tx, p.min_ty, p.max_tx, p.max_ty, 0);
        const unsigned int dk = depth_key(p.z, opt.key_mode);
        f.depth_keys[0][vid] = dk;
        f.depth_order[0][vid] = (unsigned int)vid;
        kor = dk;
        knot = ~(unsigned long long)dk & 0xFFFFFFFFull;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        kor |= __shfl_xor_sync(0xffffffffu, kor, o);
        knot |= __shfl_xor_sync(0xffffffffu, knot, o);
    }
    if (lane == 0 && block_vis) {
        atomicOr(&s.key_or, kor);
        atomicOr(&s.key_or_not, knot);
    }
    __syncthreads();
    if (tid == 0) {
        if (block_vis) {
            atomicOr(&ctrl->depth_sort.key_or, s.key_or);
            atomicOr(&ctrl->depth_sort.key_or_not, s.key_or_not);
        }
        if ((long long)blk == total_blocks - 1) {
            ctrl->n_visible = (unsigned int)(vis_base + block_vis);
            ctrl->depth_sort.n = vis_base + block_vis;
        }
    }
}

/* Pairs of an emission warp resolved to their splats per window. */
constexpr int kEmitWindow = 256;
constexpr int kEmitPerLane = kEmitWindow / 32;
static_assert(kEmitPerLane == 8, "two 16-byte slot groups per lane");

constexpr int kEmitWarps = kEmitThreads / 32;
constexpr int kEmitMaxRounds = 4;

struct EmitSmem {
    /* per warp and window slot: 1 + the lane whose splat holds the pair */
    __align__(16) unsigned int owner[kEmitThreads / 32][kEmitWindow];
    unsigned int blk;
    unsigned int warp_pairs[kEmitMaxRounds][kEmitWarps], warp_tiles[kEmitMaxRounds][kEmitWarps];
    unsigned long long base;             /* the blocks before: instances and pairs (pack_counts) */
    /* per splat: its first pair (block-relative), cells per rectangle row,
     * the batch-wide id of its first cell, cells per view row */
    uint4 run[kEmitThreads];
    /* per splat: 1 / (cells per rectangle row), as bits, for the row of a
     * pair; its visible index */
    uint2 aux[kEmitThreads];
    unsigned long long rect[kEmitThreads];
    unsigned int hist[4][256];            /* the CTA's cell ids: counts of each digit value */
    unsigned int cut, cut_tiles, kept;    /* at the instance capacity (emit_cut) */
};
static_assert(kEmitThreads == 256, "one emission thread per digit value clears and adds the block's counts");

/* Owners of the warp's window [a, a + kEmitWindow): slot k of s.owner[warp]
 * gets 1 + the lane whose splat holds pair a + k (block-relative). Returns
 * the window's pair count. */
__device__ __forceinline__ unsigned int emit_window_owners(EmitSmem& s, int warp, int lane, unsigned int a,
                                                           unsigned int excl, unsigned int cnt, unsigned int w_end) {
    unsigned int* own = s.owner[warp];
    uint4* o4 = reinterpret_cast<uint4*>(own) + lane * 2;
    o4[0] = make_uint4(0u, 0u, 0u, 0u);
    o4[1] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    if (cnt && excl + cnt > a && excl < a + kEmitWindow) own[(excl > a ? excl : a) - a] = (unsigned int)lane + 1u;
    __syncwarp();
    /* inclusive prefix maximum: eight consecutive slots per lane, then
     * across the lanes */
    const uint4 g0 = o4[0], g1 = o4[1];
    unsigned int m[kEmitPerLane] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
    for (int k = 1; k < kEmitPerLane; ++k) m[k] = max(m[k], m[k - 1]);
    unsigned int x = m[kEmitPerLane - 1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x = max(x, y);
    }
    unsigned int pre = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) pre = 0u;
    o4[0] = make_uint4(max(pre, m[0]), max(pre, m[1]), max(pre, m[2]), max(pre, m[3]));
    o4[1] = make_uint4(max(pre, m[4]), max(pre, m[5]), max(pre, m[6]), max(pre, m[7]));
    __syncwarp();
    return w_end - a < (unsigned int)kEmitWindow ? w_end - a : kEmitWindow;
}

/* Row of block-relative pair j of splat lo in its rectangle of cells (rows
 * outer, columns inner) and *column. */
__device__ __forceinline__ unsigned int emit_row(const EmitSmem& s, int lo, const uint4& rn, unsigned int j,
                                                 unsigned int* column) {
    const unsigned int w = rn.y;
    const unsigned int q = j - rn.x;
    /* q / w through the reciprocal (exact after one correction step while
     * q < 2^20), integer division beyond */
    unsigned int row;
    if (q < (1u << 20)) {
        row = (unsigned int)((float)q * __uint_as_float(s.aux[lo].x));
        if (row * w > q) --row;
        else if ((row + 1u) * w <= q) ++row;
    } else {
        row = q / w;
    }
    *column = q - row * w;
    return row;
}

/* The block in which the instances reach the capacity (`room` of its own are
 * kept): the first splat that does not fit wholly (s.cut), how many of its
 * tiles do (s.cut_tiles, row-major in its rectangle, a prefix of its cells)
 * and the block's pairs up to there (s.kept). One thread; a frame that
 * overflows is rendered again. */
__device__ __noinline__ void emit_cut(EmitSmem& s, unsigned int room, int n) {
    s.cut = (unsigned int)n;
    s.cut_tiles = 0u;
    s.kept = 0u;
    unsigned long long used = 0ull;
    for (int k = 0; k < n; ++k) {
        const unsigned long long r = s.rect[k];
        const unsigned int w = (unsigned int)(rect_max_tx(r) - rect_min_tx(r) + 1);
        const unsigned int h = (unsigned int)(rect_max_ty(r) - rect_min_ty(r) + 1);
        if (used + (unsigned long long)w * h <= room) {
            used += (unsigned long long)w * h;
            continue;
        }
        const unsigned int left = room - (unsigned int)used;
        s.cut = (unsigned int)k;
        s.cut_tiles = left;
        const unsigned int row = left / w, col = left - row * w;   /* `row` whole rows and `col` tiles of the next */
        const unsigned int cx0 = rect_min_tx(r) / kCellSide, cy0 = rect_min_ty(r) / kCellSide, cw = s.run[k].y;
        unsigned int cells = 0u;
        if (row > 0) cells = cw * ((rect_min_ty(r) + row - 1) / kCellSide - cy0 + 1);
        if (col > 0) {
            const unsigned int before = cw * ((rect_min_ty(r) + row) / kCellSide - cy0);
            cells = max(cells, before + (rect_min_tx(r) + col - 1) / kCellSide - cx0 + 1);
        }
        s.kept = s.run[k].x + cells;
        return;
    }
}

/* A splat's rectangle in cells, and its tile and cell counts. */
struct CellRect {
    unsigned int tiles;   /* below 2^24, so that 256 of them fit 32 bits */
    unsigned int cx, cy, cw, pairs;
};

__device__ __forceinline__ CellRect cell_rect(unsigned long long r) {
    const unsigned int mnx = rect_min_tx(r), mny = rect_min_ty(r), mxx = rect_max_tx(r), mxy = rect_max_ty(r);
    CellRect c;
    c.tiles = (mxx - mnx + 1u) * (mxy - mny + 1u);
    c.cx = mnx / kCellSide;
    c.cy = mny / kCellSide;
    c.cw = mxx / kCellSide - c.cx + 1u;
    c.pairs = c.cw * (mxy / kCellSide - c.cy + 1u);
    return c;
}

/* A warp whose splats touch at most this many cells each writes them one
 * splat per lane; beyond, its lanes share the pairs evenly (a splat over the
 * whole image would hold its warp up). */
constexpr unsigned int kEmitLaneCells = 16;

/* kRounds rounds of 256 consecutive splats of the depth order per ticket: one
 * pair per cell that a splat's rectangle touches (batch-wide cell id and tile
 * mask, visible index), in depth order, cells row-major. Tickets are taken in
 * order, and a ticket's splats sum up their predecessors' instances and pairs
 * by decoupled look-back.
 *
 * The emission also does the cell sort's preparation, so that the sort
 * needs no pass of its own over the pairs: it counts the digit values of the
 * cell ids it writes (per CTA in shared memory, added to the sort's histogram
 * once all its tickets are done) and clears the sort's look-back descriptors of
 * the 256 * sort_items-key tiles that start among its pairs. It also fills the
 * cells' ranges with (-1, -1) for the sort's last pass and the tiles' with zeros
 * for the lists' counts.
 *
 * Instances (the tiles of the rectangles) are only counted here; those
 * beyond the capacity are left out of the pairs, so that the lists hold the
 * first `capacity` instances of the depth order, row-major per splat.
 *
 * Bound by the random 8-byte gathers of the rectangles, and before that by
 * the look-back: the resident CTAs start together, so inclusive sums travel
 * 32 tickets per step of about 0.45 us, and with 256 splats per ticket 1 M
 * splats waited 40 of 57 us. Four rounds per ticket make the chain a quarter
 * as long and keep four gathers per thread in flight: 57 -> 41 us at 1 M
 * splats and 1080p, 123 -> 74 at 2 M and 4K, 850 -> 570 for 64 views of
 * 300 k. Below three tickets of 1024 per SM one round spreads the splats
 * over more CTAs (250 k splats: 23 us, against 33 with four). Wider look-back
 * steps (8 descriptors per lane) and a scan in kernels of its own were slower
 * (1 M: 78 and 61 us). */
template <int kRounds>
__global__ void __launch_bounds__(kEmitThreads, 6)
emit_kernel(const ViewTable* __restrict__ vt, LumenGpuFrame f, Control* ctrl, unsigned long long* lb,
            unsigned int* sort_lb, long long sort_lb_tiles, int sort_tile_keys, bool wide) {
    chain_begin();
    __shared__ EmitSmem s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long V = ctrl->n_visible;
    const unsigned int* order = ctrl->depth_sort.sorted_buffer ? f.depth_order[1] : f.depth_order[0];
    const unsigned int cap = (unsigned int)f.instance_capacity;   /* below 2^30 */
    /* the digits of the cell ids, which are below the batch's cell count */
    const long long n_cells = vt->hdr.total_cells;
    const bool packed = n_cells <= kPackedCells;
    const CellDigits digits(n_cells);
    const int nd = wide ? 1 : digits.n, bits = wide ? 9 : digits.bits;   /* nine bits: in two rows of counts */
    const unsigned int digit_mask = (1u << bits) - 1u;
    const int rows = wide ? 2 : nd;
    for (int d = 0; d < 4; ++d) s.hist[d][tid] = 0u;
    if (int* ranges = cell_ranges(f, ctrl, vt)) {
        const long long nthreads = (long long)gridDim.x * blockDim.x;
        for (long long j = (long long)blockIdx.x * blockDim.x + tid; j < 2 * n_cells; j += nthreads) ranges[j] = -1;
    }
    for (long long j = (long long)blockIdx.x * blockDim.x + tid; j < 2 * vt->hdr.total_tiles;
         j += (long long)gridDim.x * blockDim.x)
        f.ranges[j] = 0;
    unsigned int kor = 0u, knot = 0u;
    unsigned long long tile_sum = 0ull;
    for (;;) {
        if (tid == 0) s.blk = atomicAdd(&ctrl->emit_ticket, 1u);
        __syncthreads();
        const int blk = (int)s.blk;
        const long long p0 = (long long)blk * (kRounds * kEmitThreads);
        if (p0 >= V) break;   /* past the visible splats: no look-back waits on it */
        /* every round's splat of the thread (the gathers in flight together) */
        unsigned int vis[kRounds], first_pair[kRounds];
        unsigned long long rects[kRounds];
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
            const long long p = p0 + q * kEmitThreads + tid;
            vis[q] = p < V ? order[p] : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int q = 0; q < kRounds; ++q) rects[q] = vis[q] != 0xFFFFFFFFu ? f.rects[vis[q]] : 0ull;
        /* in-round scans over the warp's pairs, its sums to shared memory */
#pragma unroll
        for (int q = 0; q < kRounds; ++q) {
            const CellRect c = cell_rect(rects[q]);
            const unsigned int tiles = vis[q] != 0xFFFFFFFFu ? c.tiles : 0u, pairs = vis[q] != 0xFFFFFFFFu ? c.pairs : 0u;
            unsigned int x = pairs;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            first_pair[q] = x - pairs;
            const unsigned int warp_tiles = __reduce_add_sync(0xffffffffu, tiles);
            if (lane == 31) {
                s.warp_pairs[q][warp] = x;
                s.warp_tiles[q][warp] = warp_tiles;
            }
        }
        __syncthreads();
        if (warp == 0) {
            /* the block's sums, round by round, saturated as in the descriptors */
            unsigned long long block = 0ull;
            for (int q = 0; q < kRounds; ++q) {
                const unsigned int p = __reduce_add_sync(0xffffffffu, lane < kEmitWarps ? s.warp_pairs[q][lane] : 0u);
                const unsigned int t = __reduce_add_sync(0xffffffffu, lane < kEmitWarps ? s.warp_tiles[q][lane] : 0u);
                block = add_counts(block, pack_counts(min(t, kSaturated), min(p, kSaturated)));
                tile_sum += t;
            }
            if (lane == 0) st_volatile_u64(lb + blk, (blk == 0 ? kDescIncl64 : kDescAgg64) | block);
            const unsigned long long e = blk > 0 ? lookback_counts(lb, blk, &ctrl->error_flags) : 0ull;
            if (lane == 0) {
                s.base = e;
                if (blk > 0) st_volatile_u64(lb + blk, kDescIncl64 | add_counts(e, block));
            }
        }
        __syncthreads();
        unsigned long long base = s.base;
        for (int q = 0; q < kRounds && p0 + q * kEmitThreads < V; ++q) {
            const unsigned int v = vis[q];
            const unsigned long long r = rects[q];
            CellRect c = cell_rect(r);
            unsigned int cell0 = 0u, cells_x = 0u;
            if (v != 0xFFFFFFFFu) {
                const ViewDesc& vd = vt->view[rect_view(r)];
                cells_x = (unsigned int)vd.cells_x;
                cell0 = (unsigned int)vd.cell_begin + c.cy * cells_x + c.cx;
            } else {
                c.pairs = 0u;
            }
            unsigned int excl = first_pair[q], block_pairs = 0u, block_tiles = 0u;
#pragma unroll
            for (int w = 0; w < kEmitWarps; ++w) {
                if (w == warp) excl += block_pairs;
                block_pairs += s.warp_pairs[q][w];
                block_tiles += s.warp_tiles[q][w];
            }
            const unsigned int tile_base = (unsigned int)(base >> 31) & 0x7FFFFFFFu;
            const unsigned int pair_base = (unsigned int)base & 0x7FFFFFFFu;
            /* the capacity is reached in this block or before it */
            const bool over = tile_base + min(block_tiles, kSaturated) > cap;
            unsigned int kept_pairs = block_pairs, cut = kEmitThreads;
            const bool lanes = !over && __reduce_max_sync(0xffffffffu, c.pairs) <= kEmitLaneCells;
            if (!lanes) {
                s.rect[tid] = r;
                s.run[tid] = make_uint4(excl, c.cw, cell0, cells_x);
                s.aux[tid] = make_uint2(__float_as_uint(1.0f / (float)c.cw), v);
                __syncwarp();
            }
            if (over) {
                __syncthreads();
                if (tid == 0) {
                    const long long left = V - p0 - q * kEmitThreads;
                    emit_cut(s, tile_base < cap ? cap - tile_base : 0u, (int)(left < kEmitThreads ? left : kEmitThreads));
                    if (s.cut_tiles) {   /* keys without masks: the lists form them again */
                        ctrl->cut_splat = s.aux[s.cut].y + 1u;
                        ctrl->cut_tiles = s.cut_tiles;
                    }
                }
                __syncthreads();
                kept_pairs = s.kept;
                cut = s.cut;
            }
            auto count = [&](unsigned int cell) {
                kor |= cell;
                knot |= ~cell;
                if (nd == 0) return;   /* one cell: nothing to sort */
                atomicAdd(&s.hist[0][0] + (cell & digit_mask), 1u);
                for (int d = 1; d < nd; ++d) atomicAdd(&s.hist[d][(cell >> (bits * d)) & digit_mask], 1u);
            };
            if (lanes) {
                /* A cell's mask is what the rectangle's four sides leave of
                 * it; a side matters in its own row or column of cells only. */
                const unsigned int left = 0x1111u * ((0xFu << (rect_min_tx(r) % kCellSide)) & 0xFu);
                const unsigned int right = 0x1111u * (0xFu >> (kCellSide - 1 - rect_max_tx(r) % kCellSide));
                const unsigned int top = (0xFFFFu << (4 * (rect_min_ty(r) % kCellSide))) & 0xFFFFu;
                const unsigned int bottom = 0xFFFFu >> (4 * (kCellSide - 1 - rect_max_ty(r) % kCellSide));
                const unsigned int last_row = (unsigned int)rect_max_ty(r) / kCellSide - c.cy;
                unsigned int cell = cell0, col = 0u, row = 0u;
                unsigned int* key = f.keys[0] + pair_base + excl;
                unsigned int* val = f.vals[0] + pair_base + excl;
                for (unsigned int k = 0; k < c.pairs; ++k) {
                    const unsigned int mask = (col == 0u ? left : 0xFFFFu) & (col + 1u == c.cw ? right : 0xFFFFu) &
                                              (row == 0u ? top : 0xFFFFu) & (row == last_row ? bottom : 0xFFFFu);
                    key[k] = packed ? mask * (unsigned int)kPackedCells + cell : cell;
                    val[k] = v;
                    count(cell);
                    ++cell;
                    if (++col == c.cw) {
                        col = 0u;
                        ++row;
                        cell += cells_x - c.cw;
                    }
                }
                __syncwarp();
            } else {
                /* The warp's pairs (those of its 32 splats, consecutive in the
                 * block's order), kEmitWindow at a time. Each splat marks the
                 * slot where its run of pairs enters the window (the splat
                 * already running at the window's start marks slot 0); a prefix
                 * maximum over the marks then gives every slot its splat without
                 * a search, and consecutive lanes write consecutive pairs. */
                const unsigned int my_end = excl + c.pairs;
                const unsigned int w_begin = __shfl_sync(0xffffffffu, excl, 0);
                const unsigned int w_end = min(__shfl_sync(0xffffffffu, my_end, 31), kept_pairs);
                for (unsigned int a = w_begin; a < w_end; a += kEmitWindow) {
                    const unsigned int nwin = emit_window_owners(s, warp, lane, a, excl, c.pairs, w_end);
                    for (unsigned int jj = lane; jj < nwin; jj += 32) {
                        const int lo = warp * 32 + (int)s.owner[warp][jj] - 1;
                        const uint4 rn = s.run[lo];
                        unsigned int column;
                        const unsigned int row = emit_row(s, lo, rn, a + jj, &column);
                        const unsigned long long rect = s.rect[lo];
                        const unsigned int cell = rn.z + row * rn.w + column;
                        const unsigned int pos = pair_base + a + jj;   /* below the capacity, like the instances */
                        if (pos >= cap) continue;
                        unsigned int key = cell;
                        if (packed) {
                            const int x = (int)(rect_min_tx(rect) / kCellSide + column) * kCellSide;
                            const int y = (int)(rect_min_ty(rect) / kCellSide + row) * kCellSide;
                            unsigned int mask = cell_mask(rect, x, y);
                            if (over && (unsigned int)lo == cut) mask = cut_mask(rect, x, y, mask, s.cut_tiles);
                            key |= mask << 16;
                        }
                        f.keys[0][pos] = key;
                        f.vals[0][pos] = s.aux[lo].y;
                        count(cell);
                    }
                    __syncwarp();
                }
            }
            /* look-back descriptors of the sort tiles whose first key is one of
             * this block's pairs (every tile of the sort has one) */
            {
                const unsigned int i0 = min(pair_base, cap), i1 = min(pair_base + kept_pairs, cap);
                const unsigned int tk = (unsigned int)sort_tile_keys;
                const unsigned int t0 = (i0 + tk - 1u) / tk;
                unsigned int t1 = (i1 + tk - 1u) / tk;
                if ((long long)t1 > sort_lb_tiles) t1 = (unsigned int)sort_lb_tiles;
                const int row = wide ? kWideCells : 256;
                for (int d = 0; d < nd; ++d) {
                    unsigned int* region = sort_lb + (size_t)d * (size_t)lookback_rows(sort_lb_tiles) * 256;
                    for (unsigned int t = t0; t < t1; ++t)
                        for (int j = tid; j < row; j += kEmitThreads) {
                            region[(size_t)t * row + j] = 0u;
                            if (t % kLookbackGroup == 0)   /* its group's row */
                                region[((size_t)sort_lb_tiles + t / kLookbackGroup) * row + j] = 0u;
                        }
                }
            }
            if (tid == 0) {
                const bool last = p0 + (q + 1) * kEmitThreads >= V;
                if (over ? tile_base <= cap : last) ctrl->cell_sort.n = (unsigned long long)(pair_base + kept_pairs);
                if (over && last) atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_CAPACITY);
            }
            base = add_counts(base, pack_counts(min(block_tiles, kSaturated), min(block_pairs, kSaturated)));
            if (over) __syncthreads();
            __syncwarp();
        }
        __syncthreads();
    }
    for (int d = 0; d < rows; ++d) {
        const unsigned int n = s.hist[d][tid];
        if (n) atomicAdd(&ctrl->cell_sort.hist[d][tid], n);
    }
    kor = __reduce_or_sync(0xffffffffu, kor);
    knot = __reduce_or_sync(0xffffffffu, knot);
    if (lane == 0 && (kor | knot)) {
        atomicOr(&ctrl->cell_sort.key_or, (unsigned long long)kor);
        atomicOr(&ctrl->cell_sort.key_or_not, (unsigned long long)knot);
    }
    if (tid == 0 && tile_sum) atomicAdd(&ctrl->n_instances, tile_sum);
}

/* ---------------------------------------------------------------------
 * Gaussian-major batch projection. Views of one scene in a batch share
 * every input of the projection but the camera, so a unit of work is one
 * 128-Gaussian block of a distinct scene, projected into every view of
 * that scene: its 236 bytes per Gaussian are read once per batch instead of
 * once per view. The visible indices stay the per-view-major order of
 * project_kernel (view v's block b at the position the blocks before it in
 * (view, block) order leave), so every output is the one-view-at-a-time
 * pipeline's. Three launches:
 *   batch_count_kernel:   per unit and view, the block's visible count
 *                         (geometry only: 44 bytes per Gaussian);
 *   batch_offsets_kernel: exclusive scan of the counts in (view, block)
 *                         order (decoupled look-back over 2048-count tiles),
 *                         written over the counts;
 *   batch_project_kernel: per unit, the SH rows staged once, then for every
 *                         view the full projection, the record, index,
 *                         rectangle and depth key at the view's offset.
 * --------------------------------------------------------------------- */

constexpr int kOffsetsThreads = 1024;
constexpr int kOffsetsItems = 8;    /* 8192 counts per tile: one tile for a 1M-Gaussian view */
constexpr int kOffsetsTile = kOffsetsThreads * kOffsetsItems;
/* resident projection CTAs per SM: 64 registers, 8 x 24.6 KB of staged SH rows */
constexpr int kBatchProjectCtas = 8;

struct BatchProjSmem {
    DevCamera cam;
    unsigned long long unit;
    unsigned int warp_tot[kProjThreads / 32];
    unsigned long long key_or, key_or_not;
};

/* The counts (u32 per (view, block)) and, after them, the scan's
 * descriptors, in the project look-back region of the scratch. */
__device__ __forceinline__ unsigned long long* offsets_desc(unsigned long long* lb, long long total_blocks) {
    return lb + (total_blocks + 1) / 2;
}

/* The unit's Gaussian parameters (zeros past the scene's end). */
struct UnitParams {
    float mx, my, mz;
    Prepared pr;
};

__device__ __forceinline__ UnitParams load_unit_params(const LumenGpuGaussians& g, long long i,
                                                       const LumenRenderOptions& opt) {
    UnitParams u;
    u.mx = u.my = u.mz = 0.0f;
    u.pr.ok = false;
    u.pr.op = 0.0f;
    u.pr.s00 = u.pr.s01 = u.pr.s02 = u.pr.s11 = u.pr.s12 = u.pr.s22 = 0.0f;
    if (i < g.count) {
        const float* m = g.means + i * 3;
        const float* sc = g.scales + i * 3;
        const float4 q = __ldg(reinterpret_cast<const float4*>(g.quats) + i);
        u.mx = __ldg(m); u.my = __ldg(m + 1); u.mz = __ldg(m + 2);
        u.pr = prepare_gaussian(__ldg(sc), __ldg(sc + 1), __ldg(sc + 2), Quat{q.x, q.y, q.z, q.w},
                                __ldg(g.opacities + i), opt);
    }
    return u;
}

template <bool kPersistent>
__global__ void __launch_bounds__(kProjThreads)
batch_count_kernel(const ViewTable* __restrict__ vt, LumenRenderOptions opt, Control* ctrl,
                   unsigned long long* lb) {
    chain_begin();
    __shared__ BatchProjSmem s;
    const int tid = threadIdx.x;
    const int n_views = vt->hdr.n_views;
    const long long total_units = vt->hdr.total_units;
    unsigned int* counts = reinterpret_cast<unsigned int*>(lb);
    for (;;) {
        if (kPersistent) {
            if (tid == 0) s.unit = atomicAdd(&ctrl->count_ticket, 1u);
            __syncthreads();
        } else if (tid == 0) {
            s.unit = blockIdx.x;
        }
        __syncthreads();
        const long long u = (long long)s.unit;
        if (u >= total_units) break;
        const int lead = find_view_by_unit(vt, n_views, u);
        const long long b = u - vt->view[lead].unit_begin;
        const UnitParams up = load_unit_params(vt->view[lead].g, b * kProjThreads + tid, opt);
        for (int v = lead; v >= 0; v = vt->view[v].group_next) {
            copy_camera(s.cam, vt->view[v].dcam);
            __syncthreads();
            const bool vis = project_prepared<false>(s.cam, up.mx, up.my, up.mz, up.pr, nullptr, opt).visible;
            const int c = __syncthreads_count(vis);
            if (tid == 0) counts[vt->view[v].block_begin + b] = (unsigned int)c;
        }
        if (!kPersistent) break;
        __syncthreads();
    }
}

/* Exclusive scan of the (view, block) visible counts in place; the total
 * is the batch's visible count. */
__global__ void __launch_bounds__(kOffsetsThreads)
batch_offsets_kernel(const ViewTable* __restrict__ vt, Control* ctrl, unsigned long long* lb) {
    chain_begin();
    __shared__ unsigned int warp_tot[kOffsetsThreads / 32];
    __shared__ unsigned int tile_s;
    __shared__ unsigned long long base_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const long long nb = vt->hdr.total_blocks;
    const long long ntiles = (nb + kOffsetsTile - 1) / kOffsetsTile;
    unsigned int* counts = reinterpret_cast<unsigned int*>(lb);
    unsigned long long* desc = offsets_desc(lb, nb);
    for (;;) {
        if (tid == 0) tile_s = atomicAdd(&ctrl->offsets_ticket, 1u);
        __syncthreads();
        const long long t = tile_s;
        if (t >= ntiles) break;
        const long long i0 = t * kOffsetsTile + (long long)tid * kOffsetsItems;
        unsigned int c[kOffsetsItems];
        unsigned int sum = 0;
#pragma unroll
        for (int k = 0; k < kOffsetsItems; ++k) {
            c[k] = i0 + k < nb ? counts[i0 + k] : 0u;
            sum += c[k];
        }
        unsigned int tot = 0;
        const unsigned int ex = block_exclusive_scan<kOffsetsThreads>(sum, warp_tot, &tot);
        if (tid == 0) st_volatile_u64(desc + t, (t == 0 ? kDescIncl64 : kDescAgg64) | tot);
        if (warp == 0) {
            const unsigned long long e = t > 0 ? lookback64(desc, (int)t, &ctrl->error_flags) : 0ull;
            if (lane == 0) {
                base_s = e;
                if (t > 0) st_volatile_u64(desc + t, kDescIncl64 | (e + tot));
            }
        }
        __syncthreads();
        unsigned long long run = base_s + ex;
#pragma unroll
        for (int k = 0; k < kOffsetsItems; ++k) {
            if (i0 + k < nb) counts[i0 + k] = (unsigned int)run;
            run += c[k];
        }
        if (tid == 0 && t == ntiles - 1) {
            ctrl->n_visible = (unsigned int)(base_s + tot);
            ctrl->depth_sort.n = base_s + tot;
        }
        __syncthreads();
    }
}

template <bool kPersistent>
__global__ void __launch_bounds__(kProjThreads, kBatchProjectCtas)
batch_project_kernel(const ViewTable* __restrict__ vt, LumenRenderOptions opt, LumenGpuFrame f, Control* ctrl,
                     const unsigned long long* lb) {
    chain_begin();
    __shared__ BatchProjSmem s;
    extern __shared__ float4 sh_stage[];   /* kProjThreads x 12: the unit's SH coefficients */
    const int tid = threadIdx.x, lane = tid & 31;
    const int n_views = vt->hdr.n_views;
    const long long total_units = vt->hdr.total_units;
    const unsigned int* offsets = reinterpret_cast<const unsigned int*>(lb);
    for (;;) {
        if (tid == 0) {
            s.unit = kPersistent ? (unsigned long long)atomicAdd(&ctrl->proj_ticket, 1u) : blockIdx.x;
            s.key_or = 0ull;
            s.key_or_not = 0ull;
        }
        __syncthreads();
        const long long u = (long long)s.unit;
        if (u >= total_units) break;
        const int lead = find_view_by_unit(vt, n_views, u);
        const LumenGpuGaussians& g = vt->view[lead].g;
        const long long b = u - vt->view[lead].unit_begin;
        const long long i0 = b * kProjThreads, i = i0 + tid;
        {
            const long long count = g.count;
            const int nblk = (int)(count - i0 < kProjThreads ? count - i0 : kProjThreads);
            const float4* src = reinterpret_cast<const float4*>(g.sh + i0 * 48);
            for (int c = tid; c < nblk * 12; c += kProjThreads) {
                const int t = c / 12, q = c - 12 * t;
                cp_async16(sh_stage + 12 * t + (q ^ sh_swizzle(t)), src + c);
            }
            cp_async_commit();
        }
        const UnitParams up = load_unit_params(g, i, opt);
        const bool in_scene = i < g.count;
        cp_async_wait_all();
        unsigned long long kor = 0ull, knot = 0ull;
        for (int v = lead; v >= 0; v = vt->view[v].group_next) {
            copy_camera(s.cam, vt->view[v].dcam);
            __syncthreads();
            const Projected p = project_prepared<true>(s.cam, up.mx, up.my, up.mz, up.pr,
                                                       reinterpret_cast<const float*>(sh_stage + tid * 12), opt,
                                                       sh_swizzle(tid));
            const long long blk = vt->view[v].block_begin + b;
            if (f.radii && in_scene) f.radii[blk * kProjThreads + tid] = p.visible ? p.radius : 0;
            unsigned int n_vis = 0;
            const unsigned int vis_local = block_exclusive_scan<kProjThreads>(p.visible ? 1u : 0u, s.warp_tot, &n_vis);
            if (p.visible) {
                const unsigned long long vid = (unsigned long long)offsets[blk] + vis_local;
                float4* dst = reinterpret_cast<float4*>(f.records + vid);
                dst[0] = make_float4(p.cx, p.cy, p.z, p.op);
                dst[1] = make_float4(p.ic00, p.ic01, p.ic11, 0.0f);
                dst[2] = make_float4(p.r, p.g, p.b, 0.0f);
                f.visible_ids[vid] = (unsigned int)i;
                f.rects[vid] = pack_rect(p.min_tx, p.min_ty, p.max_tx, p.max_ty, v);
                const unsigned int dk = depth_key(p.z, opt.key_mode);
                f.depth_keys[0][vid] = dk;
                f.depth_order[0][vid] = (unsigned int)vid;
                kor |= dk;
                knot |= ~(unsigned long long)dk & 0xFFFFFFFFull;
            }
            __syncthreads();   /* s.cam and s.warp_tot are rewritten for the next view */
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            kor |= __shfl_xor_sync(0xffffffffu, kor, o);
            knot |= __shfl_xor_sync(0xffffffffu, knot, o);
        }
        if (lane == 0 && (kor | knot)) {
            atomicOr(&s.key_or, kor);
            atomicOr(&s.key_or_not, knot);
        }
        __syncthreads();
        if (tid == 0 && (s.key_or | s.key_or_not)) {
            atomicOr(&ctrl->depth_sort.key_or, s.key_or);
            atomicOr(&ctrl->depth_sort.key_or_not, s.key_or_not);
        }
        if (!kPersistent) break;
        __syncthreads();
    }
}

static int resident_ctas(const void* kernel, int threads, size_t smem) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm <= 0)
        per_sm = 1;
    return per_sm;
}

static int g_emit_per_sm[2] = {0, 0}, g_batch_count_per_sm = 0, g_batch_project_per_sm = 0;   /* emit: one and four rounds */
constexpr size_t kProjStageBytes = (size_t)kProjThreads * 48 * sizeof(float);

/* Kernel attributes and the occupancy of the persistent kernels, set and
 * queried once (before any capture). */
void prime_persistent_launches() {
    cudaFuncSetAttribute(project_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kProjStageBytes);
    g_emit_per_sm[0] = resident_ctas((const void*)emit_kernel<1>, kEmitThreads, 0);
    g_emit_per_sm[1] = resident_ctas((const void*)emit_kernel<kEmitMaxRounds>, kEmitThreads, 0);
    cudaFuncSetAttribute(batch_project_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kProjStageBytes);
    cudaFuncSetAttribute(batch_project_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)kProjStageBytes);
    g_batch_count_per_sm = resident_ctas((const void*)batch_count_kernel<true>, kProjThreads, 0);
    g_batch_project_per_sm = resident_ctas((const void*)batch_project_kernel<true>, kProjThreads, kProjStageBytes);
}

/* Gaussian-major projection of a batch: n_units is the batch's unit count
 * (plain launches: one CTA per unit) or 0 for persistent launches, which
 * read the count from the table. */
void launch_batch_project(const ViewTable* vt, const LumenRenderOptions& opt, const LumenGpuFrame& f,
                          Control* ctrl, unsigned long long* lb, long long n_units, long long n_blocks,
                          bool persistent, int num_sms, cudaStream_t st) {
    if (persistent) {
        const int pc = g_batch_count_per_sm > 0 ? g_batch_count_per_sm : 1;
        launch_chained(batch_count_kernel<true>, dim3(pc * num_sms), dim3(kProjThreads), 0, st, vt, opt, ctrl, lb);
        launch_chained(batch_offsets_kernel, dim3(2 * num_sms), dim3(kOffsetsThreads), 0, st, vt, ctrl, lb);
        const int pp = g_batch_project_per_sm > 0 ? g_batch_project_per_sm : 1;
        launch_chained(batch_project_kernel<true>, dim3(pp * num_sms), dim3(kProjThreads), kProjStageBytes, st, vt,
                       opt, f, ctrl, (const unsigned long long*)lb);
        return;
    }
    if (n_units <= 0) return;
    const long long tiles = (n_blocks + kOffsetsTile - 1) / kOffsetsTile;
    launch_chained(batch_count_kernel<false>, dim3((unsigned int)n_units), dim3(kProjThreads), 0, st, vt, opt, ctrl,
                   lb);
    launch_chained(batch_offsets_kernel, dim3((unsigned int)(tiles > 0 ? tiles : 1)), dim3(kOffsetsThreads), 0, st,
                   vt, ctrl, lb);
    launch_chained(batch_project_kernel<false>, dim3((unsigned int)n_units), dim3(kProjThreads), kProjStageBytes, st,
                   vt, opt, f, ctrl, (const unsigned long long*)lb);
}

/* One view of n_blocks blocks. */
void launch_project(const ViewTable* vt, const LumenRenderOptions& opt, const LumenGpuFrame& f, Control* ctrl,
                    unsigned long long* lb, long long n_blocks, cudaStream_t st) {
    if (n_blocks <= 0) return;
    launch_chained(project_kernel, dim3((unsigned int)n_blocks), dim3(kProjThreads), kProjStageBytes, st, vt, opt, f,
                   ctrl, lb);
}

/* sort_lb: the cell sort's look-back region (sort_lb_tiles descriptor
 * tiles per digit) for digit passes of sort_tile_keys keys per tile. */
void launch_emit(const ViewTable* vt, const LumenGpuFrame& f, Control* ctrl, unsigned long long* lb,
                 unsigned int* sort_lb, long long sort_lb_tiles, int sort_tile_keys, bool wide, long long n_blocks,
                 bool persistent, int num_sms, cudaStream_t st) {
    if (n_blocks <= 0) return;
    auto run = [&](auto kernel, int rounds) {
        const int per_sm = g_emit_per_sm[rounds > 1];
        const long long resident = (long long)(per_sm > 0 ? per_sm : 1) * num_sms;
        const long long blocks = (n_blocks * kProjThreads + rounds * kEmitThreads - 1) / (rounds * kEmitThreads);
        launch_chained(kernel, dim3((unsigned int)(persistent || blocks > resident ? resident : blocks)),
                       dim3(kEmitThreads), 0, st, vt, f, ctrl, lb, sort_lb, sort_lb_tiles, sort_tile_keys, wide);
    };
    if (n_blocks * kProjThreads >= 3ll * num_sms * kEmitMaxRounds * kEmitThreads)
        run(emit_kernel<kEmitMaxRounds>, kEmitMaxRounds);
    else
        run(emit_kernel<1>, 1);
}

}  // namespace lumen
