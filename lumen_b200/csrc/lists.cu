/*
 * lists.cu - the tiles' splat lists from the sorted (cell, splat) pairs.
 *
 * Reference: the key sort of rasterize_scene (src/raster/pipeline.mojo:152-166
 * with radix_sort_64bit, src/raster/radix_sort.mojo:39-87) and
 * TileRangeIndex.build_from_sorted_keys, src/raster/binning.mojo:51-73: the
 * instances ordered by (tile, depth key, visible index), and each tile's
 * first and last position, (-1, -1) where it has none.
 *
 * The emission writes one pair per cell (4x4 tiles) that a splat touches, in
 * depth order, and the cell sort keeps that order within a cell. Here each
 * cell's list is split over its 16 tiles by the pairs' tile masks, in order:
 *
 *   list_count_kernel   per segment of 256 pairs of a cell (or of a part of a
 *                       long cell): the instances of each of its tiles before it
 *   list_scan_kernel    an exclusive scan of the tiles' counts: the ranges, the
 *                       touched tiles, each view's first instance
 *   list_write_kernel   per segment: a vote per tile and 32 pairs gives every
 *                       instance its position
 *
 * Why two levels: sorting the instances themselves by tile ranks every one of
 * them twice (two digit passes, about 120 instructions per instance and pass)
 * and moves 8 B per instance five times. A splat covers about 7 tiles but 2
 * cells, so the ranked pairs are 3 to 4 times fewer, and the split needs no
 * ranking. The instances are written once. From the depth order to the ranges,
 * emission included, this took (us, before -> after): 1 M splats at 1080p
 * 160 -> 115, 2 M at 4K 455 -> 235, 64 views of 300 k at 720p 2400 -> 1320,
 * 512 splats at 800x600 34 -> 32.
 */
#include "splat_common.cuh"

namespace lumen {

namespace {

constexpr int kCountThreads = 256;
constexpr int kCountWarps = kCountThreads / 32;
/* At most so many CTAs per SM, whatever the cells: a persistent launch, sized for
 * the most cells that its buffers hold, spent 8 us on starting 64 per SM. */
constexpr int kCountCtas = 16;
constexpr int kScanThreads = 1024;
constexpr int kWriteThreads = 128;
constexpr int kWriteWarps = kWriteThreads / 32;
constexpr int kWriteCtas = 6;                   /* per SM */
constexpr int kSegment = 256;                   /* pairs of a cell that a warp counts and writes at a time */
constexpr int kLongCell = 24576;                /* cells of more pairs are counted in parts, */
constexpr int kWindow = 16384;                  /* cut at multiples of so many sorted pairs */
constexpr int kCellTiles = kCellSide * kCellSide;

/* A cell in its view. */
struct Cell {
    int x, y;                /* its first tile */
    int tiles_x, tiles_y;
    long long tile_begin;
    /* batch-wide id of its tile k (bit k of the masks), or -1 beyond the view */
    __device__ __forceinline__ long long tile(int k) const {
        const int tx = x + k % kCellSide, ty = y + k / kCellSide;
        return tx < tiles_x && ty < tiles_y ? tile_begin + (long long)ty * tiles_x + tx : -1;
    }
};

__device__ __forceinline__ Cell find_cell(const ViewTable* vt, int n_views, long long cell) {
    const ViewDesc& vd = vt->view[n_views == 1 ? 0 : find_view_by_cell(vt, n_views, cell)];
    const int local = (int)(cell - vd.cell_begin);
    Cell c;
    c.y = local / vd.cells_x * kCellSide;
    c.x = local % vd.cells_x * kCellSide;
    c.tiles_x = vd.tiles_x;
    c.tiles_y = (vd.cam.height + kTile - 1) / kTile;
    c.tile_begin = vd.tile_begin;
    return c;
}

/* The first of n sorted keys whose cell is `cell` or above, by a whole warp
 * (32 probes per step). */
__device__ __forceinline__ int first_of_cell(const unsigned int* __restrict__ keys, int n, unsigned int id_mask,
                                             unsigned int cell) {
    const int lane = threadIdx.x & 31;
    int lo = 0, len = n;   /* the answer is in [lo, lo + len] */
    while (len > 0) {
        const int step = (len + 31) / 32;
        const int at = lo + lane * step;
        const bool below = lane * step < len && (keys[at] & id_mask) < cell;
        const int k = __popc(__ballot_sync(0xffffffffu, below));   /* the first k probes are below */
        if (k == 0) return lo;
        const int end = lo + len;
        lo += (k - 1) * step + 1;
        len = min(step - 1, end - lo);
    }
    return lo;
}


/* Tiles per scan group: at most kTileGroups groups. */
__device__ __forceinline__ long long tile_group_size(long long n_tiles) {
    long long g = kScanThreads;
    while (g * kTileGroups < n_tiles) g *= 2;
    return g;
}

struct SortedPairs {
    const unsigned int* keys;
    const unsigned int* vals;
    int n;
    bool packed;
    unsigned int cut_splat, cut_tiles;   /* of the control block */
};

/* The tile mask of a sorted pair of the cell whose first tile is (x, y). */
__device__ __forceinline__ unsigned int pair_mask(const SortedPairs& in, unsigned int key, unsigned int v,
                                                  const uint64_t* __restrict__ rects, int x, int y) {
    if (in.packed) return key >> 16;
    const unsigned long long rect = rects[v];
    const unsigned int mask = cell_mask(rect, x, y);
    return v + 1u == in.cut_splat ? cut_mask(rect, x, y, mask, in.cut_tiles) : mask;
}

/* kPacked: the cells are known to be few enough for packed keys (in one form
 * for both kinds of key, the code that forms masks cost 64 views of 300 k 23 us). */
template <bool kPacked>
__device__ __forceinline__ SortedPairs sorted_pairs(const LumenGpuFrame& f, const Control* ctrl,
                                                    const ViewTable* vt) {
    const unsigned int b = ctrl->cell_sort.sorted_buffer;
    const long long n = (long long)ctrl->cell_sort.n;
    return {b ? f.keys[1] : f.keys[0], b ? f.vals[1] : f.vals[0],
            (int)(n < f.instance_capacity ? n : f.instance_capacity), kPacked || vt->hdr.total_cells <= kPackedCells,
            ctrl->cut_splat, ctrl->cut_tiles};
}

/* A segment: up to 256 consecutive pairs of one part of a cell, as the count
 * kernel leaves it for the write kernel. They lie in the cell sort's look-back
 * rows, which nothing reads once it is done (2 B per instance that the frame can
 * hold, against 80 B per 256 pairs and per part, and 64 B per part). Without
 * enough room, a warp writes a whole cell. */
struct Segment {
    int first;
    unsigned int n_part;        /* its pairs (10 bits), and its part's number in the cell */
    unsigned int tile0;         /* the cell's first tile, and the view's tiles per row */
    int tiles_x;
    unsigned int before[kCellTiles];   /* per tile, its instances in the part's pairs before */
};
static_assert(sizeof(Segment) == 80, "16-byte aligned");

/* Scratch after the cell sort: the tiles' order (u32 per tile), if there is to
 * be one, then the parts' totals, then the segments. offset: of p in the
 * frame's scratch. */
struct Room {
    unsigned char* p;
    long long bytes, offset;
    long long order_min, order_max;   /* frames of so many tiles get an order */
};

__device__ __forceinline__ bool has_order(const Room& room, const ViewTable* vt) {
    const long long n = vt->hdr.total_tiles;
    return n >= room.order_min && n <= room.order_max && n * 4 <= room.bytes;
}

/* The work items of the count: a cell, or (from n_cells on) a window of
 * sorted pairs that lies in a long cell which starts before it. Part 0 of a
 * cell is the cell's item; part k the window k after the one that the cell starts
 * in. total: per item and tile, the part's instances. Without more pairs than a
 * long cell has, there are no windows and no totals. */
struct SegmentRoom {
    unsigned int (*total)[kCellTiles];
    Segment* p;
    long long n;
};

__device__ __forceinline__ long long count_items(const ViewTable* vt, int n_pairs) {
    return vt->hdr.total_cells + (n_pairs > kLongCell ? (n_pairs + kWindow - 1) / kWindow : 0);
}

__device__ __forceinline__ SegmentRoom segment_room(const Room& room, const ViewTable* vt, int n_pairs) {
    const long long order = has_order(room, vt) ? (vt->hdr.total_tiles * 4 + 15) / 16 * 16 : 0;
    const long long totals =
        n_pairs > kLongCell ? count_items(vt, n_pairs) * (long long)sizeof(unsigned int[kCellTiles]) : 0;
    return {reinterpret_cast<unsigned int(*)[kCellTiles]>(room.p + order),
            reinterpret_cast<Segment*>(room.p + order + totals),
            max(room.bytes - order - totals, 0ll) / (long long)sizeof(Segment)};
}

/* Class of a tile's list length n: higher for longer lists. */
__device__ __forceinline__ int length_class(unsigned int n) {
    const int log2 = 31 - __clz((int)(n | 1u));
    return n < 2u ? (int)n : 2 * log2 + (int)((n >> (log2 - 1)) & 1u);
}

__device__ __forceinline__ bool has_room(const SegmentRoom& room, const ViewTable* vt, int n_pairs) {
    return n_pairs / kSegment + count_items(vt, n_pairs) <= room.n;
}

/* The cell's range among the sorted pairs to bounds[0], bounds[1]: as the
 * cell sort's last pass left it, or searched by two warps when there was none
 * (every pair in one cell) or no room for the ranges. A barrier must follow. */
__device__ __forceinline__ void find_bounds(int* bounds, const SortedPairs& in, const int* ranges, long long cell) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (ranges) {
        if (tid < 2) bounds[tid] = ranges[2 * cell + tid];
    } else if (warp < 2) {
        const unsigned int id_mask = in.packed ? (unsigned int)(kPackedCells - 1) : 0xFFFFFFFFu;
        const int at = first_of_cell(in.keys, in.n, id_mask, (unsigned int)cell + (unsigned int)warp);
        if (lane == 0) bounds[warp] = at;
    }
}

/* One CTA per item, eight segments at a time (a warp each, all its keys'
 * reads in flight, the next eight's before these are counted). Bound by the
 * latency of those reads (4 B per pair, once), about 0.6 us per step of 2048
 * pairs, so long cells are counted in parts by as many CTAs: a cell of 2 M pairs
 * by one CTA took 590 us (2 M splats in a 64x64 image: the frame 1.81 ms, in
 * parts 1.26, and 1.22 with the instances sorted by tile; 1 M in 128x72 0.70,
 * 0.52 and 0.54). With cells of 8192 pairs already in parts, 2 M splats at 4K
 * counted 31 us instead of 23. A part's counts start at 0 (the write
 * kernel adds the totals of the parts before); the tiles' totals are added up by
 * atomics, and the last part to arrive knows them. */
template <bool kPacked>
__global__ void __launch_bounds__(kCountThreads)
list_count_kernel(const ViewTable* __restrict__ vt, LumenGpuFrame f, Control* ctrl, Room scratch) {
    chain_begin();
    const bool order = has_order(scratch, vt);
    constexpr int kReads = kSegment / 32;
    __shared__ int bounds[2];
    __shared__ unsigned int slot_s;
    __shared__ unsigned int count[2][kCountWarps][kCellTiles];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SortedPairs in = sorted_pairs<kPacked>(f, ctrl, vt);
    const SegmentRoom room = segment_room(scratch, vt, in.n);
    const bool noted = has_room(room, vt, in.n);
    const int* cells = ctrl->cells_by_sort ? cell_ranges(f, ctrl, vt) : nullptr;
    const long long n_cells = vt->hdr.total_cells, group = tile_group_size(vt->hdr.total_tiles);
    const long long n_items = count_items(vt, in.n);
    const unsigned int id_mask = in.packed ? (unsigned int)(kPackedCells - 1) : 0xFFFFFFFFu;
    const int n_views = vt->hdr.n_views;
    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int window = item < n_cells ? -1 : (int)(item - n_cells);
        const long long cell = window < 0 ? item : (long long)(in.keys[(long long)window * kWindow] & id_mask);
        if (cell >= n_cells) {   /* self-check: a key that names no cell */
            if (tid == 0) atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
            continue;
        }
        find_bounds(bounds, in, cells, cell);
        const Cell c = find_cell(vt, n_views, cell);
        __syncthreads();
        const int cell_first = bounds[0], cell_end = bounds[1];
        const bool in_parts = cell_end - cell_first > kLongCell;
        /* the item's pairs */
        int first = cell_first, end = cell_end;
        unsigned int part = 0u;
        if (window >= 0) {
            first = window * kWindow;
            part = (unsigned int)(window - cell_first / kWindow);
            if (!in_parts || cell_first >= first) first = end;   /* the cell's own item has them */
        }
        if (in_parts) end = (int)min((long long)end, ((long long)first / kWindow + 1) * kWindow);
        if (window >= 0 && first >= end) {
            __syncthreads();
            continue;
        }
        const int n_seg = first < end ? (end - first + kSegment - 1) / kSegment : 0;
        if (tid == 0 && n_seg) slot_s = noted ? atomicAdd(&ctrl->n_segments, (unsigned int)n_seg) : 0u;
        unsigned int m[kReads], base = 0u;   /* base: lane k < 16, tile k's instances so far */
        auto read = [&](int seg) {
#pragma unroll
            for (int u = 0; u < kReads; ++u) {
                const int i = first + seg * kSegment + 32 * u + lane;
                m[u] = i < end ? pair_mask(in, in.keys[i], in.packed ? 0u : in.vals[i], f.rects, c.x, c.y) : 0u;
            }
        };
        read(warp);
        for (int s0 = 0, buf = 0; s0 < n_seg; s0 += kCountWarps, buf ^= 1) {
            const int seg = s0 + warp;
            /* per lane: 16 counts in the bytes of four words (at most 8 each) */
            unsigned int sum[4] = {0u, 0u, 0u, 0u};
#pragma unroll
            for (int u = 0; u < kReads; ++u)
#pragma unroll
                for (int q = 0; q < 4; ++q) sum[q] += (((m[u] >> (4 * q)) & 0xFu) * 0x00204081u) & 0x01010101u;
            read(seg + kCountWarps);
            unsigned int mine = 0u;   /* lane 4 q + column: the tile's count */
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                /* columns 0 and 2, 1 and 3 as 16-bit fields */
                const unsigned int even = __reduce_add_sync(0xffffffffu, sum[q] & 0x00FF00FFu);
                const unsigned int odd = __reduce_add_sync(0xffffffffu, (sum[q] >> 8) & 0x00FF00FFu);
                if ((lane >> 2) == q) mine = ((lane & 1 ? odd : even) >> (lane & 2 ? 16 : 0)) & 0xFFFFu;
            }
            if (lane < kCellTiles) count[buf][warp][lane] = mine;
            __syncthreads();
            if (lane < kCellTiles) {
                unsigned int before = base;
#pragma unroll
                for (int w = 0; w < kCountWarps; ++w) {
                    const unsigned int n = count[buf][w][lane];
                    if (w < warp) before += n;
                    base += n;
                }
                if (noted && seg < n_seg) room.p[slot_s + seg].before[lane] = before;
            } else if (lane == kCellTiles && noted && seg < n_seg) {
                const int i0 = first + seg * kSegment;
                const unsigned int n = end - i0 < kSegment ? (unsigned int)(end - i0) : (unsigned int)kSegment;
                *reinterpret_cast<int4*>(room.p + slot_s + seg) =
                    make_int4(i0, (int)(n | part << 10), (int)(c.tile_begin + (long long)c.y * c.tiles_x + c.x), c.tiles_x);
            }
        }
        if (warp == 0) {
            const long long t = lane < kCellTiles ? c.tile(lane) : -1;
            if (t >= 0 && base) atomicAdd(&ctrl->group_total[t / group], base);
            unsigned int total = base;
            bool known = true;
            if (!in_parts) {
                if (t >= 0) f.ranges[2 * t + 1] = (int)base;
            } else {
                if (noted && lane < kCellTiles) room.total[item][lane] = base;
                /* the emission has zeroed the ranges; the first tile's other
                 * word counts the parts that have arrived */
                if (t >= 0) atomicAdd(f.ranges + 2 * t + 1, (int)base);
                __threadfence();
                __syncwarp();
                int arrived = lane == 0 ? atomicAdd(f.ranges + 2 * t, 1) : 0;
                arrived = __shfl_sync(0xffffffffu, arrived, 0);
                known = arrived == (cell_end - 1) / kWindow - cell_first / kWindow;
                __threadfence();
                if (known && t >= 0) total = (unsigned int)__ldcg(f.ranges + 2 * t + 1);
            }
            if (order && known) {
                const unsigned int tiles = __ballot_sync(0xffffffffu, t >= 0);
                const int cls = length_class(total);
                if (t >= 0) {
                    const unsigned int same = __match_any_sync(tiles, cls);
                    if (lane == __ffs(same) - 1) atomicAdd(&ctrl->class_total[cls], (unsigned int)__popc(same));
                }
            }
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kScanThreads)
list_scan_kernel(ViewTable* vt, int* __restrict__ ranges, Control* ctrl, Room room) {
    chain_begin();
    __shared__ unsigned int class_start[kTileClasses], class_n[kTileClasses], class_base[kTileClasses];
    __shared__ unsigned int warp_tot[kScanThreads / 32];
    __shared__ unsigned int base_s;
    const int tid = threadIdx.x, lane = tid & 31;
    const long long n_tiles = vt->hdr.total_tiles, group = tile_group_size(n_tiles);
    const int n_views = vt->hdr.n_views;
    if (blockIdx.x == 0 && tid == 0) {
        ctrl->list_buffer = ctrl->cell_sort.sorted_buffer ^ 1u;
        ctrl->depth_varying = ctrl->depth_sort.varying;
        ctrl->depth_buffer = ctrl->depth_sort.sorted_buffer;
        if (has_order(room, vt)) ctrl->order_offset = (unsigned int)(room.offset / 256);
    }
    /* longest lists first: a class starts after the tiles of all higher ones */
    unsigned int* order = has_order(room, vt) ? reinterpret_cast<unsigned int*>(room.p) : nullptr;
    if (order) {
        const int cls = kTileClasses - 1 - tid;
        unsigned int all;
        const unsigned int before = block_exclusive_scan<kScanThreads>(cls >= 0 ? ctrl->class_total[cls] : 0u, warp_tot, &all);
        if (cls >= 0) class_start[cls] = before;
        __syncthreads();
    }
    unsigned int touched = 0, id_or = 0, id_or_not = 0;
    for (long long g = blockIdx.x; g * group < n_tiles; g += gridDim.x) {
        unsigned int total = 0;
        const unsigned int before = tid < g ? ctrl->group_total[tid] : 0u;   /* kTileGroups == kScanThreads */
        block_exclusive_scan<kScanThreads>(before, warp_tot, &total);
        if (tid == 0) base_s = total;
        __syncthreads();
        for (long long t0 = g * group; t0 < (g + 1) * group && t0 < n_tiles; t0 += kScanThreads) {
            const long long t = t0 + tid;
            const bool valid = t < n_tiles;
            const unsigned int n = valid ? (unsigned int)ranges[2 * t + 1] : 0u;
            const unsigned int start = base_s + block_exclusive_scan<kScanThreads>(n, warp_tot, &total);
            if (valid) {
                ranges[2 * t] = n ? (int)start : -1;
                ranges[2 * t + 1] = n ? (int)(start + n) : -1;
            }
            if (order) {
                if (tid < kTileClasses) class_n[tid] = 0u;
                __syncthreads();
                const int cls = length_class(n);
                const unsigned int rank = valid ? atomicAdd(&class_n[cls], 1u) : 0u;
                __syncthreads();
                if (tid < kTileClasses && class_n[tid])
                    class_base[tid] = class_start[tid] + atomicAdd(&ctrl->class_taken[tid], class_n[tid]);
                __syncthreads();
                if (valid) order[class_base[cls] + rank] = (unsigned int)t;
            }
            if (n) {
                ++touched;
                id_or |= (unsigned int)t;
                id_or_not |= ~(unsigned int)t;
            }
            /* a view's first instance is the smallest start among its tiles */
            const unsigned int s0 = n ? start : 0xFFFFFFFFu;
            const int v = !valid ? -1 : n_views > 1 ? find_view_by_tile(vt, n_views, t) : 0;
            const int v0 = __shfl_sync(0xffffffffu, v, 0);
            if (__all_sync(0xffffffffu, v == v0 || v < 0)) {
                const unsigned int m = __reduce_min_sync(0xffffffffu, s0);
                if (lane == 0 && m != 0xFFFFFFFFu)
                    atomicMin(reinterpret_cast<unsigned long long*>(&vt->view[v0].inst_begin), (unsigned long long)m);
            } else if (n) {
                atomicMin(reinterpret_cast<unsigned long long*>(&vt->view[v].inst_begin), (unsigned long long)start);
            }
            __syncthreads();
            if (tid == 0) base_s += total;
            __syncthreads();
        }
    }
    touched = __reduce_add_sync(0xffffffffu, touched);
    id_or = __reduce_or_sync(0xffffffffu, id_or);
    id_or_not = __reduce_or_sync(0xffffffffu, id_or_not);
    if (lane == 0 && touched) {
        atomicAdd(&ctrl->touched_tiles, touched);
        atomicOr(&ctrl->tile_or, id_or);
        atomicOr(&ctrl->tile_or_not, id_or_not);
    }
}

/* A warp per segment: per tile and 32 pairs, a vote tells the lanes whose
 * pair touches the tile, and they write its next instances. No warp waits for
 * another: a segment's instances of a tile start at the tile's first position
 * plus those of the cell's segments before, and segments are handed out
 * evenly whatever cells they belong to (a warp per cell and 256 pairs, cell by
 * cell, left a tail at long lists: 9 mixed views 193 us against 35).
 * Bound by the votes' population counts (XU 52 %), issue (57 %) and the short
 * runs' partial writes: 24 warps per SM are best (64 views of 300 k: the three
 * kernels 464 us, with 32 warps 480, with 48 and segments of 128 pairs 769); a
 * transpose and a gather in shared memory took half as many instructions again
 * (2 M at 4K: 98 against 71 us). */
template <bool kPacked>
__global__ void __launch_bounds__(kWriteThreads, kWriteCtas)
list_write_kernel(const ViewTable* __restrict__ vt, LumenGpuFrame f, Control* ctrl, Room scratch) {
    chain_begin();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const SortedPairs in = sorted_pairs<kPacked>(f, ctrl, vt);
    const SegmentRoom room = segment_room(scratch, vt, in.n);
    const bool noted = has_room(room, vt, in.n);
    const unsigned int id_mask = in.packed ? (unsigned int)(kPackedCells - 1) : 0xFFFFFFFFu;
    const unsigned int out = ctrl->list_buffer;
    unsigned int* __restrict__ kout = out ? f.keys[1] : f.keys[0];
    unsigned int* __restrict__ vout = out ? f.vals[1] : f.vals[0];
    const long long n_work = noted ? (long long)ctrl->n_segments : vt->hdr.total_cells;
    const long long n_tiles = vt->hdr.total_tiles;
    const unsigned int below = lanemask_lt();
    for (long long w = (long long)blockIdx.x * kWriteWarps + warp; w < n_work; w += (long long)gridDim.x * kWriteWarps) {
        int i0, end, tiles_x, cx = 0, cy = 0;
        unsigned int tile0, before = 0u;
        if (noted) {
            const int4 seg = *reinterpret_cast<const int4*>(room.p + w);
            i0 = seg.x;
            end = seg.x + (seg.y & 1023);
            tile0 = (unsigned int)seg.z;
            tiles_x = seg.w;
            if (lane < kCellTiles) before = room.p[w].before[lane];
            if (const int part = (int)((unsigned int)seg.y >> 10)) {
                /* the parts of the cell before, two at a time */
                const long long cell = min((long long)(in.keys[i0] & id_mask), vt->hdr.total_cells - 1);
                const long long window = vt->hdr.total_cells + i0 / kWindow;   /* the part's own item */
                unsigned int sum = 0u;
#pragma unroll 4
                for (int k = lane / kCellTiles; k < part; k += 2)
                    sum += room.total[k ? window - part + k : cell][lane % kCellTiles];
                before += sum + __shfl_down_sync(0xffffffffu, sum, kCellTiles);
            }
            if (!in.packed) {
                const ViewDesc& vd = vt->view[find_view_by_tile(vt, vt->hdr.n_views, tile0)];
                cx = (int)((tile0 - vd.tile_begin) % tiles_x);
                cy = (int)((tile0 - vd.tile_begin) / tiles_x);
            }
        } else {
            i0 = first_of_cell(in.keys, in.n, id_mask, (unsigned int)w);
            end = first_of_cell(in.keys, in.n, id_mask, (unsigned int)w + 1u);
            const Cell c = find_cell(vt, vt->hdr.n_views, w);
            tile0 = (unsigned int)(c.tile_begin + (long long)c.y * c.tiles_x + c.x);
            tiles_x = c.tiles_x;
            cx = c.x;
            cy = c.y;
        }
        if (i0 >= end) continue;
        /* lane k < 16: tile k's next position and its end (the ids of tiles
         * beyond the view are other tiles', or none; no mask names them) */
        const long long my_tile = (long long)tile0 + lane / kCellSide * tiles_x + lane % kCellSide;
        const bool mine = lane < kCellTiles && my_tile < n_tiles;
        unsigned int at = mine ? (unsigned int)max(f.ranges[2 * my_tile], 0) + before : 0u;
        const unsigned int at_end =
            mine ? (unsigned int)min(max(f.ranges[2 * my_tile + 1], 0), (int)f.instance_capacity) : 0u;
        for (; i0 < end; i0 += kSegment) {
            unsigned int m[kSegment / 32], v[kSegment / 32];
#pragma unroll
            for (int g = 0; g < kSegment / 32; ++g) {
                const int i = i0 + g * 32 + lane;
                v[g] = i < end ? in.vals[i] : 0u;
                m[g] = i < end ? pair_mask(in, in.keys[i], v[g], f.rects, cx, cy) : 0u;
            }
            unsigned int written = 0u;   /* lane k: the segment's instances of tile k */
            bool fits = true;
#pragma unroll
            for (int k = 0; k < kCellTiles; ++k) {
                unsigned int pos = __shfl_sync(0xffffffffu, at, k);
                const unsigned int pos0 = pos, stop = __shfl_sync(0xffffffffu, at_end, k);
                const unsigned int tile = tile0 + (unsigned int)(k / kCellSide * tiles_x + k % kCellSide);
#pragma unroll
                for (int g = 0; g < kSegment / 32; ++g) {
                    const bool hit = (m[g] >> k) & 1u;
                    const unsigned int b = __ballot_sync(0xffffffffu, hit);
                    const unsigned int p = pos + __popc(b & below);
                    if (hit && p < stop) {
                        kout[p] = tile;
                        vout[p] = v[g];
                    }
                    pos += __popc(b);
                }
                fits = fits && pos <= stop | pos == pos0;
                if (lane == k) written = pos - pos0;
            }
            at += written;
            /* self-check: more instances than were counted */
            if (!fits && lane == 0) atomicOr(&ctrl->error_flags, LUMEN_GPU_ERR_BOUNDS);
        }
    }
}

int grid_of(long long n, long long cap) { return (int)(n < 1 ? 1 : n < cap ? n : cap); }

}  // namespace

/* n_cells, n_tiles: the batch's, or upper bounds for a persistent launch
 * (the kernels read the batch's from the table; grids are strided). order_most:
 * the most tiles of a batch that may be composited in one launch, which goes by
 * the tiles' order. */
void launch_lists(ViewTable* vt, const LumenGpuFrame& f, Control* ctrl, unsigned char* scratch, long long room_offset,
                  long long room_bytes, long long n_cells, long long n_tiles, long long order_most, int num_sms,
                  cudaStream_t st) {
    /* Longest lists first: a tile with a long list that starts late runs on
     * alone. Of use from one and a half to ten tiles per resident CTA of the
     * compositor. Compositor, in tile order and longest first: 100 k splats at
     * 999x563 (2268 tiles) 58 -> 40 us and its adjoint 87 -> 70, 250 k at
     * 1279x719 (3600) 113 -> 88, 1 M at 1080p (8160) 155 -> 151. With fewer (50 k
     * at 640x480, 1200 tiles) it gains nothing and the order costs 2 us; with
     * more, neighbouring tiles no longer share their splats in the L2 (2 M at
     * 4K, 32400 tiles: 288 -> 301). */
    const long long line = (long long)kCompositeBlocksPerSm * num_sms;
    const Room room{scratch + room_offset, room_bytes, room_offset, line + line / 2,
                    order_most < 10 * line ? order_most : 10 * line};
    const bool packed = n_cells <= kPackedCells;
    const long long windows = f.instance_capacity / kWindow;
    launch_chained(packed ? list_count_kernel<true> : list_count_kernel<false>,
                   dim3(grid_of(n_cells + windows, (long long)kCountCtas * num_sms)), dim3(kCountThreads), 0, st,
                   (const ViewTable*)vt, f, ctrl, room);
    launch_chained(list_scan_kernel, dim3(grid_of((n_tiles + kScanThreads - 1) / kScanThreads, 2ll * num_sms)),
                   dim3(kScanThreads), 0, st, vt, f.ranges, ctrl, room);
    const long long most = f.instance_capacity / kSegment + n_cells + windows;   /* segments, or cells */
    launch_chained(packed ? list_write_kernel<true> : list_write_kernel<false>,
                   dim3(grid_of((most + kWriteWarps - 1) / kWriteWarps, kWriteCtas * num_sms)), dim3(kWriteThreads), 0,
                   st, (const ViewTable*)vt, f, ctrl, room);
}

}  // namespace lumen
