/*
 * sort.cu - stable LSD radix sort of (key, value) pairs on the device.
 *
 * Reference: radix_sort_64bit, src/raster/radix_sort.mojo:39-87 (eight
 * stable 8-bit LSD passes with 256 buckets).
 *
 * B200 design (onesweep, Adinets & Merrill 2022), for 32- or 64-bit keys:
 *  - one histogram pass reads the keys once and counts every digit that
 *    varies (the frame's cell sort needs none: the emission that writes the
 *    pairs counts their digits). A digit is constant when no two keys differ in
 *    that byte (the OR of all keys and the OR of all complemented keys,
 *    gathered by the kernel that produced them, tell which); a pass over a
 *    constant digit leaves a stable sort unchanged, so it is skipped on the
 *    device.
 *  - each digit pass is one persistent kernel: a CTA takes 4096-key tiles in
 *    ticket order, counts the tile's digits and publishes the counts at
 *    once, ranks its keys with a warp-level multisplit (a shared match mask
 *    per digit; stable: warp order, then item order, then lane order)
 *    straight into shared memory, and then resolves the global
 *    digit offsets by decoupled look-back over earlier tiles. Keys are
 *    written out in digit runs.
 *  - every wait on another CTA's descriptor is bounded.
 * Per pass and pair: (sizeof key + 4) B read and written.
 */
#include "splat_common.cuh"

namespace lumen {

__device__ __forceinline__ unsigned int varying_digits(const SortControl* c, int nbytes, int bits = 8) {
    const unsigned long long v = c->key_or & c->key_or_not;
    unsigned int m = 0;
    for (int d = 0; d < nbytes; ++d)
        if ((v >> (bits * d)) & ((1ull << bits) - 1ull)) m |= 1u << d;
    return m;
}

__device__ __forceinline__ long long sort_count(const SortControl* c, long long capacity) {
    const long long k = (long long)c->n;
    return k < capacity ? k : capacity;
}

/* Histogram of every varying digit; clears the look-back regions of the
 * passes that will run.
 *
 * Each thread counts runs of kRun consecutive keys: equal digits in a row
 * are summed in a register and added to the warp's shared histogram once
 * per run: keys that come in runs (sorted before, or equal in a high byte)
 * cost a few atomics, random digits one shared atomic per key, with no
 * warp-wide match. */
template <typename KeyT>
__global__ void __launch_bounds__(256)
histogram_kernel(const KeyT* __restrict__ keys, long long capacity, SortControl* sc, unsigned int* lb,
                 long long lb_tiles_cap, int tile_keys) {
    chain_begin();
    constexpr int kBytes = (int)sizeof(KeyT);
    constexpr int kRun = kBytes == 8 ? 8 : 16;           /* 64 bytes of keys per thread and run */
    /* a histogram set per warp (per pair of warps for 8-byte keys, to stay
     * within 32 KB) so warps do not contend on the same shared bins */
    constexpr int kWarps = kBytes == 8 ? 4 : 8;
    __shared__ unsigned int h[kWarps][kBytes][256];
    const int tid = threadIdx.x, warp = (tid >> 5) % kWarps;
    const long long K = sort_count(sc, capacity);
    const unsigned int varying = K > 1 ? varying_digits(sc, kBytes) : 0u;
    for (int j = tid; j < kWarps * kBytes * 256; j += 256) (&h[0][0][0])[j] = 0u;
    __syncthreads();
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    const long long gtid = (long long)blockIdx.x * blockDim.x + tid;
    const bool vec = ((uintptr_t)keys & 15u) == 0;   /* runs start 64-byte apart from the base */
    if (varying) {
        for (long long c = gtid; c * kRun < K; c += nthreads) {
            const long long i0 = c * kRun;
            KeyT k[kRun];
            const int nk = (int)(K - i0 < kRun ? K - i0 : kRun);
            if (nk == kRun && vec) {
                const uint4* src = reinterpret_cast<const uint4*>(keys + i0);
#pragma unroll
                for (int q = 0; q < kRun * kBytes / 16; ++q) {
                    const uint4 v = src[q];
                    reinterpret_cast<uint4*>(k)[q] = v;
                }
            } else {
#pragma unroll
                for (int r = 0; r < kRun; ++r) k[r] = r < nk ? keys[i0 + r] : (KeyT)0;
            }
#pragma unroll
            for (int d = 0; d < kBytes; ++d) {
                if (!(varying & (1u << d))) continue;
                unsigned int prev = (unsigned int)((k[0] >> (8 * d)) & 0xFF), run = 1;
#pragma unroll
                for (int r = 1; r < kRun; ++r) {
                    if (r >= nk) break;
                    const unsigned int b = (unsigned int)((k[r] >> (8 * d)) & 0xFF);
                    if (b == prev) {
                        ++run;
                    } else {
                        atomicAdd(&h[warp][d][prev], run);
                        prev = b;
                        run = 1;
                    }
                }
                atomicAdd(&h[warp][d][prev], run);
            }
        }
    }
    __syncthreads();
    if (varying) {
        for (int j = tid; j < kBytes * 256; j += 256) {
            const int d = j >> 8, b = j & 255;
            unsigned int c = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) c += h[w][d][b];
            if ((varying & (1u << d)) && c) atomicAdd(&sc->hist[d][b], c);
        }
        const long long tiles = (K + tile_keys - 1) / tile_keys;
        for (int d = 0; d < kBytes; ++d) {
            if (!(varying & (1u << d))) continue;
            unsigned int* region = lb + (size_t)d * (size_t)lookback_rows(lb_tiles_cap) * 256;
            for (long long j = gtid; j < tiles * 256; j += nthreads) region[j] = 0u;
            const long long groups = (tiles + kLookbackGroup - 1) / kLookbackGroup;
            for (long long j = gtid; j < groups * 256; j += nthreads) region[lb_tiles_cap * 256 + j] = 0u;
        }
    }
    if (blockIdx.x == 0 && tid == 0) {
        sc->varying = varying;
        sc->sorted_buffer = (unsigned int)(__popc(varying) & 1);
    }
}

/* kThreads: threads and digit values of the pass, 256 or 512 (the cell sort's
 * single pass over 257 to 512 cells). */
template <typename KeyT, int kItems, int kThreads = kSortThreads>
struct PassSmem {
    static constexpr int kSets = kThreads == 256 ? 2 : 1;
    KeyT keys[kThreads * kItems];
    unsigned int vals[kThreads * kItems];
    unsigned int whist[kThreads / 32][kThreads];
    unsigned int match[kSets][kThreads / 32][kThreads];   /* per item parity and warp: lanes holding each digit */
    unsigned int digit_start[kThreads];
    long long gbase[kThreads];
    unsigned int goffset[kThreads];
    unsigned int warp_sums[kThreads / 32];
    unsigned int tile;
};

/* Sum over earlier tiles of digit t's count. Within the tile's group of 16
 * the tiles' rows are walked back; beyond, a group is one step: its last
 * tile's row if that is inclusive by now, or else its sum, to which every tile
 * has added its count (and 1 in the upper bits: complete at 16). A walk over
 * every earlier tile, when all resident CTAs start at once, reads about half
 * a row per pair of tiles, 100 MB for 444 tiles, which bound the passes. The
 * rows are read kLookbackWindow at a time (independent loads); one that is
 * not there yet stops the window, and the walk resumes from it. */
constexpr int kLookbackWindow = 4;
constexpr unsigned int kGroupOne = 1u << 20;   /* 16 tiles of at most 6144 keys stay below */

template <int kRow>
__device__ __forceinline__ unsigned int lookback_digit(const unsigned int* lb, const unsigned int* groups, int tile,
                                                       int t, unsigned int* err) {
    unsigned int excl = 0;
    int spins = 0;
    const int g0 = tile / kLookbackGroup;
    for (int j = tile - 1; j >= g0 * kLookbackGroup;) {
        unsigned int d[kLookbackWindow];
#pragma unroll
        for (int w = 0; w < kLookbackWindow; ++w)
            d[w] = j - w >= g0 * kLookbackGroup ? ld_volatile_u32(lb + (size_t)(j - w) * kRow + t) : 0u;
        bool stalled = false;
#pragma unroll
        for (int w = 0; w < kLookbackWindow; ++w) {
            if (stalled || j < g0 * kLookbackGroup) continue;
            const unsigned int v = d[w];
            if (!(v >> 30)) {
                stalled = true;
            } else {
                excl += v & kDescMask32;
                if ((v >> 30) == 2) return excl;
                --j;
            }
        }
        if (stalled) {
            if (++spins >= kSpinLimit) {
                atomicOr(err, LUMEN_GPU_ERR_SPIN_TIMEOUT);
                return excl;
            }
            __nanosleep(32);
        }
    }
    for (int g = g0 - 1; g >= 0;) {
        unsigned int last[kLookbackWindow], sum[kLookbackWindow];
#pragma unroll
        for (int w = 0; w < kLookbackWindow; ++w) {
            const int gw = g - w;
            last[w] = gw >= 0 ? ld_volatile_u32(lb + ((size_t)gw * kLookbackGroup + kLookbackGroup - 1) * kRow + t) : 0u;
            sum[w] = gw >= 0 ? ld_volatile_u32(groups + (size_t)gw * kRow + t) : 0u;
        }
        bool stalled = false;
#pragma unroll
        for (int w = 0; w < kLookbackWindow; ++w) {
            if (stalled || g < 0) continue;
            if ((last[w] >> 30) == 2) return excl + (last[w] & kDescMask32);
            if (sum[w] / kGroupOne == (unsigned int)kLookbackGroup) {
                excl += sum[w] % kGroupOne;
                --g;
            } else {
                stalled = true;
            }
        }
        if (stalled) {
            if (++spins >= kSpinLimit) {
                atomicOr(err, LUMEN_GPU_ERR_SPIN_TIMEOUT);
                return excl;
            }
            __nanosleep(32);
        }
    }
    return excl;
}

/* The frame's cell sort: its last digit pass also writes the cells' ranges
 * (first, end) from the runs of equal cells that it sees. ctrl == nullptr for
 * every other sort. */
struct CellSink {
    Control* ctrl;
    const ViewTable* vt;
    LumenGpuFrame frame;
};

/* Key j of a pass tile (nvalid keys, in sorted order in shared memory) went
 * to global position pos. A digit's keys go to consecutive positions, so a
 * run of equal cells inside the pass tile covers consecutive positions: the
 * cell's range starts at the smallest run start over all pass tiles and ends
 * after the largest run end (the ranges hold (-1, -1) before: -1 is the
 * largest unsigned value, so the minimum replaces it). */
template <typename KeyT>
__device__ __forceinline__ void cell_edges(int* ranges, unsigned int id_mask, const KeyT* skeys, int j, int nvalid,
                                           KeyT kk, long long pos) {
    const unsigned int c = (unsigned int)kk & id_mask;
    if (j == 0 || ((unsigned int)skeys[j - 1] & id_mask) != c)
        atomicMin(reinterpret_cast<unsigned int*>(ranges + 2 * (size_t)c), (unsigned int)pos);
    if (j + 1 == nvalid || ((unsigned int)skeys[j + 1] & id_mask) != c)
        atomicMax(ranges + 2 * (size_t)c + 1, (int)(pos + 1));
}

/* Resident CTAs per SM of a pass. */
template <typename KeyT, int kItems, int kThreads>
constexpr int kPassCtas = sizeof(KeyT) == 4 && kThreads == 256 ? (kItems <= 8 ? 4 : kItems <= 16 ? 3 : 2) : 2;

/* kItems keys per thread: tiles of kThreads * kItems keys. kCellDigits: digits
 * of the width that CellDigits gives (a constant width where it is 8: the
 * depth passes of 250 k splats are 1 us faster each). */
template <typename KeyT, int kItems, int kThreads = kSortThreads, bool kCellDigits = false>
__global__ void __launch_bounds__(kThreads, (kPassCtas<KeyT, kItems, kThreads>))
onesweep_pass_kernel(KeyT* k0, unsigned int* v0, KeyT* k1, unsigned int* v1, long long capacity, SortControl* sc,
                     unsigned int* lb_all, long long lb_tiles_cap, unsigned int* err, int digit, CellSink sink) {
    chain_begin();
    constexpr int kTileKeys = kThreads * kItems;
    constexpr int kWarps = kThreads / 32;
    const int bits = kThreads != 256 ? 9 : kCellDigits ? CellDigits(sink.vt->hdr.total_cells).bits : 8;
    const unsigned int digit_mask = (1u << bits) - 1u;   /* a digit's bits */
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using Smem = PassSmem<KeyT, kItems, kThreads>;
    Smem& s = *reinterpret_cast<Smem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    /* the digits that vary, from the producer's key statistics (the same
     * rule as the histogram kernel's, for sorts whose histogram the producer
     * counted) */
    unsigned int varying = sort_count(sc, capacity) > 1 ? varying_digits(sc, (int)sizeof(KeyT), kThreads == 256 ? bits : 8) : 0u;
    if (kThreads != 256) varying = varying ? 1u : 0u;   /* one digit */
    if (blockIdx.x == 0 && tid == 0) {
        sc->varying = varying;
        sc->sorted_buffer = (unsigned int)(__popc(varying) & 1);
    }
    if (!(varying & (1u << digit))) return;
    const int src = __popc(varying & ((1u << digit) - 1u)) & 1;
    const KeyT* __restrict__ kin = src ? k1 : k0;
    const unsigned int* __restrict__ vin = src ? v1 : v0;
    KeyT* __restrict__ kout = src ? k0 : k1;
    unsigned int* __restrict__ vout = src ? v0 : v1;
    const long long K = sort_count(sc, capacity);
    const long long ntiles = (K + kTileKeys - 1) / kTileKeys;
    const int shift = bits * digit;
    unsigned int* lb = lb_all + (size_t)digit * (size_t)lookback_rows(lb_tiles_cap) * kThreads;
    unsigned int* groups = lb + (size_t)lb_tiles_cap * kThreads;
    int* edges = nullptr;
    unsigned int id_mask = 0xFFFFFFFFu;
    if (sizeof(KeyT) == 4 && sink.ctrl && (varying >> digit) == 1u) {   /* the pass over the highest varying byte */
        edges = cell_ranges(sink.frame, sink.ctrl, sink.vt);
        if (sink.vt->hdr.total_cells <= kPackedCells) id_mask = (unsigned int)(kPackedCells - 1);
        if (edges && blockIdx.x == 0 && tid == 0) sink.ctrl->cells_by_sort = 1u;
    }

    /* global exclusive offsets of this digit's buckets */
    {
        const unsigned int c = (&sc->hist[0][0])[digit * 256 + tid];
        unsigned int x = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s.warp_sums[warp] = x;
        __syncthreads();
        unsigned int wb = 0;
        for (int w = 0; w < warp; ++w) wb += s.warp_sums[w];
        s.goffset[tid] = wb + x - c;
        __syncthreads();
    }

    /* the match masks start clear; each item's leaders clear what it set */
    for (int j = tid; j < Smem::kSets * kWarps * kThreads; j += kThreads) (&s.match[0][0][0])[j] = 0u;

    for (;;) {
        if (tid == 0) s.tile = atomicAdd(&sc->pass_ticket[digit], 1u);
        __syncthreads();
        const long long tile = s.tile;
        if (tile >= ntiles) break;
        const long long base = tile * kTileKeys;

        /* warp w owns keys [base + w*512, +512); item i of lane l is base + w*512 + i*32 + l */
        KeyT k[kItems];
        unsigned int v[kItems];
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            const long long idx = base + warp * (kItems * 32) + it * 32 + lane;
            const bool valid = idx < K;
            k[it] = valid ? kin[idx] : (KeyT)0;
            v[it] = valid ? vin[idx] : 0u;
        }
        const long long wbase = base + warp * (kItems * 32);
        for (int b = lane; b < kThreads; b += 32) s.whist[warp][b] = 0u;
        __syncwarp();
        /* the tile's digit counts come first (per-warp shared histograms; the
         * order of the increments does not matter), so that the tile's
         * aggregate is published before its keys are ranked and the
         * look-back chain of the tiles after it moves on sooner */
#pragma unroll
        for (int it = 0; it < kItems; ++it)
            if (wbase + it * 32 + lane < K) atomicAdd(&s.whist[warp][(unsigned int)((k[it] >> shift) & digit_mask)], 1u);
        __syncthreads();
        /* digit t: warp-exclusive offsets and the tile's count */
        const int t = tid;
        unsigned int run = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const unsigned int c = s.whist[w][t];
            s.whist[w][t] = run;
            run += c;
        }
        const unsigned int count = run;
        st_volatile_u32(lb + (size_t)tile * kThreads + t, (tile == 0 ? kDescIncl32 : kDescAgg32) | count);
        atomicAdd(groups + (size_t)(tile / kLookbackGroup) * kThreads + t, kGroupOne + count);
        {
            unsigned int x = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                unsigned int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (lane == 31) s.warp_sums[warp] = x;
            __syncthreads();
            unsigned int wb = 0;
            for (int w = 0; w < warp; ++w) wb += s.warp_sums[w];
            s.digit_start[t] = wb + x - count;
        }
        __syncthreads();
        /* warp-level stable multisplit (warp order, then item order, then
         * lane order): each lane sets its bit in the shared mask of its
         * digit, so after a warp barrier the mask names the lanes holding the
         * same digit (one shared atomic per key, where a ballot per digit bit
         * costs eight vote and select steps and a match instruction slows
         * down with the number of distinct digits). The lowest such lane
         * advances the warp's running count of the digit, which starts at its
         * warp-exclusive offset, and clears the mask; a key's rank is then its
         * place in the tile's digit run and it goes straight to its slot in
         * shared memory. Items alternate between two mask sets, so the
         * clearing of one item's masks needs no barrier of its own before the
         * next item sets the other set. */
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            const bool valid = wbase + it * 32 + lane < K;
            const unsigned int d = (unsigned int)((k[it] >> shift) & digit_mask);
            unsigned int* mk = s.match[it % Smem::kSets][warp];
            if (valid) atomicOr(&mk[d], 1u << lane);
            __syncwarp();
            const unsigned int peers = valid ? mk[d] : 0u;
            unsigned int prior = 0;
            if (valid) prior = s.whist[warp][d];
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) {
                s.whist[warp][d] = prior + __popc(peers);
                mk[d] = 0u;
            }
            if (valid) {
                const unsigned int pos = s.digit_start[d] + prior + __popc(peers & lanemask_lt());
                s.keys[pos] = k[it];
                s.vals[pos] = v[it];
            }
            if (Smem::kSets == 1) __syncwarp();   /* the masks are clear before the next item sets them */
        }
        /* the look-back runs once the keys are in shared memory (their
         * registers are free for a wide window of descriptors) */
        unsigned int excl = 0;
        if (tile > 0) {
            excl = lookback_digit<kThreads>(lb, groups, (int)tile, t, err);
            st_volatile_u32(lb + (size_t)tile * kThreads + t, kDescIncl32 | (excl + count));
        }
        s.gbase[t] = (long long)s.goffset[t] + (long long)excl - (long long)s.digit_start[t];
        __syncthreads();
        const int nvalid = (int)((K - base) < kTileKeys ? (K - base) : kTileKeys);
        if (nvalid == kTileKeys) {
#pragma unroll
            for (int it = 0; it < kItems; ++it) {
                const int j = it * kThreads + tid;
                const KeyT kk = s.keys[j];
                const unsigned int d = (unsigned int)((kk >> shift) & digit_mask);
                const long long out = s.gbase[d] + j;
                kout[out] = kk;
                vout[out] = s.vals[j];
                if (edges) cell_edges(edges, id_mask, s.keys, j, kTileKeys, kk, out);
            }
        } else {
            for (int j = tid; j < nvalid; j += kThreads) {
                const KeyT kk = s.keys[j];
                const unsigned int d = (unsigned int)((kk >> shift) & digit_mask);
                const long long out = s.gbase[d] + j;
                kout[out] = kk;
                vout[out] = s.vals[j];
                if (edges) cell_edges(edges, id_mask, s.keys, j, nvalid, kk, out);
            }
        }
        __syncthreads();
    }
}

/* A whole sort of up to 131072 keys in one launch, by one cluster of CTAs.
 * Each CTA holds an equal run of the keys and runs a pass as above, but the
 * digit counts of the CTAs before it come from their shared memory (a cluster
 * barrier instead of descriptors to wait for), and the next pass starts at a
 * cluster barrier instead of a launch. The pairs move between the CTAs through
 * the L2.
 *
 * A sort of so few keys is bound by latency: with the histogram and a launch
 * per digit, most of it went to launches (2.5 us each on the device, 4 us to
 * issue) and the passes' fixed 7 to 10 us. The sort of the depth keys, before
 * and after: 512 splats 27 -> 11 us, 50 k 34 -> 20, 100 k 40 -> 24, and four
 * launches fewer. Up to 1024 keys one CTA does, up to 8192 eight (a key per
 * thread; the largest portable cluster), beyond them sixteen where the device
 * takes such a cluster (100 k keys: 24 us against 31 with eight). At 250 k keys
 * the digit passes over the whole GPU are faster (65 us against 89), and eight
 * CTAs hold 131072 keys (16 per thread), hence the limit. */
constexpr int kClusterThreads = 1024;
constexpr int kClusterItems = 16;
constexpr int kClusterCtas = 8;
constexpr int kClusterKeys = kClusterThreads * kClusterItems;   /* per CTA */
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kCountParts = kClusterThreads / 256;
static int g_cluster_ctas = kClusterCtas;   /* for more than a key per thread of eight CTAs */

struct ClusterSmem {
    unsigned int keys[kClusterKeys], vals[kClusterKeys];
    unsigned int whist[kClusterWarps][256];
    unsigned int match[kClusterWarps][256];
    unsigned int part[kCountParts][256];
    unsigned int count[256];          /* the CTA's digit counts, read by the whole cluster */
    unsigned int digit_start[256];
    unsigned int gbase[256];
    unsigned int warp_sums[8];
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }

/* The word at p of the cluster's CTA rank. */
__device__ __forceinline__ unsigned int cluster_read(const unsigned int* p, unsigned int rank) {
    unsigned int addr = (unsigned int)__cvta_generic_to_shared(p), v;
    asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(addr) : "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

/* Exclusive scan of x over threads 0 to 255 (the other threads only keep the
 * barriers). */
__device__ __forceinline__ unsigned int digit_scan(unsigned int x, unsigned int* warp_sums) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int incl = x;
    if (warp < 8) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) warp_sums[warp] = incl;
    }
    __syncthreads();
    if (warp < 8)
        for (int w = 0; w < warp; ++w) incl += warp_sums[w];
    return incl - x;
}

__global__ void __launch_bounds__(kClusterThreads, 1)
cluster_sort_kernel(unsigned int* k0, unsigned int* v0, unsigned int* k1, unsigned int* v1, long long capacity,
                    SortControl* sc) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ClusterSmem& s = *reinterpret_cast<ClusterSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned int rank, ctas;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(ctas));
    const int K = (int)sort_count(sc, capacity);   /* at most ctas * kClusterKeys */
    const unsigned int varying = K > 1 ? varying_digits(sc, 4) : 0u;
    if (rank == 0 && tid == 0) {
        sc->varying = varying;
        sc->sorted_buffer = (unsigned int)(__popc(varying) & 1);
    }
    const int items = (K + (int)ctas * kClusterThreads - 1) / ((int)ctas * kClusterThreads);
    const int base = (int)rank * items * kClusterThreads;
    const int nvalid = min(max(K - base, 0), items * kClusterThreads);
    const int wbase = base + warp * items * 32;   /* warp w owns items * 32 consecutive keys */
    const unsigned int *kin = k0, *vin = v0;
    unsigned int *kout = k1, *vout = v1;
    for (int shift = 0; shift < 32; shift += 8) {
        if (!(varying & (1u << (shift / 8)))) continue;
        unsigned int k[kClusterItems], v[kClusterItems];
#pragma unroll
        for (int it = 0; it < kClusterItems; ++it) {
            const int i = wbase + it * 32 + lane;
            const bool valid = it < items && i < K;
            k[it] = valid ? __ldcg(kin + i) : 0u;
            v[it] = valid ? __ldcg(vin + i) : 0u;
        }
        for (int b = lane; b < 256; b += 32) {
            s.whist[warp][b] = 0u;
            s.match[warp][b] = 0u;
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < kClusterItems; ++it)
            if (it < items && wbase + it * 32 + lane < K) atomicAdd(&s.whist[warp][(k[it] >> shift) & 0xFFu], 1u);
        __syncthreads();
        /* digit t's warp-exclusive offsets, eight warps per thread */
        const int t = tid & 255, part = tid >> 8;
        unsigned int run = 0u, n[kClusterWarps / kCountParts];
#pragma unroll
        for (int w = 0; w < kClusterWarps / kCountParts; ++w) {
            n[w] = s.whist[part * (kClusterWarps / kCountParts) + w][t];
            run += n[w];
        }
        s.part[part][t] = run;
        __syncthreads();
        unsigned int before = 0u, count = 0u;
#pragma unroll
        for (int p = 0; p < kCountParts; ++p) {
            const unsigned int x = s.part[p][t];
            if (p < part) before += x;
            count += x;
        }
#pragma unroll
        for (int w = 0; w < kClusterWarps / kCountParts; ++w) {
            s.whist[part * (kClusterWarps / kCountParts) + w][t] = before;
            before += n[w];
        }
        if (part == 0) s.count[t] = count;
        cluster_arrive();   /* the counts are there once every CTA has arrived */
        const unsigned int start = digit_scan(count, s.warp_sums);
        if (part == 0) s.digit_start[t] = start;
        __syncthreads();
        /* the warp-level multisplit of the digit pass, with one set of masks */
#pragma unroll
        for (int it = 0; it < kClusterItems; ++it) {
            if (it >= items) break;
            const bool valid = wbase + it * 32 + lane < K;
            const unsigned int d = (k[it] >> shift) & 0xFFu;
            if (valid) atomicOr(&s.match[warp][d], 1u << lane);
            __syncwarp();
            const unsigned int peers = valid ? s.match[warp][d] : 0u;
            const unsigned int prior = valid ? s.whist[warp][d] : 0u;
            __syncwarp();
            if (valid) {
                if (lane == __ffs(peers) - 1) {
                    s.whist[warp][d] = prior + __popc(peers);
                    s.match[warp][d] = 0u;
                }
                const unsigned int pos = s.digit_start[d] + prior + __popc(peers & lanemask_lt());
                s.keys[pos] = k[it];
                s.vals[pos] = v[it];
            }
            __syncwarp();
        }
        cluster_wait();
        /* digit t's place among all keys, less its place in the CTA's */
        unsigned int total = 0u, earlier = 0u;
        if (part == 0)
            for (unsigned int c = 0; c < ctas; ++c) {
                const unsigned int x = cluster_read(&s.count[t], c);
                if (c < rank) earlier += x;
                total += x;
            }
        const unsigned int first = digit_scan(total, s.warp_sums);
        if (part == 0) s.gbase[t] = first + earlier - start;
        __syncthreads();
        for (int j = tid; j < nvalid; j += kClusterThreads) {
            const unsigned int kk = s.keys[j];
            const unsigned int out = s.gbase[(kk >> shift) & 0xFFu] + (unsigned int)j;
            kout[out] = kk;
            vout[out] = s.vals[j];
        }
        /* every pair of the pass is written, and no count is read any more */
        cluster_arrive();
        cluster_wait();
        kin = kin == k0 ? k1 : k0;
        vin = vin == v0 ? v1 : v0;
        kout = kout == k0 ? k1 : k0;
        vout = vout == v0 ? v1 : v0;
    }
}

/* OR and OR-of-complement of n keys and the pair count, for sorts whose
 * keys come from the caller (lumen_gpu_sort_pairs). */
template <typename KeyT>
__global__ void __launch_bounds__(256)
key_stats_kernel(const KeyT* __restrict__ keys, long long n, SortControl* sc) {
    unsigned long long o = 0ull, no = 0ull;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += nthreads) {
        const unsigned long long k = (unsigned long long)keys[i];
        o |= k;
        no |= ~k;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        o |= __shfl_xor_sync(0xffffffffu, o, off);
        no |= __shfl_xor_sync(0xffffffffu, no, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicOr(&sc->key_or, o);
        atomicOr(&sc->key_or_not, no);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->n = (unsigned long long)n;
}

/* Rebuild the reference's 64-bit keys: (tile << 32) | depth key of the
 * instance's splat. */
__global__ void sorted_keys64_kernel(const unsigned int* k0, const unsigned int* k1, const unsigned int* v0,
                                     const unsigned int* v1, const LumenSplatRecord* records, long long capacity,
                                     int key_mode, const Control* ctrl, unsigned long long* out) {
    const long long K = (long long)ctrl->n_instances < capacity ? (long long)ctrl->n_instances : capacity;
    const unsigned int* keys = ctrl->list_buffer ? k1 : k0;
    const unsigned int* vals = ctrl->list_buffer ? v1 : v0;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < K; i += nthreads) {
        const unsigned int v = vals[i];
        out[i] = ((unsigned long long)keys[i] << 32) | depth_key(records[v].depth, key_mode);
    }
}

/* key_bytes: the low bytes that can vary at all (a pass per byte is
 * launched; among those, passes over bytes that turn out constant exit at
 * once). */
template <typename KeyT, int kItems, int kThreads = kSortThreads, bool kCellDigits = false>
void launch_sort_impl(KeyT* k0, unsigned int* v0, KeyT* k1, unsigned int* v1, long long capacity, SortControl* sc,
                      unsigned int* lb, long long lb_tiles_cap, unsigned int* err, int key_bytes, int num_sms,
                      cudaStream_t st, const CellSink* sink = nullptr) {
    if (!sink) {
        /* Not chained: its blocks (32 KB of shared memory each) would take the
         * places that the producer's last blocks leave, ahead of those still
         * to come (64 views of 300 k: a batch 5.50 -> 5.39 ms without; single
         * frames 1 us). */
        ChainedLaunches chained(false);
        launch_chained(histogram_kernel<KeyT>, dim3(num_sms * 4), dim3(256), 0, st, (const KeyT*)k0, capacity, sc, lb,
                       lb_tiles_cap, kSortThreads * kItems);
    }
    const size_t smem = sizeof(PassSmem<KeyT, kItems, kThreads>);
    const int ctas_per_sm = kPassCtas<KeyT, kItems, kThreads>;   /* all CTAs resident */
    const int nd = key_bytes < (int)sizeof(KeyT) ? key_bytes : (int)sizeof(KeyT);
    for (int d = 0; d < nd; ++d)
        launch_chained(onesweep_pass_kernel<KeyT, kItems, kThreads, kCellDigits>, dim3(num_sms * ctas_per_sm), dim3(kThreads), smem, st,
                       k0, v0, k1, v1, capacity, sc, lb, lb_tiles_cap, err, d, sink ? *sink : CellSink{});
}

/* items: keys per thread of a digit pass, 8, 16 or 24 (tiles of 2048, 4096
 * or 6144 keys); lb_tiles_cap must hold ceil(capacity / (256 * items))
 * tiles. */
template <bool kCellDigits>
static void launch_sort_items(unsigned int* k0, unsigned int* v0, unsigned int* k1, unsigned int* v1,
                              long long capacity, SortControl* sc, unsigned int* lb, long long lb_tiles_cap,
                              unsigned int* err, int items, int key_bytes, const CellSink* sink, int num_sms,
                              cudaStream_t st) {
    auto run = [&](auto kernel) { kernel(k0, v0, k1, v1, capacity, sc, lb, lb_tiles_cap, err, key_bytes, num_sms, st, sink); };
    if (items == 8) run(launch_sort_impl<unsigned int, 8, kSortThreads, kCellDigits>);
    else if (items == 24) run(launch_sort_impl<unsigned int, 24, kSortThreads, kCellDigits>);
    else run(launch_sort_impl<unsigned int, 16, kSortThreads, kCellDigits>);
}

void launch_sort32(unsigned int* k0, unsigned int* v0, unsigned int* k1, unsigned int* v1, long long capacity,
                   SortControl* sc, unsigned int* lb, long long lb_tiles_cap, unsigned int* err, int items,
                   int key_bytes, int num_sms, cudaStream_t st) {
    if (capacity <= (long long)kClusterCtas * kClusterKeys && key_bytes >= 4) {
        const int ctas = capacity <= kClusterThreads                  ? 1
                         : capacity <= kClusterCtas * kClusterThreads ? kClusterCtas
                                                                      : g_cluster_ctas;
        launch_chained_cluster(cluster_sort_kernel, ctas, dim3(ctas), dim3(kClusterThreads), sizeof(ClusterSmem), st,
                               k0, v0, k1, v1, capacity, sc);
        return;
    }
    launch_sort_items<false>(k0, v0, k1, v1, capacity, sc, lb, lb_tiles_cap, err, items, key_bytes, nullptr, num_sms,
                             st);
}

/* The frame's cell sort: the emission has counted the pairs' digits, cleared
 * the look-back tiles and filled the cells' ranges with -1, so only the digit
 * passes run, the last of which writes the ranges. */
void launch_cell_sort(const LumenGpuFrame& f, Control* ctrl, const ViewTable* vt, unsigned int* lb,
                      long long lb_tiles_cap, int items, CellDigits digits, bool wide, bool persistent, int num_sms,
                      cudaStream_t st) {
    const CellSink sink{ctrl, vt, f};
    if (wide) {
        launch_sort_impl<unsigned int, kWideItems, kWideCells>(
            f.keys[0], f.vals[0], f.keys[1], f.vals[1], f.instance_capacity, &ctrl->cell_sort, lb, lb_tiles_cap,
            &ctrl->error_flags, 1, num_sms, st, &sink);
        return;
    }
    /* persistent launches learn the cells, and with them the width, on the device */
    auto run = persistent || digits.bits != 8 ? launch_sort_items<true> : launch_sort_items<false>;
    run(f.keys[0], f.vals[0], f.keys[1], f.vals[1], f.instance_capacity, &ctrl->cell_sort, lb, lb_tiles_cap,
        &ctrl->error_flags, items, digits.n, &sink, num_sms, st);
}

void launch_sort64(unsigned long long* k0, unsigned int* v0, unsigned long long* k1, unsigned int* v1,
                   long long capacity, SortControl* sc, unsigned int* lb, long long lb_tiles_cap, unsigned int* err,
                   int num_sms, cudaStream_t st) {
    launch_sort_impl<unsigned long long, kSort64Items>(k0, v0, k1, v1, capacity, sc, lb, lb_tiles_cap, err, 8,
                                                       num_sms, st);
}

void launch_key_stats64(const unsigned long long* keys, long long n, SortControl* sc, int num_sms, cudaStream_t st) {
    key_stats_kernel<unsigned long long><<<num_sms * 2, 256, 0, st>>>(keys, n, sc);
}

void launch_sorted_keys64(const LumenGpuFrame& f, const Control* ctrl, int key_mode, unsigned long long* out,
                          int num_sms, cudaStream_t st) {
    sorted_keys64_kernel<<<num_sms * 4, 256, 0, st>>>(f.keys[0], f.keys[1], f.vals[0], f.vals[1], f.records,
                                                      (long long)f.instance_capacity, key_mode, ctrl, out);
}

void configure_sort_kernels() {
    cudaFuncSetAttribute(cluster_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ClusterSmem));
    /* a cluster of 16 where the device can hold one */
    cudaFuncSetAttribute(cluster_sort_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * kClusterCtas);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = sizeof(ClusterSmem);
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2 * kClusterCtas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, cluster_sort_kernel, &cfg) == cudaSuccess && clusters > 0)
        g_cluster_ctas = 2 * kClusterCtas;
    else
        cudaGetLastError();
    auto allow = [](auto kernel, size_t smem) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    };
    allow(onesweep_pass_kernel<unsigned int, 8>, sizeof(PassSmem<unsigned int, 8>));
    allow(onesweep_pass_kernel<unsigned int, 16>, sizeof(PassSmem<unsigned int, 16>));
    allow(onesweep_pass_kernel<unsigned int, 24>, sizeof(PassSmem<unsigned int, 24>));
    allow(onesweep_pass_kernel<unsigned int, 8, kSortThreads, true>, sizeof(PassSmem<unsigned int, 8>));
    allow(onesweep_pass_kernel<unsigned int, 16, kSortThreads, true>, sizeof(PassSmem<unsigned int, 16>));
    allow(onesweep_pass_kernel<unsigned int, 24, kSortThreads, true>, sizeof(PassSmem<unsigned int, 24>));
    cudaFuncSetAttribute(onesweep_pass_kernel<unsigned int, kWideItems, kWideCells>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(PassSmem<unsigned int, kWideItems, kWideCells>));
    cudaFuncSetAttribute(onesweep_pass_kernel<unsigned long long, kSort64Items>,
                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(PassSmem<unsigned long long, kSort64Items>));
}

}  // namespace lumen
