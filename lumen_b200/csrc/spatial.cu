/*
 * spatial.cu - picking on the device (include/lumen_spatial.h): the LBVH
 * build and closest-splat ray casts.
 *
 * Reference: LBVH.build_from_cloud (src/spatial/bvh.mojo:45-120),
 * compute_morton_3d / expand_bits_10_to_30 (src/spatial/morton.mojo:7-46),
 * AABB3f.expand_point / expand_box / intersect_ray (src/spatial/aabb.mojo:47-98),
 * raycast_closest_splat (src/spatial/raycast.mojo:30-95), Ray3f and
 * PinholeCamera.generate_ray (src/scene/camera.mojo:12-21, 85-90).
 *
 * Build, all on one stream:
 *   K1 bbox_kernel      the cloud's box: per-axis min and max of the positions
 *                       (NaN skipped, as add_gaussian's comparisons skip it),
 *                       reduced with atomicMax on order-preserving bit keys
 *   K2 morton_kernel    one 30-bit code per Gaussian, index as the value, and
 *                       which bits of the codes vary (the sort skips digits
 *                       that do not; a kernel of its own for this took 5 us)
 *   K3 the library's stable onesweep radix sort (32-bit keys, 4 digit passes)
 *   K4 bvh_levels_kernel, once per ten levels: a block writes 1024 leaves
 *                       (or loads 1024 nodes of the level reached so far)
 *                       and builds their ancestors ten levels up in shared
 *                       memory, one barrier per level. Parents pair adjacent
 *                       nodes, so 1024 aligned nodes never need another
 *                       block's: each parent is built once, in the
 *                       reference's order (left box expanded by the right),
 *                       and the nodes equal the reference's level-by-level
 *                       pairing bit for bit (1M leaves: two launches).
 *                       Node numbering is the reference's: leaves, then each
 *                       level's parents.
 * Casts: eight lanes per ray walk the hierarchy three levels at a time, the
 * nearest nodes first (cast_ray); the hits are those of the reference's
 * depth-first order bit for bit, ties included. Rays for which that order
 * could show, and hierarchies that are not as the build leaves them for the
 * Gaussians as they are now (check_nodes_kernel), are cast in that order by
 * one thread (cast_ray_in_order).
 *
 * Memory: the build reads 24 B per Gaussian twice and writes 32 B per node
 * (n + ceil(n / 2) + ceil(n / 4) + ... nodes, about 64 MB for 1M Gaussians) plus the sort's traffic.
 */
#include "splat_common.cuh"
#include "../../include/lumen_spatial.h"

namespace lumen {
LumenStatus map_cuda(cudaError_t e);
LumenStatus status_from_flags(unsigned int flags);
int device_sm_count();
void configure_once();
void launch_sort32(unsigned int* k0, unsigned int* v0, unsigned int* k1, unsigned int* v1, long long capacity,
                   SortControl* sc, unsigned int* lb, long long lb_tiles_cap, unsigned int* err, int items,
                   int key_bytes, int num_sms, cudaStream_t st);

namespace {

constexpr int kMaxLevels = 40;        /* 2^30 leaves need 31 levels */
constexpr int kRayStack = 64;         /* a traversal holds at most levels + 1 entries */

struct BvhControl {
    SortControl sort;
    unsigned int error_flags;
    unsigned int lo[3];               /* max of ~key(p): the minimum, 0 when none */
    unsigned int hi[3];               /* max of key(p): the maximum, 0 when none */
};

struct BvhLevels {
    int n_levels;
    long long start[kMaxLevels];
    long long count[kMaxLevels];
};

struct BvhLayout {
    size_t control_off, keys0_off, vals0_off, keys1_off, vals1_off, lb_off, total;
    long long sort_tiles;
    size_t zeroed() const { return keys0_off; }
};

BvhLevels make_levels(long long n) {
    BvhLevels L;
    L.n_levels = 0;
    if (n <= 0) return L;
    long long start = 0, count = n;
    L.start[0] = 0;
    L.count[0] = n;
    L.n_levels = 1;
    while (count > 1) {                                    /* bvh.mojo:96-117 */
        start += count;
        count = (count + 1) / 2;
        L.start[L.n_levels] = start;
        L.count[L.n_levels] = count;
        ++L.n_levels;
    }
    return L;
}

long long node_count_of(long long n) {
    if (n <= 0) return 0;
    const BvhLevels L = make_levels(n);
    return L.start[L.n_levels - 1] + 1;
}

BvhLayout make_layout(long long n) {
    BvhLayout B;
    B.sort_tiles = (n + kSortTileMin - 1) / kSortTileMin;
    B.control_off = 0;
    B.keys0_off = align_up(sizeof(BvhControl), 256);
    B.vals0_off = align_up(B.keys0_off + (size_t)n * 4, 256);
    B.keys1_off = align_up(B.vals0_off + (size_t)n * 4, 256);
    B.vals1_off = align_up(B.keys1_off + (size_t)n * 4, 256);
    B.lb_off = align_up(B.vals1_off + (size_t)n * 4, 256);
    B.total = align_up(B.lb_off + (size_t)4 * (size_t)lookback_rows(B.sort_tiles > 0 ? B.sort_tiles : 1) * 256 * 4, 256);
    return B;
}

/* order-preserving key of a float (NaN excluded by the callers) */
__device__ __forceinline__ unsigned int ord_key(float f) {
    const unsigned int b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float ord_value(unsigned int k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

__global__ void __launch_bounds__(256)
bbox_kernel(const float* __restrict__ means, long long n, BvhControl* ctrl) {
    __shared__ unsigned int s_lo[3][8], s_hi[3][8];
    unsigned int lo[3] = {0u, 0u, 0u}, hi[3] = {0u, 0u, 0u};
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const float p = means[i * 3 + c];
            if (p == p) {                                  /* gaussian_cloud.mojo:36-42 skip NaN */
                const unsigned int k = ord_key(p);
                lo[c] = max(lo[c], ~k);
                hi[c] = max(hi[c], k);
            }
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        lo[c] = __reduce_max_sync(0xffffffffu, lo[c]);
        hi[c] = __reduce_max_sync(0xffffffffu, hi[c]);
        if (lane == 0) {
            s_lo[c][warp] = lo[c];
            s_hi[c][warp] = hi[c];
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        const int c = threadIdx.x;
        unsigned int a = 0u, b = 0u;
        for (int w = 0; w < 8; ++w) {
            a = max(a, s_lo[c][w]);
            b = max(b, s_hi[c][w]);
        }
        if (a) atomicMax(&ctrl->lo[c], a);
        if (b) atomicMax(&ctrl->hi[c], b);
    }
}

/* expand_bits_10_to_30, morton.mojo:7-18 */
__device__ __forceinline__ unsigned int expand_bits(unsigned int val) {
    unsigned int v = val & 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

/* compute_morton_3d, morton.mojo:21-46 (a NaN coordinate counts as 0) */
__device__ __forceinline__ unsigned int morton3(float nx, float ny, float nz) {
    float c[3] = {nx, ny, nz};
    unsigned int q[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float v = c[k];
        if (v < 0.0f) v = 0.0f;
        else if (v > 1.0f) v = 1.0f;
        q[k] = v == v ? (unsigned int)(v * 1023.0f) : 0u;
    }
    return expand_bits(q[0]) | (expand_bits(q[1]) << 1) | (expand_bits(q[2]) << 2);
}

__global__ void __launch_bounds__(256)
morton_kernel(const float* __restrict__ means, long long n, BvhControl* __restrict__ ctrl,
              unsigned int* __restrict__ keys, unsigned int* __restrict__ vals) {
    /* the box as add_gaussian leaves it: min from 1e9, max from -1e9 */
    float mn[3], inv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        float lo = (float)1e9, hi = (float)-1e9;
        const unsigned int a = ctrl->lo[c], b = ctrl->hi[c];
        if (a) {
            const float v = ord_value(~a);
            if (v < lo) lo = v;
        }
        if (b) {
            const float v = ord_value(b);
            if (v > hi) hi = v;
        }
        const float extent = hi - lo;                                    /* bvh.mojo:52-58 */
        mn[c] = lo;
        inv[c] = 1.0f / (extent > (float)0.001 ? extent : 1.0f);
    }
    unsigned int key_or = 0u, key_or_not = 0u;
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        const float nx = (means[i * 3 + 0] - mn[0]) * inv[0];                /* bvh.mojo:64-72 */
        const float ny = (means[i * 3 + 1] - mn[1]) * inv[1];
        const float nz = (means[i * 3 + 2] - mn[2]) * inv[2];
        const unsigned int code = morton3(nx, ny, nz);
        keys[i] = code;
        vals[i] = (unsigned int)i;
        key_or |= code;
        key_or_not |= ~code;
    }
    /* the sort's key statistics, one atomic per block and word */
    __shared__ unsigned int block_or, block_or_not;
    if (threadIdx.x == 0) block_or = block_or_not = 0u;
    __syncthreads();
    key_or = __reduce_or_sync(0xffffffffu, key_or);
    key_or_not = __reduce_or_sync(0xffffffffu, key_or_not);
    if ((threadIdx.x & 31) == 0) {
        atomicOr(&block_or, key_or);
        atomicOr(&block_or_not, key_or_not);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicOr(&ctrl->sort.key_or, (unsigned long long)block_or);
        atomicOr(&ctrl->sort.key_or_not, (unsigned long long)block_or_not);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ctrl->sort.n = (unsigned long long)n;
}

struct Box {
    float mn[3], mx[3];
};

__device__ __forceinline__ Box load_box_cg(const LumenBvhNode* node, int* left, int* right) {
    const float4 a = __ldcg(reinterpret_cast<const float4*>(node));
    const float4 b = __ldcg(reinterpret_cast<const float4*>(node) + 1);
    if (left) *left = __float_as_int(a.w);
    if (right) *right = __float_as_int(b.w);
    return Box{{a.x, a.y, a.z}, {b.x, b.y, b.z}};
}

__device__ __forceinline__ void store_node(LumenBvhNode* node, const Box& b, int left, int right) {
    float4* p = reinterpret_cast<float4*>(node);
    __stcg(p, make_float4(b.mn[0], b.mn[1], b.mn[2], __int_as_float(left)));
    __stcg(p + 1, make_float4(b.mx[0], b.mx[1], b.mx[2], __int_as_float(right)));
}

/* A leaf's box: position +- 3 x the largest scale (bvh.mojo:78-93). */
__device__ __forceinline__ Box leaf_box(const float* __restrict__ means, const float* __restrict__ scales, long long g) {
    float r = scales[g * 3 + 0];
    if (scales[g * 3 + 1] > r) r = scales[g * 3 + 1];
    if (scales[g * 3 + 2] > r) r = scales[g * 3 + 2];
    const float r3 = r * 3.0f;
    Box leaf;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const float pc = means[g * 3 + c];
        leaf.mn[c] = pc - r3;
        leaf.mx[c] = pc + r3;
    }
    return leaf;
}

/* AABB3f.expand_point, aabb.mojo:47-54 */
__device__ __forceinline__ void expand_point(Box& b, const float p[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
        if (p[c] < b.mn[c]) b.mn[c] = p[c];
#pragma unroll
    for (int c = 0; c < 3; ++c)
        if (p[c] > b.mx[c]) b.mx[c] = p[c];
}

/* Levels of the hierarchy built per launch: a block takes 1024 consecutive
 * nodes of level L0 (for L0 = 0 it first writes them as leaves) and builds
 * their ancestors up to level L0 + 10 in shared memory, one level per
 * barrier; parents pair adjacent nodes exactly as bvh.mojo:96-117 does, so
 * a block's subtree never needs another block's nodes. */
constexpr int kRefitSpan = 10;
constexpr int kRefitNodes = 1 << kRefitSpan;
constexpr int kRefitThreads = 256;

__global__ void __launch_bounds__(kRefitThreads)
bvh_levels_kernel(const float* __restrict__ means, const float* __restrict__ scales, long long n,
                  const BvhControl* __restrict__ ctrl, const unsigned int* __restrict__ v0,
                  const unsigned int* __restrict__ v1, LumenBvhNode* __restrict__ nodes,
                  int* __restrict__ splat_index, BvhLevels lv, int L0) {
    __shared__ Box cur[kRefitNodes];
    __shared__ Box nxt[kRefitNodes / 2];
    const int tid = threadIdx.x;
    const long long b = blockIdx.x;
    const long long first = b * kRefitNodes;
    const long long cnt0 = lv.count[L0];
    const int m0 = (int)(cnt0 - first < kRefitNodes ? cnt0 - first : kRefitNodes);
    if (L0 == 0) {
        const unsigned int* perm = ctrl->sort.sorted_buffer ? v1 : v0;
        for (int k = tid; k < m0; k += kRefitThreads) {
            const long long i = first + k;
            const long long g = perm[i];
            const Box leaf = leaf_box(means, scales, g);
            store_node(nodes + i, leaf, -1, -1);
            splat_index[i] = (int)g;
            cur[k] = leaf;
        }
    } else {
        for (int k = tid; k < m0; k += kRefitThreads)
            cur[k] = load_box_cg(nodes + lv.start[L0] + first + k, nullptr, nullptr);
    }
    __syncthreads();
    Box* src = cur;
    Box* dst = nxt;
    for (int sft = 1; sft <= kRefitSpan && L0 + sft < lv.n_levels; ++sft) {
        const int L = L0 + sft;
        const long long pfirst = first >> sft;                 /* this block's first parent at level L */
        const long long pend = ((first + kRefitNodes) >> sft) < lv.count[L] ? ((first + kRefitNodes) >> sft)
                                                                             : lv.count[L];
        const int np = (int)(pend - pfirst);
        for (int k = tid; k < np; k += kRefitThreads) {
            const long long pg = pfirst + k;
            const long long left = lv.start[L - 1] + 2 * pg;
            const bool has_right = 2 * pg + 1 < lv.count[L - 1];
            Box bx = src[2 * k];
            if (has_right) {
                expand_point(bx, src[2 * k + 1].mn);           /* AABB3f.expand_box, aabb.mojo:56-58 */
                expand_point(bx, src[2 * k + 1].mx);
            }
            store_node(nodes + lv.start[L] + pg, bx, (int)left, has_right ? (int)(left + 1) : -1);
            dst[k] = bx;
        }
        __syncthreads();
        /* ping-pong: the next level reads what this one wrote (an odd level
         * writes at most 512 parents, into the smaller buffer) */
        Box* t = src;
        src = dst;
        dst = t;
    }
}

struct RayState {
    float o[3], d[3], inv[3];
};

/* Vec3f.normalized, vector.mojo:106-110 */
__device__ __forceinline__ void normalize3(const float v[3], float out[3]) {
    const float l = sqrtf(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]);
    if (l > (float)0.000001) {
        out[0] = v[0] / l;
        out[1] = v[1] / l;
        out[2] = v[2] / l;
    } else {
        out[0] = out[1] = out[2] = 0.0f;
    }
}

/* AABB3f.intersect_ray, aabb.mojo:60-98 (the reciprocals are the same on
 * every call, so they are taken once per ray) */
__device__ __forceinline__ bool intersect(const float4& a, const float4& b, const RayState& r, float t_min,
                                          float t_max) {
    const float t1x = (a.x - r.o[0]) * r.inv[0], t2x = (b.x - r.o[0]) * r.inv[0];
    const float t1y = (a.y - r.o[1]) * r.inv[1], t2y = (b.y - r.o[1]) * r.inv[1];
    const float t1z = (a.z - r.o[2]) * r.inv[2], t2z = (b.z - r.o[2]) * r.inv[2];
    const float tx_min = fminf(t1x, t2x), tx_max = fmaxf(t1x, t2x);
    const float ty_min = fminf(t1y, t2y), ty_max = fmaxf(t1y, t2y);
    const float tz_min = fminf(t1z, t2z), tz_max = fmaxf(t1z, t2z);
    const float t_enter = fmaxf(fmaxf(tx_min, ty_min), tz_min);
    const float t_exit = fminf(fminf(tx_max, ty_max), tz_max);
    return !(t_enter > t_exit || t_exit < t_min || t_enter > t_max);
}

struct CastArgs {
    const LumenBvhNode* nodes;
    const int* splat_index;   /* n_leaves entries */
    long long node_count, root, n_gauss, n_leaves;
    const float* means;
    const float* scales;
    float max_dist;
};

/* The splat of leaf idx against the ray (raycast.mojo:62-88): whether it lies
 * within three radii, with the distance along the ray and the closest point. */
__device__ __forceinline__ bool leaf_hit(const CastArgs& A, const RayState& r, int idx, float limit, int* splat,
                                         float* t, float point[3]) {
    /* leaves are nodes [0, n_leaves) of a built hierarchy; a damaged one
     * cannot make the read leave the array */
    const int s = (long long)idx < A.n_leaves ? A.splat_index[idx] : -1;
    if (s < 0 || (long long)s >= A.n_gauss) return false;
    const float cx = A.means[(long long)s * 3], cy = A.means[(long long)s * 3 + 1], cz = A.means[(long long)s * 3 + 2];
    const float ocx = cx - r.o[0], ocy = cy - r.o[1], ocz = cz - r.o[2];
    const float t_proj = ocx * r.d[0] + ocy * r.d[1] + ocz * r.d[2];
    if (!(t_proj > 0.0f && t_proj <= limit)) return false;
    const float px = r.o[0] + r.d[0] * t_proj, py = r.o[1] + r.d[1] * t_proj, pz = r.o[2] + r.d[2] * t_proj;
    const float dx = px - cx, dy = py - cy, dz = pz - cz;
    const float dist = sqrtf(dx * dx + dy * dy + dz * dz);
    float rad = A.scales[(long long)s * 3];
    if (A.scales[(long long)s * 3 + 1] > rad) rad = A.scales[(long long)s * 3 + 1];
    if (A.scales[(long long)s * 3 + 2] > rad) rad = A.scales[(long long)s * 3 + 2];
    if (!(dist <= rad * 3.0f)) return false;
    *splat = s;
    *t = t_proj;
    point[0] = px;
    point[1] = py;
    point[2] = pz;
    return true;
}

__device__ __forceinline__ LumenRayHit no_hit(const CastArgs& A) {
    LumenRayHit h;
    h.hit = 0;
    h.splat_index = -1;
    h.point[0] = h.point[1] = h.point[2] = 0.0f;
    h.distance = A.node_count == 0 || A.root < 0 ? (float)1e9 : A.max_dist;
    return h;
}

__device__ __forceinline__ RayState ray_state(const float origin[3], const float dir[3]) {
    RayState r;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        r.o[c] = origin[c];
        r.d[c] = dir[c];
        r.inv[c] = 1.0f / (dir[c] != 0.0f ? dir[c] : (float)1e-6);
    }
    return r;
}

/* raycast_closest_splat, raycast.mojo:30-95, in the reference's own order:
 * depth first, the left child pushed before the right, so leaves are visited
 * in descending order, each against the closest hit so far. */
__device__ __forceinline__ LumenRayHit cast_ray_in_order(const CastArgs& A, const float origin[3], const float dir[3]) {
    LumenRayHit best = no_hit(A);
    if (A.node_count == 0 || A.root < 0) return best;
    const RayState r = ray_state(origin, dir);
    int stack[kRayStack];
    int sp = 0;
    stack[sp++] = (int)A.root;
    /* a built hierarchy visits each node at most once; the bound and the
     * index check keep a damaged one from looping or reading out of range */
    for (long long visits = 0; sp > 0 && visits <= A.node_count; ++visits) {
        const int idx = stack[--sp];
        if (idx < 0 || (long long)idx >= A.node_count) continue;
        const float4 a = __ldg(reinterpret_cast<const float4*>(A.nodes + idx));
        const float4 b = __ldg(reinterpret_cast<const float4*>(A.nodes + idx) + 1);
        if (!intersect(a, b, r, 0.0f, best.distance)) continue;
        const int left = __float_as_int(a.w), right = __float_as_int(b.w);
        if (left == -1 && right == -1) {
            int splat;
            float t, point[3];
            if (leaf_hit(A, r, idx, best.distance, &splat, &t, point) && t < best.distance) {
                best.hit = 1;
                best.splat_index = splat;
                best.distance = t;
                best.point[0] = point[0];
                best.point[1] = point[1];
                best.point[2] = point[2];
            }
        } else {
            /* at most levels + 1 entries: 32 below 2^30 leaves */
            if (left >= 0 && sp < kRayStack) stack[sp++] = left;
            if (right >= 0 && sp < kRayStack) stack[sp++] = right;
        }
    }
    return best;
}

/* A box test for the near-first cast: exactly intersect()'s decision on
 * t_enter > t_exit and t_exit < 0, and *t_near, a lower bound of t_enter and
 * of the distance of every hit inside the box, whatever the rounding of the
 * slab products (slack: the bound on a hit point's rounding error along an
 * axis, per unit of 1 / d). */
__device__ __forceinline__ bool box_ahead(const float4& a, const float4& b, const RayState& r, const float ainv[3],
                                          float slack, float* t_enter_out, float* t_near) {
    const float t1x = (a.x - r.o[0]) * r.inv[0], t2x = (b.x - r.o[0]) * r.inv[0];
    const float t1y = (a.y - r.o[1]) * r.inv[1], t2y = (b.y - r.o[1]) * r.inv[1];
    const float t1z = (a.z - r.o[2]) * r.inv[2], t2z = (b.z - r.o[2]) * r.inv[2];
    const float tx_min = fminf(t1x, t2x), tx_max = fmaxf(t1x, t2x);
    const float ty_min = fminf(t1y, t2y), ty_max = fmaxf(t1y, t2y);
    const float tz_min = fminf(t1z, t2z), tz_max = fmaxf(t1z, t2z);
    const float t_enter = fmaxf(fmaxf(tx_min, ty_min), tz_min);
    const float t_exit = fminf(fminf(tx_max, ty_max), tz_max);
    /* each axis' entry moved back by 2^-19 of the box's extent along it and
     * by the slack */
    constexpr float k = 1.0f / (1 << 19);
    const float nx = __fmaf_rn(-slack, ainv[0], __fmaf_rn(-k, tx_max - tx_min, tx_min));
    const float ny = __fmaf_rn(-slack, ainv[1], __fmaf_rn(-k, ty_max - ty_min, ty_min));
    const float nz = __fmaf_rn(-slack, ainv[2], __fmaf_rn(-k, tz_max - tz_min, tz_min));
    *t_enter_out = t_enter;
    *t_near = fmaxf(fmaxf(nx, ny), nz);
    return !(t_enter > t_exit || t_exit < 0.0f);
}

/* Eight lanes cast a ray together. Node i of level l of the built hierarchy
 * has the nodes 2^s i .. 2^s i + 2^s - 1 of level l - s below it, consecutive
 * in memory, so the hierarchy is walked three levels at a time: lane k of the
 * group loads and tests the k-th of the (up to) eight descendants, and the
 * group pushes those ahead of the best hit, the farthest first. */
constexpr int kCastLanes = 8;
constexpr int kCastThreads = 256;
constexpr int kCastStack = 80;   /* 7 left behind per three levels (2^30 leaves: 10 steps) and 8 new ones */

/* The levels' first nodes and sizes, in shared memory (indexed per group). */
struct CastLevels {
    int n_levels;
    unsigned int start[kMaxLevels], count[kMaxLevels];
};

__device__ __forceinline__ void copy_levels(CastLevels& s, const BvhLevels& lv) {
    if (threadIdx.x == 0) s.n_levels = lv.n_levels;
    if (threadIdx.x < kMaxLevels) {
        s.start[threadIdx.x] = (unsigned int)lv.start[threadIdx.x];   /* below 2^31 nodes */
        s.count[threadIdx.x] = (unsigned int)lv.count[threadIdx.x];
    }
    __syncthreads();
}

struct CastEntry {
    unsigned int node;   /* index within its level, and level / 3 in the top five bits */
    float t_near;
};

/* raycast_closest_splat with the nearest nodes first, which prunes most of
 * the tree once the first hits are found: the reference's order visits
 * leaves from the last to the first wherever they lie. Bound by the latency
 * of the node reads (a chain of about one 256-byte read per three levels), so
 * the lanes of a ray read their nodes side by side. 65 536 rays of a block of
 * pixels into 1 M Gaussians on a B200, over several places of the block: 4.2
 * to 6.1 ms in the reference's order with one thread per ray, 0.56 to 1.43
 * with the nearer child first, 0.37 to 0.83 with eight lanes per ray.
 *
 * The result is the reference's bit for bit, where the nodes are as the build
 * leaves them for the Gaussians as they are now (check_nodes_kernel). Their
 * boxes contain their children's, and float subtraction and multiplication are monotone,
 * so a leaf whose box passes has ancestors that pass. A leaf with a hit at
 * t_proj normally has t_enter <= t_proj (its box contains the hit point), and
 * then the reference keeps it exactly when t_proj is below the best so far:
 * its result is the least t_proj, and among equal ones the leaf that it
 * visits first, the one with the highest index, in whatever order the leaves
 * are taken here. Rounding can leave t_enter above t_proj when the ray
 * touches the sphere beside a face of the box; what the reference then does
 * depends on its order. Such a leaf is never pruned here before it is seen,
 * as t_near is below t_proj, and when one with t_proj up to the best so far
 * is seen, the whole ray is cast in the reference's order. So is a ray whose
 * origin or reciprocals are not ordinary numbers.
 *
 * Every lane of the group returns the hit, or false for a ray to be cast in
 * the reference's order. */
__device__ __forceinline__ bool cast_ray(const CastArgs& A, const CastLevels& lv, const float origin[3],
                                         const float dir[3], bool active, CastEntry* stack, LumenRayHit& best) {
    const int lane = threadIdx.x & 31, k = lane & (kCastLanes - 1), g0 = lane & ~(kCastLanes - 1);
    const unsigned int group = 0xFFu << g0;
    best = no_hit(A);
    const RayState r = ray_state(origin, dir);
    bool in_order = false;
    float ainv[3], far = 0.0f;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        ainv[c] = fabsf(r.inv[c]);
        far = fmaxf(far, fabsf(r.o[c]));
        if (!(ainv[c] < 1e30f && fabsf(r.o[c]) < 1e30f)) in_order = true;
    }
    active = active && !in_order;
    /* 2^-19 (|o| + t) bounds the rounding of a hit point at distance t
     * (three roundings of 2^-24 per coordinate) and of the box face beside
     * it, with room */
    constexpr float ulps = 1.0f / (1 << 19);
    float slack = ulps * (far + best.distance);
    int best_leaf = -1, sp = 0;
    int level = lv.n_levels - 1;
    unsigned int node = 0u;
    while (active) {
        const int below = level > 0 ? (level - 1) / 3 * 3 : 0;
        const unsigned int child = (node << (level - below)) + (unsigned int)k;
        bool pass = k < (1 << (level - below)) && child < lv.count[below];
        float te = INFINITY, tn = 0.0f;
        if (pass) {
            const LumenBvhNode* at = A.nodes + (lv.start[below] + child);
            const float4 a = __ldg(reinterpret_cast<const float4*>(at));
            const float4 b = __ldg(reinterpret_cast<const float4*>(at) + 1);
            pass = box_ahead(a, b, r, ainv, slack, &te, &tn) && !(tn > best.distance);
        }
        const unsigned int passed = (__ballot_sync(group, pass) >> g0) & 0xFFu;
        if (below != 0) {
            if (passed) {
                /* the descendants on the stack, the farthest lowest */
                int place = 0;
#pragma unroll
                for (int o = 1; o < kCastLanes; ++o) {
                    const float tj = __shfl_xor_sync(group, te, o);
                    place += ((passed >> (k ^ o)) & 1u) && (tj > te || (tj == te && (k ^ o) > k));
                }
                if (pass) stack[sp + place] = CastEntry{child | ((unsigned int)(below / 3) << 27), tn};
                sp += __popc(passed);
                __syncwarp(group);
            }
        } else if (passed) {
            float t = INFINITY, point[3];
            int splat = -1, leaf = (int)child;
            const bool hit = pass && leaf_hit(A, r, leaf, best.distance, &splat, &t, point);
            if (__any_sync(group, hit && !(te <= t))) {
                in_order = true;
                break;
            }
            if (!(hit && (t < best.distance || (best.hit && leaf > best_leaf)))) splat = -1;
            if (__any_sync(group, splat >= 0)) {
                /* the least t, and of equal ones the highest leaf */
#pragma unroll
                for (int o = 1; o < kCastLanes; o <<= 1) {
                    const float t2 = __shfl_xor_sync(group, t, o);
                    const int s2 = __shfl_xor_sync(group, splat, o), l2 = __shfl_xor_sync(group, leaf, o);
                    if (s2 >= 0 && (splat < 0 || t2 < t || (t2 == t && l2 > leaf))) {
                        t = t2;
                        splat = s2;
                        leaf = l2;
                    }
                }
                best.hit = 1;
                best.splat_index = splat;
                best.distance = t;
                best_leaf = leaf;
                slack = ulps * (far + t);
            }
        }
        active = false;
        while (sp > 0 && !active) {
            const CastEntry e = stack[--sp];
            active = !(e.t_near > best.distance);
            node = e.node & 0x7FFFFFFu;
            level = 3 * (int)(e.node >> 27);
        }
        __syncwarp(group);   /* the entry is read by all before its slot is written again */
    }
    if (best.hit) {
#pragma unroll
        for (int c = 0; c < 3; ++c) best.point[c] = r.o[c] + r.d[c] * best.distance;
    }
    return !in_order;
}

/* What cast_ray rests on is checked before every cast: the Gaussians may have
 * moved since the build, and the nodes are the caller's memory. Rays through
 * nodes that do not pass are cast in the reference's order, which follows the
 * links and the boxes whatever they hold. Nothing but the hits is at hand to
 * carry the finding to the cast, so a block that finds such a node marks every
 * hit record, unless a block before it has come to the last; the cast leaves
 * marked records alone (and marks those of rays that it gives up), and a pass
 * with a thread per ray casts their rays. A record that holds the mark by chance
 * only costs its ray the slower way; no hit looks like it. */
__device__ __forceinline__ uint4 in_order_mark() {
    return make_uint4(0x7A3C91E5u, 0x1D80F24Bu, 0xC5E76A03u, 0x3B9F58D2u);
}

__device__ __forceinline__ bool marked_in_order(const LumenRayHit* hit) {
    const unsigned int* w = reinterpret_cast<const unsigned int*>(hit);
    const uint4 m = in_order_mark();
    return w[0] == m.x && w[1] == m.y && w[2] == m.z && w[3] == m.w;
}

__device__ __forceinline__ void mark_in_order(LumenRayHit* hit) {
    unsigned int* w = reinterpret_cast<unsigned int*>(hit);
    const uint4 m = in_order_mark();
    w[0] = m.x;
    w[1] = m.y;
    w[2] = m.z;
    w[3] = m.w;
}

/* Whether node i is as the build leaves it: a leaf holds the box of its
 * Gaussian; a parent the links to its two children (or one) of the level
 * below, and a box that contains theirs. A NaN passes no comparison. */
__device__ __forceinline__ bool node_as_built(const CastArgs& A, const CastLevels& lv, long long i) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(A.nodes + i));
    const float4 b = __ldg(reinterpret_cast<const float4*>(A.nodes + i) + 1);
    const int left = __float_as_int(a.w), right = __float_as_int(b.w);
    if (i < A.n_leaves) {
        const int g = A.splat_index[i];
        if (g < 0 || (long long)g >= A.n_gauss) return false;
        const Box box = leaf_box(A.means, A.scales, g);
        return left == -1 && right == -1 && a.x == box.mn[0] && a.y == box.mn[1] && a.z == box.mn[2] &&
               b.x == box.mx[0] && b.y == box.mx[1] && b.z == box.mx[2];
    }
    int level = 1;
    while (level + 1 < lv.n_levels && i >= (long long)lv.start[level + 1]) ++level;
    const long long first = 2 * (i - (long long)lv.start[level]);
    const long long child = (long long)lv.start[level - 1] + first;
    const bool two = first + 1 < (long long)lv.count[level - 1];
    if ((long long)left != child || right != (two ? left + 1 : -1)) return false;
    for (int k = 0; k < (two ? 2 : 1); ++k) {
        const float4 c = __ldg(reinterpret_cast<const float4*>(A.nodes + child + k));
        const float4 d = __ldg(reinterpret_cast<const float4*>(A.nodes + child + k) + 1);
        if (!(a.x <= c.x && a.y <= c.y && a.z <= c.z && b.x >= d.x && b.y >= d.y && b.z >= d.z)) return false;
    }
    return true;
}

__global__ void __launch_bounds__(256)
check_nodes_kernel(CastArgs A, BvhLevels levels, LumenRayHit* __restrict__ hits, long long n_rays) {
    __shared__ CastLevels lv;
    copy_levels(lv, levels);
    const long long stride = (long long)gridDim.x * blockDim.x;
    int found = 0;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < A.node_count; i += stride)
        found |= !node_as_built(A, lv, i);
    if (!__syncthreads_or(found) || marked_in_order(hits + n_rays - 1)) return;
    for (long long i = threadIdx.x; i < n_rays; i += blockDim.x) mark_in_order(hits + i);
}

/* The rays of a cast: the caller's (kPick false), or those through pixels of
 * a view. */
struct RaySource {
    const LumenRay* rays;
    const float* pixels;
    LumenViewCamera cam;
};

struct CameraTurn {
    Quat q, qi;
};

template <bool kPick>
__device__ __forceinline__ CameraTurn camera_turn(const RaySource& src) {
    if (!kPick) return {};
    /* PinholeCamera keeps its rotation normalised (camera.mojo:37-40) */
    const Quat q = q_normalized({src.cam.rotation[0], src.cam.rotation[1], src.cam.rotation[2], src.cam.rotation[3]});
    return {q, q_inverse(q)};
}

template <bool kPick>
__device__ __forceinline__ LumenRay ray_of(const RaySource& src, const CameraTurn& turn, long long i) {
    LumenRay r;
    if (!kPick) {
        const LumenRay given = src.rays[i];
        r = given;
        normalize3(given.direction, r.direction);                                  /* Ray3f.__init__, camera.mojo:16-18 */
        return r;
    }
    /* generate_ray, camera.mojo:85-90 */
    const float v[3] = {(src.pixels[2 * i] - src.cam.cx) / src.cam.fx, (src.pixels[2 * i + 1] - src.cam.cy) / src.cam.fy,
                        1.0f};
    float dc[3];
    normalize3(v, dc);
    const Quat rq = q_mul(q_mul(turn.q, Quat{0.0f, dc[0], dc[1], dc[2]}), turn.qi);   /* rotate_vec, quaternion.mojo:80-87 */
    const float dw[3] = {rq.x, rq.y, rq.z};
    normalize3(dw, r.direction);                                                   /* Ray3f */
    r.origin[0] = src.cam.position[0];
    r.origin[1] = src.cam.position[1];
    r.origin[2] = src.cam.position[2];
    return r;
}

/* Eight lanes per ray; records that are marked, and those of rays that
 * cast_ray gives up, are left marked. */
template <bool kPick>
__global__ void __launch_bounds__(kCastThreads)
cast_kernel(CastArgs A, BvhLevels lv, RaySource src, long long n_rays, LumenRay* __restrict__ rays_out,
            LumenRayHit* __restrict__ hits) {
    __shared__ CastEntry stacks[kCastThreads / kCastLanes][kCastStack];
    __shared__ CastLevels levels;
    copy_levels(levels, lv);
    const int group = threadIdx.x / kCastLanes;
    const bool writes = (threadIdx.x & (kCastLanes - 1)) == 0;
    const CameraTurn turn = camera_turn<kPick>(src);
    const long long stride = (long long)gridDim.x * (kCastThreads / kCastLanes);
    /* warps stay whole: the last rays of a warp may be idle */
    for (long long i0 = (long long)blockIdx.x * (kCastThreads / kCastLanes) + (group & ~3); i0 < n_rays; i0 += stride) {
        const long long i = i0 + (group & 3);
        const bool active = i < n_rays;
        const LumenRay ray = ray_of<kPick>(src, turn, active ? i : i0);
        if (kPick && rays_out && writes && active) rays_out[i] = ray;
        const bool marked = active && marked_in_order(hits + i);
        LumenRayHit h;
        const bool done = cast_ray(A, levels, ray.origin, ray.direction, active && !marked, stacks[group], h);
        __syncwarp();   /* the mark is read by all before the record is written */
        if (active && !marked && writes) {
            if (done) hits[i] = h;
            else mark_in_order(hits + i);
        }
    }
}

/* One thread per ray, in the reference's order: all rays, or those of marked
 * records. */
constexpr int kInOrderThreads = 128;

template <bool kPick>
__global__ void __launch_bounds__(kInOrderThreads)
cast_in_order_kernel(CastArgs A, RaySource src, long long n_rays, bool all, LumenRay* __restrict__ rays_out,
                     LumenRayHit* __restrict__ hits) {
    const CameraTurn turn = camera_turn<kPick>(src);
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_rays; i += stride) {
        if (!all && !marked_in_order(hits + i)) continue;
        const LumenRay ray = ray_of<kPick>(src, turn, i);
        if (kPick && all && rays_out) rays_out[i] = ray;
        hits[i] = cast_ray_in_order(A, ray.origin, ray.direction);
    }
}

unsigned int cast_grid(long long n, long long per_block, long long per_sm) {
    long long g = (n + per_block - 1) / per_block;
    const long long cap = (long long)device_sm_count() * per_sm;
    if (g > cap) g = cap;
    return (unsigned int)(g < 1 ? 1 : g);
}

/* A thread per ray in the reference's order at once, without the check and the
 * second pass, where there is little to prune: into 256 Gaussians at most
 * (300 of a box: both 46 us, whatever the rays), and with many rays, where the
 * eight lanes are bound by instructions, into some thousands: 65 536 rays into
 * 2000 (4000, 8000) Gaussians 88 (121, 183) us against 136 (152, 157), 2 M rays 612
 * (892, 1379) against 1540 (1689, 1893). With fewer rays the eight lanes are as
 * fast or faster (16 384 into 2000: 64 us against 74; one ray into 1 M: 149
 * against 967, of which the check takes 35). A cast from a node other than the
 * root follows the links. */
bool casts_in_order(const CastArgs& A, long long n_rays) {
    return A.root != A.node_count - 1 || A.n_leaves <= 256 ||
           (n_rays > 32768 && A.n_leaves <= (n_rays > 131072 ? 8192 : 4096));
}

template <bool kPick>
LumenStatus cast(const CastArgs& A, const RaySource& src, long long n_rays, LumenRay* rays_out, LumenRayHit* hits,
                 cudaStream_t s) {
    const bool in_order = casts_in_order(A, n_rays);
    if (!in_order) {
        const BvhLevels lv = make_levels(A.n_leaves);
        check_nodes_kernel<<<cast_grid(A.node_count, 256, 8), 256, 0, s>>>(A, lv, hits, n_rays);
        cast_kernel<kPick><<<cast_grid(n_rays, kCastThreads / kCastLanes, 64), kCastThreads, 0, s>>>(A, lv, src, n_rays,
                                                                                                  rays_out, hits);
    }
    cast_in_order_kernel<kPick><<<cast_grid(n_rays, kInOrderThreads, 16), kInOrderThreads, 0, s>>>(
        A, src, n_rays, in_order, rays_out, hits);
    return map_cuda(cudaGetLastError());
}

bool bvh_ok(const LumenGpuBvh* b, const LumenGpuGaussians* g) {
    if (!b || !g || b->leaf_count < 0 || b->leaf_count >= (1ll << 30) || b->leaf_count != g->count) return false;
    if (b->node_count != node_count_of(b->leaf_count)) return false;
    if (b->node_count > 0 && (!b->nodes || !b->splat_index || !g->means || !g->scales)) return false;
    if (((uintptr_t)b->nodes) & 15u) return false;
    return true;
}

}  // namespace
}  // namespace lumen

using namespace lumen;

extern "C" {

int64_t lumen_bvh_node_count(int64_t n) { return node_count_of(n); }

size_t lumen_gpu_bvh_scratch_bytes(int64_t n) { return n < 0 ? 0 : make_layout(n).total; }

LumenStatus lumen_gpu_bvh_build(const LumenGpuGaussians* g, LumenGpuBvh* bvh, void* scratch, size_t scratch_bytes,
                                void* stream) {
    if (!g || !bvh || g->count < 0 || g->count >= (1ll << 30)) return LUMEN_ERROR_INVALID_ARGUMENT;
    const long long n = g->count;
    if (n == 0) {
        bvh->leaf_count = 0;
        bvh->node_count = 0;
        bvh->root_index = -1;
        return LUMEN_SUCCESS;
    }
    if (!g->means || !g->scales || !bvh->nodes || !bvh->splat_index || !scratch) return LUMEN_ERROR_INVALID_ARGUMENT;
    if (((uintptr_t)bvh->nodes | (uintptr_t)scratch) & 15u) return LUMEN_ERROR_INVALID_ARGUMENT;
    const BvhLayout B = make_layout(n);
    if (scratch_bytes < B.total) return LUMEN_ERROR_INVALID_ARGUMENT;
    const BvhLevels lv = make_levels(n);
    configure_once();
    cudaStream_t s = (cudaStream_t)stream;
    unsigned char* base = (unsigned char*)scratch;
    BvhControl* ctrl = (BvhControl*)(base + B.control_off);
    unsigned int* k0 = (unsigned int*)(base + B.keys0_off);
    unsigned int* v0 = (unsigned int*)(base + B.vals0_off);
    unsigned int* k1 = (unsigned int*)(base + B.keys1_off);
    unsigned int* v1 = (unsigned int*)(base + B.vals1_off);
    unsigned int* lb = (unsigned int*)(base + B.lb_off);
    cudaError_t e = cudaMemsetAsync(base, 0, B.zeroed(), s);
    if (e != cudaSuccess) return map_cuda(e);
    const int sms = device_sm_count();
    long long grid = (n + 255) / 256;
    if (grid > (long long)sms * 8) grid = (long long)sms * 8;
    bbox_kernel<<<(unsigned int)grid, 256, 0, s>>>(g->means, n, ctrl);
    morton_kernel<<<(unsigned int)grid, 256, 0, s>>>(g->means, n, ctrl, k0, v0);
    /* 2048-key tiles while 4096-key ones would leave SMs idle */
    const int items = n <= 3ll * sms * kSortTile ? 8 : 16;
    launch_sort32(k0, v0, k1, v1, n, &ctrl->sort, lb, B.sort_tiles, &ctrl->error_flags, items, 4, sms, s);
    for (int L0 = 0; L0 + 1 < lv.n_levels; L0 += kRefitSpan) {
        const long long blocks = (lv.count[L0] + kRefitNodes - 1) / kRefitNodes;
        bvh_levels_kernel<<<(unsigned int)blocks, kRefitThreads, 0, s>>>(g->means, g->scales, n, ctrl, v0, v1,
                                                                         bvh->nodes, bvh->splat_index, lv, L0);
    }
    if (lv.n_levels == 1)   /* a single leaf: the kernel writes it without climbing */
        bvh_levels_kernel<<<1, kRefitThreads, 0, s>>>(g->means, g->scales, n, ctrl, v0, v1, bvh->nodes,
                                                      bvh->splat_index, lv, 0);
    if ((e = cudaGetLastError()) != cudaSuccess) return map_cuda(e);
    unsigned int h_flags = 0;
    e = cudaMemcpyAsync(&h_flags, &ctrl->error_flags, sizeof(h_flags), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return map_cuda(e);
    bvh->leaf_count = n;
    bvh->node_count = node_count_of(n);
    bvh->root_index = bvh->node_count - 1;
    return status_from_flags(h_flags);
}

LumenStatus lumen_gpu_raycast(const LumenGpuBvh* bvh, const LumenGpuGaussians* g, const LumenRay* rays,
                              int64_t n_rays, float max_dist, LumenRayHit* hits, void* stream) {
    if (!bvh_ok(bvh, g) || n_rays < 0) return LUMEN_ERROR_INVALID_ARGUMENT;
    if (n_rays == 0) return LUMEN_SUCCESS;
    if (!rays || !hits) return LUMEN_ERROR_INVALID_ARGUMENT;
    const CastArgs A{bvh->nodes, bvh->splat_index, bvh->node_count, bvh->root_index, g->count, bvh->leaf_count,
                     g->means, g->scales, max_dist};
    return cast<false>(A, RaySource{rays, nullptr, {}}, n_rays, nullptr, hits, (cudaStream_t)stream);
}

LumenStatus lumen_gpu_pick_pixels(const LumenGpuBvh* bvh, const LumenGpuGaussians* g, const LumenViewCamera* cam,
                                  const float* pixels_xy, int64_t n, float max_dist, LumenRay* rays,
                                  LumenRayHit* hits, void* stream) {
    if (!bvh_ok(bvh, g) || !cam || n < 0) return LUMEN_ERROR_INVALID_ARGUMENT;
    if (n == 0) return LUMEN_SUCCESS;
    if (!pixels_xy || !hits) return LUMEN_ERROR_INVALID_ARGUMENT;
    const CastArgs A{bvh->nodes, bvh->splat_index, bvh->node_count, bvh->root_index, g->count, bvh->leaf_count,
                     g->means, g->scales, max_dist};
    return cast<true>(A, RaySource{nullptr, pixels_xy, *cam}, n, rays, hits, (cudaStream_t)stream);
}

}  // extern "C"
