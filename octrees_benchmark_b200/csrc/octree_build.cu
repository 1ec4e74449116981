// Linear-octree build over the SFC-sorted keys.
//
// Reference path replaced: LinearOctree::buildOctree (inc/structures/linear_octree.hpp:
// 567-605): the cornerstone leaf iteration (buildOctreeLeaves 458-471 with
// rebalanceDecision / calculateNodeOp / processNode / computeNodeCounts), then
// createUnsortedLayout, a sort of the Warren-Salmon prefixes, linkTree,
// computeInternalRanges and computeGeometry (336-565).
//
// Why a top-down construction gives the same arrays.  In the reference's
// iteration a leaf is split when its count exceeds maxPointsLeaf (and level <
// 21) and 8 sibling leaves merge when their summed count is <= maxPointsLeaf.
// Starting from the root, every split node had count > maxPointsLeaf, so its
// 8 children always sum above it and no merge ever fires: the converged tree
// is exactly "split every node with more than maxPointsLeaf points, down to
// level 21".  Sorting the nodes by their placeholder-bit prefix (1 followed by
// the 3*level key bits) orders them level by level and, inside a level, by key:
// breadth-first order.  So the node of child c of the j-th internal node of
// level l sits at level_start[l+1] + 8 j + c, and offsets[] of the k-th
// internal node of level l+1 is level_start[l+2] + 8 k.  internalRanges of a
// node are the lower_bounds of its start and end key in the sorted keys, and
// its centre is PointEncoder::getCenter of its start key.
//
// Kernels: every level at once.  The sorted keys alone say which nodes split: the
// octant of level l that holds key i has more than M = maxPointsLeaf points past
// i's first if key i + M still lies in it, so with e the level to which key i
// shares its octant with key i - 1 and d (at most 20) that to which it shares it
// with key i + M, the split nodes whose first point is i are those of levels e + 1
// to d.  Their number per level and block of keys (k_level_count), its scan over
// the blocks (k_level_scan) and their order inside a block give every split node
// its rank in its level, and so the place of its 8 children (k_level_list);
// k_level_children finds the children's ranges by search from i on, 8 lanes a
// node.  No level waits for another, as it did for a grid barrier and a dependent
// search each when one cooperative launch went down level by level.
//
// Bound: latency below ~1M points (four launches of 3 to 12 us), above that the
// two reads of the keys and the sectors of the searches.  Device time, level by
// level -> now: 20k points (Hilbert, leaf 32) 61 -> 28 us, 1M (Morton, leaf 128)
// 113 -> 30, 10M (Hilbert, leaf 64) 194 -> 132 (count 30, scan 7, list 41, children
// 53; with the children searched by the warp that found their node 236 in all).
#include "cloud.h"
#include "sfc.cuh"

namespace octb {

namespace {

constexpr int kLvWarps = 8;
constexpr int kLvThreads = 32 * kLvWarps;
constexpr int kLvRows = 8;                           // rows of 32 keys a warp takes
constexpr uint32_t kLvTile = kLvThreads * kLvRows;   // keys of a block
constexpr int kSplitLevels = (int)kMaxDepth;         // levels 0 .. 20 can split

struct BoxGeom {
    BoxD box;
    LevelGeom geom;
};

// lower_bound over [lo, hi).  Ranges longer than kKaryMin are
// first narrowed kKaryWays-fold per step by kKaryWays - 1 independent probes
// (one round trip each step instead of log2(kKaryWays) dependent ones: the top
// levels' searches span millions of keys), then bisected.
constexpr uint32_t kKaryWays = 8;
constexpr uint32_t kKaryMin = 32;
static_assert(kKaryMin >= kKaryWays, "a k-ary step needs a stride of at least one key");

__device__ __forceinline__ uint32_t lower_bound_keys(const uint64_t* __restrict__ keys, uint32_t lo, uint32_t hi,
                                                     uint64_t v) {
    while (hi - lo > kKaryMin) {
        // keys [lo, hi) ascending; the answer lies in [lo, hi]
        const uint32_t s = (hi - lo) / kKaryWays;
        uint32_t below = 0;  // probes lo + p s (p = 1 .. ways - 1) under v: a prefix of them
#pragma unroll
        for (uint32_t p = 1; p < kKaryWays; ++p) below += keys[lo + p * s] < v ? 1u : 0u;
        const uint32_t nlo = below ? lo + below * s + 1 : lo;
        if (below < kKaryWays - 1) hi = lo + (below + 1) * s;
        lo = nlo;
    }
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (keys[mid] < v) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Levels to which two keys share their octant (0 .. 21).
__device__ __forceinline__ int shared_levels(uint64_t a, uint64_t b) {
    const uint64_t x = a ^ b;
    if (x == 0) return (int)kMaxDepth;
    const int top = 63 - __clzll((long long)x);  // a key has 63 bits
    return top >= 62 ? 0 : (62 - top) / 3;
}

// e and d of key i: the nodes of levels e + 1 .. d split and begin with it (none when d <= e).
__device__ __forceinline__ void split_levels(uint64_t prev, uint64_t key, uint64_t far, bool first, bool reaches,
                                             int& e, int& d) {
    e = first ? -1 : shared_levels(prev, key);
    d = reaches ? min(shared_levels(key, far), kSplitLevels - 1) : -1;
}

// Per block of keys and level, the split nodes that begin in it (counts[level * blocks + block]); per warp, the
// rows that begin any.  A key whose difference to key i + M is above that to key i - 1 begins none, so few keys
// get to their levels: two reads of the keys bound this kernel.
__global__ void __launch_bounds__(kLvThreads) k_level_count(const uint64_t* __restrict__ keys, uint64_t n, uint32_t M,
                                                            uint32_t* __restrict__ counts, uint8_t* __restrict__ rows) {
    __shared__ uint32_t s_cnt[kLvWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t base = (uint64_t)blockIdx.x * kLvTile + (uint64_t)warp * (32 * kLvRows) + lane;
    uint64_t key[kLvRows], far[kLvRows];
#pragma unroll
    for (int r = 0; r < kLvRows; ++r) {
        const uint64_t i = base + 32 * r;
        key[r] = i < n ? keys[i] : 0ull;
        far[r] = i + M < n ? keys[i + M] : 0ull;
    }
    uint64_t before = lane == 0 && base > 0 && base < n ? keys[base - 1] : 0ull;  // lane 0: the key before the row
    uint32_t mine = 0, any = 0;  // lane l: split nodes of level l
#pragma unroll
    for (int r = 0; r < kLvRows; ++r) {
        const uint64_t i = base + 32 * r;
        uint64_t prev = __shfl_up_sync(0xffffffffu, key[r], 1);
        if (lane == 0) prev = before;
        before = __shfl_sync(0xffffffffu, key[r], 31);
        const bool reaches = i + M < n;
        if (!__any_sync(0xffffffffu, reaches && (i == 0 || (key[r] ^ far[r]) < (prev ^ key[r])))) continue;
        int e, d;
        split_levels(prev, key[r], far[r], i == 0, reaches, e, d);
        const bool has = d > e;
        if (!__any_sync(0xffffffffu, has)) continue;
        any |= 1u << r;
        const int lo = __reduce_min_sync(0xffffffffu, has ? e + 1 : kSplitLevels);
        const int hi = __reduce_max_sync(0xffffffffu, has ? d : -1);
#pragma unroll 1
        for (int l = lo; l <= hi; ++l) {
            const uint32_t m = __ballot_sync(0xffffffffu, e < l && l <= d);
            if (lane == l) mine += __popc(m);
        }
    }
    s_cnt[warp][lane] = mine;
    if (lane == 0) rows[(uint64_t)blockIdx.x * kLvWarps + warp] = (uint8_t)any;
    __syncthreads();
    if (threadIdx.x < kSplitLevels) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < kLvWarps; ++w) c += s_cnt[w][threadIdx.x];
        counts[(uint64_t)threadIdx.x * gridDim.x + blockIdx.x] = c;
    }
}

// One block per level: its counts become exclusive prefixes over the blocks, its total goes to level_internal.
__global__ void __launch_bounds__(1024) k_level_scan(uint32_t* __restrict__ counts, uint32_t blocks, BuildCtl* ctl) {
    __shared__ uint32_t s_sum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t* c = counts + (uint64_t)blockIdx.x * blocks;
    uint32_t carry = 0;
    for (uint32_t b = 0; b < blocks; b += 1024) {
        const uint32_t v = b + tid < blocks ? c[b + tid] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, off);
            if (lane >= off) x += y;
        }
        if (lane == 31) s_sum[warp] = x;
        __syncthreads();
        uint32_t w = s_sum[lane];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        const uint32_t before = warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0u;
        if (b + tid < blocks) c[b + tid] = carry + before + x - v;
        carry += __shfl_sync(0xffffffffu, w, 31);
        __syncthreads();
    }
    if (tid == 0) ctl->level_internal[blockIdx.x] = carry;
}

// Where the levels begin, from the split nodes of each: the first node of level l (start[l]) and the split nodes
// of the levels before it (split[l]).  One warp; returns the nodes of the tree.
__device__ __forceinline__ unsigned long long level_table(const BuildCtl* ctl, uint32_t* start, uint32_t* split) {
    const int lane = threadIdx.x & 31;
    const uint32_t c = lane < kSplitLevels ? ctl->level_internal[lane] : 0u;
    unsigned long long x = c;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    const unsigned long long all = __shfl_sync(0xffffffffu, x, 31);
    if (lane == 0) start[0] = 0;
    if (lane < kSplitLevels) {
        start[lane + 1] = (uint32_t)(1 + 8 * (x - c));
        split[lane] = (uint32_t)(x - c);
    }
    if (lane == kSplitLevels) split[lane] = (uint32_t)all;
    return 1 + 8 * all;
}

// Every split node, in the order of the nodes: its first point and its own place (x, y of list[]).
__global__ void __launch_bounds__(kLvThreads) k_level_list(const uint64_t* __restrict__ keys, uint64_t n, uint32_t M,
                                                           const uint32_t* __restrict__ counts,
                                                           const uint8_t* __restrict__ rows, uint2* __restrict__ list,
                                                           uint32_t node_cap, BuildCtl* ctl, uint32_t* err) {
    __shared__ uint32_t s_start[kMaxDepth + 2], s_split[kMaxDepth + 2];
    __shared__ unsigned long long s_total;
    __shared__ uint32_t s_cnt[kLvWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        const unsigned long long total = level_table(ctl, s_start, s_split);
        const uint32_t used = __ballot_sync(0xffffffffu, lane < kSplitLevels && ctl->level_internal[lane] != 0);
        if (lane == 0) {
            s_total = total;
            if (blockIdx.x == 0) {
                if (total > node_cap) {
                    ctl->need_nodes = (uint32_t)(total < 0xffffffffull ? total : 0xffffffffull);
                    set_err(err, kErrNodeCapacity);
                } else {
                    ctl->n_total = (uint32_t)total;
                    ctl->n_internal = (uint32_t)(total / 8);
                    ctl->max_depth_seen = 32 - __clz(used);  // the deepest split level + 1
                }
            }
        }
    }
    // split nodes per level of the warp's rows, and of those before them
    const uint64_t base = (uint64_t)blockIdx.x * kLvTile + (uint64_t)warp * (32 * kLvRows) + lane;
    const uint32_t any = base - lane < n ? rows[(uint64_t)blockIdx.x * kLvWarps + warp] : 0u;
    auto levels = [&](int r, uint64_t& key, int& e, int& d) {
        const uint64_t i = base + 32 * r;
        key = i < n ? keys[i] : 0ull;
        const uint64_t far = i + M < n ? keys[i + M] : 0ull;
        uint64_t prev = __shfl_up_sync(0xffffffffu, key, 1);
        if (lane == 0 && i > 0 && i < n) prev = keys[i - 1];
        split_levels(prev, key, far, i == 0, i + M < n, e, d);
    };
    uint32_t mine = 0;
#pragma unroll 1
    for (uint32_t rem = any; rem; rem &= rem - 1) {
        uint64_t key;
        int e, d;
        levels(__ffs(rem) - 1, key, e, d);
        const bool has = d > e;
        const int lo = __reduce_min_sync(0xffffffffu, has ? e + 1 : kSplitLevels);
        const int hi = __reduce_max_sync(0xffffffffu, has ? d : -1);
#pragma unroll 1
        for (int l = lo; l <= hi; ++l) {
            const uint32_t m = __ballot_sync(0xffffffffu, e < l && l <= d);
            if (lane == l) mine += __popc(m);
        }
    }
    s_cnt[warp][lane] = mine;
    __syncthreads();
    if (!any || s_total > node_cap) return;  // (the host grows the node arrays and runs again)
    uint32_t pre = lane < kSplitLevels ? counts[(uint64_t)lane * gridDim.x + blockIdx.x] : 0u;
    for (int w = 0; w < warp; ++w) pre += s_cnt[w][lane];
#pragma unroll 1
    for (uint32_t rem = any; rem; rem &= rem - 1) {
        const int r = __ffs(rem) - 1;
        uint64_t key;
        int e, d;
        levels(r, key, e, d);
        const bool has = d > e;
        const int lo = __reduce_min_sync(0xffffffffu, has ? e + 1 : kSplitLevels);
        const int hi = __reduce_max_sync(0xffffffffu, has ? d : -1);
        // the level above: its split nodes before the row, and those of the row up to the lane
        uint32_t up = lo > 0 ? __shfl_sync(0xffffffffu, pre, lo - 1) : 0u;
#pragma unroll 1
        for (int l = lo; l <= hi; ++l) {
            const bool begins = e < l && l <= d;
            const uint32_t m = __ballot_sync(0xffffffffu, begins);
            const uint32_t at = __shfl_sync(0xffffffffu, pre, l) + __popc(m & lanemask_lt());
            if (begins) {
                // child `digit` of the last split node of the level above that begins at or before the key
                const uint32_t digit = (uint32_t)((key >> (3 * (kMaxDepth - l))) & 7u);
                const uint32_t node = l ? s_start[l] + 8u * (up - 1u) + digit : 0u;
                list[s_split[l] + at] = make_uint2((uint32_t)(base + 32 * r), node);
            }
            up = at + (begins ? 1u : 0u);
            if (lane == l) pre += __popc(m);
        }
    }
}

// The children of every split node, 8 lanes a node.
template <int ENC>
__global__ void __launch_bounds__(kLvThreads) k_level_children(const uint64_t* __restrict__ keys, uint64_t n,
                                                               uint32_t M, const BoxGeom* __restrict__ bgp,
                                                               const uint2* __restrict__ list,
                                                               uint32_t* __restrict__ offsets,
                                                               uint2* __restrict__ ranges,
                                                               double* __restrict__ centers, uint32_t node_cap,
                                                               const BuildCtl* __restrict__ ctl) {
    __shared__ BoxGeom bg;
    __shared__ uint32_t s_start[kMaxDepth + 2], s_split[kMaxDepth + 2];
    __shared__ unsigned long long s_total;
    for (uint32_t t = threadIdx.x; t < sizeof(BoxGeom) / 8; t += kLvThreads)
        reinterpret_cast<double*>(&bg)[t] = reinterpret_cast<const double*>(bgp)[t];
    if (threadIdx.x < 32) {
        const unsigned long long total = level_table(ctl, s_start, s_split);
        if (threadIdx.x == 0) s_total = total;
    }
    __syncthreads();
    if (s_total > node_cap) return;
    const uint32_t total = (uint32_t)s_total, splits = total / 8;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        double c[3];
        node_center<ENC>(0ull, 0, bg.box, bg.geom, c);
        centers[0] = c[0];
        centers[1] = c[1];
        centers[2] = c[2];
        ranges[0] = make_uint2(0u, (uint32_t)n);
        if (splits == 0) offsets[0] = 0u;
    }
    const int c = threadIdx.x & 7;
    const uint32_t stride = gridDim.x * (kLvThreads / 8);
    const uint32_t rounds = (splits + stride - 1) / stride;  // whole warps: the lanes of a node shuffle
    uint32_t t = blockIdx.x * (kLvThreads / 8) + (threadIdx.x >> 3);
#pragma unroll 1
    for (uint32_t round = 0; round < rounds; ++round, t += stride) {
        const bool on = t < splits;
        const uint2 me = on ? list[t] : make_uint2(0u, 0u);
        const uint32_t first = me.x;
        int l = 0;  // the last level that begins at or before t
#pragma unroll
        for (int b = 16; b > 0; b >>= 1)
            if (l + b < kSplitLevels && s_split[l + b] <= t) l += b;
        const uint64_t key = on ? keys[first] : 0ull;
        const uint64_t step = node_range(l + 1);
        const uint64_t start = key & ~(8ull * step - 1ull);
        // where child c ends
        const uint64_t v = start + (uint64_t)(c + 1) * step;
        uint32_t end = first;
        if (on && key < v) {
            // the first few levels' nodes are a large part of the keys; else a bracket first: seven doublings
            // of M / 8 keys at once, as most split nodes hold up to 8 M
            uint64_t lo = (uint64_t)first + 1, hi = n;
            if (l > 4) {
                uint64_t at = first, s = M / 8 + 1;
#pragma unroll 1
                for (;;) {
                    uint32_t below = 0;
#pragma unroll
                    for (int q = 0; q < 7; ++q) below += at + (s << q) < n && keys[at + (s << q)] < v ? 1u : 0u;
                    if (below) lo = at + (s << (below - 1)) + 1;
                    if (below < 7) {
                        hi = min(n, at + (s << below));
                        break;
                    }
                    at += s << 6;
                    s <<= 6;
                }
            }
            end = lower_bound_keys(keys, (uint32_t)lo, (uint32_t)hi, v);
        }
        const uint32_t prev = __shfl_up_sync(0xffffffffu, end, 1);
        if (!on) continue;
        const uint32_t child = s_start[l + 1] + 8u * (t - s_split[l]) + c;
        const uint32_t begin = c ? prev : first;
        double cc[3];
        node_center<ENC>(start + (uint64_t)c * step, l + 1, bg.box, bg.geom, cc);
        ranges[child] = make_uint2(begin, end);
        centers[3ull * child] = cc[0];
        centers[3ull * child + 1] = cc[1];
        centers[3ull * child + 2] = cc[2];
        // a child that splits is in the list itself, and gets its link there
        if (!(end - begin > M && l + 1 < kSplitLevels)) offsets[child] = 0u;
        if (c == 0 && me.y < total) offsets[me.y] = child;
    }
}

int sm_count_b(int device) {
    int v = 148;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
    return v;
}

}  // namespace

cudaError_t launch_build(Cloud& c, bool* capacity_ok) {
    cudaError_t e;
    *capacity_ok = true;
    const uint64_t n = c.n;
    const uint32_t M = c.params.max_points_leaf;
    if (c.node_capacity == 0) {
        // nodes = 1 + 8 * internal; a level holds at most n / (M + 1) internal nodes
        const uint64_t per_level = n / ((uint64_t)M + 1) + 1;
        uint64_t cap = 8 * 3 * per_level + 9;
        if (cap > 0xfffffff0ull) cap = 0xfffffff0ull;
        c.node_capacity = (uint32_t)cap;
    }
    const uint64_t cap = c.node_capacity;
    const uint32_t blocks = (uint32_t)(n ? (n + kLvTile - 1) / kLvTile : 1);
    if ((e = c.offsets.reserve(4 * (cap + 1))) != cudaSuccess) return e;
    if ((e = c.ranges.reserve(8 * cap)) != cudaSuccess) return e;
    if ((e = c.centers.reserve(24 * cap)) != cudaSuccess) return e;
    if ((e = c.lv_counts.reserve(4ull * kSplitLevels * blocks)) != cudaSuccess) return e;
    if ((e = c.lv_rows.reserve((uint64_t)kLvWarps * blocks)) != cudaSuccess) return e;
    if ((e = c.lv_list.reserve(sizeof(uint2) * (cap / 8 + 1))) != cudaSuccess) return e;
    if ((e = c.d_build.reserve(sizeof(BuildCtl))) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(c.d_build.ptr, 0, sizeof(BuildCtl), c.stream)) != cudaSuccess) return e;
    const uint64_t* keys = c.keys.as<uint64_t>();
    uint32_t* counts = c.lv_counts.as<uint32_t>();
    uint8_t* rows = c.lv_rows.as<uint8_t>();
    BuildCtl* ctl = c.d_build.as<BuildCtl>();
    uint2* list = c.lv_list.as<uint2>();
    const uint64_t most = cap / 8 + 1;  // split nodes
    const uint64_t want = (8 * most + kLvThreads - 1) / kLvThreads;
    const uint64_t full = (uint64_t)sm_count_b(c.device) * 8;
    const unsigned grid = (unsigned)(want < full ? want : full);
    k_level_count<<<blocks, kLvThreads, 0, c.stream>>>(keys, n, M, counts, rows);
    k_level_scan<<<kSplitLevels, 1024, 0, c.stream>>>(counts, blocks, ctl);
    k_level_list<<<blocks, kLvThreads, 0, c.stream>>>(keys, n, M, counts, rows, list, (uint32_t)cap, ctl,
                                                      c.d_err.as<uint32_t>());
    auto children = c.params.encoder == OCT_ENC_HILBERT_3D ? k_level_children<5> : k_level_children<1>;
    children<<<grid, kLvThreads, 0, c.stream>>>(keys, n, M, c.d_box.as<BoxGeom>(), list, c.offsets.as<uint32_t>(),
                                                c.ranges.as<uint2>(), c.centers.as<double>(), (uint32_t)cap, ctl);
    return cudaGetLastError();
}

// A kernel of this file's device code, for preload_kernels.
const void* kernel_anchor_octree_build() { return reinterpret_cast<const void*>(&k_level_children<1>); }

}  // namespace octb
