// k nearest neighbours over the linear octree.
//
// Reference path replaced: LinearOctree::knn (inc/structures/linear_octree.hpp:
// 899-942), a best-first search over one heap of octants (keyed by the
// clamp-to-box distance, distPointOctantSquared 854-878) and points (keyed by
// distPointsSquared 844-851) that stops after min(n, k) points.
//
// B200 design: one warp per query walks the tree depth-first, nearest child
// first (children of a node are judged on 8 lanes and ordered by their
// lower bound), and prunes every octant whose lower bound exceeds the current
// k-th distance.  The k best (squared distance, index) pairs live in a sorted
// list in shared memory; leaf points that beat the k-th pair are appended to a
// candidate buffer with a ballot, and a full buffer is sorted (descending) and
// bitonic-merged into the list.  All distances are the reference's FP64 expressions, so the
// returned squared distances are bitwise the reference's, and ordering by
// (distance, index) resolves ties at the k-th distance by the lowest index.
#include <algorithm>
#include <cfloat>

#include "cloud.h"
#include "search_kernels.cuh"

namespace octb {

namespace {

constexpr int kKnnWarps = 4;
constexpr int kKnnThreads = 32 * kKnnWarps;
constexpr int kKnnStack = 8 * (kMaxDepth + 1);

struct KnnArgs {
    const double* xs;
    const double* ys;
    const double* zs;
    const uint32_t* offsets;
    const uint2* ranges;
    const double* centers;
    const LevelGeom* geom;
    const double* q;
    uint64_t nq;
    uint32_t k;
    uint32_t* idx;
    double* d2;
    uint32_t* counts;
    uint32_t* err;
    const uint32_t* order;  // query visiting order (curve order), or nullptr
    uint32_t bucket;        // subtrees with at most this many points are scanned as one range
    const DynGroup* grp;    // table launch (k_knn<LCAP, true>): sizes and requests on the device
    const unsigned long long* nq_dev;  // the query count in device memory (else nq)
};

__device__ __forceinline__ bool pair_less(double da, uint32_t ia, double db, uint32_t ib) {
    return (da < db) || (da == db && ia < ib);
}

// Bitonic sort of N (power of two) pairs in shared memory into descending order, one warp.
template <int N>
__device__ __forceinline__ void warp_bitonic_sort_desc(double* d, uint32_t* ix) {
    const int lane = threadIdx.x & 31;
    for (int size = 2; size <= N; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            for (int i = lane; i < N / 2; i += 32) {
                const int lo = ((i & ~(stride - 1)) << 1) | (i & (stride - 1));
                const int hi = lo + stride;
                const bool asc = (lo & size) != 0;  // mirrored network: the last stage runs descending
                const double a = d[lo], b = d[hi];
                const uint32_t ia = ix[lo], ib = ix[hi];
                const bool swap = asc ? pair_less(b, ib, a, ia) : pair_less(a, ia, b, ib);
                if (swap) {
                    d[lo] = b; d[hi] = a;
                    ix[lo] = ib; ix[hi] = ia;
                }
            }
            __syncwarp();
        }
    }
}

// A bitonic sequence of N (power of two) pairs into ascending order, one warp.
template <int N>
__device__ __forceinline__ void warp_bitonic_merge(double* d, uint32_t* ix) {
    const int lane = threadIdx.x & 31;
    for (int stride = N >> 1; stride > 0; stride >>= 1) {
        for (int i = lane; i < N / 2; i += 32) {
            const int lo = ((i & ~(stride - 1)) << 1) | (i & (stride - 1));
            const int hi = lo + stride;
            const double a = d[lo], b = d[hi];
            const uint32_t ia = ix[lo], ib = ix[hi];
            if (pair_less(b, ib, a, ia)) {
                d[lo] = b; d[hi] = a;
                ix[lo] = ib; ix[hi] = ia;
            }
        }
        __syncwarp();
    }
}

// LCAP: list capacity (power of two >= k); the candidate buffer has LCAP slots too.
// MULTI: a table launch (the batched engine): each query's request gives its
// cloud (kept per warp in shared memory), k and output slots.
// CARRY: children's records are read when their parent is expanded and carried
// on the stack (no dependent loads at a pop, empty leaves never pushed, subtrees
// of at most `bucket` points scanned as one range); without it (the plain path)
// a popped node's record is read then, one leaf at a time.
#define KV(f) (MULTI ? s_view[warp].f : a.f)
template <int LCAP, bool MULTI, bool CARRY = true>
__global__ void __launch_bounds__(kKnnThreads) k_knn(KnnArgs a) {
    constexpr int P = 2 * LCAP;
    extern __shared__ __align__(16) unsigned char smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // per warp: list+buffer (P pairs) and the traversal stack (node, depth, lower bound)
    double* base_d = reinterpret_cast<double*>(smem);
    double* sd = base_d + (size_t)warp * P;
    double* st_lb = base_d + (size_t)kKnnWarps * P + (size_t)warp * kKnnStack;
    uint32_t* base_u = reinterpret_cast<uint32_t*>(base_d + (size_t)kKnnWarps * (P + kKnnStack));
    uint32_t* si = base_u + (size_t)warp * P;
    // stack entry: a range [st_a, st_b) to scan, or (st_b == 0xffffffff) an internal node whose first child is st_a
    uint32_t* st_a = base_u + (size_t)kKnnWarps * P + (size_t)warp * kKnnStack;
    uint32_t* st_b = base_u + (size_t)kKnnWarps * (P + kKnnStack) + (size_t)warp * kKnnStack;
    uint8_t* st_depth =
        reinterpret_cast<uint8_t*>(base_u + (size_t)kKnnWarps * (P + 2 * kKnnStack)) + (size_t)warp * kKnnStack;
    __shared__ double s_rad[MULTI ? kKnnWarps : 1][kMaxDepth + 1][3];
    __shared__ CloudView s_view[MULTI ? kKnnWarps : 1];
    double (*s_radii)[3] = s_rad[MULTI ? warp : 0];
    if (!MULTI) {
        for (int i = threadIdx.x; i < (kMaxDepth + 1) * 3; i += kKnnThreads)
            (&s_radii[0][0])[i] = (&a.geom->radii[0][0])[i];
        __syncthreads();
    }
    const SearchReq* reqs = nullptr;
    uint32_t nreq = 1, cur_cloud = 0xffffffffu;
    uint64_t q0 = 0, nq = a.nq;
    if (MULTI) {
        reqs = a.grp->reqs;
        nreq = a.grp->nreq;
        q0 = a.grp->q_begin;
        nq = a.grp->nq;
    } else if (a.nq_dev) {
        nq = *a.nq_dev;
    }
    const uint64_t nwarps = (uint64_t)gridDim.x * kKnnWarps;
    for (uint64_t w = (uint64_t)blockIdx.x * kKnnWarps + warp; w < nq; w += nwarps) {
        const uint64_t qpos = q0 + w;
        const uint64_t q = a.order ? a.order[qpos] : qpos;
        uint32_t K = a.k;
        uint64_t o = q * (uint64_t)K;  // first output slot of this query
        const double* qc = a.q + 3 * q;
        if (MULTI) {  // the request whose positions contain q (q_begin ascending)
            uint32_t lo = 0, hi = nreq;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (reqs[mid].q_begin <= q) lo = mid;
                else hi = mid;
            }
            const SearchReq& rq = reqs[lo];
            if (rq.cloud_id != cur_cloud) {
                __syncwarp();
                const double* gr = &rq.cv.geom->radii[0][0];
                for (int t = lane; t < (kMaxDepth + 1) * 3; t += 32) (&s_radii[0][0])[t] = gr[t];
                if (lane == 0) s_view[warp] = rq.cv;
                cur_cloud = rq.cloud_id;
                __syncwarp();
            }
            K = rq.k;
            const uint64_t ql = q - rq.q_begin;
            o = rq.out_begin + ql * (uint64_t)K;
            qc = rq.centers + 3 * ql;
        }
        const double p[3] = {qc[0], qc[1], qc[2]};
        for (int i = lane; i < P; i += 32) {
            sd[i] = INFINITY;
            si[i] = 0xffffffffu;
        }
        __syncwarp();
        uint32_t nl = 0;        // entries in the sorted list sd[0, LCAP)
        uint32_t nb = 0;        // entries in the buffer sd[LCAP, 2 LCAP)
        double thr = INFINITY;  // k-th best distance (when nl == K)
        uint32_t thr_i = 0xffffffffu;
        bool failed = false;

        auto merge = [&]() {
            // the list half is sorted already: sort the buffer half descending, then one
            // bitonic merge of (ascending list, descending buffer) sorts all P pairs
            warp_bitonic_sort_desc<LCAP>(sd + LCAP, si + LCAP);
            warp_bitonic_merge<P>(sd, si);
            uint32_t tot = nl + nb;
            nl = tot < K ? tot : K;
            nb = 0;
            for (int i = (int)nl + lane; i < P; i += 32) {
                sd[i] = INFINITY;
                si[i] = 0xffffffffu;
            }
            __syncwarp();
            if (nl == K) {
                thr = sd[K - 1];
                thr_i = si[K - 1];
            }
        };

        // stack of (range or first child, depth, lower bound); the root's bound is 0
        // (linear_octree.hpp:904).  Child records are read when their parent is
        // expanded, so a popped entry needs no further dependent loads; empty leaves
        // are never pushed and subtrees of at most `bucket` points are scanned as one
        // range (extra points cannot change the k best pairs).
        if constexpr (CARRY) {
            const uint32_t fc0 = KV(offsets)[0];
            const uint2 rg0 = KV(ranges)[0];
            const bool scan0 = fc0 == 0 || rg0.y - rg0.x <= a.bucket;
            if (lane == 0) {
                st_a[0] = scan0 ? rg0.x : fc0;
                st_b[0] = scan0 ? rg0.y : 0xffffffffu;
                st_depth[0] = 0;
                st_lb[0] = 0.0;
            }
        } else if (lane == 0) {
            st_a[0] = 0;  // the root node
            st_depth[0] = 0;
            st_lb[0] = 0.0;
        }
        __syncwarp();
        int sp = 1;
        while (sp > 0 && !failed) {
            --sp;
            uint32_t ea = st_a[sp], eb = st_b[sp];
            const double lb = st_lb[sp];
            const uint32_t depth = st_depth[sp];
            __syncwarp();
            if (lb > thr) continue;
            if constexpr (!CARRY) {  // plain: the popped node's record
                const uint32_t node = ea;
                const uint32_t fcn = KV(offsets)[node];
                if (fcn == 0) {
                    const uint2 rg = KV(ranges)[node];
                    ea = rg.x;
                    eb = rg.y;
                } else {
                    ea = fcn;
                    eb = 0xffffffffu;
                }
            }
            if (eb != 0xffffffffu) {
                // points [ea, eb): distances, candidates into the buffer
                for (uint32_t b = ea; b < eb; b += 32) {
                    const uint32_t i = b + lane;
                    double d = INFINITY;
                    bool cand = false;
                    if (i < eb) {
                        d = dist_pp(p[0], p[1], p[2], KV(xs)[i], KV(ys)[i], KV(zs)[i]);
                        cand = pair_less(d, i, thr, thr_i);
                    }
                    uint32_t m = __ballot_sync(0xffffffffu, cand);
                    if (nb + __popc(m) > (uint32_t)LCAP) {
                        merge();
                        cand = cand && pair_less(d, i, thr, thr_i);
                        m = __ballot_sync(0xffffffffu, cand);
                    }
                    if (cand) {
                        const uint32_t slot = LCAP + nb + __popc(m & lanemask_lt());
                        sd[slot] = d;
                        si[slot] = i;
                    }
                    nb += __popc(m);
                    __syncwarp();
                }
            } else {
                // internal: lower bounds and records of the 8 children, nearest pushed last
                const uint32_t fc = ea;
                const uint32_t cd = depth + 1;
                double clb = INFINITY;
                bool keep = false;
                uint32_t ca = 0, cb = 0;
                if (lane < 8) {
                    const uint32_t child = fc + lane;
                    clb = dist_po(p, KV(centers) + 3ull * child, s_radii[cd]);
                    if constexpr (CARRY) {
                        const uint32_t cfc = KV(offsets)[child];
                        const uint2 rg = KV(ranges)[child];
                        if (cfc && rg.y - rg.x > a.bucket) {
                            ca = cfc;
                            cb = 0xffffffffu;
                            keep = !(clb > thr);
                        } else {
                            ca = rg.x;
                            cb = rg.y;
                            keep = (rg.y > rg.x) && !(clb > thr);
                        }
                    } else {
                        ca = child;  // its record is read when it is popped
                        keep = !(clb > thr);
                    }
                }
                const uint32_t km = __ballot_sync(0xffffffffu, keep) & 0xffu;
                const int nk = __popc(km);
                if (sp + nk > kKnnStack) {
                    failed = true;
                    break;
                }
                // position among kept children by descending (lb, lane): farthest deepest
                int pos = 0;
#pragma unroll
                for (int o = 0; o < 8; ++o) {
                    const double ol = __shfl_sync(0xffffffffu, clb, o);
                    const bool ok = (km >> o) & 1u;
                    if (ok && o != lane && ((ol > clb) || (ol == clb && o > lane))) ++pos;
                }
                if (keep) {
                    const int slot = sp + pos;
                    st_a[slot] = ca;
                    st_b[slot] = cb;
                    st_lb[slot] = clb;
                    st_depth[slot] = (uint8_t)cd;
                }
                __syncwarp();
                sp += nk;
            }
        }
        if (failed) set_err(a.err, kErrStackOverflow);
        if (nb > 0) merge();
        for (uint32_t j = lane; j < K; j += 32) {
            if (j < nl) {
                a.idx[o + j] = si[j];
                a.d2[o + j] = sd[j];
            } else {
                a.idx[o + j] = 0xffffffffu;
                a.d2[o + j] = INFINITY;
            }
        }
        if (lane == 0 && a.counts) a.counts[q] = nl;
        __syncwarp();
    }
}

template <int LCAP>
size_t knn_smem() {
    const size_t P = 2 * LCAP;
    const size_t per = P + kKnnStack;
    return (size_t)kKnnWarps * (per * 8 + (per + kKnnStack) * 4 + kKnnStack) + 16;
}

template <int LCAP>
cudaError_t launch_l(const KnnArgs& a, int grid, cudaStream_t s, bool carry) {
    const size_t smem = knn_smem<LCAP>();
    cudaError_t e;
    if (carry) {
        if ((e = cudaFuncSetAttribute(k_knn<LCAP, false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem)) != cudaSuccess)
            return e;
        k_knn<LCAP, false, true><<<grid, kKnnThreads, smem, s>>>(a);
    } else {
        if ((e = cudaFuncSetAttribute(k_knn<LCAP, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem)) != cudaSuccess)
            return e;
        k_knn<LCAP, false, false><<<grid, kKnnThreads, smem, s>>>(a);
    }
    return cudaGetLastError();
}

// Table launch of the list kernel (the engine's kNN groups with 64 < k <= LCAP).
template <int LCAP>
cudaError_t launch_l_table(const DynGroup* d_grp, const uint32_t* order, uint32_t bucket, uint32_t* idx, double* d2,
                           uint32_t* counts, uint32_t* err, int grid, cudaStream_t s) {
    KnnArgs a{};
    a.grp = d_grp;
    a.bucket = bucket;
    a.order = order;
    a.idx = idx;
    a.d2 = d2;
    a.counts = counts;
    a.err = err;
    k_knn<LCAP, true><<<grid, kKnnThreads, knn_smem<LCAP>(), s>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Register kNN for k <= 64: one warp per query, the k best (distance, index)
// pairs held in registers as a sorted list (R = 1 or 2 entries per lane,
// element j = r * 32 + lane).  Leaf points that beat the k-th pair collect in a
// 32-entry shared buffer; a full buffer is merged into the list by a register
// bitonic sort + merge (xor shuffles, no shared-memory sort).  Children are judged with their ranges and first-child links loaded at
// expansion time, so empty leaves are never pushed and a popped entry needs no
// further dependent loads before its points are read.
// ---------------------------------------------------------------------------

template <int R>
struct RegList {
    double d[R];
    uint32_t i[R];
};

template <int R>
__device__ __forceinline__ void reglist_kth(const RegList<R>& L, uint32_t K, double& td, uint32_t& ti) {
    const int r = (int)(K - 1) >> 5, src = (int)(K - 1) & 31;
    double d = L.d[0];
    uint32_t i = L.i[0];
#pragma unroll
    for (int rr = 1; rr < R; ++rr)
        if (rr == r) {
            d = L.d[rr];
            i = L.i[rr];
        }
    td = __shfl_sync(0xffffffffu, d, src);
    ti = __shfl_sync(0xffffffffu, i, src);
}

// Compare-exchange with the lane `lane ^ j`: keep the smaller pair when
// `keep_min`, else the larger.
__device__ __forceinline__ void cx_xor(double& d, uint32_t& i, int j, bool keep_min) {
    const double pd = __shfl_xor_sync(0xffffffffu, d, j);
    const uint32_t pi = __shfl_xor_sync(0xffffffffu, i, j);
    const bool partner_less = pair_less(pd, pi, d, i);
    if (partner_less == keep_min) {
        d = pd;
        i = pi;
    }
}

// Ascending bitonic sort of one pair per lane (32 pairs).
__device__ __forceinline__ void warp_sort32(double& d, uint32_t& i) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) cx_xor(d, i, j, ((lane & j) == 0) == ((lane & k) == 0));
}

// Sort a bitonic sequence of 32 pairs (one per lane) ascending.
__device__ __forceinline__ void warp_bitonic_merge32(double& d, uint32_t& i) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) cx_xor(d, i, j, (lane & j) == 0);
}

// Merge 32 unsorted candidate pairs (one per lane, +inf for none) into the
// sorted register list, keeping the smallest 32 * R pairs.  For R = 2: the 32
// smallest of (upper half, candidates) are min(upper[l], sorted_cand[31 - l]),
// and the 64 smallest of everything are the lower half merged with those.
template <int R>
__device__ __forceinline__ void reglist_merge32(RegList<R>& L, double cd, uint32_t ci) {
    const int lane = threadIdx.x & 31;
    warp_sort32(cd, ci);
    const double rd = __shfl_sync(0xffffffffu, cd, 31 - lane);
    const uint32_t ri = __shfl_sync(0xffffffffu, ci, 31 - lane);
    double md = L.d[R - 1];
    uint32_t mi = L.i[R - 1];
    if (pair_less(rd, ri, md, mi)) {
        md = rd;
        mi = ri;
    }
    warp_bitonic_merge32(md, mi);
    if constexpr (R == 1) {
        L.d[0] = md;
        L.i[0] = mi;
    } else {
        // lower half L0 (ascending) against reversed M: min goes low, max goes high
        const double xd = __shfl_sync(0xffffffffu, md, 31 - lane);
        const uint32_t xi = __shfl_sync(0xffffffffu, mi, 31 - lane);
        double lo_d = L.d[0], hi_d = xd;
        uint32_t lo_i = L.i[0], hi_i = xi;
        if (pair_less(xd, xi, lo_d, lo_i)) {
            hi_d = lo_d;
            hi_i = lo_i;
            lo_d = xd;
            lo_i = xi;
        }
        warp_bitonic_merge32(lo_d, lo_i);
        warp_bitonic_merge32(hi_d, hi_i);
        L.d[0] = lo_d;
        L.i[0] = lo_i;
        L.d[1] = hi_d;
        L.i[1] = hi_i;
    }
}

struct KnnTableArgs {
    SearchReq single;        // the request of a single-cloud search (grp == null)
    const DynGroup* grp;     // sizes and request table of a batch group (device)
    uint64_t nq;             // queries of a single-request launch
    const uint32_t* order;   // visiting order (global query positions), or null
    uint32_t bucket;
    uint32_t* idx;
    double* d2;
    uint32_t* counts;
    uint32_t* err;
    double est;              // > 0: provisional k-th distance from the first range's density (factor), 0: off
    const unsigned long long* nq_dev;  // single-request launch: the query count in device memory (else nq)
};

// MULTI 0: one request in the kernel parameters; 1: a request table, the
// current request's cloud pointers in shared memory; 2: a request table whose
// requests are all on the cloud single.cv (kernel parameters)
#define KRQ(f) (MULTI ? reqs[ri].f : a.single.f)
#define KRQV(f) (MULTI == 1 ? s_view[warp].f : a.single.cv.f)
template <int R, int MULTI>
__global__ void __launch_bounds__(kKnnThreads, 8) k_knn_reg(KnnTableArgs a) {
    __shared__ uint32_t st_a[kKnnWarps][kKnnStack];   // leaf: first point; internal: first child
    __shared__ uint32_t st_b[kKnnWarps][kKnnStack];   // leaf: end point; internal: 0xffffffff
    __shared__ double st_lb[kKnnWarps][kKnnStack];
    __shared__ uint8_t st_depth[kKnnWarps][kKnnStack];
    __shared__ double s_rad[kKnnWarps][kMaxDepth + 1][3];
    __shared__ double s_bd[kKnnWarps][32];
    __shared__ uint32_t s_bi[kKnnWarps][32];
    __shared__ CloudView s_view[MULTI == 1 ? kKnnWarps : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double (*s_radii)[3] = s_rad[warp];
    uint32_t cur_cloud = 0xffffffffu;
    uint32_t* sa = st_a[warp];
    uint32_t* sb = st_b[warp];
    double* sl = st_lb[warp];
    uint8_t* sd = st_depth[warp];
    const SearchReq* reqs = nullptr;
    uint32_t nreq = 1;
    uint64_t q0 = 0, nq = a.nq;
    if (MULTI) {
        reqs = a.grp->reqs;
        nreq = a.grp->nreq;
        q0 = a.grp->q_begin;
        nq = a.grp->nq;
    } else if (a.nq_dev) {
        nq = *a.nq_dev;
    }
    const uint64_t nwarps = (uint64_t)gridDim.x * kKnnWarps;
    for (uint64_t w = (uint64_t)blockIdx.x * kKnnWarps + warp; w < nq; w += nwarps) {
        const uint64_t qpos = q0 + w;
        const uint64_t q = a.order ? a.order[qpos] : qpos;  // global query position
        uint32_t ri = 0;
        if (MULTI) {  // the request whose positions contain q (q_begin ascending)
            uint32_t lo = 0, hi = nreq;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (reqs[mid].q_begin <= q) lo = mid;
                else hi = mid;
            }
            ri = lo;
        }
        if (KRQ(cloud_id) != cur_cloud) {
            __syncwarp();
            const double* gr = &KRQ(cv.geom)->radii[0][0];
            for (int t = lane; t < (kMaxDepth + 1) * 3; t += 32) (&s_radii[0][0])[t] = gr[t];
            if (MULTI == 1 && lane == 0) s_view[warp] = reqs[ri].cv;
            cur_cloud = KRQ(cloud_id);
            __syncwarp();
        }
        const uint32_t K = KRQ(k);
        const uint64_t ql = q - KRQ(q_begin);
        const double* qc = KRQ(centers);
        const double p[3] = {qc[3 * ql], qc[3 * ql + 1], qc[3 * ql + 2]};
        RegList<R> L;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            L.d[r] = INFINITY;
            L.i[r] = 0xffffffffu;
        }
        uint32_t nl = 0;
        double thr = INFINITY;
        uint32_t thr_i = 0xffffffffu;
        bool failed = false;
        uint32_t nb = 0;  // candidates waiting in the shared buffer
        double* bd = s_bd[warp];
        uint32_t* bi = s_bi[warp];
        // Provisional threshold: at the first point range the search reaches (the
        // query's own cell, nearest first), the squared radius holding about
        // `est` x k points at that cell's points per unit of xy area.  Nodes and
        // points beyond it are skipped; every point within it is still visited
        // (lower bounds never exceed distances), so if at least k points lie
        // within it the k best are exact, and otherwise the query runs again
        // without it.
        bool est_pending = a.est > 0.0, est_used = false;
        for (int attempt = 0; attempt < 2; ++attempt) {
        auto merge_buf = [&]() {
            const double cdv = (lane < (int)nb) ? bd[lane] : (double)INFINITY;
            const uint32_t civ = (lane < (int)nb) ? bi[lane] : 0xffffffffu;
            __syncwarp();
            reglist_merge32<R>(L, cdv, civ);
            nl = (nl + nb < K) ? nl + nb : K;
            nb = 0;
            if (nl == K) reglist_kth<R>(L, K, thr, thr_i);
        };
        // root (bound 0, linear_octree.hpp:904)
        {
            const uint32_t fc0 = KRQV(offsets)[0];
            const uint2 rg0 = KRQV(ranges)[0];
            const bool scan0 = fc0 == 0 || rg0.y - rg0.x <= a.bucket;
            if (lane == 0) {
                sa[0] = scan0 ? rg0.x : fc0;
                sb[0] = scan0 ? rg0.y : 0xffffffffu;
                sl[0] = 0.0;
                sd[0] = 0;
            }
        }
        __syncwarp();
        int sp = 1;
        while (sp > 0) {
            --sp;
            const uint32_t ea = sa[sp], eb = sb[sp];
            const double lb = sl[sp];
            const uint32_t depth = sd[sp];
            __syncwarp();
            if (lb > thr) continue;
            if (eb != 0xffffffffu) {
                if (est_pending) {
                    est_pending = false;
                    const double area = 4.0 * s_radii[depth][0] * s_radii[depth][1];
                    if (area > 0.0) {
                        thr = a.est * (double)K * area / (3.14159265358979323846 * (double)(eb - ea));
                        thr_i = 0xffffffffu;  // with the pair order this accepts d <= thr
                        est_used = true;
                    }
                }
                // leaf [ea, eb): candidates beat the k-th pair
                for (uint32_t b = ea; b < eb; b += 32) {
                    const uint32_t i = b + lane;
                    double d = INFINITY;
                    bool cand = false;
                    if (i < eb) {
                        d = dist_pp(p[0], p[1], p[2], KRQV(xs)[i], KRQV(ys)[i], KRQV(zs)[i]);
                        cand = pair_less(d, i, thr, thr_i);
                    }
                    uint32_t m = __ballot_sync(0xffffffffu, cand);
                    if (nb + __popc(m) > 32) {
                        merge_buf();
                        cand = cand && pair_less(d, i, thr, thr_i);
                        m = __ballot_sync(0xffffffffu, cand);
                    }
                    if (cand) {
                        const uint32_t slot = nb + __popc(m & lanemask_lt());
                        bd[slot] = d;
                        bi[slot] = i;
                    }
                    nb += __popc(m);
                    __syncwarp();
                }
                continue;
            }
            // internal: judge the 8 children (bound, first child / range), nearest on top
            const uint32_t fc = ea;
            const uint32_t cd = depth + 1;
            double clb = INFINITY;
            bool keep = false;
            uint32_t ca = 0, cb = 0;
            if (lane < 8) {
                const uint32_t child = fc + lane;
                clb = dist_po(p, KRQV(centers) + 3ull * child, s_radii[cd]);
                const uint32_t cfc = KRQV(offsets)[child];
                const uint2 rg = KRQV(ranges)[child];
                if (cfc && rg.y - rg.x > a.bucket) {
                    ca = cfc;
                    cb = 0xffffffffu;
                    keep = !(clb > thr);
                } else {
                    // a leaf, or a small subtree scanned as one range: extra points can only be
                    // rejected by the k-th pair, so the k best pairs are unchanged
                    ca = rg.x;
                    cb = rg.y;
                    keep = (rg.y > rg.x) && !(clb > thr);  // an empty leaf holds no candidate
                }
            }
            const uint32_t km = __ballot_sync(0xffffffffu, keep) & 0xffu;
            const int nk = __popc(km);
            if (sp + nk > kKnnStack) {
                failed = true;
                break;
            }
            int pos = 0;
#pragma unroll
            for (int o = 0; o < 8; ++o) {
                const double ol = __shfl_sync(0xffffffffu, clb, o);
                const bool ok = (km >> o) & 1u;
                if (ok && o != lane && ((ol > clb) || (ol == clb && o > lane))) ++pos;
            }
            if (keep) {
                const int slot = sp + pos;
                sa[slot] = ca;
                sb[slot] = cb;
                sl[slot] = clb;
                sd[slot] = (uint8_t)cd;
            }
            __syncwarp();
            sp += nk;
        }
        if (nb) merge_buf();
        if (!(est_used && nl < K) || failed) break;
        // fewer than k points within the provisional threshold: again, without it
#pragma unroll
        for (int r = 0; r < R; ++r) {
            L.d[r] = INFINITY;
            L.i[r] = 0xffffffffu;
        }
        nl = 0;
        thr = INFINITY;
        thr_i = 0xffffffffu;
        est_used = false;
        __syncwarp();
        }
        if (failed) set_err(a.err, kErrStackOverflow);
        const uint64_t o = KRQ(out_begin) + ql * (uint64_t)K;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t j = (uint32_t)(r * 32 + lane);
            if (j < K) {
                a.idx[o + j] = (j < nl) ? L.i[r] : 0xffffffffu;
                a.d2[o + j] = (j < nl) ? L.d[r] : (double)INFINITY;
            }
        }
        if (lane == 0 && a.counts) a.counts[q] = nl;
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// Curve-ordered kNN: one query per warp, a walk that collects every point within
// a provisional distance and ranks the collected points at the end.
//
// With a good provisional threshold the walk needs no order, no sorted list and
// no merges: it is a radius search whose hits (squared distance, index) go to a
// buffer of `cap` pairs in shared memory; if at least k pairs came in, the k
// best are among them.  As the order is free, a step takes up to four nodes off
// the stack, the 32 lanes judging their 32 children at once, and the point
// ranges it finds are gathered and tested as one run of points, 32 lanes full
// whatever the ranges' lengths.
//
// The final ranking is a counting sort: squared distances in the plane are
// close to uniform, so `bins` equal bins of [0, threshold] hold one or two pairs
// each; a pair's rank is its bin's start plus the pairs of the bin that precede
// it by (distance, index), and the pair is written to that output slot.  (When a
// bin holds more than kBinMany pairs the bins are taken again over the logarithm
// of the distances, so far outliers do not press the others into one bin; if one
// still does, the pairs are sorted.)  A
// buffer that runs full keeps the bins that hold its k smallest pairs and the
// threshold drops to the largest pair kept.
//
// Thresholds: a warp takes `chunk` consecutive queries at a time, and every one
// after the first of a run starts at kGrpSeed x the largest k-th distance of those
// before it, each faded by kSeedFade a query (the k-th distance varies slowly along the curve;
// longer runs widen the stretch of the curve that the warps work on at once,
// which costs L2 hits).  Every kKnnHeadStride-th query (of k = 1 every 64th) is a head: heads are handed
// out first; the first query of a run (and each query handed out alone at the
// end) starts from the nearest head of its request that has finished.  A query
// without a seed (one whose centre lies outside the cloud's box among them), and a query that found fewer than k pairs within its seeded
// threshold, takes the k-th distance among the first 2 k points (3/2 k of k > 256) that a
// best-first walk comes to (knn_near_ranges): an upper bound of its k-th
// distance, so the walk that follows always suffices.  What is left (a stack or a buffer that cannot hold a
// degenerate input) is appended to a fallback list that the sorted-list kernels
// complete exactly.
//
// F32 (k <= 64): points are first tested in FP32 (centre-relative copies)
// against an FP32 bound of the threshold (knn_f32_threshold); only points not
// rejected take the FP64 distance.
//
// Bound: latency and issue (500k queries of k = 50 on the 10M-point tile: 3.7k
// warp instructions a query where the sorted lists of four queries a warp took
// 5.6k; 0.6 of a warp instruction a cycle and scheduler, dependent loads the
// largest stall).  Two things cost more than they look: code that no longer fits
// the instruction cache (the loops below are not unrolled: 3.42 -> 2.87 ms) and
// shared memory, which is taken from the L1 that serves neighbouring queries
// (2 KB more a block: 2.87 -> 2.97 ms).  Whole calls before (groups of four with
// sorted lists for k <= 64, bitonic merges in shared memory above) and now:
//   10M-point tile: 500k, k = 50 3700 -> 2754 us; 50k, k = 50 1069 -> 430; 5k, k = 50
//   497 -> 195; 200, k = 50 345 -> 105; 5M: 30k, k = 250 2300 -> 627; 3k, k = 900
//   2400 -> 610.  k = 1: see kHeadBitsOne.
// ---------------------------------------------------------------------------

constexpr int kGrpWarps = 4;
constexpr int kGrpThreads = 32 * kGrpWarps;
constexpr int kGrpStack = 200;        // nodes: 60 while four are taken at a time, then 7 more a level at most
constexpr uint32_t kGrpRanges = 64;   // ranges gathered before they are tested
constexpr int kScanBlocks = 2;        // 32-point blocks in flight (k = 50, 500k: 1 3.02 ms, 2 2.85, 4 3.22)
constexpr double kGrpSeed = 1.5;      // provisional threshold / largest recent k-th distance of the run
constexpr double kSeedFade = 0.95;    // what an earlier k-th distance counts for a query later (0.7: +8 % at k = 10)
// In the place of the slot a query seeds from: a head seeds no slot of the run, a centre outside the box none at all.
constexpr uint32_t kHeadSeed = 0xfffffffeu, kNoSeed = 0xfffffffdu;
constexpr uint32_t kBinMany = 48;
// Heads, as a power of two: every 16th query, of k = 1 every 64th.  A head starts cold, which for k = 1 costs several
// times what the others do, and the head's distance is as good a start from further away (0 for centres at cloud
// points).  200k, 500k and 1M centres at cloud points, every 16th -> every 64th, in us: 10M-point tile 429, 889,
// 1655 -> 398, 798, 1476 (sorted lists of four queries a warp 442, 841, 1567), 1M points at 20 a m^2 363, 787, 1504
// -> 338, 718, 1358 (357, 715, 1358); beside the points 749, 1660, 3096 -> 737, 1575, 2983.
constexpr uint32_t kHeadBits = 4, kHeadBitsOne = 6;
static_assert(kKnnHeadStride == 1u << kHeadBits, "every kKnnHeadStride-th query is a head");

struct KnnGroupArgs {
    SearchReq single;                 // one request (grp == null)
    const DynGroup* grp;              // a batch group: sizes and requests on the device
    uint64_t packets;                 // single: queries
    const uint32_t* order;            // visiting order (global query positions), or null
    uint32_t bucket;
    uint32_t cap;                     // pairs of a query's buffer (a multiple of 32, at least k + 32 kScanBlocks)
    uint32_t bins;                    // bins of the ranking (a multiple of 128)
    uint32_t* idx;
    double* d2;
    uint32_t* counts;
    uint32_t* err;
    double est;                       // > 0: queries are seeded; else every one starts from the points next to it
    uint32_t* packet_ctr;             // [0] runs of `chunk` queries, [1] single queries at the end, [2] heads
    uint32_t chunk;                   // pairs of consecutive queries per fetch (>= 1)
    uint32_t heads;                   // 1: every kKnnHeadStride-th query is a head, taken first
    double* head_kth;                 // per head: the largest k-th distance it found (NaN: not yet, < 0: none)
    unsigned long long* stats;        // FP32 filter: point tests, FP64 tests, band hits (may be null)
    uint32_t* fb_list;                // queries left to the sorted-list kernels (global positions; a batch group's
                                      // entries start at its q_begin)
    unsigned long long* fb_count;
};

// FP32 filter of the group kNN: a point whose FP32 squared distance D_f to
// the query exceeds the returned value has an exact squared distance above
// thr.  Per axis a = p - centre (|a| <= A, the box radius) and b = q - centre
// (|b| <= B) are each rounded once to FP32 from their FP64 differences, and
// delta_f = fl32(a_f - b_f); with u = 2^-24, |delta_f - delta| <= 1.0002 u
// (A + B + |delta|).  For D <= thr (|delta| <= s = sqrt thr, M = A + B + s):
// |sum delta_f^2 - D| <= 2 * 1.0002 u M sqrt(3) s + 3.0012 u^2 M^2, and the
// FP32 product and two fused adds add at most 3.0001 u sum delta_f^2 <=
// 3.0001 u (s + 1.733 u M)^2.  The threshold is thr plus twice that bound,
// rounded up to FP32.  ab = A + B.
__device__ __forceinline__ float knn_f32_threshold(double thr, double ab) {
    if (!(thr < (double)INFINITY)) return INFINITY;
    const double u = 5.9604644775390625e-08;  // 2^-24
    const double sr = sqrt(thr) * (1.0 + 1.0e-12);
    const double M = ab + sr;
    const double t = sr + 1.74 * u * M;
    const double err = 3.47 * u * M * sr + 3.01 * u * u * M * M + 3.01 * u * t * t;
    return __double2float_ru(thr + 2.0 * err);
}

// Squared distances (>= 0, or +inf) to bins, non-decreasing: linear in the
// distance (shift < 0), or in the bits of its FP32 value (its logarithm).
struct BinMap {
    float scale;
    uint32_t lo;
    int shift;
    bool crowded;  // a bin holds more than kBinMany pairs all the same
    __device__ __forceinline__ uint32_t bin(double d, uint32_t bins) const {
        if (shift < 0) {
            const int b = (int)((float)d * scale);  // NaN (inf * 0) converts to 0
            return (uint32_t)b < bins ? (uint32_t)b : bins - 1;
        }
        const uint32_t v = __float_as_uint((float)d);
        const uint32_t b = v < lo ? 0u : (v - lo) >> shift;
        return b < bins ? b : bins - 1;
    }
};

// Bins of the n pairs at d, none above `top` (one warp): hist[b] becomes the number of pairs below bin b.
__device__ __forceinline__ BinMap knn_bin_pairs(const double* d, uint32_t n, double top, uint32_t* hist,
                                                uint32_t bins) {
    const int lane = threadIdx.x & 31;
    BinMap m;
    m.scale = top > 0.0 && top < (double)INFINITY ? (float)bins / (float)top : 0.0f;
    m.lo = 0;
    m.shift = -1;
    m.crowded = false;
    uint4* h4 = reinterpret_cast<uint4*>(hist);  // 128 bins a step, four on a lane
#pragma unroll 1
    for (int tries = 0;; ++tries) {
        __syncwarp();
#pragma unroll 1
        for (uint32_t b = 0; b < bins; b += 128) h4[b / 4 + lane] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
#pragma unroll 1
        for (uint32_t e = lane; e < n; e += 32) atomicAdd(&hist[m.bin(d[e], bins)], 1u);
        __syncwarp();
        uint32_t below = 0, most = 0;
#pragma unroll 1
        for (uint32_t b = 0; b < bins; b += 128) {
            uint4 c = h4[b / 4 + lane];
            const uint32_t sum = c.x + c.y + c.z + c.w;
            most = max(most, max(max(c.x, c.y), max(c.z, c.w)));
            uint32_t ex = sum;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, ex, off);
                if (lane >= off) ex += y;
            }
            const uint32_t all = __shfl_sync(0xffffffffu, ex, 31);
            ex += below - sum;
            below += all;
            c.w = ex + c.x + c.y + c.z;
            c.z = ex + c.x + c.y;
            c.y = ex + c.x;
            c.x = ex;
            h4[b / 4 + lane] = c;
        }
        m.crowded = __any_sync(0xffffffffu, most > kBinMany);
        if (tries == 0 && m.crowded) {
            // over the logarithm of the distances instead, unless they are all one (to FP32)
            uint32_t lo = 0xffffffffu, hi = 0;
#pragma unroll 1
            for (uint32_t e = lane; e < n; e += 32) {
                const uint32_t v = __float_as_uint((float)d[e]);  // zero (the query itself) goes to the first bin
                if (v) lo = v < lo ? v : lo;
                hi = v > hi ? v : hi;
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            if (hi > lo) {
                m.lo = lo;
                m.shift = 32 - __clz((hi - lo) / bins);  // (hi - lo) >> shift < bins
                continue;
            }
        }
        __syncwarp();
        return m;
    }
}

// n pairs into ascending order by (distance, index), one warp: Batcher's odd-even merge sort, which takes any n.
// For distances that crowd into one bin (points that are given many times), where ranking each pair against the
// others of its bin is quadratic: 20k queries of k = 1000 on points given 1500 times 85.5 -> 3.1 ms, k = 250 on
// points given 300 times 2.41 -> 0.63; other clouds take the time they took.
__device__ __noinline__ void knn_sort_pairs(double* d, uint32_t* ix, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
#pragma unroll 1
    for (uint32_t p = 1; p < n; p <<= 1) {
#pragma unroll 1
        for (uint32_t k = p; k > 0; k >>= 1) {
            const uint32_t off = k & (p - 1);  // (k mod p)
#pragma unroll 1
            for (uint32_t t = lane;; t += 32) {
                const uint32_t x = off + (((t & ~(k - 1)) << 1) | (t & (k - 1))), y = x + k;
                if (y >= n) break;
                if (((x ^ y) & ~(2 * p - 1)) == 0) {  // of the same run of 2 p
                    const double a = d[x], b = d[y];
                    const uint32_t ia = ix[x], ib = ix[y];
                    if (pair_less(b, ib, a, ia)) {
                        d[x] = b;
                        d[y] = a;
                        ix[x] = ib;
                        ix[y] = ia;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// The K best of n pairs by that sort, to their output slots; returns the K-th distance (< 0: none).
__device__ __noinline__ double knn_write_sorted(double* d, uint32_t* ix, uint32_t n, uint32_t K, uint32_t* idx,
                                                double* d2) {
    knn_sort_pairs(d, ix, n);
#pragma unroll 1
    for (uint32_t t = threadIdx.x & 31; t < K; t += 32) {
        idx[t] = t < n ? ix[t] : 0xffffffffu;
        d2[t] = t < n ? d[t] : (double)INFINITY;
    }
    return n >= K ? d[K - 1] : -1.0;
}

// The K best of n > 32 pairs by their bins, to their output slots; returns the K-th distance (< 0: none).  Out of
// line: as part of the walk's kernel it takes registers and instruction cache from it (500k queries of k = 50
// 2782 -> 2738 us, 100k of k = 10 460 -> 450).
__device__ __noinline__ double knn_rank_pairs(double* bd, uint32_t* bi, uint16_t* ord, uint32_t* hist, uint32_t n,
                                              double thr, uint32_t K, uint32_t bins, uint32_t* idx, double* d2) {
    const uint32_t lane = threadIdx.x & 31;
    const BinMap bm = knn_bin_pairs(bd, n, thr, hist, bins);
    if (bm.crowded) return knn_write_sorted(bd, bi, n, K, idx, d2);
    double kth = -1.0;
#pragma unroll 1
    for (uint32_t e = lane; e < n; e += 32) ord[atomicAdd(&hist[bm.bin(bd[e], bins)], 1u)] = (uint16_t)e;
    __syncwarp();
#pragma unroll 1
    for (uint32_t t = lane; t < n; t += 32) {
        const uint32_t e = ord[t];
        const double dd = bd[e];
        const uint32_t ii = bi[e];
        const uint32_t b = bm.bin(dd, bins);
        const uint32_t f = b ? hist[b - 1] : 0u, l = hist[b];  // the bin's pairs in ord
        uint32_t rank = f;
        if (f < K && l - f > 1)
#pragma unroll 1
            for (uint32_t x = f; x < l; ++x) {
                const uint32_t g = ord[x];
                rank += pair_less(bd[g], bi[g], dd, ii) ? 1u : 0u;
            }
        if (rank < K) {
            idx[rank] = ii;
            d2[rank] = dd;
            if (rank == K - 1) kth = dd;
        }
    }
#pragma unroll 1
    for (uint32_t t = n + lane; t < K; t += 32) {
        idx[t] = 0xffffffffu;
        d2[t] = (double)INFINITY;
    }
    const uint32_t kb = __ballot_sync(0xffffffffu, kth >= 0.0);
    return kb ? __shfl_sync(0xffffffffu, kth, 31 - __clz(kb)) : -1.0;
}

// The K-th smallest of the n squared distances at d as FP32 bits: radix selection, seven bits a pass.
__device__ __noinline__ uint32_t knn_kth_bits(const double* d, uint32_t n, uint32_t K, uint32_t* hist) {
    const int lane = threadIdx.x & 31;
    uint4* h4 = reinterpret_cast<uint4*>(hist);
    uint32_t prefix = 0, left = K;  // the bits so far; the K-th is the left-th smallest of those that begin so
#pragma unroll 1
    for (int shift = 25; shift >= -3; shift -= 7) {
        const int sh = shift < 0 ? 0 : shift, bits = shift < 0 ? 4 : 7;
        __syncwarp();
        h4[lane] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
#pragma unroll 1
        for (uint32_t e = lane; e < n; e += 32) {
            const unsigned long long v = __float_as_uint((float)d[e]);
            if ((v >> (sh + bits)) == prefix) atomicAdd(&hist[(uint32_t)(v >> sh) & ((1u << bits) - 1u)], 1u);
        }
        __syncwarp();
        const uint4 c = h4[lane];
        const uint32_t sum = c.x + c.y + c.z + c.w;
        uint32_t in = sum;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, in, off);
            if (lane >= off) in += y;
        }
        const int at = __ffs(__ballot_sync(0xffffffffu, in >= left)) - 1;  // (n >= K: some lane)
        uint32_t r = left - (in - sum), digit = 4 * lane;
        if (r > c.x) {
            r -= c.x;
            ++digit;
            if (r > c.y) {
                r -= c.y;
                ++digit;
                if (r > c.z) {
                    r -= c.z;
                    ++digit;
                }
            }
        }
        left = __shfl_sync(0xffffffffu, r, at);
        prefix = (prefix << bits) | __shfl_sync(0xffffffffu, digit, at);
    }
    __syncwarp();
    return prefix;
}

// A full buffer of n >= K pairs: its K smallest are kept, at the front, with the others of the K-th's bin;
// returns how many pairs those are and the largest of them.  More than `most` of them: the bins are given up
// for the K-th distance itself (to FP32).  Out of line: the walks that call it stay short enough for the
// instruction cache.
struct KnnCut {
    double top;
    uint32_t n;
};
__device__ __noinline__ KnnCut knn_cut(double* d, uint32_t* ix, uint32_t n, double top, uint32_t K, uint32_t most,
                                       uint32_t* hist, uint32_t bins) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    if (!(top < (double)INFINITY)) {
        top = 0.0;
#pragma unroll 1
        for (uint32_t e = lane; e < n; e += 32) top = fmax(top, d[e]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, off));
    }
    const BinMap bm = knn_bin_pairs(d, n, top, hist, bins);
    // pairs below the first bin that starts at or past K (hist ascends)
    uint32_t kept = n;
#pragma unroll 1
    for (uint32_t b = lane; b < bins; b += 32) kept = hist[b] >= K ? min(kept, hist[b]) : kept;
    kept = __reduce_min_sync(0xffffffffu, kept);
    const bool exact = kept > most;
    const uint32_t kth = exact ? knn_kth_bits(d, n, K, hist) : 0u;
    KnnCut c;
    c.n = 0;
    c.top = 0.0;
#pragma unroll 1
    for (uint32_t t = 0; t < n; t += 32) {
        const uint32_t e = t + lane;
        double dd = 0.0;
        uint32_t ii = 0;
        bool keep = false;
        if (e < n) {
            dd = d[e];
            ii = ix[e];
            keep = exact ? __float_as_uint((float)dd) <= kth : hist[bm.bin(dd, bins)] < K;
        }
        const uint32_t kb = __ballot_sync(0xffffffffu, keep);
        if (keep) {  // at or below the lanes' own positions
            const uint32_t o = c.n + __popc(kb & lanemask_lt());
            d[o] = dd;
            ix[o] = ii;
            c.top = fmax(c.top, dd);
        }
        c.n += __popc(kb);
        __syncwarp();
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) c.top = fmax(c.top, __shfl_xor_sync(0xffffffffu, c.top, off));
    return c;
}

// Open nodes of a cold query that are kept, by the buffer (k <= 64: up to 128 points are looked for).
__host__ __device__ constexpr int knn_open_nodes(uint32_t cap) { return cap <= 192 ? kGrpStack / 2 : kGrpStack; }

// Bytes of dynamic shared memory of one warp: pairs, bins, and the bounds of a cold query's open nodes, whose place
// the ranking's order of the pairs takes when no node is open any more.  (Shared memory is L1 cache that the walks
// lack: at k = 44 and 13, 1.6 KB a block more for the bounds cost 2 to 3 % of the time.)
__host__ __device__ constexpr size_t knn_group_bytes(uint32_t cap, uint32_t bins) {
    const size_t open = 4 * (size_t)knn_open_nodes(cap), ord = 2 * (size_t)cap;
    return (size_t)cap * 12 + (size_t)bins * 4 + (open > ord ? open : ord);
}

// A cold query's first points: nodes and ranges taken best first (the smallest bound of all that are open, as
// octants are thin slabs and a depth-first walk would leave a near one for last) until the ranges (to `list`)
// hold knn_near_points(K) points.  An entry is a node's first child and their depth, or a range's node and depth 255.
// Returns when the list is full; the state is carried from call to call.
__host__ __device__ constexpr uint32_t knn_near_points(uint32_t K) { return K <= 256 ? 2 * K : K + K / 2; }
struct KnnNear {
    int open;        // open entries
    uint32_t taken;  // points of the ranges so far
    uint32_t m;      // ranges of this call
};
__device__ __noinline__ KnnNear knn_near_ranges(const uint32_t* offsets, const uint2* ranges, const double* centers,
                                                const double (*radii)[3], double x, double y, double z, uint32_t K,
                                                uint32_t bucket, KnnNear st, uint32_t* fcs, uint8_t* depths,
                                                float* keys, int room, uint2* list) {
    const int lane = threadIdx.x & 31;
    const double p[3] = {x, y, z};
    st.m = 0;
#pragma unroll 1
    while (st.open > 0 && st.taken < knn_near_points(K) && st.m < kGrpRanges) {
        uint32_t key = 0xffffffffu;  // (bounds are not negative: their bits ascend as they do)
        int at = 0;
#pragma unroll 1
        for (int t = lane; t < st.open; t += 32) {
            const uint32_t kt = __float_as_uint(keys[t]);
            if (kt < key) {
                key = kt;
                at = t;
            }
        }
        const uint32_t least = __reduce_min_sync(0xffffffffu, key);
        at = __shfl_sync(0xffffffffu, at, __ffs(__ballot_sync(0xffffffffu, key == least)) - 1);
        const uint32_t fc = fcs[at], depth = depths[at];
        --st.open;
        __syncwarp();
        if (lane == 0) {  // the last entry takes its place
            fcs[at] = fcs[st.open];
            depths[at] = depths[st.open];
            keys[at] = keys[st.open];
        }
        if (depth == 255u) {
            const uint2 rg = ranges[fc];
            if (lane == 0) list[st.m] = rg;
            ++st.m;
            st.taken += rg.y - rg.x;
            __syncwarp();
            continue;
        }
        const uint32_t child = fc + (lane & 7);
        const uint2 rg = ranges[child];
        const uint32_t cfc = offsets[child], n = rg.y - rg.x;
        const float lb = (float)dist_po(p, centers + 3ull * child, radii[depth]);
        const bool some = lane < 8 && n, whole = cfc == 0 || n <= bucket;
        const uint32_t sm = __ballot_sync(0xffffffffu, some);
        __syncwarp();
        if (some) {
            const int to = st.open + __popc(sm & lanemask_lt());
            fcs[to] = whole ? child : cfc;
            depths[to] = whole ? (uint8_t)255 : (uint8_t)(depth + 1);
            keys[to] = lb;
        }
        st.open += __popc(sm);
        __syncwarp();
        if (st.open + 7 > room) {
            // no room for the next node's children: the far half of the bounds' span goes, and again until half the
            // entries are left (any K points bound the K-th distance; halves of the span and not of the largest
            // bound, as the bounds of a query far from the cloud differ by little)
            uint32_t least_left = 0xffffffffu, most = 0;
#pragma unroll 1
            for (int t = lane; t < st.open; t += 32) {
                least_left = min(least_left, __float_as_uint(keys[t]));
                most = max(most, __float_as_uint(keys[t]));
            }
            const float low = __uint_as_float(__reduce_min_sync(0xffffffffu, least_left));
            float span = __uint_as_float(__reduce_max_sync(0xffffffffu, most)) - low;
#pragma unroll 1
            for (int tries = 0; st.open > room / 2 && span > 0.0f && tries < 24; ++tries) {
                span *= 0.5f;
                int left = 0;
#pragma unroll 1
                for (int t = 0; t < st.open; t += 32) {
                    uint32_t f = 0;
                    float k = 0.0f;
                    uint8_t d = 0;
                    const bool in = t + lane < st.open;
                    if (in) {
                        f = fcs[t + lane];
                        d = depths[t + lane];
                        k = keys[t + lane];
                    }
                    const bool stay = in && k - low <= span;
                    const uint32_t sb = __ballot_sync(0xffffffffu, stay);
                    if (stay) {  // at or below the lanes' own positions
                        const int to = left + __popc(sb & lanemask_lt());
                        fcs[to] = f;
                        depths[to] = d;
                        keys[to] = k;
                    }
                    left += __popc(sb);
                    __syncwarp();
                }
                st.open = left;
            }
            if (st.open > room / 2) st.open = room / 2;  // (equal bounds)
        }
    }
    return st;
}

template <int MULTI, bool F32>
__global__ void __launch_bounds__(kGrpThreads, 7) k_knn_group(KnnGroupArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_n[kGrpWarps];               // pairs in the buffer
    __shared__ uint32_t st_fc[kGrpWarps][kGrpStack];  // first child of a node
    __shared__ uint8_t st_d[kGrpWarps][kGrpStack];    // its children's depth
    __shared__ uint2 s_rg[kGrpWarps][kGrpRanges];
    // the nodes that the warp's last walks passed one by one from the root (centre, first child), by
    // depth: a walk starts at the deepest that holds its whole ball
    __shared__ double s_pc[kGrpWarps][kMaxDepth + 1][3];
    __shared__ uint32_t s_pf[kGrpWarps][kMaxDepth + 1];
    // level radii: per warp for a table of clouds, once per block for one cloud
    __shared__ double s_rad[MULTI == 1 ? kGrpWarps : 1][kMaxDepth + 1][3];
    __shared__ CloudView s_view[MULTI == 1 ? kGrpWarps : 1];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double (*s_radii)[3] = s_rad[MULTI == 1 ? warp : 0];
    if (MULTI != 1) {
        const double* gr = &a.single.cv.geom->radii[0][0];
#pragma unroll 1
        for (int t = threadIdx.x; t < (kMaxDepth + 1) * 3; t += kGrpThreads) (&s_rad[0][0][0])[t] = gr[t];
        __syncthreads();
    }
    if (MULTI != 1 && lane < 3) s_pc[warp][0][lane] = a.single.cv.centers[lane];
    __syncwarp();
    const uint32_t cap = a.cap, bins = a.bins;
    unsigned char* mine = smem + (size_t)warp * knn_group_bytes(cap, bins);
    double* bd = reinterpret_cast<double*>(mine);
    uint32_t* bi = reinterpret_cast<uint32_t*>(mine + (size_t)cap * 8);
    uint32_t* hist = bi + cap;
    uint16_t* ord = reinterpret_cast<uint16_t*>(hist + bins);
    uint32_t* sf = st_fc[warp];
    uint8_t* sdp = st_d[warp];
    float* sk = reinterpret_cast<float*>(ord);  // bounds of a cold query's open nodes
    uint2* list = s_rg[warp];
    uint32_t* np = &s_n[warp];
    unsigned long long f_tests = 0, f_64 = 0, f_band = 0;
    uint32_t cur_cloud = 0xffffffffu;
    const SearchReq* reqs = nullptr;
    uint32_t nreq = 1;
    // query positions of a launch fit 32 bits (positions are u32 in the order arrays)
    uint32_t packets = (uint32_t)a.packets;
    uint32_t fb_base = 0;  // the fallback entries of a batch group start at its first position
    if (MULTI) {
        reqs = a.grp->reqs;
        nreq = a.grp->nreq;
        packets = (uint32_t)a.grp->packets;
        fb_base = (uint32_t)a.grp->q_begin;
    }
    // heads (every S-th query) go out first, one at a time; the others are slots:
    // slot s is the s-th query that is not a head (every query without heads)
    const bool far = (MULTI ? a.grp->kmax : a.single.k) == 1;
    const uint32_t sbits = far ? kHeadBitsOne : kHeadBits, S = 1u << sbits;
    const bool heads = a.heads != 0;
    const uint32_t n_heads = heads ? (packets + S - 1) >> sbits : 0;
    const uint32_t slots = packets - n_heads;
    bool heads_left = n_heads != 0;
    // slots [0, p_chunked) go out in chunks, the rest one at a time
    const uint32_t nw = gridDim.x * kGrpWarps;
    // (runs no longer than leave every warp four of them)
    const uint32_t chunk = max(1u, min(2 * a.chunk, slots / (4 * nw)));
    const uint32_t p_chunked = (chunk > 1 && slots > 2 * nw) ? (slots - 2 * nw) / chunk * chunk : 0;
    uint32_t next = 0, chunk_end = 0;
    double (*pc)[3] = s_pc[warp];
    uint32_t* pf = s_pf[warp];
    uint32_t path_len = 0;
    // the warp's last slot and request; the query after it on the curve, read ahead (lane t < 3: coordinate t)
    uint32_t seed_slot = 0xfffffffeu, seed_ri = 0;
    uint32_t ahead_pos = 0xffffffffu, ahead_q = 0;
    double ahead_c = 0.0;
    double run_kth = -1.0;  // the largest recent k-th distance of the run (< 0: none)

    for (;;) {
        uint32_t slot = 0xffffffffu;  // the head's number when a head
        bool head = false;
        if (heads_left) {
            uint32_t h = 0;
            if (lane == 0) h = atomicAdd(&a.packet_ctr[2], 1u);
            h = __shfl_sync(0xffffffffu, h, 0);
            if (h < n_heads) head = true, slot = h;
            else heads_left = false;
        }
        if (!head) {
            if (next < chunk_end) {
                slot = next++;
            } else {
                uint32_t v = 0;
                if (lane == 0) v = atomicAdd(&a.packet_ctr[0], 1u);
                v = __shfl_sync(0xffffffffu, v, 0);
                const uint64_t c0 = (uint64_t)v * chunk;
                if (c0 < p_chunked) {
                    slot = (uint32_t)c0;
                    next = slot + 1;
                    chunk_end = slot + chunk;
                } else {
                    uint32_t s = 0;
                    if (lane == 0) s = atomicAdd(&a.packet_ctr[1], 1u);
                    s = __shfl_sync(0xffffffffu, s, 0);
                    if ((uint64_t)p_chunked + s >= slots) break;
                    slot = p_chunked + s;
                    next = chunk_end = 0;
                }
            }
            if (slot >= slots) break;
        }
        const uint32_t packet = head ? slot << sbits : !heads ? slot : slot + (far ? slot / ((1u << kHeadBitsOne) - 1) : slot / ((1u << kHeadBits) - 1)) + 1;
        uint32_t ri = 0;
        if (MULTI) {  // the request of this query (packet_begin ascending over the table)
            uint32_t lo = 0, hi = nreq;
#pragma unroll 1
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (reqs[mid].packet_begin <= packet) lo = mid;
                else hi = mid;
            }
            ri = lo;
        }
        if (MULTI == 1 && reqs[ri].cloud_id != cur_cloud) {  // this warp's level radii and cloud follow the query's
            __syncwarp();
            const double* gr = &reqs[ri].cv.geom->radii[0][0];
#pragma unroll 1
            for (int t = lane; t < (kMaxDepth + 1) * 3; t += 32) (&s_radii[0][0])[t] = gr[t];
            if (lane == 0) s_view[warp] = reqs[ri].cv;
            if (lane < 3) pc[0][lane] = reqs[ri].cv.centers[lane];
            cur_cloud = reqs[ri].cloud_id;
            path_len = 0;
            __syncwarp();
        }
        const uint32_t K = KRQ(k);
        const uint32_t q_begin = (uint32_t)KRQ(q_begin);
        const uint32_t pos = q_begin + (packet - (uint32_t)KRQ(packet_begin));
        // seed: the queries before this one in the warp's run, else (between heads) the
        // nearest head of the same request
        if (head || slot != seed_slot + 1 || ri != seed_ri) run_kth = -1.0;
        double seed = run_kth;
        if (seed < 0.0 && heads && !head) {
            const uint32_t pb = (uint32_t)KRQ(packet_begin);
            const uint32_t pe = pb + (uint32_t)(KRQ(q_end) - KRQ(q_begin));
            const uint32_t hlo = packet >> sbits, hhi = hlo + 1;  // heads hlo S < packet < hhi S
            const bool lo_ok = hlo * S >= pb, hi_ok = hhi < n_heads && hhi * S < pe;
            const bool use_hi = hi_ok && (!lo_ok || hhi * S - packet < packet - hlo * S);
            // a head not finished yet reads NaN: no seed (nothing waits for it)
            if (use_hi || lo_ok) seed = __ldcg(&a.head_kth[use_hi ? hhi : hlo]);
        }
        bool cold = !(a.est > 0.0 && seed >= 0.0);
        if (pos != ahead_pos) {
            ahead_q = a.order ? a.order[pos] : pos;
            ahead_c = lane < 3 ? KRQ(centers)[3ull * (ahead_q - q_begin) + lane] : 0.0;
        }
        const uint64_t q = ahead_q;
        const uint64_t ql = q - q_begin;
        const double p[3] = {__shfl_sync(0xffffffffu, ahead_c, 0), __shfl_sync(0xffffffffu, ahead_c, 1),
                             __shfl_sync(0xffffffffu, ahead_c, 2)};
        ahead_pos = next < chunk_end && pos + 1 < (uint32_t)KRQ(q_end) && (!heads || ((packet + 1) & (S - 1))) ? pos + 1 : 0xffffffffu;
        if (ahead_pos != 0xffffffffu) ahead_q = a.order ? a.order[ahead_pos] : ahead_pos;
        // A centre outside the cloud's box (by more than rounding) starts cold and seeds no other: its k-th distance is
        // decided by how far it is from the cloud, and a ball a little larger holds much of the cloud.  20k centres
        // around a cube of 500k points, k = 10: 570 -> 220 us, beside a plane 1056 -> 274; centres inside keep their time
        bool outside = false;
        if (lane < 3) outside = fabs(ahead_c - pc[0][lane]) > 1.000001 * s_radii[0][lane];
        outside = __any_sync(0xffffffffu, outside);
        cold = cold || outside;
        seed_slot = outside ? kNoSeed : head ? kHeadSeed : slot;
        double thr = cold ? (double)INFINITY : kGrpSeed * seed;
        // FP32 filter: query - box centre in FP32, the FP32 threshold, and A + B (box radius +
        // |query - centre|_inf) for new thresholds
        float qx = 0.0f, qy = 0.0f, qz = 0.0f, tf = 0.0f;
        double ab = 0.0;
        if constexpr (F32) {
            const BoxD* bx = KRQV(box);
            const double bqx = dsub(p[0], bx->center[0]);
            const double bqy = dsub(p[1], bx->center[1]);
            const double bqz = dsub(p[2], bx->center[2]);
            const double A = smax(smax(bx->radii[0], bx->radii[1]), bx->radii[2]);
            const double B = smax(smax(fabs(bqx), fabs(bqy)), fabs(bqz));
            ab = (A + B) * (1.0 + 1.0e-12);
            qx = (float)bqx;
            qy = (float)bqy;
            qz = (float)bqz;
        }
        bool ok = true;       // false: left to the fallback
        double kth = -1.0;    // the k-th distance, when k pairs were found
#pragma unroll 1
        for (int attempt = 0; attempt < 2; ++attempt) {
            // phase 0 (cold): the points of the query's own node, for a threshold; phase 1: every point
            // within the threshold
#pragma unroll 1
            for (int phase = cold ? 0 : 1; phase < 2; ++phase) {
                int sp = 0;
                uint32_t m = 0, taken = 0;  // ranges gathered; points of phase 0
                uint2 rg0 = make_uint2(0u, 0u);
                uint32_t fc0 = 0, depth0 = 1;  // children to judge first, and their depth
                if (phase == 0) {
                    thr = (double)INFINITY;
                    fc0 = KRQV(offsets)[0];
                    if (fc0) {  // the root
                        if (lane == 0) {
                            sf[0] = fc0;
                            sdp[0] = 1;
                            sk[0] = 0.0f;
                        }
                        sp = 1;
                    }
                } else if (path_len) {
                    // the deepest node of the path that holds the whole ball, by margins above what a squared distance
                    // loses below the FP64 range (3 x 2^-1075) and above the rounding of coordinates, keys and node
                    // boxes (to the size of the cloud's box): every node outside it is beyond the threshold.  Squares
                    // are compared (an FP64 root: +0.4 % at k = 50); no square is above an infinite threshold
                    const double r2 = thr * 1.000002 + 2.0e-323;
                    bool holds = (uint32_t)lane < path_len;
                    if (holds && lane) {
#pragma unroll
                        for (int t = 0; t < 3; ++t) {
                            const double c = pc[lane][t];
                            const double in = s_radii[lane][t] - fabs(p[t] - c) -
                                              1.0e-12 * (fabs(p[t]) + fabs(c) + s_radii[0][t]);
                            holds = holds && in > 0.0 && in * in > r2;
                        }
                    }
                    path_len = 32 - __clz(__ballot_sync(0xffffffffu, holds));
                    fc0 = pf[path_len - 1];
                    depth0 = path_len;
                } else {
                    rg0 = KRQV(ranges)[0];
                    fc0 = KRQV(offsets)[0];
                    if (fc0) {  // the root
                        if (lane == 0) pf[0] = fc0;
                        path_len = 1;
                    }
                }
                if constexpr (F32) tf = knn_f32_threshold(thr, ab);
                if (phase == 0) {
                } else if (fc0 == 0) {
                    if (lane == 0) list[0] = rg0;
                    m = 1;
                } else {
                    if (lane == 0) {
                        sf[0] = fc0;
                        sdp[0] = (uint8_t)depth0;
                    }
                    sp = 1;
                }
                if (lane == 0) *np = 0;
                __syncwarp();
#pragma unroll 1
                for (;;) {
                    if (phase == 0) {
                        const KnnNear st = knn_near_ranges(KRQV(offsets), KRQV(ranges), KRQV(centers), s_radii, p[0], p[1],
                                                           p[2], K, a.bucket, KnnNear{sp, taken, 0}, sf, sdp, sk,
                                                           knn_open_nodes(cap), list);
                        sp = st.taken < knn_near_points(K) ? st.open : 0;
                        taken = st.taken;
                        m = st.m;
                    }
                    if (phase == 0 || sp == 0 || m > kGrpRanges - 32) {
                        // the gathered ranges, 32 of them at a time as one run of points: lane l's range holds
                        // [first, end) of the run, starting at point first + base
#pragma unroll 1
                        for (uint32_t r0 = 0; r0 < m; r0 += 32) {
                            const uint2 rg = r0 + lane < m ? list[r0 + lane] : make_uint2(0u, 0u);
                            const uint32_t len = rg.y - rg.x;
                            uint32_t end = len;
#pragma unroll
                            for (int off = 1; off < 32; off <<= 1) {
                                const uint32_t y = __shfl_up_sync(0xffffffffu, end, off);
                                if (lane >= off) end += y;
                            }
                            const uint32_t first = end - len, base = rg.x - first;
                            const uint32_t total = __shfl_sync(0xffffffffu, end, 31);
#pragma unroll 1
                            for (uint32_t b = 0; b < total; b += 32 * kScanBlocks) {
                                const uint32_t have = *np;
                                __syncwarp();  // read by every lane before any adds to it
                                uint32_t i[kScanBlocks];
                                double px[kScanBlocks], py[kScanBlocks], pz[kScanBlocks];
                                float4 pt[kScanBlocks];
#pragma unroll
                                for (int u = 0; u < kScanBlocks; ++u) {
                                    const uint32_t bu = b + 32 * u;
                                    if (u && bu >= total) break;
                                    // the lane's range: ranges begun before bu, plus those that begin at or below it
                                    const uint32_t before = __popc(__ballot_sync(0xffffffffu, first < bu));
                                    const uint32_t starts = __reduce_or_sync(
                                        0xffffffffu, (len && first - bu < 32u) ? 1u << (first - bu) : 0u);
                                    const int r = (int)(before + __popc(starts & (2u * (1u << lane) - 1u))) - 1;
                                    // (lanes past the end read the last point again)
                                    i[u] = __shfl_sync(0xffffffffu, base, r) + min(bu + lane, total - 1);
                                    if constexpr (F32) {
                                        pt[u] = KRQV(crel)[i[u]];
                                    } else {
                                        px[u] = KRQV(xs)[i[u]];
                                        py[u] = KRQV(ys)[i[u]];
                                        pz[u] = KRQV(zs)[i[u]];
                                    }
                                }
                                if (have + 32 * kScanBlocks > cap) {
                                    // no room for a whole step: the K smallest pairs (to a bin) are kept, the threshold
                                    // drops to the largest of them
                                    KnnCut c = knn_cut(bd, bi, have, thr, K, cap - 32 * kScanBlocks, hist, bins);
                                    if (c.n + 32 * kScanBlocks > cap) {  // equal distances that fill the buffer
                                        ok = false;
                                        c.n = 0;
                                        c.top = -1.0;  // takes no more points
                                    }
                                    __syncwarp();
                                    if (lane == 0) *np = c.n;
                                    thr = c.top;
                                    if constexpr (F32) tf = knn_f32_threshold(thr, ab);
                                    __syncwarp();
                                }
#pragma unroll
                                for (int u = 0; u < kScanBlocks; ++u) {
                                    if (u && b + 32 * u >= total) break;
                                    const bool in = b + 32 * u + lane < total;
                                    double d = 0.0;
                                    bool cand = false;
                                    if constexpr (F32) {
                                        const float dx = pt[u].x - qx, dy = pt[u].y - qy, dz = pt[u].z - qz;
                                        const float df = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
                                        if (in) {
                                            ++f_tests;
                                            if (!(df > tf)) {  // near the threshold or inside: the exact FP64 test
                                                d = dist_pp(p[0], p[1], p[2], KRQV(xs)[i[u]], KRQV(ys)[i[u]],
                                                            KRQV(zs)[i[u]]);
                                                cand = d <= thr;
                                                ++f_64;
                                                f_band += cand ? 0u : 1u;
                                            }
                                        }
                                    } else {
                                        d = dist_pp(p[0], p[1], p[2], px[u], py[u], pz[u]);
                                        cand = in && d <= thr;
                                    }
                                    if (cand) {
                                        const uint32_t at = atomicAdd(np, 1u);
                                        bd[at] = d;
                                        bi[at] = i[u];
                                    }
                                }
                                __syncwarp();
                            }
                        }
                        m = 0;
                        if (sp == 0) break;
                        __syncwarp();
                        if (phase == 0) continue;
                    }
                    // up to four nodes: lane (node lane / 8, child lane % 8)
                    const int take = sp > 32 ? 1 : sp < 4 ? sp : 4;
                    const int from = sp - 1 - (lane >> 3);
                    bool near = false;
                    uint32_t cfc = 0, cd = 0;
                    uint2 rg = make_uint2(0u, 0u);
                    double oc[3] = {0.0, 0.0, 0.0};
                    if ((lane >> 3) < take) {
                        cd = sdp[from];
                        const uint32_t child = sf[from] + (lane & 7);
                        cfc = KRQV(offsets)[child];
                        rg = KRQV(ranges)[child];
#pragma unroll
                        for (int t = 0; t < 3; ++t) oc[t] = KRQV(centers)[3ull * child + t];
                        near = !(dist_po(p, oc, s_radii[cd]) > thr) && rg.y != rg.x;
                    }
                    const bool whole = cfc == 0 || rg.y - rg.x <= a.bucket;
                    const uint32_t mr = __ballot_sync(0xffffffffu, near && whole);
                    const uint32_t mn = __ballot_sync(0xffffffffu, near && !whole);
                    sp -= take;
                    if (sp + __popc(mn) > kGrpStack) {
                        ok = false;
                        break;
                    }
                    if (near) {
                        if (whole) {
                            list[m + __popc(mr & lanemask_lt())] = rg;
                        } else {
                            const int at = sp + __popc(mn & lanemask_lt());
                            sf[at] = cfc;
                            sdp[at] = (uint8_t)(cd + 1);
                        }
                    }
                    if (sp == 0 && m == 0 && mr == 0 && __popc(mn) == 1) {
                        // one node still, below the path's last: the path goes on with it
                        const int from_lane = __ffs(mn) - 1;
                        if (__shfl_sync(0xffffffffu, cd, from_lane) == path_len) {
                            if (lane == from_lane) {
                                pf[path_len] = cfc;
#pragma unroll
                                for (int t = 0; t < 3; ++t) pc[path_len][t] = oc[t];
                            }
                            ++path_len;
                        }
                    }
                    m += __popc(mr);
                    sp += __popc(mn);
                    __syncwarp();
                }
                __syncwarp();
                if (phase == 0) {
                    if (*np >= K) thr = knn_cut(bd, bi, *np, thr, K, cap - 32 * kScanBlocks, hist, bins).top;
                    __syncwarp();
                }
            }
            if (!ok) break;
            const uint32_t n = *np;
            if (n < K && thr < (double)INFINITY) {  // the seeded threshold was too small
                ok = attempt == 0;
                cold = true;
                __syncwarp();
                continue;
            }
            if (ahead_pos != 0xffffffffu && lane < 3) ahead_c = KRQ(centers)[3ull * (ahead_q - q_begin) + lane];
            const uint64_t o = KRQ(out_begin) + ql * (uint64_t)K;
            if (lane == 0 && a.counts) a.counts[q] = n < K ? n : K;
            if (n <= 32) {  // a pair a lane, ranked against each of the others
                const double dd = (uint32_t)lane < n ? bd[lane] : (double)INFINITY;
                const uint32_t ii = (uint32_t)lane < n ? bi[lane] : 0xffffffffu;
                uint32_t rank = 0;
#pragma unroll 1
                for (uint32_t t = 0; t < n; ++t)
                    rank += pair_less(__shfl_sync(0xffffffffu, dd, t), __shfl_sync(0xffffffffu, ii, t), dd, ii);
                if ((uint32_t)lane >= n) rank = lane;  // empty slots
                if (rank < K) {
                    a.idx[o + rank] = ii;
                    a.d2[o + rank] = dd;
                }
#pragma unroll 1
                for (uint32_t t = 32 + lane; t < K; t += 32) {
                    a.idx[o + t] = 0xffffffffu;
                    a.d2[o + t] = (double)INFINITY;
                }
                const uint32_t kb = __ballot_sync(0xffffffffu, rank == K - 1 && (uint32_t)lane < n);
                kth = kb ? __shfl_sync(0xffffffffu, dd, 31 - __clz(kb)) : -1.0;
                break;
            }
            kth = knn_rank_pairs(bd, bi, ord, hist, n, thr, K, bins, a.idx + o, a.d2 + o);
            break;
        }
        if (!ok && lane == 0) {
            const unsigned long long f = atomicAdd(a.fb_count, 1ull);
            a.fb_list[fb_base + f] = (uint32_t)q;
        }
        if (!ok) ahead_pos = 0xffffffffu;  // not read
        run_kth = fmax(kth, kSeedFade * run_kth);
        seed_ri = ri;
        if (seed_slot == kHeadSeed && lane == 0) __stcg(&a.head_kth[slot], kth);
        __syncwarp();
    }
    if constexpr (F32) {
        if (a.stats) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                f_tests += __shfl_xor_sync(0xffffffffu, f_tests, off);
                f_64 += __shfl_xor_sync(0xffffffffu, f_64, off);
                f_band += __shfl_xor_sync(0xffffffffu, f_band, off);
            }
            if (lane == 0) {
                atomicAdd(&a.stats[0], f_tests);
                atomicAdd(&a.stats[1], f_64);
                atomicAdd(&a.stats[2], f_band);
            }
        }
    }
}

// Buffer pairs and bins for lists of up to k pairs: a seeded walk collects about 1.4 k.
uint32_t knn_group_cap(uint32_t k) { return (knn_near_points(k) + 32 * kScanBlocks + 31) / 32 * 32; }
uint32_t knn_group_bins(uint32_t k) { return k <= 128 ? 128 : k <= 256 ? 256 : k <= 512 ? 512 : 1024; }

// blocks_per_sm > 0 caps the resident blocks (room for a kernel running beside it).
template <int MULTI, bool F32>
cudaError_t launch_group(KnnGroupArgs g, uint32_t kmax, int sms, cudaStream_t s, int blocks_per_sm) {
    g.cap = knn_group_cap(kmax);
    g.bucket /= 4;
    g.bins = knn_group_bins(kmax);
    const size_t smem = kGrpWarps * knn_group_bytes(g.cap, g.bins);
    cudaError_t e;
    if (smem > (32u << 10) &&
        (e = cudaFuncSetAttribute(k_knn_group<MULTI, F32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kGrpWarps * knn_group_bytes(knn_group_cap(1024), 1024)))) != cudaSuccess)
        return e;
    int per = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_knn_group<MULTI, F32>, kGrpThreads, smem) !=
            cudaSuccess ||
        per < 1)
        per = 1;
    if (blocks_per_sm > 0 && blocks_per_sm < per) per = blocks_per_sm;
    uint64_t grid = (uint64_t)sms * per;
    if (!g.grp) {
        const uint64_t want = (g.packets + kGrpWarps - 1) / kGrpWarps;
        if (want < grid) grid = want;
    }
    if (grid == 0) return cudaSuccess;
    k_knn_group<MULTI, F32><<<(int)grid, kGrpThreads, smem, s>>>(g);
    return cudaGetLastError();
}

// The search of a launch.  With seeding, every kKnnHeadStride-th query is a
// head: the heads go out first and start from their own nodes; every other
// query starts from those before it in its run or, when it leads its run, from
// the nearest head that has finished.  packet_ctr holds 3 counters (zeroed);
// head_kth one double per head, set to NaN here.  fp32: the FP32-filter form
// (every cloud of the launch has its centre-relative FP32 copy).
template <int MULTI>
cudaError_t launch_group_seeded(KnnGroupArgs g, uint32_t kmax, int sms, cudaStream_t s, int blocks_per_sm,
                                double* head_kth, size_t head_bytes, bool fp32) {
    g.heads = g.est > 0.0 && head_kth ? 1 : 0;
    g.head_kth = head_kth;
    if (g.heads) {
        const cudaError_t e = cudaMemsetAsync(head_kth, 0xff, head_bytes, s);
        if (e != cudaSuccess) return e;
    }
    if (fp32) return launch_group<MULTI, true>(g, kmax, sms, s, blocks_per_sm);
    return launch_group<MULTI, false>(g, kmax, sms, s, blocks_per_sm);
}

int sm_count_k(int device) {
    int v = 148;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
    return v;
}

}  // namespace

cudaError_t launch_knn_table(int device, cudaStream_t s, const DynGroup* d_grp, const SearchReq* single, uint64_t nq,
                             uint32_t kmax, const uint32_t* d_order, uint32_t bucket, uint32_t* d_idx, double* d_d2,
                             uint32_t* d_counts, uint32_t* d_err, int blocks_per_sm, double est) {
    if (!d_grp && nq == 0) return cudaSuccess;
    KnnTableArgs a{};
    a.single = single ? *single : SearchReq{};
    a.grp = d_grp;
    a.nq = nq;
    a.order = d_order;
    a.bucket = bucket;
    a.idx = d_idx;
    a.d2 = d_d2;
    a.counts = d_counts;
    a.err = d_err;
    a.est = est;
    const int sms = sm_count_k(device);
    const uint64_t cap = (uint64_t)sms * (blocks_per_sm > 0 ? blocks_per_sm : 16);
    const uint64_t want = d_grp ? cap : (nq + kKnnWarps - 1) / kKnnWarps;
    const int grid = (int)(want < cap ? want : cap);
    if (d_grp) {
        if (kmax > 64) {  // the shared-memory list kernel, blocks per SM as its list fits
            auto lgrid = [&](size_t smem) { return sms * (int)std::max<size_t>(1, (224u << 10) / (smem + 3072)); };
            if (kmax <= 128) return launch_l_table<128>(d_grp, d_order, bucket, d_idx, d_d2, d_counts, d_err,
                                                        lgrid(knn_smem<128>()), s);
            if (kmax <= 256) return launch_l_table<256>(d_grp, d_order, bucket, d_idx, d_d2, d_counts, d_err,
                                                        lgrid(knn_smem<256>()), s);
            if (kmax <= 512) return launch_l_table<512>(d_grp, d_order, bucket, d_idx, d_d2, d_counts, d_err,
                                                        lgrid(knn_smem<512>()), s);
            return launch_l_table<1024>(d_grp, d_order, bucket, d_idx, d_d2, d_counts, d_err, lgrid(knn_smem<1024>()),
                                        s);
        }
        if (single) {  // every request of the group on the cloud single->cv
            if (kmax <= 32) k_knn_reg<1, 2><<<grid, kKnnThreads, 0, s>>>(a);
            else k_knn_reg<2, 2><<<grid, kKnnThreads, 0, s>>>(a);
        } else {
            if (kmax <= 32) k_knn_reg<1, 1><<<grid, kKnnThreads, 0, s>>>(a);
            else k_knn_reg<2, 1><<<grid, kKnnThreads, 0, s>>>(a);
        }
    } else {
        if (kmax <= 32) k_knn_reg<1, 0><<<grid, kKnnThreads, 0, s>>>(a);
        else k_knn_reg<2, 0><<<grid, kKnnThreads, 0, s>>>(a);
    }
    return cudaGetLastError();
}

cudaError_t launch_knn_group_table(int device, cudaStream_t s, const DynGroup* d_grp, DynGroup* d_fb,
                                   const SearchReq* single, uint32_t kmax, const uint32_t* d_order, uint32_t bucket,
                                   uint32_t* d_idx, double* d_d2, uint32_t* d_counts, uint32_t* d_err,
                                   uint32_t* d_packet_ctr, uint32_t* d_fb_list, double est, uint32_t chunk,
                                   int blocks_per_sm, double* d_head_kth, size_t head_bytes, bool fp32,
                                   unsigned long long* d_stats) {
    if (kmax > 1024) return cudaErrorInvalidValue;
    cudaError_t e;
    if ((e = cudaMemsetAsync(d_packet_ctr, 0, 12, s)) != cudaSuccess) return e;
    // a batch whose radius results outgrew their arrays runs again from the same table: the queries handed back
    // are counted from 0 each time (the list has one entry a query)
    if ((e = cudaMemsetAsync(&d_fb->nq, 0, sizeof(d_fb->nq), s)) != cudaSuccess) return e;
    KnnGroupArgs g{};
    g.single = single ? *single : SearchReq{};
    g.grp = d_grp;
    g.order = d_order;
    g.bucket = bucket;
    g.idx = d_idx;
    g.d2 = d_d2;
    g.counts = d_counts;
    g.err = d_err;
    g.est = est;
    g.packet_ctr = d_packet_ctr;
    g.chunk = chunk > 0 ? chunk : 1;
    g.fb_list = d_fb_list;
    g.stats = d_stats;
    g.fb_count = reinterpret_cast<unsigned long long*>(&d_fb->nq);
    const int sms = sm_count_k(device);
    const int bps = blocks_per_sm;
    e = single ? launch_group_seeded<2>(g, kmax, sms, s, bps, d_head_kth, head_bytes, fp32)
               : launch_group_seeded<1>(g, kmax, sms, s, bps, d_head_kth, head_bytes, fp32);
    if (e != cudaSuccess) return e;
    // the queries handed back, exactly and without the provisional threshold
    return launch_knn_table(device, s, d_fb, single, 0, kmax, d_fb_list, bucket, d_idx, d_d2, d_counts, d_err,
                            bps, 0.0);
}

cudaError_t prepare_knn_dyn() {
    cudaError_t e;
    if ((e = cudaFuncSetAttribute(k_knn<128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)knn_smem<128>())) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_knn<256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)knn_smem<256>())) != cudaSuccess)
        return e;
    if ((e = cudaFuncSetAttribute(k_knn<512, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)knn_smem<512>())) != cudaSuccess)
        return e;
    return cudaFuncSetAttribute(k_knn<1024, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)knn_smem<1024>());
}

static SearchReq knn_request(const Cloud& c, const double* d_centers, uint64_t nq, uint32_t k) {
    SearchReq r{};
    r.cv = cloud_view(c);
    r.centers = d_centers;
    r.q_begin = 0;
    r.q_end = nq;
    r.k = k;
    return r;
}

static cudaError_t launch_list(const KnnArgs& a, uint32_t k, int grid, cudaStream_t s, bool carry) {
    if (k <= 32) return launch_l<32>(a, grid, s, carry);
    if (k <= 64) return launch_l<64>(a, grid, s, carry);
    if (k <= 128) return launch_l<128>(a, grid, s, carry);
    if (k <= 256) return launch_l<256>(a, grid, s, carry);
    if (k <= 512) return launch_l<512>(a, grid, s, carry);
    return launch_l<1024>(a, grid, s, carry);
}

cudaError_t launch_knn(Cloud& c, const double* d_centers, uint64_t nq, uint32_t k, uint32_t* d_idx, double* d_d2,
                       uint32_t* d_counts) {
    if (nq == 0 || k == 0) return cudaSuccess;
    KnnArgs a{};
    a.xs = c.xs.as<double>();
    a.ys = c.ys.as<double>();
    a.zs = c.zs.as<double>();
    a.offsets = c.offsets.as<uint32_t>();
    a.ranges = c.ranges.as<uint2>();
    a.centers = c.centers.as<double>();
    a.geom = reinterpret_cast<const LevelGeom*>(c.d_box.as<unsigned char>() + sizeof(BoxD));
    a.q = d_centers;
    a.nq = nq;
    a.k = k;
    a.idx = d_idx;
    a.d2 = d_d2;
    a.counts = d_counts;
    a.err = c.d_err.as<uint32_t>();
    a.bucket = c.packet ? c.knn_bucket : 0;  // the plain path descends to the leaves
    a.order = nullptr;
    if (c.packet) {  // curve-ordered queries: neighbouring warps share octants in cache
        cudaError_t e;
        if ((e = launch_query_order(c, d_centers, nq, &a.order)) != cudaSuccess) return e;
    }
    const uint64_t want = (nq + kKnnWarps - 1) / kKnnWarps;
    const uint64_t cap = (uint64_t)sm_count_k(c.device) * 16;
    const int grid = (int)(want < cap ? want : cap);
    if (c.packet && (k > 64 || c.knn_packet)) {
        // the FP32 filter (k <= 64): centre-relative FP32 points, built on first use
        cudaError_t e;
        const bool f32 = fp32_on_knn(c.fp32_filter) && k <= 64;
        if (f32 && !c.crel_built) {
            if ((e = launch_center_rel(c)) != cudaSuccess) return e;
            c.crel_built = true;
        }
        const SearchReq r = knn_request(c, d_centers, nq, k);
        // the curve-ordered search, then the exact sorted-list kernels for the queries it hands back
        if ((e = c.packet_ctr.reserve(256)) != cudaSuccess) return e;
        if ((e = c.knn_fb.reserve(16 + 4 * nq)) != cudaSuccess) return e;
        const size_t head_bytes = 8 * (nq / kKnnHeadStride + 1);
        if ((e = c.knn_heads.reserve(head_bytes)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(c.packet_ctr.ptr, 0, 12, c.stream)) != cudaSuccess) return e;
        if ((e = cudaMemsetAsync(c.knn_fb.ptr, 0, 8, c.stream)) != cudaSuccess) return e;
        KnnGroupArgs g{};
        g.single = r;
        g.grp = nullptr;
        g.packets = nq;
        g.order = a.order;
        g.bucket = c.knn_bucket;
        g.idx = d_idx;
        g.d2 = d_d2;
        g.counts = d_counts;
        g.err = c.d_err.as<uint32_t>();
        g.est = c.knn_est;
        g.packet_ctr = c.packet_ctr.as<uint32_t>();
        g.chunk = c.knn_chunk;
        g.fb_count = c.knn_fb.as<unsigned long long>();
        g.fb_list = reinterpret_cast<uint32_t*>(c.knn_fb.as<unsigned char>() + 16);
        g.stats = f32 ? c.stats.as<unsigned long long>() + 2 : nullptr;  // oct_knn_filter_stats
        const int sms = sm_count_k(c.device);
        double* heads = c.knn_heads.as<double>();
        KernelClock clk(c, 1);
        e = launch_group_seeded<0>(g, k, sms, c.stream, 0, heads, head_bytes, f32);
        clk.stop();
        if (e != cudaSuccess) return e;
        if (k > 64) {
            a.order = g.fb_list;
            a.nq_dev = g.fb_count;
            return launch_list(a, k, grid, c.stream, true);
        }
        KnnTableArgs f{};
        f.single = r;
        f.nq = nq;
        f.nq_dev = g.fb_count;
        f.order = g.fb_list;
        f.bucket = c.knn_bucket;
        f.idx = d_idx;
        f.d2 = d_d2;
        f.counts = d_counts;
        f.err = g.err;
        f.est = 0.0;  // exact without the provisional threshold
        if (k <= 32) k_knn_reg<1, 0><<<grid, kKnnThreads, 0, c.stream>>>(f);
        else k_knn_reg<2, 0><<<grid, kKnnThreads, 0, c.stream>>>(f);
        return cudaGetLastError();
    }
    if (c.packet) {  // k <= 64, one query per warp
        const SearchReq r = knn_request(c, d_centers, nq, k);
        return launch_knn_table(c.device, c.stream, nullptr, &r, nq, k, a.order, c.knn_bucket, d_idx, d_d2, d_counts,
                                c.d_err.as<uint32_t>(), 0, c.knn_est);
    }
    return launch_list(a, k, grid, c.stream, false);
}

// A kernel of this file's device code, for preload_kernels.
const void* kernel_anchor_knn_search() { return reinterpret_cast<const void*>(&k_knn_reg<2, 0>); }

}  // namespace octb
