// Batched ("packet") radius search: neighbors / neighborsPrune / neighborsStruct
// for 1 to 16 spatially ordered queries per warp (FP32 counts: to 32; packet_width).
//
// Reference path replaced: the same as radius_search.cu - singleTraversal
// (inc/structures/linear_octree.hpp:653-686) with the criteria and leaf actions of
// neighborsStruct (695-736), neighborsPrune (746-784) and neighbors (796-816).
//
// B200 design.  The query centres are first ordered along the cloud's curve
// (launch_query_order), so the queries of a warp are neighbours in space and
// need almost the same octants.  The warp walks the tree once for all of them:
// at every internal node the lanes judge the 8 children for four queries at a
// time (the reference's predicates, bit for bit), and a child is pushed with two
// masks - the queries for which it is fully inside (they get its whole range
// when it is popped) and those that must descend into it.  Pushing the
// children lowest octant last keeps every query's output in ascending order.
// Leaves (the transposed test): the lanes load 32 consecutive points of up to
// kLeafGroup neighbouring leaves and test them against one query of the leaves'
// masks at a time; the ballot is that query's hit mask, stored in one coalesced
// write, or cut into the runs that neighborsStruct returns.  Fully-inside ranges
// are written by the whole warp.  Packets are handed out by an atomic counter so
// that long and short packets balance.
//
// Bound: instruction issue (2.5k warp instructions per query at r = 2.5 on the
// 10M-point tile, DRAM below 5 % of peak): the pair loop takes about 1k of them,
// the child tests 0.6k.  500k queries there: 2122 us with one leaf at a time and
// one pass per four active queries, 1904 us with the leaf groups, 1638 us with
// the aligned fours (no bit search per query), 24-byte stack records and the
// one-chunk fast path of the hit store; 100k circles of 593 points over leaves
// of 32 on a 2M-point tile 1899 -> 1416 -> 1159 us; 50k neighborsStruct squares
// (count + fill, one lane per query over a leaf's points, then one pass of this
// form) 4.9 -> 1.2 ms.
//
// Output: count pass + scan + fill at the scanned offsets, or one pass in which
// every query appends its results to its own chain of 64-entry chunks (see
// k_radius_packet's CHUNK form) that k_chunk_compact moves into the CSR array.
//
// FP32 variant (the precision form): each sorted point also has FP32
// coordinates relative to its leaf's centre (x, y, z computed in FP64 and
// rounded once; w = their L1 norm).  A lane tests its query, made relative to
// the same centre, in FP32; a point whose FP32 result lies within a rigorous
// error band of the decision boundary is re-tested in FP64 on the original
// coordinates with the reference's expression, so every decision is still the
// reference's.  Band (sphere / circle, inside iff d2 < r2 / d2 <= r2):
//   |d2_fp32 - d2| <= 2^-23 (|q|_1 + |p|_1 + 1.74 r) r + 3 2^-24 d2 near the
//   boundary, plus 2^-24 r2 for rounding r2 to FP32; the band used is 2 to 4
//   times that:  2^-21 ((|q|_1 + |p|_1 + 2 r) r + r2).
// Cube / square: per axis, the interval bounds bmin = c - r and bmax = c + r
// (FP64) are made leaf-relative and rounded to FP32; an axis is certain when
// its margin exceeds 2^-22 (|p_i| + |bound_i|).
#include <algorithm>
#include <cfloat>

#include "cloud.h"
#include "search_kernels.cuh"

namespace octb {

namespace {

constexpr int kPkWarps = 4;
constexpr int kPkThreads = 32 * kPkWarps;
constexpr int kPkStack = 8 * (kMaxDepth + 1);
constexpr uint32_t kChunk = kResultChunk;  // entries per result chunk (one-pass mode)
constexpr uint32_t kNoChunk = 0xffffffffu;
constexpr uint32_t kNotOpen = 0xffffffffu;
constexpr int kLeafGroup = 8;  // leaves tested as one run of points

struct PacketArgs {
    SearchReq single;           // the request of a single-cloud search (grp == null); with
                                // one_cloud, single.cv is the cloud of every request of grp
    const DynGroup* grp;        // sizes and request table of a batch group (device)
    uint64_t packets;           // packets of a single-request launch
    uint32_t width;             // queries per packet of a single-request launch (1 to 16; FP32 counts: to 32)
    bool one_cloud;             // host dispatch: grp's requests all search single.cv
    const uint32_t* order;      // query visiting order (global positions), or null
    unsigned long long* counts;
    unsigned long long* counts2;
    const unsigned long long* offs;
    uint32_t* out;
    uint64_t out_cap;
    uint32_t* packet_ctr;
    unsigned long long* stats;  // [0] point tests, [1] FP64 re-tests
    uint32_t* err;
    // one-pass mode: each query's results go to its own chain of kChunk-entry chunks
    uint32_t* chunk_pool;       // chunk_cap x kChunk entries
    uint2* chunk_rec;           // the query position a chunk belongs to, its number in the query's chain (chunk_cap)
    uint32_t* chunk_ctr;        // chunks handed out
    uint32_t chunk_cap;
};

// Per-lane FP32 context of one leaf.
struct LeafCtx {
    float qx, qy, qz;  // query centre relative to the leaf centre
    float r2f;         // radius^2 rounded to FP32 (sphere, circle)
    float b0, b1;      // band = b0 + b1 * |p|_1 (sphere, circle)
    float lo[3], hi[3], tlo[3], thi[3];  // relative interval bounds and their tolerances (cube, square)
};

template <int KT>
__device__ __forceinline__ void leaf_ctx(const SearchKernel& k, const double* lc, LeafCtx& c) {
    c.qx = (float)dsub(k.c[0], lc[0]);
    c.qy = (float)dsub(k.c[1], lc[1]);
    c.qz = (float)dsub(k.c[2], lc[2]);
    const float r = (float)k.r;
    if constexpr (KT == kSphere || KT == kCircle) {
        const float q1 = fabsf(c.qx) + fabsf(c.qy) + ((KT == kSphere) ? fabsf(c.qz) : 0.0f);
        c.r2f = (float)k.r2;
        const float s = 4.76837158203125e-07f;  // 2^-21
        c.b0 = s * ((q1 + 2.0f * r) * r + c.r2f) + FLT_MIN;
        c.b1 = s * r;
    } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            c.lo[a] = (float)dsub(k.bmin[a], lc[a]);
            c.hi[a] = (float)dsub(k.bmax[a], lc[a]);
            c.tlo[a] = 2.384185791015625e-07f * fabsf(c.lo[a]);  // 2^-22 |bound|
            c.thi[a] = 2.384185791015625e-07f * fabsf(c.hi[a]);
        }
    }
}

// FP32 test: 1 inside, 0 outside, -1 undecided (re-test in FP64).
template <int KT>
__device__ __forceinline__ int f32_test(const LeafCtx& c, float4 p) {
    if constexpr (KT == kSphere || KT == kCircle) {
        const float dx = p.x - c.qx, dy = p.y - c.qy;
        float d2 = __fmaf_rn(dy, dy, __fmul_rn(dx, dx));
        if constexpr (KT == kSphere) {
            const float dz = p.z - c.qz;
            d2 = __fmaf_rn(dz, dz, d2);
        }
        const float band = __fmaf_rn(c.b1, p.w, c.b0);
        if (d2 < c.r2f - band) return 1;
        if (d2 > c.r2f + band) return 0;
        return -1;
    } else {
        constexpr int D = (KT == kCube) ? 3 : 2;
        const float pv[3] = {p.x, p.y, p.z};
        const float tp = 2.384185791015625e-07f * p.w;  // 2^-22 |p|_1 >= 2^-22 |p_i|
        bool sure_in = true;
#pragma unroll
        for (int a = 0; a < D; ++a) {
            const float ml = pv[a] - c.lo[a], mh = c.hi[a] - pv[a];
            const float tl = tp + c.tlo[a], th = tp + c.thi[a];
            if (ml < -tl || mh < -th) return 0;
            sure_in = sure_in && (ml > tl) && (mh > th);
        }
        return sure_in ? 1 : -1;
    }
}

// MULTI 0: one request, read from the kernel parameters (constant-bank
// operands, no registers held).  1: a request table; the cloud pointers of the
// warp's current request live in shared memory (RQV), so the hot loops do not
// re-load them from the table.  2: a request table whose requests are all on
// one cloud, whose pointers are kernel parameters again (no shared-memory
// reads in the hot loops).
#define RQ(f) (MULTI ? reqs[cur_req].f : a.single.f)
#define RQV(f) (MULTI == 1 ? s_view[warp].f : a.single.cv.f)

// Query parameters of lane j for the transposed leaf and child tests, one
// 48-byte row per query so that a test reads them with 16-byte loads: sphere /
// circle (c0, c1, c2, r2, r, -), cube / square (bmin0..2, bmax0..2).
constexpr int kQpRow = 6;
__device__ __forceinline__ double2 ld_d2(const double* p) { return *reinterpret_cast<const double2*>(p); }
__device__ __forceinline__ float4 ld_f4(const float* p) { return *reinterpret_cast<const float4*>(p); }

template <int KT>
__device__ __forceinline__ void put_query(double (*q)[kQpRow], int lane, const SearchKernel& k) {
    if constexpr (KT == kSphere || KT == kCircle) {
        q[lane][0] = k.c[0];
        q[lane][1] = k.c[1];
        q[lane][2] = k.c[2];
        q[lane][3] = k.r2;
        q[lane][4] = k.r;
    } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            q[lane][a] = k.bmin[a];
            q[lane][3 + a] = k.bmax[a];
        }
    }
}

// Lane j's SearchKernel back from put_query's copy: the fields the box tests,
// the leaf tests and the FP32 context read (bounds of a sphere / circle are
// recomputed by init's own expressions, so they are the same values).
template <int KT>
__device__ __forceinline__ SearchKernel kernel_of(const double (*q)[kQpRow], int j) {
    SearchKernel k;
    if constexpr (KT == kSphere || KT == kCircle) {
        const double2 a = ld_d2(&q[j][0]), b = ld_d2(&q[j][2]);
        k.c[0] = a.x;
        k.c[1] = a.y;
        k.c[2] = b.x;
        k.r2 = b.y;
        k.r = q[j][4];
#pragma unroll
        for (int a2 = 0; a2 < 3; ++a2) {
            k.bmin[a2] = dsub(k.c[a2], k.r);
            k.bmax[a2] = dadd(k.c[a2], k.r);
        }
    } else {  // cube / square tests read the bounds only
        const double2 a = ld_d2(&q[j][0]), b = ld_d2(&q[j][2]), c = ld_d2(&q[j][4]);
        k.r = k.r2 = 0.0;
        k.c[0] = k.c[1] = k.c[2] = 0.0;
        k.bmin[0] = a.x;
        k.bmin[1] = a.y;
        k.bmin[2] = b.x;
        k.bmax[0] = b.y;
        k.bmax[1] = c.x;
        k.bmax[2] = c.y;
    }
    return k;
}

// FP32 leaf context of lane j's query for the transposed FP32 test, one row
// per query: sphere / circle (qx, qy, qz, r2f | b0, b1, -, -), cube / square
// (lo0..2, hi0 | hi1, hi2, tlo0, tlo1 | tlo2, thi0..2).
template <int KT>
__device__ __forceinline__ void put_ctx(float* row, const LeafCtx& c) {
    if constexpr (KT == kSphere || KT == kCircle) {
        row[0] = c.qx;
        row[1] = c.qy;
        row[2] = c.qz;
        row[3] = c.r2f;
        row[4] = c.b0;
        row[5] = c.b1;
    } else {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            row[a] = c.lo[a];
            row[3 + a] = c.hi[a];
            row[6 + a] = c.tlo[a];
            row[9 + a] = c.thi[a];
        }
    }
}
template <int KT>
__device__ __forceinline__ LeafCtx get_ctx(const float* row) {
    LeafCtx c;
    if constexpr (KT == kSphere || KT == kCircle) {
        const float4 a = ld_f4(row);
        const float2 b = *reinterpret_cast<const float2*>(row + 4);
        c.qx = a.x;
        c.qy = a.y;
        c.qz = a.z;
        c.r2f = a.w;
        c.b0 = b.x;
        c.b1 = b.y;
    } else {
        const float4 a = ld_f4(row), b = ld_f4(row + 4), d = ld_f4(row + 8);
        c.lo[0] = a.x;
        c.lo[1] = a.y;
        c.lo[2] = a.z;
        c.hi[0] = a.w;
        c.hi[1] = b.x;
        c.hi[2] = b.y;
        c.tlo[0] = b.z;
        c.tlo[1] = b.w;
        c.tlo[2] = d.x;
        c.thi[0] = d.y;
        c.thi[1] = d.z;
        c.thi[2] = d.w;
    }
    return c;
}

// Bits 0, 8, 16 and 24 of x as a 4-bit number (the products land on distinct bits: no carries).
__device__ __forceinline__ uint32_t four_bits(uint32_t x) { return (((x & 0x01010101u) * 0x01020408u) >> 24) & 15u; }

// is_inside of lane j's query for point p: the same expressions, operand for operand.
template <int KT>
__device__ __forceinline__ bool inside_of(const double (*q)[kQpRow], int j, double px, double py, double pz) {
    if constexpr (KT == kSphere) {
        const double2 a = ld_d2(&q[j][0]), b = ld_d2(&q[j][2]);
        return dsq3(dsub(px, a.x), dsub(py, a.y), dsub(pz, b.x)) < b.y;
    } else if constexpr (KT == kCircle) {
        const double2 a = ld_d2(&q[j][0]), b = ld_d2(&q[j][2]);
        return dsq2(dsub(px, a.x), dsub(py, a.y)) <= b.y;
    } else {
        const double2 a = ld_d2(&q[j][0]), b = ld_d2(&q[j][2]), c = ld_d2(&q[j][4]);
        // bmin = (a.x, a.y, b.x), bmax = (b.y, c.x, c.y)
        if constexpr (KT == kCube)
            return px >= a.x && px <= b.y && py >= a.y && py <= c.x && pz >= b.x && pz <= c.y;
        else
            return px >= a.x && px <= b.y && py >= a.y && py <= c.x;
    }
}

// MODE 0 counts, 1 fills at scanned offsets, 2 (one pass) appends each query's
// results to its own chain of kChunk-entry chunks taken from a pool (contiguous
// chunks for one long range, so positions stay linear); per query the count is
// written, per chunk its query and its number in the chain, and k_chunk_compact
// moves every chunk into the CSR array after the scan.  A neighborsStruct range
// takes two entries.
//
// Leaves are tested in groups: up to kLeafGroup leaves that are next on the stack
// (ascending, possibly with gaps) form one run of points, 32 of them on the lanes
// at a time, each lane with its own leaf's query masks.  Leaves hold 10 to 30
// points (empty octants are dropped), so a leaf at a time leaves half the lanes
// idle and pays a stack pop per leaf.
template <int KT, int ALGO, int MODE, bool F32, int MULTI>
__global__ void __launch_bounds__(kPkThreads) k_radius_packet(PacketArgs a) {
    // The leaf test is transposed: the lanes hold consecutive points and test them
    // against one query of the masks at a time, so every lane does useful work and
    // the ballot is that query's hit mask.  The FP32 form reads the points'
    // leaf-relative coordinates and each query's context for the leaf (made once
    // per leaf by the query's own lane, so its groups are single leaves); a point
    // inside the error band is re-tested in FP64.
    constexpr bool kRanges = (ALGO == kStruct);
    constexpr bool kChain = (MODE == 2);
    constexpr int kGroup = F32 ? 1 : kLeafGroup;
    constexpr int kCtxF = (KT == kSphere || KT == kCircle) ? 8 : 12;  // floats of a query's FP32 leaf context row
    __shared__ __align__(16) float s_ctx[F32 ? kPkWarps : 1][32][kCtxF];
    __shared__ CloudView s_view[MULTI == 1 ? kPkWarps : 1];
    __shared__ uint32_t st_node[F32 ? kPkWarps : 1][kPkStack];
    __shared__ uint4 st_nd[kPkWarps][kPkStack];  // first child (0 for a leaf), point range, depth
    __shared__ uint2 st_qm[kPkWarps][kPkStack];  // query masks: overlapping, fully inside
    __shared__ double s_rad[kPkWarps][kMaxDepth + 1][3];
    __shared__ __align__(16) double s_qp[kPkWarps][32][kQpRow];

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double (*s_radii)[3] = s_rad[warp];
    uint32_t cur_cloud = 0xffffffffu;
    uint32_t cur_req = 0;
    const SearchReq* reqs = nullptr;
    uint32_t nreq = 1;
    uint64_t packets = a.packets;
    uint32_t width = a.width;
    if (MULTI) {
        reqs = a.grp->reqs;
        nreq = a.grp->nreq;
        packets = a.grp->packets;
        width = a.grp->width;
    }
    const uint32_t lbit = 1u << lane;
    uint32_t* sn = st_node[F32 ? warp : 0];
    uint4* sf = st_nd[warp];
    uint2* sm = st_qm[warp];
    unsigned long long n_tests = 0, n_retests = 0;
    bool dry = false;  // the chunk pool has run out

    for (;;) {
        uint32_t packet = 0;
        if (lane == 0) packet = atomicAdd(a.packet_ctr, 1u);
        packet = __shfl_sync(0xffffffffu, packet, 0);
        if (packet >= packets) break;
        // the request of this packet: packet_begin is ascending over the table
        if (MULTI) {
            uint32_t lo = 0, hi = nreq;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (reqs[mid].packet_begin <= packet) lo = mid;
                else hi = mid;
            }
            cur_req = lo;
        }
        if (RQ(cloud_id) != cur_cloud) {  // this warp's level radii and cloud follow the packet's cloud
            __syncwarp();
            const double* gr = &RQ(cv.geom)->radii[0][0];
            for (int t = lane; t < (kMaxDepth + 1) * 3; t += 32) (&s_radii[0][0])[t] = gr[t];
            if (MULTI == 1 && lane == 0) s_view[warp] = reqs[cur_req].cv;
            cur_cloud = RQ(cloud_id);
            __syncwarp();
        }
        const uint64_t q_begin = RQ(q_begin);
        const uint64_t i = q_begin + (uint64_t)width * (packet - RQ(packet_begin)) + lane;
        const bool valid = (uint32_t)lane < width && i < RQ(q_end);
        const uint64_t qg = valid ? (a.order ? (uint64_t)a.order[i] : i) : q_begin;  // global query position
        const uint64_t ql = qg - q_begin;                                              // within the request
        const uint32_t qi = (uint32_t)qg;
        const double* qc = RQ(centers);
        const double* qrad = RQ(radii);
        const uint32_t approx_cut = kRanges ? RQ(approx_cut) : 0u;
        const bool approx_upper = kRanges && RQ(approx_upper) != 0;
        SearchKernel k;
        k.init(qc[3 * ql], qc[3 * ql + 1], qc[3 * ql + 2], qrad ? qrad[ql] : RQ(radius));
        __syncwarp();  // the previous packet's reads of s_qp are done
        put_query<KT>(s_qp[warp], lane, k);  // read by the other lanes after a __syncwarp
        // per lane (its own query): results (ranges for neighborsStruct), points of the ranges,
        // where the fill starts
        uint32_t cnt = 0, cnt2 = 0;
        unsigned long long base = 0;
        if (MODE == 1 && valid) base = a.offs[qi];
        bool overflow = false;
        uint32_t open_at = kNotOpen;  // neighborsStruct: first point of the run that crosses into the next 32 points
        // one-pass mode: this lane's chain (current chunk, entries used in it); its chunks are full up to the
        // current one, so the count says how many there are
        uint32_t ck_cur = kNoChunk, ck_fill = kChunk;

        // Reserve n > 0 entries at the end of lane j's chain (warp-uniform call):
        // returns where they go - the first `room` continue chunk `cur`, the rest
        // are linear from chunk `nc` on (new chunks taken as one contiguous run).
        // A pool that is too small leaves the chain full: nothing more is stored,
        // the counts stay exact and the host runs again.  A warp that has met its
        // end does not ask again: with every further hit asking the one counter, a
        // batch over 16 clouds whose pool held half the results was searched in
        // 8.7 ms (4.1 with room), and the first batch of an engine took 37.3 ms
        // where it takes 32.4.
        struct ChunkPos {
            uint32_t cur, fill, room, nc;
        };
        auto chain_len = [&]() -> uint32_t {  // before the results being added are counted
            return kRanges ? (cnt + kChunk / 2 - 1) / (kChunk / 2) : (cnt + kChunk - 1) / kChunk;
        };
        auto chunk_reserve = [&](int j, uint32_t n) -> ChunkPos {
            ChunkPos p;
            p.cur = __shfl_sync(0xffffffffu, ck_cur, j);
            p.fill = __shfl_sync(0xffffffffu, ck_fill, j);
            p.room = kChunk - p.fill;
            p.nc = kNoChunk;
            if (n > p.room) {
                const uint32_t m = (n - p.room + kChunk - 1) / kChunk;
                uint32_t nc = kNoChunk;  // (above any capacity)
                if (lane == j && !dry) nc = atomicAdd(a.chunk_ctr, m);
                nc = __shfl_sync(0xffffffffu, nc, j);
                const bool fits = (uint64_t)nc + m <= a.chunk_cap;
                if (fits) {
                    p.nc = nc;
                    if (m > 1) {  // the chunks after the first, which is lane j's to record
                        const uint32_t owner = __shfl_sync(0xffffffffu, qi, j), num = __shfl_sync(0xffffffffu, chain_len(), j);
                        for (uint32_t t = 1 + lane; t < m; t += 32) {
                            a.chunk_rec[nc + t] = make_uint2(owner, num + t);
                        }
                    }
                } else {
                    dry = true;
                }
                if (lane == j) {
                    if (fits) {
                        a.chunk_rec[nc] = make_uint2(qi, chain_len());
                        ck_cur = nc + m - 1;
                        ck_fill = n - p.room - (m - 1) * kChunk;
                    } else {
                        ck_fill = kChunk;
                    }
                }
            } else if (lane == j) {
                ck_fill += n;
            }
            return p;
        };
        auto chunk_store = [&](const ChunkPos& p, uint32_t r, uint32_t v) {
            if (r < p.room) a.chunk_pool[(uint64_t)p.cur * kChunk + p.fill + r] = v;
            else if (p.nc != kNoChunk) a.chunk_pool[(uint64_t)p.nc * kChunk + (r - p.room)] = v;
        };
        // neighborsStruct, a range to the lane's own query (lanes diverge): chunks hold whole pairs
        auto lane_range = [&](uint32_t f, uint32_t l) {
            if (MODE == 1) {
                const unsigned long long o = base + cnt;
                if (o < a.out_cap) {
                    a.out[2 * o] = f;
                    a.out[2 * o + 1] = l;
                } else {
                    overflow = true;
                }
            }
            if (kChain) {
                bool room = ck_fill < kChunk;
                if (!room) {
                    const uint32_t nc = dry ? kNoChunk : atomicAdd(a.chunk_ctr, 1u);
                    if (nc < a.chunk_cap) {
                        a.chunk_rec[nc] = make_uint2(qi, chain_len());
                        ck_cur = nc;
                        ck_fill = 0;
                        room = true;
                    } else {
                        dry = true;
                    }
                }
                if (room) {
                    uint32_t* d = a.chunk_pool + (uint64_t)ck_cur * kChunk + ck_fill;
                    d[0] = f;
                    d[1] = l;
                    ck_fill += 2;
                }
            }
            cnt += 1;
            cnt2 += l - f;
        };

        // Query j's hits among the lanes' points (lane's point `idx`): appended in ascending order.
        // neighborsStruct: starts bit v = lane v is the first point of its leaf, cont = lane 31's leaf
        // goes on in the next 32 points; the maximal runs inside one leaf become ranges.
        auto take = [&](int j, bool in, uint32_t idx, uint32_t starts, bool cont) {
            const uint32_t hb = __ballot_sync(0xffffffffu, in);
            if constexpr (!kRanges) {
                (void)starts;
                (void)cont;
                if (!hb) return;
                const uint32_t n = __popc(hb), rank = __popc(hb & lanemask_lt());
                if constexpr (kChain) {
                    const uint32_t fill = __shfl_sync(0xffffffffu, ck_fill, j);
                    if (fill + n <= kChunk) {
                        const uint32_t cur = __shfl_sync(0xffffffffu, ck_cur, j);
                        if (in) a.chunk_pool[(uint64_t)cur * kChunk + (fill + rank)] = idx;
                        if (lane == j) ck_fill = fill + n;
                    } else {
                        const ChunkPos p = chunk_reserve(j, n);
                        if (in) chunk_store(p, rank, idx);
                    }
                } else if constexpr (MODE == 1) {
                    const unsigned long long o = __shfl_sync(0xffffffffu, base + cnt, j) + rank;
                    if (in) {
                        if (o < a.out_cap) a.out[o] = idx;
                        else overflow = true;
                    }
                }
                if (lane == j) cnt += n;
            } else {
                const uint32_t oa = __shfl_sync(0xffffffffu, open_at, j);
                const bool opened = oa != kNotOpen;
                if (!hb && !opened) return;
                const uint32_t rs = hb & (~(hb << 1) | starts) & ~(opened ? 1u : 0u);  // first points of runs
                uint32_t re = hb & (~(hb >> 1) | (starts >> 1));                       // last points of runs
                const bool stays = cont && (hb >> 31);
                if (stays) re &= 0x7fffffffu;
                const uint32_t closed = (opened && !(hb & 1u)) ? 1u : 0u;  // the open run ended with the last 32 points
                const uint32_t m = __popc(re) + closed;
                if (MODE != 0 && m) {
                    const uint32_t below = rs & (lanemask_lt() | lbit);
                    const uint32_t f = below ? idx - (uint32_t)(lane - (31 - __clz(below))) : oa;
                    const uint32_t r = closed + __popc(re & lanemask_lt());
                    const bool ends = (re >> lane) & 1u;
                    if constexpr (kChain) {
                        const ChunkPos p = chunk_reserve(j, 2 * m);
                        if (closed && lane == 0) {
                            chunk_store(p, 0, oa);
                            chunk_store(p, 1, idx);
                        }
                        if (ends) {
                            chunk_store(p, 2 * r, f);
                            chunk_store(p, 2 * r + 1, idx + 1);
                        }
                    } else {
                        const unsigned long long o = __shfl_sync(0xffffffffu, base + cnt, j);
                        if (o + m <= a.out_cap) {
                            if (closed && lane == 0) {
                                a.out[2 * o] = oa;
                                a.out[2 * o + 1] = idx;
                            }
                            if (ends) {
                                a.out[2 * (o + r)] = f;
                                a.out[2 * (o + r) + 1] = idx + 1;
                            }
                        } else {
                            overflow = true;
                        }
                    }
                }
                uint32_t next_open = kNotOpen;
                if (stays) {
                    const uint32_t last = __shfl_sync(0xffffffffu, idx, 31);
                    next_open = rs ? last - (uint32_t)__clz(rs) : oa;
                }
                if (lane == j) {
                    cnt += m;
                    cnt2 += __popc(hb);
                    open_at = next_open;
                }
            }
        };

        // The `g` leaves from stack slot `top` down: their points against the queries that overlap them
        // (lanes < g hold the leaves' ranges and masks).
        auto scan_leaves = [&](int top, int g) {
            uint2 rg = make_uint2(0u, 0u);
            uint32_t lo = 0, li = 0;
            if (lane < g) {
                const uint4 nd = sf[top - lane];
                const uint2 qm = sm[top - lane];
                rg = make_uint2(nd.y, nd.z);
                lo = qm.x;
                li = qm.y;
                n_tests += (unsigned long long)__popc(lo) * (rg.y - rg.x);
            }
            if constexpr (F32) {  // each query of the leaf's mask: its context, from its own lane
                const uint32_t mask = __shfl_sync(0xffffffffu, lo, 0);
                const uint32_t node = sn[top];
                __syncwarp();
                if ((mask >> lane) & 1u) {
                    LeafCtx ctx;
                    leaf_ctx<KT>(kernel_of<KT>(s_qp[warp], lane), RQV(centers) + 3ull * node, ctx);
                    put_ctx<KT>(s_ctx[warp][lane], ctx);
                }
                __syncwarp();
            }
            // first: the leaves' points as one run; leaf l holds [first, first + length) of it
            const uint32_t len = rg.y - rg.x;
            if (MODE == 0 && !kRanges && __any_sync(0xffffffffu, li != 0)) {
                // counted: a leaf's points for all the queries that hold it at once (one query at a time: FP32 counts
                // of 100k cubes of 6 m on a dense tile 2524 us, so 2345; FP64 1424, 1259)
                for (int l = 0; l < g; ++l) {
                    const uint32_t mask = __shfl_sync(0xffffffffu, li, l), n = __shfl_sync(0xffffffffu, len, l);
                    if (mask & lbit) cnt += n;
                }
                li = 0;
            }
            uint32_t end = len;
#pragma unroll
            for (int off = 1; off < kGroup; off <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, end, off);
                if (lane >= off) end += y;
            }
            const uint32_t first = end - len;
            const uint32_t total = __shfl_sync(0xffffffffu, end, kGroup - 1);  // lanes g .. kGroup - 1 add 0
            for (uint32_t b = 0; b < total; b += 32) {
                const uint32_t v = b + lane;
                const bool in_range = v < total;
                uint32_t idx, mo, mi, uni, starts = 0;
                bool cont = false;
                if constexpr (kGroup == 1) {
                    idx = __shfl_sync(0xffffffffu, rg.x, 0) + v;
                    mo = __shfl_sync(0xffffffffu, lo, 0);
                    mi = __shfl_sync(0xffffffffu, li, 0);
                    uni = mo | mi;
                    if (kRanges) {
                        starts = b == 0 ? 1u : 0u;
                        cont = total > b + 32;
                    }
                } else {
                    // the lane's leaf: leaves begun before b, plus those that begin at or below the lane
                    const bool is = lane < g;
                    const uint32_t before = __popc(__ballot_sync(0xffffffffu, is && first < b));
                    const bool here = is && first >= b && first < b + 32;
                    starts = __reduce_or_sync(0xffffffffu, here ? 1u << (first - b) : 0u);
                    const int e = (int)(before + __popc(starts & (lanemask_lt() | lbit))) - 1;
                    idx = __shfl_sync(0xffffffffu, rg.x - first, e) + v;
                    mo = __shfl_sync(0xffffffffu, lo, e);
                    mi = __shfl_sync(0xffffffffu, li, e);
                    uni = __reduce_or_sync(0xffffffffu, (is && first < b + 32 && end > b) ? (lo | li) : 0u);
                    if (kRanges) cont = __any_sync(0xffffffffu, is && first < b + 32 && end > b + 32);
                }
                double px = 0.0, py = 0.0, pz = 0.0;
                float4 pf = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (in_range) {
                    if constexpr (F32) {
                        pf = RQV(rel)[idx];
                    } else {
                        px = RQV(xs)[idx];
                        py = RQV(ys)[idx];
                        pz = RQV(zs)[idx];
                    }
                } else {
                    mo = mi = 0;
                }
                for (uint32_t rem = uni; rem;) {
                    const int j = 31 - __clz(rem);
                    const uint32_t jb = 1u << j;
                    rem ^= jb;
                    if constexpr (F32) {
                        bool in = (mi & jb) != 0;
                        if (mo & jb) {
                            const int r = f32_test<KT>(get_ctx<KT>(s_ctx[warp][j]), pf);
                            if (r < 0) {  // inside the error band: the reference's FP64 expression decides
                                in = inside_of<KT>(s_qp[warp], j, RQV(xs)[idx], RQV(ys)[idx], RQV(zs)[idx]);
                                ++n_retests;
                            } else {
                                in = r > 0;
                            }
                        }
                        take(j, in, idx, starts, cont);
                    } else {
                        // two queries at a time: their FP64 tests are independent, so their latencies
                        // overlap instead of adding up
                        const int j2 = rem ? 31 - __clz(rem) : j;
                        const uint32_t jb2 = rem ? 1u << j2 : 0u;
                        rem ^= jb2;
                        const bool t1 = inside_of<KT>(s_qp[warp], j, px, py, pz);
                        const bool t2 = inside_of<KT>(s_qp[warp], j2, px, py, pz);
                        take(j, ((t1 ? mo : mi) | mi) & jb, idx, starts, cont);
                        if (jb2) take(j2, ((t2 ? mo : mi) | mi) & jb2, idx, starts, cont);
                    }
                }
            }
        };

        // root: continuationCriterion(0, 0)
        bool over = false, in = false;
        if (valid) {
            if constexpr (ALGO == kNeighbors) {
                over = box_overlap<KT>(k, RQV(centers), s_radii[0]);
            } else {
                const int j = box_intersect<KT>(k, RQV(centers), s_radii[0]);
                in = (j == kInside);
                over = (j == kOverlap);
            }
        }
        int sp_top = 0;
        {
            const uint32_t mo = __ballot_sync(0xffffffffu, over);
            const uint32_t mi = __ballot_sync(0xffffffffu, in);
            if (mo | mi) {
                const uint32_t fc0 = RQV(offsets)[0];
                const uint2 rg0 = RQV(ranges)[0];
                if (lane == 0) {
                    if (F32) sn[0] = 0;
                    sf[0] = make_uint4(fc0, rg0.x, rg0.y, 0u);
                    sm[0] = make_uint2(mo, mi);
                }
                sp_top = 1;
            }
        }
        __syncwarp();
        while (sp_top > 0) {
            --sp_top;
            const uint4 nd = sf[sp_top];
            const uint32_t fc = nd.x;
            const uint2 nrg = make_uint2(nd.y, nd.z);
            if (fc == 0 && nrg.x != nrg.y) {
                // a leaf: with it the leaves that follow on the stack
                int g = 1;
                if (kGroup > 1) {
                    const int s = sp_top - lane;
                    bool leaf = lane < kGroup && s >= 0 && sf[s].x == 0;
                    if (kRanges && leaf) leaf = sf[s].y != sf[s].z;  // an empty inside leaf adds its own empty range
                    g = __ffs(~__ballot_sync(0xffffffffu, leaf)) - 1;
                }
                scan_leaves(sp_top, g);
                sp_top -= g - 1;
                __syncwarp();
                continue;
            }
            const uint2 qm = sm[sp_top];
            const uint32_t mo = qm.x, mi = qm.y, depth = nd.w;
            __syncwarp();
            if constexpr (kRanges) {
                if (mi & lbit) lane_range(nrg.x, nrg.y);
            } else if (mi) {
                // a fully-inside node: every lane of mi adds the node's whole range; the
                // warp writes it for one lane at a time, 32 consecutive indices per store
                const uint32_t len = nrg.y - nrg.x;
                if (MODE != 0 && len) {
                    uint32_t rem = mi;
                    while (rem) {
                        const int j = __ffs(rem) - 1;
                        rem &= rem - 1;
                        if constexpr (kChain) {
                            const ChunkPos p = chunk_reserve(j, len);
                            for (uint32_t t = lane; t < len; t += 32) chunk_store(p, t, nrg.x + t);
                        } else {
                            const unsigned long long o0 = __shfl_sync(0xffffffffu, base + cnt, j);
                            for (uint32_t t = lane; t < len; t += 32) {
                                const unsigned long long o = o0 + t;
                                if (o < a.out_cap) a.out[o] = nrg.x + t;
                                else overflow = true;
                            }
                        }
                    }
                }
                if (mi & lbit) cnt += len;
            }
            if (mo == 0 || fc == 0) continue;
            const uint32_t cd = depth + 1;
            // lane j (< 8) keeps child j's first-child link, range and lane masks
            uint32_t my_fc = 0, my_mo = 0, my_mi = 0;
            uint2 my_rg = make_uint2(0u, 0u);
            if (lane < 8) {
                my_fc = RQV(offsets)[fc + lane];
                my_rg = RQV(ranges)[fc + lane];
            }
            // neighborsApprox (linear_octree.hpp:979-985): below its precision level a
            // child is cut before any box test, its whole range added in upper-bound mode
            const bool cut = kRanges && approx_cut != 0 && cd >= approx_cut;
            {
                // child tests transposed: lane = (query slot lane / 8, child lane % 8), four
                // consecutive queries of the packet at a time (those next to each other on the
                // curve mostly reach the same nodes), skipping fours the node does not concern;
                // each lane tests with the query's own SearchKernel and the child's centre, as
                // the per-query walk does
                const double* ocp = RQV(centers) + 3ull * (fc + (lane & 7));
                const double oc[3] = {ocp[0], ocp[1], ocp[2]};
                int q0 = 0;
                for (uint32_t rem = mo; rem; rem >>= 4, q0 += 4) {
                    if (!(rem & 15u)) continue;
                    bool o = false, n = false;
                    const SearchKernel kq = kernel_of<KT>(s_qp[warp], q0 + (lane >> 3));
                    if constexpr (ALGO == kNeighbors) {
                        o = box_overlap<KT>(kq, oc, s_radii[cd]);
                    } else if (cut) {
                        n = approx_upper;
                    } else {
                        const int jj = box_intersect<KT>(kq, oc, s_radii[cd]);
                        n = (jj == kInside);
                        o = (jj == kOverlap);
                    }
                    // bit 8 s + c of a ballot: query q0 + s against child c; lane c gathers its four bits
                    const uint32_t bo = __ballot_sync(0xffffffffu, o);
                    my_mo |= four_bits(bo >> (lane & 7)) << q0;
                    if constexpr (ALGO != kNeighbors) {
                        const uint32_t bi = __ballot_sync(0xffffffffu, n);
                        my_mi |= four_bits(bi >> (lane & 7)) << q0;
                    }
                }
                my_mo &= mo;
                my_mi &= mo;
            }
            if (lane < 8 && my_fc == 0 && my_rg.x == my_rg.y) {  // empty leaf: nothing to scan or add
                my_mo = 0;
                if (!kRanges) my_mi = 0;  // neighborsStruct still adds its empty range
            }
            const uint32_t pushm = __ballot_sync(0xffffffffu, lane < 8 && (my_mo | my_mi) != 0);
            const int np = __popc(pushm);
            if (sp_top + np > kPkStack) {
                overflow = true;
                break;
            }
            if ((pushm >> lane) & 1u) {
                // lowest octant on top of the stack
                const int slot = sp_top + __popc(pushm >> (lane + 1));
                if (F32) sn[slot] = fc + lane;
                sf[slot] = make_uint4(my_fc, my_rg.x, my_rg.y, cd);
                sm[slot] = make_uint2(my_mo, my_mi);
            }
            __syncwarp();
            sp_top += np;
        }
        if (overflow) set_err(a.err, MODE == 1 ? kErrOutputCapacity : kErrStackOverflow);
        if (MODE != 1 && valid) {
            a.counts[qi] = cnt;
            if (kRanges) a.counts2[qi] = cnt2;
        }
        __syncwarp();
    }
    if (kChain && __any_sync(0xffffffffu, dry) && lane == 0) set_err(a.err, kErrChunkCapacity);
    if (a.stats) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            n_tests += __shfl_down_sync(0xffffffffu, n_tests, off);
            n_retests += __shfl_down_sync(0xffffffffu, n_retests, off);
        }
        if (lane == 0) {
            atomicAdd(&a.stats[0], n_tests);
            atomicAdd(&a.stats[1], n_retests);
        }
    }
}

// FP32 leaf-relative coordinates: one warp per node; leaves write their points.
__global__ void k_leaf_rel(const double* __restrict__ xs, const double* __restrict__ ys,
                           const double* __restrict__ zs, const uint32_t* __restrict__ offsets,
                           const uint2* __restrict__ ranges, const double* __restrict__ centers, uint32_t n_total,
                           float4* __restrict__ rel) {
    const uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= n_total) return;
    const uint32_t node = (uint32_t)w;
    if (offsets[node] != 0) return;
    const uint2 rg = ranges[node];
    const double cx = centers[3ull * node], cy = centers[3ull * node + 1], cz = centers[3ull * node + 2];
    for (uint32_t i = rg.x + lane; i < rg.y; i += 32) {
        float4 v;
        v.x = (float)dsub(xs[i], cx);
        v.y = (float)dsub(ys[i], cy);
        v.z = (float)dsub(zs[i], cz);
        // L1 norm, rounded up so that it bounds the exact L1 norm of the FP32 (x, y, z)
        v.w = __fadd_ru(__fadd_ru(fabsf(v.x), fabsf(v.y)), fabsf(v.z));
        rel[i] = v;
    }
}

int sm_count_p(int device) {
    int v = 148;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device);
    return v;
}

// mode: 0 count, 1 fill at known offsets, 2 one pass into result chunks
template <int KT, int ALGO, int MULTI>
cudaError_t launch_pk_m(const PacketArgs& a, int mode, bool fp32, int grid, cudaStream_t s) {
    if constexpr (MULTI == 2 && ALGO == kStruct) {  // batches do not search neighborsStruct
        return cudaErrorInvalidValue;
    }
    if (mode == 2) {
        if (fp32) k_radius_packet<KT, ALGO, 2, true, MULTI><<<grid, kPkThreads, 0, s>>>(a);
        else k_radius_packet<KT, ALGO, 2, false, MULTI><<<grid, kPkThreads, 0, s>>>(a);
    } else if (mode == 1) {
        if (fp32) k_radius_packet<KT, ALGO, 1, true, MULTI><<<grid, kPkThreads, 0, s>>>(a);
        else k_radius_packet<KT, ALGO, 1, false, MULTI><<<grid, kPkThreads, 0, s>>>(a);
    } else {
        if (fp32) k_radius_packet<KT, ALGO, 0, true, MULTI><<<grid, kPkThreads, 0, s>>>(a);
        else k_radius_packet<KT, ALGO, 0, false, MULTI><<<grid, kPkThreads, 0, s>>>(a);
    }
    return cudaGetLastError();
}

template <int KT, int ALGO>
cudaError_t launch_pk(const PacketArgs& a, int mode, bool fp32, int grid, cudaStream_t s) {
    if (a.grp) {
        if (a.one_cloud) return launch_pk_m<KT, ALGO, 2>(a, mode, fp32, grid, s);
        return launch_pk_m<KT, ALGO, 1>(a, mode, fp32, grid, s);
    }
    return launch_pk_m<KT, ALGO, 0>(a, mode, fp32, grid, s);
}

template <int KT>
cudaError_t launch_pk_a(const PacketArgs& a, int algo, int mode, bool fp32, int grid, cudaStream_t s) {
    switch (algo) {
        case kNeighbors: return launch_pk<KT, kNeighbors>(a, mode, fp32, grid, s);
        case kStruct: return launch_pk<KT, kStruct>(a, mode, fp32, grid, s);
        default: return launch_pk<KT, kPrune>(a, mode, fp32, grid, s);
    }
}

// Result chunks into the CSR array, every chunk by itself: its query's count and offset and its number in the
// chain say where its entries go.  A warp takes up to 32 chunks at a time, their records in coalesced reads, and copies
// kCompactBatch of them a step, the loads of all before any store.  Bound: HBM (8 bytes a result), and the
// sectors that a query's last chunk leaves half empty.  Following each query's links from chunk to chunk, four
// queries in lockstep, took 133 us for the 36.8M results of 500k queries, 195 for 59M in long chains and 981 for
// a 16-cloud batch; this form takes 106, 118 and 661.
constexpr int kCompactBatch = 4;
static_assert(kChunk == 64, "a chunk is two 32-entry rows");

__global__ void __launch_bounds__(256) k_chunk_compact(const unsigned long long* __restrict__ counts,
                                                       const unsigned long long* __restrict__ offs,
                                                       const uint2* __restrict__ rec,
                                                       const uint32_t* __restrict__ pool,
                                                       const uint32_t* __restrict__ ctr, uint32_t chunk_cap,
                                                       uint32_t* __restrict__ out, uint64_t out_cap, uint64_t n,
                                                       const uint64_t* d_n, uint32_t per, uint32_t* err) {
    // per: entries of a result (1 index, or 2 for a range); counts and offsets count results
    if (d_n) n = *d_n;
    const int lane = threadIdx.x & 31;
    const uint64_t chunks = min(*ctr, chunk_cap);
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    uint32_t S = kCompactBatch;  // chunks a warp takes at a time: as many as keep every warp busy
    while (S < 32 && S * nwarps < chunks) S <<= 1;
    bool bad = false;  // a chunk without a query (the pool ran over, which the search reported), or no room
    for (uint64_t c0 = (((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * S; c0 < chunks; c0 += nwarps * S) {
        const uint64_t c = c0 + lane;
        uint32_t len = 0;
        unsigned long long dst = 0;
        if ((uint32_t)lane < S && c < chunks) {
            const uint2 r = rec[c];
            const uint32_t q = r.x;
            if (q < n) {
                const unsigned long long total = counts[q] * per, at = (unsigned long long)r.y * kChunk;
                if (at < total) {
                    len = total - at < kChunk ? (uint32_t)(total - at) : kChunk;
                    dst = offs[q] * per + at;
                    if (dst + len > out_cap) {
                        bad = true;
                        len = 0;
                    }
                }
            } else {
                bad = true;
            }
        }
        for (uint32_t t = 0; t < S && c0 + t < chunks; t += kCompactBatch) {
            uint32_t v[kCompactBatch][2], m[kCompactBatch];
            unsigned long long d[kCompactBatch];
#pragma unroll
            for (int b = 0; b < kCompactBatch; ++b) {
                m[b] = __shfl_sync(0xffffffffu, len, t + b);
                d[b] = __shfl_sync(0xffffffffu, dst, t + b);
                const uint32_t* src = pool + (c0 + t + b) * kChunk + lane;
                if ((uint32_t)lane < m[b]) v[b][0] = src[0];
                if ((uint32_t)lane + 32 < m[b]) v[b][1] = src[32];
            }
#pragma unroll
            for (int b = 0; b < kCompactBatch; ++b) {
                uint32_t* to = out + d[b] + lane;
                if ((uint32_t)lane < m[b]) to[0] = v[b][0];
                if ((uint32_t)lane + 32 < m[b]) to[32] = v[b][1];
            }
        }
    }
    if (bad) set_err(err, kErrOutputCapacity);
}

// The sum of mix64 over each query's results (the count is the search's), a chunk a warp; hashes zeroed before.
__global__ void __launch_bounds__(256) k_chunk_hash(const unsigned long long* __restrict__ counts,
                                                    const uint2* __restrict__ rec,
                                                    const uint32_t* __restrict__ pool,
                                                    const uint32_t* __restrict__ ctr, uint32_t chunk_cap,
                                                    unsigned long long* __restrict__ hashes, uint64_t n,
                                                    uint32_t* err) {
    const int lane = threadIdx.x & 31;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t chunks = min(*ctr, chunk_cap);
    for (uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < chunks; c += nwarps) {
        const uint2 r = rec[c];
        const uint32_t q = r.x;
        if (q >= n) {  // the pool ran over (reported by the search kernel)
            if (lane == 0) set_err(err, kErrOutputCapacity);
            continue;
        }
        const unsigned long long total = counts[q], at = (unsigned long long)r.y * kChunk;
        unsigned long long h = 0;
        if (at + lane < total) h += mix64(pool[c * kChunk + lane]);
        if (at + lane + 32 < total) h += mix64(pool[c * kChunk + lane + 32]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) h += __shfl_xor_sync(0xffffffffu, h, off);
        if (lane == 0) atomicAdd(&hashes[q], h);
    }
}

}  // namespace

// FP32 (x, y, z) of every point relative to the box centre, each rounded once
// from the FP64 difference; w = 0.
__global__ void k_center_rel(const double* __restrict__ xs, const double* __restrict__ ys,
                             const double* __restrict__ zs, const BoxD* __restrict__ box, uint64_t n,
                             float4* __restrict__ out) {
    const double cx = box->center[0], cy = box->center[1], cz = box->center[2];
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x)
        out[i] = make_float4((float)dsub(xs[i], cx), (float)dsub(ys[i], cy), (float)dsub(zs[i], cz), 0.0f);
}

cudaError_t launch_center_rel(Cloud& c) {
    cudaError_t e;
    if ((e = c.crel.reserve(16 * (c.n ? c.n : 1))) != cudaSuccess) return e;
    if (c.n == 0) return cudaSuccess;
    const uint64_t want = (c.n + 255) / 256;
    const unsigned grid = (unsigned)(want < 148ull * 16 ? want : 148ull * 16);
    k_center_rel<<<grid, 256, 0, c.stream>>>(c.xs.as<double>(), c.ys.as<double>(), c.zs.as<double>(),
                                             c.d_box.as<BoxD>(), c.n, c.crel.as<float4>());
    return cudaGetLastError();
}

cudaError_t launch_leaf_rel(Cloud& c) {
    cudaError_t e;
    if ((e = c.rel.reserve(16 * (c.n ? c.n : 1))) != cudaSuccess) return e;
    if (c.n == 0 || c.n_total == 0) return cudaSuccess;
    const uint64_t threads = 32ull * c.n_total;
    k_leaf_rel<<<(unsigned)((threads + 255) / 256), 256, 0, c.stream>>>(
        c.xs.as<double>(), c.ys.as<double>(), c.zs.as<double>(), c.offsets.as<uint32_t>(), c.ranges.as<uint2>(),
        c.centers.as<double>(), c.n_total, c.rel.as<float4>());
    return cudaGetLastError();
}

CloudView cloud_view(const Cloud& c) {
    CloudView v;
    v.xs = c.xs.as<double>();
    v.ys = c.ys.as<double>();
    v.zs = c.zs.as<double>();
    v.rel = c.rel.as<float4>();
    v.crel = c.crel_built ? c.crel.as<float4>() : nullptr;
    v.offsets = c.offsets.as<uint32_t>();
    v.ranges = c.ranges.as<uint2>();
    v.centers = c.centers.as<double>();
    v.geom = reinterpret_cast<const LevelGeom*>(c.d_box.as<unsigned char>() + sizeof(BoxD));
    v.box = c.d_box.as<BoxD>();
    v.encoder = c.params.encoder;
    v.pad = 0;
    return v;
}

// Queries per packet: the widest of 1, 2, ... 16 that still leaves every resident warp (8 blocks per SM)
// two packets.  A wide packet reads each node once for all its queries, but it is one warp's serial walk:
// kernel time of sphere r = 2.5 searches of the 10M-point tile at widths 1 / 2 / 4 / 8 / 16 / 32, in us:
//   100 centres 71 / 100 / 137 / 225 / 420 / 843     30k 342 / 315 / 311 / 367 / 536 / 849
//   2k   105 / 125 / 159 / 262 / 435 / 849           100k 968 / 688 / 588 / 588 / 664 / 772
//   8k   176 / 198 / 265 / 385 / 626 / 1063          500k 4476 / 2618 / 1959 / 1735 / 1638 / 1720
// (with circles of 560 points on a dense tile 100k: 2256 / 1560 / 1238 / 1159 / 1333 / 1937).
// FP32 counts take 32 as well (widest): a leaf's contexts are made by all lanes at once, and there are no results
// to append: 500k squares of 3 m 5029 us at 16, 4795 at 32, spheres of 0.5 m 531, 507; FP32 lists are faster at 16.
uint32_t packet_width(uint64_t nq, int device, uint32_t widest) {
    const uint64_t packets = (uint64_t)sm_count_p(device) * kPkWarps * 8 * 2;
    uint32_t w = widest;
    while (w > 1 && (nq + w - 1) / w < packets) w >>= 1;
    return w;
}

cudaError_t launch_radius_table(int device, cudaStream_t s, int kernel, int algo, int mode, bool fp32,
                                const DynGroup* d_grp, const SearchReq* single, uint64_t packets, uint32_t width,
                                const uint32_t* d_order, unsigned long long* d_counts, unsigned long long* d_counts2,
                                const unsigned long long* d_offsets, uint32_t* d_out, uint64_t out_capacity,
                                uint32_t* d_packet_ctr, unsigned long long* d_stats, uint32_t* d_err,
                                int blocks_per_sm, const ChunkArgs* chunks) {
    cudaError_t e;
    if (!d_grp && packets == 0) return cudaSuccess;
    if ((e = cudaMemsetAsync(d_packet_ctr, 0, 4, s)) != cudaSuccess) return e;
    PacketArgs a;
    a.single = single ? *single : SearchReq{};
    a.grp = d_grp;
    a.one_cloud = d_grp != nullptr && single != nullptr;  // a batch on one cloud: its view in `single`
    a.packets = packets;
    a.width = width;
    a.order = d_order;
    a.counts = d_counts;
    a.counts2 = d_counts2;
    a.offs = d_offsets;
    a.out = d_out;
    a.out_cap = out_capacity;
    a.packet_ctr = d_packet_ctr;
    a.stats = d_stats;
    a.err = d_err;
    a.chunk_pool = chunks ? chunks->pool : nullptr;
    a.chunk_rec = chunks ? chunks->rec : nullptr;
    a.chunk_ctr = chunks ? chunks->ctr : nullptr;
    a.chunk_cap = chunks ? chunks->cap : 0;
    if (mode == 2 && (!chunks || (algo == kStruct && !d_counts2))) return cudaErrorInvalidValue;
    // persistent grid: warps take packets from the counter until none is left
    const uint64_t cap = (uint64_t)sm_count_p(device) * (blocks_per_sm > 0 ? blocks_per_sm : 12);
    const uint64_t want = d_grp ? cap : (packets + kPkWarps - 1) / kPkWarps;
    const int grid = (int)(want < cap ? want : cap);
    switch (kernel) {
        case kCircle: return launch_pk_a<kCircle>(a, algo, mode, fp32, grid, s);
        case kSquare: return launch_pk_a<kSquare>(a, algo, mode, fp32, grid, s);
        case kCube: return launch_pk_a<kCube>(a, algo, mode, fp32, grid, s);
        default: return launch_pk_a<kSphere>(a, algo, mode, fp32, grid, s);
    }
}

cudaError_t launch_chunk_hash(int device, cudaStream_t s, const unsigned long long* d_counts, const ChunkArgs& chunks,
                              unsigned long long* d_hashes, uint64_t n, uint32_t* d_err) {
    if (n == 0) return cudaSuccess;
    const cudaError_t e = cudaMemsetAsync(d_hashes, 0, 8 * n, s);
    if (e != cudaSuccess) return e;
    const uint64_t cap = (uint64_t)sm_count_p(device) * 8;
    const uint64_t want = ((uint64_t)chunks.cap + 7) / 8;
    const int grid = (int)(want < cap ? want : cap);
    k_chunk_hash<<<grid, 256, 0, s>>>(d_counts, chunks.rec, chunks.pool, chunks.ctr, chunks.cap, d_hashes,
                                      n, d_err);
    return cudaGetLastError();
}

cudaError_t launch_chunk_compact(int device, cudaStream_t s, const unsigned long long* d_counts,
                                 const unsigned long long* d_offsets, const ChunkArgs& chunks, uint32_t* d_out,
                                 uint64_t out_capacity, uint64_t n, const uint64_t* d_n, uint32_t* d_err,
                                 uint32_t per) {
    if ((!d_n && n == 0) || chunks.cap == 0) return cudaSuccess;
    const uint64_t cap = (uint64_t)sm_count_p(device) * 8;
    // a single search's chunks: its results' and a last one of every query
    const uint64_t most = d_n ? chunks.cap : std::min<uint64_t>(chunks.cap, out_capacity / kChunk + n + 1);
    const uint64_t want = (most + 31) / 32;  // 8 warps of at least kCompactBatch chunks a block
    const int grid = (int)(want < cap ? want : cap);
    k_chunk_compact<<<grid, 256, 0, s>>>(d_counts, d_offsets, chunks.rec, chunks.pool, chunks.ctr,
                                         chunks.cap, d_out, out_capacity, n, d_n, per, d_err);
    return cudaGetLastError();
}

cudaError_t launch_radius_packet(Cloud& c, int kernel, int algo, int mode, bool fp32, const double* d_centers,
                                 uint64_t nq, const double* d_radii, double radius, const uint32_t* d_order,
                                 unsigned long long* d_counts, unsigned long long* d_counts2,
                                 const unsigned long long* d_offsets, uint32_t* d_out, uint64_t out_capacity,
                                 const ChunkArgs* chunks) {
    cudaError_t e;
    if (nq == 0) return cudaSuccess;
    if ((e = c.packet_ctr.reserve(256)) != cudaSuccess) return e;
    SearchReq r{};
    r.cv = cloud_view(c);
    r.centers = d_centers;
    r.radii = d_radii;
    r.radius = radius;
    r.q_begin = 0;
    r.q_end = nq;
    r.packet_begin = 0;
    r.out_begin = 0;
    r.k = 0;
    r.cloud_id = 0;
    r.approx_cut = c.approx_cut;
    r.approx_upper = (uint32_t)c.approx_upper;
    KernelClock clk(c, 0);
    const uint32_t w = packet_width(nq, c.device, fp32 && mode == 0 ? 32 : 16);
    e = launch_radius_table(c.device, c.stream, kernel, algo, mode, fp32, nullptr, &r, (nq + w - 1) / w, w, d_order,
                            d_counts, d_counts2, d_offsets, d_out, out_capacity, c.packet_ctr.as<uint32_t>(),
                            c.stats.as<unsigned long long>(), c.d_err.as<uint32_t>(), 0, chunks);
    clk.stop();
    return e;
}

// A kernel of this file's device code, for preload_kernels.
const void* kernel_anchor_radius_packet() { return reinterpret_cast<const void*>(&k_center_rel); }

}  // namespace octb
