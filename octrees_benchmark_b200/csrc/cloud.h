// Host-side state of one device-resident cloud (the object behind oct_cloud)
// and the launchers each .cu file provides.  Internal to the library.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <string>
#include <utility>
#include <vector>

#include "../../include/octree_b200.h"
#include "oct_common.cuh"

namespace octb {

// A grow-only device allocation.  Bound to a memory pool and a stream (a
// cloud's arrays), its storage comes from the pool in that stream's order
// (cudaMallocFromPoolAsync / cudaFreeAsync): building or destroying a cloud
// then waits for nothing but its own stream, where cudaMalloc / cudaFree would
// wait for all work on the device (every other cloud's and engine's).
// Unbound, it uses cudaMalloc / cudaFree.
struct DevBuf {
    void* ptr = nullptr;
    size_t bytes = 0;
    cudaMemPool_t pool = nullptr;
    const cudaStream_t* stream = nullptr;  // the owner's current stream (followed when the owner switches it)
    bool slice = false;                    // part of the owner's slab: nothing to free
    void bind(cudaMemPool_t p, const cudaStream_t* s) {
        pool = p;
        stream = s;
    }
    cudaError_t reserve(size_t want) {
        if (want <= bytes) return cudaSuccess;
        release();
        size_t b = want < 256 ? 256 : want;
        cudaError_t e = pool ? cudaMallocFromPoolAsync(&ptr, b, pool, *stream) : cudaMalloc(&ptr, b);
        if (e == cudaSuccess) bytes = b;
        else ptr = nullptr;
        return e;
    }
    // The storage becomes [p, p + b) of a slab the owner holds (and frees after this array's release).
    void take_slice(void* p, size_t b) {
        release();
        ptr = p;
        bytes = b;
        slice = true;
    }
    void release() {
        if (ptr && !slice) {
            if (pool) cudaFreeAsync(ptr, *stream);
            else cudaFree(ptr);
        }
        ptr = nullptr;
        bytes = 0;
        slice = false;
    }
    template <class T>
    T* as() const { return static_cast<T*>(ptr); }
};

// The memory pool of every cloud's arrays on a device (created on first use,
// kept for the process; it holds all freed storage for reuse, until oct_trim_cloud_memory gives it back).
cudaMemPool_t cloud_pool(int device);
// The stream of a destroyed cloud, kept for the next one (at most kIdleStreams a device: creating and destroying a
// stream costs a small cloud as much as its sort); stream_get creates one when none is idle, idle_streams_drop
// destroys the idle ones.  Each is idle or owned by one cloud, so no two users share one.  One is kept, not more: the
// pool counts what a cloud freed as its stream's until that stream is gone, and an allocation on another stream asks
// every such stream first.  After 16 clouds were destroyed, building one of 73k points took 247 us with one stream
// kept, 354 with 4, 790 with 16 and 426 with none.
constexpr size_t kIdleStreams = 1;
cudaError_t stream_get(int device, cudaStream_t* out);
void stream_put(int device, cudaStream_t s);
void idle_streams_drop(int device);
// Pinned host blocks of kPinnedBlock bytes, reused across clouds (cudaFreeHost can wait for the device).
constexpr size_t kPinnedBlock = 4096;
constexpr size_t kPinnedRunOffset = 3072;  // the split sort's RunCtl on its way to the device
void* pinned_block_get();
void pinned_block_put(void* p);

// Device-side record of the sort (one per cloud): the 8 digit histograms of
// the keys, their exclusive scans, which passes are skipped (all keys share
// the digit) and one tile counter per pass.
struct SortCtl {
    unsigned long long offs[8][256];
    uint32_t hist[8][256];
    uint32_t skip[8];
    uint32_t tile_ctr[8];
    uint32_t bbox_ctr;
    uint32_t pad;
};

// Octree build bookkeeping written by the device.
struct BuildCtl {
    uint32_t level_internal[kMaxDepth + 2];  // split nodes of each level
    uint32_t n_total;
    uint32_t n_internal;
    uint32_t max_depth_seen;
    uint32_t need_nodes;                  // nodes the tree needs (valid when kErrNodeCapacity)
};

// Device pointers of one built cloud, as the search kernels read them.
struct CloudView {
    const double* xs;
    const double* ys;
    const double* zs;
    const float4* rel;          // FP32 leaf-relative points (packet FP32 path), may be null
    const float4* crel;         // FP32 points relative to the box centre (group kNN FP32 path), may be null
    const uint32_t* offsets;
    const uint2* ranges;
    const double* centers;
    const LevelGeom* geom;      // per-level radii
    const BoxD* box;            // the cloud's Box (anchor frame of its keys)
    int32_t encoder;            // OCT_ENC_MORTON_3D or OCT_ENC_HILBERT_3D
    uint32_t pad;
};

// One request of a search launch (device copy).  A launch covers a table of
// requests; every query of the launch has a global position q in
// [q_begin, q_end) of its request, and outputs are indexed by q.
struct SearchReq {
    CloudView cv;
    const double* centers;      // the request's nq x 3 centres
    const double* radii;        // per-query radii (radius requests) or null
    double radius;              // radius when radii is null
    uint64_t q_begin, q_end;    // global query positions of this request
    uint64_t packet_begin;      // first packet of the request in the launch
    uint64_t out_begin;         // kNN: first output slot (previous requests' nq * k)
    uint32_t k;                 // kNN k
    uint32_t cloud_id;          // distinct per cloud within the table (radii reload key)
    uint32_t approx_cut;        // neighborsStruct: 0, or neighborsApprox's precisionLevel + 1
    uint32_t approx_upper;      // neighborsApprox: 1 adds the ranges of the cut octants
};

// Launch sizes of one kernel group of a batch, in device memory.  The host
// writes them before the batch runs, so one launch configuration (and one
// captured graph) serves batches of any size.
struct DynGroup {
    const SearchReq* reqs;      // the group's requests (device), positions ascending
    uint32_t nreq;
    uint32_t kmax;              // kNN: largest k of the group
    uint64_t packets;           // packets of the group
    uint64_t width;             // radius: queries per packet (packet_width)
    uint64_t q_begin;           // first query position of the group
    uint64_t nq;                // queries of the group
};

// Register kNN: provisional k-th distance = this factor x the radius that holds k
// points at the density of the query's first cell (exact either way).
constexpr double kKnnEstimate = 1.2;
// Curve-ordered kNN: consecutive queries a warp takes at a time, in pairs (the later
// ones start from the k-th distances of those before them).  10M-point tile, 500k
// queries of k = 50: runs of 8 take 2.74 ms, of 16 2.87, of 32 3.23 (L2 and L1 hits).
constexpr uint32_t kKnnGroupChunk = 4;
// its heads: every kKnnHeadStride-th query (of k = 1 every fourth of those) is searched first,
// from its own node; the others start from a neighbouring query's k-th distance
constexpr uint32_t kKnnHeadStride = 16;
struct Cloud {
    oct_params params{};
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    uint64_t n = 0;
    bool sorted = false;
    bool built = false;
    int radius_group = 8;
    std::string last_error;

    DevBuf slab;            // one allocation the arrays sized by the point count are cut from
    // points
    DevBuf xyz_in;          // AoS input (n x 3 f64), as uploaded
    DevBuf xs, ys, zs;      // SFC-sorted coordinates, SoA f64
    DevBuf keys, keys_alt;  // u64 keys (sorted result lives in `keys`)
    DevBuf perm, perm_alt;  // u32 input position of each sorted point
    DevBuf keys_hi, keys_hi_alt;  // u32 upper key halves (the split sort)
    DevBuf run_pv, run_pv_alt;    // u64 lower key half << 32 | input position (the split sort)
    DevBuf run_ctl, run_list;     // the split sort's run bookkeeping
    DevBuf run_long;              // its runs longer than 4096 points (LongRun entries)
    int split_sel = 0;            // which keys_hi / run_pv buffer holds the split sort's result
    int split_sort = 1;           // sort the upper halves, then the runs (0: the 8-pass sort)
    DevBuf sort_status;     // onesweep look-back words
    uint32_t sort_epoch = 0;
    DevBuf d_ctl;           // SortCtl
    DevBuf d_box;           // BoxD
    DevBuf d_err;           // uint32 error word
    BoxD box{};             // host copy
    LevelGeom geom{};       // host copy

    // tree
    DevBuf offsets;  // u32, n_total + 1
    DevBuf ranges;   // uint2 (first, last) per node
    DevBuf centers;  // 3 x f64 per node (AoS)
    DevBuf lv_counts; // build scratch: split nodes per level and block of keys
    DevBuf lv_rows;   // build scratch: rows of keys that begin split nodes, per warp
    DevBuf lv_list;   // build scratch: the split nodes
    DevBuf parts;     // bounding-box partials
    DevBuf d_build;  // BuildCtl
    uint32_t node_capacity = 0;
    uint32_t n_total = 0, n_internal = 0, n_leaf = 0, max_depth_seen = 0;

    // query scratch
    DevBuf q_centers, q_radii, q_counts, q_offsets, q_out, q_out2, q_scan_tmp;
    // query ordering (packet searches): keys, order, look-back words, histograms
    DevBuf qs_keys, qs_keys_alt, qs_ord, qs_ord_alt, qs_status, qs_ctl;
    uint32_t qs_epoch = 0;
    DevBuf packet_ctr;  // dynamic packet counters
    DevBuf knn_fb;      // collecting kNN: fallback count (u64) at 0, fallback query list (u32) from byte 16
    DevBuf knn_heads;   // collecting kNN: the heads' k-th distances (f64 per head)
    DevBuf stats;       // device counters: points tested, FP64 band re-tests, ...
    // FP32 leaf-relative coordinates (x, y, z, 0) per sorted point, built on demand
    DevBuf rel;
    bool rel_built = false;
    DevBuf crel;  // FP32 (x, y, z) - box centre per point, for the group kNN's FP32 filter
    bool crel_built = false;
    // search configuration (oct_set_search_config)
    int packet = 1;
    int fp32_filter = 0;  // 0, OCT_FP32_ALL, OCT_FP32_RADIUS or OCT_FP32_KNN
    int knn_packet = 1;  // kNN (packet path): the collecting search, else sorted lists (k <= 64)
    uint32_t knn_bucket = 256;
    int two_pass = 0;   // 1: packet radius searches count, then fill (no result chunks)
    // neighborsStruct searches of the current call: 0, or neighborsApprox's precisionLevel + 1
    // (children deeper than that level are cut; approx_upper adds their ranges)
    uint32_t approx_cut = 0;
    int approx_upper = 0;
    // per-axis radii of the current call (the Vector-radii overloads, cube and square): device pointer to
    // nq x 3 half extents (axes_stride 3) or one (x, y, z) for every query (axes_stride 0); nullptr otherwise
    const double* axes = nullptr;
    uint32_t axes_stride = 0;
    DevBuf q_axes;
    double knn_est = kKnnEstimate;  // kNN provisional threshold: the sorted lists' factor; the collecting search seeds its queries unless 0
    uint32_t knn_chunk = kKnnGroupChunk;  // collecting kNN: pairs of consecutive queries per warp fetch
    // one-pass radius search: result chunk pool, each chunk's query and place in its chain, counter
    DevBuf ck_pool, ck_rec, ck_ctr;

    // pinned host staging for small readbacks
    void* pinned = nullptr;

    // oct_search_timing: CUDA events on the cloud's stream around the main search kernel of each call
    // (kind 0: the packet radius search, 1: the group kNN), summed by oct_search_kernel_times
    bool time_kernels = false;
    std::vector<cudaEvent_t> ev_free;
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_pend[2];
    double kernel_ms[2] = {0.0, 0.0};
    uint64_t kernel_launches[2] = {0, 0};
};

// Records the start of a timed kernel on the cloud's stream (no-op unless timing is on); stop() records the end.
struct KernelClock {
    Cloud& c;
    int kind;
    cudaEvent_t a = nullptr, b = nullptr;
    KernelClock(Cloud& cl, int k) : c(cl), kind(k) {
        if (!c.time_kernels) return;
        for (cudaEvent_t* e : {&a, &b}) {
            if (!c.ev_free.empty()) {
                *e = c.ev_free.back();
                c.ev_free.pop_back();
            } else if (cudaEventCreate(e) != cudaSuccess) {
                *e = nullptr;
            }
        }
        if (a && b) cudaEventRecord(a, c.stream);
    }
    void stop() {
        if (a && b) {
            cudaEventRecord(b, c.stream);
            c.ev_pend[kind].emplace_back(a, b);
        } else {
            if (a) c.ev_free.push_back(a);
            if (b) c.ev_free.push_back(b);
        }
        a = b = nullptr;
    }
};

// ---- launchers (each returns a cudaError_t of the launch) ----
// upper_hist_only: the split sort follows (the lower digits' histograms are not needed)
cudaError_t launch_bbox_encode(Cloud& c, const double* d_xyz_aos, bool upper_hist_only = false);
// The arrays that the sort of n points needs, cut from one allocation (c.slab, empty before; a failure leaves
// them to be allocated one by one).  Sixteen allocations and frees less: 40 us of a cloud's life.
void reserve_point_arrays(Cloud& c, uint64_t n);
cudaError_t launch_sort_split(Cloud& c, const uint32_t skip[8], const double* d_xyz_aos, int* out_sel);
cudaError_t launch_sort_long(Cloud& c, const double* d_xyz_aos, uint32_t l_count, uint32_t l_total);
cudaError_t launch_sort_passes(Cloud& c, const uint32_t skip[8], int* final_sel);
cudaError_t launch_gather(Cloud& c, const double* d_xyz_aos, const uint32_t* d_perm, int sel);
cudaError_t launch_build(Cloud& c, bool* capacity_ok);
cudaError_t launch_radius(Cloud& c, int kernel, int algo, int group, bool fill, const double* d_centers,
                          uint64_t nq, const double* d_radii, double radius, unsigned long long* d_counts,
                          unsigned long long* d_counts2, const unsigned long long* d_offsets, uint32_t* d_out,
                          uint64_t out_capacity);
cudaError_t launch_scan_u64(Cloud& c, const unsigned long long* d_in, unsigned long long* d_out, uint64_t n);
cudaError_t launch_query_order(Cloud& c, const double* d_centers, uint64_t nq, const uint32_t** d_order);
cudaError_t launch_leaf_rel(Cloud& c);
// FP32 coordinates relative to the box centre (group kNN FP32 filter), into c.crel.
cudaError_t launch_center_rel(Cloud& c);
struct ChunkArgs;
// mode as launch_radius_table (0 count, 1 fill, 2 one pass into `chunks`)
cudaError_t launch_radius_packet(Cloud& c, int kernel, int algo, int mode, bool fp32, const double* d_centers,
                                 uint64_t nq, const double* d_radii, double radius, const uint32_t* d_order,
                                 unsigned long long* d_counts, unsigned long long* d_counts2,
                                 const unsigned long long* d_offsets, uint32_t* d_out, uint64_t out_capacity,
                                 const ChunkArgs* chunks = nullptr);
// Result chunks of the one-pass radius search: `cap` chunks of 64 entries, the query each belongs to and its
// number in that query's chain (chunk k holds entries 64 k on), and the hand-out counter.
struct ChunkArgs {
    uint32_t* pool;
    uint2* rec;  // query, number in the chain
    uint32_t* ctr;
    uint32_t cap;
};
constexpr uint32_t kResultChunk = 64;
// The chunks of arrays as they are now: an array that could not be grown is empty, and so is the pool then.
inline ChunkArgs chunk_args(const DevBuf& pool, const DevBuf& rec, const DevBuf& ctr) {
    const uint64_t a = pool.bytes / (4ull * kResultChunk), b = rec.bytes / sizeof(uint2);
    const uint64_t cap = a < b ? a : b;
    return ChunkArgs{pool.as<uint32_t>(), rec.as<uint2>(), ctr.as<uint32_t>(),
                     (uint32_t)(cap < 0xfffffff0ull ? cap : 0xfffffff0ull)};
}

// Queries per packet (1 to `widest`: 16, or 32 where FP32 searches count) of a packet radius launch over nq queries.
uint32_t packet_width(uint64_t nq, int device, uint32_t widest = 16);
// Packet radius search.  Either one request (`single`, host copy, `packets`
// packets of `width` queries) or the group of a batch (`d_grp`, sizes read on the device); with
// both, every request of the group is on the cloud `single->cv` (kernel
// parameters instead of per-request views).
// mode: 0 count, 1 fill at d_offsets, 2 one pass into `chunks` (counts and
// the chunks' records written; neighborsStruct also writes d_counts2).
cudaError_t launch_radius_table(int device, cudaStream_t s, int kernel, int algo, int mode, bool fp32,
                                const DynGroup* d_grp, const SearchReq* single, uint64_t packets, uint32_t width,
                                const uint32_t* d_order, unsigned long long* d_counts, unsigned long long* d_counts2,
                                const unsigned long long* d_offsets, uint32_t* d_out, uint64_t out_capacity,
                                uint32_t* d_packet_ctr, unsigned long long* d_stats, uint32_t* d_err,
                                int blocks_per_sm = 0, const ChunkArgs* chunks = nullptr);
// Per query, the sum of splitmix64's output function over its result chunks.
cudaError_t launch_chunk_hash(int device, cudaStream_t s, const unsigned long long* d_counts, const ChunkArgs& chunks,
                              unsigned long long* d_hashes, uint64_t n, uint32_t* d_err);
// Result chunks into CSR (after the counts are scanned into d_offsets);
// per = 2 for ranges (two entries a result; d_out and out_capacity count entries).
cudaError_t launch_chunk_compact(int device, cudaStream_t s, const unsigned long long* d_counts,
                                 const unsigned long long* d_offsets, const ChunkArgs& chunks, uint32_t* d_out,
                                 uint64_t out_capacity, uint64_t n, const uint64_t* d_n, uint32_t* d_err,
                                 uint32_t per = 1);
// kNN, one warp per query.  Either one request (`single`, nq queries, k <= 64,
// register lists) or the group of a batch (`d_grp`, kmax = the group's largest
// k: register lists up to 64, shared-memory lists up to 1024).
cudaError_t launch_knn_table(int device, cudaStream_t s, const DynGroup* d_grp, const SearchReq* single, uint64_t nq,
                             uint32_t kmax, const uint32_t* d_order, uint32_t bucket, uint32_t* d_idx, double* d_d2,
                             uint32_t* d_counts, uint32_t* d_err, int blocks_per_sm = 0, double est = 0.0);
// Curve-ordered kNN of a batch group, then the sorted-list kernels over the queries it hands back.  d_fb: the
// fallback group (requests, kmax and q_begin of d_grp; its nq is set to 0
// here, so that the launch can be repeated); d_fb_list: one entry per query position of the batch; d_packet_ctr:
// three counters; blocks_per_sm > 0 caps the resident blocks of both launches.
cudaError_t launch_knn_group_table(int device, cudaStream_t s, const DynGroup* d_grp, DynGroup* d_fb,
                                   const SearchReq* single, uint32_t kmax, const uint32_t* d_order, uint32_t bucket,
                                   uint32_t* d_idx, double* d_d2, uint32_t* d_counts, uint32_t* d_err,
                                   uint32_t* d_packet_ctr, uint32_t* d_fb_list, double est, uint32_t chunk,
                                   int blocks_per_sm, double* d_head_kth, size_t head_bytes, bool fp32,
                                   unsigned long long* d_stats);
CloudView cloud_view(const Cloud& c);
// Batched engine: the sort of query keys with device-side sizes (encode_sort.cu),
// and the shared-memory limits of the table kNN list kernels (knn_search.cu).
cudaError_t prepare_sort_dyn();
cudaError_t prepare_knn_dyn();
size_t sort_tile_keys();
cudaError_t launch_sort_dyn(int device, cudaStream_t s, uint64_t* k0, uint64_t* k1, uint32_t* v0, uint32_t* v1,
                            const uint64_t* d_n, uint64_t max_n, int passes, SortCtl* ctl,
                            unsigned long long* status, const uint32_t* d_epoch, uint32_t* err,
                            uint32_t** result_vals);
cudaError_t launch_knn(Cloud& c, const double* d_centers, uint64_t nq, uint32_t k, uint32_t* d_idx, double* d_d2,
                       uint32_t* d_counts);

// oct_search_config.fp32_filter: which searches run their FP32 filter.
inline bool fp32_on_radius(int f) { return f == OCT_FP32_ALL || f == OCT_FP32_RADIUS; }
inline bool fp32_on_knn(int f) { return f == OCT_FP32_ALL || f == OCT_FP32_KNN; }

// One kernel of each source file's device code (each file is its own device
// library), and the loading of every kernel of those libraries on a device
// (capi.cu).  Under lazy module loading, the CUDA default, a kernel is loaded
// at its first launch and the load can wait for the work in flight on the
// device; a server meeting a kernel variant for the first time mid-stream
// would hold its batches that long.  preload_kernels loads them all once per
// device up front.
const void* kernel_anchor_capi();
const void* kernel_anchor_encode_sort();
const void* kernel_anchor_engine();
const void* kernel_anchor_knn_search();
const void* kernel_anchor_octree_build();
const void* kernel_anchor_radius_packet();
const void* kernel_anchor_radius_search();
int preload_kernels(int device);

}  // namespace octb

// The object behind the ABI's oct_cloud handle.
struct oct_cloud_s {
    octb::Cloud c;
};
