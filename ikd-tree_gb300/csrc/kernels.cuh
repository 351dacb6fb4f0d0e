// Host-side launchers shared between the translation units of libikdg.
#pragma once
#include <cuda_runtime.h>

#include <utility>
#include <stdint.h>

#include "common.cuh"

namespace ikdg {

// A mutation or a build is a chain of short launches in one stream, each needing the
// one before.  launch_chain lets a kernel's blocks come up while its predecessor
// drains (programmatic stream serialization); every kernel launched so calls
// chain_begin first, which waits until all earlier work of the stream is complete and
// visible, then lets the next one come up.  What
// the chain writes is read with plain or L2 loads, never as read-only data
// (const __restrict__, __ldg): the reader is up while it is written.  Not used for
// queries (one or two launches) nor under capture.  Waiting blocks hold no more
// than one kernel's worth of places: a kernel lets the next one come up only once it
// runs itself.  14,400-point scan into 500,000 points 431 -> 393 us, small edits of
// 100,000 points 502 -> 465, a build of 2,000,000 points 1054 -> 1000.
__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// The first launch of this thread's chains that was refused since the last look.  A
// chain with a launch missing leaves a wrong tree: the call that issued it looks before
// it waits.
inline thread_local cudaError_t chain_refused = cudaSuccess;
inline cudaError_t take_chain_refused() {
    const cudaError_t e = chain_refused;
    chain_refused = cudaSuccess;
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}
template <class... P, class... A>
inline void launch_chain_if(bool chain, unsigned cluster, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem,
                            cudaStream_t s, A&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    int n = 0;
    if (chain) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = cluster;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        ++n;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
    // (launches outside a chain: left as the thread's last error, as with <<<>>>)
    if (chain && e != cudaSuccess && chain_refused == cudaSuccess) chain_refused = e;
}
template <class... P, class... A>
inline void launch_chain(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t s, A&&... args) {
    launch_chain_if(true, 1, kernel, grid, block, smem, s, std::forward<A>(args)...);
}


// ---- sort.cu ----------------------------------------------------------------
// Exclusive prefix sum of n int32 / int64 values; `total` (device, nullable) receives
// the sum.  `temp` must hold scan_temp_bytes(n) bytes.
size_t scan_temp_bytes(long long n);
// chain: launched with launch_chain.
void exclusive_scan(const int* in, int* out, long long n, int* total, void* temp, cudaStream_t s, bool chain = false);
void exclusive_scan(const long long* in, long long* out, long long n, long long* total, void* temp, cudaStream_t s);

// Stable LSD radix sort of `batch` independent (key, value) arrays of length n
// stored `stride` elements apart, on the low `bits` bits of the key (a
// multiple of 8).  The result lands back in keys / vals; the *_alt buffers are
// scratch of the same shape.  `temp` must hold sort_temp_bytes(n, batch).
size_t sort_temp_bytes(long long n, int batch);
// With copy_back = false an odd number of passes leaves the result in the
// alt buffers, and the call returns true.
bool radix_sort_pairs(uint32_t* keys, uint32_t* vals, uint32_t* keys_alt, uint32_t* vals_alt, long long n,
                      int batch, long long stride, int bits, void* temp, cudaStream_t s, bool copy_back = true, bool chain = false);

// ---- build.cu ---------------------------------------------------------------
// Batched subtree build.  `pts` holds the points of `njobs` jobs back to back
// (job j = [job_off[j], job_off[j+1])), each as {x, y, z, id}.  Every job
// becomes a balanced subtree of leaves holding at most `fill` points, split at
// the median of the longest AABB axis, and is linked into the child slot
// `job_link[j]` (= parent * 2 + side) together with its AABB and counts.  The pools'
// free stacks are settled by the snapshot or job-finish kernel that follows.
// Open segments of the large splitter at one level, and their tiles: a block of a
// launch over tiles b takes tile[b] = {s, e, segment, tile of the segment}.
struct SplitLevel {
    int4* seg;       // {s, e, link, -}
    uint32_t* box;   // 6 per segment: keys of the AABB's low, then high corner
    int* cand_n;     // candidates listed
    int4* tile;      // tiles of SPLIT_TILE points
    int4* htile;     // tiles of HIST_TILE points
    unsigned long long* n;  // segments, tiles, htiles in one word (split_take)
};
struct BuildScratch {
    float4* pts[3];      // 3 x [n] points between levels; [2]: those of segments that left the splitter
    int4* small;         // segments for finish_split_kernel  {s, e, link, -}
    int4* local_jobs;    // segments for the local builder
    int* nseg;           // [2] device counters (small, local)
    SplitLevel split[2]; // large segments of two levels
    int* hist;           // bins per large segment
    int2* pick;          // {bin, rank in it}
    uint2* thr;          // {key, position} of the split point
    int2* kids;          // large segments of the children (-1: small, -2: dropped)
    int* tile_left;      // left points per tile, then their prefix
    uint2* cand;         // [n] {key, position} of the picked bins' points
};
size_t build_scratch_bytes(long long n, int njobs);
void carve_build_scratch(void* base, long long n, int njobs, BuildScratch* bs);
int build_levels(long long max_job, int fill);
void build_subtrees(const DevTree& t, const float4* pts, long long n, const int* job_off, const int* job_link,
                    int njobs, long long max_job, int fill, const BuildScratch& bs, cudaStream_t s);

// ---- query.cu ---------------------------------------------------------------
// Batched kNN.  `temp` must hold knn_temp_bytes(nq, k) bytes of device
// scratch: the query binning (QBIN_BINS counters, a key and a permutation
// entry per query, for batches of at least QBIN_MIN_QUERIES) and, for
// k > KNN_GROUP_MAX, k slot indices per query.  A group of lanes searches each
// query, with the candidate list in registers, for k <= KNN_GROUP_MAX; beyond,
// a thread does, with the list in the output rows.
constexpr int KNN_GROUP_MAX = 64;
constexpr int QBIN_BITS = 16;
constexpr int QBIN_BINS = 1 << QBIN_BITS;
constexpr long long QBIN_MIN_QUERIES = 2048;
// Whether a batch is sorted by default (by 16 levels).  Sorted neighbours share what
// they fetch and walk alike, which pays where the search is long against the sort (30 to
// 60 us per million queries): many queries on a small map, long lists on a map beyond
// the L2 cache, or very many queries.  With k <= 2 such a batch goes to a thread per
// query, which issues less than a group when 32 neighbours walk alike.  Device buffers,
// unsorted / sorted (us), surfaces unless said:
//   20k points, 1.5M queries: k = 1 426 / 360 (a thread each), k = 2 537 / 470, k = 5
//   836 / 779, 600k queries: k = 8 455 / 431, k = 32 1886 / 1611;
//   200k: 1.5M, k = 1 493 / 430, k = 5 890 / 844, uniform 950 / 962;
//   3M uniform: 1M, k = 1 339 / 378, k = 8 988 / 1030, 5M, k = 8 one per cent apart;
//   20M slab: 1M, k = 16 1107 / 1064, k = 5 829 / 804, 500k k = 5 on 10M 484 / 498.
// The lines (slots, queries) lie where surfaces gain more than uniform maps lose; up to
// 500k queries nothing is sorted.  Host buffers: only the long lists on large maps (a
// sorted batch's rows come back by copy).
constexpr int QBIN_AUTO_BITS = 16;
constexpr long long KNN_THREAD_QUERIES = 900000;
inline int knn_auto_bits(long long nq, int k, long long slots, bool host) {
    const bool large_map = k >= 8 && slots >= 12000000 && nq >= 1 << 19;
    const bool small_map = slots < 300000 && nq >= 1 << 19 && nq * k >= 4500000;
    const bool threads = k <= 2 && nq >= (slots < 2000000 ? KNN_THREAD_QUERIES : 1 << 21);
    const bool sort = large_map || (!host && (threads || (k > 2 && (small_map || nq >= 4000000))));
    return sort ? QBIN_AUTO_BITS : 0;
}
size_t knn_temp_bytes(long long nq, int k);
// Host-pointer kNN calls of at most this many queries (and k <= KNN_GROUP_MAX)
// run on pooled per-call streams with the tree's lock held shared, so
// concurrent callers search at the same time.
constexpr long long SMALL_KNN_QUERIES = 4096;
// Allocation-free kNN: limit on the batch size and the device address of the
// shared scratch array (looked up on the first call per device).
constexpr long long NOALLOC_MAX_QUERIES = 1 << 18;
cudaError_t noalloc_scratch(int device, void** ptr);
size_t noalloc_scratch_bytes();
// `bin_bits` (0 = off, at most QBIN_BITS) levels of the tree order the queries
// before the search.
// host_out: the outputs are host memory the GPU writes directly (each warp's
// rows then leave as coalesced 16-byte spans through shared memory).
void launch_knn(const DevTree& t, const float* q, int q_stride, long long nq, int k, float max_sq,
                int* out_id, float* out_d2, float* out_xyz, int* out_cnt, void* temp, int bin_bits,
                cudaStream_t s, bool host_out = false);
// Box (mode 0) and radius (mode 1) search.  `temp` holds range_temp_bytes(nq,
// passes) bytes.  passes: RANGE_COUNT counts the hits first (*total, nullable, receives
// their number), without it the counts in temp are those of an earlier call
// with the same queries; RANGE_LOG keeps the hits found while counting for the
// writing (of this call or of that later one, which passes it too).  offsets
// (nq + 1 entries) are written; with ids, the hits too.  Boxes are {min xyz, max
// xyz}; radius queries are {x, y, z} with a per-query radius (r_stride floats
// apart).  With capacity >= 0, a query whose hits would end past it is skipped
// (raising ERR_OUTPUT).
constexpr int RANGE_COUNT = 1, RANGE_LOG = 2;
size_t range_temp_bytes(long long nq, int passes);
void launch_range(const DevTree& t, int mode, const float* q, int q_stride, const float* radius, int r_stride,
                  long long nq, void* temp, int passes, long long* offsets, int* ids, float* xyz, long long capacity,
                  long long* total, cudaStream_t s);

// ---- batch.cu ---------------------------------------------------------------------
// One request of a multi-tree batch: a kNN, box or radius search of nq queries
// on trees[tree].  Phase 1 (search) covers chunks [c1, c1 + n1) of the
// phase's chunk numbering; range requests also take phase-2 (write) chunks
// [c2, c2 + n2).  A chunk is the work a warp takes at once: `per` queries.
constexpr int BATCH_THREADS = 128;
constexpr int BATCH_CHUNK = 32;       // queries per chunk, at most
constexpr int BATCH_KNN_STEP = 8;     // kNN queries a warp searches side by side
constexpr int BATCH_KMAX = 16;
constexpr int BATCH_RANGE_CLASS = 3;  // box / radius requests; 0..2: kNN, k <= 4, 8, 16
enum BatchKind : int { BATCH_KNN = 0, BATCH_BOX = 1, BATCH_RADIUS = 2 };

struct BatchReq {
    long long c1, n1, c2, n2;
    const float* q;
    const float* radius;
    long long nq;
    int kind, tree, q_stride, r_stride;
    int k, per;
    float max_sq;
    int* ids;
    float* d2;
    float* xyz;
    int* cnt;
    long long* offsets;  // range: nq + 1 entries, CSR within the request
    long long cbase;     // range: first entry of this request in the batch count array
    long long capacity;  // range: ids / xyz capacity
    long long* total;    // range: device total (nullable)
    const int* perm;     // query at position i of the request's run order (nullptr: in order)
};

// The range requests' hit log (see RangeLog in search.cuh), one first chunk per
// phase-2 chunk of queries.
struct BatchLog {
    void* pool;
    unsigned* next;
    long long warps, chunks;
};
size_t batch_log_bytes(long long chunks);
// Chunks of the log for this many phase-2 chunks of queries.
long long batch_log_chunks(long long warps);

// Register class of a kNN request with this k (k <= BATCH_KMAX): 0..2;
// range requests are class BATCH_RANGE_CLASS.
int batch_kclass(int k);
// Resident CTAs (whole GPU) of the persistent search kernel of a class;
// `height`: the tallest tree of the batch (sizes the stacks).
int batch_search_grid(int kclass, int height);
int batch_write_grid(int height);
// Phase 1 over requests [r0, r1), all of register class kclass, whose chunks
// are [c_begin, c_end); ctr: a zeroed device counter.
void launch_batch_search(const DevTree* trees, const BatchReq* reqs, const long long* req_c1, int r0, int r1,
                         long long c_begin, long long c_end, int kclass, int height, long long* counts,
                         const BatchLog& log, unsigned long long* ctr, int grid, cudaStream_t s);
// Spatial order of every request's queries: key = request position in the
// high bits, Morton code of the query (kNN / radius: the point; box: its
// centre) in the tree's root box below; vals = query index in its request.
// qstart: first query of each request in [0, total) (n + 1 entries).
void launch_batch_keys(const DevTree* trees, const BatchReq* reqs, const long long* qstart, int n, long long total,
                       int req_bits, uint32_t* keys, uint32_t* vals, cudaStream_t s);
// Phase 2 over the range requests listed in ridx[0..nr) (ascending c2, chunks
// [0, c_end)); goff: exclusive scan of the batch count array.
void launch_batch_write(const DevTree* trees, const BatchReq* reqs, const int* ridx, const long long* req_c2, int nr,
                        long long c_end, int height, const long long* goff, const BatchLog& log, unsigned long long* ctr,
                        int grid, cudaStream_t s);

// ---- register.cu ---------------------------------------------------------------
// The pose travels as a kernel argument: R row-major, t.  planes: 2 float4 per
// point ({n,d} and a point c on the plane).  partial: per-block double sums
// (reg_blocks(n) entries of 1 (loss) or 6 (adjoint) doubles).
struct RegPose {
    double R[9], t[3];
};
int reg_blocks(long long n);
void launch_transform(const float* p, long long n, const RegPose& pose, float* w, cudaStream_t s);
void launch_plane_residual(const float* p, const RegPose& pose, long long n, int k, const float* nb, const int* cnt,
                           float thresh, float4* planes, float* res, int* valid, double* partial, cudaStream_t s);
void launch_adjoint(const float* p, long long n, const RegPose& pose, const float4* planes, const float* res,
                    const int* valid, float dl, float* grad_p, double* partial, cudaStream_t s);

// ---- update.cu --------------------------------------------------------------
struct UpdateScratch;
}  // namespace ikdg
