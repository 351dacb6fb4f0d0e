// Batched searches: Nearest_Search, Box_Search, Radius_Search, one launch per
// call; the traversal bodies and their semantics are in search.cuh.
#include <cuda_runtime.h>

#include <mutex>

#include "search.cuh"

namespace ikdg {
namespace {

using search::FINF;

constexpr int KNN_THREADS = search::KNN_CTA;
inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Stores n floats (or int bits) from shared memory to dst with the whole CTA:
// 16-byte stores where dst is 16-byte aligned, 4-byte stores otherwise.  src is
// 16-byte aligned.
__device__ __forceinline__ void block_store(float* dst, const float* src, int n) {
    int done = 0;
    if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
        const int n4 = n >> 2;
        for (int i = threadIdx.x; i < n4; i += KNN_THREADS)
            reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
        done = n4 << 2;
    }
    for (int i = done + threadIdx.x; i < n; i += KNN_THREADS) dst[i] = src[i];
}

// kNN, k <= 64: KNN_THREADS / KNN_G queries per CTA.  Dynamic shared memory: the
// threads' stack columns (`entries` each).  STAGED: the outputs are host memory;
// the CTA's rows are one span of every array (no permutation), are staged over
// the stacks once its queries are done and leave as 16-byte stores.
template <int R, bool STAGED, bool EARLY>
__global__ void __launch_bounds__(KNN_THREADS) knn_group_kernel(DevTree t, const float* __restrict__ q, int q_stride,
                                                                long long nq, int k, float max_sq, search::KnnOut o,
                                                                const int* __restrict__ perm, int entries, int per_warp) {
    extern __shared__ __align__(16) unsigned char knn_sm[];
    const search::KnnLane g;
    // query of this group among the CTA's; groups past per_warp idle
    const int gw = (threadIdx.x & 31) / search::KNN_G, gi = (threadIdx.x >> 5) * per_warp + gw;
    const int queries = KNN_THREADS / 32 * per_warp;
    const long long tid = (long long)blockIdx.x * queries + gi;
    const bool valid = gw < per_warp && tid < nq;
    long long qi = valid ? tid : 0;
    if (!STAGED && valid && perm != nullptr) qi = __ldg(perm + tid);
    const float qx = valid ? q[qi * q_stride + 0] : 0.f;
    const float qy = valid ? q[qi * q_stride + 1] : 0.f;
    const float qz = valid ? q[qi * q_stride + 2] : 0.f;
    float ld[R];
    int ls[R];
    search::knn_group<R, EARLY>(t, g, valid, qx, qy, qz, k, max_sq, reinterpret_cast<int2*>(knn_sm) + threadIdx.x, entries,
                         per_warp * search::KNN_G / 2, ld, ls);
    if (!STAGED) {
        search::knn_write_rows<R>(t, g, valid, ld, ls, k, qi, o);
        return;
    }
    __syncthreads();  // the stacks are dead: stage the rows over them
    float* st = reinterpret_cast<float*>(knn_sm);
    search::KnnOut so;
    so.id = reinterpret_cast<int*>(st);
    so.d2 = st + queries * k;
    so.xyz = o.xyz != nullptr ? st + 2 * queries * k : nullptr;
    so.cnt = reinterpret_cast<int*>(st + 5 * queries * k);
    search::knn_write_rows<R>(t, g, valid, ld, ls, k, gi, so);
    __syncthreads();
    const long long q0 = (long long)blockIdx.x * queries;
    const int rows = (int)min((long long)queries, nq - q0);
    block_store(reinterpret_cast<float*>(o.id + q0 * k), reinterpret_cast<const float*>(so.id), rows * k);
    block_store(o.d2 + q0 * k, so.d2, rows * k);
    if (o.xyz != nullptr) block_store(o.xyz + q0 * k * 3, so.xyz, rows * k * 3);
    if (o.cnt != nullptr) block_store(reinterpret_cast<float*>(o.cnt + q0), reinterpret_cast<const float*>(so.cnt), rows);
}

// Batches of at most this many queries get a warp per query (its other groups
// idle): no query waits for another one's steps.  1M-point map, host clock around
// one call, a warp each / eight a warp: 1,000 queries k = 5 29.0 / 36.2 us, k = 32 57 / 83;
// 4,000 queries 34.8 / 39.7 and 90 / 88, but 14.1 / 12.3 (k = 5) a call when calls on
// several trees overlap; 15,000 queries 71.7 / 41.8.
constexpr long long KNN_SPREAD_QUERIES = 2048;

// Batches of at most this many queries are bound by the chain of a query and load a
// bucket's slots beside its fill count; larger ones by issue and occupancy.  3M points, k
// = 5, us a call alone, after the count / beside it: 1 query 25.8 / 24.7, 2,000 34.6 / 32.3,
// 15,000 50.6 / 46.0, 30,000 56.5 / 53.4, 45,000 66.5 / 73.9, 80,000 97.9 / 102.5 (k = 32
// gains up to 80,000, 2 %).
constexpr long long KNN_EARLY_QUERIES = 32768;

template <int R>
void knn_group_launch(const DevTree& t, const float* q, int q_stride, long long nq, int k, float max_sq,
                      const search::KnnOut& o, const int* perm, bool staged, cudaStream_t s) {
    const int per_warp = nq <= KNN_SPREAD_QUERIES ? 1 : 32 / search::KNN_G;
    const int queries = KNN_THREADS / 32 * per_warp;
    const unsigned grid = blocks_for(nq, queries);
    const int entries = search::knn_stack_entries(t.height);
    const size_t stacks = (size_t)KNN_THREADS * entries * sizeof(int2);
    const size_t rows = (size_t)queries * (5 * k + 1) * sizeof(float);
    const size_t smem = staged && rows > stacks ? rows : stacks;
    const bool early = nq <= KNN_EARLY_QUERIES;
    auto kernel = staged ? (early ? knn_group_kernel<R, true, true> : knn_group_kernel<R, true, false>)
                         : (early ? knn_group_kernel<R, false, true> : knn_group_kernel<R, false, false>);
    kernel<<<grid, KNN_THREADS, smem, s>>>(t, q, q_stride, nq, k, max_sq, o, perm, entries, per_warp);
}

// Box (MODE 0) and radius (MODE 1) searches, `per` consecutive queries a warp.
// Counting: counts[qi], the warp's sum in warp_sum and, with a log, its hits.
template <int MODE>
__global__ void __launch_bounds__(search::RANGE_CTA) range_count_kernel(DevTree t, const float* __restrict__ q,
                                                                        int q_stride, const float* __restrict__ radius,
                                                                        int r_stride, long long nq, int per,
                                                                        long long* __restrict__ counts,
                                                                        long long* __restrict__ warp_sum,
                                                                        search::RangeLog log, int entries) {
    extern __shared__ __align__(16) unsigned char range_sm[];
    const search::RangeWarp w = search::range_warp_carve<false>(range_sm, entries);
    const int lane = threadIdx.x & 31;
    const long long wi = ((long long)blockIdx.x * search::RANGE_CTA + threadIdx.x) >> 5;
    const long long qi = wi * per + lane;
    const bool valid = lane < per && qi < nq;
    if (valid) search::range_put_query<MODE>(w, lane, q + qi * q_stride, MODE == 1 ? radius[qi * r_stride] : 0.f);
    w.cnt[lane] = 0;
    search::RangeLog wl = log;
    if (wi * per >= nq) wl.pool = nullptr;  // the grid's last warps: no queries, no chunk
    search::LogCursor lc(wl, wi);
    search::range_warp<MODE, false>(t, w, __ballot_sync(0xffffffffu, valid), entries, wl, lc, 0, 0, nullptr, nullptr);
    lc.close();
    __syncwarp();
    const int c = valid ? w.cnt[lane] : 0;
    if (valid) counts[qi] = c;
    long long sum = c;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0 && wi * per < nq) warp_sum[wi] = sum;
}

// The CSR offsets (nq + 1 entries) from the counts and the scanned warp sums.
// With ids, the logged hits are written from the queries' offsets on (a warp
// without a log searches again); with a capacity (>= 0), a query whose hits
// would end past it writes nothing and raises ERR_OUTPUT.
template <int MODE>
__global__ void __launch_bounds__(search::RANGE_CTA, 8) range_write_kernel(DevTree t, const float* __restrict__ q,
                                                                        int q_stride, const float* __restrict__ radius,
                                                                        int r_stride, long long nq, int per,
                                                                        const long long* __restrict__ counts,
                                                                        const long long* __restrict__ warp_off,
                                                                        long long* __restrict__ offsets,
                                                                        int* __restrict__ ids, float* __restrict__ xyz,
                                                                        long long capacity, search::RangeLog log,
                                                                        int entries) {
    extern __shared__ __align__(16) unsigned char range_sm[];
    const int lane = threadIdx.x & 31;
    const long long wi = ((long long)blockIdx.x * search::RANGE_CTA + threadIdx.x) >> 5;
    const long long qi = wi * per + lane;
    const bool valid = lane < per && qi < nq;
    const long long c = valid ? counts[qi] : 0;
    long long inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const long long v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
    }
    const long long start = (wi * per < nq ? warp_off[wi] : 0) + inc - c;
    if (valid) {
        offsets[qi] = start;
        if (qi == nq - 1) offsets[nq] = start + c;
    }
    if (ids == nullptr) return;
    const search::RangeWarp w = search::range_warp_carve<true>(range_sm, entries);
    bool go = c > 0;
    if (go && capacity >= 0 && start + c > capacity) {
        atomicOr(&t.st->err, ERR_OUTPUT);
        go = false;
    }
    const unsigned todo = __ballot_sync(0xffffffffu, go);
    if (todo == 0) return;
    // The log holds every query's hits: it serves unless one is to be left out.
    const int2* first = log.pool != nullptr ? log.pool + wi * search::LOG_CHUNK : nullptr;
    const bool all = todo == __ballot_sync(0xffffffffu, c > 0);
    if (first != nullptr && all && __ldg(&first->x) >= 0) {
        search::range_replay(t, w, log, first, start, start + c, ids, xyz);
        return;
    }
    if (go) search::range_put_query<MODE>(w, lane, q + qi * q_stride, MODE == 1 ? radius[qi * r_stride] : 0.f);
    search::LogCursor lc(search::RangeLog{nullptr, nullptr, 0, 0}, 0);
    search::range_warp<MODE, true>(t, w, todo, entries, log, lc, start, start + c, ids, xyz);
}

// A thread per query: k > 64 (K = 0), or k = K and very many sorted queries.
template <int K>
__global__ void __launch_bounds__(KNN_THREADS) knn_thread_kernel(DevTree t, const float* __restrict__ q, int q_stride,
                                                               long long nq, int k, float max_sq, search::KnnOut o,
                                                               int* __restrict__ slots, const int* __restrict__ perm) {
    const long long tid = (long long)blockIdx.x * KNN_THREADS + threadIdx.x;
    const bool valid = tid < nq;
    long long qi = valid ? tid : 0;
    if (valid && perm != nullptr) qi = __ldg(perm + tid);
    const float qx = valid ? q[qi * q_stride + 0] : 0.f;
    const float qy = valid ? q[qi * q_stride + 1] : 0.f;
    const float qz = valid ? q[qi * q_stride + 2] : 0.f;
    search::knn_thread_body<K>(t, valid, qi, qx, qy, qz, k, max_sq, o, slots);
}

// ---- query binning -----------------------------------------------------------
// Each query descends the top QBIN_BITS levels of the tree by the split planes;
// the left/right path, left-aligned to QBIN_BITS bits, is an in-order index of
// a k-d cell.  A counting sort on it puts queries of the same or neighbouring
// cells into the same warp, so the threads of a warp traverse nearly the same
// nodes and leaves.
__global__ void qbin_kernel(DevTree t, const float* __restrict__ q, int q_stride, long long nq, int* __restrict__ key,
                            int* __restrict__ hist, int nbits) {
    long long qi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (qi >= nq) return;
    const float p[3] = {q[qi * q_stride], q[qi * q_stride + 1], q[qi * q_stride + 2]};
    int code = __float_as_int(__ldg(&t.node[3].x));
    int bits = 0, depth = 0;
    while (code > 0 && depth < nbits) {
        const float4 f3 = __ldg(t.node + 4 * code + 3);
        const int go = p[__float_as_int(f3.w)] < f3.z ? 0 : 1;
        bits = (bits << 1) | go;
        code = go ? __float_as_int(f3.y) : __float_as_int(f3.x);
        ++depth;
    }
    bits <<= (nbits - depth);
    key[qi] = bits;
    atomicAdd(hist + bits, 1);
}

__global__ void qbin_scatter_kernel(const int* __restrict__ key, long long nq, int* __restrict__ cursor,
                                    int* __restrict__ perm) {
    long long qi = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (qi >= nq) return;
    int pos = atomicAdd(cursor + key[qi], 1);
    perm[pos] = (int)qi;
}

}  // namespace

size_t knn_temp_bytes(long long nq, int k) {
    size_t b = 0;
    if (nq >= QBIN_MIN_QUERIES) b += sizeof(int) * (2 * QBIN_BINS + 2 * nq) + scan_temp_bytes(QBIN_BINS) + 1024;
    if (k > KNN_GROUP_MAX) b += sizeof(int) * nq * k + 256;
    return b;
}

void launch_knn(const DevTree& t, const float* q, int q_stride, long long nq, int k, float max_sq, int* out_id,
                float* out_d2, float* out_xyz, int* out_cnt, void* temp, int bin_bits, cudaStream_t s,
                bool host_out) {
    if (nq <= 0) return;
    char* tp = (char*)temp;
    const int* perm = nullptr;
    const int nbins = 1 << bin_bits;
    if (nq >= QBIN_MIN_QUERIES && bin_bits > 0) {
        int* hist = (int*)tp;
        int* offs = hist + nbins;
        int* key = offs + nbins;
        int* pm = key + nq;
        char* stemp = (char*)(pm + nq);
        stemp = (char*)(((uintptr_t)stemp + 255) & ~(uintptr_t)255);
        tp = stemp + ((scan_temp_bytes(QBIN_BINS) + 255) / 256) * 256;
        cudaMemsetAsync(hist, 0, sizeof(int) * nbins, s);
        qbin_kernel<<<blocks_for(nq, 256), 256, 0, s>>>(t, q, q_stride, nq, key, hist, bin_bits);
        exclusive_scan(hist, offs, nbins, nullptr, stemp, s);
        qbin_scatter_kernel<<<blocks_for(nq, 256), 256, 0, s>>>(key, nq, offs, pm);
        perm = pm;
    }
    const search::KnnOut o{out_id, out_d2, out_xyz, out_cnt};
    if (k > KNN_GROUP_MAX) {
        knn_thread_kernel<0><<<blocks_for(nq, KNN_THREADS), KNN_THREADS, 0, s>>>(t, q, q_stride, nq, k, max_sq, o,
                                                                              (int*)tp, perm);
        return;
    }
    if (perm != nullptr && k <= 2 && nq >= KNN_THREAD_QUERIES) {
        auto kernel = k == 1 ? knn_thread_kernel<1> : knn_thread_kernel<2>;
        kernel<<<blocks_for(nq, KNN_THREADS), KNN_THREADS, 0, s>>>(t, q, q_stride, nq, k, max_sq, o, nullptr, perm);
        return;
    }
    const bool staged = host_out && perm == nullptr;
#define IKDG_KNN(R) knn_group_launch<R>(t, q, q_stride, nq, k, max_sq, o, perm, staged, s)
    if (k <= 4)
        IKDG_KNN(1);
    else if (k <= 8)
        IKDG_KNN(2);
    else if (k <= 16)
        IKDG_KNN(4);
    else if (k <= 32)
        IKDG_KNN(8);
    else
        IKDG_KNN(16);
#undef IKDG_KNN
}

// ---- kNN without allocation -----------------------------------------------------
// Scratch of the allocation-free kNN entry point (ikdg_knn_device_noalloc): the
// query sort's bin counters, bin offsets, per-query keys and permutation, and
// the prefix-sum partials, for at most NOALLOC_MAX_QUERIES queries.  It is a
// file-scope device array, so it exists on every GPU that loads the library
// until the process exits, and every call shares it.
constexpr size_t NOALLOC_SCRATCH_BYTES = ((size_t)(2 * QBIN_BINS + 2 * NOALLOC_MAX_QUERIES) * sizeof(int) + 4096 +
                                          64 * 1024);
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_SCRATCH_BYTES];

namespace {
std::mutex g_noalloc_mu;
void* g_noalloc_ptr[256] = {};
}  // namespace

// Device address of the scratch array on the current device.  Looked up once
// per device (the first call on a device does this set-up, which is why that
// first call must not happen inside a stream capture); later calls reuse it.
cudaError_t noalloc_scratch(int device, void** ptr) {
    if (device < 0 || device >= 256) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (g_noalloc_ptr[device] == nullptr) {
        void* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess) return e;
        g_noalloc_ptr[device] = p;
    }
    *ptr = g_noalloc_ptr[device];
    return cudaSuccess;
}

size_t noalloc_scratch_bytes() { return NOALLOC_SCRATCH_BYTES; }

namespace {

// Queries per warp: as many as leave about RANGE_WARPS warps, so that small
// batches spread over the GPU and large ones fill their warps' windows.
constexpr long long RANGE_WARPS = 4864;  // 32 per SM
int range_per(long long nq) {
    int per = 1;
    while (per < search::RANGE_QUERIES && nq / (2 * per) >= RANGE_WARPS) per *= 2;
    return per;
}

}  // namespace

namespace {

// Chunks of the hit log beyond one per warp: four per warp (100k radius
// searches of 0.5-5 m on a 1M-point map take 2.5), 64 MB at most.
long long log_extra(long long warps) { return warps * 4 < 65536 ? warps * 4 : 65536; }

struct RangeTemp {
    long long* counts;
    long long* sums;
    long long* offs;
    void* scan;
    unsigned* next;
    int2* pool;
    size_t bytes;
    RangeTemp(void* base, long long nq, long long warps, bool log) {
        char* p = (char*)base;
        auto take = [&](size_t b) {
            char* r = p;
            p += (b + 255) & ~(size_t)255;
            return (void*)r;
        };
        counts = (long long*)take(sizeof(long long) * nq);
        sums = (long long*)take(sizeof(long long) * warps);
        offs = (long long*)take(sizeof(long long) * warps);
        scan = take(scan_temp_bytes(warps));
        next = (unsigned*)take(sizeof(unsigned));
        pool = log ? (int2*)take(sizeof(int2) * search::LOG_CHUNK * (warps + log_extra(warps))) : nullptr;
        bytes = (size_t)(p - (char*)base);
    }
};

long long range_warps(long long nq) { return (nq + range_per(nq) - 1) / range_per(nq); }

}  // namespace

size_t range_temp_bytes(long long nq, int passes) {
    return RangeTemp(nullptr, nq, range_warps(nq), passes & RANGE_LOG).bytes + 256;
}

void launch_range(const DevTree& t, int mode, const float* q, int q_stride, const float* radius, int r_stride,
                  long long nq, void* temp, int passes, long long* offsets, int* ids, float* xyz, long long capacity,
                  long long* total, cudaStream_t s) {
    if (nq <= 0) return;
    const int per = range_per(nq);
    const long long warps = range_warps(nq);
    const RangeTemp w((void*)(((uintptr_t)temp + 255) & ~(uintptr_t)255), nq, warps, passes & RANGE_LOG);
    const search::RangeLog log{w.pool, w.next, warps, warps + log_extra(warps)};
    const unsigned grid = blocks_for(warps, search::RANGE_CTA / 32);
    const int entries = search::range_stack_entries(t.height);
    constexpr int WARPS = search::RANGE_CTA / 32;
    const size_t sm_count = WARPS * search::range_warp_bytes(entries, false);
    const size_t sm_write = ids != nullptr ? WARPS * search::range_warp_bytes(entries, true) : 0;
    if (passes & RANGE_COUNT) {
        if (log.pool != nullptr) cudaMemsetAsync(w.next, 0, sizeof(unsigned), s);
        if (mode == 0)
            range_count_kernel<0><<<grid, search::RANGE_CTA, sm_count, s>>>(t, q, q_stride, radius, r_stride, nq, per,
                                                                            w.counts, w.sums, log, entries);
        else
            range_count_kernel<1><<<grid, search::RANGE_CTA, sm_count, s>>>(t, q, q_stride, radius, r_stride, nq, per,
                                                                            w.counts, w.sums, log, entries);
        exclusive_scan(w.sums, w.offs, warps, total, w.scan, s);
    }
    if (mode == 0)
        range_write_kernel<0><<<grid, search::RANGE_CTA, sm_write, s>>>(t, q, q_stride, radius, r_stride, nq, per,
                                                                        w.counts, w.offs, offsets, ids, xyz, capacity,
                                                                        log, entries);
    else
        range_write_kernel<1><<<grid, search::RANGE_CTA, sm_write, s>>>(t, q, q_stride, radius, r_stride, nq, per,
                                                                        w.counts, w.offs, offsets, ids, xyz, capacity,
                                                                        log, entries);
}

}  // namespace ikdg
