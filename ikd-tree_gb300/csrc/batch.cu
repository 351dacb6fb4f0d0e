// Multi-tree batched searches: many kNN / box / radius requests over many
// trees in one persistent launch per phase.  The reference has no batched
// form; every request has the semantics of its per-call search (search.cuh).
//
// Work is cut into chunks of up to BATCH_CHUNK queries; each warp takes
// the next chunk index from a device counter, finds the request it belongs to
// by a binary search over the requests' first chunks, and runs that request's
// search body on it.  So small requests of many trees fill the GPU together,
// no launch is spent per request, and no warp waits for another (a warp with
// a heavy query does not hold up the rest of its CTA).
#include <cuda_runtime.h>

#include <mutex>

#include "search.cuh"

namespace ikdg {
namespace {

constexpr int WARPS_PER_CTA = BATCH_THREADS / 32;

// Last r in [lo, hi) with starts[r] <= c (starts ascending, starts[lo] <= c).
__device__ __forceinline__ int find_req(const long long* __restrict__ starts, int lo, int hi, long long c) {
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(starts + mid) <= c)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Phase 1 for one class: KC 0..2 are kNN requests with k <= 4, 8, 16 (four lanes
// per query, the list in 1, 2 or 4 registers a lane), producing their final rows;
// KC = BATCH_RANGE_CLASS box and radius requests (per-query hit counts in
// counts[cbase + qi]).  One kernel per class keeps each at its own register
// count.  entries: stack entries, per thread (kNN) or per warp (range), in dynamic
// shared memory.
template <int KC>
__global__ void __launch_bounds__(BATCH_THREADS) batch_search_kernel(const DevTree* __restrict__ trees,
                                                                     const BatchReq* __restrict__ reqs,
                                                                     const long long* __restrict__ req_c1, int r0,
                                                                     int r1, long long c_begin, long long c_end,
                                                                     long long* __restrict__ counts,
                                                                     search::RangeLog log,
                                                                     unsigned long long* __restrict__ ctr,
                                                                     int entries) {
    constexpr int G = search::KNN_G, R = KC == 0 ? 1 : KC == 1 ? 2 : 4;
    extern __shared__ __align__(16) int2 batch_sm[];
    const int lane = threadIdx.x & 31;
    for (;;) {
        // Each warp takes its own chunk: no warp waits for another.
        long long c = 0;
        int r = -1;
        if (lane == 0) {
            c = c_begin + (long long)atomicAdd(ctr, 1ull);
            r = c < c_end ? find_req(req_c1, r0, r1, c) : -1;
        }
        c = __shfl_sync(0xffffffffu, c, 0);
        r = __shfl_sync(0xffffffffu, r, 0);
        if (c >= c_end) break;
        const BatchReq& Rq = reqs[r];
        const DevTree t = trees[Rq.tree];
        if constexpr (KC < BATCH_RANGE_CLASS) {
            static_assert(G * BATCH_KNN_STEP == 32 && BATCH_THREADS == search::KNN_CTA, "a warp's queries, the stack columns");
            const search::KnnLane g;
            int2* stk = batch_sm + threadIdx.x;
            const search::KnnOut o{Rq.ids, Rq.d2, Rq.xyz, Rq.cnt};
            const long long q0 = (c - Rq.c1) * Rq.per;
            for (int i = 0; i < Rq.per && q0 + i < Rq.nq; i += BATCH_KNN_STEP) {
                long long qi = q0 + i + lane / G;
                const bool valid = qi < Rq.nq;
                if (valid && Rq.perm != nullptr) qi = __ldg(Rq.perm + qi);
                if (!valid) qi = 0;
                const float* q = Rq.q + qi * Rq.q_stride;
                const float qx = valid ? q[0] : 0.f, qy = valid ? q[1] : 0.f, qz = valid ? q[2] : 0.f;
                float ld[R];
                int ls[R];
                search::knn_group<R>(t, g, valid, qx, qy, qz, Rq.k, Rq.max_sq, stk, entries, 16, ld, ls);
                search::knn_write_rows<R>(t, g, valid, ld, ls, Rq.k, qi, o);
            }
        } else {
            const search::RangeWarp w =
                search::range_warp_carve<false>(reinterpret_cast<unsigned char*>(batch_sm), entries);
            long long qi = (c - Rq.c1) * Rq.per + lane;
            const bool valid = lane < Rq.per && qi < Rq.nq;
            if (valid && Rq.perm != nullptr) qi = __ldg(Rq.perm + qi);
            w.cnt[lane] = 0;
            const unsigned todo = __ballot_sync(0xffffffffu, valid);
            search::LogCursor lc(log, Rq.c2 + (c - Rq.c1));
            if (Rq.kind == BATCH_BOX) {
                if (valid) search::range_put_query<0>(w, lane, Rq.q + qi * Rq.q_stride, 0.f);
                search::range_warp<0, false>(t, w, todo, entries, log, lc, 0, 0, nullptr, nullptr);
            } else {
                if (valid) search::range_put_query<1>(w, lane, Rq.q + qi * Rq.q_stride, Rq.radius[qi * Rq.r_stride]);
                search::range_warp<1, false>(t, w, todo, entries, log, lc, 0, 0, nullptr, nullptr);
            }
            lc.close();
            __syncwarp();
            if (valid) counts[Rq.cbase + qi] = w.cnt[lane];
            __syncwarp();
        }
    }
}

// Phase 2: range requests write their CSR offsets and, where the request's
// capacity holds the query's results, the ids / points.
__global__ void __launch_bounds__(BATCH_THREADS, 6) batch_write_kernel(const DevTree* __restrict__ trees,
                                                                    const BatchReq* __restrict__ reqs,
                                                                    const int* __restrict__ ridx,
                                                                    const long long* __restrict__ req_c2, int nr,
                                                                    long long c_end,
                                                                    const long long* __restrict__ goff,
                                                                    search::RangeLog log,
                                                                    unsigned long long* __restrict__ ctr, int entries) {
    extern __shared__ __align__(16) int2 batch_sm[];
    const search::RangeWarp w =
        search::range_warp_carve<true>(reinterpret_cast<unsigned char*>(batch_sm), entries);
    const int lane = threadIdx.x & 31;
    for (;;) {
        long long c = 0;
        int r = -1;
        if (lane == 0) {
            c = (long long)atomicAdd(ctr, 1ull);
            r = c < c_end ? __ldg(ridx + find_req(req_c2, 0, nr, c)) : -1;
        }
        c = __shfl_sync(0xffffffffu, c, 0);
        r = __shfl_sync(0xffffffffu, r, 0);
        if (c >= c_end) break;
        const BatchReq& R = reqs[r];
        const DevTree t = trees[R.tree];
        const long long at = (c - R.c2) * R.per + lane;
        bool go = lane < R.per && at < R.nq;
        const long long qi = go && R.perm != nullptr ? (long long)__ldg(R.perm + at) : at;
        const long long base = goff[R.cbase];
        long long o = 0, n = 0;
        if (go && at == 0) {
            const long long tot = goff[R.cbase + R.nq] - base;
            R.offsets[R.nq] = tot;
            if (R.total != nullptr) *R.total = tot;
        }
        if (go) {
            o = goff[R.cbase + qi] - base;
            n = goff[R.cbase + qi + 1] - goff[R.cbase + qi];
            R.offsets[qi] = o;
            if (n == 0 || R.ids == nullptr) {
                go = false;
            } else if (o + n > R.capacity) {
                atomicOr(&t.st->err, ERR_OUTPUT);
                go = false;
            }
        }
        const unsigned todo = __ballot_sync(0xffffffffu, go);
        if (todo == 0) continue;
        const int2* first = log.pool + c * search::LOG_CHUNK;
        if (todo == __ballot_sync(0xffffffffu, n > 0) && __ldg(&first->x) >= 0) {
            search::range_replay(t, w, log, first, o, o + n, R.ids, R.xyz);
            continue;
        }
        search::LogCursor lc(search::RangeLog{nullptr, nullptr, 0, 0}, 0);
        if (R.kind == BATCH_BOX) {
            if (go) search::range_put_query<0>(w, lane, R.q + qi * R.q_stride, 0.f);
            search::range_warp<0, true>(t, w, todo, entries, log, lc, o, o + n, R.ids, R.xyz);
        } else {
            if (go) search::range_put_query<1>(w, lane, R.q + qi * R.q_stride, R.radius[qi * R.r_stride]);
            search::range_warp<1, true>(t, w, todo, entries, log, lc, o, o + n, R.ids, R.xyz);
        }
        __syncwarp();
    }
}

// Every third bit of a 10-bit value (Morton interleave).
__device__ __forceinline__ uint32_t spread3(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

__global__ void batch_key_kernel(const DevTree* __restrict__ trees, const BatchReq* __restrict__ reqs,
                                 const long long* __restrict__ qstart, int n, long long total, int req_bits,
                                 uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= total) return;
    const int p = find_req(qstart, 0, n, g);
    const BatchReq& R = reqs[p];
    const long long qi = g - qstart[p];
    float c[3];
    const float* q = R.q + qi * R.q_stride;
    for (int a = 0; a < 3; ++a) c[a] = R.kind == BATCH_BOX ? 0.5f * (q[a] + q[3 + a]) : q[a];
    // the root's box is the left-child box of the sentinel record (node 0)
    const float4 f0 = trees[R.tree].node[0], f1 = trees[R.tree].node[1];
    const float lo[3] = {f0.x, f0.y, f0.z}, hi[3] = {f0.w, f1.x, f1.y};
    uint32_t m = 0;
    for (int a = 0; a < 3; ++a) {
        const float t = (c[a] - lo[a]) / (hi[a] - lo[a]);
        const int v = hi[a] > lo[a] && t > 0.f ? (t < 1.f ? (int)(t * 1024.f) : 1023) : 0;
        m |= spread3((uint32_t)min(v, 1023)) << a;
    }
    const int mb = 32 - req_bits;  // Morton bits kept below the request position
    keys[g] = ((uint32_t)p << mb) | (mb >= 30 ? m : m >> (30 - mb));
    vals[g] = (uint32_t)qi;
}

std::mutex g_grid_mu;

// Dynamic shared memory of a search kernel class, its stack entries.
static_assert(BATCH_THREADS == search::RANGE_CTA, "range warps per CTA");
size_t class_smem(int kc, int height) {
    return kc < BATCH_RANGE_CLASS
               ? sizeof(int2) * search::knn_stack_entries(height) * BATCH_THREADS
               : WARPS_PER_CTA * search::range_warp_bytes(search::range_stack_entries(height), false);
}
int class_entries(int kc, int height) {
    return kc < BATCH_RANGE_CLASS ? search::knn_stack_entries(height) : search::range_stack_entries(height);
}
size_t write_smem(int height) {
    return WARPS_PER_CTA * search::range_warp_bytes(search::range_stack_entries(height), true);
}

int resident_grid(const void* fn, size_t smem = 0) {
    // On a failed query the grid falls back to one CTA per SM (or 1); the
    // kernels are correct for any grid size.
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) sms = 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, BATCH_THREADS, smem) != cudaSuccess) per_sm = 1;
    cudaGetLastError();
    return (sms > 0 ? sms : 1) * (per_sm > 0 ? per_sm : 1);
}

search::RangeLog to_log(const BatchLog& l) { return search::RangeLog{(int2*)l.pool, l.next, l.warps, l.chunks}; }

typedef void (*SearchKernel)(const DevTree*, const BatchReq*, const long long*, int, int, long long, long long,
                             long long*, search::RangeLog, unsigned long long*, int);
SearchKernel search_kernel(int kc) {
    return kc == 0 ? batch_search_kernel<0> : kc == 1 ? batch_search_kernel<1> : kc == 2 ? batch_search_kernel<2>
                                                                              : batch_search_kernel<BATCH_RANGE_CLASS>;
}

}  // namespace

size_t batch_log_bytes(long long chunks) { return sizeof(int2) * search::LOG_CHUNK * (size_t)chunks; }
long long batch_log_chunks(long long warps) { return warps + (warps * 4 < 131072 ? warps * 4 : 131072); }

int batch_kclass(int k) { return k <= 4 ? 0 : k <= 8 ? 1 : 2; }

int batch_search_grid(int kclass, int height) {
    std::lock_guard<std::mutex> lock(g_grid_mu);
    return resident_grid((const void*)search_kernel(kclass), class_smem(kclass, height));
}

int batch_write_grid(int height) {
    std::lock_guard<std::mutex> lock(g_grid_mu);
    return resident_grid((const void*)batch_write_kernel, write_smem(height));
}

void launch_batch_search(const DevTree* trees, const BatchReq* reqs, const long long* req_c1, int r0, int r1,
                         long long c_begin, long long c_end, int kclass, int height, long long* counts,
                         const BatchLog& log, unsigned long long* ctr, int grid, cudaStream_t s) {
    if (c_end <= c_begin || r1 <= r0) return;
    const long long ctas = (c_end - c_begin + WARPS_PER_CTA - 1) / WARPS_PER_CTA;
    const unsigned g = (unsigned)(ctas < grid ? ctas : grid);
    search_kernel(kclass)<<<g, BATCH_THREADS, class_smem(kclass, height), s>>>(
        trees, reqs, req_c1, r0, r1, c_begin, c_end, counts, to_log(log), ctr, class_entries(kclass, height));
}

void launch_batch_keys(const DevTree* trees, const BatchReq* reqs, const long long* qstart, int n, long long total,
                       int req_bits, uint32_t* keys, uint32_t* vals, cudaStream_t s) {
    if (total <= 0 || n <= 0) return;
    batch_key_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(trees, reqs, qstart, n, total, req_bits, keys,
                                                                      vals);
}

void launch_batch_write(const DevTree* trees, const BatchReq* reqs, const int* ridx, const long long* req_c2, int nr,
                        long long c_end, int height, const long long* goff, const BatchLog& log, unsigned long long* ctr,
                        int grid, cudaStream_t s) {
    if (c_end <= 0 || nr <= 0) return;
    const long long ctas = (c_end + WARPS_PER_CTA - 1) / WARPS_PER_CTA;
    const unsigned g = (unsigned)(ctas < grid ? ctas : grid);
    batch_write_kernel<<<g, BATCH_THREADS, write_smem(height), s>>>(trees, reqs, ridx, req_c2, nr, c_end, goff,
                                                                   to_log(log), ctr,
                                                                   search::range_stack_entries(height));
}

}  // namespace ikdg
