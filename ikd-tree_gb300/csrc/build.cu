// Batched, level-synchronous subtree builder.
//
// Replaces the recursive BuildTree (ikd-Tree/ikd_Tree.cpp:573-622), used both
// by Build (:352-364) and by the rebuilds of Rebuild (:624-645).  The split
// rule is kept: every segment is cut at its median on the longest axis of its
// AABB (first axis wins ties, :593-595).  Unlike the reference, internal nodes
// hold no point: segments of at most `fill` points become leaf buckets.
//
// All jobs of a call are built together, on one of three paths chosen by the
// largest job:
// * small (every job <= LB_SMALL points): one CTA per job builds the whole
//   subtree in shared memory (local_build_kernel);
// * medium (jobs <= SPLIT_MIN): one CTA per job splits it in shared memory down to
//   LB_SMALL-point segments (finish_split_kernel: radix-selected median, stable
//   partition), then the local builder finishes them;
// * large: segments above SPLIT_MIN points are split one level at a time by
//   many CTAs each (split_* kernels: histogram of the split axis, the bin that
//   holds the median, selection among that bin's few points, stable partition),
//   the rest goes the medium way.
// All three cut a segment of n points at the point of rank n / 2 on its axis,
// ties in input order (every partition is stable), so they follow one split
// rule.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <climits>

#include "kernels.cuh"
#include "split_grid.h"

namespace ikdg {
namespace {

__device__ __forceinline__ float coord4(const float4& p, int a) { return a == 0 ? p.x : (a == 1 ? p.y : p.z); }

__global__ void init_segs_kernel(const int* job_off, const int* job_link, int njobs,
                                 int4* segs, int* nseg) {
    chain_begin();
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j == 0) nseg[0] = njobs;
    if (j >= njobs) return;
    segs[j] = make_int4(job_off[j], job_off[j + 1], job_link[j], 0);
}

// ---- CTA-local builder ----------------------------------------------------------
// One block builds a whole subtree of up to MAXN points in shared memory:
// three index arrays, each sorted on one coordinate (one bitonic network sorts
// the three arrays of (coordinate key, input position) together), are stably
// partitioned level by level, so every open segment is the same position range
// in all three and its AABB is read off the ends of the ranges.  Per level: one
// thread per open segment takes its node or leaf (the split point is the middle
// of the range on the split axis, which already holds the left half in place);
// one pass over positions marks each point's side and fills the leaves; a block
// prefix sum of the left flags of the two other arrays and a scatter partition
// them.
//
// With leaves of at most `fill` >= 8 points an open segment holds >= 9
// points, so a level has at most 2 * MAXN / 9 < SEGS open segments.
//
// Shape: 1,024 points on 256 threads (about 55 KB of shared memory, four blocks
// per SM); each thread owns four positions and one open segment at most.
constexpr int LB_SMALL = 1024;
constexpr uint16_t LB_DONE = 0xffff;

template <int MAXN, int THREADS>
struct LbShared {
    static constexpr int SEGS = THREADS;
    float4 P[MAXN];            // the job's points by local id (input order)
    uint16_t ord0[3][MAXN];    // index arrays, one per axis (local ids)
    union {
        struct {
            uint16_t ord1[3][MAXN];  // the other buffer of the partition
            uint16_t seg_of[MAXN];   // open segment of a position, LB_DONE once in a leaf
            uint32_t scanv[MAXN];    // exclusive prefix of packed left flags
            uint8_t side[MAXN];      // per local id: 1 = goes right
        } a;
        unsigned long long K[3][MAXN];  // sort keys, only before the first level
    } u;
    uint16_t ss[2][SEGS], se[2][SEGS];
    int slink[2][SEGS];
    int swide[2][SEGS];        // wide record above the segment's parent, its position there
    uint8_t swpos[2][SEGS];
    int snode[SEGS];           // node or leaf index, -1 when allocation failed
    uint16_t snext[SEGS];      // first child segment of a node
    int8_t saxis[SEGS];        // split axis, -1 for leaves
    uint32_t wsum[THREADS / 32];
    PoolRun run_leaf, run_node;
    int free_leaf_n, free_node_n;  // free-stack sizes when the runs were taken
    uint32_t level_total;          // leaves (low 16 bits) and nodes of the current level
    int nseg[2];
    int overflow;
};
static_assert(4 * (sizeof(LbShared<LB_SMALL, 256>) + 1024) <= 228 * 1024, "four local builders per SM");

__device__ __forceinline__ float key_float(uint32_t k) {
    uint32_t u = (k & 0x80000000u) ? (k ^ 0x80000000u) : ~k;
    return __uint_as_float(u);
}

// Ascending bitonic sort of K[a][0 .. size) for the three arrays at once, size a
// power of two of at most 4 * THREADS.  Thread t holds elements 4 t .. 4 t + 3 of
// each array in registers: partners up to 64 elements apart are in the thread or
// the warp, only longer strides go through shared memory (6 of the 55 steps for
// 1,024 elements; every step went through it before, which bound the sort by
// shared-memory bandwidth).
template <int MAXN, int THREADS>
__device__ void lb_bitonic3(unsigned long long (*K)[MAXN], int size) {
    static_assert(MAXN == 4 * THREADS, "four elements per thread");
    typedef unsigned long long u64;
    const int e0 = threadIdx.x * 4;
    u64 v[3][4];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int r = 0; r < 4; ++r) v[a][r] = e0 + r < size ? K[a][e0 + r] : ~0ull;
    for (int kk = 2; kk <= size; kk <<= 1) {
        int j = kk >> 1;
        if (j >= 128) {
            for (; j >= 128; j >>= 1) {
                __syncthreads();
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int r = 0; r < 4; ++r) K[a][e0 + r] = v[a][r];
                __syncthreads();
                const bool keep_min = ((e0 & j) == 0) == ((e0 & kk) == 0);
#pragma unroll
                for (int a = 0; a < 3; ++a)
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const u64 o = K[a][(e0 + r) ^ j];
                        v[a][r] = (o < v[a][r]) == keep_min ? o : v[a][r];
                    }
            }
        }
        for (; j >= 4; j >>= 1) {
            const bool keep_min = ((e0 & j) == 0) == ((e0 & kk) == 0);
#pragma unroll
            for (int a = 0; a < 3; ++a)
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const u64 o = __shfl_xor_sync(0xffffffffu, v[a][r], j >> 2);
                    v[a][r] = (o < v[a][r]) == keep_min ? o : v[a][r];
                }
        }
        // strides 2 and 1 inside the thread
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            auto cx = [&](int x, int y, bool up) {
                const u64 p = v[a][x], q = v[a][y];
                const bool sw = (p > q) == up;
                v[a][x] = sw ? q : p;
                v[a][y] = sw ? p : q;
            };
            const bool up = (e0 & kk) == 0;
            if (j == 2) {
                cx(0, 2, up);
                cx(1, 3, up);
            }
            if (kk == 2) {
                cx(0, 1, true);
                cx(2, 3, false);
            } else {
                cx(0, 1, up);
                cx(2, 3, up);
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int r = 0; r < 4; ++r) K[a][e0 + r] = v[a][r];
    __syncthreads();
}

// Nodes and leaves of the subtree the builders make from n points with leaf
// fill `fill`: a segment of more than `fill` points is a node whose children
// hold n / 2 and n - n / 2 points, so the sizes of one level take at most two
// consecutive values.
__device__ __forceinline__ void subtree_counts(int n, int fill, int* nodes, int* leaves) {
    int lo = n, c_lo = 1, c_hi = 0;  // c_lo segments of lo points, c_hi of lo + 1
    int nn = 0, nl = 0;
    for (int guard = 0; guard < 40 && c_lo + c_hi > 0; ++guard) {
        int n_lo = 0, n_hi = 0, next = 0;
        bool have = false;
        for (int h = 0; h < 2; ++h) {
            const int size = lo + h, c = h ? c_hi : c_lo;
            if (c == 0) continue;
            if (size <= fill) {
                nl += c;
                continue;
            }
            nn += c;
            const int a = size / 2, b = size - size / 2;  // b == a or a + 1
            if (!have) {
                next = a;
                have = true;
            }
            // children sizes at this level are next or next + 1
            n_lo += (a == next ? c : 0) + (b == next ? c : 0);
            n_hi += (a == next + 1 ? c : 0) + (b == next + 1 ? c : 0);
        }
        lo = next;
        c_lo = n_lo;
        c_hi = n_hi;
    }
    *nodes = nn;
    *leaves = nl;
}

template <int MAXN, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS >= 1024 ? 1 : 4) local_build_kernel(DevTree t, const float4* pts,
                                                                 const int4* jobs, const int* njobs,
                                                                 int max_jobs, int fill) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char lb_raw[];
    constexpr int PPT = MAXN / THREADS;
    constexpr int SEGS = THREADS;
    static_assert(MAXN % THREADS == 0 && PPT == 4 && MAXN <= 65535, "local builder shape");
    static_assert(2 * MAXN / 9 < SEGS, "segment table too small");
    LbShared<MAXN, THREADS>& sm = *reinterpret_cast<LbShared<MAXN, THREADS>*>(lb_raw);
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    // The producers count past the capacity when it overflows (and flag it):
    // never read beyond the job array.
    const int nj = min(*njobs, max_jobs);
    for (int job = blockIdx.x; job < nj; job += gridDim.x) {
        const int4 jb = jobs[job];
        const int n = jb.y - jb.x;
        if (n > MAXN || n < 0 || fill < 8) {  // cannot happen: the host guarantees all three
            if (tid == 0) atomicOr(&t.st->err, ERR_SEG);
            continue;
        }
        for (int i = tid; i < n; i += THREADS) sm.P[i] = pts[(long long)jb.x + i];
        int size = 2;
        while (size < n) size <<= 1;
        __syncthreads();
        for (int i = tid; i < size; i += THREADS) {
            if (i < n) {
                const float4 p = sm.P[i];
                sm.u.K[0][i] = ((unsigned long long)float_key(p.x) << 32) | (unsigned)i;
                sm.u.K[1][i] = ((unsigned long long)float_key(p.y) << 32) | (unsigned)i;
                sm.u.K[2][i] = ((unsigned long long)float_key(p.z) << 32) | (unsigned)i;
            } else {
                sm.u.K[0][i] = sm.u.K[1][i] = sm.u.K[2][i] = ~0ull;
            }
        }
        __syncthreads();
        lb_bitonic3<MAXN, THREADS>(sm.u.K, size);
        for (int i = tid; i < n; i += THREADS) {
            sm.ord0[0][i] = (uint16_t)sm.u.K[0][i];
            sm.ord0[1][i] = (uint16_t)sm.u.K[1][i];
            sm.ord0[2][i] = (uint16_t)sm.u.K[2][i];
        }
        __syncthreads();  // the sort keys are dead from here on
        for (int i = tid; i < n; i += THREADS) sm.u.a.seg_of[i] = 0;
        if (tid == 0) {
            sm.nseg[0] = 1;
            sm.nseg[1] = 0;
            sm.overflow = 0;
            sm.ss[0][0] = 0;
            sm.se[0][0] = (uint16_t)n;
            sm.slink[0][0] = jb.z;
            const int2 wi = t.winfo[jb.z >> 1];
            sm.swide[0][0] = wi.x;
            sm.swpos[0][0] = (uint8_t)wi.y;
            // The whole subtree's nodes and leaves from the pools at once
            // (its shape follows from n and the fill); level l takes the
            // indices after those of levels 0 .. l-1.
            int nn = 0, nl = 0;
            subtree_counts(n, fill, &nn, &nl);
            sm.free_leaf_n = t.st->free_leaf_n;
            sm.free_node_n = t.st->free_node_n;
            sm.run_leaf = pool_reserve(&t.st->free_leaf_taken, sm.free_leaf_n, &t.st->leaf_top, nl);
            sm.run_node = pool_reserve(&t.st->free_node_taken, sm.free_node_n, &t.st->node_top, nn);
        }
        __syncthreads();
        uint16_t(*oc)[MAXN] = sm.ord0;
        uint16_t(*on)[MAXN] = sm.u.a.ord1;
        int cb = 0;
        const int i0 = tid * PPT;
        int leaf_base = 0, node_base = 0;  // indices of the runs taken by earlier levels
        for (int level = 0; level < 64; ++level) {
            const int S = sm.nseg[cb];
            if (S == 0) break;
            // One thread per open segment: a leaf, or a node with its axis,
            // its split value and two child segments.  The level's leaves and
            // nodes are ranked by ballots and taken from the pools with one
            // reservation each.
            const int sg = tid;
            const bool live = sg < S;
            int s = 0, e = 0, link = 0;
            if (live) {
                s = sm.ss[cb][sg];
                e = sm.se[cb][sg];
                link = sm.slink[cb][sg];
            }
            const int cnt = e - s;
            const bool is_leaf = live && cnt <= fill, is_node = live && cnt > fill;
            const unsigned lm = __ballot_sync(0xffffffffu, is_leaf), nm = __ballot_sync(0xffffffffu, is_node);
            if (lane == 0) sm.wsum[warp] = (uint32_t)__popc(lm) | ((uint32_t)__popc(nm) << 16);
            __syncthreads();
            if (warp == 0) {
                const uint32_t w = lane < THREADS / 32 ? sm.wsum[lane] : 0u;
                uint32_t wi = w;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
                    if (lane >= o) wi += y;
                }
                if (lane < THREADS / 32) sm.wsum[lane] = wi - w;
                if (lane == 31) sm.level_total = wi;
            }
            __syncthreads();
            const uint32_t level_total = sm.level_total;
            if (live) {
                const uint32_t wb = sm.wsum[warp];
                const unsigned below = (1u << lane) - 1u;
                const int parent = link >> 1, side = link & 1;
                const int2 wi = make_int2(sm.swide[cb][sg], sm.swpos[cb][sg]);
                Box3 b = empty_box();
                if (cnt > 0)
                    for (int a = 0; a < 3; ++a) {
                        b.lo[a] = coord4(sm.P[oc[a][s]], a);
                        b.hi[a] = coord4(sm.P[oc[a][e - 1]], a);
                    }
                sm.saxis[sg] = -1;
                sm.snode[sg] = -1;
                if (is_leaf) {
                    const int L = pool_pick(sm.run_leaf, t.free_leaf, sm.free_leaf_n, t.leaf_cap,
                                            leaf_base + (int)(wb & 0xffffu) + __popc(lm & below), t.st,
                                            ERR_POOL_LEAF);
                    sm.snode[sg] = L;
                    if (L >= 0) {
                        t.leaf_n[L] = cnt;
                        t.lparent[L] = link;
                        write_child_box(t.node, parent, side, b);
                        write_child_code(t.node, parent, side, leaf_code(L));
                        write_child_cnt(t.ncnt, parent, side, cnt, 0);
                        wide_link(t, wi, side, leaf_code(L), b, cnt);
                    }
                } else {
                    const int X = pool_pick(sm.run_node, t.free_node, sm.free_node_n, t.node_cap,
                                            node_base + (int)(wb >> 16) + __popc(nm & below), t.st, ERR_POOL);
                    float ext[3];
                    for (int a = 0; a < 3; ++a) ext[a] = __fsub_rn(b.hi[a], b.lo[a]);
                    int axis = 0;
                    if (ext[1] > ext[axis]) axis = 1;
                    if (ext[2] > ext[axis]) axis = 2;
                    const int mid = s + cnt / 2;
                    const int r = X >= 0 ? atomicAdd(&sm.nseg[cb ^ 1], 2) : 0;
                    if (X >= 0 && r + 1 >= SEGS) {  // cannot happen by the bound above; guard anyway
                        atomicOr(&t.st->err, ERR_SEG);
                        sm.overflow = 1;
                    } else if (X >= 0) {
                        sm.snode[sg] = X;
                        sm.saxis[sg] = (int8_t)axis;
                        sm.snext[sg] = (uint16_t)r;
                        t.node[4 * X + 3] = make_float4(__int_as_float(0), __int_as_float(0),
                                                        coord4(sm.P[oc[axis][mid]], axis), __int_as_float(axis));
                        t.nparent[X] = link;
                        int h = 0;
                        for (int m = cnt; m > fill; m -= m / 2) ++h;
                        t.nheight[X] = h;
                        write_child_box(t.node, parent, side, b);
                        write_child_code(t.node, parent, side, X);
                        write_child_cnt(t.ncnt, parent, side, cnt, 0);
                        wide_link(t, wi, side, X, b, cnt);
                        const int2 wx = wide_below(wi, side, X);
                        t.winfo[X] = wx;
                        sm.swide[cb ^ 1][r] = sm.swide[cb ^ 1][r + 1] = wx.x;
                        sm.swpos[cb ^ 1][r] = sm.swpos[cb ^ 1][r + 1] = (uint8_t)wx.y;
                        sm.ss[cb ^ 1][r] = (uint16_t)s;
                        sm.se[cb ^ 1][r] = (uint16_t)mid;
                        sm.slink[cb ^ 1][r] = X * 2;
                        sm.ss[cb ^ 1][r + 1] = (uint16_t)mid;
                        sm.se[cb ^ 1][r + 1] = (uint16_t)e;
                        sm.slink[cb ^ 1][r + 1] = X * 2 + 1;
                    }
                }
            }
            __syncthreads();
            if (sm.overflow) break;
            leaf_base += (int)(level_total & 0xffffu);
            node_base += (int)(level_total >> 16);
            // Leaves take their points; node segments mark each point's side
            // from its position in the split axis's array.
#pragma unroll
            for (int r = 0; r < PPT; ++r) {
                const int i = i0 + r;
                if (i >= n) break;
                const int sg = sm.u.a.seg_of[i];
                if (sg == LB_DONE) continue;
                const int ax = sm.saxis[sg];
                const int s = sm.ss[cb][sg];
                if (ax < 0) {
                    const int L = sm.snode[sg];
                    if (L >= 0) {
                        float4 q = sm.P[oc[0][i]];
                        q.w = __uint_as_float(__float_as_uint(q.w) & ID_MASK);
                        t.pts[(long long)L * LEAF_CAP + (i - s)] = q;
                    }
                } else {
                    const int mid = s + (sm.se[cb][sg] - s) / 2;
                    sm.u.a.side[oc[ax][i]] = i >= mid ? 1 : 0;
                }
            }
            __syncthreads();
            // Packed left flags of the two arrays that are not the split
            // axis's: (axis + 1) % 3 in the low half, (axis + 2) % 3 in the high.
            uint32_t v[PPT];
            uint32_t sum = 0;
#pragma unroll
            for (int r = 0; r < PPT; ++r) {
                const int i = i0 + r;
                uint32_t f = 0;
                if (i < n) {
                    const int sg = sm.u.a.seg_of[i];
                    if (sg != LB_DONE) {
                        const int ax = sm.saxis[sg];
                        if (ax >= 0) {
                            const int b1 = ax == 2 ? 0 : ax + 1, b2 = ax == 0 ? 2 : ax - 1;
                            f = (uint32_t)(sm.u.a.side[oc[b1][i]] ^ 1) | ((uint32_t)(sm.u.a.side[oc[b2][i]] ^ 1) << 16);
                        }
                    }
                }
                v[r] = sum;
                sum += f;
            }
            uint32_t inc = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
                if (lane >= o) inc += y;
            }
            if (lane == 31) sm.wsum[warp] = inc;
            __syncthreads();
            if (warp == 0) {
                uint32_t w = lane < THREADS / 32 ? sm.wsum[lane] : 0u;
                uint32_t wi = w;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
                    if (lane >= o) wi += y;
                }
                if (lane < THREADS / 32) sm.wsum[lane] = wi - w;
            }
            __syncthreads();
            const uint32_t tbase = sm.wsum[warp] + inc - sum;
#pragma unroll
            for (int r = 0; r < PPT; ++r)
                if (i0 + r < n) sm.u.a.scanv[i0 + r] = tbase + v[r];
            __syncthreads();
            // Scatter: the split axis's array keeps its order, the other two
            // are partitioned stably; positions move to the child segments.
            if (tid == 0) sm.nseg[cb] = 0;  // every thread read it at the top of the level
#pragma unroll
            for (int r = 0; r < PPT; ++r) {
                const int i = i0 + r;
                if (i >= n) break;
                const int sg = sm.u.a.seg_of[i];
                if (sg == LB_DONE) continue;
                const int ax = sm.saxis[sg];
                if (ax < 0) {
                    sm.u.a.seg_of[i] = LB_DONE;
                    continue;
                }
                const int s = sm.ss[cb][sg];
                const int mid = s + (sm.se[cb][sg] - s) / 2;
                const int b1 = ax == 2 ? 0 : ax + 1, b2 = ax == 0 ? 2 : ax - 1;
                const uint32_t rel = sm.u.a.scanv[i] - sm.u.a.scanv[s];
                on[ax][i] = oc[ax][i];
                const uint16_t j1 = oc[b1][i], j2 = oc[b2][i];
                const int c1 = (int)(rel & 0xffffu), c2 = (int)(rel >> 16);
                on[b1][sm.u.a.side[j1] ? mid + (i - s - c1) : s + c1] = j1;
                on[b2][sm.u.a.side[j2] ? mid + (i - s - c2) : s + c2] = j2;
                sm.u.a.seg_of[i] = (uint16_t)(sm.snext[sg] + (i < mid ? 0 : 1));
            }
            __syncthreads();
            uint16_t(*tmp)[MAXN] = oc;
            oc = on;
            on = tmp;
            cb ^= 1;
        }
        __syncthreads();
    }
}

// Exclusive block prefix of a per-thread value; the block total goes to
// *total.  The shared words are free for reuse when it returns.
template <int THREADS>
__device__ __forceinline__ uint32_t block_scan_u32(uint32_t v, uint32_t* wsum, uint32_t* tot, uint32_t* total) {
    static_assert(THREADS <= 32 * 32, "one warp scans the warp sums");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < THREADS / 32 ? wsum[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < THREADS / 32) wsum[lane] = wi - w;
        if (lane == 31) *tot = wi;
    }
    __syncthreads();
    const uint32_t r = wsum[warp] + inc - v;
    *total = *tot;
    __syncthreads();
    return r;
}

// ---- segments of at most SPLIT_MIN points ------------------------------------------------
// A block takes a whole segment into shared memory, splits it down to LB_SMALL-
// point pieces there (at most three splits, the points of the open piece in
// registers meanwhile) and writes the pieces out for the local builder.  (One
// launch per level with every pass over a segment in L2: 160 us for a 2M-point
// build, 61 us now.)
constexpr int FIN_THREADS = 512;
constexpr int FIN_ROUNDS = SPLIT_MIN / FIN_THREADS;
constexpr int FIN_WARPS = FIN_THREADS / 32;

struct FinShared {
    float4 P[SPLIT_MIN];
    int hist[256];
    uint32_t red[FIN_WARPS][6];
    uint32_t cnt[FIN_ROUNDS * FIN_WARPS];  // packed (below, equal) counts, then their prefix
    uint32_t box[6];
    int3 open[4];                          // {s, e, link} pieces to split
    int nopen, node, axis, digit, rank;
};

__global__ void __launch_bounds__(FIN_THREADS, 2) finish_split_kernel(DevTree t, const float4* src,
                                                                      const int4* segs, const int* nseg,
                                                                      int max_segs, float4* __restrict__ out,
                                                                      int4* __restrict__ local_jobs, int* nlocal,
                                                                      int max_local, int fill) {
    chain_begin();
    extern __shared__ __align__(16) unsigned char fin_raw[];
    FinShared& sm = *reinterpret_cast<FinShared*>(fin_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int S = min(*nseg, max_segs);
    auto local = [&](int s, int e, int link) {  // one thread
        const int r = atomicAdd(nlocal, 1);
        if (r < max_local) local_jobs[r] = make_int4(s, e, link, 0);
        else atomicOr(&t.st->err, ERR_SEG);
    };
    for (int q = blockIdx.x; q < S; q += gridDim.x) {
        const int4 sg = segs[q];
        const int s0 = sg.x, total = sg.y - sg.x;
        __syncthreads();  // the previous segment's shared words are free again
        if (total > SPLIT_MIN || total < 0) {  // cannot happen: the lists hold such segments only
            if (tid == 0) atomicOr(&t.st->err, ERR_SEG);
            continue;
        }
#pragma unroll
        for (int r = 0; r < FIN_ROUNDS; ++r)
            if (r * FIN_THREADS + tid < total) sm.P[r * FIN_THREADS + tid] = src[s0 + r * FIN_THREADS + tid];
        if (tid == 0) {
            sm.nopen = 0;
            if (total > LB_SMALL) sm.open[sm.nopen++] = make_int3(0, total, sg.z);
            else local(s0, s0 + total, sg.z);
        }
        __syncthreads();
        while (sm.nopen > 0) {
            const int3 o = sm.open[sm.nopen - 1];
            const int s = o.x, cnt = o.y - o.x, m = cnt / 2, link = o.z;
            __syncthreads();  // everyone has the piece
            if (tid == 0) --sm.nopen;
            float4 p[FIN_ROUNDS];
            uint32_t mn[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, mx[3] = {0u, 0u, 0u};
#pragma unroll
            for (int r = 0; r < FIN_ROUNDS; ++r) {
                const int i = r * FIN_THREADS + tid;
                if (i < cnt) {
                    p[r] = sm.P[s + i];
                    const uint32_t kx = float_key(p[r].x), ky = float_key(p[r].y), kz = float_key(p[r].z);
                    mn[0] = min(mn[0], kx), mx[0] = max(mx[0], kx);
                    mn[1] = min(mn[1], ky), mx[1] = max(mx[1], ky);
                    mn[2] = min(mn[2], kz), mx[2] = max(mx[2], kz);
                }
            }
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                mn[a] = __reduce_min_sync(0xffffffffu, mn[a]);
                mx[a] = __reduce_max_sync(0xffffffffu, mx[a]);
                if (lane == 0) sm.red[warp][a] = mn[a], sm.red[warp][3 + a] = mx[a];
            }
            __syncthreads();
            if (warp == 0) {
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const uint32_t lo = __reduce_min_sync(0xffffffffu, lane < FIN_WARPS ? sm.red[lane][a] : 0xffffffffu);
                    const uint32_t hi = __reduce_max_sync(0xffffffffu, lane < FIN_WARPS ? sm.red[lane][3 + a] : 0u);
                    if (lane == 0) sm.box[a] = lo, sm.box[3 + a] = hi;
                }
                __syncwarp();
                if (lane == 0) {
                    Box3 b;
                    float ext[3];
                    for (int a = 0; a < 3; ++a) {
                        b.lo[a] = key_float(sm.box[a]);
                        b.hi[a] = key_float(sm.box[3 + a]);
                        ext[a] = __fsub_rn(b.hi[a], b.lo[a]);
                    }
                    int axis = 0;
                    if (ext[1] > ext[axis]) axis = 1;
                    if (ext[2] > ext[axis]) axis = 2;
                    const int X = alloc_node(t);
                    sm.node = X;
                    sm.axis = axis;
                    if (X >= 0) {
                        const int parent = link >> 1, side = link & 1;
                        t.nparent[X] = link;
                        int h = 0;
                        for (int k = cnt; k > fill; k -= k / 2) ++h;
                        t.nheight[X] = h;
                        write_child_box(t.node, parent, side, b);
                        write_child_code(t.node, parent, side, X);
                        write_child_cnt(t.ncnt, parent, side, cnt, 0);
                        const int2 wi = t.winfo[parent];
                        wide_link(t, wi, side, X, b, cnt);
                        t.winfo[X] = wide_below(wi, side, X);
                    }
                }
            }
            __syncthreads();
            const int X = sm.node, axis = sm.axis;
            if (X < 0) continue;  // the pool is exhausted (flagged by alloc_node): the points are dropped
            uint32_t key[FIN_ROUNDS];
#pragma unroll
            for (int r = 0; r < FIN_ROUNDS; ++r)
                key[r] = r * FIN_THREADS + tid < cnt ? float_key(coord4(p[r], axis)) : 0xffffffffu;
            uint32_t v = 0;
            int rank = m;
            for (int b = 32; b > 0; b -= 8) {
                if (tid < 256) sm.hist[tid] = 0;
                __syncthreads();
#pragma unroll
                for (int r = 0; r < FIN_ROUNDS; ++r)
                    if (r * FIN_THREADS + tid < cnt && (b < 32 ? key[r] >> b : 0u) == v)
                        atomicAdd(&sm.hist[(key[r] >> (b - 8)) & 255u], 1);
                __syncthreads();
                if (warp == 0) {
                    int c[8], sum = 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) c[j] = sm.hist[lane * 8 + j], sum += c[j];
                    int inc = sum;
#pragma unroll
                    for (int k = 1; k < 32; k <<= 1) {
                        const int y = __shfl_up_sync(0xffffffffu, inc, k);
                        if (lane >= k) inc += y;
                    }
                    int r = rank - (inc - sum);
                    if (r >= 0 && r < sum) {  // exactly one lane
                        int d = 0;
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (r < c[j]) {
                                d = j;
                                break;
                            }
                            r -= c[j];
                        }
                        sm.digit = lane * 8 + d;
                        sm.rank = r;
                    }
                }
                __syncthreads();
                v = (v << 8) | (uint32_t)sm.digit;
                rank = sm.rank;
            }
            if (tid == 0)
                t.node[4 * X + 3] = make_float4(__int_as_float(0), __int_as_float(0), key_float(v), __int_as_float(axis));
            // Stable partition: points in order of (round, thread).
            const uint32_t need = (uint32_t)rank;  // keys equal to v that go left
            unsigned lt[FIN_ROUNDS], eq[FIN_ROUNDS];
#pragma unroll
            for (int r = 0; r < FIN_ROUNDS; ++r) {
                const bool in = r * FIN_THREADS + tid < cnt;
                lt[r] = __ballot_sync(0xffffffffu, in && key[r] < v);
                eq[r] = __ballot_sync(0xffffffffu, in && key[r] == v);
                if (lane == 0) sm.cnt[r * FIN_WARPS + warp] = (uint32_t)__popc(lt[r]) | ((uint32_t)__popc(eq[r]) << 16);
            }
            __syncthreads();
            if (warp == 0) {
                constexpr int PER = FIN_ROUNDS * FIN_WARPS / 32;
                uint32_t c[PER], sum = 0;
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    c[j] = sum;
                    sum += sm.cnt[lane * PER + j];
                }
                uint32_t inc = sum;
#pragma unroll
                for (int k = 1; k < 32; k <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, inc, k);
                    if (lane >= k) inc += y;
                }
                __syncwarp();
#pragma unroll
                for (int j = 0; j < PER; ++j) sm.cnt[lane * PER + j] = inc - sum + c[j];
            }
            __syncthreads();
            const unsigned below = (1u << lane) - 1u;
#pragma unroll
            for (int r = 0; r < FIN_ROUNDS; ++r) {
                const int i = r * FIN_THREADS + tid;
                if (i < cnt) {
                    const uint32_t base = sm.cnt[r * FIN_WARPS + warp];
                    const uint32_t l = (base & 0xffffu) + __popc(lt[r] & below), q2 = (base >> 16) + __popc(eq[r] & below);
                    const uint32_t lb = l + min(q2, need);
                    const bool left = key[r] < v || (key[r] == v && q2 < need);
                    sm.P[s + (left ? (int)lb : m + i - (int)lb)] = p[r];  // (left: lb < m; right: below cnt)
                }
            }
            if (tid == 0) {
                for (int c = 0; c < 2; ++c) {
                    const int cs = c == 0 ? s : s + m, ce = c == 0 ? s + m : s + cnt;
                    if (ce - cs > LB_SMALL) sm.open[sm.nopen++] = make_int3(cs, ce, X * 2 + c);
                    else local(s0 + cs, s0 + ce, X * 2 + c);
                }
            }
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < FIN_ROUNDS; ++r)
            if (r * FIN_THREADS + tid < total) out[s0 + r * FIN_THREADS + tid] = sm.P[r * FIN_THREADS + tid];
    }
}

// ---- multi-block splitter for large segments ------------------------------------------------
// Segments above SPLIT_MIN points: one level per round of five launches, every
// segment cut into tiles of SPLIT_TILE points, a block per tile (split_grid.h).
//   hist      keys on the split axis into SPLIT_BINS bins over the segment's range
//   pick      the bin that holds the point of rank n / 2 (a block per segment)
//   classify  per tile the points of lower bins; the picked bin's points, (key,
//             position), into the segment's candidate list
//   select    the (key, position) of rank n / 2 among the candidates, the tiles'
//             left counts and their prefix sum, the node, the child segments (a
//             block per segment)
//   scatter   stable partition by (key, position), the children's AABBs
// A uniform segment's candidates are ~1/1,000 of it; a stray point far away or many
// equal keys put most of the segment on the list (select_large).
// This took the place of sorting the three coordinates once and partitioning the
// three sorted index arrays per level with random gathers of the sides (109
// launches): a 2M-point build moves 16 instead of ~100 bytes per point and level
// and takes 700 us of kernels (370 of them these) against 1,950 us.  Bound by L2
// bandwidth (level passes) and by the latency of the per-segment blocks.
constexpr int SPLIT_THREADS = 256;
constexpr int SPLIT_ROUNDS = 8;  // points per thread
constexpr int SPLIT_BINS = 2048;
constexpr int HIST_THREADS = 1024;
static_assert(SPLIT_TILE == SPLIT_THREADS * SPLIT_ROUNDS && HIST_TILE == HIST_THREADS * SPLIT_ROUNDS, "points per thread");
constexpr int SPLIT_CACHE = 4096;  // candidates kept in shared memory by select

// The split axis of a segment (longest extent, first on ties) and its bins: equal
// widths over the segment's range.  The bin grows with the coordinate (every
// operation rounds monotonically), which is all the selection needs; an outlier
// that stretches the range makes the candidate lists longer.  (Bins of the
// ordered keys put a quarter of an octave into each where the range spans zero:
// 20k candidates also where the points are even.)
struct SplitAxis {
    int axis;
    float lo, scale;
    __device__ __forceinline__ int bin(float x) const {
        const int b = (int)__fmul_rn(__fsub_rn(x, lo), scale);
        return min(max(b, 0), SPLIT_BINS - 1);
    }
};
__device__ __forceinline__ SplitAxis split_axis(const uint32_t* box) {
    const float x = key_float(box[0]), y = key_float(box[1]), z = key_float(box[2]);
    float ext = __fsub_rn(key_float(box[3]), x);
    const float ey = __fsub_rn(key_float(box[4]), y), ez = __fsub_rn(key_float(box[5]), z);
    SplitAxis r{0, x, 0.f};
    if (ey > ext) r.axis = 1, r.lo = y, ext = ey;
    if (ez > ext) r.axis = 2, r.lo = z, ext = ez;
    r.scale = __fdiv_rn((float)SPLIT_BINS, ext);
    return r;
}

// First tile of a segment in the tile arrays: segments hold more than SPLIT_MIN
// = 2 tiles of points, so s / 1024 leaves room for every segment's own tiles.
__device__ __forceinline__ int split_tile0(int s) { return s >> 10; }
static_assert(SPLIT_TILE == 2048 && SPLIT_MIN >= 2 * SPLIT_TILE, "tile array layout");

__device__ __forceinline__ void split_box_reset(uint32_t* box) {
    for (int a = 0; a < 3; ++a) {
        box[a] = 0xffffffffu;
        box[3 + a] = 0u;
    }
}

// A level's counters in one word, so that one addition gives a new segment its index and
// the places of its tiles: segments from bit 42 on, tiles from bit 21, htiles below (n is
// below 2^30, so there are at most 2^18 segments and 2^20 tiles).
struct SplitCount {
    int segs, tiles, htiles;
};
__device__ __forceinline__ SplitCount split_unpack(unsigned long long v) {
    return SplitCount{(int)(v >> 42), (int)(v >> 21 & 0x1fffffu), (int)(v & 0x1fffffu)};
}
// Opens segment [s, e) below `link` (one thread); its index, or -1 when the list is full
// (flagged), and where its tiles go.
__device__ __forceinline__ SplitCount split_take(const SplitLevel& lv, int cap, int s, int e, int link, DevStatus* st) {
    const int tiles = (e - s + SPLIT_TILE - 1) / SPLIT_TILE, htiles = (e - s + HIST_TILE - 1) / HIST_TILE;
    SplitCount c = split_unpack(atomicAdd(lv.n, (1ull << 42) | (unsigned long long)tiles << 21 | (unsigned long long)htiles));
    if (c.segs >= cap) {  // cannot happen: see split_grid.h
        atomicOr(&st->err, ERR_SEG);
        c.segs = -1;
        return c;
    }
    lv.seg[c.segs] = make_int4(s, e, link, 0);
    lv.cand_n[c.segs] = 0;
    split_box_reset(lv.box + 6 * c.segs);
    return c;
}
// Lists the tiles of a segment split_take opened (the whole block).
template <int THREADS>
__device__ __forceinline__ void split_list(const SplitLevel& lv, const SplitCount& c, int s, int e) {
    const int tiles = (e - s + SPLIT_TILE - 1) / SPLIT_TILE, htiles = (e - s + HIST_TILE - 1) / HIST_TILE;
    for (int i = threadIdx.x; i < tiles; i += THREADS) lv.tile[c.tiles + i] = make_int4(s, e, c.segs, i);
    for (int i = threadIdx.x; i < htiles; i += THREADS) lv.htile[c.htiles + i] = make_int4(s, e, c.segs, i);
}
__device__ __forceinline__ int split_segs(const SplitLevel& lv, int cap) { return min(split_unpack(*lv.n).segs, cap); }

// Jobs above SPLIT_MIN points open the splitter's first level; the others go to
// the small list, their points copied to `exits` (a block per job).
__global__ void __launch_bounds__(SPLIT_THREADS) split_open_kernel(const float4* pts,
                                                                   const int* job_off,
                                                                   const int* job_link, int njobs,
                                                                   SplitLevel lv, int cap, float4* __restrict__ exits,
                                                                   int4* __restrict__ small, int* nsmall, int max_small,
                                                                   DevStatus* st) {
    chain_begin();
    __shared__ SplitCount at;
    for (int j = blockIdx.x; j < njobs; j += gridDim.x) {
        const int s = job_off[j], e = job_off[j + 1];
        const bool big = e - s > SPLIT_MIN;
        __syncthreads();
        if (threadIdx.x == 0) {
            if (big) {
                at = split_take(lv, cap, s, e, job_link[j], st);
            } else {
                const int r = atomicAdd(nsmall, 1);
                if (r >= max_small)
                    atomicOr(&st->err, ERR_SEG);
                else
                    small[r] = make_int4(s, e, job_link[j], 0);
            }
        }
        __syncthreads();
        if (!big)
            for (int i = s + threadIdx.x; i < e; i += SPLIT_THREADS) exits[i] = pts[i];
        else if (at.segs >= 0)
            split_list<SPLIT_THREADS>(lv, at, s, e);
    }
}

// A point into a thread's box; the warp's boxes into a shared one (reset before).
__device__ __forceinline__ void split_grow(uint32_t* b, const float4& p) {
    const uint32_t k[3] = {float_key(p.x), float_key(p.y), float_key(p.z)};
    for (int a = 0; a < 3; ++a) {
        b[a] = min(b[a], k[a]);
        b[3 + a] = max(b[3 + a], k[a]);
    }
}
__device__ __forceinline__ void split_flush(uint32_t* sm, const uint32_t* b) {
    for (int a = 0; a < 3; ++a) {
        const uint32_t lo = __reduce_min_sync(0xffffffffu, b[a]), hi = __reduce_max_sync(0xffffffffu, b[3 + a]);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(sm + a, lo);
            atomicMax(sm + 3 + a, hi);
        }
    }
}

__global__ void __launch_bounds__(SPLIT_THREADS) split_box_kernel(const float4* pts, SplitLevel lv,
                                                                  int max_tiles) {
    chain_begin();
    __shared__ uint32_t sm[6];
    const int4 sg = lv.tile[blockIdx.x];
    if ((int)blockIdx.x >= min(split_unpack(*lv.n).tiles, max_tiles)) return;
    const int q = sg.z, t0 = sg.x + sg.w * SPLIT_TILE;
    if (threadIdx.x == 0) split_box_reset(sm);
    __syncthreads();
    uint32_t b[6];
    split_box_reset(b);
    for (int i = t0 + threadIdx.x; i < min(t0 + SPLIT_TILE, sg.y); i += SPLIT_THREADS) split_grow(b, pts[i]);
    split_flush(sm, b);
    __syncthreads();
    if (threadIdx.x < 3) atomicMin(lv.box + 6 * q + threadIdx.x, sm[threadIdx.x]);
    else if (threadIdx.x < 6) atomicMax(lv.box + 6 * q + threadIdx.x, sm[threadIdx.x]);
}

__global__ void __launch_bounds__(HIST_THREADS) split_hist_kernel(const float4* pts, SplitLevel lv,
                                                                   int max_tiles, int* __restrict__ hist) {
    chain_begin();
    __shared__ int h[SPLIT_BINS];
    const int4 sg = lv.htile[blockIdx.x];
    if ((int)blockIdx.x >= min(split_unpack(*lv.n).htiles, max_tiles)) return;
    const int q = sg.z, t0 = sg.x + sg.w * HIST_TILE;
    const SplitAxis ax = split_axis(lv.box + 6 * q);
    for (int i = threadIdx.x; i < SPLIT_BINS; i += HIST_THREADS) h[i] = 0;
    __syncthreads();
    const float* c = reinterpret_cast<const float*>(pts) + ax.axis;
#pragma unroll
    for (int r = 0; r < SPLIT_ROUNDS; ++r) {
        const int i = t0 + r * HIST_THREADS + threadIdx.x;
        if (i < sg.y) atomicAdd(&h[ax.bin(c[4ll * i])], 1);
    }
    __syncthreads();
    int* g = hist + (long long)q * SPLIT_BINS;
    for (int i = threadIdx.x; i < SPLIT_BINS; i += HIST_THREADS)
        if (h[i]) atomicAdd(g + i, h[i]);
}

// pick[i] = {bin of the point of rank n / 2, its rank among the bin's points}.
// The bins are left zero for the next level.
__global__ void __launch_bounds__(SPLIT_THREADS) split_pick_kernel(SplitLevel lv, SplitLevel nx, int cap,
                                                                   int* __restrict__ hist, int2* __restrict__ pick) {
    chain_begin();
    __shared__ uint32_t wsum[SPLIT_THREADS / 32], tot;
    const int q = blockIdx.x;
    if (q == 0 && threadIdx.x == 0) *nx.n = 0;  // select fills it
    if (q >= split_segs(lv, cap)) return;
    const int4 sg = lv.seg[q];
    constexpr int PER = SPLIT_BINS / SPLIT_THREADS;
    int4* g = reinterpret_cast<int4*>(hist + (long long)q * SPLIT_BINS) + threadIdx.x * (PER / 4);
    int c[PER], sum = 0;
#pragma unroll
    for (int i = 0; i < PER / 4; ++i) {
        const int4 v = g[i];
        c[4 * i] = v.x, c[4 * i + 1] = v.y, c[4 * i + 2] = v.z, c[4 * i + 3] = v.w;
        sum += v.x + v.y + v.z + v.w;
        g[i] = make_int4(0, 0, 0, 0);
    }
    uint32_t total;
    int r = (sg.y - sg.x) / 2 - (int)block_scan_u32<SPLIT_THREADS>((uint32_t)sum, wsum, &tot, &total);
    if (r >= 0 && r < sum) {  // exactly one thread
        int d = threadIdx.x * PER;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
            if (r < c[i]) {
                d += i;
                break;
            }
            r -= c[i];
        }
        pick[q] = make_int2(d, r);
    }
}

__global__ void __launch_bounds__(SPLIT_THREADS) split_classify_kernel(const float4* pts, SplitLevel lv,
                                                                       int max_tiles,
                                                                       const int2* pick,
                                                                       int* __restrict__ tile_left,
                                                                       uint2* __restrict__ cand) {
    chain_begin();
    __shared__ int less;
    const int4 sg = lv.tile[blockIdx.x];
    if ((int)blockIdx.x >= min(split_unpack(*lv.n).tiles, max_tiles)) return;
    const int q = sg.z, tile = sg.w, t0 = sg.x + tile * SPLIT_TILE;
    const SplitAxis ax = split_axis(lv.box + 6 * q);
    const int bin = pick[q].x;
    if (threadIdx.x == 0) less = 0;
    __syncthreads();
    const float* c = reinterpret_cast<const float*>(pts) + ax.axis;
    const int lane = threadIdx.x & 31;
    int mine = 0, picked = 0;
    float x[SPLIT_ROUNDS];
    unsigned eq[SPLIT_ROUNDS];
#pragma unroll
    for (int r = 0; r < SPLIT_ROUNDS; ++r) {
        const int i = t0 + r * SPLIT_THREADS + threadIdx.x;
        x[r] = i < sg.y ? c[4ll * i] : 0.f;
        const int b = i < sg.y ? ax.bin(x[r]) : SPLIT_BINS;
        mine += b < bin ? 1 : 0;
        eq[r] = __ballot_sync(0xffffffffu, b == bin);
        picked += __popc(eq[r]);
    }
    if (picked) {  // one addition per warp: the bin can hold all of the tile
        int at = 0;
        if (lane == 0) at = atomicAdd(lv.cand_n + q, picked);
        at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
        for (int r = 0; r < SPLIT_ROUNDS; ++r) {
            const int i = t0 + r * SPLIT_THREADS + threadIdx.x;
            if (eq[r] >> lane & 1)
                cand[sg.x + at + __popc(eq[r] & ((1u << lane) - 1u))] = make_uint2(float_key(x[r]), (uint32_t)(i - sg.x));
            at += __popc(eq[r]);
        }
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0 && mine) atomicAdd(&less, mine);
    __syncthreads();
    if (threadIdx.x == 0) tile_left[split_tile0(sg.x) + tile] = less;
}

// A bin with more points than select keeps in shared memory: a stray point far away, heavy
// tails, towns far apart or many equal coordinates put nearly all of a segment into one.
// The list is then read by a cluster of blocks, with every thread's next eight items in
// flight, in digits of 11 bits (three of the key, at most three of the position), and
// the tiles' counts take one addition per warp and tile.  A build of 2M points, one block
// and digits of 8 bits / this: one point at 1e9 m 6861 / 1437 us, four towns 5346 / 1324,
// Cauchy 8012 / 1510, all equal 10526 / 1544 (evenly spread: 874 / 870).
struct SplitDigit {
    int digit, rank, count;
};
constexpr int SELECT_BITS = 11;
constexpr int SELECT_BINS = 1 << SELECT_BITS;
constexpr int SELECT_CLUSTER = 8;      // blocks, at most, for a segment
constexpr long long SELECT_SHARE = 32768;  // points per block (every block reads all the others' bins)

// f(item) for this block's share of the list.
template <int THREADS, class F>
__device__ __forceinline__ void select_each(const uint2* list, int c, int blocks, int block, F f) {
    const int step = blocks * THREADS;
    for (int base = block * THREADS + threadIdx.x; base - (int)threadIdx.x < c; base += 8 * step) {
        uint2 e[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
            e[u] = base + u * step < c ? list[base + u * step] : make_uint2(0u, 0xffffffffu);  // (no such position)
#pragma unroll
        for (int u = 0; u < 8; ++u) f(e[u]);
    }
}

// The key and position of rank `rank` among the c items of a list, and the left counts of
// the tiles (tl) for those before it: by all blocks of the cluster.  mem: 2 * SELECT_BINS
// ints of shared memory.
template <int THREADS>
__device__ void select_large(const uint2* list, int c, int cnt, int rank, int* tl, int* mem, uint32_t* wsum,
                             uint32_t* tot, SplitDigit* sd, uint32_t& v, uint32_t& p) {
    const cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int blocks = (int)cl.num_blocks(), block = (int)cl.block_rank();
    constexpr int PER = SELECT_BINS / THREADS;
    int pass = 0;
    // One digit: digit(item), -1 for an item that no longer matches.  The histograms of
    // two passes take turns, so one cluster barrier a pass will do.
    auto step = [&](auto digit) {
        int* h = mem + (pass++ & 1) * SELECT_BINS;
        for (int i = threadIdx.x; i < SELECT_BINS; i += THREADS) h[i] = 0;
        __syncthreads();
        select_each<THREADS>(list, c, blocks, block, [&](const uint2& e) {
            const int d = e.y == 0xffffffffu ? -1 : digit(e);
            if (d >= 0) atomicAdd(&h[d], 1);
        });
        cl.sync();
        int n[PER], sum = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) n[j] = 0;
        for (int k = 0; k < blocks; ++k) {
            const int* o = cl.map_shared_rank(h, k) + threadIdx.x * PER;
#pragma unroll
            for (int j = 0; j < PER; ++j) n[j] += o[j];
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) sum += n[j];
        uint32_t total;
        int r = rank - (int)block_scan_u32<THREADS>((uint32_t)sum, wsum, tot, &total);
        if (r >= 0 && r < sum) {  // exactly one thread
            int d = 0;
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                if (r < n[j]) {
                    d = j;
                    break;
                }
                r -= n[j];
            }
            *sd = SplitDigit{(int)threadIdx.x * PER + d, r, n[d]};
        }
        __syncthreads();
        const SplitDigit g = *sd;
        __syncthreads();
        rank = g.rank;
        return g;
    };
    v = p = 0;
    for (int b = 32; b > 0;) {
        const int w = min(b, SELECT_BITS);
        const SplitDigit g = step([&](const uint2& e) {
            return (b < 32 ? e.x >> b : 0u) == v ? (int)((e.x >> (b - w)) & ((1u << w) - 1u)) : -1;
        });
        v = (v << w) | (uint32_t)g.digit;
        b -= w;
    }
    for (int b = 32 - __clz(cnt); b > 0;) {
        const int w = min(b, SELECT_BITS);
        const SplitDigit g = step([&](const uint2& e) {
            return e.x == v && (e.y >> b) == p ? (int)((e.y >> (b - w)) & ((1u << w) - 1u)) : -1;
        });
        p = (p << w) | (uint32_t)g.digit;
        b -= w;
    }
    const int lane = threadIdx.x & 31;
    select_each<THREADS>(list, c, blocks, block, [&](const uint2& e) {
        const bool left = e.y != 0xffffffffu && (e.x < v || (e.x == v && e.y < p));
        const int tile = left ? (int)(e.y / SPLIT_TILE) : -1;
        const unsigned same = __match_any_sync(0xffffffffu, tile);
        if (left && lane == __ffs(same) - 1) atomicAdd(tl + tile, __popc(same));
    });
    __threadfence();
    cl.sync();  // the first block goes on with the counts; nobody's shared memory is read any more
}

// One 8-bit (or narrower) step of a radix selection: digit(i) of the items that
// still match (-1: not), rank -> the digit that holds the rank, the rank inside
// it and the items of that digit.
template <int THREADS, class F>
__device__ __forceinline__ SplitDigit split_digit(int n, int rank, int* hist, SplitDigit* out, F digit) {
    for (int i = threadIdx.x; i < 256; i += THREADS) hist[i] = 0;
    __syncthreads();
    for (int base = threadIdx.x; base < n; base += 4 * THREADS) {
        int d[4];  // four items in flight
#pragma unroll
        for (int u = 0; u < 4; ++u) d[u] = base + u * THREADS < n ? digit(base + u * THREADS) : -1;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (d[u] >= 0) atomicAdd(&hist[d[u]], 1);
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int c[8], sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = hist[lane * 8 + j], sum += c[j];
        int inc = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        int r = rank - (inc - sum);
        if (r >= 0 && r < sum) {  // exactly one lane
            int d = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (r < c[j]) {
                    d = j;
                    break;
                }
                r -= c[j];
            }
            *out = SplitDigit{lane * 8 + d, r, c[d]};
        }
    }
    __syncthreads();
    const SplitDigit o = *out;
    __syncthreads();
    return o;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) split_select_kernel(DevTree t, SplitLevel lv, SplitLevel nx, int cap,
                                                                     const int2* pick,
                                                                     int* __restrict__ tile_left,
                                                                     const uint2* cand,
                                                                     uint2* __restrict__ thr, int2* __restrict__ kids,
                                                                     int4* __restrict__ small, int* nsmall, int max_small,
                                                                     int fill) {
    chain_begin();
    __shared__ uint2 cache[SPLIT_CACHE];
    __shared__ int hist[256];
    __shared__ SplitDigit sd;
    __shared__ uint32_t wsum[THREADS / 32], tot, spos;
    const int blocks = (int)cooperative_groups::this_cluster().num_blocks(), q = blockIdx.x / blocks;
    if (q >= split_segs(lv, cap)) return;
    const bool lead = blockIdx.x % blocks == 0;
    const int c = lv.cand_n[q];
    if (!lead && c <= SPLIT_CACHE) return;
    const int4 sg = lv.seg[q];
    const int s = sg.x, cnt = sg.y - sg.x, m = cnt / 2, link = sg.z;
    const SplitAxis ax = split_axis(lv.box + 6 * q);
    const uint2* list = cand + s;
    int* tl = tile_left + split_tile0(s);  // the tiles' left counts: so far the lower bins'
    uint32_t v = 0, p = 0;
    if (c > SPLIT_CACHE) {
        select_large<THREADS>(list, c, cnt, pick[q].y, tl, reinterpret_cast<int*>(cache), wsum, &tot, &sd, v, p);
        if (!lead) return;
    } else {
        for (int i = threadIdx.x; i < c; i += THREADS) cache[i] = list[i];
        __syncthreads();
        // The key of rank n / 2, eight bits at a time.
        int rank = pick[q].y, same = c;
        for (int b = 32; b > 0; b -= 8) {
            const SplitDigit r = split_digit<THREADS>(c, rank, hist, &sd, [&](int i) {
                const uint32_t k = cache[i].x;
                return (b < 32 ? k >> b : 0u) == v ? (int)((k >> (b - 8)) & 255u) : -1;
            });
            v = (v << 8) | (uint32_t)r.digit;
            rank = r.rank;
            same = r.count;
        }
        // Among equal keys the position of that rank.
        if (same > 1) {
            for (int b = 32 - __clz(cnt); b > 0;) {
                const int w = min(b, 8);
                const SplitDigit r = split_digit<THREADS>(c, rank, hist, &sd, [&](int i) {
                    const uint2 e = cache[i];
                    return e.x == v && (e.y >> b) == p ? (int)((e.y >> (b - w)) & ((1u << w) - 1u)) : -1;
                });
                p = (p << w) | (uint32_t)r.digit;
                rank = r.rank;
                b -= w;
            }
        } else {
            for (int i = threadIdx.x; i < c; i += THREADS)
                if (cache[i].x == v) spos = cache[i].y;
            __syncthreads();
            p = spos;
        }
        // the candidates before (v, p)
        for (int i = threadIdx.x; i < c; i += THREADS) {
            const uint2 e = cache[i];
            if (e.x < v || (e.x == v && e.y < p)) atomicAdd(tl + e.y / SPLIT_TILE, 1);
        }
        __syncthreads();
    }
    const int tiles = (cnt + SPLIT_TILE - 1) / SPLIT_TILE;
    uint32_t carry = 0;
    for (int base = 0; base < tiles; base += THREADS) {
        const int i = base + threadIdx.x;
        const uint32_t x = i < tiles ? (uint32_t)__ldcg(tl + i) : 0u;
        uint32_t total;
        const uint32_t ex = block_scan_u32<THREADS>(x, wsum, &tot, &total);
        if (i < tiles) tl[i] = (int)(carry + ex);
        carry += total;
    }
    // The node and its children: the splitter's next level or the small list.
    __shared__ SplitCount open[2];
    if (threadIdx.x == 0) {
        open[0].segs = open[1].segs = -1;
        if (carry != (uint32_t)m) atomicOr(&t.st->err, ERR_SEG);  // cannot happen: the selection found rank m
        thr[q] = make_uint2(v, p);
        const int X = alloc_node(t);
        int2 kid = make_int2(-2, -2);  // the pool is exhausted (flagged): the points are dropped
        if (X >= 0) {
            Box3 b;
            for (int a = 0; a < 3; ++a) {
                b.lo[a] = key_float(lv.box[6 * q + a]);
                b.hi[a] = key_float(lv.box[6 * q + 3 + a]);
            }
            const int parent = link >> 1, side = link & 1;
            t.nparent[X] = link;
            int h = 0;
            for (int k = cnt; k > fill; k -= k / 2) ++h;
            t.nheight[X] = h;
            t.node[4 * X + 3] =
                make_float4(__int_as_float(0), __int_as_float(0), key_float(v), __int_as_float(ax.axis));
            write_child_box(t.node, parent, side, b);
            write_child_code(t.node, parent, side, X);
            write_child_cnt(t.ncnt, parent, side, cnt, 0);
            const int2 wi = t.winfo[parent];
            wide_link(t, wi, side, X, b, cnt);
            t.winfo[X] = wide_below(wi, side, X);
            for (int k = 0; k < 2; ++k) {
                const int cs = k == 0 ? s : s + m, ce = k == 0 ? s + m : s + cnt;
                if (ce - cs > SPLIT_MIN) {
                    open[k] = split_take(nx, cap, cs, ce, X * 2 + k, t.st);
                } else {
                    const int r = atomicAdd(nsmall, 1);
                    if (r >= max_small)
                        atomicOr(&t.st->err, ERR_SEG);
                    else
                        small[r] = make_int4(cs, ce, X * 2 + k, 0);
                }
            }
            kid = make_int2(open[0].segs, open[1].segs);
        }
        kids[q] = kid;
    }
    __syncthreads();
    for (int k = 0; k < 2; ++k)
        if (open[k].segs >= 0) split_list<THREADS>(nx, open[k], k == 0 ? s : s + m, k == 0 ? s + m : s + cnt);
}

// Points before (v, p) go left, the others right, both in order: to `dst`, or to
// `exits` where the child leaves the splitter.  64 registers, so that four blocks share
// an SM (2M points, nine levels: 157 us with 74, 130).
__global__ void __launch_bounds__(SPLIT_THREADS, 4) split_scatter_kernel(const float4* src, SplitLevel lv,
                                                                      SplitLevel nx, int max_tiles,
                                                                      const int* tile_left,
                                                                      const uint2* thr,
                                                                      const int2* kids,
                                                                      float4* __restrict__ dst,
                                                                      float4* __restrict__ exits) {
    chain_begin();
    constexpr int WARPS = SPLIT_THREADS / 32, WARP_PTS = SPLIT_TILE / WARPS;
    __shared__ uint32_t sm[12];
    __shared__ int wleft[WARPS];
    const int4 sg = lv.tile[blockIdx.x];
    if ((int)blockIdx.x >= min(split_unpack(*lv.n).tiles, max_tiles)) return;
    const int q = sg.z, tile = sg.w, t0 = sg.x + tile * SPLIT_TILE;
    const int2 kd = kids[q];
    if (kd.x == -2) return;
    int run = tile_left[split_tile0(sg.x) + tile];  // left points before this warp's
    const int axis = split_axis(lv.box + 6 * q).axis;
    const uint2 th = thr[q];
    const int m = (sg.y - sg.x) / 2;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x < 2) split_box_reset(sm + 6 * threadIdx.x);
    // A warp's consecutive points, 32 a round.
    const int w0 = t0 + warp * WARP_PTS;
    float4 p[SPLIT_ROUNDS];
    unsigned lm[SPLIT_ROUNDS];
    int left = 0;
#pragma unroll
    for (int r = 0; r < SPLIT_ROUNDS; ++r) {
        const int i = w0 + 32 * r + lane;
        bool l = false;
        if (i < sg.y) {
            p[r] = src[i];
            const uint32_t k = float_key(coord4(p[r], axis));
            l = k < th.x || (k == th.x && (uint32_t)(i - sg.x) < th.y);
        }
        lm[r] = __ballot_sync(0xffffffffu, l);
        left += __popc(lm[r]);
    }
    if (lane == 0) wleft[warp] = left;
    __syncthreads();
    for (int w = 0; w < warp; ++w) run += wleft[w];
    float4* dl = kd.x >= 0 ? dst : exits;
    float4* dr = kd.y >= 0 ? dst : exits;
    uint32_t bl[6], br[6];
    split_box_reset(bl);
    split_box_reset(br);
#pragma unroll
    for (int r = 0; r < SPLIT_ROUNDS; ++r) {
        const int i = w0 + 32 * r + lane;
        if (i < sg.y) {
            const int before = run + __popc(lm[r] & ((1u << lane) - 1u));
            const bool l = lm[r] >> lane & 1;
            const int to = l ? sg.x + before : m + (i - before);
            if (to < sg.y) (l ? dl : dr)[to] = p[r];  // (always: select checked the left count)
            if (l && kd.x >= 0) split_grow(bl, p[r]);
            if (!l && kd.y >= 0) split_grow(br, p[r]);
        }
        run += __popc(lm[r]);
    }
    if (kd.x >= 0) split_flush(sm, bl);
    if (kd.y >= 0) split_flush(sm + 6, br);
    __syncthreads();
    if (threadIdx.x < 12) {
        const int a = threadIdx.x % 6, kid = threadIdx.x < 6 ? kd.x : kd.y;
        if (kid >= 0) {
            if (a < 3) atomicMin(nx.box + 6 * kid + a, sm[threadIdx.x]);
            else atomicMax(nx.box + 6 * kid + a, sm[threadIdx.x]);
        }
    }
}

void launch_local(unsigned grid, const DevTree& t, const float4* pts, const int4* jobs, const int* njobs, int max_jobs,
                  int fill, cudaStream_t s) {
    launch_chain(local_build_kernel<LB_SMALL, 256>, grid, 256, sizeof(LbShared<LB_SMALL, 256>), s, t, pts, jobs, njobs, max_jobs,
                                                                                       fill);
}

// The local builder's shared memory is above the 48 KB default: opt in once
// per device.  Returns the device's SM count: the block-per-job kernels run
// one resident wave at most, each block looping over jobs.
int lb_prepare() {
    static std::atomic<int> sms[64];
    int dev = 0;
    cudaGetDevice(&dev);
    dev &= 63;
    int n = sms[dev].load(std::memory_order_acquire);
    if (n > 0) return n;
    cudaFuncSetAttribute(local_build_kernel<LB_SMALL, 256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)sizeof(LbShared<LB_SMALL, 256>));
    cudaFuncSetAttribute(finish_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(FinShared));
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 1;
    sms[dev].store(n, std::memory_order_release);
    return n;
}

__global__ void reset_count_kernel(unsigned long long* c) { chain_begin(); *c = 0; }

inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Bounds on the lists of one call: segments of at most SPLIT_MIN points and jobs of
// the local builder (a whole job or a piece of at least 512 points: half of a
// segment above LB_SMALL points); segments of the large splitter.
long long max_segs_bound(long long n, int njobs) { return (long long)njobs + n / 512 + 2; }

size_t align_up(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

int build_levels(long long max_job, int fill) {
    int d = 0;
    while (max_job > fill) {
        max_job = max_job - max_job / 2;
        ++d;
    }
    return d + 1;
}

namespace {

struct ScratchCarver {
    char* base;
    size_t off = 0;
    template <class T>
    T* take(size_t count) {
        T* r = (T*)(base + off);
        off += align_up(sizeof(T) * count);
        return r;
    }
};

size_t carve(void* base, long long n, int njobs, BuildScratch* bs) {
    const long long ms = max_segs_bound(n, njobs);
    // the large splitter's lists, only for calls that can use it
    const long long sp = n > SPLIT_MIN ? split_segs_cap(n) : 0;
    ScratchCarver c{(char*)base};
    for (int i = 0; i < 3; ++i) bs->pts[i] = c.take<float4>(i == 0 || sp ? n : 0);
    bs->small = c.take<int4>(ms);
    bs->local_jobs = c.take<int4>(ms);
    bs->nseg = c.take<int>(2);
    for (int i = 0; i < 2; ++i) {
        bs->split[i].seg = c.take<int4>(sp);
        bs->split[i].box = c.take<uint32_t>(6 * sp);
        bs->split[i].cand_n = c.take<int>(sp);
        bs->split[i].tile = c.take<int4>(sp ? split_tiles_cap(n) : 0);
        bs->split[i].htile = c.take<int4>(sp ? split_htiles_cap(n) : 0);
        bs->split[i].n = c.take<unsigned long long>(1);
    }
    bs->hist = c.take<int>(SPLIT_BINS * sp);
    bs->pick = c.take<int2>(sp);
    bs->thr = c.take<uint2>(sp);
    bs->kids = c.take<int2>(sp);
    bs->tile_left = c.take<int>(sp ? n / 1024 + 2 : 0);
    bs->cand = c.take<uint2>(sp ? n : 0);
    return c.off;
}

}  // namespace

size_t build_scratch_bytes(long long n, int njobs) {
    BuildScratch bs;
    return carve(nullptr, n, njobs, &bs);
}

void carve_build_scratch(void* base, long long n, int njobs, BuildScratch* bs) { carve(base, n, njobs, bs); }

void build_subtrees(const DevTree& t, const float4* pts, long long n, const int* job_off, const int* job_link,
                    int njobs, long long max_job, int fill, const BuildScratch& bs, cudaStream_t s) {
    if (njobs <= 0) return;
    const long long sms = lb_prepare();
    const int T = 256;
    const long long nn = n > 0 ? n : 1;
    const long long ms = max_segs_bound(nn, njobs);
    // Block-per-job grids: local builders run four per SM, finishing blocks two.
    auto grid = [&](long long jobs, long long per_sm) { return (unsigned)std::min(jobs, per_sm * sms); };
    if (max_job <= LB_SMALL) {
        // Every job fits the local builder: one launch builds them all.
        launch_chain(init_segs_kernel, blocks_for(njobs, T), T, 0, s, job_off, job_link, njobs, bs.local_jobs, bs.nseg);
        launch_local(grid(njobs, 4), t, pts, bs.local_jobs, bs.nseg, njobs, fill, s);
        return;
    }
    // Counters: segments of at most SPLIT_MIN points, local jobs.
    int *nsmall = bs.nseg, *nlocal = bs.nseg + 1;
    cudaMemsetAsync(bs.nseg, 0, 2 * sizeof(int), s);
    const float4* small_pts = bs.pts[2];
    if (max_job <= SPLIT_MIN) {
        launch_chain(init_segs_kernel, blocks_for(njobs, T), T, 0, s, job_off, job_link, njobs, bs.small, nsmall);
        small_pts = pts;
    } else {
        // Large segments, one level per round, until all of them are small.
        const int cap = (int)split_segs_cap(nn);
        launch_chain(reset_count_kernel, 1, 1, 0, s, bs.split[0].n);
        cudaMemsetAsync(bs.hist, 0, sizeof(int) * SPLIT_BINS * (size_t)cap, s);
        launch_chain(split_open_kernel, grid(njobs, 8), SPLIT_THREADS, 0, s, pts, job_off, job_link, njobs, bs.split[0], cap,
                                                                   bs.pts[2], bs.small, nsmall, (int)ms, t.st);
        long long size = max_job;
        for (int lv = 0; size > SPLIT_MIN; ++lv) {
            const SplitGrid g = split_grid(nn, njobs, lv);
            const unsigned segs = (unsigned)g.segs, blocks = (unsigned)g.tiles, hblocks = (unsigned)g.htiles;
            const int mt = (int)g.tiles, mh = (int)g.htiles;
            const SplitLevel &cur = bs.split[lv & 1], &nx = bs.split[(lv + 1) & 1];
            const float4* src = lv == 0 ? pts : bs.pts[(lv + 1) & 1];
            float4* dst = bs.pts[lv & 1];
            if (lv == 0) launch_chain(split_box_kernel, blocks, SPLIT_THREADS, 0, s, src, cur, mt);
            launch_chain(split_hist_kernel, hblocks, HIST_THREADS, 0, s, src, cur, mh, bs.hist);
            launch_chain(split_pick_kernel, segs, SPLIT_THREADS, 0, s, cur, nx, cap, bs.hist, bs.pick);
            launch_chain(split_classify_kernel, blocks, SPLIT_THREADS, 0, s, src, cur, mt, bs.pick, bs.tile_left, bs.cand);
            // Few segments can have many candidates each.
            unsigned k = 1;
            while (k < SELECT_CLUSTER && size >= 2 * k * SELECT_SHARE && 2 * k * segs <= 256) k *= 2;
            if (segs <= 64)
                launch_chain_if(true, k, split_select_kernel<1024>, k * segs, 1024, 0, s, t, cur, nx, cap, bs.pick, bs.tile_left, bs.cand,
                                                                         bs.thr, bs.kids, bs.small, nsmall, (int)ms,
                                                                         fill);
            else
                launch_chain(split_select_kernel<256>, segs, 256, 0, s, t, cur, nx, cap, bs.pick, bs.tile_left, bs.cand,
                                                                       bs.thr, bs.kids, bs.small, nsmall, (int)ms,
                                                                       fill);
            launch_chain(split_scatter_kernel, blocks, SPLIT_THREADS, 0, s, src, cur, nx, mt, bs.tile_left, bs.thr, bs.kids,
                                                                  dst, bs.pts[2]);
            size -= size / 2;
        }
    }
    launch_chain(finish_split_kernel, grid(ms, 2), FIN_THREADS, sizeof(FinShared), s, t, small_pts, bs.small, nsmall, (int)ms,
                                                                            bs.pts[0], bs.local_jobs, nlocal, (int)ms,
                                                                            fill);
    launch_local(grid(ms, 4), t, bs.pts[0], bs.local_jobs, nlocal, (int)ms, fill, s);
}

}  // namespace ikdg
