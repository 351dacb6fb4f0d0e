// Device bodies of the searches, shared by the per-call kernels (query.cu)
// and the persistent multi-tree batch kernel (batch.cu).
//
// Semantics (the drop-in contract):
//   * kNN (Nearest_Search / Search, ikd-Tree/ikd_Tree.cpp:366-397, :868-1013):
//     the k valid points with the smallest squared distance, among those with
//     sq_dist <= max_dist^2, ascending.  Ties at equal distance are broken by
//     the smaller point id (the reference leaves them to traversal order).  A
//     subtree is skipped only when its AABB lower bound exceeds the current
//     k-th distance or max_dist^2, so the result is exact.
//   * Box_Search (:399-404, :1015-1044): every valid p with min <= p < max.
//   * Radius_Search (:406-411, :1046-1087): every valid p with
//     sq_dist(p, q) <= r*r in float.  Whole subtrees are taken when their
//     farthest corner is inside (an exact float bound), so no point at the
//     boundary is admitted or lost by rounding.
#pragma once

#include "kernels.cuh"

namespace ikdg {
namespace search {

constexpr float FINF = __builtin_huge_valf();

// Packed pairs of floats (two rounded operations per instruction; the results
// are those of the scalar forms).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// 32 consecutive bytes from a 32-byte-aligned address, one 256-bit load
// (read-only data: the compiler may schedule it freely).
struct Quad2 {
    f32x2 v[4];
};
__device__ __forceinline__ Quad2 ld_quad2(const void* p) {
    Quad2 q;
    asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
        : "=l"(q.v[0]), "=l"(q.v[1]), "=l"(q.v[2]), "=l"(q.v[3])
        : "l"(p));
    return q;
}

// box_dist of two children of a wide record at once: the gap of an axis is
// max(lo - q, q - hi, 0), whose square is axis_gap's bit for bit.  The sums are
// scalar: packed ones were contracted with the packed squares, and a bound that
// is not rounded like sq_dist prunes points that tie with the k-th.
__device__ __forceinline__ f32x2 gap2(f32x2 lo, f32x2 hi, f32x2 q) {
    float a0, a1, b0, b1;
    unpack2(sub2(lo, q), a0, a1);
    unpack2(sub2(q, hi), b0, b1);
    const f32x2 g = pack2(max3(a0, b0, 0.f), max3(a1, b1, 0.f));
    return mul2(g, g);
}
__device__ __forceinline__ void box_dist2(f32x2 lx, f32x2 ly, f32x2 lz, f32x2 hx, f32x2 hy, f32x2 hz, f32x2 qx,
                                          f32x2 qy, f32x2 qz, float& d0, float& d1) {
    float x0, x1, y0, y1, z0, z1;
    unpack2(gap2(lx, hx, qx), x0, x1);
    unpack2(gap2(ly, hy, qy), y0, y1);
    unpack2(gap2(lz, hz, qz), z0, z1);
    d0 = __fadd_rn(__fadd_rn(x0, y0), z0);
    d1 = __fadd_rn(__fadd_rn(x1, y1), z1);
}

// sq_dist(q, p) of a stored slot {x, y, z, id}, x and y packed.
__device__ __forceinline__ float slot_dist(f32x2 qxy, float qz, f32x2 xy, float z) {
    const f32x2 d = sub2(qxy, xy);
    float sx, sy;
    unpack2(mul2(d, d), sx, sy);
    const float dz = __fsub_rn(qz, z);
    return __fadd_rn(__fadd_rn(sx, sy), __fmul_rn(dz, dz));
}

// ---- kNN, k <= 64: a group of four lanes per query over the wide records --------------
//
// A group's step is a node step (one 256-byte wide record, two children a lane)
// or a leaf step (half a bucket, 16 slots, four a lane).  A node step goes on
// with the nearest child; every lane stacks the rest of its own children that
// can still hold a result, with their box distances, in a shared-memory column
// of its own.  A leaf step inserts the slots that can enter the list, smallest
// first, at most k of them.  The list is sorted by (distance, id) and lives in
// the group's registers, entry lane * R + r, as (distance, slot); ids are read
// where two distances tie and at the end.  A subtree is skipped when its box distance exceeds
// min(max_dist^2, current k-th distance).
//
// The groups of a warp step together: node steps for the groups that hold a
// record until half of them hold a leaf, then one leaf step for those (in a
// simulated schedule over 1M points the extremes, at once and when all do, cost
// 15 % and 6 % more).
//
// 1M-point map, k = 5, kernel time before (a thread per query over the binary
// records) / now: 1 query 23.6 / 13.2 us, 15k of a LiDAR scan 51 / 21 us, 100k
// 144 / 93 us (96 / 68 us
// a call when calls on three trees overlap); 20M points, 1M queries, k = 16:
// 1595 / 1026 us a call.
// Bound by instruction issue (the tree is served from L2 and the chain of a
// query is ~15 loads): a thread per query over the binary records issued less
// per node but took 27 dependent loads a query, 96 steps a warp (its 32 queries
// wait for one another) and one thread's time per slot.
constexpr int KNN_G = 4;           // lanes per query
constexpr int KNN_LEAF_STEP = 16;  // slots per leaf step
constexpr int KNN_CTA = 128;       // threads per CTA of every kernel that uses the stacks

// Entries of a lane's stack for a tree of this height: every wide record on a
// path (the top one and one for every three levels) leaves at most the lane's
// two children.
__host__ __device__ constexpr int knn_stack_entries(int height) { return 2 * (1 + (height + 2) / 3) + 1; }

struct KnnOut {
    int* id;
    float* d2;
    float* xyz;  // nullable
    int* cnt;    // nullable
};

struct KnnLane {
    int lane, sl, gs;  // lane of the warp, of the group; the group's first lane
    unsigned gmask;    // the group's lanes
    __device__ __forceinline__ KnnLane() {
        lane = threadIdx.x & 31;
        sl = lane & (KNN_G - 1);
        gs = lane & ~(KNN_G - 1);
        gmask = ((1u << KNN_G) - 1u) << gs;
    }
};

// Searches one query per group; every lane of the warp calls it together
// (groups without a query pass valid = false).  stk: this thread's stack
// column in shared memory, `entries` entries KNN_CTA apart.  half_lanes: lanes
// of half the warp's queries.  Leaves the sorted list in ld / ls (slot -1: no
// entry).
// EARLY: a bucket's slots are loaded beside its fill count, not after it, which shortens
// the chain of a query and costs registers and loads of empty slots (KNN_EARLY_QUERIES).
template <int R, bool EARLY = false>
__device__ __forceinline__ void knn_group(const DevTree& t, const KnnLane& g, bool valid, float qx, float qy, float qz,
                                          int k, float max_sq, int2* stk, int entries, int half_lanes, float (&ld)[R],
                                          int (&ls)[R]) {
    constexpr int G = KNN_G, S = KNN_LEAF_STEP / G;
    constexpr unsigned ALL = 0xffffffffu, DEAD = 0xffffffffu;
    constexpr int DONE = 0x7fffffff;
    static_assert(WIDE == 2 * G, "two children per lane");
#pragma unroll
    for (int r = 0; r < R; ++r) {
        ld[r] = FINF;
        ls[r] = -1;
    }
    const f32x2 qx2 = pack2(qx, qx), qy2 = pack2(qy, qy), qz2 = pack2(qz, qz), qxy = pack2(qx, qy);
    float lim = max_sq;  // min(max_sq, k-th distance)
    const int wl = g.gs + (k - 1) / R, wr = (k - 1) % R;  // where the k-th entry lives
    int sp = 0, half = 0;
    int cur = valid ? t.start : DONE;  // a record's node, a leaf's code or DONE
    int lev = 0;                 // level of the record `cur` (records above it on its path)
    bool full = false;           // a stack overflowed (cannot happen: see knn_stack_entries)
    int steps = 0;
    bool ties = false;           // the warp's last leaf step met equal distances

    while (true) {
        if (++steps > t.max_visits) {
            if (cur != DONE && g.sl == 0) atomicOr(&t.st->err, ERR_LOOP);
            break;
        }
        const unsigned leaves = __ballot_sync(ALL, cur < 0);
        const bool node = (unsigned)cur < (unsigned)DONE;
        bool pop;
        if (__popc(leaves) < half_lanes && __any_sync(ALL, node)) {
            const char* a = reinterpret_cast<const char*>(t.wide + (long long)(node ? cur : 0) * 16) + 64 * g.sl;
            const Quad2 u = ld_quad2(a), v = ld_quad2(a + 32);
            float d0, d1, lx0, lx1, hx0, hx1, c0, c1;
            box_dist2(u.v[0], u.v[1], u.v[2], u.v[3], v.v[0], v.v[1], qx2, qy2, qz2, d0, d1);
            unpack2(u.v[0], lx0, lx1);
            unpack2(u.v[3], hx0, hx1);
            unpack2(v.v[2], c0, c1);
            // Key: the distance with the child's index in its low three bits
            // (they only order the visits).  Empty slots have lo > hi.
            const bool al0 = node && d0 <= lim && lx0 <= hx0, al1 = node && d1 <= lim && lx1 <= hx1;
            const unsigned key0 = al0 ? (__float_as_uint(d0) & ~7u) | (unsigned)(2 * g.sl) : DEAD;
            const unsigned key1 = al1 ? (__float_as_uint(d1) & ~7u) | (unsigned)(2 * g.sl + 1) : DEAD;
            unsigned m = min(key0, key1);
            m = min(m, __shfl_xor_sync(ALL, m, 1));
            m = min(m, __shfl_xor_sync(ALL, m, 2));
            // Entry: the code, and the distance with the record's level in
            // its low five bits.
            const bool p0 = al0 && key0 != m, p1 = al1 && key1 != m;
            full = full || (p0 && p1 ? sp + 1 : p0 || p1 ? sp : 0) >= entries;
            if (p0 && sp < entries)
                stk[KNN_CTA * sp++] = make_int2(__float_as_int(c0), (__float_as_int(d0) & ~31) | lev);
            if (p1 && sp < entries)
                stk[KNN_CTA * sp++] = make_int2(__float_as_int(c1), (__float_as_int(d1) & ~31) | lev);
            const int code = __shfl_sync(ALL, __float_as_int((m & 1) ? c1 : c0), g.gs + (int)((m >> 1) & 3u));
            pop = node && m == DEAD;
            if (node) cur = code;
            ++lev;
        } else {
            if (leaves == 0) break;
            const bool act = cur < 0;
            const int L = act ? code_leaf(cur) : 0;
            const int j0 = half * KNN_LEAF_STEP + S * g.sl;
            const int s0 = L * LEAF_CAP + j0;
            Quad2 slots[S / 2];
            if (EARLY && act) {
#pragma unroll
                for (int i = 0; i < S / 2; ++i) slots[i] = ld_quad2(t.pts + (long long)s0 + 2 * i);
            }
            const int n = act ? min(__ldg(t.leaf_n + L), LEAF_CAP) : 0;
            unsigned key[S];
#pragma unroll
            for (int i = 0; i < S; ++i) key[i] = DEAD;
            if (act) {
#pragma unroll
                for (int i = 0; i < S; i += 2) {
                    const Quad2 p = EARLY ? slots[i / 2] : ld_quad2(t.pts + (long long)s0 + i);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        float z, w;
                        unpack2(p.v[2 * e + 1], z, w);
                        const float d = slot_dist(qxy, qz, p.v[2 * e], z);
                        const bool ok = j0 + i + e < n && !(__float_as_uint(w) & F_DEL) && d <= lim;
                        key[i + e] = ok ? __float_as_uint(d) : DEAD;
                    }
                }
            }
            // The candidates enter one a round and group, the nearest first; one with
            // the k-th distance may still enter by its id.
            unsigned m;
            float pd;
            int slot, ps;
            bool go;
            auto nearest = [&]() {  // false: no group has one left
                const unsigned mine = min(min(key[0], key[1]), min(key[2], key[3]));
                m = min(mine, __shfl_xor_sync(ALL, mine, 1));
                m = min(m, __shfl_xor_sync(ALL, m, 2));
                go = m <= __float_as_uint(lim);  // (DEAD is above every distance)
                return __any_sync(ALL, go);
            };
            auto take = [&]() {  // its slot; the entry before this lane's first
                const unsigned mine = min(min(key[0], key[1]), min(key[2], key[3]));
                const int ml = __ffs(__ballot_sync(ALL, mine == m) & g.gmask) - 1;
                const bool is0 = key[0] == m, is1 = key[1] == m, is2 = key[2] == m;
                slot = __shfl_sync(ALL, s0 + (is0 ? 0 : is1 ? 1 : is2 ? 2 : 3), ml);
                if (g.lane == ml) {
                    if (is0)
                        key[0] = DEAD;
                    else if (is1)
                        key[1] = DEAD;
                    else if (is2)
                        key[2] = DEAD;
                    else
                        key[3] = DEAD;
                }
                pd = __shfl_up_sync(ALL, ld[R - 1], 1, G);
                ps = __shfl_up_sync(ALL, ls[R - 1], 1, G);
                if (g.sl == 0) pd = -1.f;
            };
            auto kth = [&]() {
                float w = ld[0];
#pragma unroll
                for (int r = 1; r < R; ++r)
                    if (r == wr) w = ld[r];
                return __shfl_sync(ALL, w, wl);
            };
            // Candidates as far as the k-th entry whose ids keep them out.
            auto drop = [&]() {
                const float kd = kth();
                int ks = ls[0];
#pragma unroll
                for (int r = 1; r < R; ++r)
                    if (r == wr) ks = ls[r];
                ks = __shfl_sync(ALL, ks, wl);
                if (!(act && ks >= 0 && kd == lim)) return;
                const int kid = (int)(__float_as_uint(__ldg(&t.pts[ks].w)) & ID_MASK);
#pragma unroll
                for (int i = 0; i < S; ++i)
                    if (key[i] == __float_as_uint(kd) && (int)(__float_as_uint(__ldg(&t.pts[s0 + i].w)) & ID_MASK) > kid)
                        key[i] = DEAD;
            };
            // (not for short lists: the test of the step before costs them 5 % of every
            // search, and a first round is cheap)
            if (R >= 8 && ties) drop();
            ties = false;
            while (nearest()) {
                const float md = __uint_as_float(m);
                bool tie = false;
#pragma unroll
                for (int r = 0; r < R; ++r) tie = tie || ld[r] == md;
                ties = __any_sync(ALL, tie && go);
                if (ties) break;
                take();
                // Sorted shift: an entry above the candidate takes its predecessor,
                // or the candidate if that is below it.
#pragma unroll
                for (int r = R - 1; r >= 0; --r) {
                    const float bd = r > 0 ? ld[r > 0 ? r - 1 : 0] : pd;
                    const int bs = r > 0 ? ls[r > 0 ? r - 1 : 0] : ps;
                    if (go && ld[r] > md) {
                        ls[r] = bd > md ? bs : slot;
                        ld[r] = fmaxf(bd, md);
                    }
                }
                lim = fminf(max_sq, kth());
            }
            // The rest of a step with equal distances, the smaller id first, in a loop
            // of its own: the one above is the hot one.  Where many points coincide,
            // whole buckets tie with the k-th entry: those that its id keeps out leave
            // at once, not one a round.  (300,000 points on 1,728 places,
            // 20k queries, k = 1 / 5 / 16 / 32: 463 /
            // 725 / 1121 / 2407 us without, 242 / 328 / 642 / 1484 with; 300 queries, k = 5,
            // on 300,000 equal points 147 ms, 40.)
            while (ties && nearest()) {
                const float md = __uint_as_float(m);
                take();
                const int id = go ? (int)(__float_as_uint(__ldg(&t.pts[slot].w)) & ID_MASK) : 0;
                bool ahead[R];  // entry r stays before the candidate
#pragma unroll
                for (int r = 0; r < R; ++r)
                    ahead[r] = ld[r] < md || (ld[r] == md && ls[r] >= 0 && go &&
                                              (int)(__float_as_uint(__ldg(&t.pts[ls[r]].w)) & ID_MASK) < id);
                bool pa = __shfl_up_sync(ALL, ahead[R - 1], 1, G);
                if (g.sl == 0) pa = true;
#pragma unroll
                for (int r = R - 1; r >= 0; --r) {
                    const bool before = r > 0 ? ahead[r > 0 ? r - 1 : 0] : pa;
                    if (go && !ahead[r]) {
                        ld[r] = before ? md : (r > 0 ? ld[r > 0 ? r - 1 : 0] : pd);
                        ls[r] = before ? slot : (r > 0 ? ls[r > 0 ? r - 1 : 0] : ps);
                    }
                }
                lim = fminf(max_sq, kth());
                drop();
            }
            pop = act && !(half == 0 && n > KNN_LEAF_STEP);
            if (act) half = pop ? 0 : 1;
        }
        // Of the columns' tops that can still hold a result, the deepest, the
        // nearest of those: so the columns hold children of the records on
        // one path only, two per record and lane.
        if (__any_sync(ALL, pop)) {
            int2 e = make_int2(DONE, 0);
            bool dead = pop && sp > 0;
            while (__any_sync(ALL, dead)) {  // drop what the bound has passed
                if (dead) {
                    e = stk[KNN_CTA * (sp - 1)];
                    if (__int_as_float(e.y & ~31) <= lim)
                        dead = false;
                    else
                        dead = --sp > 0;
                }
            }
            const unsigned key =
                pop && sp > 0 ? ((31u - (e.y & 31)) << 27) | (((unsigned)e.y >> 5) & ~3u) | (unsigned)g.sl : DEAD;
            unsigned m = min(key, __shfl_xor_sync(ALL, key, 1));
            m = min(m, __shfl_xor_sync(ALL, m, 2));
            const int code = __shfl_sync(ALL, e.x, g.gs + (int)(m & 3u));
            if (pop) {
                cur = m == DEAD ? DONE : code;
                lev = 32 - (int)(m >> 27);
                if (key == m && m != DEAD) --sp;
            }
        }
    }
    if (full) atomicOr(&t.st->err, ERR_STACK);
}

// A group's rows: entry e of query `row` at row * k + e of every array.
template <int R>
__device__ __forceinline__ void knn_write_rows(const DevTree& t, const KnnLane& g, bool valid, const float (&ld)[R],
                                               const int (&ls)[R], int k, long long row, const KnnOut& o) {
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int e = g.sl * R + r;
        const bool ok = ls[r] >= 0;
        cnt += __popc(__ballot_sync(0xffffffffu, ok && e < k) & g.gmask);
        if (!valid || e >= k) continue;
        const float4 p = ok ? __ldg(t.pts + ls[r]) : make_float4(0.f, 0.f, 0.f, 0.f);
        const long long at = row * k + e;
        o.id[at] = ok ? (int)(__float_as_uint(p.w) & ID_MASK) : -1;
        o.d2[at] = ok ? ld[r] : FINF;
        if (o.xyz != nullptr) {
            o.xyz[at * 3 + 0] = p.x;
            o.xyz[at * 3 + 1] = p.y;
            o.xyz[at * 3 + 2] = p.z;
        }
    }
    if (valid && o.cnt != nullptr && g.sl == 0) o.cnt[row] = cnt;
}

// ---- kNN, a thread per query over the binary records ---------------------------------
//
// For k > 64 (K = 0): the sorted list lives in the query's output rows, with the slot
// index of each entry in `slots` (k ints per query).  For k = K <= 2 and very many
// sorted queries: in registers (32 neighbours' walks are nearly the same, so a thread
// each issues less than a group each; see KNN_THREAD_QUERIES).  Nearer child first,
// the farther one stacked with its box distance; leaves are scanned by the warp's
// threads together, each its own.
__device__ __forceinline__ bool cand_less(float d, int id, float d2, int id2) {
    return d < d2 || (d == d2 && id < id2);
}

template <int K>
__device__ __forceinline__ void knn_thread_body(const DevTree& t, bool valid, long long qi, float qx, float qy, float qz,
                                                int k, float max_sq, const KnnOut& o, int* __restrict__ slots) {
    constexpr int PAIRS = K > 0 ? 2 : 4;  // of slots in flight
    constexpr int KR = K > 0 ? K : 1;
    float bd[KR];
    int bi[KR], bs[KR];
#pragma unroll
    for (int m = 0; m < KR; ++m) bd[m] = FINF, bi[m] = 0x7fffffff, bs[m] = -1;
    // (the three parts of a list are arrays of their own: the shifts of an insertion are
    // bound by the order of their loads and stores; 20k queries, k = 100, on 1M points
    // 7.6 ms without the qualifiers, 6.3 with)
    float* __restrict__ gd = o.d2 + qi * k;
    int* __restrict__ gi = o.id + qi * k;
    int* __restrict__ gs = slots + qi * k;
    int cnt = 0;
    float worst = FINF;
    int worst_id = 0x7fffffff;
    int st_code[MAX_STACK];
    float st_d[MAX_STACK];
    int sp = 0;
    int cur = 0;  // node code (>= 0; 0 = the sentinel record) or leaf code (< 0)
    bool done = !valid;
    int visits = 0;
    auto pop = [&]() {
        const float lim = fminf(max_sq, worst);
        while (sp > 0) {
            --sp;
            if (st_d[sp] <= lim) {
                cur = st_code[sp];
                return;
            }
        }
        done = true;
    };
    while (true) {
        while (true) {
            const bool nodework = !done && cur >= 0;
            if (!__any_sync(0xffffffffu, nodework)) break;
            if (!nodework) continue;
            if (++visits > t.max_visits) {
                atomicOr(&t.st->err, ERR_LOOP);
                done = true;
                continue;
            }
            const NodeRec r = load_node(t.node, cur);
            const int cl = r.left(), cr = r.right();
            const float lim = fminf(max_sq, worst);
            float dl = FINF, dr = FINF;
            bool vl = false, vr = false;
            if (cl != 0 && r.f0.x <= r.f0.w) {
                dl = box_dist(qx, qy, qz, r.f0.x, r.f0.y, r.f0.z, r.f0.w, r.f1.x, r.f1.y);
                vl = dl <= lim;
            }
            if (cr != 0 && r.f1.z <= r.f2.y) {
                dr = box_dist(qx, qy, qz, r.f1.z, r.f1.w, r.f2.x, r.f2.y, r.f2.z, r.f2.w);
                vr = dr <= lim;
            }
            if (vl && vr) {
                const bool left_first = dl <= dr;
                if (sp < MAX_STACK) {
                    st_code[sp] = left_first ? cr : cl;
                    st_d[sp] = left_first ? dr : dl;
                    ++sp;
                } else {
                    atomicOr(&t.st->err, ERR_STACK);
                }
                cur = left_first ? cl : cr;
            } else if (vl) {
                cur = cl;
            } else if (vr) {
                cur = cr;
            } else {
                pop();
            }
        }
        const bool leafwork = !done && cur < 0;
        if (!__any_sync(0xffffffffu, leafwork)) break;
        if (!leafwork) continue;
        // Two passes: first the slots that can enter the list are marked, with PAIRS
        // pairs of slots in flight and no branch, so the lanes stay together; then only
        // those are offered.  (Offering in one pass runs the insertion for every slot
        // at which any lane has a candidate.)
        const int L = code_leaf(cur);
        const int n = min(__ldg(t.leaf_n + L), LEAF_CAP);
        const float4* lp = t.pts + (long long)L * LEAF_CAP;
        const f32x2 qxy = pack2(qx, qy);
        unsigned marks = 0;
        for (int j0 = 0; j0 < n; j0 += 2 * PAIRS) {
            Quad2 p[PAIRS];
#pragma unroll
            for (int u = 0; u < PAIRS; ++u) p[u] = ld_quad2(lp + j0 + 2 * u);  // (slots past the fill stay in the bucket)
#pragma unroll
            for (int u = 0; u < 2 * PAIRS; ++u) {
                float z, w;
                unpack2(p[u >> 1].v[2 * (u & 1) + 1], z, w);
                const float d = slot_dist(qxy, qz, p[u >> 1].v[2 * (u & 1)], z);
                const int id = (int)(__float_as_uint(w) & ID_MASK);
                const bool in = j0 + u < n && !(__float_as_uint(w) & F_DEL) && d <= max_sq &&
                                cand_less(d, id, worst, worst_id);
                marks |= (in ? 1u : 0u) << (j0 + u);
            }
        }
        while (marks) {
            const int j = __ffs(marks) - 1;
            marks &= marks - 1;
            const float4 p = __ldg(lp + j);
            const float d = sq_dist(qx, qy, qz, p.x, p.y, p.z);
            const int id = (int)(__float_as_uint(p.w) & ID_MASK);
            if (!cand_less(d, id, worst, worst_id)) continue;
            if constexpr (K > 0) {
                float cd = d;
                int ci = id, cs = L * LEAF_CAP + j;
#pragma unroll
                for (int m = 0; m < K; ++m) {
                    const bool sw = cand_less(cd, ci, bd[m], bi[m]);
                    const float td = bd[m];
                    const int ti = bi[m], ts = bs[m];
                    bd[m] = sw ? cd : td, bi[m] = sw ? ci : ti, bs[m] = sw ? cs : ts;
                    cd = sw ? td : cd, ci = sw ? ti : ci, cs = sw ? ts : cs;
                }
                worst = bd[KR - 1];
                worst_id = bi[KR - 1];
                continue;
            }
            int pos = cnt < k ? cnt : k - 1;
            while (pos > 0 && cand_less(d, id, gd[pos - 1], gi[pos - 1])) {
                gd[pos] = gd[pos - 1];
                gi[pos] = gi[pos - 1];
                gs[pos] = gs[pos - 1];
                --pos;
            }
            gd[pos] = d;
            gi[pos] = id;
            gs[pos] = L * LEAF_CAP + j;
            if (cnt < k) ++cnt;
            if (cnt == k) {
                worst = gd[k - 1];
                worst_id = gi[k - 1];
            }
        }
        pop();
    }
    if (!valid) return;
    if constexpr (K > 0) {
#pragma unroll
        for (int j = 0; j < K; ++j) {
            const bool ok = bs[j] >= 0;
            cnt += ok ? 1 : 0;
            gi[j] = ok ? bi[j] : -1;
            gd[j] = bd[j];
            if (o.xyz != nullptr) {
                const float4 p = ok ? __ldg(t.pts + bs[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
                o.xyz[(qi * K + j) * 3 + 0] = p.x;
                o.xyz[(qi * K + j) * 3 + 1] = p.y;
                o.xyz[(qi * K + j) * 3 + 2] = p.z;
            }
        }
        if (o.cnt != nullptr) o.cnt[qi] = cnt;
        return;
    }
    for (int j = 0; j < k; ++j) {
        const bool ok = j < cnt;
        if (!ok) {
            gi[j] = -1;
            gd[j] = FINF;
        }
        if (o.xyz != nullptr) {
            const float4 p = ok ? __ldg(t.pts + gs[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
            o.xyz[(qi * k + j) * 3 + 0] = p.x;
            o.xyz[(qi * k + j) * 3 + 1] = p.y;
            o.xyz[(qi * k + j) * 3 + 2] = p.z;
        }
    }
    if (o.cnt != nullptr) o.cnt[qi] = cnt;
}

// ---- box / radius search: a warp for up to 32 queries -------------------------------
//
// The warp keeps one ordered stack of (subtree or leaf, query) items for all its
// queries: query 0's root on top, below it query 1's and so on, and every
// item's children take its place left to right.  Each step looks at the top
// RANGE_WINDOW items.  If they start with enough leaves, those are scanned, four
// lanes per leaf and four slots a lane; otherwise every record among them is
// expanded in place, four lanes per record and two children a lane.  So every
// step has work for all lanes however uneven the queries are (radii that differ
// by ten find numbers of points that differ by a thousand; in a simulated
// schedule 6.7-7.4 of a step's 8 items are used), and the leaves of a query still
// come in tree order, which is the order of its hits.
// A thread per query (the form before) kept a warp for as long as its largest
// query: 1M-point map, 100k queries, before / now, count and write kernels: box
// 197 + 227 us / 72 + 48 us, radius 650 + 861 us / 178 + 172 us.  Bound by
// instruction issue.
constexpr int RANGE_QUERIES = 32;  // queries per warp, at most
constexpr int RANGE_WINDOW = 8;    // items per step
constexpr int RANGE_FEW = 4;       // leading leaves that are worth a step of their own
constexpr int RANGE_WIDE = 96;     // stack height above which one record is expanded at a time
constexpr int RANGE_STAGE = 2 * KNN_LEAF_STEP * RANGE_WINDOW;  // hits staged at once
constexpr int RANGE_CTA = 128;

// Stack entries of a warp for a tree of this height: RANGE_WIDE, one step's
// growth, then seven per record on a path (expanded one at a time).
__host__ __device__ constexpr int range_stack_entries(int height) {
    return RANGE_WIDE + 7 * RANGE_WINDOW + 7 * (1 + (height + 2) / 3) + 1;
}

// A warp's shared memory (16-byte aligned parts).
struct RangeWarp {
    float4* q;      // [2 * RANGE_QUERIES] box {lo, hi x}, {hi y, hi z}; radius {centre, r^2}
    float* stage;   // [4 * RANGE_STAGE] hits about to be written
    int* cnt;       // [RANGE_QUERIES] hits (counting)
    int2* stack;
};
__host__ __device__ constexpr size_t range_warp_bytes(int entries, bool write) {
    return 2 * RANGE_QUERIES * sizeof(float4) +
           (write ? RANGE_STAGE * sizeof(float4) : RANGE_QUERIES * sizeof(int)) +
           ((size_t)entries * sizeof(int2) + 15) / 16 * 16;
}
template <bool WRITE>
__device__ __forceinline__ RangeWarp range_warp_carve(unsigned char* base, int entries) {
    unsigned char* p = base + (threadIdx.x >> 5) * range_warp_bytes(entries, WRITE);
    RangeWarp w{};
    w.q = reinterpret_cast<float4*>(p);
    p += 2 * RANGE_QUERIES * sizeof(float4);
    if (WRITE) {
        w.stage = reinterpret_cast<float*>(p);
        p += RANGE_STAGE * sizeof(float4);
    } else {
        w.cnt = reinterpret_cast<int*>(p);
        p += RANGE_QUERIES * sizeof(int);
    }
    w.stack = reinterpret_cast<int2*>(p);
    return w;
}

// Puts this lane's query (lane = its place among the warp's) into shared memory.
template <int MODE>
__device__ __forceinline__ void range_put_query(const RangeWarp& w, int lane, const float* q, float radius) {
    if (MODE == 0) {
        w.q[2 * lane] = make_float4(q[0], q[1], q[2], q[3]);
        w.q[2 * lane + 1] = make_float4(q[4], q[5], 0.f, 0.f);
    } else {
        w.q[2 * lane] = make_float4(q[0], q[1], q[2], __fmul_rn(radius, radius));
    }
}

// Stages a lane's hits (bits of m, slots in u and v) at places `at`, ..: points as
// words 3 at .., ids after all points.
__device__ __forceinline__ void range_stage(const RangeWarp& w, unsigned m, int at, const Quad2& u, const Quad2& v) {
    float* pt = w.stage;
    float* id = w.stage + 3 * RANGE_STAGE;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (m >> i & 1) {
            const Quad2& s = i < 2 ? u : v;
            float x, y, z, wd;
            unpack2(s.v[2 * (i & 1)], x, y);
            unpack2(s.v[2 * (i & 1) + 1], z, wd);
            pt[3 * at] = x;
            pt[3 * at + 1] = y;
            pt[3 * at + 2] = z;
            id[at] = wd;
            ++at;
        }
    }
}

// The staged hits from place s0 on leave as runs of consecutive words, one per
// query.  Groups (four lanes) with act hold one item each of query qi, their
// first hit at place `first`; `hits` ends the last.  Lane q holds query q's pos
// and lim.
__device__ __forceinline__ void range_emit(const DevTree& t, const RangeWarp& w, int s0, bool act, int qi, int first,
                                           int hits, long long& pos, long long lim, int* __restrict__ ids,
                                           float* __restrict__ xyz) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int prev = __shfl_up_sync(ALL, qi, 4);
    unsigned runs = __ballot_sync(ALL, act && (lane & 3) == 0 && (lane == 0 || prev != qi));
    while (runs) {
        const int l = __ffs(runs) - 1;
        runs &= runs - 1;
        const int s = __shfl_sync(ALL, first, l);
        const int c = (runs ? __shfl_sync(ALL, first, __ffs(runs) - 1) : hits) - s;
        if (c == 0) continue;
        const int q = __shfl_sync(ALL, qi, l);
        const long long o = __shfl_sync(ALL, pos, q);
        if (__any_sync(ALL, lane == q && pos + c > lim)) {
            if (lane == 0) atomicOr(&t.st->err, ERR_OUTPUT);
            continue;
        }
        if (lane == q) pos += c;
        const float* pt = w.stage + 3 * (s0 + s);
        const float* id = w.stage + 3 * RANGE_STAGE + s0 + s;
        int* io = ids + o;
        for (int e = lane; e < c; e += 32) io[e] = (int)(__float_as_uint(id[e]) & ID_MASK);
        if (xyz != nullptr) {
            float* xo = xyz + 3 * o;
            for (int e = lane; e < 3 * c; e += 32) xo[e] = pt[e];
        }
    }
}

// The hits a counting warp finds, so that the write pass need not search again:
// one entry {leaf * 2 + half, slot mask | query << 16} per bucket half with
// hits, in the order they are to be written, in chunks of LOG_CHUNK entries.  A
// chunk's entry 0 is {entries used, next chunk or -1}.  Warp i starts in chunk
// i; further chunks come from a counter.  A warp that finds none left, or that
// meets a covered subtree of more than LOG_COVERED points (counted as a whole),
// stores -1 used entries in its first chunk and is searched again.
constexpr int LOG_CHUNK = 128;
constexpr int LOG_COVERED = 1024;

struct RangeLog {
    int2* pool;              // nullptr: no log
    unsigned* next;          // chunks taken beyond the warps' first ones
    long long warps, chunks; // first chunks, all chunks
};

struct LogCursor {
    int2* first;
    int2* chunk;
    int used;
    bool on;
    __device__ __forceinline__ LogCursor(const RangeLog& log, long long warp) {
        on = log.pool != nullptr;
        first = chunk = on ? log.pool + warp * LOG_CHUNK : nullptr;
        used = 1;
    }
    // Room for n more entries in this chunk, or in a new one (whole warp).
    __device__ __forceinline__ void reserve(const RangeLog& log, int n) {
        if (used + n <= LOG_CHUNK) return;
        long long c = 0;
        if ((threadIdx.x & 31) == 0) {
            c = log.warps + (long long)atomicAdd(log.next, 1u);
            if (c < log.chunks) chunk[0] = make_int2(used - 1, (int)c);
        }
        c = __shfl_sync(0xffffffffu, c, 0);
        if (c >= log.chunks) {
            on = false;
            return;
        }
        chunk = log.pool + c * LOG_CHUNK;
        used = 1;
    }
    __device__ __forceinline__ void close() {
        if (first == nullptr || (threadIdx.x & 31) != 0) return;
        if (on)
            chunk[0] = make_int2(used - 1, -1);
        else
            first[0] = make_int2(-1, -1);
    }
};

// MODE 0: box, 1: radius.  Searches the queries whose bits are set in `todo`
// (their data in w.q) with the whole warp.  WRITE: the hits of query `lane` go
// to ids / xyz (nullable) from `pos` on, never past `lim` (hits there raise
// ERR_OUTPUT); otherwise they are counted in w.cnt, and logged.
template <int MODE, bool WRITE>
__device__ __forceinline__ void range_warp(const DevTree& t, const RangeWarp& w, unsigned todo, int entries,
                                           const RangeLog& log, LogCursor& lc, long long pos, long long lim,
                                           int* __restrict__ ids, float* __restrict__ xyz) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, j = lane >> 2, sub = lane & 3;
    const unsigned below = (1u << lane) - 1u;
    int sp = __popc(todo);
    // item: {node (>= 0: its record) or leaf code, query}; the first query on top
    if ((todo >> lane) & 1) w.stack[sp - 1 - __popc(todo & below)] = make_int2(t.start, lane);
    __syncwarp();
    int steps = 0;
    while (sp > 0) {
        if (++steps > t.max_visits) {
            if (lane == 0) atomicOr(&t.st->err, ERR_LOOP);
            break;
        }
        const int avail = min(sp, RANGE_WINDOW);
        // this lane's item, and with it the window: item j in lanes 4 j ..
        const int2 it = j < avail ? w.stack[sp - 1 - j] : make_int2(0, 0);
        const unsigned leafm = __ballot_sync(ALL, it.x < 0);
        int lead = (__ffs(~leafm) - 1) >> 2;  // leading leaves
        if (leafm == ALL) lead = RANGE_WINDOW;
        const float4 qa = w.q[2 * it.y];
        const float4 qb = MODE == 0 ? w.q[2 * it.y + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
        __syncwarp();  // items read before any is replaced
        if (lead == avail || lead >= RANGE_FEW) {
            const int L = code_leaf(it.x);
            const f32x2 qxy = pack2(qa.x, qa.y);
            // Hits among this lane's four slots of bucket half h, as a mask.
            Quad2 a, b;
            auto scan = [&](int h, int n) {
                unsigned m = 0;
                const float4* p = t.pts + (long long)L * LEAF_CAP + 16 * h + 4 * sub;
                a = ld_quad2(p);
                b = ld_quad2(p + 2);
                const int j0 = 16 * h + 4 * sub;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const f32x2 xy = i < 2 ? a.v[2 * (i & 1)] : b.v[2 * (i & 1)];
                    const f32x2 zw = i < 2 ? a.v[2 * (i & 1) + 1] : b.v[2 * (i & 1) + 1];
                    float z, id;
                    unpack2(zw, z, id);
                    bool in = j0 + i < n && !(__float_as_uint(id) & F_DEL);
                    if (MODE == 0) {
                        float x, y;
                        unpack2(xy, x, y);
                        in = in && x >= qa.x && x < qa.w && y >= qa.y && y < qb.x && z >= qa.z && z < qb.y;
                    } else {
                        in = in && slot_dist(qxy, qa.z, xy, z) <= qa.w;
                    }
                    m |= in ? 1u << i : 0u;
                }
                return m;
            };
            int n = 0;
            unsigned m0 = 0, m1 = 0;
            if (j < lead) {
                n = min(__ldg(t.leaf_n + L), LEAF_CAP);
                m0 = scan(0, n);
            }
            // Buckets with more than 16 slots: half the window, both halves.
            const bool over = __any_sync(ALL, n > KNN_LEAF_STEP);
            Quad2 a0 = a, b0 = b;
            if (over) {
                lead = min(lead, RANGE_WINDOW / 2);
                if (j >= lead) m0 = 0;
                if (j < lead && n > KNN_LEAF_STEP) m1 = scan(1, n);
            }
            if (!WRITE) {
                // the halves' slot masks, in every lane of the group
                unsigned v = (m0 | (m1 << 16)) << (4 * sub);
                v |= __shfl_xor_sync(ALL, v, 1);
                v |= __shfl_xor_sync(ALL, v, 2);
                const bool h0 = sub == 0 && (v & 0xffffu) != 0, h1 = sub == 0 && (v >> 16) != 0;
                if (h0 || h1) atomicAdd(&w.cnt[it.y], __popc(v));
                if (lc.on) {
                    const unsigned e0 = __ballot_sync(ALL, h0), e1 = over ? __ballot_sync(ALL, h1) : 0u;
                    lc.reserve(log, __popc(e0) + __popc(e1));
                    if (lc.on) {
                        int2* at = lc.chunk + lc.used + __popc(e0 & below) + __popc(e1 & below);
                        if (h0) *at++ = make_int2(L * 2, (int)(v & 0xffffu) | (it.y << 16));
                        if (h1) *at = make_int2(L * 2 + 1, (int)(v >> 16) | (it.y << 16));
                        lc.used += __popc(e0) + __popc(e1);
                    }
                }
            } else {
                // rank of this lane's hits: leaf by leaf, first halves before second
                const int c0 = __popc(m0), c1 = __popc(m1);
                int x = c0 | (c1 << 16);
                int y = __shfl_up_sync(ALL, x, 1, 4);
                if (sub >= 1) x += y;
                y = __shfl_up_sync(ALL, x, 2, 4);
                if (sub >= 2) x += y;
                const int tt = __shfl_sync(ALL, x, 3, 4);
                const int leaf_hits = (tt & 0xffff) + (tt >> 16);
                int z = leaf_hits;
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(ALL, z, o);
                    if (lane >= o) z += v;
                }
                const int first = z - leaf_hits, hits = __shfl_sync(ALL, z, 31);
                range_stage(w, m0, first + (x & 0xffff) - c0, a0, b0);
                if (over) range_stage(w, m1, first + (tt & 0xffff) + (x >> 16) - c1, a, b);
                __syncwarp();
                range_emit(t, w, 0, j < lead, it.y, first, hits, pos, lim, ids, xyz);
            }
            sp -= lead;
        } else {
            const bool here = j < avail;
            const bool rec = here && it.x >= 0 && (sp <= RANGE_WIDE || j == lead);
            bool al0 = here && !rec && sub == 0, al1 = false, whole = false;
            bool cov0 = false, cov1 = false;
            int k0 = it.x, k1 = 0;
            if (rec) {
                const char* p = reinterpret_cast<const char*>(t.wide + (long long)it.x * 16) + 64 * sub;
                const Quad2 u = ld_quad2(p), v = ld_quad2(p + 32);
                float lx0, lx1, ly0, ly1, lz0, lz1, hx0, hx1, hy0, hy1, hz0, hz1, f0, f1, v0, v1;
                unpack2(u.v[0], lx0, lx1);
                unpack2(u.v[1], ly0, ly1);
                unpack2(u.v[2], lz0, lz1);
                unpack2(u.v[3], hx0, hx1);
                unpack2(v.v[0], hy0, hy1);
                unpack2(v.v[1], hz0, hz1);
                unpack2(v.v[2], f0, f1);
                k0 = __float_as_int(f0);
                k1 = __float_as_int(f1);
                if (MODE == 0) {
                    // half-open, as qbox_disjoint
                    al0 = lx0 <= hx0 && qa.w > lx0 && qa.x <= hx0 && qb.x > ly0 && qa.y <= hy0 && qb.y > lz0 && qa.z <= hz0;
                    al1 = lx1 <= hx1 && qa.w > lx1 && qa.x <= hx1 && qb.x > ly1 && qa.y <= hy1 && qb.y > lz1 && qa.z <= hz1;
                } else {
                    float d0, d1;
                    box_dist2(u.v[0], u.v[1], u.v[2], u.v[3], v.v[0], v.v[1], pack2(qa.x, qa.x), pack2(qa.y, qa.y),
                              pack2(qa.z, qa.z), d0, d1);
                    al0 = lx0 <= hx0 && d0 <= qa.w;
                    al1 = lx1 <= hx1 && d1 <= qa.w;
                }
                unpack2(v.v[3], v0, v1);
                // Covered subtrees count as a whole, except small ones whose
                // leaves are to be logged.  (Leaves are scanned: the test costs
                // as much.)
                const int big = lc.on ? LOG_COVERED : 0;
                const bool try0 = !WRITE && al0 && k0 > 0 && __float_as_int(v0) > big;
                const bool try1 = !WRITE && al1 && k1 > 0 && __float_as_int(v1) > big;
                if (try0 || try1) {
                    if (MODE == 0) {
                        cov0 = qa.x <= lx0 && qa.w > hx0 && qa.y <= ly0 && qb.x > hy0 && qa.z <= lz0 && qb.y > hz0;
                        cov1 = qa.x <= lx1 && qa.w > hx1 && qa.y <= ly1 && qb.x > hy1 && qa.z <= lz1 && qb.y > hz1;
                    } else {
                        cov0 = box_far(qa.x, qa.y, qa.z, lx0, ly0, lz0, hx0, hy0, hz0) <= qa.w;
                        cov1 = box_far(qa.x, qa.y, qa.z, lx1, ly1, lz1, hx1, hy1, hz1) <= qa.w;
                    }
                    cov0 = cov0 && try0;
                    cov1 = cov1 && try1;
                    if (cov0 || cov1) {
                        whole = true;
                        atomicAdd(&w.cnt[it.y], (cov0 ? __float_as_int(v0) : 0) + (cov1 ? __float_as_int(v1) : 0));
                        al0 = al0 && !cov0;
                        al1 = al1 && !cov1;
                    }
                }
            }
            if (!WRITE && lc.on && __any_sync(ALL, whole)) lc.on = false;
            // The window's items are replaced in place, first on top.
            const unsigned b0 = __ballot_sync(ALL, al0), b1 = __ballot_sync(ALL, al1);
            const int end = sp - avail + __popc(b0) + __popc(b1);  // new height
            const int at = end - 1 - (__popc(b0 & below) + __popc(b1 & below));
            if (end > entries) {  // cannot happen: see range_stack_entries
                if (lane == 0) atomicOr(&t.st->err, ERR_STACK);
                break;
            }
            if (al0) w.stack[at] = make_int2(k0, it.y);
            if (al1) w.stack[at - (al0 ? 1 : 0)] = make_int2(k1, it.y);
            sp = end;
        }
        __syncwarp();
    }
}

// Writes the hits that a counting warp logged in the chunks from `c` on: 16
// entries a round, four lanes per entry, two entries a lane.
__device__ __forceinline__ void range_replay(const DevTree& t, const RangeWarp& w, const RangeLog& log, const int2* c,
                                             long long pos, long long lim, int* __restrict__ ids,
                                             float* __restrict__ xyz) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, j = lane >> 2, sub = lane & 3;
    while (true) {
        const int2 head = __ldg(c);
        for (int e0 = 0; e0 < head.x; e0 += 2 * RANGE_WINDOW) {
            int2 e[2];
            Quad2 a[2], b[2];
            unsigned m[2];
            bool act[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = e0 + RANGE_WINDOW * h + j;
                act[h] = i < head.x;
                e[h] = act[h] ? __ldg(c + 1 + i) : make_int2(0, 0);
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                m[h] = ((unsigned)e[h].y >> (4 * sub)) & 15u;
                if (!act[h]) m[h] = 0;
                if (m[h]) {
                    const float4* p = t.pts + (long long)(e[h].x >> 1) * LEAF_CAP + 16 * (e[h].x & 1) + 4 * sub;
                    a[h] = ld_quad2(p);
                    b[h] = ld_quad2(p + 2);
                }
            }
            // ranks of both halves of the round in one scan
            const int n0 = __popc(m[0]), n1 = __popc(m[1]);
            int x = n0 | (n1 << 16);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(ALL, x, o);
                if (lane >= o) x += v;
            }
            const int tot = __shfl_sync(ALL, x, 31);
            const int f0 = (x & 0xffff) - n0, f1 = (x >> 16) - n1, t0 = tot & 0xffff;
            range_stage(w, m[0], f0, a[0], b[0]);
            range_stage(w, m[1], t0 + f1, a[1], b[1]);
            __syncwarp();
            range_emit(t, w, 0, act[0], (e[0].y >> 16) & 31, f0, t0, pos, lim, ids, xyz);
            if (tot >> 16) range_emit(t, w, t0, act[1], (e[1].y >> 16) & 31, f1, tot >> 16, pos, lim, ids, xyz);
            __syncwarp();
        }
        if (head.y < 0) break;
        c = log.pool + (long long)head.y * LOG_CHUNK;
    }
}

}  // namespace search
}  // namespace ikdg
