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

// Leaves a warp scans per step of the range search's leaf phase.
#ifndef IKDG_RANGE_LEAF_BATCH
#define IKDG_RANGE_LEAF_BATCH 4
#endif
constexpr int RANGE_LEAF_BATCH = IKDG_RANGE_LEAF_BATCH;


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
// records) / now: 1 query 23.6 / 10 us, 15k 90 / 32 us, 100k 144 / 98 us (96 / 73 us
// a call when calls on three trees overlap); 20M points, 1M queries, k = 16:
// 1615 / 1067 us a call.
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
template <int R>
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

    while (true) {
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
            if (++steps > MAX_VISITS) {
                if (cur != DONE && g.sl == 0) atomicOr(&t.st->err, ERR_LOOP);
                break;
            }
            const bool act = cur < 0;
            const int L = act ? code_leaf(cur) : 0;
            const int j0 = half * KNN_LEAF_STEP + S * g.sl;
            const int s0 = L * LEAF_CAP + j0;
            const int n = act ? min(__ldg(t.leaf_n + L), LEAF_CAP) : 0;
            unsigned key[S];
#pragma unroll
            for (int i = 0; i < S; ++i) key[i] = DEAD;
            if (act) {
#pragma unroll
                for (int i = 0; i < S; i += 2) {
                    const Quad2 p = ld_quad2(t.pts + (long long)s0 + i);
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
            while (true) {
                // The smallest candidate of each group; one with the k-th
                // distance may still enter by its id.
                const unsigned mine = min(min(key[0], key[1]), min(key[2], key[3]));
                unsigned m = min(mine, __shfl_xor_sync(ALL, mine, 1));
                m = min(m, __shfl_xor_sync(ALL, m, 2));
                const bool go = m <= __float_as_uint(lim);  // (DEAD is above every distance)
                if (!__any_sync(ALL, go)) break;
                const int ml = __ffs(__ballot_sync(ALL, mine == m) & g.gmask) - 1;
                const bool is0 = key[0] == m, is1 = key[1] == m, is2 = key[2] == m;
                const int slot = __shfl_sync(ALL, s0 + (is0 ? 0 : is1 ? 1 : is2 ? 2 : 3), ml);
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
                const float md = __uint_as_float(m);
                float pd = __shfl_up_sync(ALL, ld[R - 1], 1, G);
                int ps = __shfl_up_sync(ALL, ls[R - 1], 1, G);
                if (g.sl == 0) pd = -1.f;
                bool tie = false;
#pragma unroll
                for (int r = 0; r < R; ++r) tie = tie || ld[r] == md;
                if (__any_sync(ALL, tie && go)) {
                    // Equal distances: the smaller id first.  (ahead: entry r
                    // stays before the candidate.)
                    const int id = go ? (int)(__float_as_uint(__ldg(t.pts + slot).w) & ID_MASK) : 0;
                    bool ahead[R];
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        ahead[r] = ld[r] < md || (ld[r] == md && ls[r] >= 0 && go &&
                                                  (int)(__float_as_uint(__ldg(t.pts + ls[r]).w) & ID_MASK) < id);
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
                } else {
                    // Sorted shift: an entry above the candidate takes its
                    // predecessor, or the candidate if that is below it.
#pragma unroll
                    for (int r = R - 1; r >= 0; --r) {
                        const float bd = r > 0 ? ld[r > 0 ? r - 1 : 0] : pd;
                        const int bs = r > 0 ? ls[r > 0 ? r - 1 : 0] : ps;
                        if (go && ld[r] > md) {
                            ls[r] = bd > md ? bs : slot;
                            ld[r] = fmaxf(bd, md);
                        }
                    }
                }
                float w = ld[0];
#pragma unroll
                for (int r = 1; r < R; ++r)
                    if (r == wr) w = ld[r];
                lim = fminf(max_sq, __shfl_sync(ALL, w, wl));
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

// ---- kNN, k > 64: a thread per query over the binary records -----------------------
//
// The sorted list lives in the query's output rows, with the slot index of each
// entry in `slots` (k ints per query).  Nearer child first, the farther one
// stacked with its box distance; leaves are scanned by the warp's threads
// together, each its own.
__device__ __forceinline__ bool cand_less(float d, int id, float d2, int id2) {
    return d < d2 || (d == d2 && id < id2);
}

__device__ __forceinline__ void knn_rows_body(const DevTree& t, bool valid, long long qi, float qx, float qy, float qz,
                                              int k, float max_sq, const KnnOut& o, int* __restrict__ slots) {
    float* gd = o.d2 + qi * k;
    int* gi = o.id + qi * k;
    int* gs = slots + qi * k;
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
            if (++visits > MAX_VISITS) {
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
        const int L = code_leaf(cur);
        const int n = min(__ldg(t.leaf_n + L), LEAF_CAP);
        for (int j = 0; j < n; ++j) {
            const float4 p = __ldg(t.pts + (long long)L * LEAF_CAP + j);
            const uint32_t w = __float_as_uint(p.w);
            if (w & F_DEL) continue;
            const float d = sq_dist(qx, qy, qz, p.x, p.y, p.z);
            const int id = (int)(w & ID_MASK);
            if (!(d <= max_sq && cand_less(d, id, worst, worst_id))) continue;
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

constexpr int RANGE_COUNT = 0, RANGE_WRITE = 1;

// MODE 0: box, MODE 1: radius.  OUT = RANGE_COUNT counts, RANGE_WRITE emits at
// the query's CSR offset.
// Box (MODE 0) / radius (MODE 1) search of query qi by this thread, with the
// leaves scanned by the whole warp.  Every lane of the warp calls this
// together; lanes without a query pass valid = false.  "While-while": in the
// node phase each thread walks its own query's nodes (a fully covered subtree
// adds its valid count from ncnt when counting, and is enumerated when
// writing) until it holds a leaf; in the leaf phase the warp takes the held
// leaves one at a time, one lane per slot (one 512-byte load per leaf), tests
// the slots against the holder's query and counts them with a ballot.  So a
// query with thousands of hits costs one warp step per leaf instead of one
// thread step per slot, while light queries keep one thread each.
// Returns this lane's hit count.  WRITE emits the hits at ids[o..],
// xyz[3 o..] in traversal order, never at or past o_lim (a hit there raises
// ERR_OUTPUT instead).  radius: one float per query, r_stride floats apart.
template <int MODE, int OUT>
__device__ __forceinline__ long long range_body(const DevTree& t, const float* __restrict__ q, int q_stride,
                                                const float* __restrict__ radius, int r_stride, long long qi,
                                                bool valid, long long o, long long o_lim, int* __restrict__ ids,
                                                float* __restrict__ xyz) {
    constexpr bool WRITE = OUT != RANGE_COUNT;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    // The query in six floats: box {lo, hi}, or radius {centre, r^2, -, -}.
    float qa[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (valid) {
        if (MODE == 0) {
            for (int a = 0; a < 6; ++a) qa[a] = q[qi * q_stride + a];
        } else {
            for (int a = 0; a < 3; ++a) qa[a] = q[qi * q_stride + a];
            const float r = radius[qi * r_stride];
            qa[3] = __fmul_rn(r, r);
        }
    }
    long long count = 0;
    int stack[MAX_STACK];
    int sp = 0;
    int cur = 0;  // item = code * 2 + covered; code 0 is the sentinel record
    bool done = !valid;
    int visits = 0;
    const float4* __restrict__ P = t.pts;
    auto pop = [&]() {
        if (sp > 0)
            cur = stack[--sp];
        else
            done = true;
    };

    while (true) {
        // Node phase.
        while (true) {
            const bool nodework = !done && (cur >> 1) >= 0;
            if (!__any_sync(0xffffffffu, nodework)) break;
            if (!nodework) continue;
            if (++visits > MAX_VISITS) {
                atomicOr(&t.st->err, ERR_LOOP);
                done = true;
                continue;
            }
            const int X = cur >> 1;
            const bool covered = cur & 1;
            const NodeRec r = load_node(t.node, X);
            const int4 c4 = WRITE ? make_int4(0, 0, 0, 0) : __ldg(t.ncnt + X);
            int next = 0;
            bool have_next = false;
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const int c = side == 0 ? r.left() : r.right();
                if (c == 0) continue;
                const Box3 b = r.box(side);
                if (box_empty(b)) continue;
                bool cov = covered;
                if (!cov) {
                    if (MODE == 0) {
                        Box3 qb;
                        for (int a = 0; a < 3; ++a) {
                            qb.lo[a] = qa[a];
                            qb.hi[a] = qa[3 + a];
                        }
                        if (qbox_disjoint(qb, b)) continue;
                        cov = qbox_covers(qb, b);
                    } else {
                        if (box_dist(qa[0], qa[1], qa[2], b.lo[0], b.lo[1], b.lo[2], b.hi[0], b.hi[1], b.hi[2]) >
                            qa[3])
                            continue;
                        cov = box_far(qa[0], qa[1], qa[2], b.lo[0], b.lo[1], b.lo[2], b.hi[0], b.hi[1], b.hi[2]) <=
                              qa[3];
                    }
                }
                if (cov && !WRITE) {
                    count += side == 0 ? (c4.x - c4.y) : (c4.z - c4.w);
                    continue;
                }
                const int it = c * 2 + (cov ? 1 : 0);
                if (!have_next) {
                    next = it;
                    have_next = true;
                } else if (sp < MAX_STACK) {
                    stack[sp++] = it;
                } else {
                    atomicOr(&t.st->err, ERR_STACK);
                }
            }
            if (have_next)
                cur = next;
            else
                pop();
        }
        // Leaf phase: the held leaves, RANGE_LEAF_BATCH at a time, one lane per
        // slot.  A bucket always has LEAF_CAP slots in the pool, so each slot
        // load is issued together with the leaf's fill count.
        const bool leafwork = !done && (cur >> 1) < 0;
        unsigned lb = __ballot_sync(0xffffffffu, leafwork);
        if (lb == 0) break;
        while (lb) {
            int src[RANGE_LEAF_BATCH];
#pragma unroll
            for (int u = 0; u < RANGE_LEAF_BATCH; ++u) {
                src[u] = lb ? __ffs(lb) - 1 : -1;
                lb &= lb - 1;
            }
            float4 p[RANGE_LEAF_BATCH];
            int nl[RANGE_LEAF_BATCH], it[RANGE_LEAF_BATCH];
#pragma unroll
            for (int u = 0; u < RANGE_LEAF_BATCH; ++u) {
                if (src[u] < 0) break;
                it[u] = __shfl_sync(0xffffffffu, cur, src[u]);
                const int L = code_leaf(it[u] >> 1);
                p[u] = __ldg(P + (long long)L * LEAF_CAP + lane);
                nl[u] = __ldg(t.leaf_n + L);
            }
#pragma unroll
            for (int u = 0; u < RANGE_LEAF_BATCH; ++u) {
                if (src[u] < 0) break;
                float h[6];
#pragma unroll
                for (int a = 0; a < 6; ++a) h[a] = __shfl_sync(0xffffffffu, qa[a], src[u]);
                bool hit = false;
                if (lane < nl[u] && !(__float_as_uint(p[u].w) & F_DEL)) {
                    if (it[u] & 1) {
                        hit = true;
                    } else if (MODE == 0) {
                        hit = p[u].x >= h[0] && p[u].x < h[3] && p[u].y >= h[1] && p[u].y < h[4] &&
                              p[u].z >= h[2] && p[u].z < h[5];
                    } else {
                        hit = sq_dist(p[u].x, p[u].y, p[u].z, h[0], h[1], h[2]) <= h[3];
                    }
                }
                const unsigned hb = __ballot_sync(0xffffffffu, hit);
                if (OUT == RANGE_WRITE) {
                    const long long base = __shfl_sync(0xffffffffu, o + count, src[u]);
                    const long long lim = __shfl_sync(0xffffffffu, o_lim, src[u]);
                    if (hit) {
                        const long long pos = base + __popc(hb & lt);
                        if (pos < lim) {
                            ids[pos] = (int)(__float_as_uint(p[u].w) & ID_MASK);
                            if (xyz != nullptr) {
                                xyz[pos * 3 + 0] = p[u].x;
                                xyz[pos * 3 + 1] = p[u].y;
                                xyz[pos * 3 + 2] = p[u].z;
                            }
                        } else {
                            atomicOr(&t.st->err, ERR_OUTPUT);
                        }
                    }
                }
                if (lane == src[u]) count += __popc(hb);
            }
        }
        if (leafwork) pop();
    }
    return count;
}

}  // namespace search
}  // namespace ikdg
