// Mutations of the device tree: point insertion, box / point deletion, box
// re-insertion, bottom-up refit with the rebalancing criteria, rebuild-job
// collection, and the exact voxel downsampling of Add_Points.
//
// Reference behaviour replaced here:
//   Add_by_point (ikd-Tree/ikd_Tree.cpp:817-866): descend by `p[axis] < split`
//     to a leaf bucket and append; a full bucket becomes a rebuild job.
//   Delete_by_range / Delete_Point_Boxes (:535-556, :647-710): every valid
//     point in the half-open box is flagged; the count of newly deleted points
//     is returned.  Whole covered subtrees are flagged without box tests.
//   Delete_by_point (:712-760): one valid point within EPSS = 1e-6 per axis is
//     flagged per input point (same_point, :1368-1371).
//   Add_by_range (:762-815): points deleted by box / point deletion (not by
//     downsampling) inside the box are restored.
//   Update / Criterion_Check / Rebuild (:1183-1323, :1089-1107, :624-645):
//     counts and AABBs are refit bottom-up along the touched paths only; a
//     node whose deleted share of slots exceeds alpha_del or whose left share
//     of valid points leaves [1 - alpha_bal, alpha_bal] is rebuilt, topmost
//     first.
#include <cuda_runtime.h>

#include <climits>
#include <utility>

#include "update.cuh"

namespace ikdg {
namespace {

inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

__device__ __forceinline__ float coord4(const float4& p, int a) { return a == 0 ? p.x : (a == 1 ? p.y : p.z); }

// Appends `v` to a work list, or flags ERR_LIST when the list is full.
__device__ __forceinline__ void list_push(DevStatus* st, int* counter, int* list, int cap, int v) {
    int i = atomicAdd(counter, 1);
    if (i < cap)
        list[i] = v;
    else
        atomicOr(&st->err, ERR_LIST);
}

__device__ __forceinline__ void mark_dirty(const UpdateAux& a, DevStatus* st, int L) {
    if (atomicExch(&a.dirty_flag[L], 1) == 0) list_push(st, &st->n_items, a.items, a.list_cap, leaf_code(L));
}

// mark_dirty by a whole warp (each lane its leaf, if it wants one): one reservation
// in the list.
__device__ __forceinline__ void mark_dirty_warp(const UpdateAux& a, DevStatus* st, int L, bool want) {
    const bool fresh = want && atomicExch(&a.dirty_flag[L], 1) == 0;
    const unsigned m = __ballot_sync(0xffffffffu, fresh);
    if (m == 0) return;
    const int lane = threadIdx.x & 31, lead = __ffs(m) - 1;
    int base = 0;
    if (lane == lead) base = atomicAdd(&st->n_items, __popc(m));
    const int at = __shfl_sync(0xffffffffu, base, lead) + __popc(m & ((1u << lane) - 1u));
    if (!fresh) return;
    if (at < a.list_cap)
        a.items[at] = leaf_code(L);
    else
        atomicOr(&st->err, ERR_LIST);
}

// ---- insertion -----------------------------------------------------------------

__global__ void route_append_kernel(DevTree t, UpdateAux a, const float4* pts, long long n,
                                    const int* n_dev, int4* __restrict__ ovf_leaf, float4* __restrict__ ovf_pts) {
    chain_begin();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    long long lim = n_dev != nullptr ? (long long)*n_dev : n;
    if (i >= lim) return;
    if (t.st->err & ERR_INPUT) return;  // a non-finite input: the call changes nothing
    float4 p = pts[i];
    int code = __float_as_int(t.node[3].x);  // sentinel's left child = root
    if (code == 0) {
        atomicOr(&t.st->err, ERR_ROUTE);
        return;
    }
    int steps = 0;
    while (code > 0) {
        if (++steps > MAX_WALK) {
            atomicOr(&t.st->err, ERR_LOOP);
            return;
        }
        float4 f3 = t.node[4 * code + 3];
        int axis = __float_as_int(f3.w);
        code = coord4(p, axis) < f3.z ? __float_as_int(f3.x) : __float_as_int(f3.y);
    }
    int L = code_leaf(code);
    int slot = atomicAdd(&t.leaf_n[L], 1);
    if (slot < LEAF_CAP) {
        t.pts[(long long)L * LEAF_CAP + slot] = p;
    } else {
        int o = atomicAdd(&t.st->n_ovf, 1);
        ovf_leaf[o] = make_int4(L, 0, 0, 0);
        ovf_pts[o] = p;
    }
    mark_dirty(a, t.st, L);
}

// ---- refit -------------------------------------------------------------------

// A refit item is a dirty leaf (its code, < 0) or a rebuilt subtree (its link,
// parent * 2 + side): either way one child side of one node, so a node sees at
// most one arrival per side.
__device__ __forceinline__ int item_link(const DevTree& t, int item) {
    return item < 0 ? __ldcg(t.lparent + code_leaf(item)) : item;
}

// Items are dealt out over the warps before the lanes, so a few thousand walks run
// one to a warp: walks of one warp diverge at each meeting and wait for one another
// (14,400-point scan into 500,000 points: 40 us with the items packed into full
// warps, 17 dealt out).
__device__ __forceinline__ int first_item() {
    const int warps = gridDim.x * (blockDim.x >> 5);
    return (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) + (int)(threadIdx.x & 31) * warps;
}

// Counts into pend[X] the child sides of X that a refit will change.
__global__ void refit_mark_kernel(DevTree t, UpdateAux a, const int* items, const int* n_items) {
    chain_begin();
    const int n = min(*n_items, a.list_cap);
    for (int i = first_item(); i < n; i += gridDim.x * blockDim.x) {
        const int link = item_link(t, items[i]);
        if (link < 0) continue;
        int X = link >> 1;
        for (int steps = 0; X > 0; ++steps) {
            if (steps > MAX_WALK) {
                atomicOr(&t.st->err, ERR_LOOP);
                return;
            }
            const int up = __ldcg(t.nparent + X);  // in flight with the atomic
            if (atomicAdd(&a.pend[X], 1) > 0) break;
            X = up >> 1;
        }
    }
}

__device__ __forceinline__ int child_height(const DevTree& t, int code) {
    return code > 0 ? __ldcg(&t.nheight[code]) : 0;
}

// A leaf that must be rebuilt (a full bucket that took more points) carries this in
// job_of_leaf from the moment it is listed until the jobs are chosen.
constexpr int LEAF_VIOL = -2;

__device__ __forceinline__ void list_leaf_violator(const DevTree& t, const UpdateAux& a, int L) {
    a.job_of_leaf[L] = LEAF_VIOL;
    list_push(t.st, &t.st->n_viol, a.viol, a.list_cap, leaf_code(L));
}

// What a child side tells its node.
struct Arrival {
    Box3 b;
    int slots, del, height;
};

// The two walkers that arrive at a node hand their data over in a mailbox per side:
// two 16-byte words, written and read whole, whose two low bits of the last word
// (counts have 30) say that it is there, and the height in the exchange that decides
// who is second.
constexpr int MAIL_SPINS = 1 << 20;
__device__ __forceinline__ void mail_write(uint4* p, uint4 v) {
    asm volatile(
        "{\n\t.reg .b128 s;\n\t"
        "mov.b128 s, {%0, %1};\n\t"
        "st.relaxed.gpu.global.b128 [%2], s;\n\t}" ::"l"((unsigned long long)v.y << 32 | v.x),
        "l"((unsigned long long)v.w << 32 | v.z), "l"(p)
        : "memory");
}
__device__ __forceinline__ uint4 mail_read(const uint4* p) {
    unsigned long long lo, hi;
    asm volatile(
        "{\n\t.reg .b128 d;\n\t"
        "ld.relaxed.gpu.global.b128 d, [%2];\n\t"
        "mov.b128 {%0, %1}, d;\n\t}"
        : "=l"(lo), "=l"(hi)
        : "l"(p)
        : "memory");
    return make_uint4((unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32));
}
struct Mail {
    uint4 *own, *other;
    uint4 u, v;  // the other side's words, if they were there already
    int h;       // 0: this walker is the first of the two
};
__device__ __forceinline__ void mail_send(const UpdateAux& a, int X, int side, const Arrival& m, Mail& k) {
    k.own = a.mail + 4 * (size_t)X + 2 * side;
    k.other = a.mail + 4 * (size_t)X + 2 * (side ^ 1);
    mail_write(k.own, make_uint4(__float_as_uint(m.b.lo[0]), __float_as_uint(m.b.lo[1]), __float_as_uint(m.b.lo[2]),
                                 (unsigned)m.slots << 2 | 1u));
    mail_write(k.own + 1, make_uint4(__float_as_uint(m.b.hi[0]), __float_as_uint(m.b.hi[1]),
                                     __float_as_uint(m.b.hi[2]), (unsigned)m.del << 2 | 1u));
    k.h = atomicExch(&a.arrive[X], m.height << 2 | 1);
    k.u = mail_read(k.other);
    k.v = mail_read(k.other + 1);
}
// True for the second walker at X, which gets the first one's data in `o`; the
// mailboxes are empty again.
__device__ __forceinline__ bool mail_take(const DevTree& t, const UpdateAux& a, int X, Mail& k, Arrival& o) {
    if (k.h == 0) return false;
    // The other walker wrote its words before its exchange; what this walker
    // overtook is on its way.
    for (int i = 0; !(k.u.w & 1u) || !(k.v.w & 1u); ++i) {
        if (i > MAIL_SPINS) {
            atomicOr(&t.st->err, ERR_LOOP);
            return false;
        }
        k.u = mail_read(k.other);
        k.v = mail_read(k.other + 1);
    }
    const uint4 zero = make_uint4(0, 0, 0, 0);
    mail_write(k.own, zero);
    mail_write(k.own + 1, zero);
    mail_write(k.other, zero);
    mail_write(k.other + 1, zero);
    a.arrive[X] = 0;
    o.b.lo[0] = __uint_as_float(k.u.x), o.b.lo[1] = __uint_as_float(k.u.y), o.b.lo[2] = __uint_as_float(k.u.z);
    o.b.hi[0] = __uint_as_float(k.v.x), o.b.hi[1] = __uint_as_float(k.v.y), o.b.hi[2] = __uint_as_float(k.v.z);
    o.slots = (int)(k.u.w >> 2);
    o.del = (int)(k.v.w >> 2);
    o.height = k.h >> 2;
    return true;
}

// The rebuild criteria of a node with `slots` stored points, `del` of them deleted,
// `left` valid ones on its left, and height h.
__device__ __forceinline__ bool violates(const Criteria& c, int slots, int del, int left, int h) {
    bool viol = false;
    if (slots > c.min_size) {
        // alpha_del on stored slots; alpha_bal on valid points.  (The reference
        // weighs balance by sizes that still include lazily deleted nodes; here a
        // rebuild that purges deleted points below would then unbalance the
        // ancestors and cascade into rebuilds of ever larger subtrees, round after
        // round.)
        const float fd = (float)del / (float)slots;
        const int valid = slots - del;
        const float fb = valid > 0 ? (float)left / (float)valid : 0.5f;
        viol = fd > c.alpha_del || fb > c.alpha_bal || fb < 1.0f - c.alpha_bal;
    }
    // Height guard, keeps every traversal stack within MAX_STACK:
    // h > 2 * ceil(log2(slots / fill + 1)) + 8, without the division.
    return viol || (h > 8 && slots < (long long)max(c.fill, 1) << (((h - 7) >> 1) - 1));
}

// One thread per item walks up to the root; of the two walkers that meet at a node
// the second goes on.  Bound by the walk's chain, one link per level: the data of
// the other side comes with the exchange that decides who is second (mail_send),
// or, where the other side does not change (pend = 1, no exchange), from loads
// issued a level ahead, as are the node's links; what a level has to store and to
// check runs while its exchange is in flight.  The stored boxes and counts are
// read by nobody in this launch.  Before, each level cost the release of its
// writes, the arrival, the loads and then the arithmetic: 15 levels took 33 us,
// 17 now (14,400-point scan into 500,000 points, four refits: the call went from
// 548 to 485 us; small edits of a 100,000-point map, 26 -> 13 us: 632 -> 535).
__global__ void __launch_bounds__(128) refit_compute_kernel(DevTree t, UpdateAux a, const int* items,
                                                            const int* n_items, Criteria c) {
    chain_begin();
    const int n_it = min(*n_items, a.list_cap);
    for (int i = first_item(); i < n_it; i += gridDim.x * blockDim.x) {
        const int item = items[i];
        const int link = item_link(t, item);
        if (item < 0) a.dirty_flag[code_leaf(item)] = 0;  // nothing below reads the flag
        if (link < 0) continue;
        int X = link >> 1, side = link & 1;
        // of X: its child codes, and its other side's box where that does not change
        NodeRec r;
        int4 cc;
        int2 wi;
        int lp = 0, expect = 0;
        auto node_ahead = [&](int Y) {  // (the sentinel, Y = 0, has no parent and is not counted)
            r = load_node_cg(t.node, Y);
            cc = __ldcg(t.ncnt + Y);
            lp = __ldcg(t.nparent + Y);
            expect = __ldcg(a.pend + Y);
            wi = __ldcg(t.winfo + Y);
        };
        node_ahead(X);
        // The child `code` of X on `side`; check: a node to hold against the criteria.
        Arrival m;
        int code = item, left = 0;
        bool check = false;
        if (item < 0) {
            const int L = code_leaf(item);
            const int n = __ldcg(&t.leaf_n[L]);
            const int cnt = n < LEAF_CAP ? n : LEAF_CAP;
            m.b = empty_box();
            m.del = 0;
            const float4* lpn = t.pts + (long long)L * LEAF_CAP;
            for (int j0 = 0; j0 < cnt; j0 += 16) {
                float4 p[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) p[u] = __ldcg(lpn + j0 + u);  // (slots past the fill stay in the bucket)
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    if (j0 + u >= cnt) break;
                    if (__float_as_uint(p[u].w) & F_DEL)
                        ++m.del;
                    else
                        box_grow(m.b, p[u].x, p[u].y, p[u].z);
                }
            }
            m.slots = n;
            m.height = 0;
            if (n > LEAF_CAP) list_leaf_violator(t, a, L);  // an overflowing bucket must be split
        } else {  // the builder wrote the subtree's box and counts into X
            code = side ? r.right() : r.left();
            m.b = r.box(side);
            m.slots = side ? cc.z : cc.x;
            m.del = side ? cc.w : cc.y;
            m.height = child_height(t, code);
        }
        for (int steps = 0;; ++steps) {
            if (steps > MAX_WALK) {
                atomicOr(&t.st->err, ERR_LOOP);
                return;
            }
            const int at = X, at_side = side, up = lp;
            const int2 at_wi = wi;
            const bool meet = X > 0 && expect > 1;
            Arrival o;
            Mail k;
            if (meet) {
                mail_send(a, X, side, m, k);
            } else {
                o.b = r.box(side ^ 1);
                o.slots = side ? cc.x : cc.z;
                o.del = side ? cc.y : cc.w;
                o.height = child_height(t, side ? r.left() : r.right());
            }
            if (X > 0) node_ahead(up >> 1);
            write_child_box(t.node, at, at_side, m.b);
            write_child_cnt(t.ncnt, at, at_side, m.slots, m.del);
            wide_update(t, at_wi, at_side, code, m.b, m.slots - m.del);
            if (check) {
                t.nheight[code] = m.height;
                a.pend[code] = 0;
                if (violates(c, m.slots, m.del, left, m.height)) {
                    a.viol_flag[code] = 1;
                    list_push(t.st, &t.st->n_viol, a.viol, a.list_cap, code);
                }
            }
            if (at == 0 || (meet && !mail_take(t, a, at, k, o))) break;
            // X's own data, its children in side order
            const Arrival& l = at_side ? o : m;
            const Arrival& rr = at_side ? m : o;
            Box3 b = empty_box();
            if (!box_empty(l.b)) box_union(b, l.b);
            if (!box_empty(rr.b)) box_union(b, rr.b);
            left = l.slots - l.del;
            const int slots = l.slots + rr.slots, del = l.del + rr.del, h = 1 + max(l.height, rr.height);
            m.b = b;
            m.slots = slots;
            m.del = del;
            m.height = h;
            check = true;
            code = at;
            X = up >> 1;
            side = up & 1;
        }
    }
}


// ---- rebuild jobs ----------------------------------------------------------------

constexpr int SETTLE_THREADS = 1024;
constexpr int LIST_THREADS = 512;  // (settle_kernel<true>, which needs the registers)

// The topmost violator on the way from node X up to the root, X included (0: none).
__device__ __forceinline__ int top_violator(const DevTree& t, const UpdateAux& a, int X) {
    int top = 0;
    for (int steps = 0; X > 0; ++steps) {
        if (steps > MAX_WALK) {
            atomicOr(&t.st->err, ERR_LOOP);
            return 0;
        }
        const int flag = __ldcg(a.viol_flag + X), up = __ldcg(t.nparent + X);  // one round trip for both
        if (flag) top = X;
        X = up >> 1;
    }
    return top;
}

// A rebuild job for the subtree `code` below `link`; its index, or -1.
__device__ __forceinline__ int new_job(const DevTree& t, const UpdateAux& a, int code, int link) {
    const int j = atomicAdd(&t.st->n_jobs, 1);
    if (j >= a.list_cap) {
        atomicOr(&t.st->err, ERR_LIST);
        return -1;
    }
    a.jobs[j] = code;
    a.job_link[j] = link;
    return j;
}

// First pass over leaf L / node X: what it belongs to, into leaf_job / node_job: a
// violating node (> 0), its own job (-1 - index; leaves only) or nothing (0).  A
// violator without one above makes its job.
__device__ __forceinline__ void choose_leaf(const DevTree& t, const UpdateAux& a, int L) {
    const int lp = __ldcg(t.lparent + L), mark = __ldcg(a.job_of_leaf + L);
    int top = lp >= 0 ? top_violator(t, a, lp >> 1) : 0;
    if (mark == LEAF_VIOL) {
        int j = -1;
        if (top == 0 && lp >= 0) j = new_job(t, a, leaf_code(L), lp);
        a.job_of_leaf[L] = j;
        if (j >= 0) top = -1 - j;
    }
    a.leaf_job[L] = top;
}
__device__ __forceinline__ void choose_node(const DevTree& t, const UpdateAux& a, int X) {
    const int link = __ldcg(t.nparent + X);
    const int top = link >= 0 ? top_violator(t, a, X) : 0;
    if (top == X) a.job_of_node[X] = new_job(t, a, X, link);
    a.node_job[X] = top;
}

// Valid points among leaf L's first m slots, and those whose deletion is reported
// (acquire_removed_points).
__device__ __forceinline__ void count_slots(const DevTree& t, int L, int m, int& valid, int& reported) {
    const float* lw = reinterpret_cast<const float*>(t.pts + (long long)L * LEAF_CAP) + 3;
    valid = reported = 0;
    // eight flag words in flight (slots past the fill count stay in the bucket)
    for (int j0 = 0; j0 < m; j0 += 8) {
        float w[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) w[u] = lw[4 * (j0 + u)];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const unsigned f = __float_as_uint(w[u]);
            if (j0 + u >= m) continue;
            valid += (f & F_DEL) ? 0 : 1;
            reported += (f & (F_DEL | F_DSDEL)) == F_DEL ? 1 : 0;
        }
    }
}
__device__ __forceinline__ int count_valid(const DevTree& t, int L) {
    int valid, reported;
    count_slots(t, L, min(t.leaf_n[L], LEAF_CAP), valid, reported);
    return valid;
}

// Second pass: the index of the job (or -1) of leaf L / node X; a leaf's valid points
// are added to its job's count, as are those that found its bucket full (leaf_n counts
// them too).
__device__ __forceinline__ void count_leaf(const DevTree& t, const UpdateAux& a, int L) {
    const int top = a.leaf_job[L];
    const int j = top > 0 ? __ldcg(a.job_of_node + top) : top < 0 ? -1 - top : -1;
    a.leaf_job[L] = j;
    const int over = t.leaf_n[L] - LEAF_CAP;
    if (j >= 0) {
        atomicAdd(&a.job_count[j], count_valid(t, L) + max(over, 0));
        return;
    }
    if (over <= 0) return;
    atomicOr(&t.st->err, ERR_OVF_JOB);
    int* d = t.st->dbg;
    if (atomicCAS(&d[0], 0, 1) == 0) {
        d[1] = L;
        d[2] = t.lparent[L];
        d[3] = t.leaf_n[L];
        d[4] = a.job_of_leaf[L];
        d[5] = a.dirty_flag[L];
        int lp = t.lparent[L];
        d[6] = lp >= 0 ? a.viol_flag[lp >> 1] : -7;
        d[7] = t.st->n_ovf;
    }
}
__device__ __forceinline__ void count_node(const DevTree& t, const UpdateAux& a, int X) {
    const int top = a.node_job[X];
    a.node_job[X] = top > 0 ? __ldcg(a.job_of_node + top) : -1;
}

// job_off = exclusive prefix sum of job_count over the selected jobs,
// job_off[n_jobs] = st->job_total = the sum, st->max_job = the largest job: one
// block, its width jobs per step.
__device__ void job_scan(const DevTree& t, const UpdateAux& a) {
    __shared__ int wsum[32];
    __shared__ int carry, mx;
    const int n = min(__ldcg(&t.st->n_jobs), a.list_cap);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (threadIdx.x == 0) {
        carry = 0;
        mx = 0;
    }
    __syncthreads();
    for (int base = 0; base < n; base += blockDim.x) {
        const int i = base + threadIdx.x;
        const int v = i < n ? __ldcg(a.job_count + i) : 0;
        int inc = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) wsum[w] = inc;
        if (v > 0) atomicMax(&mx, v);
        __syncthreads();
        if (w == 0) {
            const int ws = lane < warps ? wsum[lane] : 0;
            int wi = ws;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, wi, o);
                if (lane >= o) wi += y;
            }
            wsum[lane] = wi - ws;
        }
        __syncthreads();
        const int c = carry;
        if (i < n) a.job_off[i] = c + wsum[w] + inc - v;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = c + wsum[w] + inc;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        a.job_off[n] = carry;
        t.st->job_total = carry;
        t.st->max_job = mx;
    }
}

__device__ __forceinline__ void snapshot_root(const DevTree& t) {
    int4 c = t.ncnt[0];
    t.st->root_code = __float_as_int(t.node[3].x);
    t.st->root_slots = c.x;
    t.st->root_deleted = c.y;
    int rc = t.st->root_code;
    t.st->root_height = rc > 0 ? t.nheight[rc] : 0;
}

// Pool bookkeeping after a build: the free-stack entries taken are gone.
__device__ __forceinline__ void finish_alloc(DevStatus* st) {
    st->free_node_n = max(0, st->free_node_n - st->free_node_taken);
    st->free_leaf_n = max(0, st->free_leaf_n - st->free_leaf_taken);
    st->free_node_taken = 0;
    st->free_leaf_taken = 0;
}

// All blocks of a cooperative launch meet here.  The wait is bounded: past the
// bound it raises ERR_LOOP and goes on.
constexpr int BARRIER_SPINS = 1 << 22;
__device__ __forceinline__ void grid_barrier(DevStatus* st) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned ticket = atomicAdd(&st->barrier, 1u);
        const unsigned target = (ticket / gridDim.x + 1u) * gridDim.x;
        for (int i = 0;; ++i) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&st->barrier) : "memory");
            if (v >= target) break;
            if (i > BARRIER_SPINS) {
                atomicOr(&st->err, ERR_LOOP);
                break;
            }
        }
        __threadfence();
    }
    __syncthreads();
}

// A place for each lane that wants n of something counted at `counter`: one addition
// per warp.
template <class T>
__device__ __forceinline__ T warp_places(T* counter, int n) {
    const int lane = threadIdx.x & 31;
    int inc = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
    }
    T base = 0;
    if (lane == 31 && inc) base = atomicAdd(counter, (T)inc);
    return __shfl_sync(0xffffffffu, base, 31) + (T)(inc - n);
}

// ---- the same on a map with more leaves and nodes than the device has threads: from
// the violators up, then from the jobs down

// Violator i becomes a job unless one of its ancestors violates too.
__device__ __forceinline__ void choose_violator(const DevTree& t, const UpdateAux& a, int i) {
    const int code = a.viol[i], L = code < 0 ? code_leaf(code) : 0;
    const int link = code < 0 ? __ldcg(t.lparent + L) : __ldcg(t.nparent + code);
    int j = -1;
    if (link >= 0 && top_violator(t, a, link >> 1) == 0) j = new_job(t, a, code, link);
    if (code < 0) {
        a.job_of_leaf[L] = j;
        if (j >= 0) a.leaf_job[L] = j;
    } else if (j >= 0) {
        a.job_of_node[code] = j;
        a.node_job[code] = j;
    }
}

// Everything below the jobs into a.items: leaf codes, and 2 * node + 1 for nodes whose
// children are listed too (2 * node: in the next round).  A round takes three levels, a
// thread per node; its entries follow those of the rounds before.  Ends with a grid
// barrier; returns the number of entries.
constexpr int LIST_ROUNDS = sizeof(DevStatus::level_n) / sizeof(int);
static_assert(3 * (LIST_ROUNDS - 1) > MAX_STACK, "a round takes three levels");
__device__ int list_jobs(const DevTree& t, const UpdateAux& a, int i0, int step) {
    DevStatus* st = t.st;
    const int lane = threadIdx.x & 31;
    int begin = 0, end = min(__ldcg(&st->n_jobs), a.list_cap);
    for (int i = i0; i < end; i += step) {
        const int c = __ldcg(a.jobs + i);
        a.items[i] = c < 0 ? c : 2 * c;
    }
    for (int r = 0; r < LIST_ROUNDS && end > begin; ++r) {
        for (int i = begin + i0; i - lane < end; i += step) {  // (whole warps: one reservation each)
            const int item = i < end ? __ldcg(a.items + i) : -1;
            const bool open = item > 0 && !(item & 1);
            // children, grandchildren and theirs: the loads of one level go out together
            int c[14];
            int j = 0, n = 0;
            auto kids = [&](int X, int at) {
                float2 k = make_float2(0.f, 0.f);
                if (X > 0) k = __ldcg(reinterpret_cast<const float2*>(t.node + 4 * X + 3));
                c[at] = __float_as_int(k.x);
                c[at + 1] = __float_as_int(k.y);
            };
            if (open) j = __ldcg(a.node_job + (item >> 1));
            kids(open ? item >> 1 : 0, 0);
#pragma unroll
            for (int u = 0; u < 6; ++u) kids(c[u], 2 + 2 * u);
#pragma unroll
            for (int u = 0; u < 14; ++u) n += c[u] != 0 ? 1 : 0;
            int at = end + warp_places(&st->level_n[r], n);
            if (n > 0 && at + n > a.list_cap) {
                atomicOr(&st->err, ERR_LIST);
                continue;
            }
#pragma unroll
            for (int u = 0; u < 14; ++u) {
                if (c[u] == 0) continue;
                if (c[u] < 0)
                    a.leaf_job[code_leaf(c[u])] = j;
                else
                    a.node_job[c[u]] = j;
                a.items[at++] = c[u] < 0 ? c[u] : 2 * c[u] + (u < 6 ? 1 : 0);
            }
        }
        grid_barrier(st);
        begin = end;
        end = min(end + __ldcg(&st->level_n[r]), a.list_cap);
    }
    // (a taller tree than the rounds reach: its points must not be dropped)
    for (int i = begin + i0; i < end; i += step) {
        const int item = __ldcg(a.items + i);
        if (item > 0 && !(item & 1)) atomicOr(&st->err, ERR_LIST);
    }
    return end;
}

// A listed leaf's points, those that found its bucket full included.
__device__ __forceinline__ void count_listed(const DevTree& t, const UpdateAux& a, int L) {
    atomicAdd(&a.job_count[__ldcg(a.leaf_job + L)], count_valid(t, L) + max(__ldcg(t.leaf_n + L) - LEAF_CAP, 0));
}

// After a refit: the root's snapshot and, if the refit recorded violators, the
// rebuild jobs (topmost violators), the job every leaf and node belongs to, the
// jobs' sizes and offsets; the status block goes to pinned host memory at `host`.
// Bound by the walk up the tree, a chain of dependent loads, so every leaf and node
// gets its own thread where the device has them, and there is one walk: it finds the
// topmost violator, which is the job.  One cooperative launch with two grid barriers
// replaces eight small launches and a copy (500,000 points: 60 us of kernels became
// 34 with a walk per choice and three barriers, 26 with one and two; 4 when
// there is nothing to rebuild).  14,400-point scan into 500,000 points, with two
// such launches: 624 -> 548 us, later 344 -> 338; small edits of 100,000 points
// 773 -> 632, later 455 -> 418.  LIST: from the violators up and from the jobs down
// (list_jobs), for maps where a walk from every leaf costs more than that chain of
// rounds.  select = false: no jobs, the marks are cleared.
template <bool LIST>
__global__ void __launch_bounds__(LIST ? LIST_THREADS : SETTLE_THREADS, 2) settle_kernel(DevTree t, UpdateAux a, bool select,
                                                                   DevStatus* __restrict__ host) {
    DevStatus* st = t.st;
    const int nv = min(__ldcg(&st->n_viol), a.list_cap);
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    if (i0 == 0) {
        snapshot_root(t);
        st->n_items = 0;  // the dirty list is consumed
    }
    if (nv > 0 && select) {
        const int leaf_top = min(__ldcg(&st->leaf_top), t.leaf_cap), node_top = min(__ldcg(&st->node_top), t.node_cap);
        const int all = leaf_top + node_top;
        if (LIST) {
            for (int i = i0; i < nv; i += step) choose_violator(t, a, i);
        } else {
            for (int i = i0; i < all; i += step) {
                if (i < leaf_top)
                    choose_leaf(t, a, i);
                else if (i > leaf_top)
                    choose_node(t, a, i - leaf_top);
            }
        }
        grid_barrier(st);
        for (int i = i0; i < nv; i += step) {
            const int code = a.viol[i];
            if (code > 0) a.viol_flag[code] = 0;
        }
        if (LIST) {
            const int n = list_jobs(t, a, i0, step);
            for (int i = i0; i < n; i += step) {
                const int item = __ldcg(a.items + i);
                if (item < 0) count_listed(t, a, code_leaf(item));
            }
            if (i0 == 0) st->n_queue = n;
        } else {
            for (int i = i0; i < all; i += step) {
                if (i < leaf_top)
                    count_leaf(t, a, i);
                else if (i > leaf_top)
                    count_node(t, a, i - leaf_top);
            }
        }
        grid_barrier(st);
        if (blockIdx.x == 0) job_scan(t, a);
    } else if (nv > 0) {
        for (int i = i0; i < nv; i += step) {
            const int code = a.viol[i];
            if (code > 0)
                a.viol_flag[code] = 0;
            else
                a.job_of_leaf[code_leaf(code)] = -1;
        }
        grid_barrier(st);  // every block has read n_viol
    }
    if (blockIdx.x != 0) return;
    __syncthreads();
    const int words = sizeof(DevStatus) / 4;
    for (int w = threadIdx.x; w < words; w += blockDim.x)
        reinterpret_cast<int*>(host)[w] = __ldcg(reinterpret_cast<const int*>(st) + w);
    __syncthreads();
    if (threadIdx.x == 0) st->n_viol = 0;  // the next refit records afresh
}

// The points of leaf L's job from place `pos` of out on, its deleted ones from `rem` of
// removed on.
__device__ __forceinline__ void gather_leaf(const DevTree& t, int L, int m, float4* __restrict__ out, int pos,
                                            float4* __restrict__ removed, long long rem, long long removed_cap) {
    const float4* lp = t.pts + (long long)L * LEAF_CAP;
    for (int s0 = 0; s0 < m; s0 += 8) {
        float4 pb[8];  // eight slots in flight (the bucket always has LEAF_CAP slots)
#pragma unroll
        for (int u = 0; u < 8; ++u) pb[u] = lp[s0 + u];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            if (s0 + u >= m) break;
            const float4 p = pb[u];
            const uint32_t w = __float_as_uint(p.w);
            if (!(w & F_DEL)) {
                out[pos++] = p;
            } else if (!(w & F_DSDEL)) {
                // Dropped deleted points are kept for acquire_removed_points
                // (flatten with DELETE_POINTS_REC, ikd_Tree.cpp:1338-1342).
                if (rem < removed_cap) removed[rem] = make_float4(p.x, p.y, p.z, __uint_as_float(w & ID_MASK));
                ++rem;
            }
        }
    }
}

// The points of every job into `out`, back to back; the jobs' leaves and nodes go
// to the free stacks.  One thread per leaf and node (n_queue
// of them listed in a.items, or, below zero, all of the map's) and overflow point; the shared
// counters take one addition per warp (500,000 points: 13 -> 8 us).
__global__ void job_gather_kernel(DevTree t, UpdateAux a, int n_queue, int leaf_top, int node_top, const int4* ovf_leaf,
                                  const float4* ovf_pts, int max_ovf, float4* __restrict__ out,
                                  float4* __restrict__ removed, long long removed_cap) {
    chain_begin();
    constexpr unsigned ALL = 0xffffffffu;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int all = n_queue >= 0 ? n_queue : leaf_top + node_top;
    // this thread's leaf L or node X, -1: none; whole warps stay together for the
    // shared additions
    int L = -1, X = -1;
    if (n_queue >= 0) {
        const int item = i < all ? a.items[i] : 0;
        if (item < 0) L = code_leaf(item);
        if (item > 0) X = item >> 1;
    } else if (i < leaf_top) {
        if (a.leaf_job[i] >= 0) L = i;
    } else if (i > leaf_top && i < all && a.node_job[i - leaf_top] >= 0) {
        X = i - leaf_top;
    }
    if (__any_sync(ALL, L >= 0)) {
        int m = 0, nv = 0, nd = 0, pos = 0;
        if (L >= 0) {
            const int j = a.leaf_job[L];
            m = min(t.leaf_n[L], LEAF_CAP);
            count_slots(t, L, m, nv, nd);
            pos = a.job_off[j] + atomicAdd(&a.job_fill[j], nv);
        }
        const long long rem = (long long)warp_places((unsigned long long*)&t.st->removed_n, nd);
        const int f = warp_places(&t.st->free_leaf_n, L >= 0 ? 1 : 0);
        if (L >= 0) {
            gather_leaf(t, L, m, out, pos, removed, rem, removed_cap);
            t.lparent[L] = -1;
            t.leaf_n[L] = 0;
            t.free_leaf[f] = L;
        }
    }
    if (__any_sync(ALL, X >= 0)) {
        const int f = warp_places(&t.st->free_node_n, X >= 0 ? 1 : 0);
        if (X >= 0) {
            t.nparent[X] = -1;
            t.free_node[f] = X;
        }
    }
    const int o = i - all;
    if (o < 0 || o >= min(max_ovf, t.st->n_ovf)) return;
    const int jo = a.leaf_job[ovf_leaf[o].x];
    if (jo >= 0) out[a.job_off[jo] + atomicAdd(&a.job_fill[jo], 1)] = ovf_pts[o];
}

// Resets per-job state and queues each job's parent for the follow-up refit
// (one block).
__global__ void __launch_bounds__(1024) job_finish_kernel(DevTree t, UpdateAux a) {
    chain_begin();
    const int n = min(t.st->n_jobs, a.list_cap);
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        int code = a.jobs[j];
        if (code < 0)
            a.job_of_leaf[code_leaf(code)] = -1;
        else
            a.job_of_node[code] = -1;
        a.job_count[j] = 0;
        a.job_fill[j] = 0;
        const int link = a.job_link[j];
        if (link > 1) list_push(t.st, &t.st->n_items, a.items, a.list_cap, link);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        finish_alloc(t.st);
        t.st->max_job = 0;
        t.st->n_ovf = 0;
        t.st->n_jobs = 0;
        t.st->barrier = 0;  // the next settle_kernel may have another grid
        t.st->n_queue = 0;
        for (int r = 0; r < LIST_ROUNDS; ++r) t.st->level_n[r] = 0;
    }
}

// ---- box walks by teams of four lanes ---------------------------------------------

// Ints of a team's stack for a tree of this height: every record level replaces
// one entry by at most eight.
constexpr int TEAM = 4;
constexpr int TEAM_CTA = 128;
__host__ __device__ constexpr int team_stack_entries(int height) { return 7 * (1 + (height + 2) / 3) + 1; }
size_t team_stack_bytes(int height) { return (size_t)team_stack_entries(height) * (TEAM_CTA / TEAM) * sizeof(int); }

// Every team walks its own box down the wide records: lane `sub` tests two of the
// eight children of a record, then four of the 16 slots of half a bucket.  overlap
// (lo, hi) says whether a child's box can hold a hit; leaf(L, h, n, p, on) gets the
// lane's slots 16 h + 4 sub .. of leaf L in p (n = its fill count; on = false: no leaf
// here, but the call is made by the whole warp, so it may vote) and returns true
// when the team is done.  Leaves come in descending order, halves ascending.  The
// warp's teams step together: in each step every team takes its next record or
// leaf.  Whole warps call it; teams without a box pass active = false.
template <class O, class F>
__device__ __forceinline__ void team_walk(const DevTree& t, bool active, int* stacks, O overlap, F leaf) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (TEAM - 1), gs = lane & ~(TEAM - 1);
    const int entries = team_stack_entries(t.height);
    int* stack = stacks + (threadIdx.x / TEAM) * entries;
    const unsigned below = (1u << lane) - (1u << gs);
    int sp = active ? 1 : 0;
    int cur = t.start;  // the top of the stack, in every lane of the team
    for (int steps = 0;; ++steps) {
        if (steps > t.max_visits) {
            if (sp > 0) atomicOr(&t.st->err, ERR_LOOP);
            break;
        }
        const bool node = sp > 0 && cur >= 0, lf = sp > 0 && cur < 0;
        if (!__any_sync(ALL, sp > 0)) break;
        if (__any_sync(ALL, node)) {
            bool al0 = false, al1 = false;
            int c0 = 0, c1 = 0;
            if (node) {
                const float4* p = t.wide + (long long)cur * 16 + 4 * sub;
                const float4 a = p[0], b = p[1], c = p[2], d = p[3];  // (the top records stay in L1)
                const float lo0[3] = {a.x, a.z, b.x}, hi0[3] = {b.z, c.x, c.z};
                const float lo1[3] = {a.y, a.w, b.y}, hi1[3] = {b.w, c.y, c.w};
                al0 = lo0[0] <= hi0[0] && overlap(lo0, hi0);
                al1 = lo1[0] <= hi1[0] && overlap(lo1, hi1);
                c0 = __float_as_int(d.x);
                c1 = __float_as_int(d.y);
            }
            const unsigned b0 = __ballot_sync(ALL, al0), b1 = __ballot_sync(ALL, al1);
            if (node) {
                const int at = sp - 1 + __popc(b0 & below) + __popc(b1 & below);
                sp += __popc(b0 >> gs & 15u) + __popc(b1 >> gs & 15u) - 1;
                if (sp > entries) {  // cannot happen: see team_stack_entries
                    if (sub == 0) atomicOr(&t.st->err, ERR_STACK);
                    sp = 0;
                } else {
                    if (al0) stack[at] = c0;
                    if (al1) stack[at + (al0 ? 1 : 0)] = c1;
                }
            }
        }
        if (__any_sync(ALL, lf)) {
            const int L = lf ? code_leaf(cur) : 0;
            const float4* lp = t.pts + (long long)L * LEAF_CAP + 4 * sub;
            float4 p[4];
            int n = 0;
            if (lf) {
                n = min(__ldcg(t.leaf_n + L), LEAF_CAP);
#pragma unroll
                for (int u = 0; u < 4; ++u) p[u] = __ldcg(lp + u);
            }
            bool done = leaf(L, 0, n, p, lf);
            const bool more = lf && !done && n > 16;
            if (__any_sync(ALL, more)) {
                if (more) {
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[u] = __ldcg(lp + 16 + u);
                }
                done = leaf(L, 1, n, p, more) || done;
            }
            if (lf) sp = done ? 0 : sp - 1;
        }
        __syncwarp();
        cur = sp > 0 ? stack[sp - 1] : 0;
        __syncwarp();  // read before the next step writes
    }
}

// ---- box / point deletion, box re-insertion ----------------------------------------

constexpr int DB_THREADS = 128;
constexpr int DB_WARPS = DB_THREADS / 32;
constexpr int DB_STACK = DB_THREADS * (MAX_STACK + 2);
constexpr int DB_SPLIT_BITS_MAX = 6;
constexpr long long DB_TARGET_UNITS = 1024;

// Whether child `side` of node record r (code: its index, 0 = sentinel) can
// hold deleted points of box qb: only the split planes bound those (left subtree:
// coordinates <= split, right: >= split).
__device__ __forceinline__ bool box_child(const Box3& qb, const NodeRec& r, int code, int side) {
    if (code > 0) {
        int ax = r.axis();
        float sp = r.split();
        if (side == 0 && sp < qb.lo[ax]) return false;
        if (side == 1 && qb.hi[ax] <= sp) return false;
    }
    return true;
}

// Work unit (box bi, part): the CTA walks split_bits levels down from the
// root, taking the side that bit d of `part` names at depth d, and edits the
// subtree it reaches.  A leaf met above that depth belongs to the part whose
// remaining bits are zero.  Returns the code it reaches, or INT_MIN when the
// walk was pruned.
__device__ int box_seed(const DevTree& t, const Box3& qb, int part, int split_bits) {
    NodeRec r = load_node_cg(t.node, 0);
    int code = r.left();
    if (code == 0 || !box_child(qb, r, 0, 0)) return INT_MIN;
    for (int d = 0; d < split_bits; ++d) {
        if (code < 0) return (part >> d) == 0 ? code : INT_MIN;
        r = load_node_cg(t.node, code);
        int side = (part >> d) & 1;
        int c = side == 0 ? r.left() : r.right();
        if (c == 0 || !box_child(qb, r, code, side)) return INT_MIN;
        code = c;
    }
    return code;
}

// Restores box-deleted points (Add_by_range).  One CTA per work unit (box,
// top-level subtree).  Each round the CTA pops up to DB_THREADS items off a
// shared stack; threads expand nodes (pushing the children that can hold points
// of the box) and queue leaves, then each warp edits queued leaves one slot per
// lane.
__global__ void __launch_bounds__(DB_THREADS) box_restore_kernel(DevTree t, UpdateAux a,
                                                                 const float* boxes, long long m,
                                                                 int split_bits) {
    chain_begin();
    __shared__ int stack[DB_STACK];
    __shared__ int leafq[2 * DB_THREADS];
    __shared__ int top, nleaf;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const long long units = m << split_bits;
    for (long long u = blockIdx.x; u < units; u += gridDim.x) {
        const long long bi = u >> split_bits;
        const int part = (int)(u & ((1 << split_bits) - 1));
        Box3 qb;
        for (int k = 0; k < 3; ++k) {
            qb.lo[k] = boxes[bi * 6 + k];
            qb.hi[k] = boxes[bi * 6 + 3 + k];
        }
        if (threadIdx.x == 0) {
            top = 0;
            nleaf = 0;
            int seed = box_seed(t, qb, part, split_bits);
            if (seed != INT_MIN) stack[top++] = seed;
        }
        __syncthreads();
        for (int rounds = 0;; ++rounds) {
            int cur_top = top;
            if (cur_top == 0) break;
            if (rounds > t.max_visits) {
                if (threadIdx.x == 0) atomicOr(&t.st->err, ERR_LOOP);
                break;
            }
            int n = cur_top < DB_THREADS ? cur_top : DB_THREADS;
            int base = cur_top - n;
            int code = threadIdx.x < n ? stack[base + threadIdx.x] : 0;
            __syncthreads();
            if (threadIdx.x == 0) top = base;
            __syncthreads();
            if (threadIdx.x < n) {
                if (code >= 0) {
                    NodeRec r = load_node_cg(t.node, code);
                    for (int side = 0; side < 2; ++side) {
                        int c = side == 0 ? r.left() : r.right();
                        if (c == 0 || !box_child(qb, r, code, side)) continue;
                        if (c < 0) {
                            leafq[atomicAdd(&nleaf, 1)] = c;  // <= 2 per thread
                        } else {
                            int pos = atomicAdd(&top, 1);
                            if (pos < DB_STACK)
                                stack[pos] = c;
                            else
                                atomicOr(&t.st->err, ERR_STACK);
                        }
                    }
                } else {
                    leafq[atomicAdd(&nleaf, 1)] = code;
                }
            }
            __syncthreads();
            const int nq = nleaf;
            for (int q = warp; q < nq; q += DB_WARPS) {
                const int L = code_leaf(leafq[q]);
                const int nl = t.leaf_n[L];
                float4* lp = t.pts + (long long)L * LEAF_CAP;
                bool hit = false;
                if (lane < nl && lane < LEAF_CAP) {
                    float4 p = __ldcg(lp + lane);
                    uint32_t w = __float_as_uint(p.w);
                    if ((w & F_DEL) && !(w & F_DSDEL) && qbox_holds(qb, p.x, p.y, p.z)) {
                        atomicAnd((unsigned*)&lp[lane].w, ~F_DEL);
                        hit = true;
                    }
                }
                if (__any_sync(0xffffffffu, hit) && lane == 0) mark_dirty(a, t.st, L);
            }
            __syncthreads();
            if (threadIdx.x == 0) nleaf = 0;
        }
        __syncthreads();
    }
}

// Box deletion: one warp per work unit (box, subtree `levels` records below the
// top, named by three bits of `part` a level, or top_bits for the top record, which
// may have fewer children; a leaf met above belongs to the part whose remaining bits
// are zero).  The warp keeps a stack of records and leaves
// (code * 2 + covered), takes up to eight items a step, a team of four lanes each:
// two children per lane, or four slots of a bucket half.  Above BD_WIDE entries only
// one record a step is expanded, which bounds the stack (bd_stack_entries).  Bound by
// the chain of records; the kernel it replaces walked binary nodes with four block
// barriers a level: 37 us for six boxes in 500,000 points, 13 now.
// Where many boxes leave each of them few units, a unit that is not through after
// `limit` steps puts what is on its stack on the list `spill` (as much as fits: the
// bottom, which are the largest subtrees) and a second launch takes the list, a warp per
// entry (`list`).  8,000,000 points, the call, a box of a million among 300 / 3,000 small
// ones: 10.1 / 38.2 ms without the list, 1.2 / 2.7 with it; a box of everything 18.5 /
// 283 ms and 1.8 / 17.1.
constexpr int BD_WINDOW = 8;
constexpr int BD_WIDE = 96;
constexpr int BD_LEVELS_MAX = 4;
constexpr long long BD_UNITS = 2048;
constexpr int BD_CTA = 128;
// Units per box below which a unit's work is limited (from there on the units are small
// themselves), and the limit: boxes of up to some 5,000 points stay where they are.  The
// second launch costs a call 1-2 us.
constexpr int BD_FEW_UNITS = 256;
constexpr int BD_LIMIT = 64;
constexpr int BD_SPILL_BLOCKS = 152 * 8;
__host__ __device__ constexpr int bd_stack_entries(int height) {
    return BD_WIDE + 7 * BD_WINDOW + 7 * (1 + (height + 2) / 3) + 1;
}
__global__ void __launch_bounds__(BD_CTA) box_delete_kernel(DevTree t, UpdateAux a, const float* boxes,
                                                            long long m, int levels, int top_bits,
                                                            uint32_t del_flags, long long* __restrict__ total,
                                                            bool list, int limit, int2* spill, int spill_cap) {
    chain_begin();
    extern __shared__ int stacks[];
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, sub = lane & (TEAM - 1), j = lane / TEAM;
    const unsigned below = (1u << lane) - 1u;
    const int entries = bd_stack_entries(t.height);
    int* stack = stacks + (threadIdx.x >> 5) * entries;
    const int bits = levels > 0 ? top_bits + 3 * (levels - 1) : 0;
    const long long units = list ? min(t.st->n_spill, spill_cap) : m << bits, warps = (long long)gridDim.x * (BD_CTA / 32);
    int count = 0;
    for (long long u = (long long)blockIdx.x * (BD_CTA / 32) + (threadIdx.x >> 5); u < units; u += warps) {
        const int2 sp_in = list ? spill[u] : make_int2(0, 0);
        const long long bi = list ? sp_in.y : u >> bits;
        const float* bx = boxes + bi * 6;
        Box3 qb;
        for (int k = 0; k < 3; ++k) {
            qb.lo[k] = bx[k];
            qb.hi[k] = bx[3 + k];
        }
        // down to the unit's subtree (the whole warp reads the same words)
        int part = (int)(u & ((1 << bits) - 1)), code = list ? sp_in.x >> 1 : t.start, cov = list ? sp_in.x & 1 : 0;
        bool live = true;
        for (int d = 0; !list && d < levels && live && code >= 0; ++d) {
            const int w = d == 0 ? top_bits : 3;
            const float* f =
                reinterpret_cast<const float*>(t.wide + (long long)code * 16) + wide_at(part & ((1 << w) - 1), 0);
            Box3 b;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                b.lo[k] = f[2 * k];
                b.hi[k] = f[6 + 2 * k];
            }
            code = __float_as_int(f[12]);
            part >>= w;
            live = code != 0 && !box_empty(b) && (cov || !qbox_disjoint(qb, b)) && (code > 0 || part == 0);
            cov = cov || qbox_covers(qb, b);
        }
        if (!live) continue;
        int sp = 1;
        __syncwarp();
        if (lane == 0) stack[0] = code * 2 + cov;
        __syncwarp();
        for (int steps = 0; sp > 0; ++steps) {
            if (steps > t.max_visits) {
                if (lane == 0) atomicOr(&t.st->err, ERR_LOOP);
                break;
            }
            if (limit > 0 && steps == limit) {
                // (the counter is left alone once the list is full: it must not wrap)
                int base = spill_cap;
                if (lane == 0 && __ldcg(&t.st->n_spill) < spill_cap) base = atomicAdd(&t.st->n_spill, sp);
                base = __shfl_sync(ALL, base, 0);
                const int k = base < spill_cap ? min(sp, spill_cap - base) : 0;
                for (int i = lane; i < k; i += 32) spill[base + i] = make_int2(stack[i], (int)bi);
                sp -= k;
                for (int i = lane; i - lane < sp; i += 32) {
                    const int v = i < sp ? stack[i + k] : 0;
                    __syncwarp();
                    if (i < sp) stack[i] = v;
                    __syncwarp();
                }
                if (sp == 0) break;
            }
            const int avail = min(sp, BD_WINDOW);
            const bool here = j < avail;
            const int it = here ? stack[sp - 1 - j] : 0;
            const int c = it >> 1;  // arithmetic shift: floor(it / 2)
            const bool cv = it & 1;
            const unsigned recs = __ballot_sync(ALL, here && c >= 0);  // (also: all items read)
            const bool rec = here && c >= 0 && (sp <= BD_WIDE || j == (__ffs(recs) - 1) / TEAM);
            // records: the children that overlap replace the item
            bool al0 = here && c >= 0 && !rec && sub == 0, al1 = false;
            int k0 = it, k1 = 0;
            if (rec) {
                const float4* p = t.wide + (long long)c * 16 + 4 * sub;
                const float4 x = p[0], y = p[1], z = p[2], w = p[3];  // (the top records stay in L1)
                Box3 b0, b1;
                b0.lo[0] = x.x, b0.lo[1] = x.z, b0.lo[2] = y.x, b0.hi[0] = y.z, b0.hi[1] = z.x, b0.hi[2] = z.z;
                b1.lo[0] = x.y, b1.lo[1] = x.w, b1.lo[2] = y.y, b1.hi[0] = y.w, b1.hi[1] = z.y, b1.hi[2] = z.w;
                al0 = !box_empty(b0) && (cv || !qbox_disjoint(qb, b0));
                al1 = !box_empty(b1) && (cv || !qbox_disjoint(qb, b1));
                k0 = __float_as_int(w.x) * 2 + (cv || qbox_covers(qb, b0) ? 1 : 0);
                k1 = __float_as_int(w.y) * 2 + (cv || qbox_covers(qb, b1) ? 1 : 0);
            }
            const unsigned b0 = __ballot_sync(ALL, al0), b1 = __ballot_sync(ALL, al1);
            const int end = sp - avail + __popc(b0) + __popc(b1);
            if (end > entries) {  // cannot happen: see bd_stack_entries
                if (lane == 0) atomicOr(&t.st->err, ERR_STACK);
                break;
            }
            // the first item's children on top: depth first
            const int at = end - 1 - (__popc(b0 & below) + __popc(b1 & below));
            if (al0) stack[at] = k0;
            if (al1) stack[at - (al0 ? 1 : 0)] = k1;
            sp = end;
            // leaves: all of a lane's slots and the fill count in one round trip, the
            // flags and the bucket's place in the dirty list in the next
            unsigned hits = 0;
            const int L = c < 0 ? code_leaf(c) : 0;
            float4* lp = t.pts + (long long)L * LEAF_CAP + 4 * sub;
            if (here && c < 0) {
                const int n = min(__ldcg(t.leaf_n + L), LEAF_CAP) - 4 * sub;
                float4 p[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) p[q] = __ldcg(lp + (q < 4 ? q : q + 12));
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if ((q < 4 ? q : q + 12) < n && !(__float_as_uint(p[q].w) & F_DEL) &&
                        (cv || qbox_holds(qb, p[q].x, p[q].y, p[q].z)))
                        hits |= 1u << q;
            }
            const unsigned hit = __ballot_sync(ALL, hits != 0) >> (lane & ~(TEAM - 1)) & 15u;
            unsigned old[8];
#pragma unroll
            for (int q = 0; q < 8; ++q)  // (another box of the call may have been first)
                old[q] = hits >> q & 1u ? atomicOr(reinterpret_cast<unsigned*>(lp + (q < 4 ? q : q + 12)) + 3, del_flags)
                                        : F_DEL;
            mark_dirty_warp(a, t.st, L, sub == 0 && hit != 0);
#pragma unroll
            for (int q = 0; q < 8; ++q) count += !(old[q] & F_DEL);
            __syncwarp();
        }
    }
    count = __reduce_add_sync(ALL, count);
    if (lane == 0 && count) atomicAdd((unsigned long long*)total, (unsigned long long)count);
}

// Subtree split for box edits: enough (box, subtree) units to fill the GPU
// when there are few boxes, none when there are many.
int box_split_bits(long long m) {
    int bits = 0;
    while (bits < DB_SPLIT_BITS_MAX && (m << bits) < DB_TARGET_UNITS) ++bits;
    return bits;
}

unsigned box_grid(long long units) { return (unsigned)(units < (1LL << 20) ? units : (1LL << 20)); }

// same_point (ikd_Tree.cpp:1368-1371): |a - b| < 1e-6 per axis, the float
// difference compared in double.
__device__ __forceinline__ bool same_point(float ax, float ay, float az, float bx, float by, float bz) {
    // 1e-6f is the largest float below 1e-6: the same test without doubles
    return fabsf(__fsub_rn(ax, bx)) <= 1e-6f && fabsf(__fsub_rn(ay, by)) <= 1e-6f && fabsf(__fsub_rn(az, bz)) <= 1e-6f;
}

// One team per point: the first match in the walk's order that no other team has
// taken is deleted.  Bound by the walk's chain of records (six where the binary
// walk of one thread took 17 nodes, its slots one after the other): 24 us for 1,000
// points in 100,000, 10 now.
__global__ void __launch_bounds__(TEAM_CTA) delete_points_kernel(DevTree t, UpdateAux a, const float* __restrict__ in,
                                                                 int stride, long long n) {
    chain_begin();
    extern __shared__ int stacks[];
    const long long i = ((long long)blockIdx.x * TEAM_CTA + threadIdx.x) / TEAM;
    const bool active = i < n;
    const int lane = threadIdx.x & 31, sub = lane & (TEAM - 1), gs = lane & ~(TEAM - 1);
    float q[3] = {0.f, 0.f, 0.f}, lo[3], hi[3];
    if (active)
        for (int k = 0; k < 3; ++k) q[k] = in[i * stride + k];
    // A match differs by < 1e-6 per axis; 2e-6 bounds the search box safely
    // (a larger coordinate rounds p +- 2e-6 only where no match can exist).
    for (int k = 0; k < 3; ++k) {
        lo[k] = __fsub_rn(q[k], 2e-6f);
        hi[k] = __fadd_rn(q[k], 2e-6f);
    }
    team_walk(
        t, active, stacks,
        [&](const float* l, const float* h) {
            return l[0] <= hi[0] && h[0] >= lo[0] && l[1] <= hi[1] && h[1] >= lo[1] && l[2] <= hi[2] && h[2] >= lo[2];
        },
        [&](int L, int half, int cnt, const float4* p, bool on) {
            unsigned m = 0;
            if (on) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (16 * half + 4 * sub + u < cnt && !(__float_as_uint(p[u].w) & F_DEL) &&
                        same_point(p[u].x, p[u].y, p[u].z, q[0], q[1], q[2]))
                        m |= 1u << u;
            }
            // the team's matches in slot order, until one is taken
            bool taken = false;
            while (true) {
                const unsigned any = __ballot_sync(0xffffffffu, m != 0 && !taken);
                if (any == 0) break;
                const unsigned mine = any >> gs & 15u;
                bool got = false;
                if (mine != 0 && sub == __ffs(mine) - 1) {
                    const int u = __ffs(m) - 1;
                    m &= m - 1;
                    unsigned* w = reinterpret_cast<unsigned*>(t.pts + (long long)L * LEAF_CAP + 16 * half + 4 * sub + u) + 3;
                    got = !(atomicOr(w, F_DEL) & F_DEL);
                    if (got) mark_dirty(a, t.st, L);
                }
                taken = taken || (__ballot_sync(0xffffffffu, got) >> gs & 15u) != 0;
            }
            return taken;
        });
}

__global__ void flatten_kernel(DevTree t, float4* __restrict__ out, long long* counter) {
    int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= t.st->leaf_top) return;
    if (t.lparent[L] < 0) return;
    int n = t.leaf_n[L];
    int m = n < LEAF_CAP ? n : LEAF_CAP;
    const float4* lp = t.pts + (long long)L * LEAF_CAP;
    int nv = count_valid(t, L);
    if (nv == 0) return;
    long long pos = (long long)atomicAdd((unsigned long long*)counter, (unsigned long long)nv);
    for (int s = 0; s < m; ++s) {
        float4 p = lp[s];
        if (!(__float_as_uint(p.w) & F_DEL)) out[pos++] = p;
    }
}

// Ids of every stored slot (valid or deleted) of the leaves in use; slots
// past `cap` are counted but not written.
__global__ void stored_ids_kernel(DevTree t, int* __restrict__ out, long long cap, long long* counter) {
    int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= t.st->leaf_top) return;
    if (t.lparent[L] < 0) return;
    const int m = min(t.leaf_n[L], LEAF_CAP);
    if (m == 0) return;
    const long long pos = (long long)atomicAdd((unsigned long long*)counter, (unsigned long long)m);
    const float4* lp = t.pts + (long long)L * LEAF_CAP;
    for (int s = 0; s < m; ++s)
        if (pos + s < cap) out[pos + s] = (int)(__float_as_uint(lp[s].w) & ID_MASK);
}

// The whole tree as the only violator: settle_kernel makes it the rebuild job.
__global__ void select_root_kernel(DevTree t, UpdateAux a) {
    chain_begin();
    const int code = __float_as_int(t.node[3].x);
    if (code == 0) return;
    if (code < 0) {
        list_leaf_violator(t, a, code_leaf(code));
        return;
    }
    a.viol_flag[code] = 1;
    a.viol[0] = code;
    t.st->n_viol = 1;
}

// ---- structural validation (diagnostics) ---------------------------------------------

__device__ __forceinline__ bool same_box(const Box3& a, const Box3& b) {
    for (int k = 0; k < 3; ++k)
        if (__float_as_uint(a.lo[k]) != __float_as_uint(b.lo[k]) || __float_as_uint(a.hi[k]) != __float_as_uint(b.hi[k]))
            return false;
    return true;
}

// For every live node: both children exist and point back; the child box and
// counts stored in the node equal what the child itself holds.
__device__ __forceinline__ void note_bad(DevStatus* st, int kind, int X, int side, int a0, int a1, int a2, int a3) {
    if (atomicCAS(&st->dbg[0], 0, kind) == 0) {
        st->dbg[1] = X;
        st->dbg[2] = side;
        st->dbg[3] = a0;
        st->dbg[4] = a1;
        st->dbg[5] = a2;
        st->dbg[6] = a3;
    }
}

// For every live node: both children exist and point back; the child box and
// counts stored in the node equal what the child itself holds.
__global__ void validate_nodes_kernel(DevTree t, bool at_rest, unsigned long long* bad) {
    int X = blockIdx.x * blockDim.x + threadIdx.x;
    if (X >= t.st->node_top) return;
    if (X > 0 && t.nparent[X] < 0) return;
    NodeRec r = load_node_cg(t.node, X);
    int4 cc = __ldcg(t.ncnt + X);
    unsigned long long nbad = 0;
    for (int side = 0; side < 2; ++side) {
        int c = side == 0 ? r.left() : r.right();
        int slots = side == 0 ? cc.x : cc.z, del = side == 0 ? cc.y : cc.w;
        Box3 stored = r.box(side);
        if (X == 0 && side == 1) {
            if (c != 0) {
                ++nbad;
                note_bad(t.st, 101, X, side, c, 0, 0, 0);
            }
            continue;
        }
        if (c == 0) {
            if (X != 0) {  // only an empty tree has no root
                ++nbad;
                note_bad(t.st, 102, X, side, 0, 0, 0, 0);
            }
            continue;
        }
        Box3 b = empty_box();
        int s2 = 0, d2 = 0;
        if (c > 0) {
            if (c >= t.st->node_top || t.nparent[c] != X * 2 + side) {
                ++nbad;
                note_bad(t.st, 103, X, side, c, c < t.st->node_top ? t.nparent[c] : -9, 0, 0);
                continue;
            }
            NodeRec rc = load_node_cg(t.node, c);
            int4 c4 = __ldcg(t.ncnt + c);
            Box3 bl = rc.box(0), br = rc.box(1);
            if (!box_empty(bl)) box_union(b, bl);
            if (!box_empty(br)) box_union(b, br);
            s2 = c4.x + c4.z;
            d2 = c4.y + c4.w;
        } else {
            int L = code_leaf(c);
            if (L >= t.st->leaf_top || t.lparent[L] != X * 2 + side) {
                ++nbad;
                note_bad(t.st, 104, X, side, c, L < t.st->leaf_top ? t.lparent[L] : -9, 0, 0);
                continue;
            }
            int n = t.leaf_n[L];
            // Between a refit and its rebuild jobs a leaf may hold more
            // points than slots (its overflow is queued for the rebuild).
            if ((n > LEAF_CAP && at_rest) || n < 0) {
                ++nbad;
                note_bad(t.st, 105, X, side, c, n, 0, 0);
                continue;
            }
            s2 = n;
            const int m = n < LEAF_CAP ? n : LEAF_CAP;
            for (int j = 0; j < m; ++j) {
                float4 p = __ldcg(t.pts + (long long)L * LEAF_CAP + j);
                if (__float_as_uint(p.w) & F_DEL)
                    ++d2;
                else
                    box_grow(b, p.x, p.y, p.z);
            }
        }
        // the wide records: the child's own place, and its slot if it has one
        const int2 wi = t.winfo[X];
        const int pos = wi.y * 2 + side;
        if (c > 0) {
            const int2 wc = t.winfo[c], want = wide_below(wi, side, c);
            if (wc.x != want.x || wc.y != want.y) {
                ++nbad;
                note_bad(t.st, 112, X, side, c, wc.x, wc.y, want.y);
            }
        }
        if (pos >= WIDE || c < 0) {
            const float* f = reinterpret_cast<const float*>(t.wide + (long long)wi.x * 16);
            const int s0 = wide_slot(pos);
            Box3 wb;
            for (int a = 0; a < 3; ++a) {
                wb.lo[a] = f[wide_at(s0, a)];
                wb.hi[a] = f[wide_at(s0, 3 + a)];
            }
            bool empty_rest = true;
            for (int s = 1; pos < WIDE && s < (8 >> (31 - __clz(pos))); ++s)
                empty_rest = empty_rest && __float_as_int(f[wide_at(s0 + s, 6)]) == 0 &&
                             !(f[wide_at(s0 + s, 0)] <= f[wide_at(s0 + s, 3)]);
            const int wc = __float_as_int(f[wide_at(s0, 6)]), wv = __float_as_int(f[wide_at(s0, 7)]);
            if (wc != c || wv != slots - del || !same_box(wb, stored) || !empty_rest) {
                ++nbad;
                note_bad(t.st, 113, X, side, c, wc, wv, slots - del);
            }
        }
        if (s2 != slots || d2 != del) {
            ++nbad;
            note_bad(t.st, 106, X, side, slots, s2, del, d2);
        } else if (!same_box(b, stored)) {
            ++nbad;
            int k = 0;
            while (k < 3 && __float_as_uint(b.lo[k]) == __float_as_uint(stored.lo[k]) &&
                   __float_as_uint(b.hi[k]) == __float_as_uint(stored.hi[k]))
                ++k;
            note_bad(t.st, 107, X, side, c, k, __float_as_int(k < 3 ? b.lo[k] : 0.f),
                     __float_as_int(k < 3 ? stored.lo[k] : 0.f));
        }
    }
    if (nbad) atomicAdd(bad, nbad);
}

// Every live leaf is the child its parent record names.
__global__ void validate_leaves_kernel(DevTree t, unsigned long long* bad) {
    int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= t.st->leaf_top) return;
    int lp = t.lparent[L];
    if (lp < 0) return;
    int P = lp >> 1;
    bool ok = P < t.st->node_top && (P == 0 || t.nparent[P] >= 0);
    if (ok) {
        const int* codes = reinterpret_cast<const int*>(t.node + 4 * P + 3);
        ok = codes[lp & 1] == leaf_code(L);
    }
    if (!ok) {
        atomicAdd(bad, 1ull);
        note_bad(t.st, 108, P, lp & 1, L, lp, 0, 0);
    }
}

// Refit / rebuild bookkeeping that must be clear between refits (arrival
// counters) or between calls (violation and job tags, dirty flags).
__global__ void validate_aux_nodes_kernel(DevTree t, UpdateAux a, bool at_rest, unsigned long long* bad) {
    int X = blockIdx.x * blockDim.x + threadIdx.x;
    if (X >= t.node_cap) return;
    const uint4* m = a.mail + 4 * (size_t)X;
    if (a.pend[X] != 0 || a.arrive[X] != 0 || (m[0].w | m[1].w | m[2].w | m[3].w) != 0) {
        atomicAdd(bad, 1ull);
        note_bad(t.st, 109, X, a.pend[X], a.arrive[X], X < t.st->node_top ? t.nparent[X] : -9, 0, 0);
    }
    if (at_rest && (a.viol_flag[X] != 0 || a.job_of_node[X] != -1)) {
        atomicAdd(bad, 1ull);
        note_bad(t.st, 110, X, a.viol_flag[X], a.job_of_node[X], 0, 0, 0);
    }
}

__global__ void validate_aux_leaves_kernel(DevTree t, UpdateAux a, bool at_rest, unsigned long long* bad) {
    int L = blockIdx.x * blockDim.x + threadIdx.x;
    if (L >= t.leaf_cap) return;
    if (a.dirty_flag[L] != 0 || (a.job_of_leaf[L] != -1 && (at_rest || a.job_of_leaf[L] != LEAF_VIOL))) {
        atomicAdd(bad, 1ull);
        note_bad(t.st, 111, L, a.dirty_flag[L], a.job_of_leaf[L], L < t.st->leaf_top ? t.lparent[L] : -9, 0, 0);
    }
}

__global__ void set_ll_kernel(long long* p, long long v) { chain_begin(); *p = v; }

// Empties the top wide record and places the root at position `pos` in it.
__global__ void set_top_kernel(DevTree t, int pos) {
    if (threadIdx.x == 0) t.winfo[0] = make_int2(0, pos / 2);
    wide_store(t.wide, 0, threadIdx.x, empty_box(), 0, 0);
}

__global__ void snapshot_root_kernel(DevTree t) {
    chain_begin();
    finish_alloc(t.st);
    snapshot_root(t);
}

// ---- voxel downsampling ------------------------------------------------------------
//
// Sequential semantics (Add_Points with downsample_on, ikd_Tree.cpp:422-449),
// for new point p_i in order: box = the voxel of p_i, with
// lo = floor(x / ds) * ds and hi = lo + ds in float, centre = lo + (hi - lo) / 2
// in double rounded to float; S = valid points in the half-open box; the
// winner is p_i unless a point of S is strictly closer to the centre; if
// |S| > 1 or the winner is p_i (within EPSS), S is deleted (downsample flag)
// and the winner is inserted as a new point.
//
// Parallel form: points are grouped by voxel.  A voxel's outcome depends only
// on its own S and its own new points, taken in input order, as long as no
// point lies in two voxel boxes or outside its own (float rounding can make the
// boxes of neighbouring voxels overlap or leave gaps by one ulp).  Such points
// are detected and processed alone, in input order, which keeps the result
// identical to the sequential loop.  Among points of S at the same distance
// the smaller id wins (the reference takes the first in traversal order).  A
// winner that was already in the map is re-inserted under its own id; a new
// point i of the batch gets id first_id + i.

// Bits of the voxel hash the grouper sorts by (and compares: entries of one
// hash run are the sorted neighbours with equal masked hash): three sort passes, or two where the points are so few that
// two voxels rarely share one of 65,536 values (a run with several voxels costs its
// readers a comparison per member).  14,400 points: the sort 36 -> 24 us.
constexpr long long DS_SHORT_HASH = 32768;
inline int ds_hash_bits(long long n) { return n <= DS_SHORT_HASH ? 16 : 24; }
// Hash runs longer than this go to ds_fold_big_kernel (a warp per group,
// DS_BIG_BLOCKS blocks of four warps walking the deferred list).
constexpr int DS_BIG_RUN = 16;
constexpr int DS_BIG_BLOCKS = 152;
// Blocks of the deletion by pairs (their number is only on the device).
constexpr int SPEC_BLOCKS = 152;

__device__ __forceinline__ uint32_t mix32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

__device__ __forceinline__ void voxel_axis(float c, float ds, float& f, float& lo, float& hi, float& mid) {
    f = floorf(__fdiv_rn(c, ds));
    lo = __fmul_rn(f, ds);
    hi = __fadd_rn(lo, ds);
    mid = __double2float_rn(__dadd_rn((double)lo, __dmul_rn((double)__fsub_rn(hi, lo), 0.5)));
}

// Is coordinate c inside the box range of voxel index f + df on this axis?
__device__ __forceinline__ bool in_voxel_range(float c, float f, float df, float ds) {
    float lo = __fmul_rn(__fadd_rn(f, df), ds);
    float hi = __fadd_rn(lo, ds);
    return lo <= c && c < hi;
}

__global__ void ds_prepare_kernel(DevTree t, const float* __restrict__ in, int stride, long long n, float ds,
                                  int hash_bits, DsScratch d) {
    chain_begin();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) t.st->count = n;  // end of the first sub-batch, until a point cuts it
    if (i >= n) return;
    float c[3] = {in[i * stride], in[i * stride + 1], in[i * stride + 2]};
    if (!(isfinite(c[0]) && isfinite(c[1]) && isfinite(c[2]))) atomicOr(&t.st->err, ERR_INPUT);
    float f[3], lo[3], hi[3], mid[3];
    bool clean = true;
    for (int a = 0; a < 3; ++a) {
        voxel_axis(c[a], ds, f[a], lo[a], hi[a], mid[a]);
        clean = clean && lo[a] <= c[a] && c[a] < hi[a];
        if (!(fabsf(f[a]) < 8388608.0f)) clean = false;  // f +- 1 must stay exact
    }
    if (clean)
        for (int a = 0; a < 3; ++a)
            if (in_voxel_range(c[a], f[a], -1.f, ds) || in_voxel_range(c[a], f[a], 1.f, ds)) clean = false;
    d.pts[i] = make_float4(c[0], c[1], c[2], 0.f);
    d.box_lo[i] = make_float4(lo[0], lo[1], lo[2], f[0]);
    d.box_hi[i] = make_float4(hi[0], hi[1], hi[2], f[1]);
    d.mid[i] = make_float4(mid[0], mid[1], mid[2], f[2]);
    // Grouping key: the voxel's float indices (bit patterns), exact.
    // -0.0 and +0.0 give the same box; adding +0.0 maps both to +0.0.
    int kb[3];
    for (int a = 0; a < 3; ++a) kb[a] = __float_as_int(__fadd_rn(f[a], 0.0f));
    d.key[i] = make_int4(kb[0], kb[1], kb[2], clean ? 1 : 0);
    // The bit patterns of integral floats end in long runs of zeros: each
    // component goes through the full mixer (a product of them kept only
    // ~16 bits and put up to 7 voxels on one hash).
    uint32_t h = mix32((uint32_t)kb[2] ^ 0x9e3779b9u);
    h = mix32(h ^ (uint32_t)kb[1]);
    d.hkey[0][i] = mix32(h ^ (uint32_t)kb[0]) & ((1u << hash_bits) - 1u);
    d.hval[0][i] = (uint32_t)i;
}

__device__ __forceinline__ bool same_key(const int4& a, const int4& b) { return a.x == b.x && a.y == b.y && a.z == b.z; }

// Also lays the keys and points out in sorted order (s_key, s_pts), so the
// per-group walks below read consecutive entries instead of gathering through
// hval one dependent load at a time.
__global__ void ds_leaders_kernel(long long n, DsScratch d, DevStatus* st) {
    chain_begin();
    long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    uint32_t h = d.hkey[0][j];
    const uint32_t idx = d.hval[0][j];
    int4 k = d.key[idx];
    const float4 p = d.pts[idx];
    d.s_key[j] = k;
    d.s_pts[j] = make_float4(p.x, p.y, p.z, __int_as_float((int)idx));
    for (long long jj = j - 1; jj >= 0 && d.hkey[0][jj] == h; --jj)
        if (same_key(d.key[d.hval[0][jj]], k)) return;
    int g = atomicAdd(&st->n_groups, 1);
    d.groups[g] = (int)j;
}

// Entries of the hash run starting at sorted position j, four per step
// (independent loads); f(jj, key, point) sees them in sorted order, which
// within one voxel is input order, and returns false to stop.
template <class F>
__device__ __forceinline__ void for_run(const DsScratch& d, long long n, long long j, uint32_t h, F f) {
    for (long long base = j; base < n; base += 4) {
        uint32_t hh[4];
        int4 kk[4];
        float4 pp[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const long long jj = base + u;
            hh[u] = jj < n ? __ldcg(d.hkey[0] + jj) : ~h;
            kk[u] = jj < n ? __ldcg(d.s_key + jj) : make_int4(0, 0, 0, 0);
            pp[u] = jj < n ? __ldcg(d.s_pts + jj) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (hh[u] != h) return;
            if (!f(base + u, kk[u], pp[u])) return;
        }
    }
}

// First member index >= a of group g (members are in increasing index order).
__device__ __forceinline__ long long group_first_from(const DsScratch& d, long long n, int j, long long a) {
    const uint32_t h = __ldcg(d.hkey[0] + j);
    const int4 k = __ldcg(d.s_key + j);
    long long r = -1;
    for_run(d, n, j, h, [&](long long, const int4& kk, const float4& p) {
        if (!same_key(kk, k)) return true;
        const long long idx = __float_as_int(p.w);
        if (idx >= a) {
            r = idx;
            return false;
        }
        return true;
    });
    return r;
}

__global__ void ds_h1_kernel(long long n, long long a, DsScratch d, DevStatus* st) {
    chain_begin();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *d.n_pairs = 0;  // ds_search_kernel lists its pairs afresh
        st->n_ins = 0;   // and the fold its winners
    }
    long long i = a + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (d.key[i].w) return;
    long long cut = i > a ? i : a + 1;
    atomicMin((long long*)&st->count, cut);
}

__device__ __forceinline__ Box3 group_box(const DsScratch& d, int lead) {
    const float4 blo = d.box_lo[lead], bhi = d.box_hi[lead];
    Box3 qb;
    qb.lo[0] = blo.x; qb.lo[1] = blo.y; qb.lo[2] = blo.z;
    qb.hi[0] = bhi.x; qb.hi[1] = bhi.y; qb.hi[2] = bhi.z;
    return qb;
}

// A child's box against a half-open query box (qbox_disjoint).
__device__ __forceinline__ bool half_open_overlap(const Box3& q, const float* lo, const float* hi) {
    return q.hi[0] > lo[0] && q.lo[0] <= hi[0] && q.hi[1] > lo[1] && q.lo[1] <= hi[1] && q.hi[2] > lo[2] &&
           q.lo[2] <= hi[2];
}

// Per voxel group: S = the valid stored points in the voxel's box, |S|, the
// point of S closest to the voxel centre (smaller id on ties), and whether a
// point of S also lies in a neighbouring voxel's box range on some axis (a
// float-rounding sliver: the group is then folded alone).
// One team per group; bound by the chain of its walk and, before, by one atomic on
// the pair counter per bucket with hits: now one per warp and step.  14,400-point
// scan, 9,000 groups, 500,000 stored points: 65 us with a thread per group on the
// binary nodes, 21 now.
__global__ void __launch_bounds__(TEAM_CTA) ds_search_kernel(DevTree t, long long n, long long a, DsScratch d, float ds) {
    chain_begin();
    extern __shared__ int stacks[];
    constexpr unsigned ALL = 0xffffffffu;
    const int g = (blockIdx.x * TEAM_CTA + threadIdx.x) / TEAM;
    const int lane = threadIdx.x & 31, sub = lane & (TEAM - 1);
    if (blockIdx.x == 0 && threadIdx.x == 0) *d.n_big = 0;  // ds_fold_kernel lists its deferred groups afresh
    bool active = g < t.st->n_groups && !(t.st->err & ERR_INPUT);  // a non-finite input: the call changes nothing
    long long first = -1;
    int lead = 0;
    if (active) {
        const int j = d.groups[g];
        first = group_first_from(d, n, j, a);
        if (first < 0) {
            if (sub == 0) d.g_info[g] = make_int4(0, -1, 0, 0);
            active = false;
        } else {
            lead = d.hval[0][j];
        }
    }
    const Box3 qb = active ? group_box(d, lead) : empty_box();
    const float4 mid = active ? d.mid[lead] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float fk[3] = {active ? d.box_lo[lead].w : 0.f, active ? d.box_hi[lead].w : 0.f, mid.w};
    int n0 = 0, best_slot = -1, best_id = 0x7fffffff;
    float best_d = __int_as_float(0x7f800000);
    float4 best_p = make_float4(0.f, 0.f, 0.f, 0.f);
    bool hazard = false;
    team_walk(
        t, active, stacks, [&](const float* lo, const float* hi) { return half_open_overlap(qb, lo, hi); },
        [&](int L, int half, int cnt, const float4* p, bool on) {
            const int s0 = 16 * half + 4 * sub;
            unsigned m = 0;
            if (on) {
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (s0 + u < cnt && !(__float_as_uint(p[u].w) & F_DEL) && qbox_holds(qb, p[u].x, p[u].y, p[u].z))
                        m |= 1u << u;
            }
            if (!__any_sync(ALL, m != 0)) return false;
            // the pairs (voxel, slot) of the hits, for ds_delete_pairs_kernel
            int inc = __popc(m);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(ALL, inc, o);
                if (lane >= o) inc += y;
            }
            int base = 0;
            if (lane == 31) base = atomicAdd(d.n_pairs, inc);
            int pos = __shfl_sync(ALL, base, 31) + inc - __popc(m);
            n0 += __popc(m);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                if (!(m >> u & 1)) continue;
                if (pos < d.pair_cap) d.pairs[pos] = make_int2(g, L * LEAF_CAP + s0 + u);
                ++pos;
                const float pc[3] = {p[u].x, p[u].y, p[u].z};
#pragma unroll
                for (int k = 0; k < 3; ++k)
                    hazard = hazard || in_voxel_range(pc[k], fk[k], -1.f, ds) || in_voxel_range(pc[k], fk[k], 1.f, ds);
                const float dd = sq_dist(p[u].x, p[u].y, p[u].z, mid.x, mid.y, mid.z);
                const int id = (int)(__float_as_uint(p[u].w) & ID_MASK);
                if (dd < best_d || (dd == best_d && id < best_id)) {
                    best_d = dd;
                    best_id = id;
                    best_slot = L * LEAF_CAP + s0 + u;
                    best_p = make_float4(p[u].x, p[u].y, p[u].z, 0.f);
                }
            }
            return false;
        });
    // the four lanes' results into the first (distances are >= 0: their bit
    // patterns order like the values; ids are unique)
    int all = n0;
    unsigned dmin = __float_as_uint(best_d);
    hazard = (__ballot_sync(ALL, hazard) >> (lane & ~(TEAM - 1)) & 15u) != 0;
#pragma unroll
    for (int o = 1; o < TEAM; o <<= 1) {
        all += __shfl_xor_sync(ALL, all, o);
        dmin = min(dmin, __shfl_xor_sync(ALL, dmin, o));
    }
    int imin = __float_as_uint(best_d) == dmin ? best_id : 0x7fffffff;
#pragma unroll
    for (int o = 1; o < TEAM; o <<= 1) imin = min(imin, __shfl_xor_sync(ALL, imin, o));
    if (!active) return;
    if (all == 0) {
        if (sub != 0) return;
        d.g_info[g] = make_int4(0, -1, 0x7fffffff, 0);
        d.g_best[g] = make_float4(0.f, 0.f, 0.f, best_d);
    } else if (best_slot >= 0 && __float_as_uint(best_d) == dmin && best_id == imin) {
        d.g_info[g] = make_int4(all, best_slot, best_id, hazard ? 1 : 0);
        d.g_best[g] = make_float4(best_p.x, best_p.y, best_p.z, best_d);
    }
    if (hazard && sub == 0) {
        long long cut = first > a ? first : a + 1;
        atomicMin((long long*)&t.st->count, cut);
    }
}

__global__ void __launch_bounds__(128) ds_fold_kernel(DevTree t, long long n, long long a, long long first_id,
                                                      DsScratch d) {
    chain_begin();
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31, n_groups = t.st->n_groups, all = gridDim.x * blockDim.x;
    // Groups are dealt out over the warps before the lanes (first_item): their runs
    // differ in length and the lanes of a warp wait for the longest.  14,400 points:
    // 25 us with full warps and runs of up to 64 entries, 14 + 6 (ds_fold_big_kernel)
    // with up to 16.
    for (int g0 = first_item() - lane * (all >> 5); g0 < n_groups; g0 += all) {
        const int g = g0 + lane * (all >> 5);
        bool have_ins = false;
        float cx = 0.f, cy = 0.f, cz = 0.f, cd = 0.f;
        long long cid = -1;  // id of the current winner c: a stored point keeps its id
        int triggers = 0;
        // (a non-finite input: the call changes nothing)
        if (g < n_groups && !(t.st->err & ERR_INPUT)) [&] {
            // the sub-batch ends where ds_h1_kernel found the first point that must
            // be folded alone (st->count), and holds at least one point
            const long long e = min(max((long long)t.st->count, a + 1), n);
            int j = d.groups[g];
            int4 info = d.g_info[g];
            d.g_out[g] = make_int4(0, 0, 0, 0);
            const uint32_t h = __ldcg(d.hkey[0] + j);
            if (j + DS_BIG_RUN < n && __ldcg(d.hkey[0] + j + DS_BIG_RUN) == h) {
                // a long hash run (a voxel with many points): folded by a warp
                d.big[atomicAdd(d.n_big, 1)] = g;
                return;
            }
            if (info.y == -1 && info.x == 0 && group_first_from(d, n, j, a) < 0) return;
            const int lead = d.hval[0][j];
            const int4 k = __ldcg(d.s_key + j);
            float4 mid = d.mid[lead];
            float4 best = d.g_best[g];
            const int n0 = info.x;
            bool s_is_s0 = true, del_s0 = false;
            for_run(d, n, j, h, [&](long long, const int4& kk, const float4& p) {
                if (!same_key(kk, k)) return true;
                const long long idx = __float_as_int(p.w);
                if (idx < a) return true;
                if (idx >= e) return false;  // members come in increasing index order
                float pd = sq_dist(p.x, p.y, p.z, mid.x, mid.y, mid.z);
                float wx = p.x, wy = p.y, wz = p.z, wd = pd;
                long long wid = first_id + idx;
                bool trig;
                if (s_is_s0) {
                    if (n0 > 0 && best.w < pd) {
                        wx = best.x; wy = best.y; wz = best.z; wd = best.w;
                        wid = info.z;
                    }
                    trig = n0 > 1 || same_point(p.x, p.y, p.z, wx, wy, wz);
                    if (trig) {
                        del_s0 = n0 > 0;
                        s_is_s0 = false;
                    }
                } else {
                    if (cd < pd) {
                        wx = cx; wy = cy; wz = cz; wd = cd;
                        wid = cid;
                    }
                    trig = same_point(p.x, p.y, p.z, wx, wy, wz);
                }
                if (trig) {
                    ++triggers;
                    cx = wx; cy = wy; cz = wz; cd = wd;
                    cid = wid;
                    have_ins = true;
                }
                return true;
            });
            d.g_out[g] = make_int4(del_s0 ? 1 : 0, have_ins ? 1 : 0, triggers, 0);
        }();
        // one addition per warp to each counter
        const int trig = __reduce_add_sync(ALL, triggers);
        if (lane == 0 && trig) atomicAdd((unsigned long long*)&t.st->count2, (unsigned long long)trig);
        if (have_ins && cid > MAX_ID) {
            atomicOr(&t.st->err, ERR_ID);
            have_ins = false;
        }
        const unsigned ins = __ballot_sync(ALL, have_ins);
        int q = 0;
        if (lane == 0 && ins) q = atomicAdd(&t.st->n_ins, __popc(ins));
        q = __shfl_sync(ALL, q, 0) + __popc(ins & ((1u << lane) - 1u));
        if (have_ins) d.ins[q] = make_float4(cx, cy, cz, __int_as_float((int)cid));
    }
}

// The fold of ds_fold_kernel for the groups it deferred, one warp per group,
// 32 members per step.  After the first member the fold's state is the
// current winner c, and a member p replaces c exactly when d(p) <= d(c) (a
// later point wins ties): c after member i is the minimum of the members so
// far and the initial c (the best stored point of the voxel when it has one)
// under (distance ascending, position descending), a warp prefix minimum.
// Member i triggers (the voxel's points are replaced) when it replaces c,
// when it coincides with c (same_point), or, for a voxel holding more than
// one stored point, when it is the first member.  The point inserted is the
// final c under its own id (the stored point's, or first_id + its index).
__global__ void __launch_bounds__(128) ds_fold_big_kernel(DevTree t, long long n, long long a, long long first_id,
                                                          DsScratch d) {
    chain_begin();
    const int lane = threadIdx.x & 31;
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    if (t.st->err & ERR_INPUT) return;
    const long long e = min(max((long long)t.st->count, a + 1), n);
    const int nb = *d.n_big;
    for (int b = warp; b < nb; b += nwarps) {
        const int g = d.big[b];
        const int j = d.groups[g];
        const int4 info = d.g_info[g];
        const float4 best = d.g_best[g];
        const uint32_t h = __ldcg(d.hkey[0] + j);
        const int4 k = __ldcg(d.s_key + j);
        const float4 mid = d.mid[d.hval[0][j]];
        const int n0 = info.x;
        // running c: distance, position in the run (-2: the stored best,
        // -1: none), coordinates
        float cdist = n0 > 0 ? best.w : __int_as_float(0x7f800000);
        long long cpos = n0 > 0 ? -2 : -1;
        float cx = best.x, cy = best.y, cz = best.z;
        long long cid = n0 > 0 ? (long long)info.z : -1;
        bool first_open = n0 > 1;  // the first member triggers regardless
        int triggers = 0;
        bool more = true;
        for (long long base = j; more && base < n; base += 32) {
            const long long jj = base + lane;
            const uint32_t hh = jj < n ? __ldcg(d.hkey[0] + jj) : ~h;
            const unsigned off_run = __ballot_sync(0xffffffffu, hh != h);
            // entries from the first one of another hash on are not in the run
            const int run_end = off_run ? __ffs(off_run) - 1 : 32;
            bool member = false;
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
            long long idx = -1;
            if (lane < run_end) {
                const int4 kk = __ldcg(d.s_key + jj);
                if (same_key(kk, k)) {
                    p = __ldcg(d.s_pts + jj);
                    idx = __float_as_int(p.w);
                    member = idx >= a && idx < e;
                }
            }
            // members come in increasing index order: one at or past e ends the group
            const unsigned past = __ballot_sync(0xffffffffu, idx >= e);
            const int lim = past ? __ffs(past) - 1 : run_end;
            member = member && lane < lim;
            if (off_run || past) more = false;
            const float pd = member ? sq_dist(p.x, p.y, p.z, mid.x, mid.y, mid.z) : __int_as_float(0x7f800000);
            // inclusive prefix minimum over this step's members
            float md = pd;
            int mlane = member ? lane : -1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float od = __shfl_up_sync(0xffffffffu, md, o);
                const int ol = __shfl_up_sync(0xffffffffu, mlane, o);
                // (od, ol) is earlier: it stays the minimum only if strictly smaller
                if (lane >= o && ol >= 0 && (mlane < 0 || od < md)) {
                    md = od;
                    mlane = ol;
                }
            }
            // exclusive prefix: the inclusive one of the lane before, then the carry
            float ed = __shfl_up_sync(0xffffffffu, md, 1);
            int el = __shfl_up_sync(0xffffffffu, mlane, 1);
            if (lane == 0) el = -1;
            // c before this member: the carry unless a member of this step beat it
            const bool from_step = el >= 0 && ed <= cdist;
            const float prev_d = from_step ? ed : cdist;
            const int src = from_step ? el : lane;
            const float sx = __shfl_sync(0xffffffffu, p.x, src), sy = __shfl_sync(0xffffffffu, p.y, src),
                        sz = __shfl_sync(0xffffffffu, p.z, src);
            const float prev_x = from_step ? sx : cx, prev_y = from_step ? sy : cy, prev_z = from_step ? sz : cz;
            const bool prev_none = !from_step && cpos == -1;
            const unsigned mem = __ballot_sync(0xffffffffu, member);
            const bool is_first = first_open && mem != 0 && lane == __ffs(mem) - 1;
            const bool replaces = member && pd <= prev_d;
            const bool trig = member && (replaces || is_first ||
                                         (!prev_none && same_point(p.x, p.y, p.z, prev_x, prev_y, prev_z)));
            triggers += __popc(__ballot_sync(0xffffffffu, trig));
            if (mem) first_open = false;
            // carry: the step's minimum over everything, if it beats c
            const float sd = __shfl_sync(0xffffffffu, md, 31);
            const int sl = __shfl_sync(0xffffffffu, mlane, 31);
            if (sl >= 0 && sd <= cdist) {
                cdist = sd;
                cpos = base + sl;
                cx = __shfl_sync(0xffffffffu, p.x, sl);
                cy = __shfl_sync(0xffffffffu, p.y, sl);
                cz = __shfl_sync(0xffffffffu, p.z, sl);
                cid = first_id + __shfl_sync(0xffffffffu, idx, sl);
            }
        }
        if (lane != 0) continue;
        const bool have_ins = triggers > 0;
        d.g_out[g] = make_int4(have_ins && n0 > 0 ? 1 : 0, have_ins ? 1 : 0, triggers, 0);
        if (!have_ins) continue;
        atomicAdd((unsigned long long*)&t.st->count2, (unsigned long long)triggers);
        if (cid > MAX_ID) {
            atomicOr(&t.st->err, ERR_ID);
            continue;
        }
        const int q = atomicAdd(&t.st->n_ins, 1);
        d.ins[q] = make_float4(cx, cy, cz, __int_as_float((int)cid));
    }
}

// Deletes (with the downsample flag) the stored points ds_search_kernel found
// in the boxes of the groups whose fold decided so: one thread per listed
// (group, slot) pair, no tree walk (nothing moved since the search).
__global__ void ds_delete_pairs_kernel(DevTree t, UpdateAux a, DsScratch d) {
    chain_begin();
    const int np = *d.n_pairs;
    if (np > d.pair_cap || (t.st->err & ERR_INPUT)) return;  // the list overflowed: ds_delete_kernel walks
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < np; i += gridDim.x * blockDim.x) {
        const int2 pr = d.pairs[i];
        if (!d.g_out[pr.x].x) continue;
        float* w = &t.pts[pr.y].w;
        *w = __uint_as_float(__float_as_uint(*w) | F_DEL | F_DSDEL);
        mark_dirty(a, t.st, pr.y / LEAF_CAP);
    }
}

// The same deletion by walking the tree from every voxel box, when the pair
// list overflowed.
__global__ void __launch_bounds__(TEAM_CTA) ds_delete_kernel(DevTree t, UpdateAux a, DsScratch d) {
    chain_begin();
    extern __shared__ int stacks[];
    if (*d.n_pairs <= d.pair_cap) return;  // ds_delete_pairs_kernel did it
    const int g = (blockIdx.x * TEAM_CTA + threadIdx.x) / TEAM;
    const int sub = threadIdx.x & (TEAM - 1);
    const bool active = g < t.st->n_groups && !(t.st->err & ERR_INPUT) && d.g_out[g].x;
    const Box3 qb = active ? group_box(d, d.hval[0][d.groups[g]]) : empty_box();
    team_walk(
        t, active, stacks, [&](const float* lo, const float* hi) { return half_open_overlap(qb, lo, hi); },
        [&](int L, int half, int cnt, const float4* p, bool on) {
            const int s0 = 16 * half + 4 * sub;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t w = __float_as_uint(p[u].w);
                if (!on || s0 + u >= cnt || (w & F_DEL) || !qbox_holds(qb, p[u].x, p[u].y, p[u].z)) continue;
                t.pts[(long long)L * LEAF_CAP + s0 + u].w = __uint_as_float(w | F_DEL | F_DSDEL);
                mark_dirty(a, t.st, L);
            }
            return false;
        });
}

__global__ void pack_points_kernel(DevTree t, const float* __restrict__ in, int stride, long long n, long long first_id,
                                   float4* __restrict__ out) {
    chain_begin();
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x = in[i * stride], y = in[i * stride + 1], z = in[i * stride + 2];
    if (!(isfinite(x) && isfinite(y) && isfinite(z))) atomicOr(&t.st->err, ERR_INPUT);
    long long id = first_id + i;
    if (id > MAX_ID) atomicOr(&t.st->err, ERR_ID);
    out[i] = make_float4(x, y, z, __int_as_float((int)(id & ID_MASK)));
}

// The same for tightly packed, 16-byte aligned input: a block's points come in as
// consecutive 16-byte words (the input may be host memory over the chip link).
constexpr int PACK_POINTS = 1024;
__global__ void __launch_bounds__(256) pack_dense_kernel(DevTree t, const float4* __restrict__ in, long long n,
                                                         long long first_id, float4* __restrict__ out) {
    chain_begin();
    __shared__ float4 w[PACK_POINTS * 3 / 4];
    const long long p0 = (long long)blockIdx.x * PACK_POINTS;
    const int m = (int)min((long long)PACK_POINTS, n - p0);
    const int words = m * 3 / 4;  // whole 16-byte words
    const float4* src = in + p0 * 3 / 4;
    float4 v[3];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        if (r * 256 + (int)threadIdx.x < words) v[r] = src[r * 256 + threadIdx.x];
#pragma unroll
    for (int r = 0; r < 3; ++r)
        if (r * 256 + (int)threadIdx.x < words) w[r * 256 + threadIdx.x] = v[r];
    float* f = reinterpret_cast<float*>(w);
    if ((int)threadIdx.x < m * 3 - words * 4) f[words * 4 + threadIdx.x] = reinterpret_cast<const float*>(src)[words * 4 + threadIdx.x];
    __syncthreads();
    bool bad = false;
#pragma unroll
    for (int r = 0; r < PACK_POINTS / 256; ++r) {
        const int i = r * 256 + threadIdx.x;
        if (i >= m) break;
        const float x = f[3 * i], y = f[3 * i + 1], z = f[3 * i + 2];
        bad = bad || !(isfinite(x) && isfinite(y) && isfinite(z));
        const long long id = first_id + p0 + i;
        if (id > MAX_ID) atomicOr(&t.st->err, ERR_ID);
        out[p0 + i] = make_float4(x, y, z, __int_as_float((int)(id & ID_MASK)));
    }
    if (bad) atomicOr(&t.st->err, ERR_INPUT);
}

inline size_t au(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace

void launch_route_append(const DevTree& t, const UpdateAux& a, const float4* pts, long long n, int4* ovf_leaf,
                         float4* ovf_pts, cudaStream_t s) {
    if (n <= 0) return;
    launch_chain(route_append_kernel, blocks_for(n, 256), 256, 0, s, t, a, pts, n, nullptr, ovf_leaf, ovf_pts);
}

void launch_route_append_dev_count(const DevTree& t, const UpdateAux& a, const float4* pts, long long n_bound,
                                   const int* n_dev, int4* ovf_leaf, float4* ovf_pts, cudaStream_t s) {
    if (n_bound <= 0) return;
    launch_chain(route_append_kernel, blocks_for(n_bound, 256), 256, 0, s, t, a, pts, n_bound, n_dev, ovf_leaf, ovf_pts);
}

void launch_refit(const DevTree& t, const UpdateAux& a, const int* items, const int* n_items, int max_items,
                  const Criteria& c, cudaStream_t s) {
    if (max_items <= 0) return;
    // (the number of items is on the device, the bound often far above it: the
    // grids end at what the device holds at once)
    launch_chain(refit_mark_kernel, std::min(blocks_for(max_items, 128), 152u * 8u), 128, 0, s, t, a, items, n_items);
    launch_chain(refit_compute_kernel, std::min(blocks_for(max_items, 128), 152u * 8u), 128, 0, s, t, a, items, n_items, c);
}


cudaError_t launch_settle(const DevTree& t, const UpdateAux& a, bool select, DevStatus* host, bool list, int blocks,
                          cudaStream_t s) {
    DevTree tt = t;
    UpdateAux aa = a;
    void* args[] = {&tt, &aa, &select, &host};
    return cudaLaunchCooperativeKernel(list ? (const void*)settle_kernel<true> : (const void*)settle_kernel<false>,
                                       dim3(blocks), dim3(list ? LIST_THREADS : SETTLE_THREADS), args, 0, s);
}

void launch_job_gather(const DevTree& t, const UpdateAux& a, int n_queue, int leaf_top, int node_top,
                       const int4* ovf_leaf, const float4* ovf_pts, int max_ovf, float4* out, float4* removed,
                       long long removed_cap, cudaStream_t s) {
    const long long n = (n_queue >= 0 ? (long long)n_queue : (long long)leaf_top + node_top) + max_ovf;
    if (n > 0)
        launch_chain(job_gather_kernel, blocks_for(n, 256), 256, 0, s, t, a, n_queue, leaf_top, node_top, ovf_leaf,
                     ovf_pts, max_ovf, out, removed, removed_cap);
}

void launch_job_finish(const DevTree& t, const UpdateAux& a, cudaStream_t s) {
    launch_chain(job_finish_kernel, 1, 1024, 0, s, t, a);
}

void launch_delete_boxes(const DevTree& t, const UpdateAux& a, const float* boxes, long long m, int top_bits,
                         uint32_t flags, long long* total, int2* spill, int spill_cap, cudaStream_t s) {
    if (m <= 0) return;
    // The tree is split below the top until there are units for the whole device
    // (six boxes in 500,000 points: 33 us with units of 128 buckets, 13 with
    // 16); many boxes: not at all.
    int levels = 0, bits = 0;
    while (levels < BD_LEVELS_MAX && bits < t.height && (m << bits) < BD_UNITS) bits += levels++ ? 3 : top_bits;
    const long long blocks = ((m << bits) + BD_CTA / 32 - 1) / (BD_CTA / 32);
    const size_t smem = sizeof(int) * bd_stack_entries(t.height) * (BD_CTA / 32);
    const bool few = (1 << bits) < BD_FEW_UNITS && spill_cap > 0;
    launch_chain(box_delete_kernel, box_grid(blocks), BD_CTA, smem, s, t, a, boxes, m, levels, top_bits, flags, total,
                 false, few ? BD_LIMIT : 0, spill, spill_cap);
    if (few)
        launch_chain(box_delete_kernel, BD_SPILL_BLOCKS, BD_CTA, smem, s, t, a, boxes, m, 0, top_bits, flags, total, true,
                     0, spill, spill_cap);
}

void launch_add_boxes(const DevTree& t, const UpdateAux& a, const float* boxes, long long m, cudaStream_t s) {
    if (m <= 0) return;
    int bits = box_split_bits(m);
    launch_chain(box_restore_kernel, box_grid(m << bits), DB_THREADS, 0, s, t, a, boxes, m, bits);
}

void launch_delete_points(const DevTree& t, const UpdateAux& a, const float* pts, int stride, long long n,
                          cudaStream_t s) {
    if (n <= 0) return;
    launch_chain(delete_points_kernel, blocks_for(n * TEAM, TEAM_CTA), TEAM_CTA, team_stack_bytes(t.height), s, t, a, pts, stride, n);
}

void launch_snapshot_root(const DevTree& t, cudaStream_t s) { launch_chain(snapshot_root_kernel, 1, 1, 0, s, t); }

void launch_set_top(const DevTree& t, int pos, cudaStream_t s) { set_top_kernel<<<1, WIDE, 0, s>>>(t, pos); }

void launch_set_ll(long long* p, long long v, cudaStream_t s) { launch_chain(set_ll_kernel, 1, 1, 0, s, p, v); }

void launch_validate(const DevTree& t, const UpdateAux& a, bool at_rest, long long* bad, cudaStream_t s) {
    if (t.node_cap > 0)
        validate_nodes_kernel<<<blocks_for(t.node_cap, 256), 256, 0, s>>>(t, at_rest, (unsigned long long*)bad);
    if (t.leaf_cap > 0)
        validate_leaves_kernel<<<blocks_for(t.leaf_cap, 256), 256, 0, s>>>(t, (unsigned long long*)bad);
    if (t.node_cap > 0)
        validate_aux_nodes_kernel<<<blocks_for(t.node_cap, 256), 256, 0, s>>>(t, a, at_rest, (unsigned long long*)bad);
    if (t.leaf_cap > 0)
        validate_aux_leaves_kernel<<<blocks_for(t.leaf_cap, 256), 256, 0, s>>>(t, a, at_rest, (unsigned long long*)bad);
}

void launch_flatten(const DevTree& t, float4* out, long long* counter, cudaStream_t s) {
    if (t.leaf_cap <= 0) return;
    flatten_kernel<<<blocks_for(t.leaf_cap, 256), 256, 0, s>>>(t, out, counter);
}

void launch_stored_ids(const DevTree& t, int* out, long long cap, long long* counter, cudaStream_t s) {
    if (t.leaf_cap <= 0) return;
    stored_ids_kernel<<<blocks_for(t.leaf_cap, 256), 256, 0, s>>>(t, out, cap, counter);
}

void launch_select_root(const DevTree& t, const UpdateAux& a, cudaStream_t s) {
    launch_chain(select_root_kernel, 1, 1, 0, s, t, a);
}

void launch_pack_points(const DevTree& t, const float* in, int stride, long long n, long long first_id, float4* out,
                        cudaStream_t s) {
    if (n <= 0) return;
    if (stride == 3 && (reinterpret_cast<uintptr_t>(in) & 15) == 0) {
        launch_chain(pack_dense_kernel, blocks_for(n, PACK_POINTS), 256, 0, s, t, reinterpret_cast<const float4*>(in), n, first_id,
                                                                     out);
        return;
    }
    launch_chain(pack_points_kernel, blocks_for(n, 256), 256, 0, s, t, in, stride, n, first_id, out);
}

size_t ds_scratch_bytes(long long n, long long pair_cap) {
    size_t b = 0;
    b += au(sizeof(int2) * pair_cap) + au(sizeof(int));  // pairs, n_pairs
    b += 5 * au(sizeof(float4) * n);   // pts, box_lo, box_hi, mid, ins
    b += 2 * au(sizeof(int4) * n);     // key, s_key
    b += au(sizeof(float4) * n);       // s_pts
    b += 4 * au(sizeof(uint32_t) * n); // hkey x2, hval x2
    b += au(sizeof(int) * n);          // groups
    b += 2 * au(sizeof(int4) * n);     // g_info, g_out
    b += au(sizeof(float4) * n);       // g_best
    b += au(sizeof(int) * n) + au(sizeof(int));  // big, n_big
    b += au(sort_temp_bytes(n, 1));
    return b;
}

void carve_ds_scratch(void* base, long long n, long long pair_cap, DsScratch* d) {
    char* p = (char*)base;
    auto take = [&](size_t bytes) {
        void* r = p;
        p += (bytes + 255) & ~(size_t)255;
        return r;
    };
    d->pts = (float4*)take(sizeof(float4) * n);
    d->box_lo = (float4*)take(sizeof(float4) * n);
    d->box_hi = (float4*)take(sizeof(float4) * n);
    d->mid = (float4*)take(sizeof(float4) * n);
    d->ins = (float4*)take(sizeof(float4) * n);
    d->key = (int4*)take(sizeof(int4) * n);
    d->s_key = (int4*)take(sizeof(int4) * n);
    d->s_pts = (float4*)take(sizeof(float4) * n);
    d->hkey[0] = (uint32_t*)take(sizeof(uint32_t) * n);
    d->hkey[1] = (uint32_t*)take(sizeof(uint32_t) * n);
    d->hval[0] = (uint32_t*)take(sizeof(uint32_t) * n);
    d->hval[1] = (uint32_t*)take(sizeof(uint32_t) * n);
    d->groups = (int*)take(sizeof(int) * n);
    d->g_info = (int4*)take(sizeof(int4) * n);
    d->g_out = (int4*)take(sizeof(int4) * n);
    d->g_best = (float4*)take(sizeof(float4) * n);
    d->big = (int*)take(sizeof(int) * n);
    d->n_big = (int*)take(sizeof(int));
    d->pairs = (int2*)take(sizeof(int2) * pair_cap);
    d->n_pairs = (int*)take(sizeof(int));
    d->pair_cap = (int)pair_cap;
    d->temp = (void*)p;
}

void launch_ds_prepare(const DevTree& t, const float* in, int stride, long long n, float ds, DsScratch& d,
                       cudaStream_t s) {
    if (n <= 0) return;
    launch_chain(ds_prepare_kernel, blocks_for(n, 256), 256, 0, s, t, in, stride, n, ds, ds_hash_bits(n), d);
    // (the sorted pairs stay where the last pass left them)
    if (radix_sort_pairs(d.hkey[0], d.hval[0], d.hkey[1], d.hval[1], n, 1, n, ds_hash_bits(n), d.temp, s, false, true)) {
        std::swap(d.hkey[0], d.hkey[1]);
        std::swap(d.hval[0], d.hval[1]);
    }
    launch_chain(ds_leaders_kernel, blocks_for(n, 256), 256, 0, s, n, d, t.st);
}

void launch_ds_search(const DevTree& t, long long n, float ds, long long a, DsScratch& d, int max_groups,
                      cudaStream_t s) {
    if (n - a > 0) launch_chain(ds_h1_kernel, blocks_for(n - a, 256), 256, 0, s, n, a, d, t.st);
    if (max_groups > 0)
        launch_chain(ds_search_kernel, blocks_for((long long)max_groups * TEAM, TEAM_CTA), TEAM_CTA, team_stack_bytes(t.height), s, t, n, a, d, ds);
}

void launch_ds_fold(const DevTree& t, const UpdateAux& aux, long long n, long long a, long long first_id,
                    DsScratch& d, int max_groups, cudaStream_t s) {
    if (max_groups <= 0) return;
    launch_chain(ds_fold_kernel, std::min(blocks_for(max_groups, 4), 152u * 8u), 128, 0, s, t, n, a, first_id, d);
    launch_chain(ds_fold_big_kernel, DS_BIG_BLOCKS, 128, 0, s, t, n, a, first_id, d);
    launch_chain(ds_delete_pairs_kernel, SPEC_BLOCKS, 256, 0, s, t, aux, d);
    launch_chain(ds_delete_kernel, blocks_for((long long)max_groups * TEAM, TEAM_CTA), TEAM_CTA, team_stack_bytes(t.height), s, t, aux, d);
}

}  // namespace ikdg
