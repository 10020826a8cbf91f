// 3D friends-of-friends with the reference's skip acceleration
// (rockstar(), src/rockstar.c:53-128; src/fof.c:112-255), reformulated so
// that every step is data parallel and the partition is identical.
//
// The reference visits particles in kd-tree order.  A particle i with more
// than FOF_SKIP_THRESH (16) neighbours inside r ("dense") marks all of them
// as skipped and merges with every particle within 2r that is already in a
// group.  Written as a function of the neighbour sets S_r(i):
//   * dense(i)      <=> |S_r(i)| > 16, a property of i alone;
//   * seeds         = the lexicographically-first maximal independent set of
//                     the dense particles in tree order (a dense particle is
//                     processed iff no earlier processed dense particle has
//                     it in its r-sphere);
//   * processed(i)  <=> no seed s < i has i in S_r(s);
//   * g(j)          = the first processed k with |S_r(k)| >= 2 and
//                     j in S_r(k): the moment j joins some group;
//   * the partition is the connected components of the links
//       {(k, j) : k processed, |S_r(k)| >= 2, j in S_r(k)}
//     plus {(s, j) : s seed, j in S_2r(s), g(j) <= s}.
// Sphere searches walk the same kd-tree with the same float tests as
// src/fast3tree.c:293-414, so S_r is the reference's set, node shortcut
// included.
#include <limits.h>

#include <algorithm>

#include <cooperative_groups.h>
#include <cub/cub.cuh>
#include <thrust/binary_search.h>
#include <thrust/execution_policy.h>

#include "kdtree_impl.cuh"
#include "lsort.cuh"
#include "uflabels.cuh"
#include "widths.cuh"

namespace rsg {

namespace cg = cooperative_groups;

// The reference's squared distance of a leaf point (dx = c[t] - q[t], dist
// += dx * dx for t = 0, 1, 2 in order, each rounded; src/fast3tree.c:
// 398-405), x and y subtracted and squared as one packed pair; cxy holds
// c[0], c[1].  dist starts at 0 and the first square is not negative, so
// 0 + dx0^2 is dx0^2.
__device__ __forceinline__ float dist3_p(unsigned long long cxy, float cz, const Rec &q) {
    const unsigned long long qxy = *reinterpret_cast<const unsigned long long *>(q.pos);
    float p0, p1;
    f2_split(f2_sqr(f2_sub(cxy, qxy)), p0, p1);
    const float dz = fsub(cz, q.pos[2]);
    return fadd(fadd(p0, p1), fmul(dz, dz));
}
__device__ __forceinline__ float dist3_q(unsigned long long cxy, float cz, const float4 &q) {
    float p0, p1;
    f2_split(f2_sqr(f2_sub(cxy, f2_pack(q.x, q.y))), p0, p1);
    const float dz = fsub(cz, q.z);
    return fadd(fadd(p0, p1), fmul(dz, dz));
}
// The reference's two box tests, in its operation order:
// _fast3tree_box_not_intersect_sphere and _fast3tree_box_inside_sphere
// (src/fast3tree.c:293-330).
__device__ __forceinline__ bool box_out3(const KNode<3> &nd, const float *c, float r2) {
    float d = 0.f, e;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        if ((e = fsub(c[i], nd.mn[i])) < 0) {
            d = fadd(d, fmul(e, e));
            if (d >= r2) return true;
        } else if ((e = fsub(c[i], nd.mx[i])) > 0) {
            d = fadd(d, fmul(e, e));
            if (d >= r2) return true;
        }
    }
    return false;
}
__device__ __forceinline__ bool box_inside3(const KNode<3> &nd, const float *c, float r,
                                            float r2) {
    if (fabsf(fsub(c[0], nd.mn[0])) > r) return false;
    float dist = 0.f;
#pragma unroll
    for (int i = 0; i < 3; i++) {
        float dx = fsub(nd.mn[i], c[i]);
        dx = fmul(dx, dx);
        float dx2 = fsub(c[i], nd.mx[i]);
        dx2 = fmul(dx2, dx2);
        if (dx2 > dx) dx = dx2;
        dist = fadd(dist, dx);
        if (dist > r2) return false;
    }
    return true;
}

// Sphere search (src/fast3tree.c:377-414) on tree `root` of a 3D forest.
// on_range(start, n) receives nodes that lie entirely inside the sphere
// (shortcut of :386-392), on_point(j) leaf points with dist < r^2.  Either
// returns false to stop the walk.  Callers that only want points after
// index `after` skip the nodes that hold none (the tests of every other node
// are unchanged, so the points found after `after` are the same).
template <class FR, class FP>
__device__ bool sphere3(const KNode<3> *nodes, int root, const Rec *recs, const float *c,
                        float r, int *errflag, FR on_range, FP on_point, int after = -1) {
    int stack[RSG_STACK];
    int sp = 0;
    stack[sp++] = root;
    const float r2 = fmul(r, r);
    while (sp) {
        const KNode<3> &nd = nodes[stack[--sp]];
        if (nd.start + nd.n <= after + 1) continue;
        if (box_out3(nd, c, r2)) continue;
        if (box_inside3(nd, c, r, r2)) {
            if (!on_range(nd.start, nd.n)) return false;
            continue;
        }
        if (nd.div < 0) {
            const unsigned long long cxy = f2_pack(c[0], c[1]);
            for (int k = 0; k < nd.n; k++) {
                int j = nd.start + k;
                if (dist3_p(cxy, c[2], recs[j]) < r2)
                    if (!on_point(j)) return false;
            }
            continue;
        }
        if (sp + 2 > RSG_STACK) {
            atomicExch(errflag, 1);
            return false;
        }
        stack[sp++] = nd.left + 1;  // right, visited after left
        stack[sp++] = nd.left;
    }
    return true;
}

// The same search for the 32 queries of a warp (one per lane, `active`
// lanes only) with one shared walk: a stack entry carries the lanes that
// still need the subtree and each lane applies its own tests, so every lane meets exactly
// the nodes and points of its own walk, in the same order.  A callback
// returning false ends that lane's walk; nodes holding no index after the
// lane's `after` are dropped for that lane (the points it finds after
// `after` are unchanged).
template <class FR, class FP>
__device__ void sphere3_warp(const KNode<3> *nodes, const Rec *recs, const float *c, bool active,
                             float r, int after, int *errflag, FR on_range, FP on_point) {
    const unsigned FULL = 0xffffffffu;
    const unsigned bit = 1u << (threadIdx.x & 31);
    const float r2 = fmul(r, r);
    int sn[RSG_STACK];
    unsigned sm[RSG_STACK];
    unsigned live = __ballot_sync(FULL, active);
    if (!live) return;
    int sp = 0;
    sn[sp] = 0;
    sm[sp++] = live;
    while (sp) {
        --sp;
        const int xi = sn[sp];
        const unsigned m = sm[sp] & live;
        if (!m) continue;
        const KNode<3> nd = nodes[xi];  // three 16-byte loads
        int kind = 0;  // 1 out, 2 inside, 3 leaf points, 4 descend
        if (m & bit) {
            kind = 1;
            if (nd.start + nd.n > after + 1 && !box_out3(nd, c, r2))
                kind = box_inside3(nd, c, r, r2) ? 2 : (nd.div < 0 ? 3 : 4);
        }
        bool stop = false;
        if (kind == 2) stop = !on_range(nd.start, nd.n);
        if (__any_sync(FULL, kind == 3)) {
            const unsigned long long cxy = f2_pack(c[0], c[1]);
            for (int k = 0; k < nd.n; k++) {
                int j = nd.start + k;
                if (kind == 3 && !stop && dist3_p(cxy, c[2], recs[j]) < r2) stop = !on_point(j);
            }
        }
        live &= ~__ballot_sync(FULL, stop);
        unsigned down = __ballot_sync(FULL, kind == 4) & live;
        if (down) {
            if (sp + 2 > RSG_STACK) {
                if (bit == 1u) atomicExch(errflag, 1);
                return;
            }
            sn[sp] = nd.left + 1;
            sm[sp++] = down;
            sn[sp] = nd.left;
            sm[sp++] = down;
        }
    }
}

// Warp-cooperative form of sphere3 for one query shared by the warp (the
// position c of particle q): every point after `after` of the reference
// walk's result set -- the points of the nodes it takes whole and the leaf
// points nearer than r -- is handed to exactly one lane.  All lanes call it
// together; every lane calls visit(j, valid) in converged code, once per
// round of up to 32 points (valid false on a lane without a point), so
// warp-level operations may be used inside visit.
// Down q's root-to-leaf path the reference walk only descends until a node
// it takes whole or whose other child it would enter (not out by its test,
// holding an index after `after`); the warp starts there.  From there it
// takes up to 32 nodes of a stack in shared memory per round and spreads
// the points of the whole nodes and leaves met over its lanes.  The set of
// points is the walk's; the order is not (the reference's is ascending
// index, left subtree first).  The stack takes 32 nodes at a time while 64
// slots and a tree depth of margin are free, one at a time otherwise
// (depth-first growth is bounded by the tree depth); a tree deeper than
// RSG_STACK sets errflag, as the scalar walk does.
#define RSG_WSTK 1024
template <class FV>
__device__ void warp_sphere3(const KNode<3> *nodes, const Rec *recs, int q, const float *c,
                             float r, int after, int *S, int *errflag, FV visit) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    const float r2 = fmul(r, r);
    int x = 0;
    for (int depth = 0; depth < RSG_STACK; depth++) {
        const KNode<3> &nd = nodes[x];
        if (nd.div < 0 || box_inside3(nd, c, r, r2)) break;
        const KNode<3> &L = nodes[nd.left];
        const bool inL = q < L.start + L.n;
        const KNode<3> &O = inL ? nodes[nd.left + 1] : L;
        if (O.start + O.n > after + 1 && !box_out3(O, c, r2)) break;
        x = inL ? nd.left : nd.left + 1;
    }
    __syncwarp();
    if (lane == 0) S[0] = x;
    int sp = 1;
    __syncwarp();
    while (sp > 0) {
        const int take = (sp + 64 <= RSG_WSTK - RSG_STACK) ? min(sp, 32) : 1;
        const int xi = lane < take ? S[sp - 1 - lane] : -1;
        sp -= take;
        __syncwarp();
        // 0 nothing, 1 whole node, 2 leaf points, 3 descend
        int kind = 0, s0 = 0, m0 = 0, left = 0;
        if (xi >= 0) {
            const KNode<3> &nd = nodes[xi];
            if (nd.start + nd.n > after + 1 && !box_out3(nd, c, r2)) {
                kind = box_inside3(nd, c, r, r2) ? 1 : (nd.div < 0 ? 2 : 3);
                s0 = nd.start;
                m0 = nd.n;
                left = nd.left;
            }
        }
        const unsigned dm = __ballot_sync(FULL, kind == 3);
        const int room = (RSG_WSTK - sp) >> 1;  // child pairs that fit
        if (kind == 3 && __popc(dm & below) < room) {
            const int at = sp + 2 * __popc(dm & below);
            S[at] = left + 1;
            S[at + 1] = left;
        }
        if (__popc(dm) > room) {
            if (lane == 0) atomicExch(errflag, 1);
            return;
        }
        sp += 2 * __popc(dm);
        // the points after `after` of this round's whole nodes and leaves
        const bool pts = kind == 1 || kind == 2;
        const int a0 = pts ? max(s0, after + 1) : 0;
        const int np = pts ? max(0, s0 + m0 - a0) : 0;
        int incl = np;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += v;
        }
        const int total = __shfl_sync(FULL, incl, 31);
        for (int base = 0; base < total; base += 32) {
            const int flat = base + lane;
            int o = 0;
#pragma unroll
            for (int step = 16; step >= 1; step >>= 1) {
                const int v = __shfl_sync(FULL, incl, o + step - 1);
                if (v <= flat) o += step;
            }
            const int oi = __shfl_sync(FULL, incl, o), on = __shfl_sync(FULL, np, o);
            const int oa = __shfl_sync(FULL, a0, o), ok = __shfl_sync(FULL, kind, o);
            int j = -1;
            bool v = false;
            if (flat < total) {
                j = oa + (flat - (oi - on));
                v = true;
                if (ok == 2) v = dist3_p(f2_pack(c[0], c[1]), c[2], recs[j]) < r2;
            }
            visit(j, v);
        }
        __syncwarp();
    }
}

// ---- kernels --------------------------------------------------------------
__global__ void k_make_recs(const rsg_particle *p, int64_t n, Rec *recs, int *bad) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    Rec r;
    bool fin = true;
#pragma unroll
    for (int d = 0; d < 6; d++) {
        r.pos[d] = p[i].pos[d];
        fin &= isfinite(r.pos[d]);
    }
    r.ridx = (int32_t)i;
    r.aux = 0;
    recs[i] = r;
    if (!fin) atomicExch(bad, 1);
}

// Duplicate candidates: a particle equal (bitwise position, or id) to its
// successor in tree order (src/rockstar.c:379-389 compares with the next
// kept particle, which is the successor whenever nothing was removed).
__global__ void k_dup_probe(const Rec *recs, const rsg_particle *p, int64_t n, int *any) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i + 1 >= n) return;
    const Rec &a = recs[i], &b = recs[i + 1];
    bool same = true;
#pragma unroll
    for (int d = 0; d < 6; d++) same &= (__float_as_uint(a.pos[d]) == __float_as_uint(b.pos[d]));
    if (same || p[a.ridx].id == p[b.ridx].id) atomicExch(any, 1);
}

// Sequential duplicate removal, only run when k_dup_probe found one.
__global__ void k_dedupe_serial(Rec *recs, const rsg_particle *p, int64_t n, int64_t *n_out) {
    if (blockIdx.x || threadIdx.x) return;
    if (n < 2) { *n_out = n; return; }
    int64_t last = n - 1;
    for (int64_t i = n - 2; i >= 0; i--) {
        bool same = true;
        for (int d = 0; d < 6; d++)
            same &= (__float_as_uint(recs[i].pos[d]) == __float_as_uint(recs[last].pos[d]));
        if (same || p[recs[last].ridx].id == p[recs[i].ridx].id) {
            n--;
            recs[i] = recs[n];
            continue;
        }
        last = i;
    }
    *n_out = n;
}

// Warp forms of the searches: queries are list[0..nq) (ascending particle
// indices, so a warp's queries are neighbours in the tree), or all
// particles when list is null.
__device__ __forceinline__ bool warp_query(const int *list, int nq, int *q) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    *q = (t < nq) ? (list ? list[t] : t) : -1;
    return *q >= 0;
}
__device__ __forceinline__ bool warp_idle(int nq) {
    return (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u) >= nq;
}
// |S_r(i)| capped at 17 (the reference only asks whether it exceeds 16).
// Half the particles of a volume are dense, and most of those have 17 of
// their neighbours in the sphere among the RSG_CNT_WIN particles on either
// side of them in tree order, so these are tried first, from shared memory: a
// point nearer than r is in S_r by whichever way the walk meets it (no box that
// holds it is out, its offsets being no more than the point's).  The lanes left
// walk the tree from the root.  The walk is what the kernel waits for (83% of the issue
// slots, 18 lanes active): 17.6 -> 10.2 ms at 33.5M particles, 4.45 -> 2.64 at
// 8.4M, 3.9 -> 1.8 on the cluster; the window costs at most 65 tests a lane.
#define RSG_CNT_T 128
#define RSG_CNT_WIN 32
__global__ void __launch_bounds__(RSG_CNT_T) k_count_w(const KNode<3> *nodes, const Rec *recs,
                                                       int n, float r, uint8_t *cnt, int *err) {
    __shared__ float4 tile[RSG_CNT_T + 2 * RSG_CNT_WIN];
    const int b0 = blockIdx.x * RSG_CNT_T - RSG_CNT_WIN;
    const float INF = __int_as_float(0x7f800000);
    for (int e = threadIdx.x; e < RSG_CNT_T + 2 * RSG_CNT_WIN; e += RSG_CNT_T)
        tile[e] = b0 + e >= 0 && b0 + e < n ? *reinterpret_cast<const float4 *>(recs + b0 + e)
                                            : make_float4(INF, INF, INF, 0.f);
    __syncthreads();
    if (warp_idle(n)) return;
    int i;
    const bool act = warp_query(nullptr, n, &i);
    const float4 q = tile[threadIdx.x + RSG_CNT_WIN];
    const float c[3] = {q.x, q.y, q.z}, r2 = fmul(r, r);
    const unsigned long long cxy = f2_pack(c[0], c[1]);
    int k = act ? 0 : 17;
    for (int e = 0; e <= 2 * RSG_CNT_WIN && __any_sync(0xffffffffu, k < 17); e++)
        k += dist3_q(cxy, c[2], tile[threadIdx.x + e]) < r2;
    const bool walk = k < 17;
    if (walk) k = 0;
    sphere3_warp(
        nodes, recs, c, walk, r, -1, err,
        [&](int s, int m) { k += m; return k <= 16; },
        [&](int j) { k++; return k <= 16; });
    if (act) cnt[i] = (uint8_t)(k > 17 ? 17 : k);
}
// ---- later dense neighbours, by group -------------------------------------
// Dense particles are named here by their place in the tree-ordered list of
// the dense ones.  The list is cut into groups of 32; bit l of a mask stands
// for place 32 g + l.  Group g's list says which dense places j > k lie in
// S_r(k) of its places k: (j, mask) for one j and the places k whose sphere
// holds it, or (first, count) for a range of j beyond the group that every
// place of the run (below) holds.  skip[j] counts the k.
// The group's particles are neighbours in the tree, so in a halo a node or
// point mostly lies inside or outside the spheres of all of them: 32 nodes,
// then 32 points, are tested against the particles' box by one lane each,
// nodes inside become ranges, and only the points between the two bounds are
// tested by every lane.  Consecutive dense particles can lie far apart (a
// jump between clusters, or across a high split of the tree), so a group is
// worked in runs: the particles within RSG_REACH linking lengths of the first
// one left, along every axis.  (At a quarter of the 512^3 volume the walks
// take 59, 39, 30 and 28 ms for 0.25, 0.5, 1 and 2.)
// A list of single pairs, one thread per particle in a shared walk, took two
// walks (counts, then entries) and 4 B a pair: 121 ms for the 7.9e9 pairs of
// that volume.
// The bounds are exact in the reference's own float arithmetic: a box's or a
// point's nearest and farthest offsets bound every lane's offsets, and
// rounding is monotone, so the sums of their squares in the same order bound
// the lane's sums.  A point is in S_r(k) when its distance is below r^2, or
// equal to it when the walk takes one of the point's nodes whole
// (glist_whole).  So nodes and points whose near bound equals r^2 are kept (a
// node at r of its particles can lie in the far corner of one taken whole), and
// only those whose far bound is below it are taken without a test.
#define RSG_REACH 2.0f
#define RSG_GE 128           // entries per chunk of a group's list
#define RSG_GSTK 512
#define RSG_RANGE 0x80000000u
struct __align__(16) GChunk {
    uint2 e[RSG_GE];         // (j, mask) or (RSG_RANGE | first, count)
    int n;                   // entries
    unsigned mask;           // the places of the run it belongs to
    int group, ord;          // the chunk is its group's ord-th
};
struct GLists {
    GChunk *pool;
    int cap;                 // chunks of the pool
    unsigned *cursor;        // hands the chunks out; those asked for beyond cap are not
                             // kept, so it may pass any width (see has_place)
    int *nch;                // chunks per group
};
// Whether the reference's walk takes a node holding leaf x whole for the
// query c: the topmost node that is out or inside decides.
__device__ __noinline__ bool glist_whole(const KNode<3> *nodes, int x, const float *c, float r,
                                         float r2) {
    bool res = false;
    for (; x >= 0; x = nodes[x].parent) {
        if (box_out3(nodes[x], c, r2)) res = false;
        else if (box_inside3(nodes[x], c, r, r2)) res = true;
    }
    return res;
}
// Least and greatest squared distance between the group's box [lo, hi] and
// the box [mn, mx].
__device__ __forceinline__ void group_bounds(const float *lo, const float *hi, const float *mn,
                                             const float *mx, float &near, float &far) {
    near = far = 0.f;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const float a = fsub(mx[d], lo[d]), b = fsub(hi[d], mn[d]);
        const float e = fmaxf(fmaxf(-a, -b), 0.f), f = fmaxf(fabsf(a), fabsf(b));
        near = fadd(near, fmul(e, e));
        far = fadd(far, fmul(f, f));
    }
}
// Lists of the groups [g0, g1); dpfx holds the dense particles before every
// index.  COUNT adds the points to skip[], the ranges to its differences
// diff[], and all pairs to *pairs.
template <bool COUNT>
__global__ void __launch_bounds__(128) k_glist(const KNode<3> *nodes, const Rec *recs,
                                               const int *dense, int nd, int g0, int g1, float r,
                                               const uint8_t *cnt, const int *dpfx, GLists G,
                                               int *skip, int *diff, unsigned long long *pairs,
                                               int *err) {
    __shared__ int stk[4][RSG_GSTK];
    __shared__ uint2 stage[4][64];
    const unsigned FULL = 0xffffffffu;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = g0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (g >= g1) return;
    const unsigned below = (1u << lane) - 1u;
    const float r2 = fmul(r, r), reach = RSG_REACH * fabsf(r);
    int *S = stk[w];
    uint2 *buf = stage[w];
    const bool act = 32 * g + lane < nd;
    const int k = act ? dense[32 * g + lane] : INT_MAX;
    const int k31 = __shfl_sync(FULL, k, 31);
    float c[3];
#pragma unroll
    for (int d = 0; d < 3; d++) c[d] = act ? recs[k].pos[d] : 0.f;
    const unsigned long long cxy = f2_pack(c[0], c[1]);
    int nch = 0;  // chunks asked for
    unsigned long long np = 0;
    bool lost = false;
    for (unsigned pending = __ballot_sync(FULL, act); pending;) {
        const int lead = __ffs(pending) - 1;
        bool mine = (pending >> lane) & 1u;
        float lo[3], hi[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const float cl = __shfl_sync(FULL, c[d], lead);
            mine &= lane == lead || fabsf(fsub(c[d], cl)) <= reach;
        }
#pragma unroll
        for (int d = 0; d < 3; d++) {
            lo[d] = ord2f(__reduce_min_sync(FULL, mine ? f2ord(c[d]) : 0xffffffffu));
            hi[d] = ord2f(__reduce_max_sync(FULL, mine ? f2ord(c[d]) : 0u));
        }
        const unsigned run = __ballot_sync(FULL, mine);
        pending &= ~run;
        const int kmin = __shfl_sync(FULL, k, lead);
        const int kmax = __shfl_sync(FULL, k, 31 - __clz(run));
        int ne = 0, ns = 0, chunk = -1;  // entries in the chunk, staged; the chunk
        auto flush = [&](int m) {        // the first m <= 32 staged entries
            if (ne == RSG_GE || ne == 0) {
                unsigned nc = 0;
                if (lane == 0) nc = atomicAdd(G.cursor, 1u);
                nc = __shfl_sync(FULL, nc, 0);
                lost |= !has_place(nc, G.cap);
                if (lane == 0 && !lost) {
                    if (ne == RSG_GE) G.pool[chunk].n = RSG_GE;
                    G.pool[nc].mask = run;
                    G.pool[nc].group = g;
                    G.pool[nc].ord = nch;
                }
                nch++;
                chunk = (int)nc;
                ne = 0;
            }
            if (!lost && lane < m) G.pool[chunk].e[ne + lane] = buf[lane];
            ne += m;
        };
        auto append = [&](bool v, uint2 e) {  // one entry per lane with v
            const unsigned em = __ballot_sync(FULL, v);
            if (v) buf[ns + __popc(em & below)] = e;
            ns += __popc(em);
            __syncwarp();
            if (ns >= 32) {
                flush(32);
                ns -= 32;
                const uint2 rest = buf[32 + lane];
                __syncwarp();
                buf[lane] = rest;
                __syncwarp();
            }
        };
        // down the tree while only one child can hold points of the lists
        int x = 0;
        for (int depth = 0; depth < RSG_STACK; depth++) {
            const int left = nodes[x].left;
            if (nodes[x].div < 0) break;
            const KNode<3> ch = nodes[left + (lane & 1)];
            float near, far;
            group_bounds(lo, hi, ch.mn, ch.mx, near, far);
            const unsigned in =
                __ballot_sync(FULL, ch.start + ch.n > kmin + 1 && !(near > r2)) & 3u;
            if (in == 3u) break;
            if (in == 0u) {
                x = -1;
                break;
            }
            x = left + (in >> 1);
        }
        if (lane == 0) S[0] = x;
        int sp = x >= 0;
        __syncwarp();
        while (sp > 0) {
            const int take = (sp + 64 <= RSG_GSTK - RSG_STACK) ? min(sp, 32) : 1;
            const int xi = lane < take ? S[sp - 1 - lane] : -1;
            sp -= take;
            __syncwarp();
            int kind = 0, s0 = 0, m0 = 0, left = 0;  // 1 whole node, 2 leaf points, 3 descend
            if (xi >= 0) {
                const KNode<3> nd3 = nodes[xi];
                float near, far;
                group_bounds(lo, hi, nd3.mn, nd3.mx, near, far);
                if (nd3.start + nd3.n > kmin + 1 && !(near > r2)) {
                    kind = far < r2 ? 1 : (nd3.div < 0 ? 2 : 3);
                    s0 = nd3.start;
                    m0 = nd3.n;
                    left = nd3.left;
                }
            }
            const unsigned dm = __ballot_sync(FULL, kind == 3);
            if (__popc(dm) > ((RSG_GSTK - sp) >> 1)) {  // reported by the call: no list
                if (lane == 0) {
                    atomicExch(err, 1);
                    G.nch[g] = nch;
                    if (ne > 0 && !lost) G.pool[chunk].n = ne;
                }
                return;
            }
            if (kind == 3) {
                const int at = sp + 2 * __popc(dm & below);
                S[at] = left + 1;
                S[at + 1] = left;
            }
            sp += 2 * __popc(dm);
            // whole nodes beyond the run's own places: ranges
            bool rg = kind == 1 && s0 > kmax;
            if (__any_sync(FULL, rg)) {
                int first = 0, many = 0;
                if (rg) {
                    first = dpfx[s0];
                    many = dpfx[s0 + m0] - first;
                    kind = 0;
                    if (COUNT && many) {
                        atomicAdd(&diff[first], __popc(run));
                        atomicSub(&diff[first + many], __popc(run));
                        np += (unsigned long long)many * __popc(run);
                    }
                }
                append(many > 0, make_uint2(RSG_RANGE | (unsigned)first, (unsigned)many));
            }
            // the points after kmin of the round's other whole nodes and leaves
            const int a0 = max(s0, kmin + 1);
            const int pn = kind == 1 || kind == 2 ? max(0, s0 + m0 - a0) : 0;
            int incl = pn;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(FULL, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(FULL, incl, 31);
            for (int base = 0; base < total; base += 32) {
                const int flat = base + lane;
                int o = 0;
#pragma unroll
                for (int step = 16; step >= 1; step >>= 1) {
                    const int v = __shfl_sync(FULL, incl, o + step - 1);
                    if (v <= flat) o += step;
                }
                const int oi = __shfl_sync(FULL, incl, o), on = __shfl_sync(FULL, pn, o);
                const int oa = __shfl_sync(FULL, a0, o), ok = __shfl_sync(FULL, kind, o);
                const int ox = __shfl_sync(FULL, xi, o);
                int j = -1;
                bool all = false, some = false;
                if (flat < total) {
                    j = oa + (flat - (oi - on));
                    if (cnt[j] > 16) {
                        all = ok == 1;
                        if (!all) {
                            const float4 q = *reinterpret_cast<const float4 *>(recs + j);
                            const float p[3] = {q.x, q.y, q.z};
                            float near, far;
                            group_bounds(lo, hi, p, p, near, far);
                            all = far < r2;
                            some = !all && !(near > r2);
                        }
                    }
                }
                unsigned mask = all ? run : 0u;
                if (__any_sync(FULL, all && j <= kmax)) {  // among the run's own places
                    int p = 0;                             // particles of the group below j
#pragma unroll
                    for (int step = 16; step >= 1; step >>= 1)
                        if (__shfl_sync(FULL, k, p + step - 1) < j) p += step;
                    if (p == 31 && k31 < j) p = 32;
                    if (all && p < 32) mask &= (1u << p) - 1u;
                }
                for (unsigned todo = __ballot_sync(FULL, some); todo; todo &= todo - 1) {
                    const int b = __ffs(todo) - 1;
                    const int jb = __shfl_sync(FULL, j, b), xb = __shfl_sync(FULL, ox, b);
                    bool hit = false;
                    if (mine && k < jb) {
                        const float d = dist3_p(cxy, c[2], recs[jb]);
                        hit = d < r2 || (!(d > r2) && glist_whole(nodes, xb, c, r, r2));
                    }
                    const unsigned hm = __ballot_sync(FULL, hit);
                    if (lane == b) mask = hm;
                }
                const int dj = mask ? dpfx[j] : 0;
                if (COUNT && mask) {
                    atomicAdd(&skip[dj], __popc(mask));
                    np += __popc(mask);
                }
                append(mask != 0u, make_uint2((unsigned)dj, mask));
            }
            __syncwarp();
        }
        if (ns > 0) flush(ns);
        if (lane == 0 && ne > 0 && !lost) G.pool[chunk].n = ne;
        __syncwarp();
    }
    if (lane == 0) G.nch[g] = nch;
    if (COUNT) {
        for (int o = 16; o; o >>= 1) np += __shfl_xor_sync(FULL, np, o);
        if (lane == 0 && np) atomicAdd(pairs, np);
    }
}
__global__ void k_gchunks(const int *gch, int ng, int64_t *nch) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g <= ng) nch[g] = g < ng ? gch[g] : 0;
}
// The chunks of every group side by side: (chunk, run's places) of group g at
// table[off[g] - off0 ...].
__global__ void k_gtable(const GChunk *pool, int n, const int64_t *off, int64_t off0,
                         uint2 *table) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < n)
        table[off[pool[c].group] - off0 + pool[c].ord] = make_uint2((unsigned)c, pool[c].mask);
}
// The seeds' searches run one warp per seed (warp_sphere3): a seed's
// spheres hold hundreds to thousands of points, and its neighbours in tree
// order are mostly skipped particles with no search of their own, so a
// thread per particle would leave the warp to one lane.
#define RSG_SEED_WARPS 4
#define SEED_LOOP(ns)                                                                  \
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < (ns);               \
         t += (gridDim.x * blockDim.x) >> 5)
// Every point after seed s of S_r(s) is skipped (src/rockstar.c:75-77), and
// g(j) over the seeds' spheres (see k_gtime_r), in one walk: apart the two took
// 3.0 and 3.8 ms at 33.5M particles.
__global__ void __launch_bounds__(RSG_SEED_WARPS * 32)
    k_seed_mark_w(const KNode<3> *nodes, const Rec *recs, const int *seeds, int ns, float r,
                  uint8_t *skipped, int *gtime, int *err) {
    __shared__ int stk[RSG_SEED_WARPS][RSG_WSTK];
    int *S = stk[threadIdx.x >> 5];
    SEED_LOOP(ns) {
        const int k = seeds[t];
        const float c[3] = {recs[k].pos[0], recs[k].pos[1], recs[k].pos[2]};
        warp_sphere3(nodes, recs, k, c, r, -1, S, err, [&](int j, bool v) {
            if (!v) return;
            if (j > k) skipped[j] = 1;
            atomicMin(&gtime[j], k);
        });
    }
}
// f(k) of the seeds (see k_fptr3): the first particle of S_r(k) in walk
// order -- the smallest index -- labelled before k
__global__ void __launch_bounds__(RSG_SEED_WARPS * 32)
    k_fptr_seed_w(const KNode<3> *nodes, const Rec *recs, const int *seeds, int ns, float r,
                  const int *gtime, int *ptr, int *err) {
    __shared__ int stk[RSG_SEED_WARPS][RSG_WSTK];
    int *S = stk[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31;
    SEED_LOOP(ns) {
        const int k = seeds[t];
        const int gk = gtime[k];
        if (gk < k) {
            if (lane == 0) ptr[k] = gk;
            continue;
        }
        const float c[3] = {recs[k].pos[0], recs[k].pos[1], recs[k].pos[2]};
        int best = INT_MAX;
        warp_sphere3(nodes, recs, k, c, r, -1, S, err, [&](int j, bool v) {
            if (v && j < best && gtime[j] < k) best = j;
        });
        best = __reduce_min_sync(0xffffffffu, best);
        if (lane == 0) ptr[k] = best == INT_MAX ? k : gtime[best];
    }
}
// Candidate merges of the seeds (see k_cand3): both spheres, S_r(k) with
// the particles labelled before k, then S_2r(k) with those labelled by k.
// A label is emitted once per sphere at its first occurrence in walk order
// (the smallest index, which is the key's last field): a per-warp hash
// table keeps the smallest index of every label met; a label that finds no
// slot is emitted at every occurrence (a repeat is a no-op merge).
#define RSG_CAND_HT 128
__device__ __forceinline__ void cand_emit(int k, int phase, int j, int F, int W, int64_t cap,
                                          unsigned long long *count, uint64_t *ckey, int32_t *cF,
                                          int32_t *cW) {
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(count, (unsigned long long)g.size());
    const unsigned long long u = g.shfl(base, 0) + g.thread_rank();
    if ((int64_t)u < cap) {
        ckey[u] = ((uint64_t)(uint32_t)k << 32) | ((uint64_t)phase << 31) | (uint32_t)j;
        cF[u] = F;
        cW[u] = W;
    }
}
__global__ void __launch_bounds__(RSG_SEED_WARPS * 32)
    k_cand_seed_w(const KNode<3> *nodes, const Rec *recs, const int *seeds, int ns, float r,
                  float r2x, const int *gtime, const int32_t *lab0, const int32_t *sfid,
                  int64_t cap, unsigned long long *count, uint64_t *ckey, int32_t *cF,
                  int32_t *cW, int *err) {
    __shared__ int stk[RSG_SEED_WARPS][RSG_WSTK];
    __shared__ int hk[RSG_SEED_WARPS][RSG_CAND_HT], hv[RSG_SEED_WARPS][RSG_CAND_HT];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int *S = stk[w], *K = hk[w], *Vv = hv[w];
    SEED_LOOP(ns) {
        const int k = seeds[t];
        const int F = sfid[k];
        const float c[3] = {recs[k].pos[0], recs[k].pos[1], recs[k].pos[2]};
        for (int phase = 0; phase < 2; phase++) {
            for (int e = lane; e < RSG_CAND_HT; e += 32) {
                K[e] = -1;
                Vv[e] = INT_MAX;
            }
            __syncwarp();
            warp_sphere3(nodes, recs, k, c, phase ? r2x : r, -1, S, err, [&](int j, bool v) {
                if (!v) return;
                const int gj = gtime[j];
                if (!(phase == 0 ? gj < k : gj <= k)) return;
                const int W = lab0[j];
                if (W == F) return;
                const unsigned h = ((unsigned)W * 2654435761u) >> 25;  // 7 bits
                for (int pr = 0; pr < 8; pr++) {
                    const int e = (h + pr) & (RSG_CAND_HT - 1);
                    const int old = atomicCAS(&K[e], -1, W);
                    if (old == -1 || old == W) {
                        atomicMin(&Vv[e], j);
                        return;
                    }
                }
                cand_emit(k, phase, j, F, W, cap, count, ckey, cF, cW);
            });
            __syncwarp();
            for (int e = lane; e < RSG_CAND_HT; e += 32)
                if (K[e] != -1) cand_emit(k, phase, Vv[e], F, K[e], cap, count, ckey, cF, cW);
            __syncwarp();
        }
    }
}

// g(j): the first processed particle k with |S_r(k)| >= 2 (in tree order)
// whose r-sphere holds j -- the moment link_particle_to_fof gives j its
// label (src/fof.c:112-140).
__global__ void k_gtime_r(const KNode<3> *nodes, const Rec *recs, int n, float r,
                          const uint8_t *cnt, const uint8_t *skipped, const uint8_t *state,
                          int *gtime, int *err) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || skipped[k] || cnt[k] < 2 || state[k] == 1) return;  // seeds: k_seed_mark_w
    float c[3] = {recs[k].pos[0], recs[k].pos[1], recs[k].pos[2]};
    sphere3(
        nodes, 0, recs, c, r, err,
        [&](int a, int m) {
            for (int j = a; j < a + m; j++) atomicMin(&gtime[j], k);
            return true;
        },
        [&](int j) {
            atomicMin(&gtime[j], k);
            return true;
        });
}

// f(k), the set event k works on (src/fof.c:116-131): k's own label when an
// earlier event gave it one, else the label of the first particle of S_r(k)
// (walk order) labelled before k, else a new set (ptr = k).  -1: no event.
__global__ void k_fptr3(const KNode<3> *nodes, const Rec *recs, int n, float r,
                        const uint8_t *cnt, const uint8_t *skipped, const uint8_t *state,
                        const int *gtime, int *ptr, int *err) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || state[k] == 1) return;  // seeds: k_fptr_seed_w
    if (skipped[k] || cnt[k] < 2) {
        ptr[k] = -1;
        return;
    }
    int gk = gtime[k];
    if (gk < k) {
        ptr[k] = gk;
        return;
    }
    int p = k;
    float c[3] = {recs[k].pos[0], recs[k].pos[1], recs[k].pos[2]};
    sphere3(
        nodes, 0, recs, c, r, err,
        [&](int a, int m) {
            for (int j = a; j < a + m; j++)
                if (gtime[j] < k) {
                    p = gtime[j];
                    return false;
                }
            return true;
        },
        [&](int j) {
            if (gtime[j] < k) {
                p = gtime[j];
                return false;
            }
            return true;
        });
    ptr[k] = p;
}

// Candidate merges of event k in walk order: for every particle of S_r(k)
// labelled before k, link_particle_to_fof joins f(k)'s set to that
// particle's set (src/fof.c:133-139); a seed then does the same for every
// particle of S_2r(k) labelled by then (link_fof_to_fof, src/fof.c:142-158,
// k_cand_seed_w).  A label equal to f(k), or one this event already
// emitted, changes nothing and is skipped.  Keys order the candidates in
// time: (k, sphere, position in the result list), the position being the
// particle index (the walk lists points in ascending index order).
#define RSG_CAND_SEEN 8
__global__ void k_cand3(const KNode<3> *nodes, const Rec *recs, int n, float r,
                        const uint8_t *cnt, const uint8_t *skipped, const uint8_t *state,
                        const int *gtime, const int32_t *lab0, const int32_t *sfid, int64_t cap,
                        unsigned long long *count, uint64_t *ckey, int32_t *cF, int32_t *cW,
                        int *err) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n || skipped[k] || cnt[k] < 2 || state[k] == 1) return;  // seeds: k_cand_seed_w
    const int F = sfid[k];
    int seen[RSG_CAND_SEEN];
    int ns = 0;
    auto visit = [&](int j) {
        int gj = gtime[j];
        if (gj < k) {
            int W = lab0[j];
            bool dup = (W == F);
            for (int q = 0; q < ns; q++) dup |= (seen[q] == W);
            if (!dup) {
                if (ns < RSG_CAND_SEEN) seen[ns++] = W;
                unsigned long long t = atomicAdd(count, 1ull);
                if ((int64_t)t < cap) {
                    ckey[t] = ((uint64_t)(uint32_t)k << 32) | (uint32_t)j;
                    cF[t] = F;
                    cW[t] = W;
                }
            }
        }
    };
    float c[3] = {recs[k].pos[0], recs[k].pos[1], recs[k].pos[2]};
    sphere3(
        nodes, 0, recs, c, r, err,
        [&](int a, int m) {
            for (int j = a; j < a + m; j++) visit(j);
            return true;
        },
        [&](int j) {
            visit(j);
            return true;
        });
}

// The ordered independent set of the dense particles (the seeds), decided
// frontier by frontier.  skip[j] holds the earlier potential skippers of dense
// place j still undecided, and in its high bits j's own fate; und is a bitmap
// of the undecided places.  A place decided in one step is worked off in the
// next: its bit is set in its group's mask of that step's parity (fresh), and
// the groups with a bit are the frontier.  A group's list is walked once for
// all the places decided (D), one warp per chunk: an undecided j held by a
// seed among them is skipped, any other is released from as many skippers as
// hold it, and a j with none left that was not skipped is a seed (all its
// earlier potential skippers are decided and none of them is a seed).  Most
// j are decided already -- a seed skips its whole sphere at once -- and cost
// a bit, a range's a word for 32.  A step lasts as long as its longest chain
// of dependent accesses, so the frontier is queued by chunks (a group in a
// halo's core has hundreds; a warp per group took 0.3 ms a step), four places
// a lane go through one atomic at a time, nothing waits for the queue
// (k_kahn_next collects it from fresh), and the undecided stretches of long
// ranges are left to the warps of k_kahn_wide.  A warp per particle over its
// list of pairs, an atomic each, took 107 ms for 7.9e9 pairs.  When the
// lists are built one chunk of groups [gbeg, gend) at a time, a place decided
// beyond has no list yet: it keeps its fate and its group is queued when its
// own chunk starts.
#define RSG_SEED 0x40000000
#define RSG_SKIPPED 0x20000000
#define RSG_FATE (RSG_SEED | RSG_SKIPPED)
struct KahnCtl {
    int now, next;  // list chunks queued for this step; collected for the next
    int par;        // parity of the step
    int iters, hit, decided, gbeg, gend;
    int done, nitems;
    int going, had;  // places decided for the next step; this step had some
    int more, pad;   // the loop goes on
};
struct KahnItem {  // a stretch of places for k_kahn_wide
    int first, count;
    int skip;      // 1: held by a seed
    int many;      // places it is released by
};
struct KahnList {
    GLists G;
    int nd, ng;
    uint2 *table, *queue;  // (chunk, run's places) by group; (chunk, group) of the step
    const int64_t *off;    // the groups' first entries of the table
    unsigned *fresh[2];
    KahnCtl *ctl;
    int *skip;
    unsigned *und;
    KahnItem *items;
    int icap;
};
// An undecided place j met in this step: `skip` as read by kahn_meet.
__device__ __forceinline__ int kahn_meet(const KahnList &L, int j, bool seed, int many) {
    return seed ? atomicOr(&L.skip[j], RSG_SKIPPED) : atomicSub(&L.skip[j], many);
}
__device__ __forceinline__ void kahn_decide(const KahnList &L, unsigned *fresh, int gend, int j,
                                            bool seed, int many, int old) {
    if (seed ? (old & RSG_FATE) != 0 : old != many) return;
    if (!seed) atomicOr(&L.skip[j], RSG_SEED);
    const int g = j >> 5;
    const unsigned bit = 1u << (j & 31);
    atomicAnd(&L.und[g], ~bit);
    if (g < gend) atomicOr(&fresh[g], bit);
}
// The bits of word w that belong to places [a, a + c).
__device__ __forceinline__ unsigned range_bits(int w, int a, int c) {
    const int lo = max(a - 32 * w, 0), hi = min(a + c - 32 * w, 32);
    return (hi >= 32 ? 0xffffffffu : (1u << hi) - 1u) & ~((1u << lo) - 1u);
}
__global__ void __launch_bounds__(256) k_kahn(KahnList L) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const KahnCtl &C = *L.ctl;
    const int now = C.now, par = C.par, gend = C.gend;
    const unsigned *cf = par ? L.fresh[1] : L.fresh[0];
    unsigned *nf = par ? L.fresh[0] : L.fresh[1];
    for (int f = w0; f < now; f += nw) {
        const uint2 item = L.queue[f];
        const GChunk &K = L.G.pool[item.x];
        const int g = (int)item.y;
        const unsigned D = cf[g];
        const int me = 32 * g + lane;
        const unsigned mask = K.mask;
        const int m = K.n;
        const unsigned Dr = mask & D;
        const unsigned Sr = __ballot_sync(FULL, me < L.nd && (L.skip[me] & RSG_SEED)) & Dr;
        uint2 ev[RSG_GE / 32];
#pragma unroll
        for (int u = 0; u < RSG_GE / 32; u++) {
            ev[u] = make_uint2(0u, 0u);
            if (32 * u + lane < m) ev[u] = __ldcs(&K.e[32 * u + lane]);
        }
#pragma unroll
        for (int u = 0; u < RSG_GE / 32; u++) {
            if (32 * u >= m) break;
            const bool rg = ev[u].x & RSG_RANGE;
            const int a = (int)(ev[u].x & ~RSG_RANGE);
            const int c = rg ? (int)ev[u].y : 1;
            const unsigned by = rg ? Dr : ev[u].y & Dr;
            const int wa = a >> 5, wb = (a + c - 1) >> 5;
            const bool wide = rg && wb - wa > 3;
            bool hit = false;
            if (by && !wide)
                for (int w = wa; w <= wb; w++)
                    hit |= (L.und[w] & range_bits(w, a, c)) != 0u;
            // the places of the entries with an undecided one, flattened
            if (__any_sync(FULL, hit)) {
                const int pn = hit ? c : 0;
                int incl = pn;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(FULL, incl, o);
                    if (lane >= o) incl += v;
                }
                const int total = __shfl_sync(FULL, incl, 31);
                for (int base = 0; base < total; base += 128) {
                    int j[4], old[4], many[4];
                    bool on[4], sd[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        on[q] = false;
                        if (base + 32 * q >= total) continue;  // uniform
                        const int flat = base + 32 * q + lane;
                        int o = 0;
#pragma unroll
                        for (int step = 16; step >= 1; step >>= 1) {
                            const int v = __shfl_sync(FULL, incl, o + step - 1);
                            if (v <= flat) o += step;
                        }
                        const int oi = __shfl_sync(FULL, incl, o);
                        const int on0 = __shfl_sync(FULL, pn, o);
                        const int oa = __shfl_sync(FULL, a, o);
                        const unsigned ob = __shfl_sync(FULL, by, o);
                        j[q] = oa + (flat - (oi - on0));
                        sd[q] = (ob & Sr) != 0u;
                        many[q] = __popc(ob);
                        on[q] = flat < total && ((L.und[j[q] >> 5] >> (j[q] & 31)) & 1u);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (on[q]) old[q] = kahn_meet(L, j[q], sd[q], many[q]);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (on[q]) kahn_decide(L, nf, gend, j[q], sd[q], many[q], old[q]);
                }
            }
            for (unsigned todo = __ballot_sync(FULL, wide); todo; todo &= todo - 1) {
                const int b = __ffs(todo) - 1;
                const int ba = __shfl_sync(FULL, a, b), bc = __shfl_sync(FULL, c, b);
                const int be = (ba + bc - 1) >> 5;
                for (int v0 = ba >> 5; v0 <= be; v0 += 32) {
                    const int w = v0 + lane;
                    const unsigned word = w <= be ? L.und[w] & range_bits(w, ba, bc) : 0u;
                    const unsigned nz = __ballot_sync(FULL, word != 0u);
                    if (!nz) continue;
                    // eight words with an undecided place: an item
                    const bool lead = (lane & 7) == 0 && ((nz >> lane) & 0xffu);
                    const unsigned lm = __ballot_sync(FULL, lead);
                    int at = 0;
                    if (lane == 0) at = atomicAdd(&L.ctl->nitems, __popc(lm));
                    at = __shfl_sync(FULL, at, 0) + __popc(lm & ((1u << lane) - 1u));
                    const bool fits = at < L.icap;
                    if (lead && fits) {
                        const int f0 = max(32 * w, ba);
                        L.items[at] = KahnItem{f0, min(32 * w + 256, ba + bc) - f0,
                                               Sr != 0u, __popc(Dr)};
                    }
                    // no room: here and now
                    for (unsigned rest = __ballot_sync(FULL, lead && !fits); rest;
                         rest &= rest - 1) {
                        const int l0 = __ffs(rest) - 1;
                        for (int q = l0; q < l0 + 8; q++) {
                            const unsigned bits = __shfl_sync(FULL, word, q);
                            if (!((bits >> lane) & 1u)) continue;
                            const int j = 32 * (v0 + q) + lane;
                            kahn_decide(L, nf, gend, j, Sr != 0u, __popc(Dr),
                                        kahn_meet(L, j, Sr != 0u, __popc(Dr)));
                        }
                    }
                }
            }
        }
    }
}
// The stretches k_kahn left, a warp each: at most 256 places of eight words.
__global__ void __launch_bounds__(256) k_kahn_wide(KahnList L) {
    const int lane = threadIdx.x & 31;
    const int w0 = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    const KahnCtl &C = *L.ctl;
    const int n = min(C.nitems, L.icap), gend = C.gend;
    unsigned *nf = C.par ? L.fresh[0] : L.fresh[1];
    for (int f = w0; f < n; f += nw) {
        const KahnItem it = L.items[f];
        int old[8];
        bool on[8];
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int j = it.first + 32 * q + lane;
            on[q] = j < it.first + it.count && ((L.und[j >> 5] >> (j & 31)) & 1u);
        }
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (on[q]) old[q] = kahn_meet(L, it.first + 32 * q + lane, it.skip != 0, it.many);
#pragma unroll
        for (int q = 0; q < 8; q++)
            if (on[q])
                kahn_decide(L, nf, gend, it.first + 32 * q + lane, it.skip != 0, it.many, old[q]);
    }
}
// Queues the chunks of the groups with decided places whose run holds one.
// All lanes of a warp call it with their group's mask (0: none); a lane goes
// through its group's chunks itself, or the warp does for it when they are
// many.
#define RSG_KLANE 16
__device__ __forceinline__ void kahn_queue(const KahnList &L, int *count, int g, unsigned D,
                                           bool step) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint2 *tab = L.table - L.off[L.ctl->gbeg];
    int64_t o = 0;
    int n = 0;
    if (D) {
        o = L.off[g];
        n = (int)(L.off[g + 1] - o);
    }
    const bool own = n <= RSG_KLANE;
    int c = 0;
    if (own)
        for (int t = 0; t < n; t++) c += (tab[o + t].y & D) != 0u;
    int incl = c;
#pragma unroll
    for (int q = 1; q < 32; q <<= 1) {
        const int v = __shfl_up_sync(FULL, incl, q);
        if (lane >= q) incl += v;
    }
    const int total = __shfl_sync(FULL, incl, 31);
    if (total) {
        int at = 0;
        if (lane == 0) at = atomicAdd(count, total);
        at = __shfl_sync(FULL, at, 0) + incl - c;
        if (own)
            for (int t = 0; t < n; t++) {
                const uint2 e = tab[o + t];
                if (e.y & D) L.queue[at++] = make_uint2(e.x, (unsigned)g);
            }
    }
    for (unsigned todo = __ballot_sync(FULL, !own); todo; todo &= todo - 1) {
        const int b = __ffs(todo) - 1;
        const int bg = __shfl_sync(FULL, g, b), bn = __shfl_sync(FULL, n, b);
        const unsigned bd = __shfl_sync(FULL, D, b);
        const int64_t bo = __shfl_sync(FULL, o, b);
        for (int t0 = 0; t0 < bn; t0 += 32) {
            uint2 e = make_uint2(0u, 0u);
            if (t0 + lane < bn) e = tab[bo + t0 + lane];
            const bool on = (e.y & bd) != 0u;
            const unsigned m = __ballot_sync(FULL, on);
            if (!m) continue;
            int at = 0;
            if (lane == 0) at = atomicAdd(count, __popc(m));
            at = __shfl_sync(FULL, at, 0) + __popc(m & ((1u << lane) - 1u));
            if (on) L.queue[at] = make_uint2(e.x, (unsigned)bg);
        }
    }
    const int dec = __reduce_add_sync(FULL, __popc(D));
    if (lane == 0 && dec) {
        atomicAdd(&L.ctl->decided, dec);
        if (step) L.ctl->going = 1;
    }
}
// Collects the next frontier from the groups' masks and clears those of the
// step just run; the last block to finish advances the step.  False when no
// place was decided or a limit was reached.  A step without decided places
// (the host loop may run some past the last) does not count.
__device__ __forceinline__ bool kahn_collect(const KahnList &L, int limit, bool counts,
                                             bool *last) {
    KahnCtl *ctl = L.ctl;
    unsigned *cf = ctl->par ? L.fresh[1] : L.fresh[0];
    const unsigned *nf = ctl->par ? L.fresh[0] : L.fresh[1];
    const int gb = ctl->gbeg, ge = ctl->gend;
    bool any = false;
    const int nt = gridDim.x * blockDim.x, t = blockIdx.x * blockDim.x + threadIdx.x;
    for (int g = gb + t; g < ge; g += nt)
        if (cf[g]) {
            cf[g] = 0u;
            any = true;
        }
    // neighbouring groups (a halo's are decided together) to different warps,
    // by the 32 bytes a read takes
    const int64_t nw = nt >> 5;
    for (int64_t s0 = t >> 5; gb + 8 * s0 < ge; s0 += 4 * nw) {
        const int64_t gl = gb + 8 * (s0 + ((t & 31) >> 3) * nw) + (t & 7);
        const int g = gl < ge ? (int)gl : ge;
        const unsigned D = g < ge ? nf[g] : 0u;
        if (__any_sync(0xffffffffu, D != 0u)) kahn_queue(L, &ctl->next, g, D, true);
    }
    any = __syncthreads_or(any);
    __threadfence();
    *last = false;
    if (threadIdx.x == 0) {
        if (any) atomicOr(&ctl->had, 1);
        __threadfence();
        *last = atomicAdd(&ctl->done, 1) == (int)gridDim.x - 1;
    }
    if (!*last) return false;
    if (counts | atomicExch(&ctl->had, 0)) ctl->iters++;
    bool more = atomicExch(&ctl->going, 0) != 0;
    ctl->now = atomicExch(&ctl->next, 0);
    ctl->done = 0;
    ctl->nitems = 0;
    ctl->par ^= 1;
    if (more && ctl->iters >= limit) {
        ctl->hit = 1;
        more = false;
    }
    ctl->more = more;
    return more;
}
__global__ void k_kahn_next(KahnList L, int limit, int counts) {
    bool last;
    kahn_collect(L, limit, counts != 0, &last);
}
__global__ void k_kahn_next_g(KahnList L, int limit, cudaGraphConditionalHandle h) {
    bool last;
    const bool more = kahn_collect(L, limit, true, &last);
    if (last) cudaGraphSetConditional(h, more ? 1u : 0u);
}
// skip[] from the points' counts and the ranges' (pre: their differences
// summed); places with no earlier potential skipper are seeds, the others
// undecided.
__global__ void k_kahn_init(int nd, const int *pre, int *skip, unsigned *und) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    bool open = false;
    if (t < nd) {
        const int v = skip[t] + pre[t];
        open = v != 0;
        skip[t] = open ? v : RSG_SEED;
    }
    const unsigned b = __ballot_sync(0xffffffffu, open);
    if ((t & 31) == 0 && t < nd) und[t >> 5] = b;
}
// A chunk's first frontier: its groups' places decided so far.  One thread
// per group, reading its 32 fates; k_kahn_start names the chunk before.
__global__ void k_kahn_chunk(KahnList L) {
    const KahnCtl &C = *L.ctl;
    const int gend = C.gend;
    unsigned *cf = C.par ? L.fresh[1] : L.fresh[0];
    for (int g0 = C.gbeg + blockIdx.x * blockDim.x; g0 < gend; g0 += gridDim.x * blockDim.x) {
        const int g = g0 + threadIdx.x;
        unsigned D = 0u;
        if (g < gend) {
            for (int l = 0; l < 32 && 32 * g + l < L.nd; l++)
                if (L.skip[32 * g + l] & RSG_FATE) D |= 1u << l;
            cf[g] = D;
        }
        if (__any_sync(0xffffffffu, D != 0u)) kahn_queue(L, &L.ctl->now, g, D, false);
    }
}
__global__ void k_kahn_start(KahnCtl *ctl, int gbeg, int gend) {
    ctl->gbeg = gbeg;
    ctl->gend = gend;
    ctl->now = ctl->next = ctl->nitems = ctl->going = ctl->had = ctl->done = 0;
}
struct ChunkTarget {
    int64_t step;
    __host__ __device__ int64_t operator()(int64_t t) const { return (t + 1) * step; }
};
// State of the dense particles: 1 a seed, 2 skipped by one (others: 0).
__global__ void k_state8(const int *dense, int nd, const int *skip, uint8_t *s8) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nd) s8[dense[t]] = (skip[t] & RSG_SEED) ? 1 : 2;
}

// Label of every particle: the smallfof of the set it joined (root null),
// or the final root of that set.
__global__ void k_lab3(const int *gtime, int n, const int32_t *sfid, const int32_t *root,
                       int32_t *lab) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    int gj = gtime[j];
    lab[j] = (gj == 0x7f7f7f7f) ? -1 : (root ? root[sfid[gj]] : sfid[gj]);
}
__global__ void k_gather_out(const Rec *recs, const rsg_particle *in, int n, rsg_particle *out) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) out[k] = in[recs[k].ridx];
}
// After the partition sort: particles without a label first, then one run
// per label in ascending order (src/fof.c:226-255 walks them in this order).
__global__ void k_run_heads3(const int32_t *lab, int n, int *head) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    head[i] = lab[i] >= 0 && (i == 0 || lab[i - 1] != lab[i]);
}
// Runs of at least MIN_HALO_PARTICLES become groups, in run order.
__global__ void k_runs3(const int *hpos, const int *nh, int n, int64_t minsz, int64_t *roff,
                        int64_t *rsz, int32_t *keep) {
    int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= *nh) return;
    int s = hpos[g];
    int e = (g + 1 < *nh) ? hpos[g + 1] : n;
    roff[g] = s;
    rsz[g] = e - s;
    keep[g] = (e - s) >= minsz;
}

__global__ void k_take2(const int32_t *idx, int m, const int32_t *a, const int32_t *b,
                        int32_t *a2, int32_t *b2) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= m) return;
    a2[t] = a[idx[t]];
    b2[t] = b[idx[t]];
}
__global__ void k_iota(int *a, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = i;
}

struct SeedFlag {
    const uint8_t *state;
    __device__ uint8_t operator()(int i) const { return state[i] == 1; }
};
struct DFlag {
    const uint8_t *c;
    __device__ uint8_t operator()(int i) const { return c[i] > 16; }
};
struct DenseI {
    __host__ __device__ int operator()(uint8_t c) const { return c > 16; }
};
static int sm_count() {
    int dev = 0, v = 0;
    RSG_CUDA(cudaGetDevice(&dev));
    RSG_CUDA(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
    return v > 0 ? v : 1;
}
// The seed frontiers of one chunk as one graph: a while node whose body runs
// a step (k_kahn, k_kahn_wide) and advances the frontier (k_kahn_next_g sets
// the loop condition), so no step waits for the host.
struct KahnGraph {
    cudaGraph_t g = nullptr;
    cudaGraphExec_t e = nullptr;
    void build(int GK, int GN, int TK, KahnList L, int limit) {
        RSG_CUDA(cudaGraphCreate(&g, 0));
        cudaGraphConditionalHandle h;
        RSG_CUDA(cudaGraphConditionalHandleCreate(&h, g, 1, cudaGraphCondAssignDefault));
        cudaGraphNodeParams cp = {};
        cp.type = cudaGraphNodeTypeConditional;
        cp.conditional.handle = h;
        cp.conditional.type = cudaGraphCondTypeWhile;
        cp.conditional.size = 1;
        cudaGraphNode_t cn, wn, xn, nn;
        RSG_CUDA(cudaGraphAddNode(&cn, g, nullptr, nullptr, 0, &cp));
        cudaGraph_t body = cp.conditional.phGraph_out[0];
        void *wargs[] = {(void *)&L};
        cudaKernelNodeParams kp = {};
        kp.func = (void *)k_kahn;
        kp.gridDim = dim3(GK);
        kp.blockDim = dim3(TK);
        kp.kernelParams = wargs;
        RSG_CUDA(cudaGraphAddKernelNode(&wn, body, nullptr, 0, &kp));
        kp.func = (void *)k_kahn_wide;
        RSG_CUDA(cudaGraphAddKernelNode(&xn, body, &wn, 1, &kp));
        void *nargs[] = {(void *)&L, (void *)&limit, (void *)&h};
        kp.func = (void *)k_kahn_next_g;
        kp.gridDim = dim3(GN);
        kp.kernelParams = nargs;
        RSG_CUDA(cudaGraphAddKernelNode(&nn, body, &xn, 1, &kp));
        RSG_CUDA(cudaGraphInstantiate(&e, g, 0));
    }
    cudaStream_t ran = nullptr;
    void run(cudaStream_t st) {
        ran = st;
        RSG_CUDA(cudaGraphLaunch(e, st));
    }
    ~KahnGraph() {
        if (ran) cudaStreamSynchronize(ran);  // not destroyed while it runs
        if (e) cudaGraphExecDestroy(e);
        if (g) cudaGraphDestroy(g);
    }
};
// Indices i < n with pred(i), ascending, into out; returns their number.
template <class Pred>
static int select_where(Arena &ar, int n, Pred pred, int *out, cudaStream_t st) {
    thrust::transform_iterator<Pred, thrust::counting_iterator<int>, uint8_t> it(
        thrust::counting_iterator<int>(0), pred);
    size_t mark = ar.used;
    int *cnt = ar.get<int>(1);
    size_t b = 0;
    cub::DeviceSelect::Flagged(nullptr, b, thrust::counting_iterator<int>(0), it, out, cnt, n, st);
    void *t = ar.take(b + 256);
    cub::DeviceSelect::Flagged(t, b, thrust::counting_iterator<int>(0), it, out, cnt, n, st);
    RSG_CHECK_LAUNCH();
    int h = 0;
    RSG_CUDA(cudaMemcpyAsync(&h, cnt, sizeof(int), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    ar.used = mark;
    return h;
}

// The later-dense list buffer of the calls whose list does not fit in the
// arena, kept per host thread (see fof3d_device).
struct ListCache {
    void *p = nullptr;
    size_t bytes = 0;
};
static thread_local ListCache g_list_cache;

struct FofOut {
    int64_t num_p;
    int64_t nfofs;
};

// Device-resident 3D FOF.  d_in: caller particles (n); d_out: permuted
// particles; d_off/d_sz: groups (capacity n/2+1).
FofOut fof3d_device(Arena &ar, const rsg_particle *d_in, int64_t n64, const rsg_config &cfg,
                    rsg_particle *d_out, int64_t *d_off, int64_t *d_sz, cudaStream_t st) {
    FofOut res{0, 0};
    if (n64 <= 0) return res;
    if (n64 >= (1ll << 31) - 2) {
        set_error(RSG_ERR_ARGS, "3D FOF supports up to 2^31-2 particles");
        throw Failure();
    }
    int n = (int)n64;
    const int T = 256;
    Rec *recs = ar.get<Rec>(n);
    int *flags = ar.get<int>(8);
    RSG_CUDA(cudaMemsetAsync(flags, 0, sizeof(int) * 8, st));
    phase_mark(st, "");
    launch(k_make_recs, nblk(n, T), T, 0, st, d_in, n, recs, flags);
    int32_t *seg = ar.get<int32_t>(2);
    int32_t hseg[2] = {0, n};
    RSG_CUDA(cudaMemcpyAsync(seg, hseg, sizeof(hseg), cudaMemcpyHostToDevice, st));
    size_t mark = ar.used;
    Forest<3> F = build_forest<3, Rec>(ar, recs, n, seg, seg + 1, 1, n, 20, st);
    launch(k_dup_probe, nblk(n, T), T, 0, st, recs, d_in, n, flags + 1);
    int hflags[8];
    RSG_CUDA(cudaMemcpyAsync(hflags, flags, sizeof(hflags), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    if (hflags[0]) {
        set_error(RSG_ERR_INPUT, "non-finite particle coordinates");
        throw Failure();
    }
    if (hflags[1]) {
        int64_t *dn = ar.get<int64_t>(1);
        launch(k_dedupe_serial, 1, 1, 0, st, recs, d_in, n, dn);
        int64_t nn = 0;
        RSG_CUDA(cudaMemcpyAsync(&nn, dn, sizeof(nn), cudaMemcpyDeviceToHost, st));
        RSG_CUDA(cudaStreamSynchronize(st));
        n = (int)nn;
        hseg[1] = n;
        RSG_CUDA(cudaMemcpyAsync(seg, hseg, sizeof(hseg), cudaMemcpyHostToDevice, st));
        ar.used = mark;
        F = build_forest<3, Rec>(ar, recs, n, seg, seg + 1, 1, n, 20, st);
    }
    res.num_p = n;
    float r = (float)(cfg.avg_particle_spacing * cfg.fof_linking_length);
    float r2x = (float)(2.0 * (double)r);
    int *err = flags + 2;

    uint8_t *cnt = ar.get<uint8_t>(n);
    phase_mark(st, "fof.tree3d");
    launch(k_count_w, nblk(n, RSG_CNT_T), RSG_CNT_T, 0, st, F.nodes, recs, n, r, cnt, err);
    phase_mark(st, "fof.count");
    // dense particles (more than 16 neighbours), in tree order
    int *dense = ar.get<int>(n);
    int nd = select_where(ar, n, DFlag{cnt}, dense, st);
    // groups of 32 dense particles, their lists of later dense neighbours and
    // every particle's pending skippers
    const int ng = (nd + 31) / 32;
    int *skip = ar.get<int>(nd + 1);
    RSG_CUDA(cudaMemsetAsync(skip, 0, sizeof(int) * (nd + 1), st));
    // dense particles before every index
    int *dpfx = ar.get<int>(n + 1);
    {
        thrust::transform_iterator<DenseI, const uint8_t *, int> dit((const uint8_t *)cnt, DenseI{});
        size_t pb = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, pb, dit, dpfx, n + 1, st);
        size_t m0 = ar.used;
        void *pt = ar.take(pb + 256);
        cub::DeviceScan::ExclusiveSum(pt, pb, dit, dpfx, n + 1, st);
        ar.used = m0;
    }
    KahnList KL;
    KL.nd = nd;
    KL.skip = skip;
    KL.und = ar.get<unsigned>(ng + 1);
    int *diff = ar.get<int>(nd + 1);
    RSG_CUDA(cudaMemsetAsync(diff, 0, sizeof(int) * (nd + 1), st));
    size_t dsb = 0;
    cub::DeviceScan::InclusiveSum(nullptr, dsb, diff, diff, nd + 1, st);
    void *dst_tmp = ar.take(dsb + 256);
    KL.ng = ng;
    KL.icap = ng < (1 << 20) ? ng + 256 : 1 << 20;
    KL.items = ar.get<KahnItem>(KL.icap);
    for (int b = 0; b < 2; b++) {
        KL.fresh[b] = ar.get<unsigned>(ng + 1);
        RSG_CUDA(cudaMemsetAsync(KL.fresh[b], 0, sizeof(unsigned) * (ng + 1), st));
    }
    KL.ctl = ar.get<KahnCtl>(1);
    RSG_CUDA(cudaMemsetAsync(KL.ctl, 0, sizeof(KahnCtl), st));
    KL.G.nch = ar.get<int>(ng + 1);
    int64_t *gn = ar.get<int64_t>(ng + 1), *go = ar.get<int64_t>(ng + 1), *gm = ar.get<int64_t>(1);
    KL.off = go;
    size_t sb = 0, mb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, sb, gn, go, ng + 1, st);
    cub::DeviceReduce::Max(nullptr, mb, gn, gm, ng + 1, st);
    const size_t gtb = (sb > mb ? sb : mb) + 256;
    void *gtmp = ar.take(gtb);
    // {cursor, pairs}
    unsigned long long *tot = ar.get<unsigned long long>(2);
    RSG_CUDA(cudaMemsetAsync(tot, 0, 2 * sizeof(*tot), st));
    KL.G.cursor = (unsigned *)tot;
    // The lists go to the arena beside what the rest of the FOF takes from it
    // (< 256 B per particle: the label derivation and the partition sort).
    // Lists that do not fit (very dense snapshots) get an allocation of
    // their own, as large as free device memory allows (less 1 GiB, or room
    // for RSG_FOF_LIST_ENTRIES entries when that is set); when not all fit,
    // they are built and walked one chunk of groups at a time, chunks in
    // order.  A fixed arena holds the lists whole or fails.  That allocation
    // stays with the host thread for its later calls, as the arena does:
    // allocating and freeing tens of gigabytes costs tens of milliseconds,
    // and the free waits for the device.
    const char *lenv = getenv("RSG_FOF_LIST_ENTRIES");
    const int64_t lforce = lenv ? atoll(lenv) : 0;
    const size_t lat = (ar.used + 255) & ~(size_t)255;
    const size_t rest = ar.fixed ? 0 : (size_t)256 * n + (64u << 20);
    // a chunk, its place in the groups' table and in a step's queue
    const size_t each = sizeof(GChunk) + 2 * sizeof(uint2);
    int64_t fit = lat + rest + 1024 < ar.cap ? (int64_t)((ar.cap - lat - rest - 1024) / each) : 0;
    if (lforce > 0 && !ar.fixed) fit = 0;
    KL.G.cap = (int)std::min<int64_t>(fit, INT_MAX / 2);
    KL.G.pool = ar.get<GChunk>(KL.G.cap);
    const int TG = 128;
    auto gblk = [&](int groups) { return nblk((int64_t)groups * 32, TG); };
    launch(k_glist<true>, gblk(ng), TG, 0, st, F.nodes, recs, (const int *)dense, nd, 0, ng, r,
           (const uint8_t *)cnt, (const int *)dpfx, KL.G, skip, diff, tot + 1, err);
    if (nd > 0) cub::DeviceScan::InclusiveSum(dst_tmp, dsb, diff, diff, nd + 1, st);
    launch(k_kahn_init, nblk(nd, T), T, 0, st, nd, (const int *)diff, skip, KL.und);
    launch(k_gchunks, nblk(ng + 1, T), T, 0, st, (const int *)KL.G.nch, ng, gn);
    sb = mb = gtb;
    cub::DeviceScan::ExclusiveSum(gtmp, sb, gn, go, ng + 1, st);
    int64_t nch = 0, ne = 0;  // chunks that the lists take, pairs
    RSG_CUDA(cudaMemcpyAsync(&nch, go + ng, sizeof(nch), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaMemcpyAsync(&ne, tot + 1, sizeof(ne), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    // chunk boundaries: groups c[t] .. c[t+1], the chunks of their lists
    std::vector<int> cb_h(2, 0);
    std::vector<int64_t> lb_h(2, 0);
    cb_h[1] = ng;
    lb_h[1] = nch;
    const bool built = nch <= KL.G.cap;
    ar.used = lat;
    if (built) {
        ar.get<GChunk>(nch);
        KL.table = ar.get<uint2>(nch);
        KL.queue = ar.get<uint2>(nch);
    } else {
        if (ar.fixed) {
            set_error(RSG_ERR_LIMIT, "device arena exhausted (%lld neighbour list chunks, room "
                      "for %d)", (long long)nch, KL.G.cap);
            throw Failure();
        }
        ListCache &lc = g_list_cache;
        size_t fb = 0, tb = 0;
        RSG_CUDA(cudaMemGetInfo(&fb, &tb));
        fb += lc.bytes;  // the kept buffer is this call's to use
        int64_t avail = fb > ((size_t)1 << 30) ? (int64_t)((fb - ((size_t)1 << 30)) / each) : 0;
        if (lforce > 0) avail = lforce / RSG_GE;
        avail = std::min<int64_t>(avail, INT_MAX / 2);
        const int64_t lcap = std::min(avail, nch);
        const size_t need = each * (size_t)(lcap > 0 ? lcap : 1);
        if (lc.bytes < need) {
            if (lc.p) RSG_CUDA(cudaFree(lc.p));
            lc.p = nullptr;
            lc.bytes = 0;
            RSG_CUDA(cudaMalloc(&lc.p, need));
            lc.bytes = need;
        }
        KL.G.pool = (GChunk *)lc.p;
        KL.G.cap = (int)lcap;
        KL.table = (uint2 *)(KL.G.pool + lcap);
        KL.queue = KL.table + lcap;
        if (lcap < nch) {
            int64_t maxl = 0;
            cub::DeviceReduce::Max(gtmp, mb, gn, gm, ng + 1, st);
            RSG_CUDA(cudaMemcpyAsync(&maxl, gm, sizeof(maxl), cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            const int64_t step = lcap - maxl;
            if (step < maxl || step * RSG_GE < (1 << 12)) {
                set_error(RSG_ERR_LIMIT, "later-dense lists need more device memory than is free");
                throw Failure();
            }
            const int64_t m = (nch + step - 1) / step;  // chunks
            int *cbd = ar.get<int>(m + 1);
            thrust::transform_iterator<ChunkTarget, thrust::counting_iterator<int64_t>, int64_t> tgt(
                thrust::counting_iterator<int64_t>(0), ChunkTarget{step});
            thrust::lower_bound(thrust::cuda::par_nosync.on(st), (const int64_t *)go, (const int64_t *)go + ng + 1, tgt,
                                tgt + (m - 1), cbd);
            cb_h.assign(m + 1, 0);
            lb_h.assign(m + 1, 0);
            RSG_CUDA(cudaMemcpyAsync(cb_h.data() + 1, cbd, sizeof(int) * (m - 1),
                                     cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            cb_h[m] = ng;
            for (int64_t t = 0; t <= m; t++)
                RSG_CUDA(cudaMemcpyAsync(&lb_h[t], go + cb_h[t], sizeof(int64_t),
                                         cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            for (int64_t t = 0; t < m; t++)
                if (lb_h[t + 1] - lb_h[t] > lcap) {
                    set_error(RSG_ERR_LIMIT, "later-dense list chunk exceeds its buffer");
                    throw Failure();
                }
        }
    }
    const int nchunks = (int)cb_h.size() - 1;
    // every step but a chunk's last decides a particle
    const int limit = nd + nchunks + 2;
    int kres = 0;
    RSG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&kres, k_kahn, 256, 0));
    const int TK = 256;
    const int GK = (int)std::min<int64_t>((int64_t)(kres > 0 ? kres : 1) * sm_count(),
                                          nch * 32 / TK + 1);
    const int GN = std::min<int>(4 * sm_count(), nblk(ng, TK));
    // the frontier steps run as a device-side graph loop; with per-launch
    // event timing, and in fixed storage (instantiating a graph may take
    // device memory), the host drives the same steps, in fixed storage a few
    // between reads of the state
    const bool host_loop = launch_stats().selecting || ar.fixed;
    const int burst = launch_stats().selecting ? 1 : 8;
    KahnGraph G;
    if (!host_loop && nd > 0) G.build(GK, GN, TK, KL, limit);
    for (int t = 0; t < nchunks; t++) {
        const int c0 = cb_h[t], c1 = cb_h[t + 1];
        if (c1 <= c0) continue;
        if (!built) {
            RSG_CUDA(cudaMemsetAsync(KL.G.cursor, 0, sizeof(int), st));
            launch(k_glist<false>, gblk(c1 - c0), TG, 0, st, F.nodes, recs, (const int *)dense, nd,
                   c0, c1, r, (const uint8_t *)cnt, (const int *)dpfx, KL.G, skip, diff, tot + 1,
                   err);
        }
        const int lc = (int)(lb_h[t + 1] - lb_h[t]);
        launch(k_gtable, nblk(lc, T), T, 0, st, (const GChunk *)KL.G.pool, lc, KL.off, lb_h[t],
               KL.table);
        launch(k_kahn_start, 1, 1, 0, st, KL.ctl, c0, c1);
        launch(k_kahn_chunk, GN, TK, 0, st, KL);
        if (!host_loop) {
            G.run(st);
            continue;
        }
        for (;;) {
            for (int b = 0; b < burst; b++) {
                launch(k_kahn, GK, TK, 0, st, KL);
                launch(k_kahn_wide, GK, TK, 0, st, KL);
                launch(k_kahn_next, GN, TK, 0, st, KL, limit, (int)(burst == 1));
            }
            KahnCtl hc;
            RSG_CUDA(cudaMemcpyAsync(&hc, KL.ctl, sizeof(hc), cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            if (!hc.more || hc.hit) break;
        }
    }
    KahnCtl kc;
    RSG_CUDA(cudaMemcpyAsync(&kc, KL.ctl, sizeof(kc), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    if (kc.hit || kc.decided != nd) {
        set_error(RSG_ERR_LIMIT, "3D FOF seed selection left %d of %d dense particles undecided",
                  nd - kc.decided, nd);
        throw Failure();
    }
    if (G.e) launch_stats().launches += 3 * (int64_t)kc.iters;
    phase_mark(st, "fof.elist");
    // non-dense particles: state 0 (never seeds)
    uint8_t *state = ar.get<uint8_t>(n);
    RSG_CUDA(cudaMemsetAsync(state, 0, n, st));
    launch(k_state8, nblk(nd, T), T, 0, st, (const int *)dense, nd, (const int *)skip, state);
    phase_mark(st, "fof.seeds");
    if (getenv("RSG_TIMING"))
        fprintf(stderr, "  [fof] dense %d, dense pairs %lld in %d chunk(s), frontier steps %d\n",
                nd, (long long)ne, nchunks, kc.iters);
    last_stats()[RSG_STAT_DENSE] = nd;
    last_stats()[RSG_STAT_DENSE_PAIRS] = ne;
    last_stats()[RSG_STAT_SEED_STEPS] = kc.iters;
    int *seeds = ar.get<int>(nd + 1);
    const int nseed = select_where(ar, n, SeedFlag{state}, seeds, st);
    const int TS = RSG_SEED_WARPS * 32;
    const int GS = (int)nblk((int64_t)nseed * 32, TS);
    uint8_t *skipped = ar.get<uint8_t>(n);
    RSG_CUDA(cudaMemsetAsync(skipped, 0, n, st));
    // labels exactly as the reference's union-find leaves them (uflabels.cuh)
    int *gtime = ar.get<int>(n);
    RSG_CUDA(cudaMemsetAsync(gtime, 0x7f, sizeof(int) * n, st));  // 0x7f7f7f7f: never
    launch(k_seed_mark_w, GS, TS, 0, st, F.nodes, recs, (const int *)seeds, nseed, r, skipped,
           gtime, err);
    launch(k_gtime_r, nblk(n, T), T, 0, st, F.nodes, recs, n, r, (const uint8_t *)cnt,
           (const uint8_t *)skipped, (const uint8_t *)state, gtime, err);
    int32_t *ptr = ar.get<int32_t>(n), *sfid = ar.get<int32_t>(n), *nsc = ar.get<int32_t>(n + 1);
    launch(k_fptr3, nblk(n, T), T, 0, st, F.nodes, recs, n, r, (const uint8_t *)cnt,
           (const uint8_t *)skipped, (const uint8_t *)state, (const int *)gtime, ptr, err);
    launch(k_fptr_seed_w, GS, TS, 0, st, F.nodes, recs, (const int *)seeds, nseed, r,
           (const int *)gtime, ptr, err);
    RSG_CHECK_LAUNCH();
    int64_t S = uf_resolve(ar, ptr, n, sfid, nsc, st);
    phase_mark(st, "fof.first_links");
    // candidate merges, in time order
    unsigned long long *ccount = ar.get<unsigned long long>(1);
    int64_t ccap = (int64_t)n / 2 + 1024;
    size_t cmark = ar.used;
    uint64_t *ckey = nullptr;
    int32_t *cF = nullptr, *cW = nullptr;
    unsigned long long hc = 0;
    int32_t *lab0 = ar.get<int32_t>(n);
    {
        // lab0[j] = f(g(j)): the set j joined when it was labelled
        launch(k_lab3, nblk(n, T), T, 0, st, (const int *)gtime, n, (const int32_t *)sfid,
               (const int32_t *)nullptr, lab0);
    }
    cmark = ar.used;
    for (int pass = 0; pass < 2; pass++) {
        ar.used = cmark;
        ckey = ar.get<uint64_t>(ccap);
        cF = ar.get<int32_t>(ccap);
        cW = ar.get<int32_t>(ccap);
        RSG_CUDA(cudaMemsetAsync(ccount, 0, sizeof(unsigned long long), st));
        launch(k_cand3, nblk(n, T), T, 0, st, F.nodes, recs, n, r, (const uint8_t *)cnt,
               (const uint8_t *)skipped, (const uint8_t *)state, (const int *)gtime,
               (const int32_t *)lab0, (const int32_t *)sfid, ccap, ccount, ckey, cF, cW, err);
        launch(k_cand_seed_w, GS, TS, 0, st, F.nodes, recs, (const int *)seeds, nseed, r, r2x,
               (const int *)gtime, (const int32_t *)lab0, (const int32_t *)sfid, ccap, ccount,
               ckey, cF, cW, err);
        RSG_CHECK_LAUNCH();
        RSG_CUDA(cudaMemcpyAsync(&hc, ccount, sizeof(hc), cudaMemcpyDeviceToHost, st));
        RSG_CUDA(cudaStreamSynchronize(st));
        if ((int64_t)hc <= ccap) break;
        ccap = (int64_t)hc;  // exact size, second pass
    }
    int64_t nc = (int64_t)hc;
    if (nc >= 0x7f7f7f7f) {
        set_error(RSG_ERR_LIMIT, "3D FOF: too many label merges (%lld)", (long long)nc);
        throw Failure();
    }
    int32_t *cF2 = ar.get<int32_t>(nc + 1), *cW2 = ar.get<int32_t>(nc + 1);
    if (nc > 0) {
        uint64_t *ckey2 = ar.get<uint64_t>(nc);
        int32_t *cidx = ar.get<int32_t>(nc), *cidx2 = ar.get<int32_t>(nc);
        launch(k_iota, nblk(nc, T), T, 0, st, cidx, (int)nc);
        size_t sb = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, sb, ckey, ckey2, cidx, cidx2, (int)nc, 0, 64, st);
        void *stmp = ar.take(sb + 256);
        cub::DeviceRadixSort::SortPairs(stmp, sb, ckey, ckey2, cidx, cidx2, (int)nc, 0, 64, st);
        launch(k_take2, nblk(nc, T), T, 0, st, (const int32_t *)cidx2, (int)nc,
               (const int32_t *)cF, (const int32_t *)cW, cF2, cW2);
    }
    int32_t *sroot = ar.get<int32_t>(S + 1);
    uf_roots(ar, cF2, cW2, nc, S, sroot, st);
    int32_t *lab = ar.get<int32_t>(n);
    launch(k_lab3, nblk(n, T), T, 0, st, (const int *)gtime, n, (const int32_t *)sfid,
           (const int32_t *)sroot, lab);
    RSG_CHECK_LAUNCH();
    phase_mark(st, "fof.labels");
    // the reference's partition sort by label (src/fof.c:184-224), then the
    // groups of build_fullfofs (src/fof.c:226-255)
    {
        std::vector<int32_t> s0(1, 0), n0(1, n);
        partition_sort_labels<Rec>(ar, recs, lab, n, s0, n0, st);
    }
    launch(k_gather_out, nblk(n, T), T, 0, st, (const Rec *)recs, d_in, n, d_out);
    int *head = ar.get<int>(n), *hpos = ar.get<int>(n), *nh = ar.get<int>(1);
    launch(k_run_heads3, nblk(n, T), T, 0, st, (const int32_t *)lab, n, head);
    size_t hb = 0;
    cub::DeviceSelect::Flagged(nullptr, hb, thrust::counting_iterator<int>(0), head, hpos, nh, n,
                               st);
    void *htmp = ar.take(hb + 256);
    cub::DeviceSelect::Flagged(htmp, hb, thrust::counting_iterator<int>(0), head, hpos, nh, n, st);
    int64_t *roff = ar.get<int64_t>(n / 2 + 1), *rsz = ar.get<int64_t>(n / 2 + 1);
    int32_t *keep = ar.get<int32_t>(n / 2 + 1);
    launch(k_runs3, nblk(n / 2 + 1, T), T, 0, st, (const int *)hpos, (const int *)nh, n,
           (int64_t)cfg.min_halo_particles, roff, rsz, keep);
    int hnh = 0;
    RSG_CUDA(cudaMemcpyAsync(&hnh, nh, sizeof(int), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    int *nk = ar.get<int>(1);
    size_t kb = 0;
    cub::DeviceSelect::Flagged(nullptr, kb, roff, keep, d_off, nk, hnh, st);
    void *ktmp = ar.take(kb + 256);
    cub::DeviceSelect::Flagged(ktmp, kb, roff, keep, d_off, nk, hnh, st);
    cub::DeviceSelect::Flagged(ktmp, kb, rsz, keep, d_sz, nk, hnh, st);
    RSG_CHECK_LAUNCH();
    RSG_CUDA(cudaMemcpyAsync(&hnh, nk, sizeof(int), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaMemcpyAsync(hflags, flags, sizeof(hflags), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    if (hflags[2]) {
        set_error(RSG_ERR_LIMIT, "kd-tree traversal stack overflow");
        throw Failure();
    }
    res.nfofs = hnh;
    last_stats()[RSG_STAT_PARTICLES] = n;
    last_stats()[RSG_STAT_GROUPS] = hnh;
    phase_mark(st, "fof.output");
    return res;
}

}  // namespace rsg
