// Level-synchronous kd-forest build on the GPU that reproduces, element for
// element, the in-place permutation of the reference's fast3tree build
// (src/fast3tree.c:736-908).
//
// The reference splits a node [0, n) at lim = 0.5f * (max + min) of its
// widest dimension with a two-pointer swap: a front pointer i walks up and,
// whenever p[i] > lim, swaps it with the back pointer j, which walks down.
// With m = #(p <= lim) the result is, in closed form:
//   * small elements before m stay put;
//   * the t-th big element before m (rank t, ascending) ends at n-1 (t = 0)
//     or one slot below the (t-1)-th small element after m counted from the
//     back;
//   * the t-th small element after m counted from the back fills the slot of
//     the t-th big element before m;
//   * big elements above the last consumed back position move down one;
//   * if the untouched tail [m, pos_last) holds two or more elements, it is
//     rotated down by one (the front pointer stops at m and swaps it with
//     each tail element in turn).
// Every element's destination is therefore a function of per-node prefix
// counts of the "big" flag, which are kept as bits with the counts before
// every word and tile (RankBits) for all nodes of a level at once.  Degenerate nodes (max == min on the split dimension) get
// lim = +inf so nothing moves, as in the reference's early return.
#pragma once
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <vector>

#include "common.cuh"

namespace rsg {

template <class RecT, int D>
struct PosOf;
template <int D>
struct PosOf<Rec, D> {
    __device__ static float get(const Rec &r, int d) { return r.pos[d]; }
};

struct PotRec {  // struct potential (src/potential.h:7-21), 48 bytes
    float pos[6], r2;
    float pad;
    double pe;
    float ke;
    int32_t flags;
};
static_assert(sizeof(PotRec) == 48, "PotRec layout");
template <int D>
struct PosOf<PotRec, D> {
    __device__ static float get(const PotRec &r, int d) { return r.pos[d]; }
};

struct MetricRec {  // struct halo_metric (src/subhalo_metric.h): pos[4] + target
    float pos[4];
    int32_t target;
    int32_t pad[3];
};
template <int D>
struct PosOf<MetricRec, D> {
    __device__ static float get(const MetricRec &r, int d) { return r.pos[d]; }
};

#define RSG_FOREST_LEVELS 4096  // deepest build accepted

// Device-side state of a forest build, so that levels run back to back
// without a host round trip; the host reads it every few levels.
struct LevelState {
    int32_t nnodes;  // nodes created so far
    int32_t err;     // 1: node capacity exceeded, 2: too many levels
    int32_t nsub[2]; // subtrees listed for each size class of k_sub_build
    int32_t ncopy;   // unsplit nodes whose records must be copied to the output
    int32_t pad[3];
    int32_t nact[RSG_FOREST_LEVELS + 2];  // nodes that level l splits
};
// A subtree that one block builds (k_sub_build): its root, the root's level
// and the buffer that holds its records.
struct SubRoot {
    int32_t node, level, src, pad;
};
// A node that a level splits.
struct ActNode {
    int32_t node, start, n, div;
    float lim;
    int32_t m, q;     // records at or below lim; big ones among the first m
    int32_t rs;       // big records before start
    int32_t next[2];  // the halves' places in the next level, -1: none
};

template <int D>
struct Forest {
    KNode<D> *nodes = nullptr;  // nodes[t] is the root of tree t
    int32_t nnodes = 0;
    int32_t ntrees = 0;
};

// ---- ranks ----------------------------------------------------------------
// The "big" flags of a level as bits, with the set bits before every word of
// a tile (2,048 elements) and before every tile: the number of flags before
// any element takes three reads.
#define RSG_TILE 2048
struct RankBits {
    uint32_t *bits;
    uint16_t *wpre;
    int32_t *tpre;  // counts, then their exclusive sums
    __device__ __forceinline__ int rank(int64_t x) const {
        return tpre[x / RSG_TILE] + wpre[x >> 5] +
               __popc(bits[x >> 5] & ((1u << (x & 31)) - 1u));
    }
    __device__ __forceinline__ bool big(int64_t x) const { return (bits[x >> 5] >> (x & 31)) & 1u; }
};
inline int64_t rank_tiles(int64_t n) { return (n + RSG_TILE - 1) / RSG_TILE; }
inline RankBits rank_alloc(Arena &ar, int64_t n, cudaStream_t st) {
    const int64_t t = rank_tiles(n);
    RankBits R;
    R.bits = ar.get<uint32_t>(t * (RSG_TILE / 32) + 1);
    R.wpre = ar.get<uint16_t>(t * (RSG_TILE / 32) + 1);
    R.tpre = ar.get<int32_t>(t + 1);
    // the word and tile after the last one (rank(n) with n a multiple of a tile)
    RSG_CUDA(cudaMemsetAsync(R.bits + t * (RSG_TILE / 32), 0, 4, st));
    RSG_CUDA(cudaMemsetAsync(R.wpre + t * (RSG_TILE / 32), 0, 2, st));
    return R;
}
// Stores a block's tile: warp w of eight holds words 8 w .. 8 w + 7 of it, the
// word 8 w + l in lane l < 8.  All threads of the block call it.
__device__ __forceinline__ void rank_store(const RankBits &R, int64_t tile, uint32_t word) {
    __shared__ int wtot[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int v = lane < 8 ? __popc(word) : 0;
    int incl = v;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 7) wtot[w] = incl;
    __syncthreads();
    int off = 0, tot = 0;
    for (int i = 0; i < 8; i++) {
        if (i < w) off += wtot[i];
        tot += wtot[i];
    }
    if (lane < 8) {
        const int64_t at = tile * (RSG_TILE / 32) + 8 * w + lane;
        R.bits[at] = word;
        R.wpre[at] = (uint16_t)(off + incl - v);
    }
    if (threadIdx.x == 0) R.tpre[tile] = tot;
}
// tpre[0 .. nt) to its exclusive sums, tpre[nt] the total (one block).
__global__ void k_rank_scan(int32_t *tpre, int32_t nt);
// Destination of element l of a segment of n (see the closed form above):
// br big elements before it, m small ones in all, q big ones among the first
// m, fb and bs the tables from the segment's start.
__device__ __forceinline__ int swap_dest(int l, int n, bool big, int br, int m, int q,
                                         const int32_t *fb, const int32_t *bs) {
    if (!big && l < m) return l;
    if (big && l < m) return (br == 0) ? n - 1 : bs[br - 1] - 1;
    if (!big) return fb[m - 1 - (l - br)];
    const int pos_last = (q > 0) ? bs[q - 1] : n;
    if (l > pos_last) return l - 1;
    if (pos_last - m >= 2) return (l == m) ? pos_last - 1 : l - 1;
    return l;
}
__device__ __forceinline__ void swap_tables(int l, bool big, int br, int m, int32_t *fb,
                                            int32_t *bs) {
    if (big && l < m) fb[br] = l;
    if (!big && l >= m) bs[m - 1 - (l - br)] = l;
}

// ---- kernels ------------------------------------------------------------

// Lists a subtree of n records for k_sub_build: class 0 (n <= sub0) from the
// front of `subs`, class 1 from its back.
__device__ __forceinline__ void list_sub(SubRoot *subs, int32_t nsubs, LevelState *ls, int sub0,
                                         int32_t node, int32_t n, int32_t level, int32_t src) {
    const int c = n > sub0;
    const int at = atomicAdd(&ls->nsub[c], 1);
    subs[c ? nsubs - 1 - at : at] = SubRoot{node, level, src, 0};
}
// Roots: trees of more than `sub` records are the first level's nodes, the
// others a block's each.
template <int D>
__global__ void k_roots(const int32_t *rstart, const int32_t *rn, int32_t ntrees, int sub, int sub0,
                        KNode<D> *nodes, ActNode *act, unsigned *cbox, int32_t *slot, SubRoot *subs,
                        int32_t nsubs, LevelState *ls) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntrees) return;
    KNode<D> &nd = nodes[t];
    nd.start = rstart[t];
    nd.n = rn[t];
    nd.div = -1;
    nd.left = -1;
    nd.parent = -1;
    nd.tree = t;
    slot[t] = -1;
    if (nd.n <= sub) {
        list_sub(subs, nsubs, ls, sub0, t, nd.n, 0, 0);
        return;
    }
    const int k = atomicAdd(&ls->nact[0], 1);
    slot[t] = k;
    ActNode a = {};
    a.node = t;
    a.start = nd.start;
    a.n = nd.n;
    a.lim = __int_as_float(0x7f800000);  // the first pass only takes the box
    act[k] = a;
    for (int d = 0; d < 2 * D; d++)
        cbox[(int64_t)k * 4 * D + d] = cbox[(int64_t)k * 4 * D + 2 * D + d] =
            d < D ? 0xffffffffu : 0u;
}
__global__ void k_root_owner(const int32_t *rstart, const int32_t *rn, int32_t ntrees,
                             const int32_t *slot, int32_t *owner);

// Split dimension and limit of a node of box b (mn then mx; src/fast3tree.c:
// 736-757).
template <int D>
__device__ __forceinline__ void split_of(const float *b, int32_t &div, float &lim) {
    int dim = D - 1;
    float dmax = fsub(b[2 * D - 1], b[D - 1]);
#pragma unroll
    for (int i = 0; i < D - 1; i++) {
        float d2 = fsub(b[D + i], b[i]);
        if (d2 > dmax) {
            dmax = d2;
            dim = i;
        }
    }
    float l = fmul(0.5f, fadd(b[D + dim], b[dim]));
    if (b[D + dim] == b[dim]) l = __int_as_float(0x7f800000);  // +inf: nothing moves
    div = dim;
    lim = l;
}
// The roots' boxes (gathered as a half each) and splits.
template <int D>
__global__ void k_root_split(KNode<D> *nodes, ActNode *act, unsigned *cbox, const LevelState *ls) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ls->nact[0]) return;
    float b[2 * D];
    unsigned *c = cbox + (int64_t)k * 4 * D;
    for (int d = 0; d < 2 * D; d++) {
        b[d] = ord2f(c[d]);
        c[d] = d < D ? 0xffffffffu : 0u;
    }
    for (int d = 0; d < D; d++) {
        nodes[act[k].node].mn[d] = b[d];
        nodes[act[k].node].mx[d] = b[D + d];
    }
    split_of<D>(b, act[k].div, act[k].lim);
}

// A warp of the level passes has 256 consecutive elements.  The segments of a
// level are intervals, and where they hold at least 256 elements each
// (`wide`) a stretch whose first and last element have one owner has no
// other: the pass then reads two owners instead of 256, and its loads do not
// wait for them.  Returns that owner, or -2 where the elements have to be
// asked one by one.
#define RSG_STRETCH 256
__device__ __forceinline__ int stretch_owner(const int32_t *owner, int64_t first, int64_t n,
                                             bool wide) {
    if (!wide || first >= n) return first >= n ? -1 : -2;
    const int64_t last = first + RSG_STRETCH - 1 < n ? first + RSG_STRETCH - 1 : n - 1;
    const int a = owner[first], b = owner[last];
    return a == b ? a : -2;
}

// One pass over the records of a level: the "big" flags as rank bits, and the
// boxes of both halves of every node.  Stretches of one node (nearly all) are
// reduced in registers, and a block of one node sends its atomics once (at the
// upper levels every warp of the grid would meet at the same few words); the
// other stretches send an atomic per value.
template <int D, class RecT>
__global__ void __launch_bounds__(256) k_lv_flags(const RecT *recs, int64_t nrec,
                                                  const int32_t *owner, const ActNode *act,
                                                  unsigned *cbox, RankBits R, bool wide) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t first = blockIdx.x * (int64_t)RSG_TILE + (threadIdx.x >> 5) * RSG_STRETCH;
    const int64_t i0 = first + lane;
    const int a0 = stretch_owner(owner, first, nrec, wide);
    __shared__ unsigned part[8][4 * D];
    __shared__ int a_s;
    if (threadIdx.x == 0) a_s = a0;
    __syncthreads();
    const bool whole = __syncthreads_and(a0 >= 0 && a0 == a_s);
    uint32_t word = 0;
    if (a0 >= 0) {
        const int dim = act[a0].div;
        const float lim = act[a0].lim;
        unsigned lo[2][D], hi[2][D];
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int d = 0; d < D; d++) {
                lo[h][d] = 0xffffffffu;
                hi[h][d] = 0u;
            }
#pragma unroll 4
        for (int u = 0; u < 8; u++) {
            const int64_t i = i0 + 32 * u;
            const bool on = i < nrec;
            float p[D];
            const RecT &r = recs[on ? i : nrec - 1];
#pragma unroll
            for (int d = 0; d < D; d++) p[d] = PosOf<RecT, D>::get(r, d);
            float v = p[0];
#pragma unroll
            for (int d = 1; d < D; d++) v = dim == d ? p[d] : v;
            const bool big = on && v > lim;
            const unsigned b = __ballot_sync(FULL, big);
            if (lane == u) word = b;
#pragma unroll
            for (int d = 0; d < D; d++) {
                const unsigned o = f2ord(p[d]);
                const unsigned o0 = on && !big ? o : 0xffffffffu, o1 = big ? o : 0xffffffffu;
                lo[0][d] = min(lo[0][d], o0);
                lo[1][d] = min(lo[1][d], o1);
                hi[0][d] = max(hi[0][d], on && !big ? o : 0u);
                hi[1][d] = max(hi[1][d], big ? o : 0u);
            }
        }
        unsigned *c = cbox + (int64_t)a0 * 4 * D;
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int d = 0; d < D; d++) {
                const unsigned a = __reduce_min_sync(FULL, lo[h][d]);
                const unsigned b = __reduce_max_sync(FULL, hi[h][d]);
                if (lane == 0 && whole) {
                    part[threadIdx.x >> 5][h * 2 * D + d] = a;
                    part[threadIdx.x >> 5][h * 2 * D + D + d] = b;
                } else if (lane == 0 && a <= b) {  // the half has a record
                    atomicMin(c + h * 2 * D + d, a);
                    atomicMax(c + h * 2 * D + D + d, b);
                }
            }
    } else if (a0 == -2) {
#pragma unroll 1
        for (int u = 0; u < 8; u++) {
            const int64_t i = i0 + 32 * u;
            const int a = i < nrec ? owner[i] : -1;
            float p[D];
            bool big = false;
            if (a >= 0) {
#pragma unroll
                for (int d = 0; d < D; d++) p[d] = PosOf<RecT, D>::get(recs[i], d);
                const int dim = act[a].div;
                float v = p[0];
#pragma unroll
                for (int d = 1; d < D; d++) v = dim == d ? p[d] : v;
                big = v > act[a].lim;
                unsigned *c = cbox + (int64_t)a * 4 * D + (big ? 2 * D : 0);
#pragma unroll
                for (int d = 0; d < D; d++) {
                    const unsigned o = f2ord(p[d]);
                    atomicMin(c + d, o);
                    atomicMax(c + D + d, o);
                }
            }
            const unsigned b = __ballot_sync(FULL, big);
            if (lane == u) word = b;
        }
    }
    rank_store(R, blockIdx.x, word);  // holds a block barrier after the loop above
    if (whole && threadIdx.x < 4 * D) {
        const bool mn = threadIdx.x % (2 * D) < D;
        unsigned v = part[0][threadIdx.x];
        for (int w = 1; w < 8; w++)
            v = mn ? min(v, part[w][threadIdx.x]) : max(v, part[w][threadIdx.x]);
        unsigned *c = cbox + (int64_t)a0 * 4 * D + threadIdx.x;
        if (mn) atomicMin(c, v);
        else atomicMax(c, v);
    }
}

// Split bookkeeping of a level (src/fast3tree.c:798-846): counts, children
// with their boxes for nodes with 0 < m < n (the rest become leaves), and
// where each child goes on: above `sub` records to the next level, above
// `leaf` to the block-built subtrees, else it is a leaf.  The level writes
// buffer `dst`; leaves and unsplit nodes that end up in the scratch buffer
// (dst 1) are listed for a copy, a child with the subtrees (a block copies
// it), an unsplit node as a segment.  Children are numbered as the threads
// take them: nothing depends on the order.
template <int D>
__global__ void k_lv_nodes(KNode<D> *nodes, ActNode *act, ActNode *nxt, const unsigned *cbox,
                           unsigned *cnext, LevelState *ls, RankBits R, int32_t level, int32_t cap,
                           int leaf, int sub, int sub0, int dst, SubRoot *subs, int32_t nsubs,
                           int2 *copies) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ls->nact[level - 1]) return;
    ActNode &A = act[k];
    const int s = A.start, n = A.n;
    const int rs = R.rank(s);
    const int m = n - (R.rank((int64_t)s + n) - rs);
    A.m = m;
    A.q = R.rank((int64_t)s + m) - rs;
    A.rs = rs;
    A.next[0] = A.next[1] = -1;
    KNode<D> &nd = nodes[A.node];
    int l = -1;
    if (m > 0 && m < n) {
        l = atomicAdd(&ls->nnodes, 2);
        if (l > cap - 2) {
            ls->err = 1;
            l = -1;
        }
    }
    if (l < 0) {
        nd.div = -1;
        nd.left = -1;
        if (dst) copies[atomicAdd(&ls->ncopy, 1)] = make_int2(s, n);
        return;
    }
    nd.div = A.div;
    nd.left = l;
    const unsigned *c = cbox + (int64_t)k * 4 * D;
    for (int h = 0; h < 2; h++) {
        float b[2 * D];
        for (int d = 0; d < 2 * D; d++) b[d] = ord2f(c[h * 2 * D + d]);
        KNode<D> ch;
        ch.start = s + (h ? m : 0);
        ch.n = h ? n - m : m;
        ch.div = -1;
        ch.left = -1;
        ch.parent = A.node;
        ch.tree = nd.tree;
        for (int d = 0; d < D; d++) {
            ch.mn[d] = b[d];
            ch.mx[d] = b[D + d];
        }
        nodes[l + h] = ch;
        if (ch.n > sub) {
            const int j = atomicAdd(&ls->nact[level], 1);
            A.next[h] = j;
            ActNode x = {};
            x.node = l + h;
            x.start = ch.start;
            x.n = ch.n;
            split_of<D>(b, x.div, x.lim);
            nxt[j] = x;
            for (int d = 0; d < 2 * D; d++)
                cnext[(int64_t)j * 4 * D + d] = cnext[(int64_t)j * 4 * D + 2 * D + d] =
                    d < D ? 0xffffffffu : 0u;
        } else if (ch.n > leaf || dst) {
            list_sub(subs, nsubs, ls, sub0, l + h, ch.n, level, dst);
        }
    }
}
// The tables of the records that change sides (see stretch_owner).
static __global__ void __launch_bounds__(256) k_lv_tables(int64_t nrec, const int32_t *owner,
                                                          const ActNode *act, RankBits R,
                                                          int32_t *fb, int32_t *bs, bool wide) {
    const int lane = threadIdx.x & 31;
    const int64_t first = blockIdx.x * (int64_t)RSG_TILE + (threadIdx.x >> 5) * RSG_STRETCH;
    const int a0 = stretch_owner(owner, first, nrec, wide);
    if (a0 == -1) return;
#pragma unroll 1
    for (int u = 0; u < 8; u++) {
        const int64_t i = first + 32 * u + lane;
        if (i >= nrec) return;
        const int k = a0 >= 0 ? a0 : owner[i];
        if (k < 0) continue;
        const ActNode &A = act[k];
        swap_tables((int)(i - A.start), R.big(i), R.rank(i) - A.rs, A.m, fb + A.start,
                    bs + A.start);
    }
}
// Records to their places; a place then belongs to the half it lies in.
template <class RecT>
__global__ void __launch_bounds__(256) k_lv_scatter(int64_t nrec, int32_t *owner,
                                                    const ActNode *act, RankBits R,
                                                    const int32_t *fb, const int32_t *bs,
                                                    const RecT *src, RecT *dst, bool wide) {
    const int lane = threadIdx.x & 31;
    const int64_t first = blockIdx.x * (int64_t)RSG_TILE + (threadIdx.x >> 5) * RSG_STRETCH;
    const int a0 = stretch_owner(owner, first, nrec, wide);
    __syncwarp();  // every lane has read the owners that are written below
    if (a0 == -1) return;
    ActNode A;
    if (a0 >= 0) A = act[a0];
#pragma unroll 2
    for (int u = 0; u < 8; u++) {
        const int64_t i = first + 32 * u + lane;
        if (i >= nrec) return;
        if (a0 < 0) {
            const int k = owner[i];
            if (k < 0) continue;
            A = act[k];
        }
        const RecT r = src[i];
        const int l = (int)(i - A.start);
        const int d = swap_dest(l, A.n, R.big(i), R.rank(i) - A.rs, A.m, A.q, fb + A.start,
                                bs + A.start);
        dst[A.start + d] = r;
        owner[i] = A.next[l >= A.m];
    }
}
// Segments (x records from x.x, x.y of them) copied as they are.
template <class RecT>
__global__ void k_copy_segs(const int2 *segs, const RecT *src, RecT *dst) {
    const int2 g = segs[blockIdx.x];
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < g.y; i += gridDim.y * blockDim.x)
        dst[g.x + i] = src[g.x + i];
}

// Builds a kd-forest over recs[0..nrec) whose trees are the segments
// (rstart[t], rn[t]) (device arrays).  Elements outside every segment are
// left alone.  `recs` is permuted in place.  Returns the forest; node
// storage comes from the arena.
template <int D, class RecT>
Forest<D> build_forest(Arena &ar, RecT *recs, int64_t nrec, const int32_t *rstart,
                       const int32_t *rn, int32_t ntrees, int64_t n_in_trees, int leaf,
                       cudaStream_t st);

}  // namespace rsg
