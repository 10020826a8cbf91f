// Exact GPU version of partition_sort_particles (src/fof.c:184-224): each
// segment is split at the midpoint of its label range with the same
// two-pointer swap that the kd-tree build uses (closed form in kdtree.cuh),
// then both halves recurse.  Segments above RSG_LS_SUB elements are split
// level-synchronously, many at once; what is left of a segment at or below
// that size is finished by one block in shared memory.
#pragma once
#include "hosttables.cuh"
#include "kdtree.cuh"

namespace rsg {

#define RSG_LS_SUB0 256  // largest segment of the small blocks
#define RSG_LS_SUB 2048  // largest segment one block finishes

// A segment that a round splits.
struct LsNode {
    int32_t start, n, pivot;
    int32_t m, q;     // elements at or below the pivot; big ones among the first m
    int32_t rs;       // big elements before start
    int32_t next[2];  // the halves' places in the next round, -1: none
};
// A segment one block finishes, and the buffer that holds it.
struct LsSub {
    int32_t start, n, src, pad;
};
// Device-side state of a sort.
#define RSG_LS_ROUNDS 200
struct LsState {
    int32_t nsub[2];  // segments listed for the two classes of block
    int32_t ncopy;    // finished segments to be copied to the output
    int32_t pad;
    int32_t ns[RSG_LS_ROUNDS + 2];  // segments that round r splits
};

// pivot = min + (max - min) / 2 (src/fof.c:201)
__device__ __forceinline__ int32_t ls_pivot(int64_t lo, int64_t hi) {
    return (int32_t)(lo + (hi - lo) / 2);
}
// Roots: segments above RSG_LS_SUB elements, in ascending order.  The first
// pass only takes their label ranges (no label is above the pivot).
static __global__ void k_ls_roots(const int2 *segs, int32_t ns, LsNode *act, int32_t *range) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns) return;
    LsNode a = {};
    a.start = segs[k].x;
    a.n = segs[k].y;
    a.pivot = 0x7fffffff;
    act[k] = a;
    for (int h = 0; h < 2; h++) {
        range[4 * k + 2 * h] = 0x7fffffff;
        range[4 * k + 2 * h + 1] = (int32_t)0x80000000;
    }
}
static __global__ void k_ls_owner(const LsNode *act, int32_t *owner) {
    const LsNode &a = act[blockIdx.x];
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < a.n; i += gridDim.y * blockDim.x)
        owner[a.start + i] = blockIdx.x;
}
// Pivots of the roots.  One whose labels are all equal splits off nothing:
// its halves are itself and nothing, and go no further.
static __global__ void k_ls_root_pivot(LsNode *act, int32_t ns, int32_t *range) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns) return;
    const int32_t lo = range[4 * k], hi = range[4 * k + 1];
    act[k].pivot = lo == hi ? 0x7fffffff : ls_pivot(lo, hi);
    range[4 * k] = 0x7fffffff;
    range[4 * k + 1] = (int32_t)0x80000000;
}
// One pass over the labels of a round: the "big" flags as rank bits and the
// label ranges of both halves (as k_lv_flags takes its boxes).
static __global__ void __launch_bounds__(256) k_ls_flags(const int32_t *lab, int64_t M,
                                                         const int32_t *owner, const LsNode *act,
                                                         int32_t *range, RankBits R) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t first = blockIdx.x * (int64_t)RSG_TILE + w * RSG_STRETCH;
    const int a0 = stretch_owner(owner, first, M, true);
    __shared__ int part[8][4];
    __shared__ int a_s;
    if (threadIdx.x == 0) a_s = a0;
    __syncthreads();
    const bool whole = __syncthreads_and(a0 >= 0 && a0 == a_s);
    uint32_t word = 0;
    if (a0 >= 0) {
        const int pivot = act[a0].pivot;
        int lo[2] = {0x7fffffff, 0x7fffffff}, hi[2] = {(int)0x80000000, (int)0x80000000};
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int64_t i = first + 32 * u + lane;
            const bool on = i < M;
            const int v = on ? lab[i] : 0;
            const bool big = on && v > pivot;
            const unsigned b = __ballot_sync(FULL, big);
            if (lane == u) word = b;
            if (on) {
                lo[0] = big ? lo[0] : min(lo[0], v);
                hi[0] = big ? hi[0] : max(hi[0], v);
                lo[1] = big ? min(lo[1], v) : lo[1];
                hi[1] = big ? max(hi[1], v) : hi[1];
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int a = __reduce_min_sync(FULL, lo[h]), b = __reduce_max_sync(FULL, hi[h]);
            if (lane == 0 && whole) {
                part[w][2 * h] = a;
                part[w][2 * h + 1] = b;
            } else if (lane == 0 && a <= b) {
                atomicMin(&range[4 * a0 + 2 * h], a);
                atomicMax(&range[4 * a0 + 2 * h + 1], b);
            }
        }
    } else if (a0 == -2) {
        for (int u = 0; u < 8; u++) {
            const int64_t i = first + 32 * u + lane;
            const int a = i < M ? owner[i] : -1;
            bool big = false;
            if (a >= 0) {
                const int v = lab[i];
                big = v > act[a].pivot;
                atomicMin(&range[4 * a + (big ? 2 : 0)], v);
                atomicMax(&range[4 * a + (big ? 3 : 1)], v);
            }
            const unsigned b = __ballot_sync(FULL, big);
            if (lane == u) word = b;
        }
    }
    rank_store(R, blockIdx.x, word);  // holds a block barrier after the loop above
    if (whole && threadIdx.x < 4) {
        int v = part[0][threadIdx.x];
        for (int q = 1; q < 8; q++)
            v = (threadIdx.x & 1) ? max(v, part[q][threadIdx.x]) : min(v, part[q][threadIdx.x]);
        if (threadIdx.x & 1) atomicMax(&range[4 * a0 + threadIdx.x], v);
        else atomicMin(&range[4 * a0 + threadIdx.x], v);
    }
}
// Counts of a round's segments, and where each half goes: one of several
// labels above RSG_LS_SUB elements to the next round, up to there to the
// block lists; one of equal labels is finished, and copied (by a block, or as
// a segment) when the round leaves it in the scratch buffer (dst 1).
static __global__ void k_ls_nodes(LsNode *act, LsNode *nxt, const int32_t *range, int32_t *rnext,
                                  LsState *st, RankBits R, int32_t round, int dst, LsSub *subs,
                                  int32_t nsubs, int2 *copies) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= st->ns[round]) return;
    LsNode &A = act[k];
    const int s = A.start, n = A.n, rs = R.rank(s);
    const int m = n - (R.rank((int64_t)s + n) - rs);
    A.m = m;
    A.q = R.rank((int64_t)s + m) - rs;
    A.rs = rs;
    for (int h = 0; h < 2; h++) {
        const int hs = h ? s + m : s, hn = h ? n - m : m;
        const int32_t lo = range[4 * k + 2 * h], hi = range[4 * k + 2 * h + 1];
        A.next[h] = -1;
        if (hn > RSG_LS_SUB) {
            if (lo != hi) {
                const int j = atomicAdd(&st->ns[round + 1], 1);
                A.next[h] = j;
                LsNode x = {};
                x.start = hs;
                x.n = hn;
                x.pivot = ls_pivot(lo, hi);
                nxt[j] = x;
                for (int g = 0; g < 2; g++) {
                    rnext[4 * j + 2 * g] = 0x7fffffff;
                    rnext[4 * j + 2 * g + 1] = (int32_t)0x80000000;
                }
            } else if (dst) {
                copies[atomicAdd(&st->ncopy, 1)] = make_int2(hs, hn);
            }
        } else if (hn > 0 && (lo != hi || dst)) {
            const int c = hn > RSG_LS_SUB0;
            const int at = atomicAdd(&st->nsub[c], 1);
            subs[c ? nsubs - 1 - at : at] = LsSub{hs, hn, dst, 0};
        }
    }
}
static __global__ void __launch_bounds__(256) k_ls_tables(int64_t M, const int32_t *owner,
                                                          const LsNode *act, RankBits R,
                                                          int32_t *fb, int32_t *bs) {
    const int lane = threadIdx.x & 31;
    const int64_t first = blockIdx.x * (int64_t)RSG_TILE + (threadIdx.x >> 5) * RSG_STRETCH;
    const int a0 = stretch_owner(owner, first, M, true);
    if (a0 == -1) return;
#pragma unroll 1
    for (int u = 0; u < 8; u++) {
        const int64_t i = first + 32 * u + lane;
        if (i >= M) return;
        const int k = a0 >= 0 ? a0 : owner[i];
        if (k < 0) continue;
        const LsNode &A = act[k];
        swap_tables((int)(i - A.start), R.big(i), R.rank(i) - A.rs, A.m, fb + A.start,
                    bs + A.start);
    }
}
// Elements to their places; a place then belongs to the half it lies in.
template <class T>
__global__ void __launch_bounds__(256) k_ls_scatter(int64_t M, int32_t *owner, const LsNode *act,
                                                    RankBits R, const int32_t *fb,
                                                    const int32_t *bs, const T *src, T *dst,
                                                    const int32_t *lsrc, int32_t *ldst) {
    const int lane = threadIdx.x & 31;
    const int64_t first = blockIdx.x * (int64_t)RSG_TILE + (threadIdx.x >> 5) * RSG_STRETCH;
    const int a0 = stretch_owner(owner, first, M, true);
    __syncwarp();  // every lane has read the owners that are written below
    if (a0 == -1) return;
    LsNode A;
    if (a0 >= 0) A = act[a0];
#pragma unroll 2
    for (int u = 0; u < 8; u++) {
        const int64_t i = first + 32 * u + lane;
        if (i >= M) return;
        if (a0 < 0) {
            const int k = owner[i];
            if (k < 0) continue;
            A = act[k];
        }
        const T r = src[i];
        const int v = lsrc[i], l = (int)(i - A.start);
        const int d = swap_dest(l, A.n, R.big(i), R.rank(i) - A.rs, A.m, A.q, fb + A.start,
                                bs + A.start);
        dst[A.start + d] = r;
        ldst[A.start + d] = v;
        owner[i] = A.next[l >= A.m];
    }
}

// One block's storage for a segment of at most S elements (at most S / 2
// splitting segments of two or more elements at a time).
template <int S>
struct LsShared {
    static constexpr int NA = S / 2;
    int32_t lab[S];           // labels by the elements' first place
    uint16_t idx[2][S];       // place -> element, before and after a level
    uint16_t own[S];          // place -> splitting segment, RSG_LS_NONE: none
    uint16_t fb[S], bs[S];    // the closed form's tables (kdtree.cuh)
    uint32_t bits[S / 32 + 1];
    int32_t wpre[S / 32 + 1];
    int32_t mn[NA][2], mx[NA][2];  // label ranges of both halves
    int32_t pivot[2][NA];
    uint16_t s[2][NA], n[2][NA], m[NA], q[NA], next[NA][2];
    int32_t nact[2];
};
#define RSG_LS_NONE 0xffff
// Label range of a half of each lane's segment: one reduction when the warp's
// lanes are of one segment, else an atomic per lane.
__device__ __forceinline__ void ls_range(int32_t (*mn)[2], int32_t (*mx)[2], int v, int k,
                                         bool big) {
    const unsigned FULL = 0xffffffffu;
    const int k0 = __shfl_sync(FULL, k, 0);
    if (__all_sync(FULL, k == k0)) {
        if (k0 == RSG_LS_NONE) return;
        const unsigned b = __ballot_sync(FULL, big);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (b == (h ? 0u : FULL)) continue;
            const bool in = big == (h == 1);
            const int lo = __reduce_min_sync(FULL, in ? v : 0x7fffffff);
            const int hi = __reduce_max_sync(FULL, in ? v : (int)0x80000000);
            if ((threadIdx.x & 31) == 0) {
                atomicMin(&mn[k0][h], lo);
                atomicMax(&mx[k0][h], hi);
            }
        }
    } else if (k != RSG_LS_NONE) {
        atomicMin(&mn[k][big], v);
        atomicMax(&mx[k][big], v);
    }
}
// Finishes one listed segment per block, all its levels in shared memory, as
// k_sub_build does a subtree: flags as bits, ranks by population counts,
// 2-byte places, the records and labels moved once at the end (from the
// scratch buffer where the rounds left them there).  A level costs the chain
// of six block barriers, where a round of the loop below costs five launches
// and passes over all the call's elements: with every level a round, the sorts
// of a 64^3 snapshot were 79 rounds.
template <class R, int S, int T>
__global__ void __launch_bounds__(T) k_ls_sub(R *W, int32_t *lab, const R *sw, const int32_t *sl,
                                              const LsSub *segs) {
    extern __shared__ __align__(16) unsigned char ls_sm[];
    LsShared<S> &h = *reinterpret_cast<LsShared<S> *>(ls_sm);
    const int t = threadIdx.x, lane = t & 31;
    const LsSub seg = segs[blockIdx.x];
    const int g0 = seg.start, n = seg.n;
    const R *from = seg.src ? sw : W;
    const int32_t *lfrom = seg.src ? sl : lab;
    const int nw = (n + 31) >> 5;
    const int span = ((n + T - 1) / T) * T;  // whole warps take part in every pass
    if (t == 0) {
        h.bits[nw] = 0;
        h.mn[0][0] = 0x7fffffff;
        h.mx[0][0] = (int32_t)0x80000000;
    }
    __syncthreads();
    for (int i = t; i < span; i += T) {
        const bool ok = i < n;
        const int v = ok ? lfrom[g0 + i] : 0;
        if (ok) {
            h.lab[i] = v;
            h.idx[0][i] = (uint16_t)i;
            h.own[i] = 0;
        }
        ls_range(h.mn, h.mx, v, ok ? 0 : RSG_LS_NONE, false);
    }
    __syncthreads();
    const bool moves = h.mn[0][0] != h.mx[0][0];
    if (!moves && !seg.src) return;
    if (t == 0) {
        h.s[0][0] = 0;
        h.n[0][0] = (uint16_t)n;
        h.pivot[0][0] = ls_pivot(h.mn[0][0], h.mx[0][0]);
        h.nact[0] = moves;
    }
    auto rank = [&](int x) {
        return h.wpre[x >> 5] + __popc(h.bits[x >> 5] & ((1u << (x & 31)) - 1u));
    };
    int cur = 0;
    for (;;) {
        __syncthreads();
        const int nact = h.nact[cur];
        if (nact == 0) break;
        for (int k = t; k < nact; k += T) {
            h.mn[k][0] = h.mn[k][1] = 0x7fffffff;
            h.mx[k][0] = h.mx[k][1] = (int32_t)0x80000000;
        }
        if (t == 0) h.nact[1 - cur] = 0;
        __syncthreads();
        for (int i = t; i < span; i += T) {
            const int k = i < n ? h.own[i] : RSG_LS_NONE;
            int v = 0;
            bool big = false;
            if (k != RSG_LS_NONE) {
                v = h.lab[h.idx[cur][i]];
                big = v > h.pivot[cur][k];
            }
            const unsigned b = __ballot_sync(0xffffffffu, big);
            if (lane == 0 && i < n) h.bits[i >> 5] = b;
            ls_range(h.mn, h.mx, v, k, big);
        }
        __syncthreads();
        if (t < 32) {
            int run = 0;
            for (int w0 = 0; w0 <= nw; w0 += 32) {
                const int w = w0 + lane;
                const int v = w < nw ? __popc(h.bits[w]) : 0;
                int inc = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, inc, o);
                    if (lane >= o) inc += u;
                }
                if (w <= nw) h.wpre[w] = run + inc - v;
                run += __shfl_sync(0xffffffffu, inc, 31);
            }
        }
        __syncthreads();
        for (int k = t; k < nact; k += T) {
            const int s = h.s[cur][k], nn = h.n[cur][k];
            const int rs = rank(s);
            const int m = nn - (rank(s + nn) - rs);
            h.m[k] = (uint16_t)m;
            h.q[k] = (uint16_t)(rank(s + m) - rs);
#pragma unroll
            for (int c = 0; c < 2; c++) {
                const int cn = c ? nn - m : m;
                int j = RSG_LS_NONE;
                if (cn >= 2 && h.mn[k][c] != h.mx[k][c]) {
                    j = atomicAdd(&h.nact[1 - cur], 1);
                    h.s[1 - cur][j] = (uint16_t)(c ? s + m : s);
                    h.n[1 - cur][j] = (uint16_t)cn;
                    h.pivot[1 - cur][j] = ls_pivot(h.mn[k][c], h.mx[k][c]);
                }
                h.next[k][c] = (uint16_t)j;
            }
        }
        __syncthreads();
        for (int i = t; i < n; i += T) {
            const int k = h.own[i];
            if (k == RSG_LS_NONE) continue;
            const int s = h.s[cur][k], l = i - s, m = h.m[k];
            const int br = rank(i) - rank(s), sr = l - br;
            const bool big = (h.bits[i >> 5] >> (i & 31)) & 1u;
            if (big && l < m) h.fb[s + br] = (uint16_t)l;
            if (!big && l >= m) h.bs[s + (m - 1 - sr)] = (uint16_t)l;
        }
        __syncthreads();
        for (int i = t; i < n; i += T) {
            const int k = h.own[i];
            const uint16_t e = h.idx[cur][i];
            if (k == RSG_LS_NONE) {
                h.idx[1 - cur][i] = e;
                continue;
            }
            const int s = h.s[cur][k], nn = h.n[cur][k], l = i - s, m = h.m[k], q = h.q[k];
            const int br = rank(i) - rank(s), sr = l - br;
            const bool big = (h.bits[i >> 5] >> (i & 31)) & 1u;
            int d;
            if (!big && l < m) {
                d = l;
            } else if (big && l < m) {
                d = (br == 0) ? nn - 1 : h.bs[s + br - 1] - 1;
            } else if (!big) {
                d = h.fb[s + (m - 1 - sr)];
            } else {
                const int pos_last = (q > 0) ? h.bs[s + q - 1] : nn;
                if (l > pos_last)
                    d = l - 1;
                else if (pos_last - m >= 2)
                    d = (l == m) ? pos_last - 1 : l - 1;
                else
                    d = l;
            }
            h.idx[1 - cur][s + d] = e;
            h.own[i] = h.next[k][l >= m];
        }
        cur ^= 1;
    }
    constexpr int V = sizeof(R) / 16, PER = S / T;
    static_assert(sizeof(R) % 16 == 0 && S % T == 0, "record vectors");
    const uint4 *sv = reinterpret_cast<const uint4 *>(from + g0);
    uint4 *dv = reinterpret_cast<uint4 *>(W + g0);
#pragma unroll 1
    for (int v = 0; v < V; v++) {
        uint4 r[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = t + u * T;
            if (i < n) r[u] = sv[(int)h.idx[cur][i] * V + v];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = t + u * T;
            if (i < n) dv[i * V + v] = r[u];
        }
    }
    for (int i = t; i < n; i += T) lab[g0 + i] = h.lab[h.idx[cur][i]];
}
template <class R, int S, int T>
void launch_ls_sub(int32_t count, R *W, int32_t *lab, const R *sw, const int32_t *sl,
                   const LsSub *segs, cudaStream_t st) {
    if (count == 0) return;
    const size_t sm = sizeof(LsShared<S>);
    RSG_CUDA(cudaFuncSetAttribute(k_ls_sub<R, S, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sm));
    launch(k_ls_sub<R, S, T>, count, T, sm, st, W, lab, sw, sl, segs);
}

// Sorts W (and its labels) inside every segment (host arrays hs/hn) the way
// the reference's recursive partition does.
#define RSG_LS_BATCH 4  // rounds between reads of the sort's state
template <class T>
void partition_sort_labels(Arena &ar, T *W, int32_t *lab, int64_t M,
                           const std::vector<int32_t> &hs, const std::vector<int32_t> &hn,
                           cudaStream_t st) {
    std::vector<int2> roots;    // the segments of the round loop
    std::vector<LsSub> c0, c1;  // those the blocks finish
    for (size_t k = 0; k < hs.size(); k++) {
        if (hn[k] > RSG_LS_SUB) roots.push_back(make_int2(hs[k], hn[k]));
        else if (hn[k] >= 2) (hn[k] > RSG_LS_SUB0 ? c1 : c0).push_back(LsSub{hs[k], hn[k], 0, 0});
    }
    const int32_t ns = (int32_t)roots.size();
    if (ns == 0 && c0.empty() && c1.empty()) return;
    size_t mark = ar.used;
    struct Head {  // the fields of LsState before ns[]
        int32_t nsub[2], ncopy, pad;
    } h = {{(int32_t)c0.size(), (int32_t)c1.size()}, 0, 0};
    static_assert(offsetof(LsState, ns) == sizeof(Head), "LsState layout");
    // listed segments are disjoint
    const int32_t nsubs = ns > 0 ? (int32_t)M : h.nsub[0] + h.nsub[1];
    LsSub *subs = ar.get<LsSub>(nsubs);
    // with no segment for the rounds nothing below waits for the stream
    HostTables tables(st);
    RSG_CUDA(tables.copy(subs, std::move(c0)));
    RSG_CUDA(tables.copy(subs + (nsubs - h.nsub[1]), std::move(c1)));
    // rounds scatter back and forth between these
    T *wb[2] = {W, nullptr};
    int32_t *lb[2] = {lab, nullptr};
    if (ns > 0) {
        const int64_t cap = M / (RSG_LS_SUB + 1) + 1;  // segments of a round
        LsNode *act[2];
        int32_t *range[2];
        for (int b = 0; b < 2; b++) {
            act[b] = ar.get<LsNode>(cap);
            range[b] = ar.get<int32_t>(4 * cap);
        }
        int2 *copies = ar.get<int2>(cap), *d_roots = ar.get<int2>(ns);
        int32_t *owner = ar.get<int32_t>(M), *fb = ar.get<int32_t>(M), *bs = ar.get<int32_t>(M);
        wb[1] = ar.get<T>(M);
        lb[1] = ar.get<int32_t>(M);
        LsState *ls = ar.get<LsState>(1);
        const RankBits R = rank_alloc(ar, M, st);
        const int32_t nt = (int32_t)rank_tiles(M);
        RSG_CUDA(tables.copy(d_roots, std::move(roots)));
        RSG_CUDA(cudaMemsetAsync(ls, 0, sizeof(LsState), st));
        // Head and ns[0]
        RSG_CUDA(tables.copy((int32_t *)ls,
                             std::vector<int32_t>{h.nsub[0], h.nsub[1], 0, 0, ns}));
        RSG_CUDA(cudaMemsetAsync(owner, 0xff, sizeof(int32_t) * M, st));
        launch(k_ls_roots, nblk(ns, 64), 64, 0, st, (const int2 *)d_roots, ns, act[0], range[0]);
        const int64_t y = M / ns / 2048;
        launch(k_ls_owner, dim3(ns, (unsigned)(y < 1 ? 1 : (y > 4096 ? 4096 : y))), 256, 0, st,
               (const LsNode *)act[0], owner);
        launch(k_ls_flags, nt, 256, 0, st, (const int32_t *)lab, M, (const int32_t *)owner,
               (const LsNode *)act[0], range[0], R);
        launch(k_ls_root_pivot, nblk(ns, 64), 64, 0, st, act[0], ns, range[0]);
        // Rounds run back to back with their counts on the device; grids are
        // sized by an upper bound of the segments (ub).  A round past the last
        // costs passes over M elements against the 12 us of a read, so large
        // calls read after every round.
        const int batch = M > (1 << 22) ? 1 : RSG_LS_BATCH;
        int64_t ub = ns;
        int32_t now = ns;
        int cur = 0;
        for (int round = 0; now > 0;) {
            for (int b = 0; b < batch; b++, round++) {
                if (round > RSG_LS_ROUNDS) {
                    set_error(RSG_ERR_LIMIT, "label partition sort did not terminate");
                    throw Failure();
                }
                const int x = round & 1;
                launch(k_ls_flags, nt, 256, 0, st, (const int32_t *)lb[cur], M,
                       (const int32_t *)owner, (const LsNode *)act[x], range[x], R);
                launch(k_rank_scan, 1, 1024, 0, st, R.tpre, nt);
                launch(k_ls_nodes, nblk(ub, 64), 64, 0, st, act[x], act[1 - x],
                       (const int32_t *)range[x], range[1 - x], ls, R, round, 1 - cur, subs, nsubs,
                       copies);
                launch(k_ls_tables, nt, 256, 0, st, M, (const int32_t *)owner,
                       (const LsNode *)act[x], R, fb, bs);
                launch(k_ls_scatter<T>, nt, 256, 0, st, M, owner, (const LsNode *)act[x], R,
                       (const int32_t *)fb, (const int32_t *)bs, (const T *)wb[cur], wb[1 - cur],
                       (const int32_t *)lb[cur], lb[1 - cur]);
                RSG_CHECK_LAUNCH();
                cur ^= 1;
                ub = std::min<int64_t>(2 * ub, cap);
            }
            RSG_CUDA(cudaMemcpyAsync(&now, &ls->ns[round], sizeof(now), cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaMemcpyAsync(&h, ls, sizeof(h), cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            ub = now;
        }
        if (h.ncopy) {
            launch(k_copy_segs<T>, dim3(h.ncopy, 64), 256, 0, st, (const int2 *)copies,
                   (const T *)wb[1], W);
            launch(k_copy_segs<int32_t>, dim3(h.ncopy, 64), 256, 0, st, (const int2 *)copies,
                   (const int32_t *)lb[1], lab);
        }
    }
    launch_ls_sub<T, RSG_LS_SUB, 512>(h.nsub[1], W, lab, (const T *)wb[1], (const int32_t *)lb[1],
                                      (const LsSub *)subs + (nsubs - h.nsub[1]), st);
    launch_ls_sub<T, RSG_LS_SUB0, 64>(h.nsub[0], W, lab, (const T *)wb[1], (const int32_t *)lb[1],
                                      (const LsSub *)subs, st);
    RSG_CHECK_LAUNCH();
    ar.used = mark;
}

}  // namespace rsg
