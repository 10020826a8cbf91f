// Exact GPU version of partition_sort_particles (src/fof.c:184-224): each
// segment is split at the midpoint of its label range with the same
// two-pointer swap that the kd-tree build uses (closed form in kdtree.cuh),
// then both halves recurse.  Segments above RSG_LS_SUB elements are split
// level-synchronously, many at once; what is left of a segment at or below
// that size is finished by one block in shared memory.
#pragma once
#include "kdtree.cuh"

namespace rsg {

#define RSG_LS_SUB0 256  // largest segment of the small blocks
#define RSG_LS_SUB 2048  // largest segment one block finishes

struct LSeg {
    int32_t *start, *n;  // active segments
    int32_t *mn, *mx;    // label range
    int32_t *m, *q;
};
// Device-side state of a sort: the round's segment count and the segments
// listed for the two classes of block.
struct LsState {
    int32_t ns;
    int32_t nsub[2];
    int32_t pad;
};

// owner[i]: the active segment holding element i (segments are disjoint and
// listed by ascending start), -1 outside every segment.
static __global__ void k_ls_owner(const int32_t *start, const int32_t *n, int32_t ns, int64_t M,
                                  int32_t *owner) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= M) return;
    int lo = 0, hi = ns - 1, k = -1;
    while (lo <= hi) {
        int mid = (lo + hi) >> 1;
        if (start[mid] <= i) {
            k = mid;
            lo = mid + 1;
        } else {
            hi = mid - 1;
        }
    }
    owner[i] = (k >= 0 && i < (int64_t)start[k] + n[k]) ? k : -1;
}
static __global__ void k_ls_init(LSeg S, int32_t ns) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ns) return;
    S.mn[k] = 0x7fffffff;
    S.mx[k] = (int32_t)0x80000000;
}
// Label range of every segment.  A thread reads ITEMS consecutive elements;
// threads whose elements all belong to one segment combine their ranges
// with the other lanes of that segment before the atomics (a large segment
// gets one atomic pair per warp instead of one per thread).
template <int ITEMS>
static __global__ void k_ls_minmax(const int32_t *lab, int64_t M, const int32_t *owner, LSeg S) {
    const unsigned FULL = 0xffffffffu;
    int64_t i0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * ITEMS;
    int first = -2;  // owner shared by all of this thread's elements, -1 mixed/none
    int cur = -1, lo = 0x7fffffff, hi = (int)0x80000000;
    for (int it = 0; it < ITEMS; it++) {
        int64_t i = i0 + it;
        int a = (i < M) ? owner[i] : -1;
        if (first == -2) first = a;
        else if (a != first) first = -1;
        if (a != cur) {
            if (cur >= 0 && first == -1) {  // mixed: this run goes out on its own
                atomicMin(&S.mn[cur], lo);
                atomicMax(&S.mx[cur], hi);
            }
            cur = a;
            lo = 0x7fffffff;
            hi = (int)0x80000000;
        }
        if (a < 0) continue;
        int v = lab[i];
        lo = min(lo, v);
        hi = max(hi, v);
    }
    bool uni = first >= 0;  // every element in one segment: combine across the warp
    unsigned grp = __match_any_sync(FULL, uni ? first : -1);
    if (uni) {
        int glo = __reduce_min_sync(grp, lo), ghi = __reduce_max_sync(grp, hi);
        if ((threadIdx.x & 31) == __ffs(grp) - 1) {
            atomicMin(&S.mn[first], glo);
            atomicMax(&S.mx[first], ghi);
        }
    } else if (cur >= 0) {
        atomicMin(&S.mn[cur], lo);
        atomicMax(&S.mx[cur], hi);
    }
}
// pivot = min + (max - min) / 2 (src/fof.c:201); a segment whose labels are
// all equal is finished (no element is "big").
__device__ __forceinline__ int32_t ls_pivot(int64_t lo, int64_t hi) {
    return (lo == hi) ? 0x7fffffff : (int32_t)(lo + (hi - lo) / 2);
}
static __global__ void k_ls_flags(const int32_t *lab, int64_t M, const int32_t *owner, LSeg S,
                           int32_t *flag) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i > M) return;
    int f = 0;
    if (i < M) {
        int a = owner[i];
        if (a >= 0) f = lab[i] > ls_pivot(S.mn[a], S.mx[a]);
    }
    flag[i] = f;
}
// m (= #small) and q (= #big before m) per segment, and which halves of
// the segments that split go on: above RSG_LS_SUB elements to the next round
// (hflag), from 2 to there to the block lists.  Grid over ub + 1, ub bounding
// the round's segments.
static __global__ void k_ls_counts(LSeg S, LsState *st, int32_t ub, const int32_t *rank,
                                   int32_t *hflag, int2 *subs, int32_t nsubs) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > ub) return;
    if (k >= st->ns) {
        hflag[2 * k] = 0;
        if (k < ub) hflag[2 * k + 1] = 0;
        return;
    }
    int s = S.start[k], n = S.n[k];
    int B = rank[s + n] - rank[s];
    int m = n - B;
    S.m[k] = m;
    S.q[k] = rank[s + m] - rank[s];
    const bool split = S.mn[k] != S.mx[k];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int hs = h ? s + m : s, hn = h ? n - m : m;
        hflag[2 * k + h] = split && hn > RSG_LS_SUB;
        if (split && hn >= 2 && hn <= RSG_LS_SUB) {
            const int c = hn > RSG_LS_SUB0;
            const int at = atomicAdd(&st->nsub[c], 1);
            subs[c ? nsubs - 1 - at : at] = make_int2(hs, hn);
        }
    }
}
static __global__ void k_ls_tables(int64_t M, const int32_t *owner, LSeg S, const int32_t *flag,
                            const int32_t *rank, int32_t *fb, int32_t *bs) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= M) return;
    int a = owner[i];
    if (a < 0) return;
    int s = S.start[a];
    int l = (int)(i - s);
    int br = rank[i] - rank[s];
    int sr = l - br;
    int m = S.m[a];
    if (flag[i] && l < m) fb[s + br] = l;
    if (!flag[i] && l >= m) bs[s + (m - 1 - sr)] = l;
}
template <class T>
__global__ void k_ls_scatter(int64_t M, const int32_t *owner, LSeg S, const int32_t *flag,
                             const int32_t *rank, const int32_t *fb, const int32_t *bs,
                             const T *src, T *dst, const int32_t *lsrc, int32_t *ldst) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= M) return;
    int a = owner[i];
    if (a < 0) return;
    int s = S.start[a], n = S.n[a];
    int l = (int)(i - s);
    int br = rank[i] - rank[s];
    int sr = l - br;
    int m = S.m[a], q = S.q[a];
    int big = flag[i];
    int d;
    if (!big && l < m) d = l;
    else if (big && l < m) d = (br == 0) ? n - 1 : bs[s + br - 1] - 1;
    else if (!big) d = fb[s + (m - 1 - sr)];
    else {
        int pos_last = (q > 0) ? bs[s + q - 1] : n;
        if (l > pos_last) d = l - 1;
        else if (pos_last - m >= 2) d = (l == m) ? pos_last - 1 : l - 1;
        else d = l;
    }
    dst[s + d] = src[i];
    ldst[s + d] = lsrc[i];
}
// After a round: every element moves to the half of its segment it now
// lies in; a half of the next round (hflag) has its compacted index (hidx),
// and the elements of the other halves are copied from the buffer the round
// wrote (src) to the output arrays when they differ: they are final, or a
// block's to finish in place.
template <class T>
__global__ void k_ls_owner_next(int64_t M, int32_t *owner, LSeg S, const int32_t *hflag,
                                const int32_t *hidx, const T *src, T *dst, const int32_t *lsrc,
                                int32_t *ldst) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= M) return;
    int a = owner[i];
    if (a < 0) return;
    int h = 2 * a + ((i - S.start[a]) < S.m[a] ? 0 : 1);
    if (hflag[h]) {
        owner[i] = hidx[h];
        return;
    }
    owner[i] = -1;
    if (src != dst) {
        dst[i] = src[i];
        ldst[i] = lsrc[i];
    }
}
// The next round's segments, with their label ranges cleared.
static __global__ void k_ls_next(LSeg S, LsState *st, int32_t ub, const int32_t *hflag,
                                 const int32_t *hidx, LSeg R) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ub || k >= st->ns) return;
    for (int h = 0; h < 2; h++) {
        if (!hflag[2 * k + h]) continue;
        const int j = hidx[2 * k + h];
        R.start[j] = h ? S.start[k] + S.m[k] : S.start[k];
        R.n[j] = h ? S.n[k] - S.m[k] : S.m[k];
        R.mn[j] = 0x7fffffff;
        R.mx[j] = (int32_t)0x80000000;
    }
}
static __global__ void k_ls_advance(LsState *st, int32_t ub, const int32_t *hidx) {
    if (threadIdx.x || blockIdx.x) return;
    st->ns = hidx[2 * ub];
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
// 2-byte places, the records and labels moved once at the end.  A level costs
// the chain of six block barriers, where a round of the loop below costs ten
// launches and passes over all the call's elements: the sorts of one level of
// a 64^3 snapshot were 79 rounds of the loop, 3 ms of launches.
template <class R, int S, int T>
__global__ void __launch_bounds__(T) k_ls_sub(R *W, int32_t *lab, const int2 *segs) {
    extern __shared__ __align__(16) unsigned char ls_sm[];
    LsShared<S> &h = *reinterpret_cast<LsShared<S> *>(ls_sm);
    const int t = threadIdx.x, lane = t & 31;
    const int g0 = segs[blockIdx.x].x, n = segs[blockIdx.x].y;
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
        const int v = ok ? lab[g0 + i] : 0;
        if (ok) {
            h.lab[i] = v;
            h.idx[0][i] = (uint16_t)i;
            h.own[i] = 0;
        }
        ls_range(h.mn, h.mx, v, ok ? 0 : RSG_LS_NONE, false);
    }
    __syncthreads();
    if (h.mn[0][0] == h.mx[0][0]) return;  // nothing moves
    if (t == 0) {
        h.s[0][0] = 0;
        h.n[0][0] = (uint16_t)n;
        h.pivot[0][0] = ls_pivot(h.mn[0][0], h.mx[0][0]);
        h.nact[0] = 1;
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
    uint4 *rv = reinterpret_cast<uint4 *>(W + g0);
#pragma unroll 1
    for (int v = 0; v < V; v++) {
        uint4 r[PER];
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = t + u * T;
            if (i < n) r[u] = rv[(int)h.idx[cur][i] * V + v];
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < PER; u++) {
            const int i = t + u * T;
            if (i < n) rv[i * V + v] = r[u];
        }
    }
    for (int i = t; i < n; i += T) lab[g0 + i] = h.lab[h.idx[cur][i]];
}
template <class R, int S, int T>
void launch_ls_sub(int32_t count, R *W, int32_t *lab, const int2 *segs, cudaStream_t st) {
    if (count == 0) return;
    const size_t sm = sizeof(LsShared<S>);
    RSG_CUDA(cudaFuncSetAttribute(k_ls_sub<R, S, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)sm));
    launch(k_ls_sub<R, S, T>, count, T, sm, st, W, lab, segs);
}

// Sorts W (and its labels) inside every segment (host arrays hs/hn) the way
// the reference's recursive partition does.
#define RSG_LS_BATCH 4  // rounds between reads of the sort's state
template <class T>
void partition_sort_labels(Arena &ar, T *W, int32_t *lab, int64_t M,
                           const std::vector<int32_t> &hs, const std::vector<int32_t> &hn,
                           cudaStream_t st) {
    std::vector<int32_t> s0, n0;  // the segments of the round loop
    std::vector<int2> c0, c1;     // those the blocks finish
    for (size_t k = 0; k < hs.size(); k++) {
        if (hn[k] > RSG_LS_SUB) {
            s0.push_back(hs[k]);
            n0.push_back(hn[k]);
        } else if (hn[k] >= 2) {
            (hn[k] > RSG_LS_SUB0 ? c1 : c0).push_back(make_int2(hs[k], hn[k]));
        }
    }
    const int32_t ns = (int32_t)s0.size();
    if (ns == 0 && c0.empty() && c1.empty()) return;
    const int T_ = 256;
    size_t mark = ar.used;
    LsState h = {};
    h.ns = ns;
    h.nsub[0] = (int32_t)c0.size();
    h.nsub[1] = (int32_t)c1.size();
    // listed segments are disjoint, of two elements or more
    const int32_t nsubs = (int32_t)(M / 2 + 1);
    int2 *subs = ar.get<int2>(nsubs);
    if (!c0.empty())
        RSG_CUDA(cudaMemcpyAsync(subs, c0.data(), sizeof(int2) * c0.size(),
                                 cudaMemcpyHostToDevice, st));
    if (!c1.empty())
        RSG_CUDA(cudaMemcpyAsync(subs + (nsubs - c1.size()), c1.data(), sizeof(int2) * c1.size(),
                                 cudaMemcpyHostToDevice, st));
    if (ns > 0) {
        const int64_t cap = M / (RSG_LS_SUB + 1) + 1;  // segments of a round
        LSeg S[2];
        for (int b = 0; b < 2; b++) {
            S[b].start = ar.get<int32_t>(cap); S[b].n = ar.get<int32_t>(cap);
            S[b].mn = ar.get<int32_t>(cap); S[b].mx = ar.get<int32_t>(cap);
            S[b].m = ar.get<int32_t>(cap); S[b].q = ar.get<int32_t>(cap);
        }
        int32_t *hflag = ar.get<int32_t>(2 * cap + 1), *hidx = ar.get<int32_t>(2 * cap + 1);
        int32_t *owner = ar.get<int32_t>(M), *flag = ar.get<int32_t>(M + 1);
        int32_t *rank = ar.get<int32_t>(M + 1);
        int32_t *fb = ar.get<int32_t>(M), *bs = ar.get<int32_t>(M);
        T *tw = ar.get<T>(M);
        int32_t *tl = ar.get<int32_t>(M);
        LsState *ls = ar.get<LsState>(1);
        size_t b1 = 0, b3 = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, b1, flag, rank, (int)(M + 1), st);
        cub::DeviceScan::ExclusiveSum(nullptr, b3, hflag, hidx, (int)(2 * cap + 1), st);
        if (b3 > b1) b1 = b3;
        void *tmp = ar.take(b1 + 256);
        size_t tb = b1 + 256;
        RSG_CUDA(cudaMemcpyAsync(S[0].start, s0.data(), 4 * ns, cudaMemcpyHostToDevice, st));
        RSG_CUDA(cudaMemcpyAsync(S[0].n, n0.data(), 4 * ns, cudaMemcpyHostToDevice, st));
        RSG_CUDA(cudaMemcpyAsync(ls, &h, sizeof(h), cudaMemcpyHostToDevice, st));
        // rounds scatter back and forth between (W, lab) and (tw, tl); an
        // element is copied to (W, lab) once, when its segment leaves the loop
        T *wb[2] = {W, tw};
        int32_t *lb[2] = {lab, tl};
        int cur = 0;
        launch(k_ls_owner, nblk(M, T_), T_, 0, st, (const int32_t *)S[0].start,
               (const int32_t *)S[0].n, ns, M, owner);
        launch(k_ls_init, nblk(ns, T_), T_, 0, st, S[0], ns);
        // Rounds run back to back with their counts on the device; grids are
        // sized by an upper bound of the segments (ub).  A round past the last
        // costs passes over M elements (0.2 ms at 33M) against the 12 us of a
        // read, so large calls read after every round.
        const int batch = M > (1 << 22) ? 1 : RSG_LS_BATCH;
        int64_t ub = ns;
        for (int round = 0; h.ns > 0;) {
            for (int b = 0; b < batch; b++, round++) {
                if (round > 200) {
                    set_error(RSG_ERR_LIMIT, "label partition sort did not terminate");
                    throw Failure();
                }
                const LSeg &A = S[round & 1], &B = S[1 - (round & 1)];
                const int32_t u = (int32_t)ub;
                launch(k_ls_minmax<8>, nblk((M + 7) / 8, T_), T_, 0, st, (const int32_t *)lb[cur],
                       M, (const int32_t *)owner, A);
                launch(k_ls_flags, nblk(M + 1, T_), T_, 0, st, (const int32_t *)lb[cur], M,
                       (const int32_t *)owner, A, flag);
                cub::DeviceScan::ExclusiveSum(tmp, tb, flag, rank, (int)(M + 1), st);
                launch(k_ls_counts, nblk(u + 1, T_), T_, 0, st, A, ls, u, (const int32_t *)rank,
                       hflag, subs, nsubs);
                launch(k_ls_tables, nblk(M, T_), T_, 0, st, M, (const int32_t *)owner, A,
                       (const int32_t *)flag, (const int32_t *)rank, fb, bs);
                launch(k_ls_scatter<T>, nblk(M, T_), T_, 0, st, M, (const int32_t *)owner, A,
                       (const int32_t *)flag, (const int32_t *)rank, (const int32_t *)fb,
                       (const int32_t *)bs, (const T *)wb[cur], wb[1 - cur],
                       (const int32_t *)lb[cur], lb[1 - cur]);
                cur ^= 1;
                cub::DeviceScan::ExclusiveSum(tmp, tb, hflag, hidx, 2 * u + 1, st);
                launch(k_ls_owner_next<T>, nblk(M, T_), T_, 0, st, M, owner, A,
                       (const int32_t *)hflag, (const int32_t *)hidx, (const T *)wb[cur], W,
                       (const int32_t *)lb[cur], lab);
                launch(k_ls_next, nblk(u, T_), T_, 0, st, A, ls, u, (const int32_t *)hflag,
                       (const int32_t *)hidx, B);
                launch(k_ls_advance, 1, 1, 0, st, ls, u, (const int32_t *)hidx);
                RSG_CHECK_LAUNCH();
                ub = std::min<int64_t>(2 * ub, cap);
            }
            RSG_CUDA(cudaMemcpyAsync(&h, ls, sizeof(h), cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            ub = h.ns;
        }
    }
    launch_ls_sub<T, RSG_LS_SUB, 512>(h.nsub[1], W, lab, (const int2 *)subs + (nsubs - h.nsub[1]),
                                      st);
    launch_ls_sub<T, RSG_LS_SUB0, 64>(h.nsub[0], W, lab, (const int2 *)subs, st);
    RSG_CHECK_LAUNCH();
    ar.used = mark;
}

}  // namespace rsg
