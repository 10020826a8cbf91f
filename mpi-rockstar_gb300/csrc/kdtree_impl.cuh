// Host driver of the level-synchronous kd-forest build (see kdtree.cuh).
#pragma once
#include "kdtree.cuh"

namespace rsg {

struct ToI64 {
    __device__ int64_t operator()(int32_t v) const { return (int64_t)v; }
};
// Fails with RSG_ERR_LIMIT when the int32 counts in[0..n) add up to more
// than an int32 offset can address: the callers scan such counts into
// int32 offsets.
inline void check_i32_total(Arena &ar, const int32_t *in, int64_t n, const char *what,
                            cudaStream_t st) {
    thrust::transform_iterator<ToI64, const int32_t *, int64_t> it(in, ToI64{});
    size_t mark = ar.used;
    int64_t *tot = ar.get<int64_t>(1);
    size_t b = 0;
    cub::DeviceReduce::Sum(nullptr, b, it, tot, (int)n, st);
    void *t = ar.take(b + 256);
    cub::DeviceReduce::Sum(t, b, it, tot, (int)n, st);
    RSG_CHECK_LAUNCH();
    int64_t h = 0;
    RSG_CUDA(cudaMemcpyAsync(&h, tot, sizeof(h), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    ar.used = mark;
    if (h > (int64_t)0x7fffffff - 1) {
        set_error(RSG_ERR_LIMIT, "%s: %lld entries exceed the 2^31 limit of one call", what,
                  (long long)h);
        throw Failure();
    }
}

#define RSG_FOREST_BATCH 4  // levels between reads of the build state

// One block's storage for a subtree of at most S records, of which at most
// NA nodes split on one level (each holds more than `leaf` records).
template <int D, int S, int NA>
struct SubShared {
    float pos[D][S];              // coordinates by the records' first place
    uint16_t idx[2][S];           // place -> record, before and after a level
    uint16_t own[S];              // place -> splitting node, RSG_NOSUB: none
    uint16_t fb[S], bs[S];        // the closed form's tables (kdtree.cuh)
    uint32_t bits[S / 32 + 1];    // "big" flags and their prefix by word
    int32_t wpre[S / 32 + 1];
    unsigned cbox[NA][2][2 * D];  // boxes of both halves (ordered integers)
    float box[2][NA][2 * D];      // boxes of the splitting nodes
    int32_t gid[2][NA];
    uint16_t s[2][NA], n[2][NA];
    float lim[NA];
    uint16_t m[NA], q[NA], srank[NA], next[NA][2];
    uint8_t div[NA], split[NA];
    int32_t nact, base, fail;
};
#define RSG_NOSUB 0xffffu

// Adds the lanes' coordinates (ordered integers are formed here) to the box
// of their node's half: one reduction per value when the warp's lanes are of
// one node (the upper levels), else an atomic per lane.
template <int D>
__device__ __forceinline__ void sub_box(unsigned (*cbox)[2][2 * D], const float *c, int k,
                                        bool big) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int k0 = __shfl_sync(FULL, k, 0);
    if (__all_sync(FULL, k == k0)) {
        if (k0 == RSG_NOSUB) return;
        const unsigned b = __ballot_sync(FULL, big);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            if (b == (h ? 0u : FULL)) continue;  // no lane in this half
            const bool in = big == (h == 1);
#pragma unroll
            for (int d = 0; d < D; d++) {
                const unsigned o = f2ord(c[d]);
                const unsigned lo = __reduce_min_sync(FULL, in ? o : 0xffffffffu);
                const unsigned hi = __reduce_max_sync(FULL, in ? o : 0u);
                if (lane == 2 * d) atomicMin(&cbox[k0][h][d], lo);
                if (lane == 2 * d + 1) atomicMax(&cbox[k0][h][D + d], hi);
            }
        }
    } else if (k != RSG_NOSUB) {
#pragma unroll
        for (int d = 0; d < D; d++) {
            const unsigned o = f2ord(c[d]);
            atomicMin(&cbox[k][big][d], o);
            atomicMax(&cbox[k][big][D + d], o);
        }
    }
}

// Builds one listed subtree per block, all its levels in shared memory: the
// level-synchronous steps of the loop below with the flags as bits, ranks by
// population counts and 2-byte places instead of moving records, which are
// moved once at the end.  Its cost is the chain of a level's six block
// barriers (about 1 us a level), hidden by the other blocks of the SM; a
// level of the loop below reads and writes every record of the call and
// costs five launches, and the levels below 2048 records are half or more of a
// build's.  2048 records are what leaves room for three
// blocks an SM in 3D (70 KB) and two in 6D (83 KB); 256-record subtrees, the
// bulk of the 6D forests, run sixteen to an SM.
// Children are numbered in the order the blocks allocate them: a node's two
// children stay neighbours, and nothing depends on any other order.
template <int D, class RecT, int S, int T, int NA>
__global__ void __launch_bounds__(T) k_sub_build(RecT *out, const RecT *scratch,
                                                 const SubRoot *roots, KNode<D> *nodes,
                                                 LevelState *ls, int32_t cap, int leaf) {
    extern __shared__ __align__(16) unsigned char sub_sm[];
    SubShared<D, S, NA> &h = *reinterpret_cast<SubShared<D, S, NA> *>(sub_sm);
    const int t = threadIdx.x, lane = t & 31;
    const SubRoot root = roots[blockIdx.x];
    const RecT *recs = root.src ? scratch : out;
    const int gs = nodes[root.node].start, n = nodes[root.node].n;
    const int tree = nodes[root.node].tree;
    const int nw = (n + 31) >> 5;
    const int span = ((n + T - 1) / T) * T;  // whole warps take part in every pass
    if (t < 4 * D) h.cbox[0][t / (2 * D)][t % (2 * D)] = t % (2 * D) < D ? 0xffffffffu : 0u;
    if (t == 0) {
        h.bits[nw] = 0;
        h.gid[0][0] = root.node;
        h.s[0][0] = 0;
        h.n[0][0] = (uint16_t)n;
        h.nact = n > leaf;
        h.fail = 0;
    }
    __syncthreads();
    for (int i = t; i < span; i += T) {
        float c[D];
        const bool ok = i < n;
#pragma unroll
        for (int d = 0; d < D; d++) {
            c[d] = ok ? PosOf<RecT, D>::get(recs[gs + i], d) : 0.f;
            if (ok) h.pos[d][i] = c[d];
        }
        if (ok) {
            h.idx[0][i] = (uint16_t)i;
            h.own[i] = 0;
        }
        sub_box<D>(h.cbox, c, ok ? 0 : (int)RSG_NOSUB, false);
    }
    __syncthreads();
    if (t < D) {
        const float lo = ord2f(h.cbox[0][0][t]), hi = ord2f(h.cbox[0][0][D + t]);
        nodes[root.node].mn[t] = lo;
        nodes[root.node].mx[t] = hi;
        h.box[0][0][t] = lo;
        h.box[0][0][D + t] = hi;
    }
    int cur = 0, level = root.level;
    auto rank = [&](int x) {
        return h.wpre[x >> 5] + __popc(h.bits[x >> 5] & ((1u << (x & 31)) - 1u));
    };
    for (;;) {
        __syncthreads();
        const int nact = h.nact;
        if (nact == 0) break;
        level++;
        // split dimension and limit (src/fast3tree.c:736-757), as split_of
        for (int k = t; k < nact; k += T) {
            const float *bx = h.box[cur][k];
            int dim = D - 1;
            float dmax = fsub(bx[2 * D - 1], bx[D - 1]);
#pragma unroll
            for (int i = 0; i < D - 1; i++) {
                float d2 = fsub(bx[D + i], bx[i]);
                if (d2 > dmax) {
                    dmax = d2;
                    dim = i;
                }
            }
            float l = fmul(0.5f, fadd(bx[D + dim], bx[dim]));
            if (bx[D + dim] == bx[dim]) l = __int_as_float(0x7f800000);
            h.div[k] = (uint8_t)dim;
            h.lim[k] = l;
#pragma unroll
            for (int d = 0; d < D; d++) {
                h.cbox[k][0][d] = h.cbox[k][1][d] = 0xffffffffu;
                h.cbox[k][0][D + d] = h.cbox[k][1][D + d] = 0u;
            }
        }
        __syncthreads();
        for (int i = t; i < span; i += T) {
            const int k = i < n ? h.own[i] : (int)RSG_NOSUB;
            float c[D];
            bool big = false;
            if (k != RSG_NOSUB) {
                const int e = h.idx[cur][i];
#pragma unroll
                for (int d = 0; d < D; d++) c[d] = h.pos[d][e];
                big = h.pos[h.div[k]][e] > h.lim[k];
            } else {
#pragma unroll
                for (int d = 0; d < D; d++) c[d] = 0.f;
            }
            const unsigned b = __ballot_sync(0xffffffffu, big);
            if (lane == 0 && i < n) h.bits[i >> 5] = b;
            sub_box<D>(h.cbox, c, k, big);
        }
        __syncthreads();
        if (t < 32) {
            // word prefix, then counts, split decisions and the children's places
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
            __syncwarp();
            const unsigned below = (1u << lane) - 1u;
            int nsplit = 0, nnext = 0;
            for (int k0 = 0; k0 < nact; k0 += 32) {
                const int k = k0 + lane;
                bool sp = false, nl = false, nr = false;
                if (k < nact) {
                    const int s = h.s[cur][k], nn = h.n[cur][k];
                    const int rs = rank(s);
                    const int m = nn - (rank(s + nn) - rs);
                    h.m[k] = (uint16_t)m;
                    h.q[k] = (uint16_t)(rank(s + m) - rs);
                    sp = m > 0 && m < nn;
                    nl = sp && m > leaf;
                    nr = sp && nn - m > leaf;
                }
                const unsigned bsp = __ballot_sync(0xffffffffu, sp);
                const unsigned bl = __ballot_sync(0xffffffffu, nl);
                const unsigned br = __ballot_sync(0xffffffffu, nr);
                if (k < nact) {
                    int at = nnext + __popc(bl & below) + __popc(br & below);
                    h.split[k] = sp;
                    h.srank[k] = (uint16_t)(nsplit + __popc(bsp & below));
                    h.next[k][0] = nl ? (uint16_t)at++ : (uint16_t)RSG_NOSUB;
                    h.next[k][1] = nr ? (uint16_t)at : (uint16_t)RSG_NOSUB;
                }
                nsplit += __popc(bsp);
                nnext += __popc(bl) + __popc(br);
            }
            if (lane == 0) {
                const int base = atomicAdd(&ls->nnodes, 2 * nsplit);
                h.base = base;
                h.nact = nnext;
                if (level > RSG_FOREST_LEVELS) {
                    atomicMax(&ls->err, 2);
                    h.fail = 1;
                }
                if (base > cap - 2 * nsplit) {
                    atomicMax(&ls->err, 1);
                    h.fail = 1;
                }
            }
        }
        __syncthreads();
        if (h.fail) return;
        // tables of the misplaced records; children (src/fast3tree.c:798-846)
        for (int i = t; i < n; i += T) {
            const int k = h.own[i];
            if (k == RSG_NOSUB) continue;
            const int s = h.s[cur][k], l = i - s, m = h.m[k];
            const int br = rank(i) - rank(s), sr = l - br;
            const bool big = (h.bits[i >> 5] >> (i & 31)) & 1u;
            if (big && l < m) h.fb[s + br] = (uint16_t)l;
            if (!big && l >= m) h.bs[s + (m - 1 - sr)] = (uint16_t)l;
        }
        for (int e = t; e < 2 * nact; e += T) {
            const int k = e >> 1, c = e & 1, a = h.gid[cur][k];
            if (!h.split[k]) {
                if (c == 0) {
                    nodes[a].div = -1;
                    nodes[a].left = -1;
                }
                continue;
            }
            const int l = h.base + 2 * h.srank[k], m = h.m[k];
            const int cs = h.s[cur][k] + (c ? m : 0), cn = c ? h.n[cur][k] - m : m;
            if (c == 0) {
                nodes[a].div = h.div[k];
                nodes[a].left = l;
            }
            KNode<D> ch;
            ch.start = gs + cs;
            ch.n = cn;
            ch.div = -1;
            ch.left = -1;
            ch.parent = a;
            ch.tree = tree;
#pragma unroll
            for (int d = 0; d < D; d++) {
                ch.mn[d] = ord2f(h.cbox[k][c][d]);
                ch.mx[d] = ord2f(h.cbox[k][c][D + d]);
            }
            nodes[l + c] = ch;
            const int j = h.next[k][c];
            if (j != RSG_NOSUB) {
                h.gid[1 - cur][j] = l + c;
                h.s[1 - cur][j] = (uint16_t)cs;
                h.n[1 - cur][j] = (uint16_t)cn;
#pragma unroll
                for (int d = 0; d < D; d++) {
                    h.box[1 - cur][j][d] = ch.mn[d];
                    h.box[1 - cur][j][D + d] = ch.mx[d];
                }
            }
        }
        __syncthreads();
        // every place's record moves to its destination (kdtree.cuh); the
        // places then belong to the node's half they lie in
        for (int i = t; i < n; i += T) {
            const int k = h.own[i];
            const uint16_t e = h.idx[cur][i];
            if (k == RSG_NOSUB) {
                h.idx[1 - cur][i] = e;
                continue;
            }
            const int s = h.s[cur][k], l = i - s, m = h.m[k], q = h.q[k];
            const int br = rank(i) - rank(s), sr = l - br;
            const bool big = (h.bits[i >> 5] >> (i & 31)) & 1u;
            int d;
            if (!big && l < m) {
                d = l;
            } else if (big && l < m) {
                d = (br == 0) ? h.n[cur][k] - 1 : h.bs[s + br - 1] - 1;
            } else if (!big) {
                d = h.fb[s + (m - 1 - sr)];
            } else {
                const int pos_last = (q > 0) ? h.bs[s + q - 1] : h.n[cur][k];
                if (l > pos_last)
                    d = l - 1;
                else if (pos_last - m >= 2)
                    d = (l == m) ? pos_last - 1 : l - 1;
                else
                    d = l;
            }
            h.idx[1 - cur][s + d] = e;
            h.own[i] = h.split[k] ? h.next[k][l >= m] : (uint16_t)RSG_NOSUB;
        }
        cur ^= 1;
    }
    if (n <= leaf && !root.src) return;  // a leaf in its place
    // the records, 16 bytes of each at a time: read by every thread before any
    // is written over (the subtree may lie in `out` already)
    constexpr int V = sizeof(RecT) / 16, PER = S / T;
    static_assert(sizeof(RecT) % 16 == 0 && S % T == 0, "record vectors");
    const uint4 *sv = reinterpret_cast<const uint4 *>(recs + gs);
    uint4 *dv = reinterpret_cast<uint4 *>(out + gs);
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
}
template <int D, class RecT, int S, int T, int NA>
void launch_sub_build(int32_t count, RecT *recs, const RecT *scratch, const SubRoot *roots,
                      KNode<D> *nodes, LevelState *ls, int32_t cap, int leaf, cudaStream_t st) {
    if (count == 0) return;
    const size_t sm = sizeof(SubShared<D, S, NA>);
    RSG_CUDA(cudaFuncSetAttribute(k_sub_build<D, RecT, S, T, NA>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
    launch(k_sub_build<D, RecT, S, T, NA>, count, T, sm, st, recs, scratch, roots, nodes, ls,
           cap, leaf);
}

template <int D, class RecT>
Forest<D> build_forest(Arena &ar, RecT *recs, int64_t nrec, const int32_t *rstart,
                       const int32_t *rn, int32_t ntrees, int64_t n_in_trees, int leaf,
                       cudaStream_t st) {
    Forest<D> F;
    F.ntrees = ntrees;
    if (ntrees == 0) return F;
    const int T = 256;
    int64_t cap = ntrees + 4 * (n_in_trees / (leaf > 1 ? leaf : 1)) + 4096;
    if (cap > 2 * n_in_trees + ntrees + 16) cap = 2 * n_in_trees + ntrees + 16;
    // Size classes of the block-built subtrees: the largest a block's tables
    // hold, at most NA nodes of more than `leaf` records each to a level.
    constexpr int S0 = 256, S1 = 2048, NA0 = D == 3 ? 24 : 16, NA1 = D == 3 ? 192 : 64;
    const int sub0 = (int)std::min<int64_t>(S0, (int64_t)NA0 * (leaf + 1));
    const int sub = (int)std::min<int64_t>(S1, (int64_t)NA1 * (leaf + 1));
    const int64_t acap = n_in_trees / (sub + 1) + 1;  // nodes of more than `sub` records
    const int32_t nsubs = (int32_t)cap;  // a node is listed once at most
    KNode<D> *nodes = ar.get<KNode<D>>(cap);
    const size_t mark = ar.used;  // everything below is released on return
    SubRoot *subs = ar.get<SubRoot>(nsubs);
    LevelState *ls = ar.get<LevelState>(1);
    int32_t *slot = ar.get<int32_t>(ntrees);
    ActNode *act[2];
    unsigned *cbox[2];
    for (int b = 0; b < 2; b++) {
        act[b] = ar.get<ActNode>(acap);
        cbox[b] = ar.get<unsigned>(acap * 4 * D);
    }
    RSG_CUDA(cudaMemsetAsync(ls, 0, sizeof(LevelState), st));
    RSG_CUDA(cudaMemcpyAsync(&ls->nnodes, &ntrees, sizeof(ntrees), cudaMemcpyHostToDevice, st));
    launch(k_roots<D>, nblk(ntrees, T), T, 0, st, rstart, rn, ntrees, sub, sub0, nodes, act[0],
           cbox[0], slot, subs, nsubs, ls);
    RSG_CHECK_LAUNCH();
    struct Head {  // the fields of LevelState before nact[]
        int32_t nnodes, err, nsub[2], ncopy, pad[3];
    } hs;
    static_assert(offsetof(LevelState, nact) == sizeof(Head), "LevelState layout");
    int32_t nact = 0;
    RSG_CUDA(cudaMemcpyAsync(&nact, &ls->nact[0], sizeof(nact), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaMemcpyAsync(&hs, ls, sizeof(hs), cudaMemcpyDeviceToHost, st));
    RSG_CUDA(cudaStreamSynchronize(st));
    RecT *buf[2] = {recs, nullptr};  // levels scatter back and forth between these
    if (nact > 0) {
        buf[1] = ar.get<RecT>(nrec);
        int32_t *owner = ar.get<int32_t>(nrec);
        int32_t *fb = ar.get<int32_t>(nrec), *bs = ar.get<int32_t>(nrec);
        int2 *copies = ar.get<int2>(acap);
        const RankBits R = rank_alloc(ar, nrec, st);
        const bool wide = sub >= RSG_STRETCH;
        const int32_t nt = (int32_t)rank_tiles(nrec);
        RSG_CUDA(cudaMemsetAsync(owner, 0xff, sizeof(int32_t) * nrec, st));
        int64_t avg = n_in_trees / ntrees, y = avg / 2048;
        dim3 g((unsigned)ntrees, (unsigned)(y < 1 ? 1 : (y > 4096 ? 4096 : y)));
        launch(k_root_owner, g, 256, 0, st, rstart, rn, ntrees, (const int32_t *)slot, owner);
        launch(k_lv_flags<D, RecT>, nt, 256, 0, st, (const RecT *)recs, nrec,
               (const int32_t *)owner, (const ActNode *)act[0], cbox[0], R, wide);
        launch(k_root_split<D>, nblk(nact, T), T, 0, st, nodes, act[0], cbox[0],
               (const LevelState *)ls);
        RSG_CHECK_LAUNCH();
        // Levels of the nodes above `sub` records run back to back with their
        // counts on the device; the host reads them every RSG_FOREST_BATCH
        // levels (every one in large calls: a level past the last costs passes
        // over nrec records).  Grids are sized by an upper bound of the nodes
        // (ub): at most twice the previous level's, and one per sub + 1 records.
        const int batch = nrec > (1 << 22) ? 1 : RSG_FOREST_BATCH;
        int64_t ub = nact;
        int level = 0, cur = 0;
        while (nact > 0) {
            for (int b = 0; b < batch; b++) {
                if (++level > RSG_FOREST_LEVELS) {
                    set_error(RSG_ERR_LIMIT, "kd-forest build exceeded %d levels", RSG_FOREST_LEVELS);
                    throw Failure();
                }
                const int x = (level - 1) & 1;
                launch(k_lv_flags<D, RecT>, nt, 256, 0, st, (const RecT *)buf[cur], nrec,
                       (const int32_t *)owner, (const ActNode *)act[x], cbox[x], R, wide);
                launch(k_rank_scan, 1, 1024, 0, st, R.tpre, nt);
                launch(k_lv_nodes<D>, nblk(ub, 64), 64, 0, st, nodes, act[x], act[1 - x],
                       (const unsigned *)cbox[x], cbox[1 - x], ls, R, level, (int32_t)cap, leaf,
                       sub, sub0, 1 - cur, subs, nsubs, copies);
                launch(k_lv_tables, nt, 256, 0, st, nrec, (const int32_t *)owner,
                       (const ActNode *)act[x], R, fb, bs, wide);
                launch(k_lv_scatter<RecT>, nt, 256, 0, st, nrec, owner, (const ActNode *)act[x],
                       R, (const int32_t *)fb, (const int32_t *)bs, (const RecT *)buf[cur],
                       buf[1 - cur], wide);
                RSG_CHECK_LAUNCH();
                cur ^= 1;
                ub = std::min<int64_t>(2 * ub, acap);
            }
            RSG_CUDA(cudaMemcpyAsync(&nact, &ls->nact[level], sizeof(nact),
                                     cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaMemcpyAsync(&hs, ls, sizeof(hs), cudaMemcpyDeviceToHost, st));
            RSG_CUDA(cudaStreamSynchronize(st));
            if (hs.err) break;
            ub = nact;
        }
        if (hs.ncopy && !hs.err)
            launch(k_copy_segs<RecT>, dim3(hs.ncopy, 64), 256, 0, st, (const int2 *)copies,
                   (const RecT *)buf[1], recs);
    }
    if (!hs.err) {
        // the larger class first: its blocks are the long ones
        launch_sub_build<D, RecT, S1, 512, NA1>(hs.nsub[1], recs, (const RecT *)buf[1],
                                                (const SubRoot *)subs + (nsubs - hs.nsub[1]),
                                                nodes, ls, (int32_t)cap, leaf, st);
        launch_sub_build<D, RecT, S0, 128, NA0>(hs.nsub[0], recs, (const RecT *)buf[1],
                                                (const SubRoot *)subs, nodes, ls, (int32_t)cap,
                                                leaf, st);
        RSG_CHECK_LAUNCH();
        RSG_CUDA(cudaMemcpyAsync(&hs, ls, sizeof(hs), cudaMemcpyDeviceToHost, st));
        RSG_CUDA(cudaStreamSynchronize(st));
    }
    if (hs.err == 2) {
        set_error(RSG_ERR_LIMIT, "kd-forest build exceeded %d levels", RSG_FOREST_LEVELS);
        throw Failure();
    }
    if (hs.err) {
        set_error(RSG_ERR_LIMIT, "kd-forest node capacity %lld exceeded", (long long)cap);
        throw Failure();
    }
    F.nodes = nodes;
    F.nnodes = hs.nnodes;
    ar.used = mark;
    return F;
}

}  // namespace rsg
