// Stage 2 on the device: edge tensors, sparse valid mask, cross-tile cost
// propagation, overlap sync, global top/right edge scan, and the stitched
// backtrace.  Every rule restates Parflex.py literally; the tile loops of the
// reference become grids over edge slots.  All slot arrays are laid out like
// the reference's 4-D arrays: [n1][n2][2][L] (edge 0 = top edge = the tile's
// last row, indexed by column; edge 1 = right edge = its last column, indexed
// by row).
//
// Every kernel takes one alignment by value or a device table of them
// (blockIdx.y: a wave of a batch), so a batch's stage 2 is as many launches as
// one alignment's.
#include <cooperative_groups.h>
#include <math_constants.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "prop_list.cuh"

namespace pfx {

namespace cg = cooperative_groups;


__device__ __forceinline__ int64_t slot(const Geo& g, int i, int j, int e, int64_t p) {
    return (((int64_t)i * g.n2 + j) * 2 + e) * g.L + p;
}

__device__ __forceinline__ void decode_start(int32_t s, int32_t* sr, int32_t* sc) {
    // _build_edge_data (Parflex.py:531-546): > 0 bottom edge, < 0 left edge,
    // 0 the corner.
    if (s > 0) { *sr = 0; *sc = s; }
    else if (s < 0) { *sr = -s; *sc = 0; }
    else { *sr = 0; *sc = 0; }
}

// Fill value kernels ------------------------------------------------------
__global__ void k_fill_f64(double* p, int64_t n, double v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        p[i] = v;
}

// 1 - sum_f a[f * lda] * b[f * ldb], every product and sum rounded in the
// order f = 0, 1, ..., d-1: the value the cost kernels store for that cell.
__device__ __forceinline__ double cost_from_features(const double* a, int64_t lda,
                                                     const double* b, int64_t ldb, int d) {
    double acc = __dmul_rn(a[0], b[0]);
    for (int f = 1; f < d; ++f) acc = __dadd_rn(acc, __dmul_rn(a[f * lda], b[f * ldb]));
    return __dsub_rn(1.0, acc);
}

// The valid marks of every pair of a table to 0 (16 bytes per thread and step;
// a plan's buffers are 256-byte aligned).
__global__ void __launch_bounds__(256) k_clear_valid(const S2Pair* __restrict__ tab) {
    const S2Pair& p = tab[blockIdx.y];
    const int64_t n = (int64_t)p.g.n1 * p.g.n2 * 2 * p.g.L;
    uint8_t* v = p.b.valid;
    const int64_t step = (int64_t)gridDim.x * 256 * 16;
    for (int64_t q = ((int64_t)blockIdx.x * 256 + threadIdx.x) * 16; q < n; q += step) {
        if (q + 16 <= n) {
            *reinterpret_cast<uint4*>(v + q) = make_uint4(0, 0, 0, 0);
        } else {
            for (int64_t x = q; x < n; ++x) v[x] = 0;
        }
    }
}

// Edge tensors + valid mask (Parflex.py:509-564, 347-373, 582-624) -------
// C: row-major cost (leading dimension g.ldc), or null to read the tile-skewed
// copy Csk (per-tile stride `skew_stride` elements; FP32 elements when `f32`,
// widened exactly to FP64), or, with An non-null, computed from the
// normalised features (An: [d][N], Bn: [d][M]).
// D_arr and L_arr start out +inf.
__global__ void __launch_bounds__(256) k_edges(const S2Pair one, const S2Pair* __restrict__ tab) {
    const S2Pair& p = tab ? tab[blockIdx.y] : one;
    const Geo g = p.g;
    const S2Buf b = p.b;
    const S2Src src = p.src;
    const int64_t total = (int64_t)g.n1 * g.n2 * 2 * g.L;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < total;
         q += (int64_t)gridDim.x * blockDim.x) {
        b.D_arr[q] = CUDART_INF;
        b.L_arr[q] = CUDART_INF;
        const int64_t pos = q % g.L;
        const int64_t te = q / g.L;
        const int e = (int)(te % 2);
        const int64_t t = te / 2;
        const int i = (int)(t / g.n2), j = (int)(t % g.n2);
        int64_t r0, c0;
        int32_t R, W;
        tile_rect(g, i, j, &r0, &c0, &R, &W);
        const int32_t elen = e == 0 ? W : R;
        if (pos >= elen) { b.edge_Cf[q] = 0.0; continue; }
        const int32_t s = b.edge_P[q];
        int32_t sr, sc;
        decode_start(s, &sr, &sc);
        const int64_t slab = b.tile_slot ? b.tile_slot[t] : t;
        const int64_t si = slab * src.skew_stride + skew_index(W, sr, sc);
        // a tile stage 1 skipped has no cost slab: its edges are +inf anyway
        b.edge_Cf[q] = slab < 0 ? 0.0
                       : src.An ? cost_from_features(src.An + r0 + sr, g.N, src.Bn + c0 + sc,
                                                     g.M, src.d)
                       : (src.C ? src.C[(r0 + sr) * g.ldc + c0 + sc]
                                : (src.f32 ? (double)static_cast<const float*>(src.Csk)[si]
                                           : static_cast<const double*>(src.Csk)[si]));
        // mandatory slots: whole top edge of the last tile row, whole right
        // edge of the last tile column, and both ends of every edge
        const bool last = e == 0 ? (i == g.n1 - 1) : (j == g.n2 - 1);
        if (last || pos == 0 || pos == elen - 1) b.valid[q] = 1;
        // starts_bot_edge of tile (i, j) marks the top edge of (i-1, j);
        // starts_left_edge marks the right edge of (i, j-1)
        if (s > 0) {
            if (i >= 1 && s < W) b.valid[slot(g, i - 1, j, 0, s)] = 1;
        } else {
            if (j >= 1) {
                int64_t pr0, pc0;
                int32_t pR, pW;
                tile_rect(g, i, j - 1, &pr0, &pc0, &pR, &pW);
                if (-s < pR) b.valid[slot(g, i, j - 1, 1, -s)] = 1;
            }
        }
    }
}

// Predecessor edge slot holding global cell (gr, gc) of tile (pi, pj)
// (Parflex.py:686-700, 822-839).
__device__ __forceinline__ bool prev_slot(const Geo& g, int pi, int pj, int64_t gr, int64_t gc,
                                          int* pe, int64_t* pp) {
    int64_t r0, c0;
    int32_t R, W;
    tile_rect(g, pi, pj, &r0, &c0, &R, &W);
    const int64_t lr = gr - r0, lc = gc - c0;
    int64_t elen;
    if (lr == R - 1) { *pe = 0; *pp = lc; elen = W; }
    else if (lc == W - 1) { *pe = 1; *pp = lr; elen = R; }
    else return false;
    return *pp >= 0 && *pp < elen;
}

// Stage-2 DP (_nb_initialize_chunks_sparse / _nb_dp_fill_chunks_sparse,
// Parflex.py:632-855), tile anti-diagonal by anti-diagonal: every slot reads
// only slots of tiles (i-1, j) and (i, j-1), so a diagonal's tiles are
// independent.

// Unconditional inheritance of position 0 on the first tile row / column.
__device__ __forceinline__ void prop_inherit(const Geo& g, S2Buf& b, int i, int j) {
    double* D = b.D_arr;
    double* Lr = b.L_arr;
    if (i == 0 && j >= 1) {
        int64_t pr0, pc0;
        int32_t pR, pW;
        tile_rect(g, 0, j - 1, &pr0, &pc0, &pR, &pW);
        D[slot(g, 0, j, 0, 0)] = __ldcg(D + slot(g, 0, j - 1, 0, pW - 1));
        Lr[slot(g, 0, j, 0, 0)] = __ldcg(Lr + slot(g, 0, j - 1, 0, pW - 1));
    } else if (j == 0 && i >= 1) {
        int64_t pr0, pc0;
        int32_t pR, pW;
        tile_rect(g, i - 1, 0, &pr0, &pc0, &pR, &pW);
        D[slot(g, i, 0, 1, 0)] = __ldcg(D + slot(g, i - 1, 0, 1, pR - 1));
        Lr[slot(g, i, 0, 1, 0)] = __ldcg(Lr + slot(g, i - 1, 0, 1, pR - 1));
    }
}

// How valid slot k gets its value: nothing to do, its own edge value (a start
// on the alignment's own border or inside the tile), another slot's value, or
// another slot's value plus its own edge value less the overlap.
enum { kPropNone, kPropOwn, kPropCopy, kPropChain };

__device__ __forceinline__ int prop_source(const Geo& g, const S2Buf& b, int64_t k, int64_t* src,
                                           int* dr, int* dc) {
    const int pos = (int)(k % g.L);
    const int64_t te = k / g.L;
    const int e = (int)(te & 1);
    const int i = (int)((te >> 1) / g.n2), j = (int)((te >> 1) % g.n2);
    int64_t r0, c0;
    int32_t R, W;
    tile_rect(g, i, j, &r0, &c0, &R, &W);
    if (pos >= (e == 0 ? W : R)) return kPropNone;
    if (pos == 0 && (i == 0) != (j == 0)) return kPropNone;  // inherited (prop_inherit)
    if (pos == 0 && i > 0 && j > 0) {
        int64_t pr0, pc0;
        int32_t pR, pW;
        if (e == 0) {
            tile_rect(g, i, j - 1, &pr0, &pc0, &pR, &pW);
            *src = slot(g, i, j - 1, 0, pW - 1);
        } else {
            tile_rect(g, i - 1, j, &pr0, &pc0, &pR, &pW);
            *src = slot(g, i - 1, j, 1, pR - 1);
        }
        return kPropCopy;
    }
    int32_t sr, sc;
    decode_start(b.edge_P[k], &sr, &sc);
    const int32_t lr = e == 0 ? R - 1 : pos, lc = e == 0 ? pos : W - 1;
    *dr = abs(lr - sr);
    *dc = abs(lc - sc);
    int pi, pj;
    if (i == 0 && j == 0) {
        return sr == 0 || sc == 0 ? kPropOwn : kPropNone;
    } else if (i == 0) {
        if (sr == 0) return kPropOwn;
        if (sc != 0) return kPropNone;
        pi = 0; pj = j - 1;
    } else if (j == 0) {
        if (sc == 0) return kPropOwn;
        if (sr != 0) return kPropNone;
        pi = i - 1; pj = 0;
    } else {
        if (sr == 0) { pi = i - 1; pj = j; }
        else if (sc == 0) { pi = i; pj = j - 1; }
        else return kPropOwn;
    }
    int pe;
    int64_t pp;
    if (!prev_slot(g, pi, pj, r0 + sr, c0 + sc, &pe, &pp)) return kPropNone;
    *src = slot(g, pi, pj, pe, pp);
    return kPropChain;
}

// Tiles (i, j) with i + j < a.
__device__ __forceinline__ int64_t tiles_before(const Geo& g, int a) {
    auto tri = [](int64_t x) { return x > 0 ? x * (x + 1) / 2 : 0; };
    return tri(a) - tri((int64_t)a - g.n1) - tri((int64_t)a - g.n2);
}

// The valid slots that depend on another slot, gathered per tile
// anti-diagonal (diagonal a's at diag_list[tiles_before(a) * 2 L ..),
// diag_count[a] of them, in no order) with the slot each reads (prop_list.cuh);
// those that do not get their value here.  Few slots are valid, so the
// propagation reads 8 bytes per such slot instead of a byte per slot, and the
// only thing left to wait for on a diagonal is the value of the slot before.
__global__ void __launch_bounds__(256) k_valid_lists(const S2Pair one,
                                                     const S2Pair* __restrict__ tab) {
    const S2Pair& p = tab ? tab[blockIdx.y] : one;
    const Geo& g = p.g;
    const S2Buf& b = p.b;
    const int64_t total = (int64_t)g.n1 * g.n2 * 2 * g.L;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total;
         k += (int64_t)gridDim.x * blockDim.x) {
        if (!b.valid[k]) continue;
        int64_t src = 0;
        int dr = 0, dc = 0;
        const int how = prop_source(g, b, k, &src, &dr, &dc);
        if (how == kPropOwn) {
            b.D_arr[k] = b.edge_D[k];
            b.L_arr[k] = (double)(dr + dc);
        } else if (how != kPropNone) {
            const int t = (int)(k / (2 * g.L)), i = t / g.n2;
            const int a = i + t % g.n2;
            // one atomic for the warp's slots of a diagonal
            const unsigned same = __match_any_sync(__activemask(), a);
            const int lane = threadIdx.x & 31, lead = __ffs(same) - 1;
            int at = 0;
            if (lane == lead) at = atomicAdd(b.diag_count + a, __popc(same));
            at = __shfl_sync(same, at, lead) + __popc(same & ((1u << lane) - 1u));
            b.diag_list[tiles_before(g, a) * 2 * g.L + at] =
                make_int2(prop_place(g.n2, 2 * g.L, a, i, k),
                          prop_back(k, src, how == kPropCopy));
        }
    }
}

// What a dependent slot adds to the slot it reads (copy: nothing).
struct PropItem {
    int64_t k, src;  // k < 0: none
    bool copy;
    double eD, eC, dr, dc;
};

// Entry v of anti-diagonal a.
__device__ __forceinline__ PropItem prop_item(const Geo& g, const S2Buf& b, int a, int2 v) {
    PropItem it;
    int i;
    it.k = prop_slot(g.n2, 2 * g.L, a, v.x, &i);
    it.src = prop_src(it.k, v.y);
    it.copy = v.y < 0;
    it.eD = b.edge_D[it.k];
    it.eC = b.edge_Cf[it.k];
    const int q = v.x % (2 * g.L);
    const bool top = q < g.L;
    const int pos = top ? q : q - g.L;
    int64_t r0, c0;
    int32_t R, W, sr, sc;
    tile_rect(g, i, a - i, &r0, &c0, &R, &W);
    decode_start(b.edge_P[it.k], &sr, &sc);
    it.dr = (double)abs((top ? R - 1 : pos) - sr);
    it.dc = (double)abs((top ? pos : W - 1) - sc);
    return it;
}

// (other SMs' values of this launch: read past L1)
__device__ __forceinline__ void prop_apply(const S2Buf& b, const PropItem& it) {
    const double prev = __ldcg(b.D_arr + it.src), len = __ldcg(b.L_arr + it.src);
    if (!isfinite(prev)) return;
    b.D_arr[it.k] = it.copy ? prev : __dsub_rn(__dadd_rn(prev, it.eD), it.eC);
    b.L_arr[it.k] = it.copy ? len : __dadd_rn(__dadd_rn(len, it.dr), it.dc);
}

// The propagation in one launch: a cluster of CTAs per alignment takes the
// diagonals in order, a cluster barrier between two.  A thread's first slot of
// a diagonal is fetched while the barrier completes, so that a diagonal costs
// one dependent read, a write and the barrier.  diag_count ends up zero again.
// Measured: 7 diagonals of 4000-column tiles 30 us (one CTA over all slots 128
// us), 39 of 2000-column tiles 112 us (a launch per diagonal 156 us).
constexpr int kPropThreads = 512;

__global__ void __launch_bounds__(kPropThreads) k_propagate(const S2Pair one,
                                                            const S2Pair* __restrict__ tab) {
    cg::cluster_group cl = cg::this_cluster();
    const S2Pair& p = tab ? tab[blockIdx.y] : one;
    const Geo g = p.g;
    S2Buf b = p.b;
    const int nthr = (int)cl.num_blocks() * kPropThreads;
    const int tid = (int)cl.block_rank() * kPropThreads + (int)threadIdx.x;
    const int nd = g.n1 + g.n2 - 1;
    auto list_of = [&](int a) { return b.diag_list + tiles_before(g, a) * 2 * g.L; };
    auto first = [&](int a, int n) {
        PropItem it;
        it.k = -1;
        if (tid < n) it = prop_item(g, b, a, list_of(a)[tid]);
        return it;
    };
    int n = b.diag_count[0];
    int n_next = nd > 1 ? b.diag_count[1] : 0;
    PropItem it = first(0, n);
    for (int a = 0; a < nd; ++a) {
        if (it.k >= 0) prop_apply(b, it);
        for (int x = tid + nthr; x < n; x += nthr) prop_apply(b, prop_item(g, b, a, list_of(a)[x]));
        const int ilo = diag_row0(g.n2, a);
        const int ihi = a < g.n1 - 1 ? a : g.n1 - 1;
        // the diagonal's tiles on the first tile row / column
        if (tid == nthr - 1 && ilo == 0) prop_inherit(g, b, 0, a);
        if (tid == nthr - 2 && a - ihi == 0) prop_inherit(g, b, ihi, 0);
        cg::cluster_group::arrival_token tok = cl.barrier_arrive();
        n = n_next;
        n_next = a + 2 < nd ? b.diag_count[a + 2] : 0;
        it = first(a + 1, n);
        cl.barrier_wait(std::move(tok));
    }
    for (int a = tid; a < nd; a += nthr) b.diag_count[a] = 0;
}

// sync_tile_overlap_edges (Parflex.py:920-969).  Loops 1 and 2 touch
// disjoint slots (edge 0 / edge 1) and their pairs are disjoint, loop 3 runs
// after both.  Work item t of 2 n1 n2 (loops 1 and 2), or of n1 n2 (loop 3).
__device__ __forceinline__ void sync_overlap(const Geo& g, const S2Buf& b, int t) {
    double* D = b.D_arr;
    double* Lr = b.L_arr;
    const int nt = g.n1 * g.n2;
    const int which = t / nt, tt = t % nt;
    const int i = tt / g.n2, j = tt % g.n2;
    int64_t r0, c0;
    int32_t R, W;
    tile_rect(g, i, j, &r0, &c0, &R, &W);
    int64_t a, c;
    if (which == 0) {
        if (j + 1 >= g.n2) return;
        a = slot(g, i, j, 0, W - 1);
        c = slot(g, i, j + 1, 0, 0);
    } else {
        if (i + 1 >= g.n1) return;
        a = slot(g, i, j, 1, R - 1);
        c = slot(g, i + 1, j, 1, 0);
    }
    const bool fa = isfinite(D[a]), fc = isfinite(D[c]);
    if (fa && !fc) { D[c] = D[a]; Lr[c] = Lr[a]; }
    else if (!fa && fc) { D[a] = D[c]; Lr[a] = Lr[c]; }
}

__device__ __forceinline__ void sync_corner(const Geo& g, const S2Buf& b, int t) {
    double* D = b.D_arr;
    double* Lr = b.L_arr;
    const int i = t / g.n2, j = t % g.n2;
    int64_t r0, c0;
    int32_t R, W;
    tile_rect(g, i, j, &r0, &c0, &R, &W);
    const int64_t tc = slot(g, i, j, 0, W - 1), rc = slot(g, i, j, 1, R - 1);
    const double dt = __ldcg(D + tc), dr = __ldcg(D + rc);
    const bool ft = isfinite(dt), fr = isfinite(dr);
    if (ft && !fr) { D[rc] = dt; Lr[rc] = __ldcg(Lr + tc); }
    else if (!ft && fr) { D[tc] = dr; Lr[tc] = __ldcg(Lr + rc); }
    else if (ft && fr && fabs(dt - dr) > 1e-10) { D[rc] = dt; Lr[rc] = __ldcg(Lr + tc); }
}

// First-minimum of (norm, index) over a CTA: smaller norm, then smaller index
// (index < 0: none).  Every thread of the CTA calls; thread 0 has the result.
__device__ __forceinline__ void block_first_min(double& n, int64_t& i, double* sn, int64_t* si) {
    auto better = [](double an, int64_t ai, double bn, int64_t bi) {
        return ai >= 0 && (bi < 0 || an < bn || (an == bn && ai < bi));
    };
    for (int o = 16; o > 0; o >>= 1) {
        const double on = __shfl_down_sync(0xffffffffu, n, o);
        const int64_t oi = __shfl_down_sync(0xffffffffu, i, o);
        if (better(on, oi, n, i)) { n = on; i = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) { sn[warp] = n; si[warp] = i; }
    __syncthreads();
    if (warp == 0) {
        const int nw = (int)blockDim.x >> 5;
        n = lane < nw ? sn[lane] : CUDART_INF;
        i = lane < nw ? si[lane] : -1;
        for (int o = 16; o > 0; o >>= 1) {
            const double on = __shfl_down_sync(0xffffffffu, n, o);
            const int64_t oi = __shfl_down_sync(0xffffffffu, i, o);
            if (better(on, oi, n, i)) { n = on; i = oi; }
        }
    }
}

// Overlap sync, then the global edge scan (_build_edge_lookups +
// _nb_scan_edges, Parflex.py:1110-1222), one cluster per alignment.  Its CTAs
// take the L-wide segments of the global top edge (s < nseg_top) and of the
// right edge in turn.  The first owner of a global top column g is tile (n1-1,
// g == 0 ? 0 : (g-1)/hop) at position g - j*hop (the last tile row is the only
// one containing row N-1, and of two tiles sharing column g the lower j is
// visited first); likewise for right-edge rows.  The global winner then comes
// from the segment winners in scan order (top segments, then right segments);
// strict < against the running best that starts at LARGE = 1e9
// (Parflex.py:1167-1168).
constexpr int kScanThreads = 1024;

// buffer_global (Parflex.py:1520), every operation rounded in its order; one
// that is no int64 excludes nothing.
__device__ __forceinline__ int64_t buffer_global(int64_t N, int64_t M, double beta) {
    const double mn = (double)(N < M ? N : M), mx = (double)(N < M ? M : N);
    const double part = __ddiv_rn(__dmul_rn(__dsub_rn(1.0, beta), mn), mx);
    const double bg = __dmul_rn(mn, __dsub_rn(1.0, part));
    return fabs(bg) < 0x1p63 ? (int64_t)bg : 0;
}

__global__ void __launch_bounds__(kScanThreads) k_scan(const S2Pair one,
                                                       const S2Pair* __restrict__ tab,
                                                       const double beta) {
    __shared__ double sn[32];
    __shared__ int64_t si[32];
    cg::cluster_group cl = cg::this_cluster();
    const S2Pair& p = tab ? tab[blockIdx.y] : one;
    const Geo g = p.g;
    const S2Buf b = p.b;
    const int64_t buf = buffer_global(g.N, g.M, beta);
    const int nb = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int nthr = nb * kScanThreads, tid = rank * kScanThreads + (int)threadIdx.x;
    const int nt = g.n1 * g.n2;
    for (int t = tid; t < 2 * nt; t += nthr) sync_overlap(g, b, t);
    cl.sync();
    for (int t = tid; t < nt; t += nthr) sync_corner(g, b, t);
    cl.sync();
    const int nst = (int)((g.M + g.L - 1) / g.L), nsr = (int)((g.N + g.L - 1) / g.L);
    for (int s = rank; s < 2 * b.max_segs; s += nb) {
        const bool top = s < b.max_segs;
        const int row = top ? 0 : 1;
        const int seg = top ? s : s - b.max_segs;
        double bn = CUDART_INF;
        int64_t bgi = -1;
        if (seg < (top ? nst : nsr)) {
            const int64_t G = top ? g.M : g.N;
            const int64_t lo = (int64_t)seg * g.L;
            const int64_t hi = lo + g.L < G ? lo + g.L : G;
            for (int64_t gi = lo + threadIdx.x; gi < hi; gi += kScanThreads) {
                const int tj_or_i = gi == 0 ? 0 : (int)((gi - 1) / g.hop);
                const int64_t k = slot(g, top ? g.n1 - 1 : tj_or_i, top ? tj_or_i : g.n2 - 1,
                                       row, gi - (int64_t)tj_or_i * g.hop);
                const double Dv = __ldcg(b.D_arr + k), Lv = __ldcg(b.L_arr + k);
                const bool in = !(buf > 0 && gi < buf) && isfinite(Dv) && !(Lv <= 0.0) &&
                                !(top && Dv >= 1e9);
                (top ? b.top_D : b.right_D)[gi] = in ? Dv : CUDART_NAN;
                (top ? b.top_L : b.right_L)[gi] = in ? Lv : 0.0;
                if (!in) continue;
                const double nrm = __ddiv_rn(Dv, Lv);
                if (nrm < bn) { bn = nrm; bgi = gi; }  // strided: gi ascends per thread
            }
        }
        block_first_min(bn, bgi, sn, si);
        if (threadIdx.x == 0) {
            int64_t* m = b.seg_meta + ((int64_t)row * b.max_segs + seg) * 6;
            if (bgi >= 0) {
                const int tj_or_i = bgi == 0 ? 0 : (int)((bgi - 1) / g.hop);
                b.seg_norm[row * b.max_segs + seg] = bn;
                m[0] = top ? g.n1 - 1 : tj_or_i;
                m[1] = top ? tj_or_i : g.n2 - 1;
                m[2] = row;
                m[3] = bgi - (int64_t)tj_or_i * g.hop;
                m[4] = top ? g.N - 1 : bgi;
                m[5] = top ? bgi : g.M - 1;
            } else {
                b.seg_norm[row * b.max_segs + seg] = CUDART_INF;
                for (int f = 0; f < 6; ++f) m[f] = -1;
            }
        }
        __syncthreads();
    }
    cl.sync();
    if (rank != 0) return;
    // the first segment, in scan order, of the least norm below 1e9
    double bn = CUDART_INF;
    int64_t bs = -1;
    for (int s = threadIdx.x; s < nst + nsr; s += kScanThreads) {
        const int row = s < nst ? 0 : 1, seg = s < nst ? s : s - nst;
        const double nrm = __ldcg(b.seg_norm + row * b.max_segs + seg);
        const bool some = __ldcg(b.seg_meta + ((int64_t)row * b.max_segs + seg) * 6) >= 0;
        if (some && nrm < 1e9 && nrm < bn) { bn = nrm; bs = s; }
    }
    block_first_min(bn, bs, sn, si);
    if (threadIdx.x == 0) {
        *b.best = bs >= 0 ? bn : 1e9;
        int64_t e[6] = {-1, -1, -1, -1, -1, -1};
        if (bs >= 0) {
            const int row = bs < nst ? 0 : 1, seg = (int)(bs < nst ? bs : bs - nst);
            const int64_t* m = b.seg_meta + ((int64_t)row * b.max_segs + seg) * 6;
            const int at[6] = {4, 5, 0, 1, 2, 3};
            for (int f = 0; f < 6; ++f) e[f] = __ldcg(m + at[f]);
        }
        for (int f = 0; f < 6; ++f) b.best_end[f] = e[f];
        b.best_end[6] = bs >= 0 ? 1 : 0;
    }
}

// Tile chain of the stitched backtrace (backtrace_and_stitch,
// Parflex.py:1032-1103).  The chain needs only the start encodings on the
// tile edges, so it is followed first and the per-tile walks run in parallel
// afterwards.  Entry fields: i j edge idx end_r end_c start_r start_c row0 col0
// rows cols.  From a start (from_best: the scan's endpoint); calls
// entry(n, E) for each and stops after entry number `last`; returns how many
// entries it visited.
struct ChainStart {
    int64_t i, j, e, x;
    int from_best;
};
constexpr int kChainMax = 101;

template <typename F>
__device__ __forceinline__ int follow_chain(const Geo& g, const S2Buf& b, const ChainStart& s,
                                            int last, F entry) {
    int64_t ci = s.i, cj = s.j, ce = s.e, cx = s.x;
    if (s.from_best) {
        if (!b.best_end[6]) return 0;
        ci = b.best_end[2]; cj = b.best_end[3]; ce = b.best_end[4]; cx = b.best_end[5];
    }
    int n = 0;
    for (int it = 0; it < kChainMax; ++it) {
        if (ci < 0 || cj < 0 || ci >= g.n1 || cj >= g.n2) break;
        int64_t r0, c0;
        int32_t R, W;
        tile_rect(g, (int)ci, (int)cj, &r0, &c0, &R, &W);
        const int32_t sv = b.edge_P[slot(g, (int)ci, (int)cj, (int)ce, cx)];
        const int32_t sr = sv >= 0 ? 0 : -sv, sc = sv >= 0 ? sv : 0;
        const int32_t E[12] = {(int32_t)ci, (int32_t)cj, (int32_t)ce, (int32_t)cx,
                               ce == 0 ? R - 1 : (int32_t)cx, ce == 0 ? (int32_t)cx : W - 1,
                               sr, sc, (int32_t)r0, (int32_t)c0, R, W};
        entry(n, E);
        if (++n > last) break;
        const int64_t gsr = r0 + sr, gsc = c0 + sc;
        if (gsr == 0 || gsc == 0) break;
        const bool corner = sr == 0 && sc == 0;
        int64_t pi, pj, pe;
        if (corner) { pi = ci - 1; pj = cj - 1; pe = 0; }
        else if (sv >= 0) { pi = ci - 1; pj = cj; pe = 0; }
        else { pi = ci; pj = cj - 1; pe = 1; }
        if (pi < 0 || pj < 0 || pi >= g.n1 || pj >= g.n2) break;
        int64_t pr0, pc0;
        int32_t pR, pW;
        tile_rect(g, (int)pi, (int)pj, &pr0, &pc0, &pR, &pW);
        int64_t pidx, pmax;
        if (corner) { pidx = pW - 1; pmax = pW; }
        else {
            pidx = pe == 0 ? gsc - pc0 : gsr - pr0;
            pmax = pe == 0 ? pW : pR;
        }
        if (pidx < 0 || pidx >= pmax) break;
        ci = pi; cj = pj; ce = pe; cx = pidx;
    }
    return n;
}

__global__ void k_stitch_chain(const Geo g, S2Buf b, const ChainStart s) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    *b.chain_len = follow_chain(g, b, s, kChainMax - 1, [&](int n, const int32_t* E) {
        for (int f = 0; f < 12; ++f) b.chain[n * 12 + f] = E[f];
    });
}

// One chain entry per CTA of one warp: walk the packed backpointers from the
// entry's end cell to its start cell (_nb_backtrace_within_chunk,
// Parflex.py:977-1012), writing global points end-first.  The CTA first
// follows the chain to its entry (every lane the same).
//
// The walk is one dependent chain, so its time is the latency of a step.  The
// backpointers of a strip are laid out [period of 16 steps tau = c + rho][row
// rho]: the words the path can need in a strip of 64 rows lie in about 20
// consecutive periods of 64 words.  They are copied to shared memory
// asynchronously while the path crosses the strip below (two buffers), and a
// step reads its word at ((tau / 16) mod 32) * 64 + rho: one shared-memory
// load and six dependent integer instructions, with (rho, tau) as the walk's
// state.  A step moves at most two rows and two columns, so min(rho, c) / 2
// steps run without a test; a step number that is none (nothing won) moves
// nowhere, which shows after them.
// Measured: tiles of 4000 rows 173 us, of 2000 rows 105 us, of 500 rows 27 us;
// with a window of words per 64 x 64 cells, loaded when the path left it, and
// every test in every step 655, 354 and 81 us.
constexpr int kWalkPeriods = 32;  // periods a buffer holds (24 are fetched)
constexpr int kWalkFetch = 24;

__global__ void __launch_bounds__(32) k_walk(const S2Pair one, const S2Pair* __restrict__ tab,
                                             const ChainStart s) {
    __shared__ __align__(16) uint32_t win[2][kWalkPeriods * 64];
    const S2Pair& p = tab ? tab[blockIdx.y] : one;
    const Geo g = p.g;
    const S2Buf b = p.b;
    const int lane = threadIdx.x, e = blockIdx.x;
    int32_t ti = -1, tj = 0, r = 0, c = 0, sr = 0, sc = 0, gro = 0, gco = 0, R = 0, W = 0;
    const int n = follow_chain(g, b, s, e == 0 ? kChainMax - 1 : e, [&](int m, const int32_t* E) {
        if (e == 0 && lane < 12) {
            int32_t v = 0;
#pragma unroll
            for (int f = 0; f < 12; ++f) v = lane == f ? E[f] : v;
            b.chain[m * 12 + lane] = v;
        }
        if (m == e) {
            ti = E[0]; tj = E[1]; r = E[4]; c = E[5]; sr = E[6]; sc = E[7];
            gro = E[8]; gco = E[9]; R = E[10]; W = E[11];
        }
    });
    if (e == 0 && lane == 0) *b.chain_len = n;
    if (ti < 0) return;
    const uint32_t* slab = b.Bw + ((int64_t)ti * g.n2 + tj) * g.b_words;
    const int32_t nP = ceil_div32(W + kStripRows - 1, kBlk);
    const uint32_t win0 = (uint32_t)__cvta_generic_to_shared(win[0]);
    constexpr uint32_t kBuf = kWalkPeriods * 64 * 4;
    // periods [hi - kWalkFetch + 1, hi] of strip k into buffer k & 1
    auto fetch = [&](int32_t k, int32_t hi) {
        if (k >= 0) {
            const uint32_t dst = win0 + (k & 1) * kBuf;
            const int32_t lo = hi - kWalkFetch + 1 > 0 ? hi - kWalkFetch + 1 : 0;
            const char* src = reinterpret_cast<const char*>(slab + (int64_t)k * nP * 64);
            for (int32_t x = lo * 16 + lane; x < (hi + 1) * 16; x += 32)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                 dst + (uint32_t)(x & (kWalkPeriods * 16 - 1)) * 16),
                             "l"(src + (int64_t)x * 16)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int2* out = reinterpret_cast<int2*>(b.seg_pts) + (int64_t)e * b.seg_cap;
    // by code, a byte each: rows moved, and rows plus columns; 0: no such step
    uint32_t mv_r = 0, mv_t = 0;
    for (int q = 0; q < g.S; ++q) {
        const int kd = g.kind[q];
        const uint32_t dr = kd == 2 ? 2 : 1, dc = kd == 1 ? 2 : 1;
        mv_r |= dr << (8 * q);
        mv_t |= (dr + dc) << (8 * q);
    }
    int32_t k = r >> 6, rho = r & 63, tau = c + rho;
    fetch(k, tau >> 4);
    fetch(k - 1, (c + 63) >> 4 < nP ? (c + 63) >> 4 : nP - 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const int32_t max_iters = R + W;
    int32_t m = 0;
    bool done = false, broke = false;
    // the code of cell (64 k + rho, tau - rho)
    auto code_at = [&](uint32_t buf, int32_t rh, int32_t ta) {
        uint32_t word;
        asm volatile("ld.shared.b32 %0, [%1];"
                     : "=r"(word)
                     : "r"(buf + (uint32_t)rh * 4 + ((uint32_t)ta & (16 * (kWalkPeriods - 1))) * 16));
        return (word >> ((ta & 15) * 2)) & 3u;
    };
    // (every lane walks and stores the same)
    while (m < max_iters) {
        const uint32_t buf = win0 + (k & 1) * kBuf;
        const int32_t row0 = 64 * k + gro;
        const int32_t cc = tau - rho;
        int32_t quick = (rho < cc ? rho : cc) >> 1;
        if (m + quick > max_iters) quick = 0;
        if (quick > 1 && rho + 64 * k > sr && cc > sc) {
            // the start lies on row 0 or column 0, out of reach of these steps
            const int32_t rho0 = rho, tau0 = tau;
            int32_t moved = 0;
#pragma unroll 4
            for (int32_t q = 0; q < quick; ++q) {
                out[m + q] = make_int2(rho + row0, tau - rho + gco);
                const uint32_t code = code_at(buf, rho, tau);
                moved = (int32_t)__byte_perm(mv_r, 0u, 0x4440u | code);
                rho -= moved;
                tau -= (int32_t)__byte_perm(mv_t, 0u, 0x4440u | code);
            }
            if (moved > 0) {
                m += quick;
            } else {  // some step was none: again, one by one
                rho = rho0;
                tau = tau0;
                quick = 0;
            }
        } else {
            quick = 0;
        }
        if (quick > 0) continue;
        // one step with every test
        const int32_t row = 64 * k + rho;
        out[m] = make_int2(row + gro, cc + gco);
        ++m;
        if (row == sr && cc == sc) { done = true; break; }
        const uint32_t code = code_at(buf, rho, tau);
        const int32_t dr = (int32_t)__byte_perm(mv_r, 0u, 0x4440u | code);
        const int32_t dt = (int32_t)__byte_perm(mv_t, 0u, 0x4440u | code);
        // no step won, or it leaves the tile
        if (dr == 0 || cc < dt - dr || row < dr) { broke = true; break; }
        rho -= dr;
        tau -= dt;
        if (rho < 0) {  // into the strip above, its periods are on their way
            --k;
            rho += 64;
            tau += 64;
            const int32_t top = (tau - rho + 63) >> 4;
            asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncwarp();  // and every lane is done with the strip below's
            fetch(k - 1, top < nP ? top : nP - 1);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!done && (broke || 64 * k + rho != sr || tau - rho != sc)) {
        out[m] = make_int2(sr + gro, sc + gco);
        ++m;
    }
    if (lane == 0) b.seg_len[e] = m;
}

// Concatenate the walks with consecutive-duplicate removal and reverse to
// start-first order.  Inside one walk consecutive points always differ, so
// only the first point of a walk can repeat the last point of the previous.
// Every CTA derives the offsets of all walks; CTA x of the grid copies the
// walks x, x + gridDim.x, ...
__global__ void __launch_bounds__(256) k_concat(const S2Pair one, const S2Pair* __restrict__ tab) {
    __shared__ int64_t off[kChainMax + 1];
    __shared__ int32_t drop[kChainMax];
    const S2Pair& p = tab ? tab[blockIdx.y] : one;
    const S2Buf b = p.b;
    const int n = *b.chain_len;
    const int2* pts = reinterpret_cast<const int2*>(b.seg_pts);
    for (int e = threadIdx.x; e < n; e += blockDim.x) {
        int d = 0;
        if (e > 0) {
            const int2 prev = pts[(int64_t)(e - 1) * b.seg_cap + b.seg_len[e - 1] - 1];
            const int2 cur = pts[(int64_t)e * b.seg_cap];
            d = prev.x == cur.x && prev.y == cur.y;
        }
        drop[e] = d;
        off[e] = b.seg_len[e] - d;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int64_t o = 0;
        for (int e = 0; e < n; ++e) {
            const int64_t len = off[e];
            off[e] = o;
            o += len;
        }
        off[n] = o;
        if (blockIdx.x == 0) *b.wp_len = o;
    }
    __syncthreads();
    const int64_t K = off[n];
    longlong2* wp = reinterpret_cast<longlong2*>(b.wp);
    for (int e = blockIdx.x; e < n; e += gridDim.x) {
        const int2* src = pts + (int64_t)e * b.seg_cap;
        const int32_t d = drop[e];
        const int64_t cnt = off[e + 1] - off[e];
        for (int64_t m = threadIdx.x; m < cnt; m += blockDim.x) {
            const int2 v = src[m + d];
            wp[K - 1 - (off[e] + m)] = make_longlong2(v.x, v.y);
        }
    }
}

// Host-side launch sequence ------------------------------------------------
cudaError_t launch_fill(double* p, int64_t n, double v, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    int64_t blocks = (n + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    k_fill_f64<<<(int)blocks, 256, 0, st>>>(p, n, v);
    count_launches(1);
    return cudaGetLastError();
}

// (64 pairs: one clear and one gather, 0.11 ms, against 128 launches over four
// streams, 0.41 ms of kernels.)
cudaError_t launch_stage2_edges(const S2Pair& one, const S2Pair* tab, int npairs,
                                cudaStream_t st) {
    const int64_t nslots = (int64_t)one.g.n1 * one.g.n2 * 2 * one.g.L;
    const unsigned blocks = (unsigned)std::min<int64_t>((nslots + 255) / 256, 8192);
    if (!tab) {
        const cudaError_t e = cudaMemsetAsync(one.b.valid, 0, (size_t)nslots, st);
        if (e != cudaSuccess) return e;
    }
    return for_pairs(npairs, [&](int q, int n) {
        const S2Pair* t = tab ? tab + q : nullptr;
        if (t) {
            k_clear_valid<<<dim3((blocks + 15) / 16, (unsigned)n), 256, 0, st>>>(t);
            count_launches(1);
        }
        k_edges<<<dim3(blocks, (unsigned)n), 256, 0, st>>>(one, t);
        count_launches(1);
        return cudaGetLastError();
    });
}

// A kernel on clusters of cn CTAs, one cluster per alignment.
template <typename K, typename... More>
static cudaError_t launch_clusters(K kern, int cn, int npairs, int threads, cudaStream_t st,
                                   const S2Pair& one, const S2Pair* tab, More... more) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cn;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return for_pairs(npairs, [&](int q, int n) {
        cfg.gridDim = dim3((unsigned)cn, (unsigned)n);
        count_launches(1);
        return cudaLaunchKernelEx(&cfg, kern, one, tab ? tab + q : nullptr, more...);
    });
}

// CTAs per alignment for `work` items: one per 2048, 1 to 8, a power of two.
static int cluster_for(int64_t work) {
    int cn = 1;
    while (cn < 8 && (int64_t)cn * 2048 < work) cn *= 2;
    return cn;
}

cudaError_t launch_stage2_prop(const S2Pair& one, const S2Pair* tab, int npairs, cudaStream_t st) {
    const Geo& g = one.g;
    const int64_t nslots = (int64_t)g.n1 * g.n2 * 2 * g.L;
    const int64_t blocks = std::min<int64_t>((nslots + 255) / 256, 8192);
    const cudaError_t e = for_pairs(npairs, [&](int q, int n) {
        k_valid_lists<<<dim3((unsigned)blocks, (unsigned)n), 256, 0, st>>>(one,
                                                                          tab ? tab + q : nullptr);
        count_launches(1);
        return cudaGetLastError();
    });
    if (e != cudaSuccess) return e;
    // about one slot in eight is valid; a cluster takes 512 to 4096 at once
    return launch_clusters(k_propagate, cluster_for((int64_t)std::min(g.n1, g.n2) * g.L),
                           npairs, kPropThreads, st, one, tab);
}

cudaError_t launch_sync_scan(const S2Pair& one, const S2Pair* tab, int npairs, double beta,
                             cudaStream_t st) {
    // a CTA per two segments, up to 8
    const int64_t segs = 2 * std::max((one.g.N + one.g.L - 1) / one.g.L,
                                      (one.g.M + one.g.L - 1) / one.g.L);
    return launch_clusters(k_scan, cluster_for(segs * 1024), npairs, kScanThreads, st, one, tab,
                           beta);
}

cudaError_t launch_stitch_chain(const Geo& g, const S2Buf& b, cudaStream_t st, int from_best,
                                int64_t si, int64_t sj, int64_t se, int64_t sx) {
    k_stitch_chain<<<1, 32, 0, st>>>(g, b, ChainStart{si, sj, se, sx, from_best});
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_stitch(const S2Pair& one, const S2Pair* tab, int npairs, cudaStream_t st,
                          int from_best, int64_t si, int64_t sj, int64_t se, int64_t sx) {
    // a path crosses at most n1 + n2 - 1 tiles, and the stitch follows 101
    const int most = std::min(kChainMax, one.g.n1 + one.g.n2);
    return for_pairs(npairs, [&](int q, int n) {
        const dim3 grid((unsigned)most, (unsigned)n);
        const S2Pair* t = tab ? tab + q : nullptr;
        k_walk<<<grid, 32, 0, st>>>(one, t, ChainStart{si, sj, se, sx, from_best});
        k_concat<<<grid, 256, 0, st>>>(one, t);
        count_launches(2);
        return cudaGetLastError();
    });
}

}  // namespace pfx
