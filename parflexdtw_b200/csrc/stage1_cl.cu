// Stage 1 for alignments with few tiles: one tile on a cluster of CTAs.
//
// The CW warps of each of the cluster's n CTAs share the strip pipeline of
// one tile (stage1_v3.cu): virtual warp v = CW * rank + warp takes strips v,
// v + n CW, ...  A tile then takes (nS - 1) lag + span steps with lag =
// max(80, span / (n CW)), and few warps per SM make a step short: 16 warps on
// an SM are issue-bound, 4 take the latency of the step's dependent FP64 chain
// (cluster_step_ns).  So a tile is spread over as many SMs as the tile count
// leaves (stage1_plan).
//
// Strip k + 1 reads strip k's last rows from a ring in its own CTA's shared
// memory.  Where producer and consumer sit in different CTAs (the last warp of
// a CTA and the first of the next) the producer also writes that ring, in the
// consumer's CTA (distributed shared memory, posted stores off the dependency
// chain), and the pairwise progress words are published at cluster scope, into
// the reader's CTA too, so every poll is local.
// Rank 0 claims the tiles; three cluster barriers per tile (claim, set-up,
// end), which every thread of every CTA reaches on every path: waits are
// bounded and a warp that gives up goes on to the tile's end barrier.
#include <cooperative_groups.h>

#include <string.h>

#include <algorithm>
#include <utility>
#include <vector>

#include "stage1_dp.cuh"
#include "tile_shape.cuh"

namespace pfx {

__device__ __forceinline__ int ld_acquire_cluster(const int* p) {
    int v;
    asm volatile("ld.acquire.cluster.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_cluster(int* p, int v) {
    asm volatile("st.release.cluster.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ bool wait_progress_cl(const int* p, int target,
                                                 const volatile int* abort) {
    for (int it = 0; it < kSpinLimit; ++it) {
        if (ld_acquire_cluster(p) >= target) return true;
        if (*abort) return false;
        __nanosleep(32);
    }
    return false;
}

// FULL: every cell's D takes its cost's place in the slab and its internal start
// encoding (Wave) goes to Psk in the same layout (the single-tile call).
template <int CW, bool STD, typename T, int QD, bool FULL>
__global__ void __launch_bounds__(CW * 32, 1)
    k_stage1_cl(const TileDesc* __restrict__ descs, const int ntiles, int* __restrict__ head,
                const Geo g, int32_t* __restrict__ status, const int RB, const int queue_at,
                int2* __restrict__ Psk) {
    using V2 = typename Vec2<T>::type;
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), nc = (int)cl.num_blocks();
    const int NWT = CW * nc;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Rings<T> rg = ring_layout<T>(smem_raw, CW, RB);  // this CTA's rings
    // progress words: [w] warp w's; [CW] the previous CTA's last warp's (this
    // CTA's warp 0 waits on it); [CW + 1] the next CTA's warp 0's (this CTA's
    // last warp waits on it) -- written by those CTAs, polled here
    int* prog = reinterpret_cast<int*>(rg.xP + CW * kXch);
    __shared__ TileDesc td;
    __shared__ Sched2 s_sc;
    __shared__ int s_item, s_abort, s_ttot;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int vw = rank * CW + warp;
    // a warp's producer is the warp before it: its ring is region warp - 1 of
    // this CTA, or for warp 0 region CW - 1, which the previous CTA's last warp
    // writes; this CTA's last warp writes region CW - 1 of the next CTA
    const int prevw = (warp + CW - 1) % CW, nextw = (warp + 1) % CW;
    const bool prev_remote = warp == 0, next_remote = warp == CW - 1;
    const int next_rank = (rank + 1) % nc, prev_rank = (rank + nc - 1) % nc;
    V2* wD = cl.map_shared_rank(rg.D, next_rank);
    int2* wP = cl.map_shared_rank(rg.P, next_rank);
    int* my_word = prog + warp;
    int* peer_word = warp == 0 ? cl.map_shared_rank(prog, prev_rank) + CW + 1
                               : cl.map_shared_rank(prog, next_rank) + CW;
    if (threadIdx.x == 0) s_abort = 0;
    cl.sync();  // every CTA runs before any access to another's shared memory
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            bool stop = false;
            for (int r = 0; r < nc; ++r) stop = stop || *cl.map_shared_rank(&s_abort, r);
            const int it = stop ? ntiles : atomicAdd(head, 1);
            for (int r = 0; r < nc; ++r) *cl.map_shared_rank(&s_item, r) = it;
        }
        cl.sync();  // the claimed tile reaches every CTA
        if (s_item >= ntiles) return;  // every CTA, nothing remote after the barrier
        if (threadIdx.x == 0) {
            td = descs[s_item];
            s_sc = make_sched2(td.R, td.W, NWT);
            s_ttot = (s_sc.nS - 1) * s_sc.lag + s_sc.span;
        }
        if (threadIdx.x < CW + 2) prog[threadIdx.x] = 0;
        __syncthreads();
        if (rank == 0) {
            // edge rows past the tile's extent stay +inf / 0 (the DP writes the rest)
            double* eD = td.eD;
            int32_t* eP = td.eP;
            for (int i = threadIdx.x; i < 2 * td.L; i += CW * 32) {
                eD[i] = CUDART_INF;
                eP[i] = 0;
            }
        }
        cl.sync();  // progress words reset in every CTA, edges filled
        const int32_t R = td.R, W = td.W;
        const Sched2& sc = s_sc;
        const int lag = sc.lag;
        const int Ttot = s_ttot;
        const V2* Ct = reinterpret_cast<const V2*>(td.Csk);

        Wave<T, QD> st;
        zero_wave(st);
        if constexpr (QD > 0)
            st.q.at = (uint32_t)__cvta_generic_to_shared(smem_raw) + queue_at +
                      warp * (QD * cost_step_bytes<T>()) + lane * (int)sizeof(V2);
        int rs = ring_start(lag, RB), ws = ring_start(64, RB);
        for (int Tb = 0; Tb < Ttot; Tb += kBlk) {
            int k = -1;
            uint2 bw = make_uint2(0u, 0u);
            if (Tb >= vw * lag) {
                const int j = (Tb - vw * lag) / (NWT * lag);
                const int kk = vw + j * NWT;
                if (kk < sc.nS && Tb < kk * lag + sc.span) k = kk;
            }
            if (k >= 0) {
                int failed = 0;
                if (lane == 0) {
                    // producer (strip k-1) has written every ring slot this block reads
                    if (k >= 1 &&
                        !(prev_remote ? wait_progress_cl(prog + CW, Tb - lag + 80, &s_abort)
                                      : wait_progress(prog + prevw, Tb - lag + 80, &s_abort)))
                        failed = 1;
                    // consumer (strip k+1) has read every slot this block overwrites
                    if (!failed && k + 1 < sc.nS &&
                        !(next_remote
                              ? wait_progress_cl(prog + CW + 1, Tb + lag - RB - 45, &s_abort)
                              : wait_progress(prog + nextw, Tb + lag - RB - 45, &s_abort)))
                        failed = 1;
                    if (failed) {
                        if (status) atomicExch(status, kStatusWaitTimeout);
                        s_abort = 1;
                    }
                }
                if (__shfl_sync(0xffffffffu, failed, 0)) break;  // to the tile's end barrier
                Block<T> b;
                b.tau0 = Tb - k * lag;
                b.Cs = Ct + (int64_t)k * sc.span * 32 + lane;
                b.span = sc.span;
                b.k = k;
                b.R = R;
                b.W = W;
                b.lane = lane;
                b.nP = sc.nP;
                const bool feeds = k + 1 < sc.nS;
                lane_addresses(b, rg, warp, feeds && !next_remote ? warp * RB + ws : -1,
                               k >= 1 ? prevw * RB + rs : -1);
                b.pD = feeds && next_remote ? wD + warp * RB + ws : nullptr;
                b.pP = feeds && next_remote ? wP + warp * RB + ws : nullptr;
                if (lane == 0 && b.tau0 + 2 * kBlk <= sc.span)
                    prefetch_next_block(Ct + (int64_t)k * sc.span * 32, b.tau0 + kBlk);
                if (b.tau0 == 0) queue_start<QD, T>(st.q, b.Cs);
                if (FULL) {
                    const int64_t at = ((int64_t)k * sc.span + b.tau0) * 32 + lane;
                    b.oD = const_cast<V2*>(Ct) + at;
                    b.oP = Psk + at;
                }
                run_block<STD, true, FULL, T, QD>(g, st, b, td, sc.nS, &bw);
            }
            rs = ring_next(rs, RB);
            ws = ring_next(ws, RB);
            __syncwarp();
            // publish first: the backpointer store below is nobody's dependency
            if (lane == 31) {
                if (prev_remote || next_remote) {
                    // also into the other CTA's copy, so that its reader polls locally
                    st_release_cluster(my_word, Tb + kBlk);
                    st_release_cluster(peer_word, Tb + kBlk);
                } else {
                    cuda::atomic_ref<int, cuda::thread_scope_block> a(*my_word);
                    a.store(Tb + kBlk, cuda::memory_order_release);
                }
            }
            if (k >= 0 && 64 * k + 2 * lane < R) {
                uint2* Bt = reinterpret_cast<uint2*>(td.Bw);
                Bt[((int64_t)k * sc.nP + ((Tb - k * lag) >> 4)) * 32 + lane] = bw;
            }
        }
        cl.sync();  // every warp of every CTA is done with this tile's rings
    }
}

// Launch configuration of nclusters clusters of cn CTAs (kernel, attributes
// and shared memory set); false when it does not fit.
struct ClConfig {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr[1];
    S1Mem mem;
};

template <int CW, bool STD, typename T, int QD, bool FULL>
static cudaError_t cl_config(const S1Mem& m, int cn, int nclusters, ClConfig* c) {
    auto kern = k_stage1_cl<CW, STD, T, QD, FULL>;
    const cudaError_t e = cudaFuncSetAttribute(
        kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)m.bytes);
    if (e != cudaSuccess) return e;
    c->mem = m;
    c->cfg = {};
    c->attr[0].id = cudaLaunchAttributeClusterDimension;
    c->attr[0].val.clusterDim.x = (unsigned)cn;
    c->attr[0].val.clusterDim.y = 1;
    c->attr[0].val.clusterDim.z = 1;
    c->cfg.blockDim = dim3(CW * 32);
    c->cfg.dynamicSmemBytes = m.bytes;
    c->cfg.attrs = c->attr;
    c->cfg.numAttrs = 1;
    c->cfg.gridDim = dim3((unsigned)(cn * nclusters));
    return cudaSuccess;
}

// max != null: only the number of clusters that can run at once; fit > 0: that
// number, where the caller has it.
template <int CW, bool STD, typename T, int QD, bool FULL>
static cudaError_t cl_launch(const S1Mem& m, int cn, const TileDesc* descs, int ntiles, int* head,
                             const Geo& g, int32_t* status, cudaStream_t st, int* max,
                             int2* Psk = nullptr, int fit = 0) {
    auto kern = k_stage1_cl<CW, STD, T, QD, FULL>;
    ClConfig c;
    cudaError_t e = cl_config<CW, STD, T, QD, FULL>(m, cn, 1, &c);
    if (e != cudaSuccess) return e;
    if (fit <= 0) e = cudaOccupancyMaxActiveClusters(&fit, kern, &c.cfg);
    if (e != cudaSuccess) return e;
    if (max) {
        *max = fit;
        return cudaSuccess;
    }
    if (fit < 1) return cudaErrorInvalidConfiguration;
    const int n = std::min(ntiles, fit);
    if (n <= 0) return cudaSuccess;
    c.cfg.gridDim = dim3((unsigned)(cn * n));
    c.cfg.stream = st;
    e = cudaLaunchKernelEx(&c.cfg, kern, descs, ntiles, head, g, status, m.rb, m.queue_at, Psk);
    count_launches(1);
    return e;
}

template <typename T>
static cudaError_t cl_dispatch(int cn, int cw, const TileDesc* descs, int ntiles, int* head,
                               const Geo& g, int32_t* status, cudaStream_t st, int* max) {
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    const Sched2 s = make_sched2(g.L, g.L, cn * cw);
    const S1Mem m = stage1_mem(s.lag, cw, cta_budget(16), (int)sizeof(T), cw < 16 ? 4 : 0);
    if (m.rb == 0) return cudaErrorInvalidValue;
#define PFX_CL(CW, QD)                                                                        \
    return std_steps                                                                          \
               ? cl_launch<CW, true, T, QD, false>(m, cn, descs, ntiles, head, g, status, st, \
                                                  max)                                      \
               : cl_launch<CW, false, T, QD, false>(m, cn, descs, ntiles, head, g, status,    \
                                                   st, max)
    if (cw == 16) PFX_CL(16, 0);
    if (m.qd == 0) return cudaErrorInvalidValue;
    if (cw == 12) PFX_CL(12, 4);
    if (cw == 8) PFX_CL(8, 4);
    if (cw == 4) PFX_CL(4, 4);
#undef PFX_CL
    return cudaErrorInvalidValue;
}

cudaError_t launch_stage1_cluster(int cn, int cw, const TileDesc* descs, int ntiles, int* head,
                                  const Geo& g, int32_t* status, bool fp32, cudaStream_t st) {
    return fp32 ? cl_dispatch<float>(cn, cw, descs, ntiles, head, g, status, st, nullptr)
                : cl_dispatch<double>(cn, cw, descs, ntiles, head, g, status, st, nullptr);
}

// The tile's full outputs from the skewed ones: 32 rows x 64 columns per CTA
// through shared memory (D and P in the cost's layout, codes from the packed
// backpointers); P = 0 on row 0 and column 0, code 3 is -1. Where the DP's
// waits ran out D is NaN, not a number that could pass for a result.
__global__ void __launch_bounds__(256)
    k_unskew(const double* __restrict__ Dsk, const int* __restrict__ Psk,
             const uint32_t* __restrict__ Bw, const int32_t* __restrict__ status, int R, int W,
             double* __restrict__ D, int32_t* __restrict__ P, int8_t* __restrict__ B) {
    __shared__ double sd[32][65];
    __shared__ int sp[32][65];
    const bool failed = *status != 0;
    const int span = ceil_div32(W + kStripRows - 1, kBlk) * kBlk;
    const int k = blockIdx.y >> 1, h = (blockIdx.y & 1) * 32, c0 = blockIdx.x * 64;
    for (int q = threadIdx.x; q < 95 * 32; q += 256) {
        const int rho = q & 31, tau = c0 + h + (q >> 5), c = tau - h - rho - c0;
        if (c < 0 || c >= 64 || tau >= span) continue;
        const int64_t at = ((int64_t)k * span + tau) * 64 + h + rho;
        sd[rho][c] = Dsk[at];
        sp[rho][c] = Psk[at];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < 32 * 64; q += 256) {
        const int x = q & 63, rho = h + (q >> 6), r = 64 * k + rho, c = c0 + x;
        if (r >= R || c >= W) continue;
        const int tau = c + rho;
        const uint32_t word = __ldg(Bw + bp_word_index2(W, r, tau));
        const int code = (int)((word >> ((tau & 15) * 2)) & 3u);
        const int64_t at = (int64_t)r * W + c;
        D[at] = failed ? __longlong_as_double(0x7ff8000000000000ll) : sd[rho - h][x];
        P[at] = r == 0 || c == 0 ? 0 : sp[rho - h][x];
        B[at] = (int8_t)(code == 3 ? -1 : code);
    }
}

// A queue of one tile.
__global__ void k_one_tile(const TileDesc d, TileDesc* __restrict__ out, int* __restrict__ head) {
    *out = d;
    head[0] = 0;
    head[1] = 0;  // status
}

// One tile with all of D, P and B as row-major outputs: cost into the skewed
// layout, the DP on one cluster with D written over the cost, and back.
// Bound by the DP's chain of steps. Against one CTA that writes each cell's
// values itself (stage1_f64.cu), 1500 x 1801: 9.4 ms of kernels -> 1.32 (DP
// 1.26, the passes before and after it 0.06); its caller has the sizes.
cudaError_t launch_tile_full(const double* C, const Geo& g, double* D, int32_t* P, int8_t* B,
                             cudaStream_t st, bool* done) {
    *done = false;
    const int R = (int)g.N, W = (int)g.M;
    const int nS = ceil_div32(R, kStripRows);
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    // as many warps as strips, four per SM up to 8 SMs, then eight
    const int cw = nS > 48 ? 8 : 4;
    S1Mem m;
    TileDesc* dd = nullptr;
    int* head = nullptr;
    int2* Psk = nullptr;
    int fit = 0;
    // max: only how many clusters of cn CTAs can be resident
    const auto cluster = [&](int cn, int* max) -> cudaError_t {
#define PFX_FULL(CW)                                                                          \
    (std_steps ? cl_launch<CW, true, double, 4, true>(m, cn, dd, 1, head, g, head + 1, st,    \
                                                      max, Psk, fit)                          \
               : cl_launch<CW, false, double, 4, true>(m, cn, dd, 1, head, g, head + 1, st,   \
                                                       max, Psk, fit))
        return cw == 8 ? PFX_FULL(8) : PFX_FULL(4);
#undef PFX_FULL
    };
    const int cn = full_tile_ctas(nS, cw, [&](int n) {
        m = stage1_mem(make_sched2(g.L, g.L, n * cw).lag, cw, cta_budget(16), 8, 4);
        fit = 0;
        if (m.rb == 0 || m.qd == 0) return false;
        if (cluster(n, &fit) == cudaSuccess) return fit > 0;
        cudaGetLastError();  // a shape that cannot be resident is no error of the caller's
        return false;
    });
    if (cn == 0) return cudaSuccess;
    // scratch: slab and P (large: from the library's own pool, taking 60 MB from
    // the default one costs about 1.5 ms), and backpointers, edges, descriptor,
    // queue head and status
    auto up = [](size_t b) { return (b + 255) & ~(size_t)255; };
    // (the tile's own strips and periods, not those of an L x L tile)
    const size_t words = (size_t)nS * ceil_div32(W + kStripRows - 1, kBlk) * kStripRows;
    const size_t slab = up(words * kBlk * 8);
    const size_t bw = up(words * 4), ed = up((size_t)2 * g.L * 12);
    char *big = nullptr, *tmp = nullptr;
    if (scratch_alloc((void**)&big, slab + slab / 2, st) != cudaSuccess ||
        cudaMallocAsync((void**)&tmp, bw + ed + 512, st) != cudaSuccess) {
        cudaGetLastError();  // no room: the caller's other way needs less
        if (big) cudaFreeAsync(big, st);
        return cudaSuccess;
    }
    double* Dsk = reinterpret_cast<double*>(big);
    Psk = reinterpret_cast<int2*>(big + slab);
    TileDesc d;
    memset(&d, 0, sizeof(d));
    d.Csk = Dsk;
    d.Bw = reinterpret_cast<uint32_t*>(tmp);
    d.eD = reinterpret_cast<double*>(tmp + bw);
    d.eP = reinterpret_cast<int32_t*>(d.eD + 2 * g.L);
    d.R = R;
    d.W = W;
    d.L = g.L;
    char* misc = tmp + bw + ed;
    dd = reinterpret_cast<TileDesc*>(misc + 256);
    head = reinterpret_cast<int*>(misc);
    k_one_tile<<<1, 1, 0, st>>>(d, dd, head);
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_relayout_skew(C, g.ldc, g, Dsk, 0, st);
    if (e == cudaSuccess) e = cluster(cn, nullptr);
    if (e == cudaSuccess) {
        k_unskew<<<dim3((unsigned)ceil_div32(W, 64), (unsigned)(2 * nS)), 256, 0, st>>>(
            Dsk, reinterpret_cast<const int*>(Psk), d.Bw, head + 1, R, W, D, P, B);
        count_launches(1);
        e = cudaGetLastError();
    }
    const cudaError_t eb = cudaFreeAsync(big, st), ef = cudaFreeAsync(tmp, st);
    *done = true;
    return e != cudaSuccess ? e : (eb != cudaSuccess ? eb : ef);
}

int stage1_cluster_max(int cn, int cw, const Geo& g, bool fp32) {
    int fit = 0;
    const cudaError_t e =
        fp32 ? cl_dispatch<float>(cn, cw, nullptr, 0, nullptr, g, nullptr, nullptr, &fit)
             : cl_dispatch<double>(cn, cw, nullptr, 0, nullptr, g, nullptr, nullptr, &fit);
    if (e != cudaSuccess) {
        cudaGetLastError();  // a shape that does not fit is no error of the caller's
        return 0;
    }
    return fit;
}

// The cluster kernel's time per step with `warps` warps on an SM (tiles of 4000
// x 4000 on 2, 4 and 8 CTAs of 4 warps: 217, 217 and 215 ns; 2 and 4 of 8: 260
// and 248; 80 of them on 2 of 12: 294; on 2 of 16: 409).
static double cluster_step_ns(int warps) {
    return warps <= 4 ? 217.0 : warps <= 8 ? 255.0 : warps <= 12 ? 300.0 : 405.0;
}

// Modelled as in stage1_queue_ns.  Measured, stage 1: 16 tiles of 4000 x 4000
// 2.71 ms on 8 CTAs (6.33 on one CTA of 16 warps, 5.17 on two), 80 tiles (17
// of them smaller) 4.29 ms with 2 CTAs of 12 warps each (6.41 on one of 16; 4.88
// on two of 16), 9 tiles of 1999 x 1999 1.14 ms on 8 CTAs (1.48 on 4 of 4 warps,
// 2.01 on one of 16), 12 tiles of 1000 x 1000 0.60 ms (0.68 on one of 8).
S1Plan stage1_plan(const Geo& g, int ntiles, bool fp32, int num_sms) {
    const int64_t whole = whole_tiles(g, g.L);
    S1Plan best{0, stage1_queue_warps(whole, g.L, num_sms), 0};
    if (ntiles > num_sms) return best;
    double t = stage1_queue_ns(whole, g.L, best.cw, num_sms);
    // the tiles' steps on one CTA of 16 warps, in queue order (largest first)
    std::vector<std::pair<int64_t, double>> alone;
    for (int i = 0; i < ntiles; ++i) {
        int64_t r0, c0;
        int32_t R, W;
        tile_rect(g, i / g.n2, i % g.n2, &r0, &c0, &R, &W);
        alone.push_back({-(int64_t)R * W, stage1_model_steps(R, W, 16)});
    }
    std::stable_sort(alone.begin(), alone.end(),
                     [](const std::pair<int64_t, double>& x, const std::pair<int64_t, double>& y) {
                         return x.first < y.first;
                     });
    for (int cw = 4; cw <= 16; cw += 4)
        for (int cn = 2; cn <= 8; cn *= 2) {
            // (more warps than strips would idle)
            if (cn * cw >= 2 * ceil_div32(g.L, kStripRows)) continue;
            const double steps = stage1_model_steps(g.L, g.L, cn * cw);
            if (steps * cluster_step_ns(cw) >= t) continue;
            // every tile on a cluster at once; or for pairs of SMs the largest,
            // and each other tile on an SM of its own
            const int fit = stage1_cluster_max(cn, cw, g, fp32);
            int big = std::min(ntiles, fit);
            if (big < ntiles) big = cn == 2 ? std::min(big, num_sms - ntiles) : 0;
            if (big <= 0) continue;
            double e = steps * cluster_step_ns(cw * ceil_div32(cn * big, num_sms));
            for (int i = big; i < ntiles; ++i)
                e = std::max(e, alone[i].second * stage1_step_ns(16, 1));
            if (e >= t) continue;
            best = S1Plan{cn, cw, big};
            t = e;
        }
    return best;
}

}  // namespace pfx
