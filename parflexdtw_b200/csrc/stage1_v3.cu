// Stage 1 (plan path): FlexDTW on every tile, two rows per lane, cost
// read from the tile-skewed layout, warps synchronised pairwise.
//
// Recurrence and tie-breaking: FlexDTW.py:326-370 (see stage1_f64.cu).
//
// Mapping.  A strip is 64 tile rows; lane i owns rows 64k+2i (A) and
// 64k+2i+1 (B) and at local step tau computes A = (64k+2i, tau-2i) and
// B = (64k+2i+1, tau-2i-1): row rho = r mod 64 sits at column tau - rho, and
// r + c = 64k + tau is the same for every cell of a warp-step.  The
// predecessors of A are lane i-1's B two steps ago ((1,1)) and three steps ago
// ((1,2): what this lane had one step earlier) and lane i-1's A three steps
// ago ((2,1)); those of B are this lane's own A two and three steps ago and
// again lane i-1's B three steps ago.  Lanes pass (D, P) of both rows through
// shared memory, one entry per lane; lane 31's entry is a slot of its strip's
// ring and lane 0 reads the previous strip's ring (see Rings).  mdist =
// (r + c) - |P| is formed in FP64 (exact: both integers).
//
// Strips start `lag` (>= 80) steps apart.  Inside a tile warps do not use CTA
// barriers: each publishes the global step it has completed (release store by
// lane 31, the ring writer) and, before a block, waits (acquire, bounded)
// until its producer has written everything the block reads and its consumer
// has read every slot the block overwrites.  A wait that runs out sets the
// status word and the CTA's abort flag; every warp then leaves the tile at its
// next wait and the CTA stops claiming tiles.
//
// Work queue.  The kernel is persistent: each CTA claims tile descriptors
// (cost slab, output addresses, shape) from a device queue with one atomic
// per tile, so the tiles of one alignment or of a whole batch of alignments
// of uneven sizes run in one launch.  Queues are ordered largest tile first.
// A CTA barrier separates consecutive tiles of a CTA (progress words are
// reset there).
//
// Selection.  Every cell takes a branch-free, division-free comparison of the
// three candidates (cross products with a 2^-46 relative margin, see
// decide_quot); cells too close to call and non-finite values go to the exact
// routine, which falls back to IEEE division.  Blocks inside the tile run a
// loop that holds nothing else; see run_block.  The cost queue runs two steps
// ahead, or four with fewer than 16 warps per tile (CostQueue).
//
// Measured (592 tiles of 2000 x 2000, B200): 6.28 ms with 8 warps per tile
// (377 Gcells/s), 6.53 with 4, against 9.47 ms (4 warps) with shuffles,
// per-lane ring selects, one loop for all blocks and the exact routine inside
// it.  An inner fast step costs 52 thread instructions per cell (79 before), 19
// of them on the half-rate FP64 pipe; a careful one 112.
#include <algorithm>

#include "stage1_dp.cuh"

namespace pfx {

// ---------------------------------------------------------------------------
// In-kernel cost (CostGen).  The CTA that claimed a tile first writes the
// tile's tile-skewed FP64 cost into its own slot, then runs the DP on it, so
// a batch needs one slot per resident CTA instead of a slab per tile, and
// CTAs in their cost phase (FP64-pipe bound) share the SMs with CTAs in their
// DP phase (issue and latency bound).  Mapping and summation order are those
// of k_cost_skew (layout.cu): units of two strips x (NW * 32) steps; the
// unit's column features are staged in shared memory split by column parity
// and the two strips' row features as one (A, B) pair per lane; each warp
// computes 32 steps of both strips in passes of 8 steps, in which 9 column
// vectors serve 32 cells of a lane.  Cells outside the tile are 0, as in the
// slabs.  The staging reuses the rings' shared memory, which holds nothing
// between tiles.
constexpr int kGenCV = 4;

__host__ __device__ constexpr int gen_window(int nw) { return nw * 32 + 66; }
__host__ __device__ inline size_t gen_smem_bytes(int nw, int d) {
    return (size_t)d * (gen_window(nw) + 128) * sizeof(double);
}

template <int NW, int DMAX>
__device__ __forceinline__ void gen_tile_cost(const double* __restrict__ fa, int lda,
                                           const double* __restrict__ fb, int ldb, int R, int W,
                                           int d, double* __restrict__ slab) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int U = NW * 32;
    constexpr int CX = gen_window(NW), CH = CX / 2;
    double* sB = reinterpret_cast<double*>(smem_raw);  // [d][2][CH]
    double* sA = sB + d * CX;                          // [d][2 strips][64 rows]
    const double2* sA2 = reinterpret_cast<const double2*>(sA);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int span = ceil_div32(W + kStripRows - 1, kBlk) * kBlk;
    const int nS = ceil_div32(R, kStripRows);
    const int nchunk = ceil_div32(span, U);
    for (int kk = 0; 2 * kk < nS; ++kk) {
        const bool two = 2 * kk + 1 < nS;
        const int rA0 = 128 * kk + 2 * lane, rB0 = rA0 + 1, rA1 = rA0 + 64, rB1 = rA1 + 1;
        double2* out0 = reinterpret_cast<double2*>(slab) + (int64_t)(2 * kk) * span * 32 + lane;
        double2* out1 = out0 + (int64_t)span * 32;
        for (int ch = 0; ch < nchunk; ++ch) {
            const int ts = ch * U;
            __syncthreads();  // every warp is done with the previous unit's features
            // the unit's features, as asynchronous copies all in flight at once
            // (zero-filled outside the tile)
            for (int q = threadIdx.x; q < d * CX; q += NW * 32) {
                const int f = q / CX, x = q - f * CX;
                const int c = ts - 64 + x;
                const bool in = c >= 0 && c < W;
                cp_async8(sB + (f * 2 + (x & 1)) * CH + (x >> 1),
                          in ? fb + (int64_t)f * ldb + c : fb, in);
            }
            if (ch == 0)
                for (int q = threadIdx.x; q < d * 128; q += NW * 32) {
                    const int f = q >> 7, r = 128 * kk + (q & 127);
                    cp_async8(sA + q, r < R ? fa + (int64_t)f * lda + r : fa, r < R);
                }
            cp_async_wait_all();
            __syncthreads();
#pragma unroll 1
            for (int blk = 0; blk < 32 / kGenCV; ++blk) {
                const int t0 = ts + 32 * warp + kGenCV * blk;  // warp-uniform
                if (t0 >= span) break;
                // b[j] holds window column x = xA0 - 1 + j, xA0 = t0 - ts + 64 - 2 lane
                const int h0 = ((t0 - ts + 64) >> 1) - lane;
                double accA0[kGenCV], accB0[kGenCV], accA1[kGenCV], accB1[kGenCV];
#pragma unroll
                for (int f = 0; f < DMAX; ++f) {
                    if (f >= d) break;
                    const double* se = sB + (f * 2) * CH;  // even x
                    const double* so = se + CH;             // odd x
                    double b[kGenCV + 1];
#pragma unroll
                    for (int j = 0; j <= kGenCV; ++j)
                        b[j] = (j & 1) ? se[h0 + (j >> 1)] : so[h0 - 1 + (j >> 1)];
                    const double2 a0 = sA2[(f * 2) * 32 + lane], a1 = sA2[(f * 2 + 1) * 32 + lane];
#pragma unroll
                    for (int v = 0; v < kGenCV; ++v) {
                        const double pA0 = __dmul_rn(a0.x, b[v + 1]);
                        const double pB0 = __dmul_rn(a0.y, b[v]);
                        const double pA1 = __dmul_rn(a1.x, b[v + 1]);
                        const double pB1 = __dmul_rn(a1.y, b[v]);
                        accA0[v] = f == 0 ? pA0 : __dadd_rn(accA0[v], pA0);
                        accB0[v] = f == 0 ? pB0 : __dadd_rn(accB0[v], pB0);
                        accA1[v] = f == 0 ? pA1 : __dadd_rn(accA1[v], pA1);
                        accB1[v] = f == 0 ? pB1 : __dadd_rn(accB1[v], pB1);
                    }
                }
#pragma unroll
                for (int v = 0; v < kGenCV; ++v) {
                    const int tau = t0 + v;
                    if (tau < span) {
                        const int cA = tau - 2 * lane, cB = cA - 1;
                        const bool inA = cA >= 0 && cA < W, inB = cB >= 0 && cB < W;
                        out0[(int64_t)tau * 32] =
                            make_double2((rA0 < R && inA) ? __dsub_rn(1.0, accA0[v]) : 0.0,
                                         (rB0 < R && inB) ? __dsub_rn(1.0, accB0[v]) : 0.0);
                        if (two)
                            out1[(int64_t)tau * 32] =
                                make_double2((rA1 < R && inA) ? __dsub_rn(1.0, accA1[v]) : 0.0,
                                             (rB1 < R && inB) ? __dsub_rn(1.0, accB1[v]) : 0.0);
                    }
                }
            }
        }
    }
    __syncthreads();  // the slot holds the whole tile before any warp's DP reads it
}

template <int NW, bool STD, typename T, bool GEN, int QD>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
    k_stage1_v3(const TileDesc* __restrict__ descs, const int ntiles_max,
                const int* __restrict__ ntiles_dev, int* __restrict__ head, const Geo g,
                int32_t* __restrict__ status, const int RB, const int queue_at, const CostGen gen) {
    using V2 = typename Vec2<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Rings<T> rg = ring_layout<T>(smem_raw, NW, RB);
    int* prog = reinterpret_cast<int*>(rg.xP + NW * kXch);
    __shared__ TileDesc td;
    __shared__ Sched2 s_sc;  // schedule of the current tile (read from smem, not held in registers)
    __shared__ int s_item, s_abort, s_ttot;
    // (the warp index through a shuffle, so that what derives from it is known
    // to be uniform in the warp and stays out of the vector registers)
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int prevw = (warp + NW - 1) % NW, nextw = (warp + 1) % NW;
    const int ntiles = ntiles_dev ? min(*ntiles_dev, ntiles_max) : ntiles_max;
    if (GEN && (int)blockIdx.x >= gen.nslots) return;  // no cost slot (the launch prevents it)
    if (threadIdx.x == 0) s_abort = 0;
    cuda::atomic_ref<int, cuda::thread_scope_block> my_prog(prog[warp]);
    for (;;) {
        if (threadIdx.x == 0) {
            const int it = atomicAdd(head, 1);
            s_item = it;
            if (it < ntiles) {
                td = descs[it];
                s_sc = make_sched2(td.R, td.W, NW);
                s_ttot = (s_sc.nS - 1) * s_sc.lag + s_sc.span;
            }
        }
        if (!GEN && threadIdx.x < NW) prog[threadIdx.x] = 0;
        __syncthreads();
        if (s_item >= ntiles || s_abort) return;
        if constexpr (GEN) {
            // the tile's cost into this CTA's slot (through the rings' shared
            // memory, so the progress words are reset afterwards)
            double* slot = gen.slots + (int64_t)blockIdx.x * gen.stride;
            if (gen.d <= 12)
                gen_tile_cost<NW, 12>(td.fa, td.lda, td.fb, td.ldb, td.R, td.W, gen.d, slot);
            else
                gen_tile_cost<NW, kGenMaxD>(td.fa, td.lda, td.fb, td.ldb, td.R, td.W, gen.d,
                                            slot);
            if (threadIdx.x < NW) prog[threadIdx.x] = 0;
        }
        {
            // edge rows past the tile's extent stay +inf / 0 (the DP writes the rest)
            double* eD = td.eD;
            int32_t* eP = td.eP;
            for (int i = threadIdx.x; i < 2 * td.L; i += NW * 32) {
                eD[i] = CUDART_INF;
                eP[i] = 0;
            }
        }
        __syncthreads();
        const int32_t R = td.R, W = td.W;
        const Sched2& sc = s_sc;
        const int lag = sc.lag;
        const int Ttot = s_ttot;
        const V2* Ct =
            GEN ? reinterpret_cast<const V2*>(gen.slots + (int64_t)blockIdx.x * gen.stride)
                : reinterpret_cast<const V2*>(td.Csk);

        Wave<T, QD> st;
        zero_wave(st);
        if constexpr (QD > 0)
            st.q.at = (uint32_t)__cvta_generic_to_shared(smem_raw) + queue_at +
                      warp * (QD * cost_step_bytes<T>()) + lane * (int)sizeof(V2);
        int rs = ring_start(lag, RB), ws = ring_start(64, RB);
        for (int Tb = 0; Tb < Ttot; Tb += kBlk) {
            int k = -1;
            if (Tb >= warp * lag) {
                const int j = (Tb - warp * lag) / (NW * lag);
                const int kk = warp + j * NW;
                if (kk < sc.nS && Tb < kk * lag + sc.span) k = kk;
            }
            if (k >= 0) {
                int failed = 0;
                if (lane == 0) {
                    // producer (strip k-1) has written every ring slot this block reads
                    if (k >= 1 && !wait_progress(prog + prevw, Tb - lag + 80, &s_abort)) failed = 1;
                    // consumer (strip k+1) has read every slot this block overwrites
                    if (!failed && k + 1 < sc.nS &&
                        !wait_progress(prog + nextw, Tb + lag - RB - 45, &s_abort))
                        failed = 1;
                    if (failed) {
                        if (status) atomicExch(status, kStatusWaitTimeout);
                        s_abort = 1;
                    }
                }
                if (__shfl_sync(0xffffffffu, failed, 0)) break;  // to the tile barrier
                Block<T> b;
                b.tau0 = Tb - k * lag;
                b.span = sc.span;
                b.k = k;
                b.R = R;
                b.W = W;
                b.lane = lane;
                b.nP = sc.nP;
                b.Cs = Ct + (int64_t)k * sc.span * 32 + lane;
                lane_addresses(b, rg, warp, k + 1 < sc.nS ? warp * RB + ws : -1,
                               k >= 1 ? prevw * RB + rs : -1);
                b.pD = nullptr;
                b.pP = nullptr;
                if (lane == 0 && b.tau0 + 2 * kBlk <= sc.span)
                    prefetch_next_block(Ct + (int64_t)k * sc.span * 32, b.tau0 + kBlk);
                if (b.tau0 == 0) queue_start<QD, T>(st.q, b.Cs);
                run_block<STD, false, false, T, QD>(g, st, b, td, sc.nS, nullptr);
            }
            rs = ring_next(rs, RB);
            ws = ring_next(ws, RB);
            __syncwarp();
            if (lane == 31) my_prog.store(Tb + kBlk, cuda::memory_order_release);
        }
        __syncthreads();  // every warp is done with this tile's rings and descriptor
    }
}

// The queue kernel's shared memory for tiles of up to L x L; gen_d > 0: at
// least the in-kernel cost's staging.
static S1Mem queue_mem(int32_t L, int nw, int vbytes, int qd, int gen_d) {
    const Sched2 s = make_sched2(L, L, nw);
    S1Mem m = stage1_mem(s.lag, nw, cta_budget(nw), vbytes, qd);
    if (m.rb && gen_d > 0) {
        const size_t gen = gen_smem_bytes(nw, gen_d);
        m.bytes = m.bytes > gen ? m.bytes : gen;
        if (m.bytes > (size_t)cta_budget(nw)) m.rb = 0;
    }
    return m;
}

// Depth of the shared-memory cost queue asked for by the queue kernel.
static int queue_qd(int nw, bool std_steps, bool gen) { return std_steps && !gen && nw < 16 ? 4 : 0; }

// Modelled time of a tile: pipeline steps times the time of a step.  A strip
// needs the one above it 80 steps ahead, published in blocks of 16; measured,
// lags below 120 steps cost as much as 120 (each block then waits for its
// producer; 164 before the strips' first blocks had a fast loop).
double stage1_model_steps(int32_t R, int32_t W, int nw) {
    const Sched2 s = make_sched2(R, W, nw);
    return (s.nS - 1) * std::max(s.lag, 120) + s.span;
}

// Time of a step (ns) with `ctas` CTAs of nw warps on an SM (tiles of 1000 x
// 1000 to 4000 x 4000).
double stage1_step_ns(int nw, int ctas) {
    if (nw == 4) return 200.0 + 55.0 * (ctas - 1);
    if (nw == 8) return ctas == 1 ? 215.0 : 315.0;
    return 305.0;
}

bool stage1_queue_fits(int32_t L, int nw) { return queue_mem(L, nw, 8, 0, 0).rb > 0; }

double stage1_queue_ns(int64_t ntiles, int32_t L, int nw, int num_sms) {
    const int slots = 16 / nw;
    const int64_t per = (int64_t)num_sms * slots;
    const int64_t full = ntiles / per, rest = ntiles % per;
    const int ctas = (int)((rest + num_sms - 1) / num_sms);
    return stage1_model_steps(L, L, nw) * (full * stage1_step_ns(nw, slots) +
                                           (rest ? stage1_step_ns(nw, ctas) : 0.0));
}

// Warps per tile: the choice of the least modelled time (stage1_queue_ns;
// the FP64 rings are the larger, so they decide what fits).  Fewer warps per
// tile fill the strip pipeline better but take longer per tile, which decides
// where the last wave of tiles leaves SMs idle (ntiles: by their area, as the
// small tiles at a matrix's edges fill in at the end: 576 whole and 24 small
// tiles of 1000 x 1000 1.81 / 2.17 ms with 4 / 8 warps, by their number 8).
// Measured with 4 / 8 / 16 warps: 399 tiles of 2000 x 2000 5.66 / 4.97 / 7.26 ms,
// 143 of them 4.66 / 2.12 / 2.00 ms; 504 tiles of 1000 x 1000 1.77 / 1.94 / 3.8
// ms, 323 of 500 x 500 0.47 / 0.61 / 1.1 ms, 25 of 500 x 500 0.33 / 0.30 ms.
int stage1_queue_warps(int64_t ntiles, int32_t L, int num_sms) {
    int best = 0;
    double t = 0.0;
    for (int nw = 4; nw <= 16; nw *= 2) {
        if (!stage1_queue_fits(L, nw)) continue;
        const double e = stage1_queue_ns(ntiles, L, nw, num_sms);
        if (!best || e < t) {
            best = nw;
            t = e;
        }
    }
    return best;
}

// CTAs of the queue kernel resident at once on this device (its grid size
// for a long queue), or 0 when it does not fit.
template <int NW, bool STD, typename T, bool GEN, int QD>
static int queue_resident(size_t smem) {
    auto kern = k_stage1_v3<NW, STD, T, GEN, QD>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return 0;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NW * 32, smem) !=
        cudaSuccess)
        return 0;
    return sms * (per_sm < 1 ? 1 : per_sm);
}

template <int NW, bool STD, typename T, bool GEN, int QD>
static cudaError_t launch_q_t(const TileDesc* descs, int ntiles, const int* ntiles_dev, int* head,
                              const Geo& g, int32_t* status, cudaStream_t st, const S1Mem& m,
                              const CostGen& gen) {
    const int resident = queue_resident<NW, STD, T, GEN, QD>(m.bytes);
    if (resident <= 0) return cudaErrorInvalidValue;
    // with the in-kernel cost every CTA needs a cost slot of its own
    if (GEN && gen.nslots < std::min(resident, ntiles)) return cudaErrorInvalidValue;
    const int grid = std::min(resident, ntiles);
    if (grid <= 0) return cudaSuccess;
    k_stage1_v3<NW, STD, T, GEN, QD><<<grid, NW * 32, m.bytes, st>>>(
        descs, ntiles, ntiles_dev, head, g, status, m.rb, m.queue_at, gen);
    count_launches(1);
    return cudaGetLastError();
}

template <int NW, typename T, bool GEN>
static cudaError_t launch_q_nw(const TileDesc* descs, int ntiles, const int* nd, int* head,
                               const Geo& g, int32_t* status, cudaStream_t st,
                               const CostGen& gen) {
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    const S1Mem m = queue_mem(g.L, NW, (int)sizeof(T), queue_qd(NW, std_steps, GEN),
                              GEN ? gen.d : 0);
    if (m.rb == 0) return cudaErrorInvalidValue;
    if constexpr (!GEN && NW < 16) {
        if (m.qd)
            return launch_q_t<NW, true, T, GEN, 4>(descs, ntiles, nd, head, g, status, st, m, gen);
    }
    return std_steps
               ? launch_q_t<NW, true, T, GEN, 0>(descs, ntiles, nd, head, g, status, st, m, gen)
               : launch_q_t<NW, false, T, GEN, 0>(descs, ntiles, nd, head, g, status, st, m, gen);
}

template <typename T, bool GEN>
static cudaError_t launch_q_type(const TileDesc* descs, int ntiles, const int* nd, int* head,
                                 const Geo& g, int32_t* status, int nw, cudaStream_t st,
                                 const CostGen& gen) {
    switch (nw) {
        case 4: return launch_q_nw<4, T, GEN>(descs, ntiles, nd, head, g, status, st, gen);
        case 8: return launch_q_nw<8, T, GEN>(descs, ntiles, nd, head, g, status, st, gen);
        default: return launch_q_nw<16, T, GEN>(descs, ntiles, nd, head, g, status, st, gen);
    }
}

cudaError_t launch_stage1_queue(const TileDesc* descs, int ntiles, const int* ntiles_dev,
                                int* head, const Geo& g, int32_t* status, int nw, bool fp32,
                                cudaStream_t st, const CostGen* gen) {
    const CostGen off{nullptr, 0, 0, 0};
    if (gen && gen->d > 0) {
        if (fp32 || gen->d > kGenMaxD || !gen->slots) return cudaErrorInvalidValue;
        return launch_q_type<double, true>(descs, ntiles, ntiles_dev, head, g, status, nw, st,
                                           *gen);
    }
    return fp32 ? launch_q_type<float, false>(descs, ntiles, ntiles_dev, head, g, status, nw, st,
                                              off)
                : launch_q_type<double, false>(descs, ntiles, ntiles_dev, head, g, status, nw,
                                               st, off);
}

template <int NW>
static int gen_slots_t(const Geo& g, int d) {
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    const S1Mem m = queue_mem(g.L, NW, 8, 0, d);
    if (m.rb == 0) return 0;
    return std_steps ? queue_resident<NW, true, double, true, 0>(m.bytes)
                     : queue_resident<NW, false, double, true, 0>(m.bytes);
}

int stage1_gen_slots(const Geo& g, int nw, int d) {
    if (d < 1 || d > kGenMaxD) return 0;
    return nw == 4    ? gen_slots_t<4>(g, d)
           : nw == 8  ? gen_slots_t<8>(g, d)
           : nw == 16 ? gen_slots_t<16>(g, d)
                      : 0;
}

// Order-preserving compaction of a tile queue by a tile mask (one CTA: a
// block-wide prefix count per chunk of 1024 descriptors).
__global__ void __launch_bounds__(1024) k_compact_descs(const TileDesc* __restrict__ in, int n,
                                                        const uint8_t* __restrict__ mask,
                                                        TileDesc* __restrict__ out,
                                                        int* __restrict__ count) {
    __shared__ int warp_sums[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c0 = 0; c0 < n; c0 += 1024) {
        const int i = c0 + (int)threadIdx.x;
        const bool keep = i < n && mask[in[i].tile];
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        const int before = __popc(bal & ((1u << lane) - 1u));
        if (lane == 0) warp_sums[warp] = __popc(bal);
        __syncthreads();
        int off = 0;
        for (int w = 0; w < warp; ++w) off += warp_sums[w];
        if (keep) out[base + off + before] = in[i];
        __syncthreads();
        if (threadIdx.x == 0) {
            int tot = 0;
            for (int w = 0; w < 32; ++w) tot += warp_sums[w];
            base += tot;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) *count = base;
}

__global__ void k_mask_slots(const uint8_t* __restrict__ mask, int n, int32_t* __restrict__ slot) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) slot[t] = mask[t] ? t : -1;
}

cudaError_t launch_mask_slots(const uint8_t* mask, int n, int32_t* slot, cudaStream_t st) {
    k_mask_slots<<<(n + 255) / 256, 256, 0, st>>>(mask, n, slot);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_compact_descs(const TileDesc* in, int n, const uint8_t* mask, TileDesc* out,
                                 int* count, cudaStream_t st) {
    k_compact_descs<<<1, 1024, 0, st>>>(in, n, mask, out, count);
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace pfx
