// Stage 1 (plan path): FlexDTW on every tile, FP64, two rows per lane, cost
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
// ahead.
//
// Measured (592 tiles of 2000 x 2000, 4 warps per tile, B200): 6.91 ms = 343
// Gcells/s, against 9.47 ms = 250 Gcells/s with shuffles, per-lane ring
// selects, one loop for all blocks and the exact routine inside it.  A fast
// step costs 52 thread instructions per cell (79 before), 19 of them on the
// half-rate FP64 pipe; a careful one 112.
#include <algorithm>
#include <cooperative_groups.h>
#include <cuda/atomic>

#include "common.cuh"

#include <math_constants.h>

namespace pfx {

constexpr int kSpinLimit = 1 << 22;

// Pulls the cost of a strip's next block of steps (kBlk steps x 32 lanes,
// contiguous in the skewed slab) into L2 with one bulk prefetch, so that the
// DP's own loads, two steps ahead, hit L2 instead of HBM.  Issued by one lane;
// the range must lie inside the strip (the caller checks).
template <typename V2>
__device__ __forceinline__ void prefetch_next_block(const V2* strip, int tau_next) {
    const V2* p = strip + (int64_t)tau_next * 32;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p),
                 "r"((uint32_t)(kBlk * 32 * sizeof(V2)))
                 : "memory");
}

// IEEE arithmetic of the DP's value type (FP64 plain form, FP32 chosen form),
// rounded to nearest, never contracted.
__device__ __forceinline__ double addr(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float addr(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double mulr(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mulr(float a, float b) { return __fmul_rn(a, b); }
template <typename T> struct Vec2;
template <> struct Vec2<double> { using type = double2; };
template <> struct Vec2<float> { using type = float2; };

// Exact RN(b/nd) < RN(a/md) (nd, md positive integers), per lane, no warp
// collectives.  Division only when the cross products cannot decide.
__device__ __forceinline__ bool qless_exact(double b, double nd, double a, double md) {
    const double U = __dmul_rn(b, md);
    const double V = __dmul_rn(a, nd);
    const double diff = __dadd_rn(V, -U);
    const double mag = __dadd_rn(fabs(U), fabs(V));
    const double tau = __dmul_rn(mag, 0x1p-48);
    if (mag >= 0x1p-950) {
        if (diff > tau) return true;
        if (-diff > tau) return false;
    }
    return __ddiv_rn(b, nd) < __ddiv_rn(a, md);
}

// FP32 form: RN32(b/nd) < RN32(a/md).  The cross products of two FP32 values
// and two integers below 2^24 are exact in FP64, so their difference has the
// sign of the exact comparison: <= 0 decides "not less"; a relative margin of
// 2^-21 (two FP32 roundings are at most 2^-24 each) decides "less"; in
// between the two IEEE divisions decide.
__device__ __forceinline__ bool qless_exact(float b, float nd, float a, float md) {
    const double U = __dmul_rn((double)b, (double)md);
    const double V = __dmul_rn((double)a, (double)nd);
    const double diff = __dadd_rn(V, -U);
    if (diff <= 0.0) return false;
    if (diff > __dmul_rn(__dadd_rn(fabs(U), fabs(V)), 0x1p-21)) return true;
    return __fdiv_rn(b, nd) < __fdiv_rn(a, md);
}

// Exact selection of one cell with r, c >= 1 (generic steps, any position).
// Start encodings are the internal ones (see Wave): a boundary predecessor's
// mdist is r + c, as the reference stores P = 0 there (FlexDTW.py:346-356).
template <bool STD, bool ALLIN, typename T>
__device__ __forceinline__ void select_exact(const Geo& g, T w_last, int r, int c, T rc, T cval,
                                          T x1D, int x1P, T x2D, int x2P, T x3D, int x3P, T& oD,
                                          int& oP, int& code) {
    int bs = -1, bP = 0;
    T bA = 0, bM = 1;
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        if (!STD && s >= g.S) continue;
        const int kd = STD ? s : g.kind[s];
        const bool inb = ALLIN || kd == 0 || (kd == 1 ? c >= 2 : r >= 2);
        if (!inb) continue;
        const T pD = kd == 0 ? x1D : (kd == 1 ? x2D : x3D);
        const int pP = kd == 0 ? x1P : (kd == 1 ? x2P : x3P);
        const bool rim = !ALLIN && (r == (kd == 2 ? 2 : 1) || c == (kd == 1 ? 2 : 1));
        const T a = addr(pD, mulr(cval, (T)g.w[s]));
        const T md = rim ? rc : addr(rc, -fabs((T)pP));
        const bool take = bs < 0 ? a < (T)CUDART_INF : qless_exact(a, md, bA, bM);
        if (take) {
            bs = s;
            bA = a;
            bM = md;
            bP = pP;
        }
    }
    if (bs < 0) {
        // reference: D[-1,-1] (still 0) + C * w[-1], P[-1,-1] (0), B = -1
        oD = addr((T)0, mulr(cval, w_last));
        oP = 0;
        code = 3;
    } else {
        oD = bA;
        code = bs;
        oP = bP;
    }
}

// Division-free decision of "the new candidate's quotient is strictly below
// the incumbent's", RN(a_new / m_new) < RN(a_inc / m_inc) with positive
// integer-valued m, for the FP64 form.  Returns whether the cross products
// decide it (else the caller divides); `win` is the answer when they do.
//   U = RN(a_new * m_inc), d = RN(a_inc * m_new - U) (one FMA) and the
//   threshold t = RN(|U| * 2^-46 + 2^-900) (one FMA).  With V the exact
//   a_inc * m_new, d's error is below 2^-53 |U| + 2^-53 |d| (plus 2^-1074
//   where a value is subnormal).
//   * |V| <= 3 |U|: |d| > t > 2^-46 |U| exceeds that error by a factor of 32,
//     so it fixes the sign of the exact V - a_new m_inc and leaves a relative
//     gap > 2^-49 between the exact quotients: their roundings cannot meet.
//   * |V| > 3 |U|: the exact difference has V's sign and |V| / 2 or more of
//     magnitude, the same conclusion.
//   |d| > t needs max(|U|, |V|) > 2^-901: no quotient is subnormal.  An
//   infinite U makes t infinite and a NaN product makes d NaN: neither
//   decides.  An infinite a_inc against a finite U decides as the reference
//   does (+inf never becomes the incumbent, -inf is never beaten).
__device__ __forceinline__ bool decide_quot(double a_new, double m_new, double a_inc,
                                            double m_inc, bool& win) {
    const double U = __dmul_rn(a_new, m_inc);
    const double d = __fma_rn(a_inc, m_new, -U);
    const double t = __fma_rn(fabs(U), 0x1p-46, 0x1p-900);
    win = d > 0.0;
    return fabs(d) > t;
}
// FP32 form: the cross products of FP32 values and integers below 2^24 are
// exact in FP64 (see the FP32 qless_exact): d <= 0 decides "not below", a
// relative margin of 2^-21 decides "below".  Infinite values never decide.
__device__ __forceinline__ bool decide_quot(float a_new, float m_new, float a_inc, float m_inc,
                                            bool& win) {
    const double U = __dmul_rn((double)a_new, (double)m_inc);
    const double V = __dmul_rn((double)a_inc, (double)m_new);
    const double d = __dadd_rn(V, -U);
    win = d > __dmul_rn(__dadd_rn(fabs(U), fabs(V)), 0x1p-21);
    return (win || d <= 0.0) && fabs(d) < CUDART_INF;
}

// Steps (1,1), (1,2), (2,1) at one cell, mdists given: branch-free selection.
// Returns false when a comparison is too close to call or a value is not
// finite; the caller then recomputes the cell with select_exact.  RIM: in1 /
// in2 say whether the (1,2) / (2,1) predecessor exists (else all do).
template <bool RIM, typename T>
__device__ __forceinline__ bool select_std(T cval, T w0, T w1, T w2, T x1D, int x1P, T m0, T x2D,
                                           int x2P, T m1, bool in1, T x3D, int x3P, T m2, bool in2,
                                           T& oD, int& oP, int& code) {
    const T a0 = addr(x1D, mulr(cval, w0));
    const T a1 = addr(x2D, mulr(cval, w1));
    const T a2 = addr(x3D, mulr(cval, w2));
    bool win1, win2;
    bool ok1 = decide_quot(a1, m1, a0, m0, win1);
    if (RIM) {
        win1 = win1 && in1;
        ok1 = in1 ? ok1 : a0 < (T)CUDART_INF;
    }
    const T bA = win1 ? a1 : a0, bM = win1 ? m1 : m0;
    bool ok2 = decide_quot(a2, m2, bA, bM, win2);
    if (RIM) {
        win2 = win2 && in2;
        ok2 = in2 ? ok2 : bA < (T)CUDART_INF;
    }
    oD = win2 ? a2 : bA;
    oP = win2 ? x3P : (win1 ? x2P : x1P);
    code = win2 ? 2 : (win1 ? 1 : 0);
    return ok1 && ok2;
}

// A warp's wavefront state between steps.  At the start of step tau: A's
// outputs 1..3 steps ago, B's output one step ago, the predecessors of this
// step's A cell -- x1 (1,1), x2 (1,2), x3 (2,1) -- already received, and the
// mdists of A's and B's (1,2) predecessors.  Start encodings are internal: a
// cell on row 0 carries its column, one on column 0 minus its row, so that a
// successor inherits its predecessor's encoding everywhere.
template <typename T>
struct Wave {
    T aD1, aD2, aD3, bD1, x1D, x2D, x3D, m1A, m1B;
    int aP1, aP2, aP3, bP1, x1P, x2P, x3P;
    typename Vec2<T>::type q[2];     // cost queue, step tau in slot tau & 1
};

// Per-warp rings of a strip's last two rows, [NW][RB] slots, RB a multiple
// of kBlk, and per-warp exchange entries, [NW][kXch].  At the start of its
// step T (counted from the tile's start) every lane stores the pair {B one
// step ago, A two steps ago} and loads its neighbour lane i-1's, which the
// next step uses as x1 and x3.  Lanes 0..30 store into their exchange entry;
// lane 31 stores into ring slot (T - 64) mod RB, which then holds rows 64k+63
// and 64k+62 of column j = tau - 64; lane 0 loads ring slot (T' - lag) mod RB
// of the previous strip, its column tau'.  So one address per lane takes the
// place of shuffles, of the ring's own loads and stores and of the selects
// between the two.  Both ring windows of a block start on a multiple of
// kBlk: no address inside a block wraps.  D is one {B, A} vector, the start
// encodings one {B, A} int2.
template <typename T>
struct Rings {
    typename Vec2<T>::type *D, *xD;
    int2 *P, *xP;
};
constexpr int kXch = 34;  // 32 lanes, shifted by one entry in odd steps, and one spare
template <typename T>
__host__ __device__ constexpr int ring_slot_bytes() {
    return (int)(sizeof(typename Vec2<T>::type) + sizeof(int2));
}
// Shared memory of nw warps' rings and exchange entries, and n progress words.
template <typename T>
__host__ __device__ constexpr size_t ring_bytes(int nw, int rb, int n) {
    return (size_t)nw * (rb + kXch) * ring_slot_bytes<T>() + n * sizeof(int);
}
template <typename T>
__device__ __forceinline__ Rings<T> ring_layout(unsigned char* smem, int nw, int rb) {
    using V2 = typename Vec2<T>::type;
    Rings<T> r;
    r.D = reinterpret_cast<V2*>(smem);
    r.xD = r.D + nw * rb;
    r.P = reinterpret_cast<int2*>(r.xD + nw * kXch);
    r.xP = r.P + nw * rb;
    return r;
}
__device__ __forceinline__ void st_pair(uint32_t aD, uint32_t aP, double b, double a, int pb,
                                        int pa) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};\nst.shared.v2.s32 [%3], {%4, %5};" ::"r"(aD),
                 "d"(b), "d"(a), "r"(aP), "r"(pb), "r"(pa)
                 : "memory");
}
__device__ __forceinline__ void st_pair(uint32_t aD, uint32_t aP, float b, float a, int pb,
                                        int pa) {
    asm volatile("st.shared.v2.f32 [%0], {%1, %2};\nst.shared.v2.s32 [%3], {%4, %5};" ::"r"(aD),
                 "f"(b), "f"(a), "r"(aP), "r"(pb), "r"(pa)
                 : "memory");
}
__device__ __forceinline__ void ld_pair(uint32_t aD, uint32_t aP, double& b, double& a, int& pb,
                                        int& pa) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%4];\nld.shared.v2.s32 {%2, %3}, [%5];"
                 : "=d"(b), "=d"(a), "=r"(pb), "=r"(pa)
                 : "r"(aD), "r"(aP)
                 : "memory");
}
__device__ __forceinline__ void ld_pair(uint32_t aD, uint32_t aP, float& b, float& a, int& pb,
                                        int& pa) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%4];\nld.shared.v2.s32 {%2, %3}, [%5];"
                 : "=f"(b), "=f"(a), "=r"(pb), "=r"(pa)
                 : "r"(aD), "r"(aP)
                 : "memory");
}
template <typename T>
__device__ __forceinline__ typename Vec2<T>::type make_v2(T x, T y) {
    typename Vec2<T>::type v;
    v.x = x;
    v.y = y;
    return v;
}

// What a block needs besides the wave state.
template <typename T>
struct Block {
    const typename Vec2<T>::type* Cs;  // the strip's cost, at this lane
    uint32_t w, r;                     // this lane's store and load addresses (P; the
    uint32_t kd;                       // D address is that times 2 (FP32 form: 1), + kd)
    typename Vec2<T>::type* pD;        // PUSH: the ring slot in a cluster peer's
    int2* pP;                          // shared memory, or null
    uint32_t incW, incR;               // and their moves per two steps (ring lanes)
    int span, tau0, k, R, W, lane, nP;
};

// Edge values of a cell on the tile's last row / last column; FP64 for stage
// 2 (exact widening in the FP32 form), P = 0 on row 0 and column 0.
template <typename T>
__device__ __forceinline__ void store_edges(const TileDesc& td, int r, int c, int R, int W, T D,
                                            int P) {
    const int p = (r == 0 || c == 0) ? 0 : P;
    if (r == R - 1) {
        td.eD[c] = (double)D;
        td.eP[c] = p;
    }
    if (c == W - 1) {
        td.eD[td.L + r] = (double)D;
        td.eP[td.L + r] = p;
    }
}

// The step's outputs enter the wave.
template <typename T>
__device__ __forceinline__ void advance(Wave<T>& st, T oAD, int oAP, T oBD, int oBP, T x1n,
                                        int p1n, T x3n, int p3n) {
    st.aD3 = st.aD2; st.aP3 = st.aP2;
    st.aD2 = st.aD1; st.aP2 = st.aP1;
    st.aD1 = oAD;    st.aP1 = oAP;
    st.bD1 = oBD;    st.bP1 = oBP;
    st.x2D = st.x1D; st.x2P = st.x1P;
    st.x1D = x1n;    st.x1P = p1n;
    st.x3D = x3n;    st.x3P = p3n;
}

// Shared address of the D pair that belongs to the P pair at p.
template <typename T>
__device__ __forceinline__ uint32_t d_address(uint32_t p, uint32_t kd) {
    return p * (2 * (uint32_t)sizeof(T) / (uint32_t)sizeof(int2)) + kd;
}

// One step of the fast loop: standard steps, every cell of the strip inside
// the tile with r >= 64, c >= 18 and off its last row and column.  Returns
// false, with the wave unchanged, when some lane's cell needs the exact
// routine.  u: the step's parity.
template <bool PUSH, typename T>
__device__ __forceinline__ bool fast_step(Wave<T>& st, const int u, T rc, T w0, T w1, T w2,
                                          uint32_t w, uint32_t r, uint32_t kd,
                                          typename Vec2<T>::type* pD, int2* pP, int lane,
                                          uint32_t& bitsA, uint32_t& bitsB) {
    constexpr int SD = 2 * (int)sizeof(T), SP = (int)sizeof(int2);
    const typename Vec2<T>::type cc = st.q[u];
    T x1n, x3n;
    int p1n, p3n;
    st_pair(d_address<T>(w, kd) + u * SD, w + u * SP, st.bD1, st.aD2, st.bP1, st.aP2);
    if (PUSH && pD && lane == 31) {
        pD[u] = make_v2<T>(st.bD1, st.aD2);
        pP[u] = make_int2(st.bP1, st.aP2);
    }
    __syncwarp();
    ld_pair(d_address<T>(r, kd) + u * SD, r + u * SP, x1n, x3n, p1n, p3n);
    const T m0A = addr(rc, -fabs((T)st.x1P));
    const T m2A = addr(rc, -fabs((T)st.x3P));
    const T m0B = addr(rc, -fabs((T)st.aP2));
    T oAD, oBD;
    int oAP, oBP, codeA, codeB;
    const bool okA = select_std<false, T>(cc.x, w0, w1, w2, st.x1D, st.x1P, m0A, st.x2D, st.x2P,
                                          st.m1A, true, st.x3D, st.x3P, m2A, true, oAD, oAP,
                                          codeA);
    const bool okB = select_std<false, T>(cc.y, w0, w1, w2, st.aD2, st.aP2, m0B, st.aD3, st.aP3,
                                          st.m1B, true, st.x2D, st.x2P, st.m1A, true, oBD, oBP,
                                          codeB);
    if (!__all_sync(0xffffffffu, okA && okB)) return false;
    bitsA = bitsA * 4 + codeA;  // the first step ends up highest
    bitsB = bitsB * 4 + codeB;
    st.m1A = addr(m0A, (T)1);
    st.m1B = addr(m0B, (T)1);
    advance(st, oAD, oAP, oBD, oBP, x1n, p1n, x3n, p3n);
    return true;
}

// One step of the careful loop (see run_block).  rim: cells on row 0 / column
// 0 or next to them may occur; mask: cells past the last row / column or on
// it.  Outputs of cells outside the tile are arbitrary (nothing inside reads
// them) but for their code, 0.
template <bool STD, bool PUSH, typename T>
__device__ __forceinline__ void careful_step(const Geo& g, Wave<T>& st, const Block<T>& b,
                                             const TileDesc& td, const int u, int t,
                                             const bool rim, const bool mask, T rc,
                                             const typename Vec2<T>::type cc, uint32_t& bitsA,
                                             uint32_t& bitsB) {
    constexpr int SD = 2 * (int)sizeof(T), SP = (int)sizeof(int2);
    const unsigned F = 0xffffffffu;
    const T w0 = (T)g.w[0], w1 = (T)g.w[1], w2 = (T)g.w[2];
    const int lane = b.lane;
    const int rA = 64 * b.k + 2 * lane, rB = rA + 1;
    const int cA = b.tau0 + t - 2 * lane, cB = cA - 1;
    T x1n, x3n;
    int p1n, p3n;
    st_pair(d_address<T>(b.w, b.kd) + u * SD, b.w + u * SP, st.bD1, st.aD2, st.bP1, st.aP2);
    if (PUSH && b.pD && lane == 31) {
        b.pD[u] = make_v2<T>(st.bD1, st.aD2);
        b.pP[u] = make_int2(st.bP1, st.aP2);
    }
    __syncwarp();
    ld_pair(d_address<T>(b.r, b.kd) + u * SD, b.r + u * SP, x1n, x3n, p1n, p3n);
    T m0A = addr(rc, -fabs((T)st.x1P));
    T m2A = addr(rc, -fabs((T)st.x3P));
    T m0B = addr(rc, -fabs((T)st.aP2));
    if (rim) {
        // predecessors on row 0 / column 0 (for (1,2) the sum carried over
        // from the previous step already is r + c)
        if (cA == 1) m0A = rc;
        if (cA == 1 || rA == 2) m2A = rc;
        if (cB == 1 || rB == 1) m0B = rc;
    }
    T oAD, oBD;
    int oAP, oBP, codeA, codeB;
    bool okA = false, okB = false;
    if (STD) {
        okA = select_std<true, T>(cc.x, w0, w1, w2, st.x1D, st.x1P, m0A, st.x2D, st.x2P, st.m1A,
                                  cA >= 2, st.x3D, st.x3P, m2A, true, oAD, oAP, codeA);
        okB = select_std<true, T>(cc.y, w0, w1, w2, st.aD2, st.aP2, m0B, st.aD3, st.aP3, st.m1B,
                                  cB >= 2, st.x2D, st.x2P, st.m1A, rB >= 2, oBD, oBP, codeB);
    }
    const bool actA = rA < b.R && cA >= 0 && cA < b.W;
    const bool actB = rB < b.R && cB >= 0 && cB < b.W;
    const bool rimA = rA == 0 || cA == 0, rimB = cB == 0;
    okA = okA || !actA || rimA;
    okB = okB || !actB || rimB;
    if (__any_sync(F, !(okA && okB))) {
        const T w_last = (T)(g.S == 1 ? g.w[0] : (g.S == 2 ? g.w[1] : g.w[2]));
        if (!okA)
            select_exact<STD, false>(g, w_last, rA, cA, rc, cc.x, st.x1D, st.x1P, st.x2D, st.x2P,
                                     st.x3D, st.x3P, oAD, oAP, codeA);
        if (!okB)
            select_exact<STD, false>(g, w_last, rB, cB, rc, cc.y, st.aD2, st.aP2, st.aD3, st.aP3,
                                     st.x2D, st.x2P, oBD, oBP, codeB);
    }
    if (rim) {
        if (rimA) { oAD = cc.x; oAP = rA == 0 ? cA : -rA; codeA = 0; }
        if (rimB) { oBD = cc.y; oBP = -rB; codeB = 0; }
    }
    if (mask) {
        if (actA) store_edges(td, rA, cA, b.R, b.W, oAD, oAP);
        if (actB) store_edges(td, rB, cB, b.R, b.W, oBD, oBP);
    }
    bitsA = bitsA * 4 + (actA ? codeA : 0);
    bitsB = bitsB * 4 + (actB ? codeB : 0);
    st.m1A = addr(m0A, (T)1);
    st.m1B = addr(m0B, (T)1);
    advance(st, oAD, oAP, oBD, oBP, x1n, p1n, x3n, p3n);
}

// The careful loop: steps t .. 15 of a block.
template <bool STD, bool PUSH, typename T>
__device__ __forceinline__ void careful_steps(const Geo& g, Wave<T>& st, Block<T>& b,
                                              const TileDesc& td, int t, const bool rim,
                                              const bool mask, T rc,
                                              const typename Vec2<T>::type* cp, int ahead,
                                              uint32_t& bitsA, uint32_t& bitsB) {
    using V2 = typename Vec2<T>::type;
    // the cost queue in step order
    V2 q0 = st.q[0], q1 = st.q[1];
    if (t & 1) {
        const V2 s = q0;
        q0 = q1;
        q1 = s;
        cp += 32;
    }
#pragma unroll 1
    for (; t < kBlk; ++t) {
        const V2 cc = q0;
        q0 = q1;
        if (t < ahead) q1 = __ldcs(cp);
        cp += 32;
        careful_step<STD, PUSH, T>(g, st, b, td, t & 1, t, rim, mask, rc, cc, bitsA, bitsB);
        rc = addr(rc, (T)1);
        if (t & 1) {
            b.w += b.incW;
            b.r += b.incR;
            if (PUSH && b.pD) {
                b.pD += 2;
                b.pP += 2;
            }
        }
    }
    st.q[0] = q0;  // kBlk is even: the next block's step 0
    st.q[1] = q1;
}

// One block of 16 steps of a strip, in two loops.
//
// The fast loop (standard steps, neither `rim` nor `mask`: every cell of the
// block inside the tile with r >= 64, c >= 18 and off its last row and column)
// has no bounds tests, no divisions and one branch per step, out of the loop
// when some cell is too close to call.  The careful loop does the rest: the
// remaining steps of such a block, and whole blocks of strip 0 or of the first
// five of a strip (`rim`), or that reach the tile's last row or column or past
// them (`mask`).  There cells on row 0 / column 0, predecessors on them (mdist
// r + c) or missing are handled by selects around the same selection, and
// undecided cells -- with other step sets than the standard one, all cells --
// take the exact routine.
//
// What bounds it: warp instructions issued, then the FP64 pipe (half rate), so
// the step is written for few of both.  mdist of a predecessor that the
// previous step also used is that step's mdist + 1 (r + c grows by one per
// step) and B's (2,1) predecessor is A's (1,2) one, so a step converts three
// start encodings; lanes exchange their rows through shared memory (see
// Rings).  The fast loop is unrolled two steps deep only and holds no rare
// code: its size decides how well it is fetched.
template <bool STD, bool PUSH, typename T>
__device__ __forceinline__ void run_block(const Geo& g, Wave<T>& st, Block<T>& b,
                                          const TileDesc& td, const bool rim, const bool mask,
                                          uint2* bw) {
    using V2 = typename Vec2<T>::type;
    const T w0 = (T)g.w[0], w1 = (T)g.w[1], w2 = (T)g.w[2];
    const int lane = b.lane;
    uint32_t bitsA = 0, bitsB = 0;
    T rc = (T)(64 * b.k + b.tau0);
    const V2* cp = b.Cs + (int64_t)(b.tau0 + 2) * 32;  // the cost two steps ahead
    const int ahead = b.span - 2 - b.tau0;
    int t = 0;
    if (STD && !rim && !mask) {
        bool good = true;
#pragma unroll 1
        for (; t < kBlk; t += 2) {
            good = fast_step<PUSH, T>(st, 0, rc, w0, w1, w2, b.w, b.r, b.kd, b.pD, b.pP, lane,
                                      bitsA, bitsB);
            if (!good) break;
            st.q[0] = __ldcs(cp);
            rc = addr(rc, (T)1);
            good = fast_step<PUSH, T>(st, 1, rc, w0, w1, w2, b.w, b.r, b.kd, b.pD, b.pP, lane,
                                      bitsA, bitsB);
            if (!good) {
                ++t;
                break;
            }
            st.q[1] = __ldcs(cp + 32);
            rc = addr(rc, (T)1);
            cp += 64;
            b.w += b.incW;
            b.r += b.incR;
            if (PUSH && b.pD) {
                b.pD += 2;
                b.pP += 2;
            }
        }
    }
    if (t < kBlk)
        careful_steps<STD, PUSH, T>(g, st, b, td, t, rim, mask, rc, cp, ahead, bitsA, bitsB);
    // step t's code belongs in bits 2t, 2t+1: reverse the sixteen pairs
    bitsA = __brev(bitsA);
    bitsB = __brev(bitsB);
    bitsA = ((bitsA >> 1) & 0x55555555u) | ((bitsA & 0x55555555u) << 1);
    bitsB = ((bitsB >> 1) & 0x55555555u) | ((bitsB & 0x55555555u) << 1);
    if (bw) {
        *bw = make_uint2(bitsA, bitsB);
    } else if (64 * b.k + 2 * lane < b.R) {
        uint2* Bt = reinterpret_cast<uint2*>(td.Bw);
        Bt[((int64_t)b.k * b.nP + (b.tau0 >> 4)) * 32 + lane] = make_uint2(bitsA, bitsB);
    }
}

template <typename T>
__device__ __forceinline__ void zero_wave(Wave<T>& st) {
    st.aD1 = st.aD2 = st.aD3 = st.bD1 = st.x1D = st.x2D = st.x3D = st.m1A = st.m1B = 0;
    st.aP1 = st.aP2 = st.aP3 = st.bP1 = st.x1P = st.x2P = st.x3P = 0;
#pragma unroll
    for (int q = 0; q < 2; ++q) st.q[q].x = st.q[q].y = 0;
}

// Ring slots at which a block at step Tb starts to read (off = lag) or write
// (off = 64); Tb = 0 here, stepped by kBlk with the blocks.
__device__ __forceinline__ int ring_start(int off, int RB) { return (RB - off % RB) % RB; }
__device__ __forceinline__ int ring_next(int s, int RB) { return s + kBlk == RB ? 0 : s + kBlk; }

// Lane addresses of a block: exchange entries, but lane 31 stores into the
// ring slot `wslot` (< 0: nobody reads the strip, its entry instead; then a
// ring another strip still reads is not overwritten) and lane 0 loads slot
// `rslot` (< 0: strip 0, which has no producer).
template <typename T>
__device__ __forceinline__ void lane_addresses(Block<T>& b, const Rings<T>& rg, int warp,
                                               int wslot, int rslot) {
    const bool w = b.lane == 31 && wslot >= 0, r = b.lane == 0 && rslot >= 0;
    const int x = warp * kXch + b.lane;
    const int y = b.lane == 0 ? x : x - 1;
    b.w = (uint32_t)__cvta_generic_to_shared(w ? rg.P + wslot : rg.xP + x);
    b.r = (uint32_t)__cvta_generic_to_shared(r ? rg.P + rslot : rg.xP + y);
    b.kd = (uint32_t)__cvta_generic_to_shared(rg.D) -
           d_address<T>((uint32_t)__cvta_generic_to_shared(rg.P), 0u);
    b.incW = w ? 2 * (int)sizeof(int2) : 0;
    b.incR = r ? 2 * (int)sizeof(int2) : 0;
}

// Bounded wait until progress word *p reaches target; gives up early when
// another warp of the CTA has already given up (*abort set).
__device__ __forceinline__ bool wait_progress(int* p, int target, const volatile int* abort) {
    cuda::atomic_ref<int, cuda::thread_scope_block> a(*p);
    for (int it = 0; it < kSpinLimit; ++it) {
        if (a.load(cuda::memory_order_acquire) >= target) return true;
        if (*abort) return false;
        __nanosleep(32);
    }
    return false;
}

// Ring length: as many slots (a multiple of kBlk) as fit the shared-memory
// limit, at most lag + 128 (enough slack that the pairwise waits rarely
// block).  0: lag is too large for the memory; the largest accepted one is
// 29 above the largest power of two of slots that fits (so the tile lengths
// a caller may ask for do not depend on the rounding here), which leaves at
// least the lag - 16 slots the waits need.  `vbytes` is the size of a DP
// value (8 for FP64, 4 for FP32).
__host__ __device__ inline int ring_len(int lag, int nw, int smem_limit, int vbytes) {
    const int per = nw * (2 * vbytes + (int)sizeof(int2));
    int pow2 = 16;
    while ((pow2 * 2) * per + nw * (int)sizeof(int) <= smem_limit) pow2 *= 2;
    if (lag - 29 > pow2) return 0;
    const int fit = ((smem_limit - (nw + 2) * (int)sizeof(int)) / per - kXch) / kBlk * kBlk;
    return lag + 128 < fit ? lag + 128 : fit;
}

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

template <int NW, bool STD, typename T, bool GEN = false>
__global__ void __launch_bounds__(NW * 32, 16 / NW)
    k_stage1_v3(const TileDesc* __restrict__ descs, const int ntiles_max,
                const int* __restrict__ ntiles_dev, int* __restrict__ head, const Geo g,
                int32_t* __restrict__ status, const int RB, const CostGen gen) {
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

        Wave<T> st;
        zero_wave(st);
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
                if (b.tau0 == 0) {
                    st.q[0] = __ldcs(b.Cs);
                    st.q[1] = __ldcs(b.Cs + 32);
                }
                // the block reaches the last row or column, or past them
                const bool mask = k > sc.nS - 2 || b.tau0 + 17 > W;
                run_block<STD, false, T>(g, st, b, td, k == 0 || b.tau0 < 80, mask, nullptr);
            }
            rs = ring_next(rs, RB);
            ws = ring_next(ws, RB);
            __syncwarp();
            if (lane == 31) my_prog.store(Tb + kBlk, cuda::memory_order_release);
        }
        __syncthreads();  // every warp is done with this tile's rings and descriptor
    }
}

// ---------------------------------------------------------------------------
// One tile on a cluster of two CTAs (16 warps each): 32 warps share the strip
// pipeline of a tile, so a tile takes about (nS - 1 + 32) / 32 strip times
// instead of (nS - 1 + 16) / 16.  For alignments with fewer tiles than SMs.
// Virtual warp v = 16 * rank + warp takes strips v, v + 32, ...; strip k + 1
// reads strip k's last rows from a ring in its own CTA's shared memory.
// Where producer and consumer sit in different CTAs (v = 15 -> 16 or
// 31 -> 0) the producer writes that ring into the consumer's CTA
// (distributed shared memory, posted stores off the dependency chain), and
// the pairwise progress words are read and written at cluster scope.
// Rank 0 claims the tiles; three cluster barriers per tile (claim, set-up,
// end), which every thread of both CTAs reaches on every path: waits are
// bounded and a warp that gives up goes on to the tile's end barrier.
constexpr int kClW = 16;   // warps per CTA
constexpr int kClN = 2;    // CTAs per cluster

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

template <bool STD, typename T>
__global__ void __launch_bounds__(kClW * 32, 1)
    k_stage1_cl(const TileDesc* __restrict__ descs, const int ntiles, int* __restrict__ head,
                const Geo g, int32_t* __restrict__ status, const int RB) {
    using V2 = typename Vec2<T>::type;
    constexpr int NWT = kClW * kClN;
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const Rings<T> rg = ring_layout<T>(smem_raw, kClW, RB);  // this CTA's rings
    // progress words: [w] warp w's; [kClW] the other CTA's last warp's (this
    // CTA's warp 0 waits on it); [kClW + 1] the other CTA's warp 0's (this
    // CTA's last warp waits on it) -- written by the other CTA, polled here
    int* prog = reinterpret_cast<int*>(rg.xP + kClW * kXch);
    __shared__ TileDesc td;
    __shared__ Sched2 s_sc;
    __shared__ int s_item, s_abort, s_ttot;
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    const int vw = rank * kClW + warp;
    const int pv = (vw + NWT - 1) % NWT, nv = (vw + 1) % NWT;
    // the producer's rings (generic address, this CTA's or the peer's)
    // a warp writes its ring into its consumer's CTA (posted stores, off the
    // dependency chain) and reads its producer's ring from its own CTA: ring
    // region w of a CTA is written by warp w of the CTA that feeds it (its own
    // warp w, or for w = kClW - 1 the other CTA's last warp)
    V2* wD = cl.map_shared_rank(rg.D, nv / kClW);
    int2* wP = cl.map_shared_rank(rg.P, nv / kClW);
    // cluster scope only where the neighbour is in the other CTA
    const bool prev_remote = pv / kClW != rank, next_remote = nv / kClW != rank;
    const bool read_remotely = warp == 0 || warp == kClW - 1;  // my progress word
    int* rprog = cl.map_shared_rank(prog, 1 - rank);  // the other CTA's words
    if (threadIdx.x == 0) s_abort = 0;
    cl.sync();  // both CTAs run before any access to the other's shared memory
    for (;;) {
        if (rank == 0 && threadIdx.x == 0) {
            const int* peer_abort = cl.map_shared_rank(&s_abort, 1);
            const int it = (s_abort || *peer_abort) ? ntiles : atomicAdd(head, 1);
            s_item = it;
            *cl.map_shared_rank(&s_item, 1) = it;
        }
        cl.sync();  // the claimed tile reaches both CTAs
        if (s_item >= ntiles) return;  // both CTAs, nothing remote after the barrier
        if (threadIdx.x == 0) {
            td = descs[s_item];
            s_sc = make_sched2(td.R, td.W, NWT);
            s_ttot = (s_sc.nS - 1) * s_sc.lag + s_sc.span;
        }
        if (threadIdx.x < kClW + 2) prog[threadIdx.x] = 0;
        __syncthreads();
        if (rank == 0) {
            // edge rows past the tile's extent stay +inf / 0 (the DP writes the rest)
            double* eD = td.eD;
            int32_t* eP = td.eP;
            for (int i = threadIdx.x; i < 2 * td.L; i += kClW * 32) {
                eD[i] = CUDART_INF;
                eP[i] = 0;
            }
        }
        cl.sync();  // progress words reset and edges filled in both CTAs
        const int32_t R = td.R, W = td.W;
        const Sched2& sc = s_sc;
        const int lag = sc.lag;
        const int Ttot = s_ttot;
        const V2* Ct = reinterpret_cast<const V2*>(td.Csk);

        Wave<T> st;
        zero_wave(st);
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
                        !(prev_remote
                              ? wait_progress_cl(prog + kClW, Tb - lag + 80, &s_abort)
                              : wait_progress(prog + pv % kClW, Tb - lag + 80, &s_abort)))
                        failed = 1;
                    // consumer (strip k+1) has read every slot this block overwrites
                    if (!failed && k + 1 < sc.nS &&
                        !(next_remote
                              ? wait_progress_cl(prog + kClW + 1, Tb + lag - RB - 45, &s_abort)
                              : wait_progress(prog + nv % kClW, Tb + lag - RB - 45, &s_abort)))
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
                               k >= 1 ? (pv % kClW) * RB + rs : -1);
                b.pD = feeds && next_remote ? wD + warp * RB + ws : nullptr;
                b.pP = feeds && next_remote ? wP + warp * RB + ws : nullptr;
                if (lane == 0 && b.tau0 + 2 * kBlk <= sc.span)
                    prefetch_next_block(Ct + (int64_t)k * sc.span * 32, b.tau0 + kBlk);
                if (b.tau0 == 0) {
                    st.q[0] = __ldcs(b.Cs);
                    st.q[1] = __ldcs(b.Cs + 32);
                }
                // the block reaches the last row or column, or past them
                const bool mask = k > sc.nS - 2 || b.tau0 + 17 > W;
                run_block<STD, true, T>(g, st, b, td, k == 0 || b.tau0 < 80, mask, &bw);
            }
            rs = ring_next(rs, RB);
            ws = ring_next(ws, RB);
            __syncwarp();
            // publish first: the backpointer store below is nobody's dependency
            if (lane == 31) {
                if (read_remotely) {
                    // also into the other CTA's copy, so that its reader polls locally
                    st_release_cluster(prog + warp, Tb + kBlk);
                    st_release_cluster(rprog + (warp == 0 ? kClW + 1 : kClW), Tb + kBlk);
                } else {
                    cuda::atomic_ref<int, cuda::thread_scope_block> a(prog[warp]);
                    a.store(Tb + kBlk, cuda::memory_order_release);
                }
            }
            if (k >= 0 && 64 * k + 2 * lane < R) {
                uint2* Bt = reinterpret_cast<uint2*>(td.Bw);
                Bt[((int64_t)k * sc.nP + ((Tb - k * lag) >> 4)) * 32 + lane] = bw;
            }
        }
        cl.sync();  // every warp of both CTAs is done with this tile's rings
    }
}

static int smem_optin() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

static int smem_per_sm() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    return v;
}

// Shared memory budget per CTA when 16/NW CTAs share an SM.
static int cta_budget(int nw) {
    const int per_cta = smem_per_sm() / (16 / nw) - 2048;  // static smem and reserve
    const int optin = smem_optin();
    return per_cta < optin ? per_cta : optin;
}

static size_t smem_bytes(int32_t L, int nw, int smem_limit, int vbytes) {
    const Sched2 s = make_sched2(L, L, nw);
    const int rb = ring_len(s.lag, nw, smem_limit, vbytes);
    if (rb == 0) return (size_t)1 << 30;  // does not fit
    return vbytes == 8 ? ring_bytes<double>(nw, rb, nw) : ring_bytes<float>(nw, rb, nw);
}

int stage1_queue_warps(int ntiles, int32_t L, int num_sms) {
    // fewer warps per tile fill the strip pipeline better (utilisation ~
    // strips / (strips - 1 + warps)) but need several tiles per SM; the
    // FP64 rings are the larger, so they decide what fits
    if ((int64_t)ntiles >= 4LL * num_sms && smem_bytes(L, 4, cta_budget(4), 8) < (1u << 30))
        return 4;
    if ((int64_t)ntiles >= 2LL * num_sms && smem_bytes(L, 8, cta_budget(8), 8) < (1u << 30))
        return 8;
    return smem_bytes(L, 16, cta_budget(16), 8) < (1u << 30) ? 16 : 0;
}

// Dynamic shared memory of the queue kernel: the rings, or the in-kernel
// cost's staging (gen_d > 0) where that is larger.
static size_t queue_smem(int32_t L, int nw, int vbytes, int gen_d) {
    const size_t ring = smem_bytes(L, nw, cta_budget(nw), vbytes);
    const size_t gen = gen_d > 0 ? gen_smem_bytes(nw, gen_d) : 0;
    return ring > gen ? ring : gen;
}

// CTAs of the queue kernel resident at once on this device (its grid size
// for a long queue), or 0 when it does not fit.
template <int NW, bool STD, typename T, bool GEN>
static int queue_resident(const Geo& g, int gen_d, size_t* smem_out) {
    const size_t smem = queue_smem(g.L, NW, (int)sizeof(T), gen_d);
    if (smem >= ((size_t)1 << 30) || smem > (size_t)cta_budget(NW)) return 0;
    auto kern = k_stage1_v3<NW, STD, T, GEN>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return 0;
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NW * 32, smem) !=
        cudaSuccess)
        return 0;
    if (smem_out) *smem_out = smem;
    return sms * (per_sm < 1 ? 1 : per_sm);
}

template <int NW, bool STD, typename T, bool GEN>
static cudaError_t launch_q_t(const TileDesc* descs, int ntiles, const int* ntiles_dev, int* head,
                              const Geo& g, int32_t* status, cudaStream_t st,
                              const CostGen& gen) {
    const int limit = cta_budget(NW);
    const Sched2 s = make_sched2(g.L, g.L, NW);
    const int rb = ring_len(s.lag, NW, limit, (int)sizeof(T));
    if (rb == 0) return cudaErrorInvalidValue;
    size_t smem = 0;
    const int resident = queue_resident<NW, STD, T, GEN>(g, GEN ? gen.d : 0, &smem);
    if (resident <= 0) return cudaErrorInvalidValue;
    // with the in-kernel cost every CTA needs a cost slot of its own
    if (GEN && gen.nslots < std::min(resident, ntiles)) return cudaErrorInvalidValue;
    const int grid = std::min(resident, ntiles);
    if (grid <= 0) return cudaSuccess;
    k_stage1_v3<NW, STD, T, GEN>
        <<<grid, NW * 32, smem, st>>>(descs, ntiles, ntiles_dev, head, g, status, rb, gen);
    count_launches(1);
    return cudaGetLastError();
}

template <bool STD, typename T>
static cudaError_t launch_cl_t(const TileDesc* descs, int ntiles, int* head, const Geo& g,
                               int32_t* status, cudaStream_t st) {
    const int limit = cta_budget(kClW);
    const Sched2 s = make_sched2(g.L, g.L, kClW * kClN);
    const int rb = ring_len(s.lag, kClW, limit, (int)sizeof(T));
    if (rb == 0) return cudaErrorInvalidValue;
    const size_t smem = ring_bytes<T>(kClW, rb, kClW + 2);
    auto kern = k_stage1_cl<STD, T>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClN;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(kClW * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(kClN * (unsigned)ntiles);
    int maxc = 0;
    e = cudaOccupancyMaxActiveClusters(&maxc, kern, &cfg);
    if (e != cudaSuccess) return e;
    if (maxc < 1) return cudaErrorInvalidConfiguration;
    const int nc = ntiles < maxc ? ntiles : maxc;
    if (nc <= 0) return cudaSuccess;
    cfg.gridDim = dim3(kClN * (unsigned)nc);
    e = cudaLaunchKernelEx(&cfg, kern, descs, ntiles, head, g, status, rb);
    count_launches(1);
    return e;
}

template <bool STD, typename T>
static int cl_max_t(const Geo& g) {
    const int limit = cta_budget(kClW);
    const Sched2 s = make_sched2(g.L, g.L, kClW * kClN);
    const int rb = ring_len(s.lag, kClW, limit, (int)sizeof(T));
    if (rb == 0) return 0;
    const size_t smem = ring_bytes<T>(kClW, rb, kClW + 2);
    auto kern = k_stage1_cl<STD, T>;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClN;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(kClW * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(kClN);
    int maxc = 0;
    if (cudaOccupancyMaxActiveClusters(&maxc, kern, &cfg) != cudaSuccess) return 0;
    return maxc;
}

int stage1_cluster_max(const Geo& g, bool fp32) {
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    if (fp32) return std_steps ? cl_max_t<true, float>(g) : cl_max_t<false, float>(g);
    return std_steps ? cl_max_t<true, double>(g) : cl_max_t<false, double>(g);
}

cudaError_t launch_stage1_cluster(const TileDesc* descs, int ntiles, int* head, const Geo& g,
                                  int32_t* status, bool fp32, cudaStream_t st) {
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    if (fp32)
        return std_steps ? launch_cl_t<true, float>(descs, ntiles, head, g, status, st)
                         : launch_cl_t<false, float>(descs, ntiles, head, g, status, st);
    return std_steps ? launch_cl_t<true, double>(descs, ntiles, head, g, status, st)
                     : launch_cl_t<false, double>(descs, ntiles, head, g, status, st);
}

template <typename T, bool GEN>
static cudaError_t launch_q_type(const TileDesc* descs, int ntiles, const int* nd, int* head,
                                 const Geo& g, int32_t* status, int nw, cudaStream_t st,
                                 const CostGen& gen) {
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    switch (nw) {
        case 4:
            return std_steps
                       ? launch_q_t<4, true, T, GEN>(descs, ntiles, nd, head, g, status, st, gen)
                       : launch_q_t<4, false, T, GEN>(descs, ntiles, nd, head, g, status, st, gen);
        case 8:
            return std_steps
                       ? launch_q_t<8, true, T, GEN>(descs, ntiles, nd, head, g, status, st, gen)
                       : launch_q_t<8, false, T, GEN>(descs, ntiles, nd, head, g, status, st, gen);
        default:
            return std_steps
                       ? launch_q_t<16, true, T, GEN>(descs, ntiles, nd, head, g, status, st, gen)
                       : launch_q_t<16, false, T, GEN>(descs, ntiles, nd, head, g, status, st,
                                                       gen);
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

int stage1_gen_slots(const Geo& g, int nw, int d) {
    if (d < 1 || d > kGenMaxD) return 0;
    const bool std_steps = g.S == 3 && g.kind[0] == 0 && g.kind[1] == 1 && g.kind[2] == 2;
    switch (nw) {
        case 4:
            return std_steps ? queue_resident<4, true, double, true>(g, d, nullptr)
                             : queue_resident<4, false, double, true>(g, d, nullptr);
        case 8:
            return std_steps ? queue_resident<8, true, double, true>(g, d, nullptr)
                             : queue_resident<8, false, double, true>(g, d, nullptr);
        case 16:
            return std_steps ? queue_resident<16, true, double, true>(g, d, nullptr)
                             : queue_resident<16, false, double, true>(g, d, nullptr);
        default:
            return 0;
    }
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
