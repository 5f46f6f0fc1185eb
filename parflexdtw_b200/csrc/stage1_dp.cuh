// The FlexDTW wavefront of the stage-1 kernels (stage1_v3.cu: one tile per
// CTA; stage1_cl.cu: one tile per cluster): a warp's strip of 64 rows, the
// rings between strips and the bounded waits.  Mapping and schedule:
// stage1_v3.cu.
#pragma once
#include <cuda/atomic>

#include "common.cuh"
#include "exchange.cuh"

#include <math_constants.h>

namespace pfx {

constexpr int kSpinLimit = 1 << 22;

// Pulls the cost of a strip's next block of steps (kBlk steps x 32 lanes,
// contiguous in the skewed slab) into L2 with one bulk prefetch, so that the
// DP's own loads, two to four steps ahead, hit L2 instead of HBM.  Issued by one lane;
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
// 2^-21 (two FP32 roundings are at most 2^-24 each) decides "less" where no
// quotient can be subnormal (the mdists' product is below 2^35); in between
// the two IEEE divisions decide.
__device__ __forceinline__ bool qless_exact(float b, float nd, float a, float md) {
    const double U = __dmul_rn((double)b, (double)md);
    const double V = __dmul_rn((double)a, (double)nd);
    const double diff = __dadd_rn(V, -U);
    if (diff <= 0.0) return false;
    const double mag = __dadd_rn(fabs(U), fabs(V));
    if (diff > __dmul_rn(mag, 0x1p-21) && mag >= 0x1p-60) return true;
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
// FP32 form: RN(a / m) itself, for 0 or 2^-80 <= |a| < 2^120 and an integer 1 <= m <
// 2^17 (twice the tile length at most, which shared memory keeps far below).
// One step of Markstein's division (IBM J. Res. Dev. 34, 1990) from the
// approximate reciprocal y, whose relative error is below 2^-22: q is within
// 5.3 ulps of a / m, so a - q m has at most 22 bits and the first FMA forms it
// exactly; the second one rounds a value within 2^-19 ulp of a / m. The
// quotient a / m is at least ulp / 2m >= 2^-18 ulp off every midpoint between two
// FP32 values (it is no midpoint itself: those times m have 25 bits or more), so
// both round alike.
__device__ __forceinline__ float quot(float a, float m) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(m));
    const float q = __fmul_rn(a, y);
    return __fmaf_rn(__fmaf_rn(-m, q, a), y, q);
}

// Steps (1,1), (1,2), (2,1) at one cell, mdists given: branch-free selection.
// Returns false when a comparison is too close to call or a value is not
// finite; the caller then recomputes the cell with select_exact.  RIM: in1 /
// in2 say whether the (1,2) / (2,1) predecessor exists (else all do).
template <bool RIM>
__device__ __forceinline__ bool select_std(double cval, double w0, double w1, double w2,
                                           double x1D, int x1P, double m0, double x2D, int x2P,
                                           double m1, bool in1, double x3D, int x3P, double m2,
                                           bool in2, double& oD, int& oP, int& code) {
    const double a0 = addr(x1D, mulr(cval, w0));
    const double a1 = addr(x2D, mulr(cval, w1));
    const double a2 = addr(x3D, mulr(cval, w2));
    bool win1, win2;
    bool ok1 = decide_quot(a1, m1, a0, m0, win1);
    if (RIM) {
        win1 = win1 && in1;
        ok1 = in1 ? ok1 : a0 < CUDART_INF;
    }
    const double bA = win1 ? a1 : a0, bM = win1 ? m1 : m0;
    bool ok2 = decide_quot(a2, m2, bA, bM, win2);
    if (RIM) {
        win2 = win2 && in2;
        ok2 = in2 ? ok2 : bA < CUDART_INF;
    }
    oD = win2 ? a2 : bA;
    oP = win2 ? x3P : (win1 ? x2P : x1P);
    code = win2 ? 2 : (win1 ? 1 : 0);
    return ok1 && ok2;
}

// FP32 form: the three quotients, correctly rounded, compared as the reference
// compares them: near ties, which a few in a hundred warp steps hold at FP32's
// precision, need no second look. Values outside quot's range go to
// select_exact (RIM: but for 0; in the fast loop that test would cost every
// cell three instructions). Against FP64 cross products, which took eight
// conversions per cell and left those near ties undecided: stage 1 of 64 pairs
// of 1000 to 8000 frames in tiles of 1000, 7.1 -> 5.3 ms.
template <bool RIM>
__device__ __forceinline__ bool select_std(float cval, float w0, float w1, float w2, float x1D,
                                           int x1P, float m0, float x2D, int x2P, float m1,
                                           bool in1, float x3D, int x3P, float m2, bool in2,
                                           float& oD, int& oP, int& code) {
    const float a0 = addr(x1D, mulr(cval, w0));
    float a1 = addr(x2D, mulr(cval, w1));
    float a2 = addr(x3D, mulr(cval, w2));
    if (RIM) {  // a missing predecessor: the incumbent again, never strictly below it
        a1 = in1 ? a1 : a0;
        m1 = in1 ? m1 : m0;
        a2 = in2 ? a2 : a0;
        m2 = in2 ? m2 : m0;
    }
    const float q0 = quot(a0, m0), q1 = quot(a1, m1), q2 = quot(a2, m2);
    const bool win1 = q1 < q0;
    const bool win2 = q2 < (win1 ? q1 : q0);
    oD = win2 ? a2 : (win1 ? a1 : a0);
    oP = win2 ? x3P : (win1 ? x2P : x1P);
    code = win2 ? 2 : (win1 ? 1 : 0);
    const bool below = fabsf(a0) + fabsf(a1) + fabsf(a2) < 0x1p120f;  // false for NaN
    if (RIM) {
        const auto fits = [](float a) { return a == 0.0f || fabsf(a) >= 0x1p-80f; };
        return below && fits(a0) && fits(a1) && fits(a2);
    }
    return below && fminf(fminf(fabsf(a0), fabsf(a1)), fabsf(a2)) >= 0x1p-80f;
}

// The cost of the coming steps.  QD = 0: two steps ahead in registers.  QD > 0:
// QD steps ahead in shared memory, by asynchronous copies (each lane reads only
// what it copied): with few warps on an SM a step takes less time than half an
// L2 round trip, and the registers can hold no deeper queue.  Measured (tiles
// of 2000 x 2000): 8 warps on an SM 3.14 -> 2.71 ms with QD = 4, no better
// with 8; 16 warps on an SM issue-bound, 2.46 -> 2.51 ms, so those keep QD = 0.
template <typename T, int QD>
struct CostQueue {
    uint32_t at;  // this lane's slot of step 0
};
template <typename T>
struct CostQueue<T, 0> {
    typename Vec2<T>::type q[2];  // step tau in slot tau & 1
};
template <typename T>
__host__ __device__ constexpr int cost_step_bytes() {
    return 32 * (int)sizeof(typename Vec2<T>::type);
}
__device__ __forceinline__ void copy_cost(uint32_t dst, const double2* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_cost(uint32_t dst, const float2* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void load_cost(uint32_t at, double2& v) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(at) : "memory");
}
__device__ __forceinline__ void load_cost(uint32_t at, float2& v) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
}
// A strip's first steps (Cs: the strip's cost at this lane, at least 64 steps).
template <int QD, typename T>
__device__ __forceinline__ void queue_start(CostQueue<T, QD>& c,
                                            const typename Vec2<T>::type* Cs) {
    if constexpr (QD == 0) {
        c.q[0] = __ldcs(Cs);
        c.q[1] = __ldcs(Cs + 32);
    } else {
#pragma unroll
        for (int i = 0; i < QD; ++i) {
            copy_cost(c.at + i * cost_step_bytes<T>(), Cs + i * 32);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }
}
// Step t's cost (u: its parity); one group per step is in flight.
template <int QD, typename T>
__device__ __forceinline__ typename Vec2<T>::type queue_take(CostQueue<T, QD>& c, const int u,
                                                             int t) {
    if constexpr (QD == 0) {
        return c.q[u];
    } else {
        asm volatile("cp.async.wait_group %0;" ::"n"(QD - 1) : "memory");
        typename Vec2<T>::type v;
        load_cost(c.at + (uint32_t)(t & (QD - 1)) * cost_step_bytes<T>(), v);
        return v;
    }
}
// The cost of step t + (QD or 2), at src, takes step t's place, if `more`.
template <int QD, typename T>
__device__ __forceinline__ void queue_next(CostQueue<T, QD>& c, const int u, int t,
                                           const typename Vec2<T>::type* src, bool more) {
    if constexpr (QD == 0) {
        if (more) c.q[u] = __ldcs(src);
    } else {
        if (more) copy_cost(c.at + (uint32_t)(t & (QD - 1)) * cost_step_bytes<T>(), src);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
}
template <int QD>
__host__ __device__ constexpr int queue_depth() {
    return QD == 0 ? 2 : QD;
}

// A warp's wavefront state between steps.  At the start of step tau: A's
// outputs 1..3 steps ago, B's output one step ago, the predecessors of this
// step's A cell -- x1 (1,1), x2 (1,2), x3 (2,1) -- already received, and the
// mdists of A's and B's (1,2) predecessors.  Start encodings are internal: a
// cell on row 0 carries its column, one on column 0 minus its row, so that a
// successor inherits its predecessor's encoding everywhere.
template <typename T, int QD>
struct Wave {
    T aD1, aD2, aD3, bD1, x1D, x2D, x3D, m1A, m1B;
    int aP1, aP2, aP3, bP1, x1P, x2P, x3P;
    CostQueue<T, QD> q;
};

// Per-warp rings of a strip's last two rows, [NW][RB] slots, RB a multiple
// of kBlk, and per-warp exchange entries, [NW][kXch].  At the start of its
// step T (counted from the tile's start) every lane stores the pair {B one
// step ago, A two steps ago} and loads its neighbour lane i-1's, which the
// next step uses as x1 and x3.  Lanes 0..30 store into their exchange entry
// (exchange.cuh: one barrier of the warp per step, and another after even
// ones); lane 31 stores into ring slot (T - 64) mod RB, which then holds rows
// 64k+63 and 64k+62 of column j = tau - 64; lane 0 loads ring slot (T' - lag) mod
// RB of the previous strip, its column tau'.  So one address per lane takes the
// place of shuffles, of the ring's own loads and stores and of the selects
// between the two.  Both ring windows of a block start on a multiple of kBlk: no
// address inside a block wraps.  D is one {B, A} vector, the start encodings one
// {B, A} int2.
template <typename T>
struct Rings {
    typename Vec2<T>::type *D, *xD;
    int2 *P, *xP;
};
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
    typename Vec2<T>::type* oD;        // FULL: D and P of every cell at step tau0, this
    int2* oP;                          // lane, in the cost's layout (oD may be the cost)
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
template <typename T, int QD>
__device__ __forceinline__ void advance(Wave<T, QD>& st, T oAD, int oAP, T oBD, int oBP, T x1n,
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

// What a strip is to its tile: rows 0 and 1 or the last row change a step; kRim:
// an inner strip's blocks that reach columns 0 and 1, the last one, or past it;
// kCorner: such blocks of strip 0 and the last strip, and all of a lone strip.
enum StripKind { kInner, kTop, kBottom, kRim, kCorner };

// One step of the fast loop: standard steps, every cell of the strip's rows
// inside the tile has c >= 17 and is off the last column.  Returns false, with
// the wave unchanged, when some lane's cell needs the exact routine.  u: the
// step's parity.  kTop: strip 0 of several (row 0 is the cost itself, rows 1
// and 2 have predecessors on it); kBottom: the last strip of several, whose
// lanes past the last row count for nothing and whose last row is stored; kRim:
// cells outside the columns count for nothing, column 0 is the cost itself,
// column 1 has predecessors on it and the last column is stored; kCorner: all
// of these.
template <StripKind KIND, bool PUSH, bool FULL, typename T, int QD>
__device__ __forceinline__ bool fast_step(Wave<T, QD>& st, const Block<T>& b,
                                          const TileDesc& td, const int u, int t, T rc, T w0, T w1, T w2, double* eD, int32_t* eP,
                                          uint32_t& bitsA, uint32_t& bitsB) {
    constexpr int SD = 2 * (int)sizeof(T), SP = (int)sizeof(int2);
    const int lane = b.lane;
    const typename Vec2<T>::type cc = queue_take<QD, T>(st.q, u, t);
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
    if (KIND == kTop) {
        if (lane == 1) m2A = rc;
        if (lane == 0) m0B = rc;
    }
    const int rA = 64 * b.k + 2 * lane;
    constexpr bool kRimmed = KIND == kRim || KIND == kCorner;
    const int cA = b.tau0 + t - 2 * lane, cB = cA - 1;  // (kRimmed)
    if (kRimmed) {
        if (cA == 1) m0A = m2A = rc;
        if (cB == 1) m0B = rc;
    }
    if (KIND == kCorner) {
        if (rA == 2) m2A = rc;
        if (rA == 0) m0B = rc;
    }
    T oAD, oBD;
    int oAP, oBP, codeA, codeB;
    bool okA = select_std<kRimmed>(cc.x, w0, w1, w2, st.x1D, st.x1P, m0A, st.x2D, st.x2P, st.m1A,
                                   !kRimmed || cA != 1, st.x3D, st.x3P, m2A, true, oAD, oAP,
                                   codeA);
    bool okB = select_std<KIND == kTop || kRimmed>(
        cc.y, w0, w1, w2, st.aD2, st.aP2, m0B, st.aD3, st.aP3, st.m1B, !kRimmed || cB != 1,
        st.x2D, st.x2P, st.m1A, KIND == kTop ? lane != 0 : KIND != kCorner || rA != 0, oBD, oBP,
        codeB);
    if (KIND == kRim) {
        if (cA == 0) {
            oAD = cc.x;
            oAP = -rA;
        }
        if (cB == 0) {
            oBD = cc.y;
            oBP = -rA - 1;
        }
        // columns 1 .. W - 1 are the ones with a selection
        const bool selA = (unsigned)(cA - 1) < (unsigned)(b.W - 1);
        const bool selB = (unsigned)(cB - 1) < (unsigned)(b.W - 1);
        okA = okA || !selA;
        okB = okB || !selB;
        codeA = selA ? codeA : 0;
        codeB = selB ? codeB : 0;
    }
    if (KIND == kCorner) {
        if (rA == 0 || cA == 0) {
            oAD = cc.x;
            oAP = rA == 0 ? cA : -rA;
        }
        if (cB == 0) {
            oBD = cc.y;
            oBP = -rA - 1;
        }
        const bool selA = (unsigned)(cA - 1) < (unsigned)(b.W - 1) && rA != 0 && rA < b.R;
        const bool selB = (unsigned)(cB - 1) < (unsigned)(b.W - 1) && rA + 1 < b.R;
        okA = okA || !selA;
        okB = okB || !selB;
        codeA = selA ? codeA : 0;
        codeB = selB ? codeB : 0;
    }
    if (KIND == kTop && lane == 0) {
        oAD = cc.x;
        oAP = b.tau0 + t;
        codeA = 0;
        okA = true;
    }
    if (KIND == kBottom) {
        okA = okA || rA >= b.R;
        okB = okB || rA + 1 >= b.R;
    }
    if (!__all_sync(0xffffffffu, okA && okB)) return false;
    if (KIND == kBottom) {
        if (rA + 1 >= b.R) codeB = 0;
        if (rA == b.R - 1 || rA + 1 == b.R - 1) {
            const bool isA = rA == b.R - 1;
            const int c = b.tau0 + t - 2 * lane - (isA ? 0 : 1);
            eD[c] = (double)(isA ? oAD : oBD);
            eP[c] = isA ? oAP : oBP;
        }
    }
    if (KIND == kRim && (cA == b.W - 1 || cB == b.W - 1)) {
        const bool isA = cA == b.W - 1;
        const int r = rA + (isA ? 0 : 1);
        eD[r] = (double)(isA ? oAD : oBD);
        eP[r] = b.W == 1 ? 0 : (isA ? oAP : oBP);
    }
    if (KIND == kCorner) {
        if (rA < b.R && (unsigned)cA < (unsigned)b.W)
            store_edges(td, rA, cA, b.R, b.W, oAD, oAP);
        if (rA + 1 < b.R && (unsigned)cB < (unsigned)b.W)
            store_edges(td, rA + 1, cB, b.R, b.W, oBD, oBP);
    }
    if (FULL) {
        b.oD[t * 32] = make_v2<T>(oAD, oBD);
        b.oP[t * 32] = make_int2(oAP, oBP);
    }
    bitsA = bitsA * 4 + codeA;  // the first step ends up highest
    bitsB = bitsB * 4 + codeB;
    st.m1A = addr(m0A, (T)1);
    st.m1B = addr(m0B, (T)1);
    advance(st, oAD, oAP, oBD, oBP, x1n, p1n, x3n, p3n);
    return true;
}

// The fast loop: steps 0 .. 15 of a block, or up to the first that needs the
// exact routine.  Returns the steps done.
template <StripKind KIND, bool PUSH, bool FULL, typename T, int QD>
__device__ __forceinline__ int fast_steps(Wave<T, QD>& st, Block<T>& b, const TileDesc& td, T& rc,
                                          T w0, T w1, T w2,
                                          const typename Vec2<T>::type*& cp, const int ahead,
                                          uint32_t& bitsA, uint32_t& bitsB) {
    double* eD = KIND == kBottom ? td.eD : KIND == kRim ? td.eD + td.L : nullptr;
    int32_t* eP = KIND == kBottom ? td.eP : KIND == kRim ? td.eP + td.L : nullptr;
    constexpr bool rimmed = KIND == kRim || KIND == kCorner;
    int t = 0;
#pragma unroll 1
    for (; t < kBlk; t += 2) {
        if (!fast_step<KIND, PUSH, FULL, T, QD>(st, b, td, 0, t, rc, w0, w1, w2, eD, eP, bitsA,
                                                bitsB))
            return t;
        queue_next<QD, T>(st.q, 0, t, cp, !rimmed || t < ahead);
        rc = addr(rc, (T)1);
        __syncwarp();  // (exchange.cuh)
        if (!fast_step<KIND, PUSH, FULL, T, QD>(st, b, td, 1, t + 1, rc, w0, w1, w2, eD, eP, bitsA,
                                                bitsB))
            return t + 1;
        queue_next<QD, T>(st.q, 1, t + 1, cp + 32, !rimmed || t + 1 < ahead);
        rc = addr(rc, (T)1);
        cp += 64;
        b.w += b.incW;
        b.r += b.incR;
        if (PUSH && b.pD) {
            b.pD += 2;
            b.pP += 2;
        }
    }
    return t;
}

// One step of the careful loop (see run_block).  rim: cells on row 0 / column
// 0 or next to them may occur; mask: cells past the last row / column or on
// it.  Outputs of cells outside the tile are arbitrary (nothing inside reads
// them) but for their code, 0.
template <bool STD, bool PUSH, bool FULL, typename T, int QD>
__device__ __forceinline__ void careful_step(const Geo& g, Wave<T, QD>& st, const Block<T>& b,
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
        okA = select_std<true>(cc.x, w0, w1, w2, st.x1D, st.x1P, m0A, st.x2D, st.x2P, st.m1A,
                                  cA >= 2, st.x3D, st.x3P, m2A, true, oAD, oAP, codeA);
        okB = select_std<true>(cc.y, w0, w1, w2, st.aD2, st.aP2, m0B, st.aD3, st.aP3, st.m1B,
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
    if (FULL) {
        b.oD[t * 32] = make_v2<T>(oAD, oBD);
        b.oP[t * 32] = make_int2(oAP, oBP);
    }
    bitsA = bitsA * 4 + (actA ? codeA : 0);
    bitsB = bitsB * 4 + (actB ? codeB : 0);
    st.m1A = addr(m0A, (T)1);
    st.m1B = addr(m0B, (T)1);
    advance(st, oAD, oAP, oBD, oBP, x1n, p1n, x3n, p3n);
}

// The careful loop: steps t .. 15 of a block.
template <bool STD, bool PUSH, bool FULL, typename T, int QD>
__device__ __forceinline__ void careful_steps(const Geo& g, Wave<T, QD>& st, Block<T>& b,
                                              const TileDesc& td, int t, const bool rim,
                                              const bool mask, T rc,
                                              const typename Vec2<T>::type* cp, int ahead,
                                              uint32_t& bitsA, uint32_t& bitsB) {
    using V2 = typename Vec2<T>::type;
    if constexpr (QD == 0) {
        if (t & 1) {  // the queue in step order: the next step's cost in q[0]
            const V2 s = st.q.q[0];
            st.q.q[0] = st.q.q[1];
            st.q.q[1] = s;
        }
    }
    if (t & 1) cp += 32;
    __syncwarp();  // (the step that left the fast loop stores its pair again)
#pragma unroll 1
    for (; t < kBlk; ++t) {
        const V2 cc = queue_take<QD, T>(st.q, 0, t);
        if constexpr (QD == 0) st.q.q[0] = st.q.q[1];
        // (the register queue's load goes before the step, which is long)
        if constexpr (QD == 0) queue_next<QD, T>(st.q, 1, t, cp, t < ahead);
        careful_step<STD, PUSH, FULL, T, QD>(g, st, b, td, t & 1, t, rim, mask, rc, cc, bitsA,
                                             bitsB);
        if constexpr (QD > 0) queue_next<QD, T>(st.q, 1, t, cp, t < ahead);
        __syncwarp();  // (exchange.cuh)
        cp += 32;
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
}

constexpr int kCornerWidth = 800;  // see run_block

// One block of 16 steps of a strip, in two loops.
//
// The fast loop (standard steps) has no divisions and one branch per step, out
// of the loop when some cell is too close to call. It has a copy for each kind
// of block: inner ones, every cell of which has all its predecessors in the
// tile and off its rim (columns from 17 to the last but one), need no tests at
// all; strip 0 and the last strip a few, because the strips after strip 0
// follow at its pace and a tile ends with its last strip; blocks at the tile's
// first and last columns selects around the selection, because a strip starts
// when the one above has done its first six blocks. With the careful loop for
// those, 12 tiles of 1000 x 1000 take 0.68 ms (0.60), 504 of them 1.85 (1.77).
// The corners' copy, for which every warp of a tile would wait to be fetched,
// is used from kCornerWidth columns on (504 tiles of 1000 x 1000 1.77 -> 1.74
// ms, 399 of 2000 x 2000 4.97 -> 4.87, 80 of 4000 x 4000 4.28 -> 4.15; but 28 of
// 100 x 100 88 -> 93 us and 25 of 500 x 500 0.295 -> 0.298 ms).
// The careful loop does the rest: the remaining steps of a block, cells too
// close to call taking the exact routine, and other step sets, with which all
// cells take it.
//
// What bounds it: warp instructions issued, then the FP64 pipe (half rate), so
// the step is written for few of both.  mdist of a predecessor that the
// previous step also used is that step's mdist + 1 (r + c grows by one per
// step) and B's (2,1) predecessor is A's (1,2) one, so a step converts three
// start encodings; lanes exchange their rows through shared memory (see
// Rings).  The fast loop is unrolled two steps deep only and holds no rare
// code: its size decides how well it is fetched.
template <bool STD, bool PUSH, bool FULL, typename T, int QD>
__device__ __forceinline__ void run_block(const Geo& g, Wave<T, QD>& st, Block<T>& b,
                                          const TileDesc& td, const int nS, uint2* bw) {
    using V2 = typename Vec2<T>::type;
    const T w0 = (T)g.w[0], w1 = (T)g.w[1], w2 = (T)g.w[2];
    const int lane = b.lane;
    uint32_t bitsA = 0, bitsB = 0;
    T rc = (T)(64 * b.k + b.tau0);
    const V2* cp = b.Cs + (int64_t)(b.tau0 + queue_depth<QD>()) * 32;  // the queue's end
    const int ahead = b.span - queue_depth<QD>() - b.tau0;
    const bool left = b.tau0 < 80, right = b.tau0 + 17 > b.W;
    const bool top = b.k == 0, bottom = b.k == nS - 1;
    int t = 0;
    if (STD) {
        if ((top || bottom) && (left || right || top == bottom)) {
            if (b.W >= kCornerWidth)
                t = fast_steps<kCorner, PUSH, FULL, T, QD>(st, b, td, rc, w0, w1, w2, cp, ahead,
                                                           bitsA, bitsB);
        } else if (left || right) {
            t = fast_steps<kRim, PUSH, FULL, T, QD>(st, b, td, rc, w0, w1, w2, cp, ahead, bitsA,
                                                    bitsB);
        } else if (top) {
            t = fast_steps<kTop, PUSH, FULL, T, QD>(st, b, td, rc, w0, w1, w2, cp, ahead, bitsA,
                                                    bitsB);
        } else if (bottom) {
            t = fast_steps<kBottom, PUSH, FULL, T, QD>(st, b, td, rc, w0, w1, w2, cp, ahead,
                                                       bitsA, bitsB);
        } else {
            t = fast_steps<kInner, PUSH, FULL, T, QD>(st, b, td, rc, w0, w1, w2, cp, ahead, bitsA,
                                                      bitsB);
        }
    }
    if (t < kBlk)
        careful_steps<STD, PUSH, FULL, T, QD>(g, st, b, td, t, top || left, bottom || right, rc,
                                              cp, ahead, bitsA, bitsB);
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

template <typename T, int QD>
__device__ __forceinline__ void zero_wave(Wave<T, QD>& st) {
    st.aD1 = st.aD2 = st.aD3 = st.bD1 = st.x1D = st.x2D = st.x3D = st.m1A = st.m1B = 0;
    st.aP1 = st.aP2 = st.aP3 = st.bP1 = st.x1P = st.x2P = st.x3P = 0;
    if constexpr (QD == 0) st.q.q[0].x = st.q.q[0].y = st.q.q[1].x = st.q.q[1].y = 0;
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
    const int x = warp * kXch + exchange_store(b.lane, 0);
    const int y = warp * kXch + exchange_load(b.lane, 0);
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
// value (8 for FP64, 4 for FP32), `queue` the bytes of the warps' cost queues.
inline int ring_len(int lag, int nw, int smem_limit, int vbytes, int queue) {
    const int per = nw * (2 * vbytes + (int)sizeof(int2));
    int pow2 = 16;
    while ((pow2 * 2) * per + nw * (int)sizeof(int) <= smem_limit) pow2 *= 2;
    if (lag - 29 > pow2) return 0;
    const int fit = ((smem_limit - queue - (nw + 6) * (int)sizeof(int)) / per - kXch) / kBlk * kBlk;
    return lag + 128 < fit ? lag + 128 : fit;
}
// Shared memory of a CTA of nw warps for tiles of up to L x L whose strips
// are `lag` steps apart.  qd is the depth asked for; 0 is taken instead where
// the queue would leave the rings less than 64 slots of slack.
struct S1Mem {
    int rb, qd;    // ring slots (0: does not fit), queue depth
    size_t bytes;
    int queue_at;  // offset of the cost queues
};
inline S1Mem stage1_mem(int lag, int nw, int smem_limit, int vbytes, int qd) {
    S1Mem m{0, 0, 0, 0};
    const int queue = nw * qd * 32 * 2 * vbytes;
    int rb = qd ? ring_len(lag, nw, smem_limit, vbytes, queue) : 0;
    m.qd = rb >= lag + 64 ? qd : 0;
    m.rb = m.qd ? rb : ring_len(lag, nw, smem_limit, vbytes, 0);
    if (m.rb == 0) return m;
    const size_t ring = vbytes == 8 ? ring_bytes<double>(nw, m.rb, nw + 2)
                                    : ring_bytes<float>(nw, m.rb, nw + 2);
    m.queue_at = (int)((ring + 15) / 16 * 16);
    m.bytes = m.qd ? (size_t)m.queue_at + queue : ring;
    return m;
}

inline int smem_optin() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    return v;
}

inline int smem_per_sm() {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    return v;
}

// Shared memory budget per CTA when 16/NW CTAs share an SM.
inline int cta_budget(int nw) {
    const int per_cta = smem_per_sm() / (16 / nw) - 2048;  // static smem and reserve
    const int optin = smem_optin();
    return per_cta < optin ? per_cta : optin;
}

}  // namespace pfx
