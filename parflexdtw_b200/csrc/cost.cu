// Cosine cost matrix C = 1 - L2norm(F1)^T L2norm(F2) in FP64
// (Parflex.py:1470 with FlexDTW.L2norm, FlexDTW.py:213-216).
//
// The reduction over the feature dimension runs in a fixed order
// (k = 0, 1, ..., d-1) with every product and sum rounded separately, the
// same order numpy uses for np.sum(F*F, axis=0) and for a left-to-right
// elementwise accumulation; the device C is therefore bit-identical to the
// deterministic host restatement the parity tests use.  With d = 12 the
// kernel is bound by the HBM write of C (8 B per cell) and FP64 issue
// (2d - 1 ops per cell).
#include "common.cuh"

namespace pfx {

// L2norm of both sequences, F (d, n) stored row-major by feature (F[k * n + i]):
// a thread per frame, features taken kNormFeat at a time so that their loads
// are in flight together (with d up to kNormFeat they are read once). Bound by
// latency: 2000 and 2400 frames of 12 features in 3.3 us, 40 features in 6.6
// (a launch per sequence, loads one by one: 6.5 and 16.8).
constexpr int kNormFeat = 16;
constexpr int kNormThreads = 64;  // small CTAs: a sequence is a few thousand frames

__global__ void __launch_bounds__(kNormThreads)
    k_l2norm_cols(const double* __restrict__ F1, const double* __restrict__ F2, int d, int64_t N,
                  int64_t M, double* __restrict__ An, double* __restrict__ Bn) {
    const int64_t t = blockIdx.x * (int64_t)kNormThreads + threadIdx.x;
    if (t >= N + M) return;
    const bool second = t >= N;
    const int64_t n = second ? M : N, i = second ? t - N : t;
    const double* F = (second ? F2 : F1) + i;
    double* out = (second ? Bn : An) + i;
    double v[kNormFeat], acc = 0.0;
    for (int k0 = 0; k0 < d; k0 += kNormFeat) {
#pragma unroll
        for (int k = 0; k < kNormFeat; ++k)
            if (k0 + k < d) v[k] = F[(int64_t)(k0 + k) * n];
#pragma unroll
        for (int k = 0; k < kNormFeat; ++k)
            if (k0 + k < d) {
                const double sq = __dmul_rn(v[k], v[k]);
                acc = k0 + k == 0 ? sq : __dadd_rn(acc, sq);
            }
    }
    const double nrm = __dadd_rn(__dsqrt_rn(acc), 1e-9);
    for (int k0 = 0; k0 < d; k0 += kNormFeat) {
        if (d > kNormFeat) {
#pragma unroll
            for (int k = 0; k < kNormFeat; ++k)
                if (k0 + k < d) v[k] = F[(int64_t)(k0 + k) * n];
        }
#pragma unroll
        for (int k = 0; k < kNormFeat; ++k)
            if (k0 + k < d) out[(int64_t)(k0 + k) * n] = __ddiv_rn(v[k], nrm);
    }
}

// One thread per output column j, looping over kRows rows; A rows staged in
// shared memory (broadcast reads), B column kept in registers when d <= 16.
template <int DMAX>
__global__ void __launch_bounds__(256) k_cost_f64(const double* __restrict__ A,
                                                  const double* __restrict__ B, int d, int64_t N,
                                                  int64_t M, double* __restrict__ C, int64_t ldc,
                                                  int rows_per_block) {
    extern __shared__ double sA[];  // [rows_per_block][d]
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.y * rows_per_block;
    const int nr = (int)((N - i0) < rows_per_block ? (N - i0) : rows_per_block);
    for (int q = threadIdx.x; q < nr * d; q += blockDim.x) {
        const int ii = q / d, k = q % d;
        sA[q] = A[(int64_t)k * N + i0 + ii];
    }
    __syncthreads();
    if (j >= M) return;
    if (DMAX > 0) {
        double bj[DMAX > 0 ? DMAX : 1];
#pragma unroll
        for (int k = 0; k < DMAX; ++k) bj[k] = k < d ? B[(int64_t)k * M + j] : 0.0;
        for (int ii = 0; ii < nr; ++ii) {
            const double* a = sA + ii * d;
            double acc = __dmul_rn(a[0], bj[0]);
#pragma unroll
            for (int k = 1; k < DMAX; ++k)
                if (k < d) acc = __dadd_rn(acc, __dmul_rn(a[k], bj[k]));
            C[(i0 + ii) * ldc + j] = __dsub_rn(1.0, acc);
        }
    } else {
        for (int ii = 0; ii < nr; ++ii) {
            const double* a = sA + ii * d;
            double acc = __dmul_rn(a[0], __ldg(B + j));
            for (int k = 1; k < d; ++k) acc = __dadd_rn(acc, __dmul_rn(a[k], __ldg(B + (int64_t)k * M + j)));
            C[(i0 + ii) * ldc + j] = __dsub_rn(1.0, acc);
        }
    }
}

cudaError_t launch_l2norm(const double* F1, const double* F2, int d, int64_t N, int64_t M,
                          double* An, double* Bn, cudaStream_t st) {
    if (d < 1 || N < 1 || M < 1) return cudaErrorInvalidValue;
    const int64_t blocks = (N + M + kNormThreads - 1) / kNormThreads;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidValue;
    k_l2norm_cols<<<(unsigned)blocks, kNormThreads, 0, st>>>(F1, F2, d, N, M, An, Bn);
    count_launches(1);
    return cudaGetLastError();
}

// Normalises F1 and F2 into An (d x N) and Bn (d x M) (caller-provided) and
// writes C (N x M, leading dimension ldc).
cudaError_t launch_cost_f64(const double* F1, const double* F2, int d, int64_t N, int64_t M,
                            double* An, double* Bn, double* C, int64_t ldc, cudaStream_t st) {
    cudaError_t e = launch_l2norm(F1, F2, d, N, M, An, Bn, st);
    if (e != cudaSuccess) return e;
    int rows = 64;
    const size_t smem = (size_t)rows * d * sizeof(double);
    if (smem > 200 * 1024) rows = (int)((200 * 1024) / (d * sizeof(double)));
    const size_t sm = (size_t)rows * d * sizeof(double);
    dim3 grid((unsigned)((M + 255) / 256), (unsigned)((N + rows - 1) / rows));
    if (d <= 16) {
        cudaFuncSetAttribute(k_cost_f64<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        k_cost_f64<16><<<grid, 256, sm, st>>>(An, Bn, d, N, M, C, ldc, rows);
    } else {
        cudaFuncSetAttribute(k_cost_f64<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
        k_cost_f64<0><<<grid, 256, sm, st>>>(An, Bn, d, N, M, C, ldc, rows);
    }
    count_launches(1);
    return cudaGetLastError();
}

}  // namespace pfx
