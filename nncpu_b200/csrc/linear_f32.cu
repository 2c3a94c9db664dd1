// 32-bit matrix products for the runs in true float32:
//   C[M, N] (+)= X[M, K] . W[N, K]^T (+ bias[N]),  X and W float32, C float32 or bfloat16.
//
// Few tokens (at most 16): a stream over the weights on the CUDA cores.  A block owns four weight rows (eight with more than four
// tokens), four warps share K: warp w takes the groups of 128 columns w, w + 4, ..., and a lane reads 16 bytes of each
// of its four rows, four groups ahead, straight into registers.  The general kernel (64 x 16 tiles through shared
// memory, scalar loads, no load in flight while it multiplies) leaves memory idle nine tenths of the time.  Measured (weights
// from memory, us here / us there): N 12288, K 2048, two tokens 16.3 (6.2 TB/s) / 212; N 2048, K 6144 8.4 (6.0 TB/s) / 601;
// sixteen tokens of N 12288 44 / 241.  From 2^20 weights on products come here (N 1024, K 1024, two tokens: 1.6 / 97;
// N 512, K 512: 1.5 / 36); below, the general kernel's one order of sums for any number of rows is kept.
// An element is summed over k in an order that K alone decides (per lane ascending, then the lanes' tree, then the
// four warps), so a row's result does not depend on how many tokens the step has, up to the 16.
//
// The reference computes these products with its float row kernels (crates/nncpu/src/kernels/mod.rs:337-360).

#include <math.h>

#define NN_LIB linear_f32
#define NN_LAUNCH_OVERLAP
#include "common.cuh"

namespace {

constexpr int kFewRows = 4;      // weight rows of a warp
constexpr int kFewWarpsK = 4;    // warps that share K

// MT: tokens (a power of two, M <= MT); WR: groups of four rows that a block owns.
template <int MT, int WR>
__global__ void __launch_bounds__(WR * kFewWarpsK * 32, MT > 4 ? 2 : 4)
f32_few_kernel(const float* __restrict__ X, const float* __restrict__ W, const void* __restrict__ bias, int bias_dt,
               void* __restrict__ C, int c_dt, int M, int N, int K, int lda, int ldc, int accumulate) {
    constexpr int V = MT * kFewRows;
    constexpr int kFewUnroll = MT > 8 ? 2 : 4;    // groups of 128 columns in flight per warp: 4 rows x 4 groups x 512 bytes
    __shared__ float part[kFewWarpsK][WR][V];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int wk = warp % kFewWarpsK, wr = warp / kFewWarpsK;
    const int row0 = ((int)blockIdx.x * WR + wr) * kFewRows;
    const float* w[kFewRows];
#pragma unroll
    for (int r = 0; r < kFewRows; ++r) w[r] = W + (size_t)min(row0 + r, N - 1) * K;   // rows past N: read, not stored

    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.0f;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 wv[kFewUnroll][kFewRows];
    // K is a multiple of 4: a lane's 16 bytes lie inside a row or outside
    auto load_weights = [&](int g) {
#pragma unroll
        for (int u = 0; u < kFewUnroll; ++u) {
            const int k = (g + u * kFewWarpsK) * 128 + lane * 4;
#pragma unroll
            for (int r = 0; r < kFewRows; ++r)
                wv[u][r] = k < K ? __ldcs(reinterpret_cast<const float4*>(w[r] + k)) : zero;
        }
    };
    let_next_kernel_start();
    load_weights(wk);                 // weights depend on no kernel; activations do
    wait_for_previous_kernels();
    const int n_groups = (K + 127) / 128;
    for (int g = wk; g < n_groups; g += kFewUnroll * kFewWarpsK) {
        if (g != wk) load_weights(g);
#pragma unroll
        for (int u = 0; u < kFewUnroll; ++u) {
            const int k = (g + u * kFewWarpsK) * 128 + lane * 4;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                // (tokens past M repeat the last one and are not stored)
                const float4 x = k < K ? *reinterpret_cast<const float4*>(X + (size_t)min(m, M - 1) * lda + k) : zero;
#pragma unroll
                for (int r = 0; r < kFewRows; ++r) {
                    float a = acc[m * kFewRows + r];
                    a = fmaf(x.x, wv[u][r].x, a);
                    a = fmaf(x.y, wv[u][r].y, a);
                    a = fmaf(x.z, wv[u][r].z, a);
                    acc[m * kFewRows + r] = fmaf(x.w, wv[u][r].w, a);
                }
            }
        }
    }
    const int base = lane_totals<V>(acc, lane);
    if constexpr (V >= 32) {
#pragma unroll
        for (int i = 0; i < V / 32; ++i) part[wk][wr][base + i] = acc[i];
    } else {
        part[wk][wr][base] = acc[0];       // lanes with the same total write the same number
    }
    __syncthreads();
    for (int e = threadIdx.x; e < V * WR; e += WR * kFewWarpsK * 32) {
        const int m = e / (WR * kFewRows), rr = e % (WR * kFewRows);
        const int row = (int)blockIdx.x * WR * kFewRows + rr;
        if (m >= M || row >= N) continue;
        float v = 0.0f;
#pragma unroll
        for (int s = 0; s < kFewWarpsK; ++s) v += part[s][rr / kFewRows][m * kFewRows + rr % kFewRows];
        if (bias) v += ld_f(bias, row, bias_dt);
        const size_t o = (size_t)m * ldc + row;
        if (accumulate) v += ld_f(C, o, c_dt);
        st_f(C, o, c_dt, v);
    }
}

template <int MT, int WR>
cudaError_t launch_few(const float* X, const float* W, const void* bias, int bias_dt, void* C, int c_dt, int M, int N, int K,
                       int lda, int ldc, int accumulate, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((N + WR * kFewRows - 1) / (WR * kFewRows)));
    cfg.blockDim = dim3(WR * kFewWarpsK * 32);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.numAttrs = overlap_attribute(attr);
    cfg.attrs = attr;
    return cudaLaunchKernelEx(&cfg, f32_few_kernel<MT, WR>, X, W, bias, bias_dt, C, c_dt, M, N, K, lda, ldc, accumulate);
}

}  // namespace

// What the products here take: rows of whole 16-byte pieces.
extern "C" int nncpu_linear_f32_supported(int M, int N, int K, int lda) {
    return M > 0 && M <= 16 && N > 0 && K > 0 && K % 4 == 0 && lda % 4 == 0;
}

extern "C" int nncpu_linear_f32(const void* X, const void* W, const void* bias, int bias_dt, void* C, int c_dt, int M, int N,
                                int K, int lda, int ldc, int accumulate, void* stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    NN_CHECK(nncpu_linear_f32_supported(M, N, K, lda) && lda >= K && ldc >= N,
             "linear (32-bit): M %d, N %d, K %d, lda %d, ldc %d", M, N, K, lda, ldc);
    NN_CHECK((uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0, "linear (32-bit): operands must be 16-byte aligned");
    const float *x = (const float*)X, *w = (const float*)W;
    // With more than four tokens the activations are what the L1 cache delivers most: two groups of rows share them.
    const cudaError_t e =
        M == 1  ? launch_few<1, 1>(x, w, bias, bias_dt, C, c_dt, M, N, K, lda, ldc, accumulate, st)
        : M == 2 ? launch_few<2, 1>(x, w, bias, bias_dt, C, c_dt, M, N, K, lda, ldc, accumulate, st)
        : M <= 4 ? launch_few<4, 1>(x, w, bias, bias_dt, C, c_dt, M, N, K, lda, ldc, accumulate, st)
        : M <= 8 ? launch_few<8, 2>(x, w, bias, bias_dt, C, c_dt, M, N, K, lda, ldc, accumulate, st)
                 : launch_few<16, 2>(x, w, bias, bias_dt, C, c_dt, M, N, K, lda, ldc, accumulate, st);
    NN_CHECK(e == cudaSuccess, "linear (32-bit): launch failed: %s", cudaGetErrorString(e));
    return 0;
}
