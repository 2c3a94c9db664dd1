// 32-bit matrix products for the runs in true float32:
//   C[M, N] (+)= X[M, K] . W[N, K]^T (+ bias[N]),  X and W float32, C float32 or bfloat16.
//
// Few tokens (at most 16): a stream over the weights on the CUDA cores.  A block owns four weight rows (eight with more than four
// tokens), four warps share K: warp w takes the groups of 128 columns w, w + 4, ..., and a lane reads 16 bytes of each
// of its four rows, four groups ahead, straight into registers.  The general kernel (64 x 16 tiles through shared
// memory, scalar loads, no load in flight while it multiplies) leaves memory idle nine tenths of the time.  Measured (weights
// from memory, us here / us there): N 12288, K 2048, two tokens 16.3 (6.2 TB/s) / 212; N 2048, K 6144 8.4 (6.0 TB/s) / 601;
// sixteen tokens of N 12288 44 / 241.  From 2^20 weights on products come here unless their rows are short (N 1024, K 1024, two
// tokens: 1.6 / 97; N 512, K 512: 1.5 / 36); below, the general kernel's one order of sums for any number of rows is kept.
// An element is summed over k in an order that K alone decides (per lane ascending, then the lanes' tree, then the
// four warps), so a row's result does not depend on how many tokens the step has, up to the 16.
//
// More tokens: the tensor cores, on numbers cut in three.  x = a + b + c, a the nearest bfloat16 number (8 bits), b the nearest one
// to the rest, c what is left: 24 bits are three times eight, so nothing of x is lost (down to 2^-110 in magnitude, from where on
// c's last bits lie below bfloat16's smallest number; see kTiny).  Of the nine products of parts, exact each, the six that
// matter are taken: b c', c b' and c c' are together at most 2^-24 of the product, half a last place of it.  They are accumulated in
// 32-bit by tcgen05.mma kind::f16.  The tensor core does not round its running sum to nearest, so it only sums 64 columns at a time
// (32 where K is short); these sums are added in registers, with float additions.  Against 64-bit sums the result is nearer than
// the CUDA cores' chain of fmaf (figures at f32_many_kernel), and a row with a single one in it passes the weights through
// unchanged.
// Weights are the 128-row operand and tokens the other one (BN of them), K may be cut into slices that a second kernel adds.
//
// The reference computes these products with its float row kernels (crates/nncpu/src/kernels/mod.rs:337-360).

#include <math.h>

#include <algorithm>

#define NN_LIB linear_f32
#define NN_LAUNCH_OVERLAP
#include "common.cuh"
#include "tcgen05.cuh"

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

// ---------------------------------------------------------------------------
// More tokens.
//
// A block's warps: 0 copies tiles of 32 columns to shared memory by TMA, 1 issues the matrix instructions, 2-7 cut what arrived
// into its parts (a and b in its place, c behind it), 8-15 add the sums of 64 columns that tensor memory holds in turn to their
// registers (two warps per quarter of the lanes, half of the tokens each) and store.
// The adders take registers over from the others: 2 x 72 + 2 x 184 a warpgroup's thread, the 4 x 128 of the launch.
//
// Bound by shared memory and by the cutting: of every number of a k-block four bytes go in by TMA, four out to the cutters,
// six in from them and twelve out to the tensor core, (128 + BN) x 6.5 cycles at 128 bytes; the kernel takes 1.3 times that.  (300
// tokens of N 12288, K 2048 took 126 of 143 us without the cutters' arithmetic, 123 without their stores, 126 with one product of parts
// instead of six.)  So BN is as large as the tokens and the two accumulators of tensor memory allow, and the cutters' work is what
// counts: conversions in pairs (cvt.rn.bf16x2) and 16-byte stores; ten cutting warps, the next group's loads ahead, or 8-byte
// stores without selects were no faster.
// Measured (weights from memory, tokens cut beforehand from 96 on): N 12288, K 2048, 17 tokens 42 us, 300 tokens 120, 600 tokens 168 (180
// TFLOP/s of true 32-bit results, where the CUDA cores' peak is 72); N 2048, K 6144, 300 tokens 64.  A layer of 300 tokens (hidden 2048): 254 us for its
// four products, 3 130 us in the general kernel.  Cut into two tf32 numbers they took 251 us, but of a quarter of all numbers
// the last bit was lost.
// Error against 64-bit sums (2-norm, N(0, 1) times N(0, 0.02)), here / the general kernel's chain of fmaf: K 64 0.6e-7 / 1.5e-7,
// 512 3.2e-7 / 4.1e-7, 2048 3.2e-7 / 8.1e-7, 6144 3.3e-7 / 1.4e-6; single products within 2.3 x 2^-24.
// ---------------------------------------------------------------------------
// What the status word says when a wait ran out (each library has its own hundred).
enum LinearF32Status : int { kTimeoutEmpty = 301, kTimeoutAccumEmpty = 302, kTimeoutCut = 303, kTimeoutFull = 304, kTimeoutAccumFull = 305 };
constexpr int kManyThreads = 16 * 32;
constexpr int kCutters = 6;            // warps 2 to 7
constexpr int kManyRegsFew = 72, kManyRegsMany = 184;
static_assert(2 * kManyRegsFew + 2 * kManyRegsMany <= 4 * 128, "no more registers than the launch has");
constexpr int kManyK = 32;             // columns of a k-block: 128 bytes, one swizzle row
// Columns that the tensor core sums by itself: its sums are cut, not rounded, at every step, which over 64 columns leaves 3.2e-7 of
// a result's 2-norm whatever K is, and over 32 columns 0.6 to 1.7e-7.  A chain of fmaf has 1.5e-7 at K 64, 2.9e-7 at 256, 3.5e-7 at
// 384, 4.1e-7 at 512; so below kShortK it is 32, which costs some 7 % there.
constexpr int kShortK = 512;
constexpr int kManyAhead = 8;          // k-blocks of weights that are asked into L2 ahead of their copies

struct ManyParams {
    const float* x;       // for results that are not finite: see below
    const float* w;
    const void* bias;
    int bias_dt;
    void* out;
    int out_dt;
    float* part;          // slices > 1: [slices, M, N]
    uint16_t *cut_ab, *cut_c;   // the tokens cut beforehand: [M][kb_total][32 a, 32 b] and [M][kb_total][32 c] (see f32_cut_kernel)
    int M, N, K, lda, ldc, accumulate;
    int tiles_a, tiles_b, slices, kb_total;
    int flush;            // k-blocks that the tensor core sums by itself
    int* status;
};

// The nearest bfloat16 numbers to two floats, the first in the lower half; and the floats they are.
__device__ __forceinline__ uint32_t nearest_bf16(float x, float y) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
__device__ __forceinline__ float lower(uint32_t two) { return __uint_as_float(two << 16); }
__device__ __forceinline__ float upper(uint32_t two) { return __uint_as_float(two & 0xFFFF0000u); }

// Shared-memory matrix descriptor of a K-major tile whose rows are 64 bytes, swizzled in 64-byte mode: groups of 8 rows are
// 512 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                  // 64-byte swizzle
    return d;
}

// Asks for a tile to come to L2.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"((uint64_t)map), "r"(x), "r"(y) : "memory");
}

// One result in plain float arithmetic over its slice of K: what a sum that is not finite is replaced by, because the cut
// of an infinity, or of a number next to the largest, is not a number (inf - inf) where the product itself may be one; and
// what a sum below kTiny is replaced by, whose numbers may be so small that their third parts are not kept.  (A sum of zero
// stays: it is that of a row of zeros, unless every number of it is below 2^-134.)
constexpr float kTiny = 0x1p-60f;
// (n is a multiple of 4 and both rows start at 16 bytes.)
__device__ __noinline__ float plain_dot(const float* x, const float* w, int n) {
    float a = 0.0f;
#pragma unroll 4
    for (int k = 0; k < n; k += 4) {
        const float4 u = *reinterpret_cast<const float4*>(x + k), v = *reinterpret_cast<const float4*>(w + k);
        a = fmaf(u.x, v.x, a);
        a = fmaf(u.y, v.y, a);
        a = fmaf(u.z, v.z, a);
        a = fmaf(u.w, v.w, a);
    }
    return a;
}

template <int BN>
constexpr int kManyStages = BN > 160 ? 3 : (BN > 96 ? 4 : 5);     // as many as shared memory holds
template <int BN>
constexpr int kManyTmemCols = BN <= 32 ? 64 : (BN <= 64 ? 128 : (BN <= 128 ? 256 : 512));     // two accumulators
template <int BN>
constexpr size_t kManySmem = tmem_block_bytes(1024 + (size_t)kManyStages<BN> * (128 + BN) * 192 + 256, kManyTmemCols<BN>);

// Eight numbers in their three parts.
__device__ __forceinline__ void cut_eight(const float (&x)[8], uint4& va, uint4& vb, uint4& vc) {
    uint32_t a[4], b[4], c[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float x0 = x[2 * j], x1 = x[2 * j + 1];
        a[j] = nearest_bf16(x0, x1);
        const float y0 = x0 - lower(a[j]), y1 = x1 - upper(a[j]);
        b[j] = nearest_bf16(y0, y1);
        c[j] = nearest_bf16(y0 - lower(b[j]), y1 - upper(b[j]));      // 7 bits at most: exact
    }
    va = make_uint4(a[0], a[1], a[2], a[3]);
    vb = make_uint4(b[0], b[1], b[2], b[3]);
    vc = make_uint4(c[0], c[1], c[2], c[3]);
}

// The tokens' parts, made once (bound by its launch: 300 tokens of K 2048 are 2 MB).  Every tile of 128 weight rows multiplies
// with all tokens, so cut where they arrive the tokens are cut N / 128 times: 160 rows of them for 128 of weights in the
// products of a 300-token prompt.  Cut beforehand, 300 tokens of N 12288 x K 2048 take 145 -> 120 us.
__global__ void __launch_bounds__(256) f32_cut_kernel(const ManyParams p) {
    let_next_kernel_start();
    wait_for_previous_kernels();
    const long i = (long)blockIdx.x * 256 + threadIdx.x;        // eight numbers each
    const int per_row = p.kb_total * (kManyK / 8);
    const int row = (int)(i / per_row), g = (int)(i % per_row), k = g * 8;
    if (row >= p.M) return;
    float x[8];
#pragma unroll
    for (int h = 0; h < 2; ++h)       // (K is a multiple of 4)
        *reinterpret_cast<float4*>(&x[4 * h]) = k + 4 * h < p.K ? *reinterpret_cast<const float4*>(p.x + (size_t)row * p.lda + k + 4 * h)
                                                              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    uint4 va, vb, vc;
    cut_eight(x, va, vb, vc);
    uint16_t* ab = p.cut_ab + ((size_t)row * p.kb_total + k / kManyK) * 64 + k % kManyK;
    *reinterpret_cast<uint4*>(ab) = va;
    *reinterpret_cast<uint4*>(ab + 32) = vb;
    *reinterpret_cast<uint4*>(p.cut_c + (size_t)row * p.kb_total * 32 + k) = vc;
}

// kCutX: the tokens' parts come ready-made by TMA (map_x their a and b, map_c their c) and only the weights are cut here.
template <int BN, bool kCutX>
__global__ void __launch_bounds__(kManyThreads, 1)
f32_many_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                const __grid_constant__ CUtensorMap map_c, const ManyParams p) {
    constexpr int kStages = kManyStages<BN>;
    // A k-block: 128 rows of weights, then BN of tokens.  128 bytes a row, as TMA brings them (128-byte swizzle) and, cut, 32 numbers
    // a and 32 numbers b; behind them 64 bytes a row of numbers c (64-byte swizzle).
    constexpr int kRawBytes = (128 + BN) * 128;
    constexpr int kStageBytes = (128 + BN) * 192;
    constexpr int kTmemCols = kManyTmemCols<BN>;
    constexpr int kCols = BN / 2;                     // columns of an adding thread
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + kStages * kStageBytes);
    uint64_t* cut = full + kStages;
    uint64_t* empty = cut + kStages;
    uint64_t* acc_full = empty + kStages;   // [2]
    uint64_t* acc_empty = acc_full + 2;     // [2]
    uint32_t* tmem_slot = (uint32_t*)(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int kCopied = 128 * 128 + BN * (kCutX ? 192 : 128);      // bytes that arrive for a stage
    let_next_kernel_start();
    const int tiles = p.tiles_a * p.tiles_b, n_items = tiles * p.slices;
    // item i: the tiles of tokens of one tile of weights stand together, so that its weights are read from memory once
    auto first_kb = [&](int slice) { return (int)((long)slice * p.kb_total / p.slices); };
    const int slice0 = (int)blockIdx.x / tiles;                        // of this block's first item
    const int n_first = kCutX ? min(kStages, first_kb(slice0 + 1) - first_kb(slice0)) : 0;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&cut[s], kCutters);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 8);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // the first weights are asked for, into L2, while the tokens are being cut: what ran before that may have written them
        for (int r = 0; r < n_first; ++r)
            tma_prefetch_2d(&map_w, (first_kb(slice0) + r) * kManyK, ((int)blockIdx.x / p.tiles_b % p.tiles_a) * 128);
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    wait_for_previous_kernels();

    if (warp < 8) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kManyRegsFew));
        if (warp == 0 && lane == 0) {
            int run = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < n_items && ok; i += gridDim.x) {
                const int n0 = (i % p.tiles_b) * BN, m0 = (i / p.tiles_b % p.tiles_a) * 128, slice = i / tiles;
                for (int kb = first_kb(slice); kb < first_kb(slice + 1); ++kb, ++run) {
                    const int s = run % kStages;
                    if (!mbar_wait(&empty[s], ((run / kStages) & 1) ^ 1)) {
                        atomicExch(p.status, kTimeoutEmpty);
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[s], kCopied);         // (rows past the end are filled with zeros and counted)
                    if (kb + kManyAhead < first_kb(slice + 1)) tma_prefetch_2d(&map_w, (kb + kManyAhead) * kManyK, m0);
                    tma_load_2d(smem + s * kStageBytes, &map_w, &full[s], kb * kManyK, m0);
                    if constexpr (kCutX) {
                        tma_load_2d(smem + s * kStageBytes + 128 * 128, &map_x, &full[s], kb * 64, n0);
                        tma_load_2d(smem + s * kStageBytes + kRawBytes + 128 * 64, &map_c, &full[s], kb * 32, n0);
                    } else {
                        tma_load_2d(smem + s * kStageBytes + 128 * 128, &map_x, &full[s], kb * kManyK, n0);
                    }
                }
            }
            // let the copies in flight land before the block gives up its shared memory
            if (!ok)
                for (int r = max(0, run - kStages); r < run; ++r) mbar_wait(&full[r % kStages], (r / kStages) & 1);
        }
        if (warp == 1 && lane == 0) {
            constexpr uint32_t idesc = instr_desc_bf16(128, BN);
            int run = 0, sum = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < n_items && ok; i += gridDim.x) {
                const int slice = i / tiles, kb1 = first_kb(slice + 1);
                int nth = 0;                                  // of the k-blocks in the sum
                for (int kb = first_kb(slice); kb < kb1; ++kb, ++run) {
                    const int s = run % kStages;
                    if (nth == 0 && !mbar_wait(&acc_empty[sum & 1], ((sum >> 1) & 1) ^ 1)) {
                        atomicExch(p.status, kTimeoutAccumEmpty);
                        ok = false;
                        break;
                    }
                    // (the tokens' parts that TMA brought belong to `full`, which the cutters have waited for, too)
                    if (!mbar_wait(&cut[s], (run / kStages) & 1) || (kCutX && !mbar_wait(&full[s], (run / kStages) & 1))) {
                        atomicExch(p.status, kTimeoutCut);
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t d = tmem_base + (uint32_t)((sum & 1) * BN);
                    const uint32_t w_at = smem_u32(smem + s * kStageBytes), x_at = w_at + 128 * 128;
                    const uint32_t w_rest = w_at + kRawBytes, x_rest = w_rest + 128 * 64;
                    // the parts' products of 16 columns each, the smallest first
                    constexpr uint8_t kOrder[6][2] = {{0, 2}, {2, 0}, {1, 1}, {0, 1}, {1, 0}, {0, 0}};
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        const int pw = kOrder[i][0], px = kOrder[i][1];
#pragma unroll
                        for (int k = 0; k < 2; ++k)
                            umma_bf16(d, pw == 2 ? smem_desc_sw64(w_rest + k * 32) : smem_desc_sw128(w_at + pw * 64 + k * 32),
                                      px == 2 ? smem_desc_sw64(x_rest + k * 32) : smem_desc_sw128(x_at + px * 64 + k * 32), idesc,
                                      (nth > 0 || i > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit(&empty[s]);
                    if (++nth == p.flush || kb + 1 == kb1) {
                        umma_commit(&acc_full[sum & 1]);
                        ++sum;
                        nth = 0;
                    }
                }
            }
        }
        if (warp >= 2) {
            // A lane cuts eight numbers of a row, four lanes a row, a warp eight rows at a time, two such groups at once.  They read
            // all of a row before they write a and b in its place, and neighbouring rows write a and b in turn: no two lanes of
            // a quarter of a warp meet in a bank, reading or writing.
            const int r = lane >> 2, c = lane & 3, r7 = r & 7;
            const int in0 = r * 128 + (((2 * c) ^ r7) << 4), in1 = r * 128 + (((2 * c + 1) ^ r7) << 4);
            const int out_a = r * 128 + ((c ^ r7) << 4), out_b = r * 128 + (((4 + c) ^ r7) << 4);
            const int out_c = r * 64 + ((c ^ ((r >> 1) & 3)) << 4);
            const bool odd = r & 1;
            int run = 0;
            bool ok = true;
            for (int i = blockIdx.x; i < n_items && ok; i += gridDim.x) {
                const int slice = i / tiles, n_kb = first_kb(slice + 1) - first_kb(slice);
                for (int kb = 0; kb < n_kb; ++kb, ++run) {
                    const int s = run % kStages;
                    if (!mbar_wait(&full[s], (run / kStages) & 1)) {
                        if (lane == 0) atomicExch(p.status, kTimeoutFull);
                        ok = false;
                        break;
                    }
                    __syncwarp();
                    uint8_t* const raw = smem + s * kStageBytes;
                    uint8_t* const rest = raw + kRawBytes;
                    constexpr int kGroups = (kCutX ? 128 : 128 + BN) / 8;
#pragma unroll 1
                    for (int g0 = warp - 2; g0 < kGroups; g0 += 2 * kCutters) {
                        const int g1 = g0 + kCutters;
                        float x[2][8];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int g = u == 0 ? g0 : g1;
                            if (g < kGroups) {
                                *reinterpret_cast<float4*>(&x[u][0]) = *reinterpret_cast<const float4*>(raw + g * 1024 + in0);
                                *reinterpret_cast<float4*>(&x[u][4]) = *reinterpret_cast<const float4*>(raw + g * 1024 + in1);
                            }
                        }
                        __syncwarp();
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int g = u == 0 ? g0 : g1;
                            if (g >= kGroups) break;
                            uint4 va, vb, vc;
                            cut_eight(x[u], va, vb, vc);
                            *reinterpret_cast<uint4*>(raw + g * 1024 + (odd ? out_b : out_a)) = odd ? vb : va;
                            *reinterpret_cast<uint4*>(raw + g * 1024 + (odd ? out_a : out_b)) = odd ? va : vb;
                            *reinterpret_cast<uint4*>(rest + g * 512 + out_c) = vc;
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&cut[s]);
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kManyRegsMany));
        const int quarter = warp & 3, half = (warp - 8) >> 2;     // the lanes and the columns that this warp adds up
        const int row_in_tile = quarter * 32 + lane;
        int sum = 0;
        bool ok = true;
        for (int i = blockIdx.x; i < n_items && ok; i += gridDim.x) {
            const int n0 = (i % p.tiles_b) * BN + half * kCols, m0 = (i / p.tiles_b % p.tiles_a) * 128, slice = i / tiles;
            const int kb0 = first_kb(slice), kb1 = first_kb(slice + 1);
            float acc[kCols];
#pragma unroll
            for (int c = 0; c < kCols; ++c) acc[c] = 0.0f;
            for (int kb = kb0; kb < kb1; kb += p.flush, ++sum) {
                if (!mbar_wait(&acc_full[sum & 1], (sum >> 1) & 1)) {
                    if (lane == 0) atomicExch(p.status, kTimeoutAccumFull);
                    ok = false;
                    break;
                }
                __syncwarp();
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((sum & 1) * BN + half * kCols);
#pragma unroll
                for (int c = 0; c < kCols; c += 16) {
                    float v[16];
                    tmem_ld16(taddr + (uint32_t)c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c + j] += v[j];
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[sum & 1]);
            }
            const int row = m0 + row_in_tile;
            if (!ok || row >= p.N) continue;
            const float b = p.slices == 1 && p.bias ? ld_f(p.bias, row, p.bias_dt) : 0.0f;
            // the lanes of a warp write neighbouring features of a token
#pragma unroll
            for (int c0 = 0; c0 < kCols; c0 += 16) {
                float old[16];
#pragma unroll
                for (int c = 0; c < 16; ++c) {       // all loads before the first store
                    const int t = n0 + c0 + c;
                    old[c] = p.slices == 1 && p.accumulate && t < p.M ? ld_f(p.out, (size_t)t * p.ldc + row, p.out_dt) : 0.0f;
                }
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    const int t = n0 + c0 + c;
                    if (t >= p.M) break;
                    float v = acc[c0 + c];
                    if (!(fabsf(v) < INFINITY) || (fabsf(v) < kTiny && v != 0.0f)) {
                        const int k0 = kb0 * kManyK;
                        v = plain_dot(p.x + (size_t)t * p.lda + k0, p.w + (size_t)row * p.K + k0, min(kb1 * kManyK, p.K) - k0);
                    }
                    if (p.slices == 1) st_f(p.out, (size_t)t * p.ldc + row, p.out_dt, (v + b) + old[c]);
                    else p.part[((size_t)slice * p.M + t) * p.N + row] = v;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
}

// Adds the slices' sums in their order, then bias and what is already there.  Bound by the slices' passes through L2; kVec: four
// features a thread (N and ldc multiples of 4, 32-bit output), else one.  A layer of 300 tokens (hidden 2048) spent 50 us
// of 329 here one feature at a time.
template <bool kVec>
__global__ void __launch_bounds__(256)
f32_slices_kernel(const ManyParams p) {
    let_next_kernel_start();
    wait_for_previous_kernels();
    const long total = (long)p.M * p.N;
    if constexpr (kVec) {
        const long e = ((long)blockIdx.x * 256 + threadIdx.x) * 4;
        if (e >= total) return;
        const int t = (int)(e / p.N), row = (int)(e % p.N);
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
        for (int s = 0; s < p.slices; ++s) {
            const float4 x = __ldcs(reinterpret_cast<const float4*>(p.part + (size_t)s * total + e));
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        if (p.bias) {
            v.x += ld_f(p.bias, row, p.bias_dt); v.y += ld_f(p.bias, row + 1, p.bias_dt);
            v.z += ld_f(p.bias, row + 2, p.bias_dt); v.w += ld_f(p.bias, row + 3, p.bias_dt);
        }
        float4* at = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.out) + (size_t)t * p.ldc + row);
        if (p.accumulate) {
            const float4 x = *at;
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        *at = v;
        return;
    }
    const long e = ((long)blockIdx.x * 256 + threadIdx.x);
    if (e >= total) return;
    const int t = (int)(e / p.N), row = (int)(e % p.N);
    float v = 0.0f;
    for (int s = 0; s < p.slices; ++s) v += p.part[(size_t)s * total + e];
    if (p.bias) v += ld_f(p.bias, row, p.bias_dt);
    const size_t o = (size_t)t * p.ldc + row;
    if (p.accumulate) v += ld_f(p.out, o, p.out_dt);
    st_f(p.out, o, p.out_dt, v);
}

// How a product is cut: tokens in equal tiles of at most 256 (a multiple of 32), K in slices.
struct ManyPlan {
    int bn, tiles_b, slices;
};

// The slices with the smallest sum of rounds of the SMs times k-blocks of a slice (six more for filling and draining a
// block's pipeline), and the passes of the slices' sums through memory, in k-blocks too: one takes some (128 + BN) x 7
// cycles; the sums pass at some 2 KB a cycle, and a launch costs 4 000 cycles.
ManyPlan many_plan(int M, int N, int K) {
    ManyPlan plan;
    plan.tiles_b = (M + 255) / 256;
    plan.bn = ((M + plan.tiles_b - 1) / plan.tiles_b + 31) / 32 * 32;
    const int kb = (K + kManyK - 1) / kManyK, sms = sm_count();
    const long tiles = (long)((N + 127) / 128) * plan.tiles_b;
    const double per_kb = (128.0 + plan.bn) * 7.0;
    plan.slices = 1;
    double best = 0.0;
    for (int s = 1; s <= 8 && (s == 1 || kb / s >= 8); ++s) {
        const double rounds = (double)((tiles * s + sms - 1) / sms);
        double cost = rounds * ((kb + s - 1) / s + 6);
        if (s > 1) cost += (4000.0 + (double)s * M * N * 8.0 / 2048.0) / per_kb;
        if (s == 1 || cost < best) {
            best = cost;
            plan.slices = s;
        }
    }
    return plan;
}

// A [rows, K] float matrix with rows of `ld` floats, in boxes of box_rows x 32.
int make_map_f32(CUtensorMap* map, const void* base, int rows, int K, long ld, int box_rows) {
    EncodeTiledFn fn = encode_tiled();
    NN_CHECK(fn != nullptr, "linear (32-bit): the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    const cuuint32_t box[2] = {(cuuint32_t)kManyK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    NN_CHECK(r == CUDA_SUCCESS, "linear (32-bit): cuTensorMapEncodeTiled failed with code %d (rows %d, K %d, ld %ld, box %d)", (int)r,
             rows, K, ld, box_rows);
    return 0;
}

// The cut tokens: [rows, cols] 16-bit parts, in boxes of box_rows x box_cols (64: a and b; 32: c).
int make_map_cut(CUtensorMap* map, const void* base, int rows, long cols, int box_rows, int box_cols) {
    EncodeTiledFn fn = encode_tiled();
    NN_CHECK(fn != nullptr, "linear (32-bit): the driver does not offer cuTensorMapEncodeTiled");
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    NN_CHECK(r == CUDA_SUCCESS, "linear (32-bit): cuTensorMapEncodeTiled failed with code %d (parts of %d rows)", (int)r, rows);
    return 0;
}

template <int BN, bool kCutX>
int launch_many(const ManyParams& p, cudaStream_t stream) {
    CUtensorMap mw, mx, mc;
    if (int e = make_map_f32(&mw, p.w, p.N, p.K, p.K, 128)) return e;
    if constexpr (kCutX) {
        if (int e = make_map_cut(&mx, p.cut_ab, p.M, (long)p.kb_total * 64, BN, 64)) return e;
        if (int e = make_map_cut(&mc, p.cut_c, p.M, (long)p.kb_total * 32, BN, 32)) return e;
    } else {
        if (int e = make_map_f32(&mx, p.x, p.M, p.K, p.lda, BN)) return e;
        mc = mx;
    }
    constexpr size_t smem = kManySmem<BN>;
    static_assert(smem <= 227 * 1024, "the stages fit shared memory");
    static bool configured[64] = {};
    if (first_use_on_this_device(configured)) {
        const cudaError_t e = cudaFuncSetAttribute(f32_many_kernel<BN, kCutX>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        NN_CHECK(e == cudaSuccess, "linear (32-bit): cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    }
    const long items = (long)p.tiles_a * p.tiles_b * p.slices;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(items < sm_count() ? items : sm_count()));
    cfg.blockDim = dim3(kManyThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    cfg.numAttrs = overlap_attribute(attr);
    cfg.attrs = attr;
    cudaError_t e = cudaSuccess;
    if constexpr (kCutX) {
        cudaLaunchConfig_t pre = cfg;
        pre.gridDim = dim3((unsigned)(((long)p.M * p.kb_total * (kManyK / 8) + 255) / 256));
        pre.blockDim = dim3(256);
        pre.dynamicSmemBytes = 0;
        e = cudaLaunchKernelEx(&pre, f32_cut_kernel, p);
        NN_CHECK(e == cudaSuccess, "linear (32-bit, cutting): launch failed: %s", cudaGetErrorString(e));
    }
    e = cudaLaunchKernelEx(&cfg, f32_many_kernel<BN, kCutX>, mw, mx, mc, p);
    NN_CHECK(e == cudaSuccess, "linear (32-bit): launch failed: %s", cudaGetErrorString(e));
    if (p.slices > 1) {
        const bool vec = p.N % 4 == 0 && p.ldc % 4 == 0 && p.out_dt == DT_F32 && (uintptr_t)p.out % 16 == 0 && (uintptr_t)p.part % 16 == 0;
        const long per = vec ? 1024 : 256;
        cfg.gridDim = dim3((unsigned)(((long)p.M * p.N + per - 1) / per));
        cfg.blockDim = dim3(256);
        cfg.dynamicSmemBytes = 0;
        e = vec ? cudaLaunchKernelEx(&cfg, f32_slices_kernel<true>, p) : cudaLaunchKernelEx(&cfg, f32_slices_kernel<false>, p);
        NN_CHECK(e == cudaSuccess, "linear (32-bit, adding slices): launch failed: %s", cudaGetErrorString(e));
    }
    return 0;
}

}  // namespace

// Floats that the parts of M tokens take where they are cut beforehand (0: cut where they arrive).  The cutting is a launch of its
// own, and with few tokens there is little of them to cut beside 128 rows of weights (us, on arrival / beforehand, N x K 12288 x
// 2048 and 2048 x 6144: 17 tokens 42.6 / 44.5 and 26.1 / 28.1, 64 tokens 46.8 / 47.5 and 29.6 / 32.3, 100 tokens 66.8 / 58.0 and
// 41.7 / 36.3, 300 tokens 145 / 120 and 74.7 / 64.1, 600 tokens 210 / 168 and 119 / 107; 100 tokens of 2048 x 2048 22.3 / 21.5).
// The parts are half as large again as the tokens, so that many tokens go through the product in bands, each a product of its own, whose
// parts take kCutMost floats at most (256 MB).  8192 tokens of K 6144 would take 302 MB beside 201 MB of tokens (N 2048: 1 240 us; in two
// bands of 151 MB, sums of slices included, 1 180 us).
constexpr int kCutFrom = 96;
constexpr long kCutMost = 1l << 26;
static long cut_floats(int M, int K) {
    return M < kCutFrom ? 0 : (long)M * ((K + kManyK - 1) / kManyK) * (kManyK * 3 / 2);
}
static int cut_band(int M, int K) {
    const long bands = (cut_floats(M, K) + kCutMost - 1) / kCutMost;
    return bands <= 1 ? M : (int)((M + 256 * bands - 1) / (256 * bands)) * 256;
}

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

// Floats of scratch that nncpu_linear_f32_many needs at these sizes (0: none).
extern "C" long nncpu_linear_f32_many_scratch(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const int band = cut_band(M, K);
    long most = 0;
    for (const int m : {band, M % band}) {
        if (m == 0) continue;
        const ManyPlan plan = many_plan(m, N, K);
        most = std::max(most, cut_floats(m, K) + (plan.slices > 1 ? (long)plan.slices * m * N : 0));
    }
    return most;
}

// The same product for any number of tokens, on the tensor cores.  `scratch`: see above.  `status` is set when a bounded wait
// runs out.
extern "C" int nncpu_linear_f32_many(const void* X, const void* W, const void* bias, int bias_dt, void* C, int c_dt, int M, int N,
                                     int K, int lda, int ldc, int accumulate, void* scratch, int* status, void* stream_) {
    cudaStream_t st = (cudaStream_t)stream_;
    NN_CHECK(M > 0 && N > 0 && K > 0 && K % 4 == 0 && lda % 4 == 0 && lda >= K && ldc >= N,
             "linear (32-bit): M %d, N %d, K %d, lda %d, ldc %d", M, N, K, lda, ldc);
    NN_CHECK((uintptr_t)X % 16 == 0 && (uintptr_t)W % 16 == 0, "linear (32-bit): operands must be 16-byte aligned");
    NN_CHECK(scratch != nullptr || many_plan(M, N, K).slices == 1, "linear (32-bit): slices of K need scratch memory (%d tokens)", M);
    const int band = scratch != nullptr ? cut_band(M, K) : M;
    for (int m0 = 0; m0 < M; m0 += band) {
        const int m = std::min(band, M - m0);
        const ManyPlan plan = many_plan(m, N, K);
        ManyParams p{(const float*)X + (size_t)m0 * lda, (const float*)W, bias, bias_dt,
                     (char*)C + (size_t)m0 * ldc * (c_dt == DT_F32 ? 4 : 2), c_dt, (float*)scratch, nullptr, nullptr, m, N, K, lda, ldc, accumulate,
                     (N + 127) / 128, plan.tiles_b, plan.slices, (K + kManyK - 1) / kManyK, K < kShortK ? 1 : 2, status};
        NN_CHECK((long)p.tiles_a * p.tiles_b * p.slices < (1L << 31), "linear (32-bit): %d tokens of %d features", M, N);
        const long floats = scratch != nullptr ? cut_floats(m, K) : 0;
        if (floats > 0) {
            NN_CHECK((uintptr_t)scratch % 16 == 0, "linear (32-bit): scratch memory must be 16-byte aligned");
            p.cut_ab = (uint16_t*)scratch;
            p.cut_c = p.cut_ab + (size_t)m * p.kb_total * 64;
            p.part = (float*)scratch + floats;
        }
        int e;
#define NN_MANY(BN_) case BN_: e = floats > 0 ? launch_many<BN_, true>(p, st) : launch_many<BN_, false>(p, st); break;
        switch (plan.bn) {
            NN_MANY(32) NN_MANY(64) NN_MANY(96) NN_MANY(128) NN_MANY(160) NN_MANY(192) NN_MANY(224)
            default: e = floats > 0 ? launch_many<256, true>(p, st) : launch_many<256, false>(p, st);
        }
#undef NN_MANY
        if (e != 0) return e;
    }
    return 0;
}
