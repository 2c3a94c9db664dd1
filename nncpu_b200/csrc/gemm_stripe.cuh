// Products of 17 to 256 tokens: the tokens are the tensor core's M operand, all of them in one tile, and every SM (or pair
// of SMs) owns a stripe of the weight matrix's rows, all of K.  Part of gemm_sm100.cu.
//
// Such a product should be a stream over the weights.  Cut into tiles of 128 weight rows it has 16 to 192 tiles for 148
// SMs, so the tiles' k-blocks had to be shared among SMs and their partial sums exchanged (through a cluster's shared
// memory up to 64 tokens, through scratch memory and a second kernel above).  Here the N operand is as many weight rows as make
// one round over the SMs (a multiple of 16), so that all SMs stream alike and nothing is exchanged.  The price is that every
// SM reads all tokens (from L2).  Up to 64 tokens a block multiplies alone (M 64), or, with long rows, two blocks share a stripe, each
// multiplies half of K and sends the other the sums of its half of the columns through distributed shared memory; above, two SMs pair up, each loads half of the
// tokens and its own weight rows, and tcgen05.mma with cta_group::2 multiplies the two halves with both stripes.
//
// A stage of the ring holds `kc` chunks of 64 columns of the tokens and of the stripe (one three-dimensional tensor copy
// each: column, row, chunk).  Only as many token rows are copied as there are; the tensor core reads the M rows all the
// same, and what it makes of the bytes behind them are rows nobody stores.
//
// The tensor core cuts its running sum at every instruction instead of rounding it, so a sum over all of K in one accumulator
// would be further from 64 bits than the slices of K that clusters and dealt-out k-blocks add (K 12288: 1.4e-5 of the 2-norm
// against 2.6e-6).  So K is summed in several accumulators one after the other, which the epilogue adds: as many as those kernels' sums
// ask for (least_stretches), eight where tensor memory has room.  Where all of a block's rows would not leave room for two, the
// stripes are narrower and a block walks through K for several of them, with two sets of accumulators in turn (us and error, one accumulator / two;
// 200 tokens: gated 24576 x 4096 57 / 62, 8.9e-6 / 4.3e-6, 65536 x 4096 111 / 121, 4.4e-6 / 2.1e-6; dealt-out k-blocks 69 and 4.5e-6, 173 and 3.7e-6).
//
// What bounds it (times at the rule that sends a product here): up to 64 tokens the instructions, of which a block issues one for 16
// columns of K whatever the width of its stripe (some 45 clk each at N 16 to 64, from the times of different widths; issued back to back
// and without a stage's wait they take 24), and some 0.14 us a stage; the weights' stream at the
// larger widths (gated 24 576 x 4 096 at 64 tokens 40.4 us, 5.0 TB/s); above 64 tokens the tokens that every SM copies beside its weights.  Neither where a unit begins its walk through K (all SMs
// read the same tokens at one time) nor copies by a warp for each operand made a difference.
#pragma once

namespace {

enum StripeMode : int { kStripe64 = 0, kStripePair128 = 1, kStripePair256 = 2, kStripeSplit64 = 3 };
// warp 0: copies, 1: instructions, 2 to 9: epilogue, two a lane quarter
constexpr int kStripeThreads = 2 * 32 + 256;

struct StripeShape {
    int bn;         // weight rows of a block's stripe (a multiple of 16)
    int h0, h1;     // and how they are dealt to the (one or two) instructions of a k step
    int trows;      // rows of tokens that a block copies (a multiple of 8)
    int parts;      // of the tokens, each with units of its own (2: more tokens than a unit multiplies, and few weight rows)
    int kc;         // chunks of 64 columns a stage
    int stages, k_stages;
    int n_tiles;    // stripes of all blocks (of a pair: 2 bn rows)
    int acc_cols;   // columns of an accumulator
    int n_buf, buf_cols, tmem_cols;   // sets of accumulators (one a tile), columns of a set, columns of all
    int k_half;     // kSplit: the first block's stages
    int seg_len;    // stages that are summed into one accumulator
    int pad;        // bytes behind the ring that the tensor core may read beyond the last stage
    int recv;       // bytes for the partner's sums
    int smem;       // bytes of dynamic shared memory (tmem_block_bytes)
};

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* map, uint32_t bar_cluster_addr, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"((uint64_t)map), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
        : "memory");
}

__device__ __forceinline__ void tma_prefetch_3d(const CUtensorMap* map, int x, int y, int z) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global [%0, {%1, %2, %3}];" ::"l"((uint64_t)map), "r"(x), "r"(y), "r"(z) : "memory");
}

// 16 results of one token, features f .. f + 15, through the plain epilogue into rows of floats (p.vec: of whole 16-byte pieces);
// y: what they are added to (already loaded).  Returns the sum of squares when a norm after this product rides on it.
__device__ __forceinline__ float stripe_store16(const GemmParams& p, int token, int f, float (&v)[16], const float4 (&y)[4]) {
    if (p.bias) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] += ld_f(p.bias, f + j, p.bias_dt);
    }
    if (p.nf.act == kActXielu || p.nf.act == kActRelu2) {
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = plain_act_f(v[j], p.nf.act, p.nf.act_a, p.nf.act_b);
    }
    if (p.accumulate) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[4 * j] += y[j].x; v[4 * j + 1] += y[j].y; v[4 * j + 2] += y[j].z; v[4 * j + 3] += y[j].w;
        }
    }
    float* const row = reinterpret_cast<float*>(p.out) + (size_t)token * p.ldc + f;
    if (p.vec) {
#pragma unroll
        for (int j = 0; j < 4; ++j) reinterpret_cast<float4*>(row)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) row[j] = v[j];
    }
    float ss = 0.0f;
    if (p.nf.xg_out != nullptr) {
        __nv_bfloat162 o[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 g = ld_f4(p.nf.gamma, f + 4 * j, p.nf.gamma_dt);
            o[2 * j] = __floats2bfloat162_rn(v[4 * j] * g.x, v[4 * j + 1] * g.y);
            o[2 * j + 1] = __floats2bfloat162_rn(v[4 * j + 2] * g.z, v[4 * j + 3] * g.w);
        }
        uint4* xg = reinterpret_cast<uint4*>(p.nf.xg_out + (size_t)token * p.rows_b + f);
        xg[0] = *reinterpret_cast<uint4*>(o);
        xg[1] = *reinterpret_cast<uint4*>(o + 4);
#pragma unroll
        for (int j = 0; j < 16; ++j) ss = fmaf(v[j], v[j], ss);
    }
    return ss;
}

template <int kMode, int kEpi>
__global__ void __launch_bounds__(kStripeThreads)
gemm_stripe_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w, const GemmParams p,
                   const StripeShape s) {
    constexpr bool kPair = kMode == kStripePair128 || kMode == kStripePair256;
    constexpr bool kSplit = kMode == kStripeSplit64;      // two blocks share a stripe, each half of K
    constexpr bool kAlone64 = kMode == kStripe64 || kSplit;
    constexpr int kM = kAlone64 ? 64 : kMode == kStripePair128 ? 128 : 256;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int bytes_x = s.kc * s.trows * 128, bytes_w = s.kc * s.bn * 128, bytes_stage = bytes_x + bytes_w;
    uint64_t* full = (uint64_t*)(smem + s.stages * bytes_stage + s.pad);
    uint64_t* empty = full + s.stages;
    uint64_t* acc_full = empty + s.stages;  // [2]
    uint64_t* acc_empty = acc_full + 2;     // [2]
    uint64_t* got = acc_empty + 2;          // kSplit: the partner's sums for this block's columns are here
    uint32_t* tmem_slot = (uint32_t*)(got + 1);
    float* recv = (float*)(((uintptr_t)(tmem_slot + 1) + 15) & ~(uintptr_t)15);   // kSplit: [column][64 rows]

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    constexpr bool kTwo = kPair || kSplit;              // blocks of a unit
    const int half = kTwo ? (int)cluster_rank() : 0;
    const int rank = kPair ? half : 0;
    const int unit_of_all = kTwo ? (int)blockIdx.x >> 1 : (int)blockIdx.x, all_units = kTwo ? (int)gridDim.x >> 1 : (int)gridDim.x;
    const int unit = unit_of_all >> (s.parts - 1), units = all_units >> (s.parts - 1);
    const int first_token = (unit_of_all & (s.parts - 1)) * 2 * s.trows + rank * s.trows;
    const int tile_n = kPair ? 2 * s.bn : s.bn;
    const int my_tiles = unit < s.n_tiles ? (s.n_tiles - unit + units - 1) / units : 0;
    // this block's part of K, in stages (kSplit: the first half or the rest)
    const int k_begin = kSplit && half ? s.k_half : 0;
    const int k_mine = kSplit ? (half ? s.k_stages - s.k_half : s.k_half) : s.k_stages;
    const int my_runs = my_tiles * k_mine;              // stages this block works through
    const int n_first = min(s.stages, my_runs);         // copies that need no free stage (they may reach into the next tile)
    const int first_row = unit * tile_n + rank * s.bn, next_row = units * tile_n;
    // One stage's copies: `st` its place in the ring, `ks` its place in K, `n0` the stripe's first row.  In a pair the first
    // block's barrier counts both blocks' copies.  (The walkers below count on by ones: a division by a number that is not known
    // beforehand costs a lone thread as long as a copy.)
    auto load_w = [&](int st, int ks, int n0) {
        uint8_t* const dst = smem + st * bytes_stage + bytes_x;
        if constexpr (kPair) tma_load_3d_pair(dst, &map_w, map_to_rank(smem_u32(&full[st]), 0), 0, n0, (k_begin + ks) * s.kc);
        else tma_load_3d(dst, &map_w, &full[st], 0, n0, (k_begin + ks) * s.kc);
    };
    auto load_x = [&](int st, int ks) {
        uint8_t* const dst = smem + st * bytes_stage;
        if constexpr (kPair) tma_load_3d_pair(dst, &map_x, map_to_rank(smem_u32(&full[st]), 0), 0, first_token, (k_begin + ks) * s.kc);
        else tma_load_3d(dst, &map_x, &full[st], 0, 0, (k_begin + ks) * s.kc);
    };
    // What may be asked for before the kernel before this one is over: up to 64 tokens the weights themselves, which that kernel must
    // not have written (as without stripes); above, it may have, and they are asked for into L2 only.
    auto first_weights = [&]() {
        for (int r = 0, ks = 0, n0 = first_row; r < n_first; ++r) {
            if constexpr (kPair) {
                tma_prefetch_3d(&map_w, 0, n0, (k_begin + ks) * s.kc);
            } else {
                mbar_expect_tx(&full[r], (uint32_t)bytes_stage);
                load_w(r, ks, n0);
            }
            if (++ks == k_mine) { ks = 0; n0 += next_row; }
        }
    };

    let_next_kernel_start();
    if (threadIdx.x == 0) {
        prefetch_tensormap(&map_w);
        prefetch_tensormap(&map_x);
        for (int i = 0; i < s.stages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], kPair ? 16 : 8);
        }
        mbar_init(got, 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        first_weights();
    }
    if (warp == 1) {
        if constexpr (kPair) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(s.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(s.tmem_cols) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if constexpr (kTwo) cluster_barrier();       // both blocks' barriers exist before anyone signals across the cluster
    else __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;
    wait_for_previous_kernels();

    if (warp == 0) {
        if (lane == 0) {
            bool ok = true;
            int ks = 0, n0 = first_row, left = my_runs - n_first;
            for (int r = 0; r < n_first; ++r) {
                if constexpr (kPair) {
                    // (the partner's copies cannot complete a phase early: see gemm_pair_kernel)
                    if (rank == 0) mbar_expect_tx(&full[r], 2u * (uint32_t)bytes_stage);
                    load_w(r, ks, n0);
                }
                load_x(r, ks);
                if (++ks == k_mine) { ks = 0; n0 += next_row; }
            }
            int st = 0, phase = 0;
            for (; left > 0; --left) {
                if (!mbar_wait(&empty[st], phase)) {
                    atomicExch(p.status, kTimeoutEmpty);
                    ok = false;
                    break;
                }
                if (rank == 0) mbar_expect_tx(&full[st], (kPair ? 2u : 1u) * (uint32_t)bytes_stage);
                load_w(st, ks, n0);
                load_x(st, ks);
                if (++ks == k_mine) { ks = 0; n0 += next_row; }
                if (++st == s.stages) { st = 0; phase ^= 1; }
            }
            if (!ok) {
                // give the copies already in flight time to land before the block gives up its shared memory
                const unsigned long long t0 = global_ns();
                while (global_ns() - t0 < 2000000ull) __nanosleep(1000);
            }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            // the whole warp walks along and elects the thread that issues
            const int n0_mma = kPair ? 2 * s.h0 : s.h0, n1_mma = kPair ? 2 * s.h1 : s.h1;
            const uint32_t idesc0 = instr_desc_bf16(kM, n0_mma), idesc1 = instr_desc_bf16(kM, n1_mma);
            const int cols1 = kMode == kStripePair256 ? 2 * s.h0 : s.h0;   // where the second instruction's columns begin
            int st = 0, phase = 0;
            bool ok = true;
            for (int it = 0; it < my_tiles && ok; ++it) {
                const int buf = s.n_buf > 1 ? it & 1 : 0;
                if (!__all_sync(0xffffffffu, mbar_wait(&acc_empty[buf], ((s.n_buf > 1 ? it >> 1 : it) & 1) ^ 1))) {
                    if (lane == 0) atomicExch(p.status, kTimeoutAccumEmpty);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t tmem_d = tmem_base + (uint32_t)(buf * s.buf_cols);
                int in_seg = 0;                       // stages of the accumulator at tmem_d
                for (int ks = 0; ks < k_mine; ++ks) {
                    if (in_seg == s.seg_len) {
                        in_seg = 0;
                        tmem_d += (uint32_t)s.acc_cols;
                    }
                    if (!__all_sync(0xffffffffu, mbar_wait(&full[st], phase))) {
                        if (lane == 0) atomicExch(p.status, kTimeoutFull);
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t stage = smem_u32(smem + st * bytes_stage);
                    if (elect_one()) {
                        for (int c = 0; c < s.kc; ++c) {
                            const uint64_t x_desc = smem_desc_sw128(stage + c * s.trows * 128);
                            const uint64_t w_desc = smem_desc_sw128(stage + bytes_x + c * s.bn * 128);
#pragma unroll
                            for (int k = 0; k < kBlockK / kUmmaK; ++k) {     // 32 bytes a step: 2 in a descriptor's units
                                const uint32_t more = (in_seg > 0 || c > 0 || k > 0) ? 1u : 0u;
                                if constexpr (kPair) umma_bf16_pair(tmem_d, x_desc + 2 * k, w_desc + 2 * k, idesc0, more);
                                else umma_bf16(tmem_d, x_desc + 2 * k, w_desc + 2 * k, idesc0, more);
                            }
                            if (kPair && s.h1 > 0) {
                                const uint64_t w1_desc = smem_desc_sw128(stage + bytes_x + c * s.bn * 128 + s.h0 * 128);
#pragma unroll
                                for (int k = 0; k < kBlockK / kUmmaK; ++k)
                                    umma_bf16_pair(tmem_d + cols1, x_desc + 2 * k, w1_desc + 2 * k, idesc1, (in_seg > 0 || c > 0 || k > 0) ? 1u : 0u);
                            }
                        }
                        if constexpr (kPair) umma_commit_pair(&empty[st]);
                        else umma_commit(&empty[st]);
                        if (ks + 1 == k_mine) {
                            if constexpr (kPair) umma_commit_pair(&acc_full[buf]);
                            else umma_commit(&acc_full[buf]);
                        }
                    }
                    __syncwarp();
                    ++in_seg;
                    if (++st == s.stages) { st = 0; phase ^= 1; }
                }
            }
        }
    } else {
        // Epilogue: a warp may read its quarter of the tensor-memory lanes; the two warps of a quarter take turns at groups of
        // 16 columns.  Where the accumulator's rows are: M 64: 16 rows in the first half of every quarter; M 128 on a
        // pair: rows 0 to 63 of this block in the first two quarters for the first block's stripe, in the last two for the
        // second's; M 256: 128 rows, the columns of both stripes.
        const int quarter = warp & 3, turn = (warp - 2) >> 2;
        const int local = kAlone64 ? (lane < 16 ? quarter * 16 + lane : 1 << 20)
                          : kMode == kStripePair128 ? (quarter & 1) * 32 + lane : quarter * 32 + lane;
        const int token = first_token + local;
        const bool t_ok = local < s.trows && token < p.rows_a;
        const int n_groups = (kMode == kStripePair256 ? 2 * s.bn : s.bn) / 16;
        auto feature_of = [&](int g) {       // the first feature of a group, within the unit's stripes
            if (kAlone64) return 16 * g;
            if (kMode == kStripePair128) return (quarter >> 1) * s.bn + 16 * g;
            int c = 16 * g, base = 0, h = s.h0;
            if (c >= 2 * s.h0) { c -= 2 * s.h0; base = s.h0; h = s.h1; }
            return c >= h ? s.bn + base + c - h : base + c;
        };
        // (a norm's producer goes through stripe_store16 whatever C's alignment)
        const bool rows16 = kEpi == kPlain && p.out_dt == DT_F32 && (p.vec || p.nf.xg_out != nullptr);
        float row_scale = 1.0f;
        if (p.nf.bins_in != nullptr && t_ok)
            row_scale = 1.0f / sqrtf(bins_total(p.nf.bins_in + (size_t)token * kBinWords) * (1.0f / (float)p.K) + p.nf.eps);
        if (p.nf.bins_clear != nullptr && blockIdx.x == 0)     // the norm before: its consumer has run
            for (int i = threadIdx.x - 64; i < p.rows_a * kBinWords; i += 256) p.nf.bins_clear[i] = 0ull;
        auto old_of = [&](int f, float4 (&y)[4]) {
            if (rows16 && p.accumulate && t_ok && f + 16 <= p.rows_b) {
                const float* const src = reinterpret_cast<const float*>(p.out) + (size_t)token * p.ldc + f;
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    y[j] = p.vec ? reinterpret_cast<const float4*>(src)[j] : make_float4(src[4 * j], src[4 * j + 1], src[4 * j + 2], src[4 * j + 3]);
            }
        };
        float4 y[4] = {};
        float ss = 0.0f;
        for (int it = 0; it < my_tiles; ++it) {
            const int n0 = (unit + it * units) * tile_n;
            const int buf = s.n_buf > 1 ? it & 1 : 0;
            // kSplit: groups of columns belong to the two blocks in turn, and a block's groups to its two warps of a quarter
            const int g_step = kSplit ? 4 : 2, g_first = kSplit ? 2 * turn + half : turn;
            if (g_first < n_groups) old_of(n0 + feature_of(g_first), y);          // asked for under the stream
            const bool done = mbar_wait(&acc_full[buf], (s.n_buf > 1 ? it >> 1 : it) & 1);
            if (!__all_sync(0xffffffffu, done)) {
                if (lane == 0) atomicExch(p.status, kTimeoutAccumFull);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * s.buf_cols);
            // a group's sums: K is summed in segments, which are added here in their order
            auto sums_of = [&](int g, float (&v)[16]) {
                tmem_ld16(taddr + (uint32_t)(16 * g), v);     // every lane takes part, whatever its row
                for (int seg = 1; seg * s.seg_len < k_mine; ++seg) {      // (four loads at once were slower: registers)
                    float w[16];
                    tmem_ld16(taddr + (uint32_t)(seg * s.acc_cols + 16 * g), w);
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += w[j];
                }
            };
            if constexpr (kSplit) {
                // the partner's columns go to its shared memory, a column of this warp's 16 rows at a time; its barrier counts
                // the eight warps that have sent theirs
                const uint32_t there = map_to_rank(smem_u32(recv + quarter * 16 + (lane & 15)), (uint32_t)(half ^ 1));
#pragma unroll 1
                for (int g = 2 * turn + (half ^ 1); g < n_groups; g += 4) {
                    float v[16];
                    __syncwarp();                            // the load is the whole warp's
                    sums_of(g, v);
                    if (lane < 16) {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(there + (uint32_t)(((g >> 1) * 16 + j) * 64 * 4)), "f"(v[j]) : "memory");
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(map_to_rank(smem_u32(got), (uint32_t)(half ^ 1)));
                if (!__all_sync(0xffffffffu, mbar_wait(got, 0))) {
                    if (lane == 0) atomicExch(p.status, kTimeoutAccumEmpty);
                    break;
                }
                asm volatile("fence.acq_rel.cluster;" ::: "memory");
            }
#pragma unroll 1
            for (int g = g_first; g < n_groups; g += g_step) {
                const int f = n0 + feature_of(g);
                if (g != g_first) old_of(f, y);
                float v[16];
                __syncwarp();                                // the load is the whole warp's
                sums_of(g, v);
                if constexpr (kSplit) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] += recv[((g >> 1) * 16 + j) * 64 + quarter * 16 + (lane & 15)];
                }
#pragma unroll
                for (int j = 0; j < 16; ++j) v[j] *= row_scale;
                if (t_ok && f < p.rows_b) {
                    if (rows16 && f + 16 <= p.rows_b) ss += stripe_store16(p, token, f, v, y);
                    else store16<kEpi>(p, token, f, v);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) {
                if constexpr (kPair) mbar_arrive_cluster(map_to_rank(smem_u32(&acc_empty[buf]), 0));
                else mbar_arrive(&acc_empty[buf]);
            }
        }
        if (p.nf.xg_out != nullptr && t_ok && my_tiles > 0) bins_add(p.nf.bins_out + (size_t)token * kBinWords, ss);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if constexpr (kTwo) cluster_barrier();       // the partner may still be reading this block's shared memory, or writing to it
    else __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if constexpr (kPair) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(s.tmem_cols) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(s.tmem_cols) : "memory");
    }
}

}  // namespace
