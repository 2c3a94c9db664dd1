// Causal attention over the cache pages in true 32-bit (queries, pages and output float32), on the CUDA cores: heads of at
// most 128 lanes in rows of whole 16-byte pieces.  The general kernel of generic.cu takes everything else; it runs one block
// per (token, head), each of whose threads walks through a whole key row by itself, one load after the other.
//
//   * decode_f32_kernel: a block takes one token, the query heads of one key/value head, and one stretch of the keys;
//     a warp reads whole rows (32 lanes x 16 bytes), eight of them in flight.  The stretches' parts meet in
//     merge_f32_kernel.  How long a row's stretches are follows from its own position and from how many stretches the
//     launch has room for, so a row's result does not depend on the rows beside it as long as that room is the same (the
//     callers': 32, in steps of more than 64 tokens 8).
//   * prompt_f32_kernel: a block takes 32 query rows (a few neighbouring tokens of one sequence times the query heads of one
//     key/value head) and walks through the pages they see; scores and outputs are 32-bit products out of shared memory, four by four
//     and four by eight numbers per thread.
// Measured, 16 heads over 4 of 128 lanes: two sequences of some 600 keys 14 us with the merge (172 in the general kernel),
// a prompt of 300 tokens 57 us (414).  The first is bound by latency (a stretch is two rounds of loads), the second by
// its few blocks: 152 walk through up to five pages, at two 32-row products of 64 keys each.
// Both take what the general kernel takes: windows, blocks, kept first keys, slopes, sinks, caps and a gate per head.
// (the reference's attention: crates/nncpu/src/model/forward.rs:382-470)

#include <math.h>

#define NN_LIB attention_f32
#define NN_LAUNCH_OVERLAP
#include "common.cuh"

namespace {

struct AttnF32 {
    const float* q;            // [n_tok, n_heads * hd]
    const float* k_pages;      // [pages, n_kv, 64, hd]
    const float* v_pages;      // [pages, n_kv, 64, vd]
    const int* block_table;
    int bt_stride;
    const int* tok_seq;
    const int* tok_pos;
    float* out;                // [n_tok, n_heads * vo]
    float* part;               // partial outputs [n_tok, n_heads, n_chunks, vd], then (maximum, sum) pairs behind them
    int n_tok, n_heads, n_kv, hd, vd, vo;
    float scale;
    int window, keep;
    float slope_base;
    const float* sinks;
    float cap;
    const float* head_gate;
    int gate_ld;
    int chunk, n_chunks;       // least keys of a stretch (a multiple of 128), most stretches of a token
    unsigned room;             // chunk * n_chunks, at most 2^31
    int t0;                    // token by token: the launch's first token
    int runs;                  // prompts: blocks a tile of tokens has for the sequences in it
};

// Keys of a stretch for the token at `pos`: the least, doubled until the token's keys fit the stretches there is room for.
__device__ __forceinline__ int stretch_of(const AttnF32& p, int pos) {
    int chunk = p.chunk;
    for (unsigned keys = p.room; keys <= (unsigned)pos; keys *= 2) chunk *= 2;      // (room is at least 128: ends below 2^32)
    return chunk;
}

__device__ __forceinline__ float slope_of(const AttnF32& p, int h) {
    return p.slope_base != 0.0f ? exp2f(-p.slope_base * (float)(h + 1) / (float)p.n_heads) : 0.0f;
}

// A score from its dot product, as the general kernel makes it.
__device__ __forceinline__ float score_of(const AttnF32& p, float dot, float slope, int away) {
    float s = dot * p.scale;
    if (p.cap != 0.0f) s = p.cap * tanhf(s / p.cap);
    return s - slope * (float)away;
}

// What an output row is multiplied by: one over the softmax's denominator, times the head's gate.
__device__ __forceinline__ float closing_factor(const AttnF32& p, int t, int h, float m, float l) {
    if (p.sinks != nullptr) l += expf(p.sinks[h] - m);
    float inv = l > 0.0f ? 1.0f / l : 0.0f;
    if (p.head_gate != nullptr) inv *= 1.0f / (1.0f + expf(0.0f - p.head_gate[(size_t)t * p.gate_ld + h]));
    return inv;
}

__device__ __forceinline__ void axpy4(float a, const float4& x, float4& y) {
    y.x = fmaf(a, x.x, y.x); y.y = fmaf(a, x.y, y.y); y.z = fmaf(a, x.z, y.z); y.w = fmaf(a, x.w, y.w);
}

constexpr int kDecodeKeys = 128;   // keys per round of a block: 32 per warp, half a page
constexpr int kTokensPerLaunch = 65535;

// GB: query heads a block takes (1, 2, 4 or 8), of the n_heads / n_kv that share a key/value head.
template <int GB>
__global__ void __launch_bounds__(128)
decode_f32_kernel(const AttnF32 p) {
    __shared__ float sc[kDecodeKeys][GB];
    __shared__ float red[4][GB];
    __shared__ __align__(16) float part_o[4][GB][128];
    let_next_kernel_start();
    wait_for_previous_kernels();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int group = p.n_heads / p.n_kv, per_kv = (group + GB - 1) / GB;
    const int kvh = blockIdx.x / per_kv, g0 = (blockIdx.x % per_kv) * GB;
    const int t = p.t0 + blockIdx.z;
    const int seq = p.tok_seq[t];
    if (seq < 0) {          // padding: zeros (from the block of the first stretch when nothing is merged)
        if (p.n_chunks == 1)
            for (int i = tid; i < GB * p.vo; i += 128)
                if (g0 + i / p.vo < group)
                    p.out[((size_t)t * p.n_heads + kvh * group + g0 + i / p.vo) * p.vo + i % p.vo] = 0.0f;
        return;
    }
    const int pos = p.tok_pos[t];
    const int first = first_visible_key(pos, p.window);
    const int chunk = stretch_of(p, pos);
    const int d4 = lane * 4;
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4 q[GB];
    float slope[GB];
#pragma unroll
    for (int g = 0; g < GB; ++g) {
        const int h = kvh * group + min(g0 + g, group - 1);       // heads past the group: computed, not stored
        q[g] = d4 < p.hd ? *reinterpret_cast<const float4*>(p.q + ((size_t)t * p.n_heads + h) * p.hd + d4) : zero;
        slope[g] = slope_of(p, h);
    }
    for (int c = blockIdx.y; c < p.n_chunks; c += gridDim.y) {
        const int begin = c * chunk, end = min(begin + chunk, pos + 1);
        if (begin > pos) break;
        float m[GB], l[GB];
        float4 o[GB];
#pragma unroll
        for (int g = 0; g < GB; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.0f;
            o[g] = zero;
        }
        for (int k0 = begin; k0 < end; k0 += kDecodeKeys) {
            if (k0 + kDecodeKeys <= first && k0 >= p.keep) continue;      // no key of this round is visible
            const int w0 = k0 + warp * 32;                                // this warp's 32 keys lie in one page
            // (a warp none of whose keys is visible stays away from its page, which a window may have given back)
            const bool any = w0 <= pos && (w0 + 31 >= first || w0 < p.keep);
            size_t row0 = 0;
            if (any) {
                const int page = p.block_table[(size_t)seq * p.bt_stride + w0 / kPage];
                row0 = ((size_t)page * p.n_kv + kvh) * kPage + w0 % kPage;
#pragma unroll 1
                for (int j0 = 0; j0 < 32; j0 += 8) {
                    float4 k[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)      // rows past the last key lie in the page all the same
                        k[j] = d4 < p.hd ? *reinterpret_cast<const float4*>(p.k_pages + (row0 + j0 + j) * p.hd + d4) : zero;
                    float dot[8 * GB];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
#pragma unroll
                        for (int g = 0; g < GB; ++g)
                            dot[j * GB + g] = fmaf(q[g].w, k[j].w, fmaf(q[g].z, k[j].z, fmaf(q[g].y, k[j].y, q[g].x * k[j].x)));
                    const int base = lane_totals<8 * GB>(dot, lane);
#pragma unroll
                    for (int i = 0; i < (8 * GB > 32 ? 8 * GB / 32 : 1); ++i)
                        (&sc[warp * 32 + j0][0])[base + i] = dot[i];
                }
            }
            __syncthreads();
            const int key = k0 + tid;
            const bool visible = key <= pos && (key >= first || key < p.keep);
            float s[GB], m_new[GB];
#pragma unroll
            for (int g = 0; g < GB; ++g) {
                s[g] = visible ? score_of(p, sc[tid][g], slope[g], pos - key) : -INFINITY;
                const float mw = warp_max(s[g]);
                if (lane == 0) red[warp][g] = mw;
            }
            __syncthreads();
#pragma unroll
            for (int g = 0; g < GB; ++g)
                m_new[g] = fmaxf(m[g], fmaxf(fmaxf(red[0][g], red[1][g]), fmaxf(red[2][g], red[3][g])));
            __syncthreads();
#pragma unroll
            for (int g = 0; g < GB; ++g) {
                const float w = visible ? expf(s[g] - m_new[g]) : 0.0f;
                sc[tid][g] = w;
                const float sum = warp_sum(w);
                if (lane == 0) red[warp][g] = sum;
            }
            __syncthreads();
#pragma unroll
            for (int g = 0; g < GB; ++g) {
                const float corr = m[g] == m_new[g] ? 1.0f : expf(m[g] - m_new[g]);     // 0 in the first round
                l[g] = l[g] * corr + ((red[0][g] + red[1][g]) + (red[2][g] + red[3][g]));
                m[g] = m_new[g];
                o[g].x *= corr; o[g].y *= corr; o[g].z *= corr; o[g].w *= corr;
            }
            if (any) {
#pragma unroll 1
                for (int j0 = 0; j0 < 32; j0 += 8) {
                    float4 v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {        // a row that the query does not see counts as zeros, whatever it holds
                        const int key_j = w0 + j0 + j;
                        const bool seen = key_j <= pos && (key_j >= first || key_j < p.keep);
                        v[j] = seen && d4 < p.vd ? *reinterpret_cast<const float4*>(p.v_pages + (row0 + j0 + j) * p.vd + d4) : zero;
                    }
#pragma unroll
                    for (int j = 0; j < 8; ++j)
#pragma unroll
                        for (int g = 0; g < GB; ++g) axpy4(sc[warp * 32 + j0 + j][g], v[j], o[g]);
                }
            }
            __syncthreads();       // the next round writes scores and sums again
        }
        // the four warps' outputs, added in warp order
#pragma unroll
        for (int g = 0; g < GB; ++g) *reinterpret_cast<float4*>(&part_o[warp][g][d4]) = o[g];
        __syncthreads();
#pragma unroll
        for (int g = 0; g < GB; ++g) {
            if (g0 + g >= group) break;
            const int h = kvh * group + g0 + g;
            const float v = (part_o[0][g][tid] + part_o[1][g][tid]) + (part_o[2][g][tid] + part_o[3][g][tid]);
            if (p.n_chunks == 1) {
                if (tid < p.vo) p.out[((size_t)t * p.n_heads + h) * p.vo + tid] = v * closing_factor(p, t, h, m[g], l[g]);
            } else {
                const size_t slot = ((size_t)t * p.n_heads + h) * p.n_chunks + c;
                if (tid < p.vd) p.part[slot * p.vd + tid] = v;
                if (tid == 0) {
                    float* ml = p.part + (size_t)p.n_tok * p.n_heads * p.n_chunks * p.vd + slot * 2;
                    ml[0] = m[g];
                    ml[1] = l[g];
                }
            }
        }
        __syncthreads();
    }
}

// Adds the stretches' parts in their order: a block per (head, token), a thread per lane of the values.
__global__ void __launch_bounds__(128)
merge_f32_kernel(const AttnF32 p) {
    let_next_kernel_start();
    wait_for_previous_kernels();
    const int h = blockIdx.x, t = p.t0 + blockIdx.y, d = threadIdx.x;
    const size_t out = ((size_t)t * p.n_heads + h) * p.vo + d;
    if (p.tok_seq[t] < 0) {
        if (d < p.vo) p.out[out] = 0.0f;
        return;
    }
    const int n = p.tok_pos[t] / stretch_of(p, p.tok_pos[t]) + 1;
    const size_t slot0 = ((size_t)t * p.n_heads + h) * p.n_chunks;
    const float* ml = p.part + (size_t)p.n_tok * p.n_heads * p.n_chunks * p.vd + slot0 * 2;
    float m = -INFINITY;
    for (int c = 0; c < n; ++c) m = fmaxf(m, ml[2 * c]);
    float l = 0.0f, acc = 0.0f;
    for (int c = 0; c < n; ++c) {
        if (ml[2 * c + 1] == 0.0f) continue;       // no key of this stretch was visible
        const float w = expf(ml[2 * c] - m);
        l = fmaf(w, ml[2 * c + 1], l);
        if (d < p.vd) acc = fmaf(w, p.part[(slot0 + c) * p.vd + d], acc);
    }
    if (d < p.vo) p.out[out] = acc * closing_factor(p, t, h, m, l);
}

// ---------------------------------------------------------------------------
// Prompts.
// ---------------------------------------------------------------------------
constexpr int kRowsQ = 32;           // query rows of a block
constexpr int kPsLd = kRowsQ + 4;    // a key's row of weights in shared memory

__device__ __forceinline__ void copy16(void* dst, const void* src, bool real) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "r"(real ? 16 : 0)
                 : "memory");
}

__global__ void __launch_bounds__(128)
prompt_f32_kernel(const AttnF32 p) {
    extern __shared__ __align__(16) float sm[];
    const int ld_q = p.hd + 4, ld_k = p.hd + 4;     // four more: rows start in different banks
    float* qs = sm;                                 // [32][hd + 4]
    float* ks = qs + kRowsQ * ld_q;                 // [64][hd + 4]
    float* vs = ks + kPage * ld_k;                  // [64][vd]
    float* ps = vs + kPage * p.vd;                  // [64][36]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int group = p.n_heads / p.n_kv, per_block = kRowsQ / group;      // tokens of a block
    // One dimension of blocks: key/value heads, then the runs of a tile (tokens of one sequence), then the tiles, the last
    // tokens' first (their walks are the longest).
    const int kvh = (int)(blockIdx.x % p.n_kv), nth = (int)(blockIdx.x / p.n_kv) % p.runs;
    const int n_tiles = (p.n_tok + per_block - 1) / per_block;
    int t0 = (n_tiles - 1 - (int)(blockIdx.x / p.n_kv) / p.runs) * per_block;
    int t1 = min(t0 + per_block, p.n_tok);
    if (p.runs > 1) {
        // this block's run; the last block of a tile takes the runs that are left
        int r = t0, run = 0;
        for (; run < nth && r < t1; ++run) {
            const int seq = p.tok_seq[r];
            for (++r; r < t1 && p.tok_seq[r] == seq; ++r) {}
        }
        if (r >= t1) return;
        t0 = r;
        if (nth + 1 < p.runs) {
            const int seq = p.tok_seq[r];
            for (++r; r < t1 && p.tok_seq[r] == seq; ++r) {}
            t1 = r;
        }
    }

    for (int i = tid; i < kRowsQ * (p.hd / 4); i += 128) {
        const int r = i / (p.hd / 4), d = (i % (p.hd / 4)) * 4;
        const int t = t0 + r / group;
        *reinterpret_cast<float4*>(qs + r * ld_q + d) =
            r < per_block * group && t < t1
                ? *reinterpret_cast<const float4*>(p.q + ((size_t)t * p.n_heads + kvh * group + r % group) * p.hd + d)
                : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    float m[4], l[4], acc[4][8], slope[4];
    int row_t[4], row_pos[4], row_first[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i, t = t0 + r / group;
        const bool real = r < per_block * group && t < t1;
        row_t[i] = real ? t : -1;
        row_pos[i] = real ? p.tok_pos[t] : -1;
        row_first[i] = real ? first_visible_key(row_pos[i], p.window) : 0;
        slope[i] = slope_of(p, kvh * group + r % group);
        m[i] = -INFINITY;
        l[i] = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    }
    // a run of tokens of one sequence after the other (a block that has the rest of a tile may hold several)
    for (int r0 = t0; r0 < t1;) {
        const int seq = p.tok_seq[r0];
        int r1 = r0 + 1;
        while (r1 < t1 && p.tok_seq[r1] == seq) ++r1;
        const int run0 = r0;
        r0 = r1;
        if (seq < 0) continue;                       // padding: its rows stay zeros
        const int last = p.tok_pos[r1 - 1];
        const PageWalk walk(first_visible_key(p.tok_pos[run0], p.window), last, p.keep);
        const int* table = p.block_table + (size_t)seq * p.bt_stride;
        auto fetch = [&](const float* pages, int width, int ld, float* dst, int i) {
            const int key0 = walk.page(i) * kPage;
            const float* src = pages + ((size_t)table[walk.page(i)] * p.n_kv + kvh) * kPage * width;
            for (int e = tid; e < kPage * (width / 4); e += 128) {
                const int k = e / (width / 4), d = (e % (width / 4)) * 4;
                copy16(dst + k * ld + d, src + (size_t)k * width + d, key0 + k <= last);   // zeros past the last key
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        fetch(p.k_pages, p.hd, ld_k, ks, 0);
        for (int i = 0; i < walk.n; ++i) {
            fetch(p.v_pages, p.vd, p.vd, vs, i);
            asm volatile("cp.async.wait_group 1;" ::: "memory");      // the keys are here, the values on their way
            __syncthreads();
            float s[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) s[a][b] = 0.0f;
            for (int d = 0; d < p.hd; d += 4) {
                float4 qv[4], kv[4];
#pragma unroll
                for (int a = 0; a < 4; ++a) qv[a] = *reinterpret_cast<const float4*>(qs + (ty * 4 + a) * ld_q + d);
#pragma unroll
                for (int b = 0; b < 4; ++b) kv[b] = *reinterpret_cast<const float4*>(ks + (tx + 16 * b) * ld_k + d);
#pragma unroll
                for (int a = 0; a < 4; ++a)
#pragma unroll
                    for (int b = 0; b < 4; ++b)
                        s[a][b] = fmaf(qv[a].w, kv[b].w, fmaf(qv[a].z, kv[b].z, fmaf(qv[a].y, kv[b].y, fmaf(qv[a].x, kv[b].x, s[a][b]))));
            }
            const int key0 = walk.page(i) * kPage;
            float w[4][4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                const bool in_run = row_t[a] >= run0 && row_t[a] < r1;
                float top = -INFINITY;
                bool visible[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int key = key0 + tx + 16 * b;
                    visible[b] = in_run && key <= row_pos[a] && (key >= row_first[a] || key < p.keep);
                    s[a][b] = visible[b] ? score_of(p, s[a][b], slope[a], row_pos[a] - key) : -INFINITY;
                    top = fmaxf(top, s[a][b]);
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
                const float m_new = fmaxf(m[a], top);
                const float corr = m[a] == m_new ? 1.0f : expf(m[a] - m_new);     // 0 on the first keys
                float sum = 0.0f;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    w[b][a] = visible[b] ? expf(s[a][b] - m_new) : 0.0f;
                    sum += w[b][a];
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                l[a] = l[a] * corr + sum;
                m[a] = m_new;
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[a][j] *= corr;
            }
#pragma unroll
            for (int b = 0; b < 4; ++b)
                *reinterpret_cast<float4*>(ps + (tx + 16 * b) * kPsLd + ty * 4) = make_float4(w[b][0], w[b][1], w[b][2], w[b][3]);
            __syncthreads();                          // every thread is done with the keys
            if (i + 1 < walk.n) {
                fetch(p.k_pages, p.hd, ld_k, ks, i + 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            // Values that are not finite would reach rows that do not see their key (0 times infinity): a page that holds
            // any is multiplied key by key with a look at who sees it.
            bool odd = false;
            for (int e = tid; e < kPage * (p.vd / 4); e += 128) {
                const float4 v = *reinterpret_cast<const float4*>(vs + e * 4);
                odd |= !(fabsf(v.x) < INFINITY && fabsf(v.y) < INFINITY && fabsf(v.z) < INFINITY && fabsf(v.w) < INFINITY);
            }
            odd = __syncthreads_or(odd) != 0;         // (the values copied by other threads are here, too)
            const int c0 = tx * 4, c1 = 64 + tx * 4;
            const int n_keys = min(kPage, last - key0 + 1);
            if (!odd) {
#pragma unroll 4
                for (int k = 0; k < n_keys; ++k) {
                    const float4 pr = *reinterpret_cast<const float4*>(ps + k * kPsLd + ty * 4);
                    const float pw[4] = {pr.x, pr.y, pr.z, pr.w};
                    float4 v0 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), v1 = v0;
                    if (c0 < p.vd) v0 = *reinterpret_cast<const float4*>(vs + k * p.vd + c0);
                    if (c1 < p.vd) v1 = *reinterpret_cast<const float4*>(vs + k * p.vd + c1);
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        acc[a][0] = fmaf(pw[a], v0.x, acc[a][0]); acc[a][1] = fmaf(pw[a], v0.y, acc[a][1]);
                        acc[a][2] = fmaf(pw[a], v0.z, acc[a][2]); acc[a][3] = fmaf(pw[a], v0.w, acc[a][3]);
                        acc[a][4] = fmaf(pw[a], v1.x, acc[a][4]); acc[a][5] = fmaf(pw[a], v1.y, acc[a][5]);
                        acc[a][6] = fmaf(pw[a], v1.z, acc[a][6]); acc[a][7] = fmaf(pw[a], v1.w, acc[a][7]);
                    }
                }
            } else {
#pragma unroll 1
                for (int k = 0; k < n_keys; ++k) {
                    const int key = key0 + k;
#pragma unroll
                    for (int a = 0; a < 4; ++a) {
                        if (!(row_t[a] >= run0 && row_t[a] < r1 && key <= row_pos[a] && (key >= row_first[a] || key < p.keep))) continue;
                        const float pw = ps[k * kPsLd + ty * 4 + a];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (c0 < p.vd) acc[a][j] = fmaf(pw, vs[k * p.vd + c0 + j], acc[a][j]);
                            if (c1 < p.vd) acc[a][4 + j] = fmaf(pw, vs[k * p.vd + c1 + j], acc[a][4 + j]);
                        }
                    }
                }
            }
            __syncthreads();                          // values and weights may be written again
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        if (row_t[a] < 0) continue;
        const int r = ty * 4 + a, t = row_t[a], h = kvh * group + r % group;
        const bool padding = p.tok_seq[t] < 0;
        const float f = padding ? 0.0f : closing_factor(p, t, h, m[a], l[a]);
        float* o = p.out + ((size_t)t * p.n_heads + h) * p.vo;
        if (tx * 4 < p.vo)
            *reinterpret_cast<float4*>(o + tx * 4) = make_float4(acc[a][0] * f, acc[a][1] * f, acc[a][2] * f, acc[a][3] * f);
        if (64 + tx * 4 < p.vo)
            *reinterpret_cast<float4*>(o + 64 + tx * 4) = make_float4(acc[a][4] * f, acc[a][5] * f, acc[a][6] * f, acc[a][7] * f);
    }
}

}  // namespace

// Heads that the kernels here take: at most 128 lanes in rows of whole 16-byte pieces, at most 32 query heads per key/value
// head.
extern "C" int nncpu_attention_f32_supported(int n_heads, int n_kv, int hd, int vd, int vo) {
    return n_kv > 0 && n_heads > 0 && n_heads % n_kv == 0 && n_heads / n_kv <= 32 && hd > 0 && hd <= 128 && hd % 4 == 0 &&
           vd > 0 && vd <= 128 && vd % 4 == 0 && vo > 0 && vo <= vd && vo % 4 == 0;
}

// chunk > 0: token by token, every token's keys in at most n_chunks stretches (more than one: `part` holds n_tok * n_heads *
// n_chunks * (vd + 2) floats) of `chunk` keys, a multiple of 128, or of its double, its quadruple and so on where the token has
// more keys than that.  chunk 0: query rows in tiles; tokens of one sequence stand together, in ascending order of position;
// n_seqs: sequences of the step, each of which gets blocks of its own in a tile (0: not known).
extern "C" int nncpu_attention_f32(const void* q, const void* k_pages, const void* v_pages, const int* block_table,
                                   int bt_stride, const int* tok_seq, const int* tok_pos, void* out, void* part, int n_tok,
                                   int n_heads, int n_kv, int hd, int vd, int vo, float scale, int window, int keep,
                                   float slope_base, const float* sinks, float cap, const float* head_gate, int gate_ld,
                                   int chunk, int n_chunks, int n_seqs, int sm_count, void* stream) {
    NN_CHECK(n_tok >= 0 && nncpu_attention_f32_supported(n_heads, n_kv, hd, vd, vo),
             "attention (32-bit): %d heads over %d, %d lanes of keys, %d of values, %d of outputs", n_heads, n_kv, hd, vd, vo);
    NN_CHECK(cap >= 0.0f && keep >= 0 && (head_gate == nullptr || gate_ld >= n_heads), "attention (32-bit): cap %f, %d kept keys, gate rows of %d",
             cap, keep, gate_ld);
    NN_CHECK((uintptr_t)q % 16 == 0 && (uintptr_t)k_pages % 16 == 0 && (uintptr_t)v_pages % 16 == 0 && (uintptr_t)out % 16 == 0,
             "attention (32-bit): queries, pages and output must be 16-byte aligned");
    NN_CHECK(chunk == 0 || (chunk > 0 && chunk % kDecodeKeys == 0 && n_chunks > 0 && (n_chunks == 1 || part != nullptr)),
             "attention (32-bit): stretches of %d keys, %d of them", chunk, n_chunks);
    if (n_tok == 0) return 0;
    cudaStream_t st = (cudaStream_t)stream;
    AttnF32 p{(const float*)q, (const float*)k_pages, (const float*)v_pages, block_table, bt_stride, tok_seq, tok_pos,
              (float*)out, (float*)part, n_tok, n_heads, n_kv, hd, vd, vo, scale, window, keep, slope_base, sinks, cap,
              head_gate, gate_ld, chunk, n_chunks, 0, 0, 1};
    const int group = n_heads / n_kv;
    if (chunk > 0) {
        p.room = (unsigned)((long)chunk * n_chunks < (1L << 31) ? (long)chunk * n_chunks : 1L << 31);
        const int gb = group >= 8 ? 8 : (group > 2 ? 4 : group);
        const int blocks_x = n_kv * ((group + gb - 1) / gb);
        // as many blocks as eight per SM ask for; a block with several stretches takes them in turn
        const long pairs = (long)blocks_x * n_tok;
        long per = (8L * sm_count + pairs - 1) / pairs;
        if (per > n_chunks) per = n_chunks;
        // both launched to start while the kernel before them ends: their launches are as long as their work
        cudaLaunchConfig_t cfg = {};
        cfg.blockDim = dim3(128);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        cfg.attrs = attr;
        cfg.numAttrs = overlap_attribute(attr);
        const auto kernel = gb == 8 ? decode_f32_kernel<8> : gb == 4 ? decode_f32_kernel<4> : gb == 2 ? decode_f32_kernel<2> : decode_f32_kernel<1>;
        // Tokens are the last dimension of the grids, which ends at 65 535: a step of more is several launches.  (With tokens
        // in the first dimension, or all in one, eight sequences of 1 000 keys took 16.5 and sixteen 24 us instead of 13.7 and 17.4.)
        for (p.t0 = 0; p.t0 < n_tok; p.t0 += kTokensPerLaunch) {
            const unsigned tokens = (unsigned)(n_tok - p.t0 < kTokensPerLaunch ? n_tok - p.t0 : kTokensPerLaunch);
            cfg.gridDim = dim3((unsigned)blocks_x, (unsigned)per, tokens);
            cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
            NN_CHECK(e == cudaSuccess, "attention (32-bit): launch failed: %s", cudaGetErrorString(e));
            if (n_chunks > 1) {
                cfg.gridDim = dim3((unsigned)n_heads, tokens);
                e = cudaLaunchKernelEx(&cfg, merge_f32_kernel, p);
                NN_CHECK(e == cudaSuccess, "attention (32-bit, merge): launch failed: %s", cudaGetErrorString(e));
            }
        }
        return 0;
    }
    const int per_block = kRowsQ / group;
    const long tiles = ((long)n_tok + per_block - 1) / per_block;
    p.runs = n_seqs > 0 && n_seqs < per_block ? n_seqs : per_block;
    NN_CHECK(tiles * n_kv * p.runs < (1L << 31), "attention (32-bit): %d tokens in tiles of %d", n_tok, per_block);
    const size_t smem = sizeof(float) * ((size_t)kRowsQ * (hd + 4) + (size_t)kPage * (hd + 4) + (size_t)kPage * vd + (size_t)kPage * kPsLd);
    static bool done[64];
    if (first_use_on_this_device(done)) {
        const cudaError_t e = cudaFuncSetAttribute(prompt_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        NN_CHECK(e == cudaSuccess, "attention (32-bit): shared memory: %s", cudaGetErrorString(e));
    }
    prompt_f32_kernel<<<(unsigned)(tiles * n_kv * p.runs), 128, smem, st>>>(p);
    NN_LAUNCH_OK("attention (32-bit)");
    return 0;
}
