// Split-KV attention of decoding / verification rows over FP8-E4M3 pages (head sizes 128 and 256, up to eight query heads per KV head).
//
// Every row reads its whole cache, so the kernel is a stream over K and V that has to keep up with HBM.  The CUDA-core kernel
// (paged_attention.cu) widens the codes into shared memory and multiplies on the FMA pipe: issue-bound at 0.11 of the measured copy
// bandwidth (32 rows of 0.4 - 8 K tokens, 24 heads on 4 KV heads of 256: 418 us, here 117 us for 287 MB, 2.5 TB/s; the last splits of
// the longest rows bound it).  Here each warp works for
// itself on every fourth run of 16 tokens, straight from global memory to tensor-core fragments (mma.sync m16n8k16, f16 operands, in
// which an E4M3 code is exact; one conversion per two codes, nothing goes through shared memory):
//   * S = Q K^T: the query heads of the KV head are rows 0-7 of A.  The order of the head's dimensions along K of the product is free
//     (the same on both sides), so that a lane's fragments are 16 consecutive codes of one token: one load, and 8 bytes of Q.
//     Q is bf16: scaled by a power of two per head it is exact in f16 down to 2^-30 of the head's largest entry; what f16 drops of smaller
//     ones is multiplied in rows 8-15 of the same product.
//   * softmax in 32 bits, online per warp.  The value row's scale 2^e f joins the weight: w = exp(s) 2^e f over the largest such product.
//   * O += P V: w is split into two f16 terms (23 bits; the largest w is 2^12 to 2^14, so that what lies 2^-36 below it still counts), the high
//     one in rows 0-7 of A and the low one in the unused rows 8-15 of the same product.  A lane's fragments of V are 16 consecutive
//     codes of four tokens; a byte permutation pairs them.
// The tensor core drops what falls below the last bit of an accumulator.  So a score is the 32-bit sum of a product per 64 dimensions, and a
// value's accumulator goes to sums in shared memory after 16 runs.  The partial sums are as exact as those of the CUDA-core kernel, which
// rounds every addition (against 64 bits: 2.5e-8 and 4.1e-8 with splits of 64 tokens, 1.5e-7 and 6.3e-7 with 4096; with scores kept as binary
// logarithms and single accumulators 1.0e-7 and 7.6e-7, in 113 us).  Two terms of w show only where single tokens with scales thousands of times the others'
// make up the result (1.3e-7 and 1.1e-7); a third product for what they drop takes 131 us.
// The warps' results meet in shared memory; the partials are those of the merge pass of paged_attention.cu.
// A row's arithmetic depends only on its position and the split length, not on the batch.
#include "ps_common.cuh"

namespace ps {

constexpr int kF8Threads = 128, kF8Warps = kF8Threads / 32, kF8Tok = 16, kF8Chain = 16;

struct AttnFp8Args {
    const __nv_bfloat16* q;                      // [rows, Hq, D]
    const uint8_t* k_pool; const uint8_t* v_pool; const float* k_scale; const float* v_scale;
    const int* block_table; int max_blocks, page_tokens, num_pages;
    const int* row_slot; const int* row_pos;
    int Hq, Hkv; float scale;
    int split_tokens, max_splits;
    float* part_acc; float* part_ml;
    uint32_t* status;
};

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t e4m3x2_to_f16x2(uint32_t two) {                  // the low 16 bits
    uint32_t h;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"((uint16_t)two));
    return h;
}
__device__ __forceinline__ float f8_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t f16x2_bits(__half lo, __half hi) { return (uint32_t)__half_as_ushort(lo) | ((uint32_t)__half_as_ushort(hi) << 16); }

// grid = (splits, Hkv, rows)
template <int D>
__global__ void __launch_bounds__(kF8Threads, 2) attn_fp8_decode_kernel(const AttnFp8Args a) {
    constexpr int KC = D / 64, VC = D / 128;         // 16-byte pieces of a lane per K token, per V token
    constexpr int QP = D + 8;                        // pitch of a head's queries (f16)
    constexpr float kLog2e = 1.4426950408889634f, kTop = 8192.f;      // 2^13: the largest f16 weight is between 2^12 and 2^14
    __shared__ __align__(16) __half s_q[16 * QP];    // the heads' queries, and behind them 2^24 times what f16 drops of them
    __shared__ float s_qs[8];                        // score factor of a head: softmax scale / power of two of its queries
    __shared__ float s_acc[kF8Warps][8 * D];         // [2 x accumulator][lane]
    __shared__ float s_m[kF8Warps][8], s_l[kF8Warps][8];
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int split = blockIdx.x, kvh = blockIdx.y, row = blockIdx.z, G = a.Hq / a.Hkv;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int visible = a.row_pos[row] + 1;
    const int begin = split * a.split_tokens, end = min(visible, begin + a.split_tokens);
    if (begin >= end) return;                        // (padding rows, and rows that another kernel of the step owns)
    const int slot = a.row_slot[row];
    const int* bt = a.block_table + (size_t)slot * a.max_blocks;

    // ---- queries: warp w stages heads w, w + 4
    for (int h = warp; h < 8; h += kF8Warps) {
        const __nv_bfloat16* src = a.q + ((size_t)row * a.Hq + kvh * G + h) * D;
        float x[D / 32], top = 0.f;
#pragma unroll
        for (int i = 0; i < D / 32; ++i) { x[i] = h < G ? bf16_to_f32(src[lane + 32 * i]) : 0.f; top = fmaxf(top, fabsf(x[i])); }
        top = warp_max(top);
        // largest entry in [2^13, 2^14); an all-zero or non-finite head is taken as it is
        int e = 0;
        if (top > 0.f && top < 3.0e38f) e = max(-126, min(126, 13 - ((int)(__float_as_uint(top) >> 23) - 127)));
        const float up = __uint_as_float((uint32_t)(e + 127) << 23);
#pragma unroll
        for (int i = 0; i < D / 32; ++i) {
            const __half q = __float2half_rn(x[i] * up);
            const float r = x[i] * up - __half2float(q);
            s_q[h * QP + lane + 32 * i] = q;
            s_q[(8 + h) * QP + lane + 32 * i] = __float2half_rn(r * 16777216.f);
        }
        if (lane == 0) s_qs[h] = a.scale / up;
    }
    __syncthreads();
    const float qs = s_qs[g];

    float o[VC * 16][4];
#pragma unroll
    for (int i = 0; i < VC * 16; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    // head g: largest score and the sum of e^(s - m_s) (this lane's tokens); the weights' reference e^r_s 2^r_e, a score and a whole number
    float m_s = -1.0e30f, l = 0.f, r_s = -1.0e30f, r_e = 0.f;
    bool bad = false;
    const size_t tok_bytes = D;
    // 16 tokens' place in the pools; false: not mapped
    auto place = [&](int tok, size_t& at) {
        const int page = bt[tok / a.page_tokens];
        if (page < 0 || page >= a.num_pages) { bad = true; return false; }
        at = ((size_t)page * a.Hkv + kvh) * a.page_tokens + tok % a.page_tokens;
        return true;
    };
    uint4 kr[2][KC];
    float ksc[4], vsc[4];
    size_t at = 0;
    bool have = false;
    auto load_k = [&](int tok) {                     // the next run's keys and row scales
        have = tok < end && place(tok, at);
        if (!have) return;
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int j = 0; j < KC; ++j) kr[n][j] = __ldg(reinterpret_cast<const uint4*>(a.k_pool + (at + 8 * n + g) * tok_bytes + 64 * j + 16 * t));
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const float2 k2 = __ldg(reinterpret_cast<const float2*>(a.k_scale + at + 8 * n + 2 * t)), v2 = __ldg(reinterpret_cast<const float2*>(a.v_scale + at + 8 * n + 2 * t));
            ksc[2 * n] = k2.x; ksc[2 * n + 1] = k2.y; vsc[2 * n] = v2.x; vsc[2 * n + 1] = v2.y;
        }
    };
    // Adds the accumulators (both terms of the weights) to the lane's sums in shared memory, times `f` and `e`, and clears them.  The
    // tensor core drops what falls below an accumulator's last bit, so no more than kF8Chain products are added to one.
    float kept = 0.f;                                // factor of the sums in shared memory to the present reference
    float* mine = s_acc[warp] + lane;
    auto flush = [&](float f, float e) {
#pragma unroll
        for (int i = 0; i < VC * 16; ++i) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                float* p = mine + 32 * (2 * i + x);
                *p = ((kept > 0.f ? *p * kept : 0.f) + (o[i][x] + o[i][x + 2])) * f * e;
            }
            o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
        }
        kept = 1.f;
    };
    int runs = 0;
    int tok = begin + kF8Tok * warp;
    load_k(tok);
    for (; tok < end; tok += kF8Tok * kF8Warps) {
        const bool live = have;                      // warp-uniform
        uint4 vr[4][VC];
        float s[4], lv[4], fv[4];
        if (live) {
            // tokens 2t, 2t + 1, 2t + 8, 2t + 9 of the run
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int i = 0; i < VC; ++i)
                    vr[n][i] = __ldg(reinterpret_cast<const uint4*>(a.v_pool + (at + 2 * t + (n & 1) + 8 * (n >> 1)) * tok_bytes + 128 * i + 16 * g));
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < KC; ++j) {
                float c[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const __half* q = s_q + g * QP + 64 * j + 16 * t + 4 * i;
                    const uint2 qa = *reinterpret_cast<const uint2*>(q);
                    const uint2 qb = *reinterpret_cast<const uint2*>(q + 8 * QP);
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        const uint32_t w = i == 0 ? kr[n][j].x : i == 1 ? kr[n][j].y : i == 2 ? kr[n][j].z : kr[n][j].w;
                        mma_f16(c[n], qa.x, qb.x, qa.y, qb.y, e4m3x2_to_f16x2(w), e4m3x2_to_f16x2(w >> 16));
                    }
                }
#pragma unroll
                for (int n = 0; n < 4; ++n) sum[n] += fmaf(1.f / 16777216.f, c[n >> 1][2 + (n & 1)], c[n >> 1][n & 1]);
            }
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                s[n] = sum[n] * (qs * ksc[n]);
                const int e = max(-126, min(126, (int)((__float_as_uint(vsc[n]) >> 23) & 255u) - 127));
                lv[n] = (float)e;
                fv[n] = vsc[n] * __uint_as_float((uint32_t)(127 - e) << 23);
            }
        }
        const int first = tok;
        load_k(tok + kF8Tok * kF8Warps);
        if (!live) continue;
        if (first + kF8Tok > end) {                  // the run's last tokens are not there: no weight, and no codes that could be NaN
#pragma unroll
            for (int n = 0; n < 4; ++n)
                if (first + 2 * t + (n & 1) + 8 * (n >> 1) >= end) {
                    s[n] = -INFINITY; lv[n] = fv[n] = 0.f;
#pragma unroll
                    for (int i = 0; i < VC; ++i) vr[n][i] = make_uint4(0, 0, 0, 0);
                }
        }
        // exponents of the weights: differences of scores and of whole numbers first, so that what is rounded is small where a weight is
        // near the largest
        float x[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) x[n] = fmaf(s[n] - r_s, kLog2e, lv[n] - r_e);
        float ms = fmaxf(fmaxf(s[0], s[1]), fmaxf(s[2], s[3])), top = fmaxf(fmaxf(x[0], x[1]), fmaxf(x[2], x[3]));
#pragma unroll
        for (int d = 1; d <= 2; d <<= 1) {
            ms = fmaxf(ms, __shfl_xor_sync(0xffffffffu, ms, d));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
        }
        ms = fmaxf(m_s, ms);
        l *= f8_ex2((m_s - ms) * kLog2e);
        m_s = ms;
        const bool up = top > 0.f;
        if (__any_sync(0xffffffffu, up)) {           // a weight above the reference
            top = fmaxf(fmaxf(fmaf(s[0] - ms, kLog2e, lv[0]), fmaf(s[1] - ms, kLog2e, lv[1])), fmaxf(fmaf(s[2] - ms, kLog2e, lv[2]), fmaf(s[3] - ms, kLog2e, lv[3])));
#pragma unroll
            for (int d = 1; d <= 2; d <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, d));
            float alpha = 1.f;
            if (up) {
                const float e = ceilf(top);
                alpha = f8_ex2(fmaf(r_s - ms, kLog2e, r_e - e));
                r_s = ms; r_e = e;
                kept *= alpha;
#pragma unroll
                for (int n = 0; n < 4; ++n) x[n] = fmaf(s[n] - r_s, kLog2e, lv[n] - r_e);
            }
#pragma unroll
            for (int i = 0; i < VC * 16; ++i) { o[i][0] *= alpha; o[i][1] *= alpha; o[i][2] *= alpha; o[i][3] *= alpha; }
        }
        __half hi[4], lo[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) {
            l += f8_ex2((s[n] - m_s) * kLog2e);
            const float w = f8_ex2(x[n]) * (fv[n] * kTop);
            hi[n] = __float2half_rn(w);
            lo[n] = __float2half_rn(w - __half2float(hi[n]));
        }
        const uint32_t a0 = f16x2_bits(hi[0], hi[1]), a1 = f16x2_bits(lo[0], lo[1]), a2 = f16x2_bits(hi[2], hi[3]), a3 = f16x2_bits(lo[2], lo[3]);
#pragma unroll
        for (int i = 0; i < VC; ++i) {
            const uint32_t v0[4] = {vr[0][i].x, vr[0][i].y, vr[0][i].z, vr[0][i].w}, v1[4] = {vr[1][i].x, vr[1][i].y, vr[1][i].z, vr[1][i].w};
            const uint32_t v2[4] = {vr[2][i].x, vr[2][i].y, vr[2][i].z, vr[2][i].w}, v3[4] = {vr[3][i].x, vr[3][i].y, vr[3][i].z, vr[3][i].w};
#pragma unroll
            for (int w = 0; w < 4; ++w)
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    // bytes 2p and 2p + 1 of both tokens, interleaved
                    const uint32_t x = __byte_perm(v0[w], v1[w], p ? 0x7362 : 0x5140), y = __byte_perm(v2[w], v3[w], p ? 0x7362 : 0x5140);
                    mma_f16(o[16 * i + 4 * w + 2 * p], a0, a1, a2, a3, e4m3x2_to_f16x2(x), e4m3x2_to_f16x2(y));
                    mma_f16(o[16 * i + 4 * w + 2 * p + 1], a0, a1, a2, a3, e4m3x2_to_f16x2(x >> 16), e4m3x2_to_f16x2(y >> 16));
                }
        }
        if (++runs == kF8Chain) { flush(1.f, 1.f); runs = 0; }
    }
    if (bad) set_status(a.status, PS_DEV_BAD_INDEX);
    // ---- this warp's sums, on the reference of the scores
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    const float f = l > 0.f ? f8_ex2((r_s - m_s) * kLog2e) / kTop : 0.f, fe = r_e < -126.f ? 0.f : __uint_as_float((uint32_t)((int)r_e + 127) << 23);
    flush(f, fe);
    if (t == 0) { s_m[warp][g] = m_s; s_l[warp][g] = l; }
    __syncthreads();
    // ---- the four warps' sums, in warp order: a lane's head and four neighbouring dimensions at a time
    if (g >= G) return;
    float c[kF8Warps], m = s_m[0][g], sum = 0.f;
#pragma unroll
    for (int w = 1; w < kF8Warps; ++w) m = fmaxf(m, s_m[w][g]);
#pragma unroll
    for (int w = 0; w < kF8Warps; ++w) { c[w] = f8_ex2((s_m[w][g] - m) * kLog2e); sum = fmaf(c[w], s_l[w][g], sum); }
    const size_t idx = ((size_t)row * a.Hq + kvh * G + g) * a.max_splits + split;
    for (int q = warp; q < VC * 8; q += kF8Warps) {
        const int i = 4 * (q >> 1), x = q & 1;       // product columns 2t + x of accumulators i .. i + 3
        float v[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < kF8Warps; ++w)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = fmaf(c[w], s_acc[w][32 * (2 * (i + j) + x) + lane], v[j]);
        *reinterpret_cast<float4*>(a.part_acc + idx * D + 128 * (i >> 4) + 32 * t + 16 * x + (i & 15)) = make_float4(v[0], v[1], v[2], v[3]);
    }
    if (warp == 0 && t == 0) { a.part_ml[2 * idx] = sum > 0.f ? m : -3.0e38f; a.part_ml[2 * idx + 1] = sum; }
}

}  // namespace ps

// Whether ps_attn_decode_fp8 serves a geometry: pages of whole 16-token runs, splits of whole runs.
PS_API int ps_attn_decode_fp8_ok(int Hq, int Hkv, int D, int page_tokens, int split_tokens) {
    return (D == 128 || D == 256) && Hkv > 0 && Hq % Hkv == 0 && Hq / Hkv <= 8 && page_tokens > 0 && page_tokens % 16 == 0 && split_tokens % 16 == 0;
}

// Partials of rows [rows, Hq, D] over FP8-E4M3 pages, for ps_paged_attention_merge.
PS_API int ps_attn_decode_fp8(const void* q, const void* k_pool, const void* v_pool, const void* k_scale, const void* v_scale,
                              const void* block_table, int max_blocks, int page_tokens, int num_pages, const void* row_slot, const void* row_pos,
                              int rows, int Hq, int Hkv, int D, float sm_scale, int split_tokens, int max_splits, int max_visible, void* part_acc,
                              void* part_ml, void* status, cudaStream_t stream) {
    using namespace ps;
    if (!ps_attn_decode_fp8_ok(Hq, Hkv, D, page_tokens, split_tokens) || rows <= 0 || rows > 65535 || ((uintptr_t)k_pool | (uintptr_t)v_pool) % 16)
        return (int)cudaErrorInvalidValue;
    AttnFp8Args a;
    a.q = (const __nv_bfloat16*)q; a.k_pool = (const uint8_t*)k_pool; a.v_pool = (const uint8_t*)v_pool; a.k_scale = (const float*)k_scale;
    a.v_scale = (const float*)v_scale; a.block_table = (const int*)block_table; a.max_blocks = max_blocks; a.page_tokens = page_tokens;
    a.num_pages = num_pages; a.row_slot = (const int*)row_slot; a.row_pos = (const int*)row_pos; a.Hq = Hq; a.Hkv = Hkv;
    a.scale = sm_scale; a.split_tokens = split_tokens; a.max_splits = max_splits; a.part_acc = (float*)part_acc;
    a.part_ml = (float*)part_ml; a.status = (uint32_t*)status;
    int n_splits = (max_visible + split_tokens - 1) / split_tokens;
    if (n_splits < 1) n_splits = 1;
    if (n_splits > max_splits) return (int)cudaErrorInvalidValue;
    const dim3 grid(n_splits, Hkv, rows);
    return D == 256 ? launch_pdl(attn_fp8_decode_kernel<256>, grid, dim3(kF8Threads), 0, stream, a)
                    : launch_pdl(attn_fp8_decode_kernel<128>, grid, dim3(kF8Threads), 0, stream, a);
}
