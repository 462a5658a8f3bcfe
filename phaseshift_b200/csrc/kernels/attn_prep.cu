// Fused attention prepare: per-head RMSNorm(1+w) on q and k, partial NeoX RoPE, and the paged
// KV append (BF16, FP8-E4M3 with one f32 scale per token x kv-head, or NVFP4 rows as laid out in kv_fp4.cuh), in one launch.
//
// The reference runs these as separate dispatches (split, two per-group RMSNorms, RoPE pair
// kernel with an f64 inv_freq table, kv_append; src/phaseshift/models/qwen35/kernels/optimized/
// attention/rope.hip:130-251, kv_append.hip:98-148).  Here a warp owns a (row, head): the
// normalised, rotated q is written to the dense q buffer, k/v go straight into their page.
//
// Layouts
//   qkv      [rows, ld_qkv] bf16: per q-head h: [2hD, 2hD+D) = q, [2hD+D, 2hD+2D) = gate;
//            then k heads at q_span + hk*D, then v heads at q_span + Hkv*D + hk*D.
//   q_out    [rows, Hq, D] bf16
//   k/v pool [num_pages, Hkv, page_tokens, D] (bf16 or e4m3) or [num_pages, Hkv, page_tokens, kv_fp4_row_bytes(D)] bytes
//            (NVFP4, kv_fp8 == 2), scales [num_pages, Hkv, page_tokens] f32
//   block_table [num_slots, max_blocks] int32; row_slot/row_pos give each row's sequence slot and position.
#include "kv_fp4.cuh"

namespace ps {

struct AttnPrepArgs {
    const __nv_bfloat16* qkv; int ld_qkv;
    int rows, Hq, Hkv, D, rotary_dim;
    const __nv_bfloat16* q_norm_w; const __nv_bfloat16* k_norm_w; float eps;
    const double* inv_freq;            // [rotary_dim/2]
    const int* row_slot; const int* row_pos;
    __nv_bfloat16* q_out;
    void* k_pool; void* v_pool; float* k_scale; float* v_scale;
    const int* block_table; int max_blocks; int page_tokens; int num_pages; int kv_fp8;
    uint32_t* status;
    int pairs;                         // rows of qkv take 4-byte loads
    int wide;                          // the queries and the pools take 4-byte stores
};

// Two neighbouring values rounded to bf16 at element `at`, which is even.
__device__ __forceinline__ void prep_store2(__nv_bfloat16* dst, int at, float x, float y, int wide) {
    if (wide) *reinterpret_cast<uint32_t*>(dst + at) = f32x2_to_bf16x2_bits(x, y);
    else { dst[at] = f32_to_bf16(x); dst[at + 1] = f32_to_bf16(y); }
}

// grid = (CTAs per row, rows), block = 8 warps; a warp takes whole heads of the row, one after the other.  The row's rotation angles --
// 64-bit sines and cosines, the same for every head -- are computed once per CTA: computed per head, as before, they were most of the
// kernel (2048 rows of 16 + 8 heads: 56 us, now 39, which is latency: a row's chain of loads, norm and turn).  D <= 512.
constexpr int kPrepWarps = 8, kPrepMaxD = 512;
__global__ void __launch_bounds__(kPrepWarps * 32) attn_prep_kernel(const AttnPrepArgs a) {
    extern __shared__ __align__(16) double s_turn[];               // [rotary_dim / 2][2]: cosine, sine
    __shared__ __align__(16) float s_vals[kPrepWarps][kPrepMaxD];       // float2 accesses
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int row = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, D = a.D, half = a.rotary_dim / 2;
    const int q_span = 2 * a.Hq * D, heads = a.Hq + 2 * a.Hkv;
    const int pos = a.row_pos[row], slot = a.row_slot[row];
    for (int i = threadIdx.x; i < half; i += kPrepWarps * 32) {
        double s, c;
        sincos((double)pos * a.inv_freq[i], &s, &c);
        s_turn[2 * i] = c; s_turn[2 * i + 1] = s;
    }
    // the row's place in the pools (a padding row of a row bucket has none: only its queries are written)
    int page = -1;
    if (slot >= 0) {
        const int blk = pos / a.page_tokens;
        if (pos >= 0 && blk < a.max_blocks) page = a.block_table[(size_t)slot * a.max_blocks + blk];
        if (page < 0 || page >= a.num_pages) { page = -1; if (threadIdx.x == 0 && blockIdx.x == 0) set_status(a.status, PS_DEV_BAD_INDEX); }
    }
    const int off = pos % a.page_tokens;
    __syncthreads();
    float* vals = s_vals[warp];
    for (int hh = blockIdx.x * kPrepWarps + warp; hh < heads; hh += gridDim.x * kPrepWarps) {
        const int kind = hh < a.Hq ? 0 : hh < a.Hq + a.Hkv ? 1 : 2;          // q, k, v
        const int head = kind == 0 ? hh : kind == 1 ? hh - a.Hq : hh - a.Hq - a.Hkv;
        const __nv_bfloat16* src = a.qkv + (size_t)row * a.ld_qkv + (kind == 0 ? 2 * head * D : q_span + (kind == 1 ? head : a.Hkv + head) * D);
        if (kind != 0 && page < 0) continue;
        float x[kPrepMaxD / 64][2], ss = 0.f;
#pragma unroll
        for (int j = 0; j < kPrepMaxD / 64; ++j) {
            const int d = 2 * lane + 64 * j;
            x[j][0] = x[j][1] = 0.f;
            if (d < D) {
                const float2 f = a.pairs ? bf16x2_bits_to_f32x2(*reinterpret_cast<const uint32_t*>(src + d)) : make_float2(bf16_to_f32(src[d]), bf16_to_f32(src[d + 1]));
                x[j][0] = f.x; x[j][1] = f.y;
                ss += f.x * f.x + f.y * f.y;
            }
        }
        if (kind != 2) {
            const float ir = rsqrtf(warp_sum(ss) / (float)D + a.eps);
            const __nv_bfloat16* w = kind == 0 ? a.q_norm_w : a.k_norm_w;
#pragma unroll
            for (int j = 0; j < kPrepMaxD / 64; ++j) {
                const int d = 2 * lane + 64 * j;
                if (d < D) { x[j][0] = x[j][0] * ir * (1.f + bf16_to_f32(w[d])); x[j][1] = x[j][1] * ir * (1.f + bf16_to_f32(w[d + 1])); }
            }
        }
        __syncwarp();                                                        // the previous head's values have been read
#pragma unroll
        for (int j = 0; j < kPrepMaxD / 64; ++j)
            if (2 * lane + 64 * j < D) *reinterpret_cast<float2*>(vals + 2 * lane + 64 * j) = make_float2(x[j][0], x[j][1]);
        __syncwarp();
        if (kind != 2)
            // NeoX half-rotate on the first rotary_dim dims: (x[i], x[i + half]) turned by pos * inv_freq[i]
            for (int i = lane; i < half; i += 32) {
                const double c = s_turn[2 * i], s = s_turn[2 * i + 1];
                const float lo = vals[i], hi = vals[i + half];
                vals[i] = (float)((double)lo * c - (double)hi * s);
                vals[i + half] = (float)((double)hi * c + (double)lo * s);
            }
        __syncwarp();
        if (kind == 0) {
            __nv_bfloat16* dst = a.q_out + ((size_t)row * a.Hq + head) * D;
            for (int d = 2 * lane; d < D; d += 64) prep_store2(dst, d, vals[d], vals[d + 1], a.wide);
            continue;
        }
        const size_t tok = ((size_t)page * a.Hkv + head) * a.page_tokens + off;
        void* pool = kind == 1 ? a.k_pool : a.v_pool;
        if (!a.kv_fp8) {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(pool) + tok * D;
            for (int d = 2 * lane; d < D; d += 64) prep_store2(dst, d, vals[d], vals[d + 1], a.wide);
            continue;
        }
        // coded rows: K after bf16 rounding of the turned value, V as given; the row's scale from its maximum
        float amax = 0.f;
        for (int d = lane; d < D; d += 32) { const float y = bf16_to_f32(f32_to_bf16(vals[d])); vals[d] = y; amax = fmaxf(amax, fabsf(y)); }
        amax = warp_max(amax);
        __syncwarp();
        float* scale = (kind == 1 ? a.k_scale : a.v_scale) + tok;
        if (a.kv_fp8 == 2) {
            const float ts = kv_fp4_token_scale(amax);
            uint8_t* dst = reinterpret_cast<uint8_t*>(pool) + tok * kv_fp4_row_bytes(D);
            for (int b = lane; b < D / 16; b += 32) {
                uint2 codes; uint8_t sf;
                kv_fp4_quant16(vals + 16 * b, ts, codes, sf);
                *reinterpret_cast<uint2*>(dst + 8 * b) = codes;
                dst[D / 2 + b] = sf;
            }
            if (lane == 0) *scale = ts;
        } else {
            const float sc = amax > 0.f ? amax / 448.f : 1.f, inv = 1.f / sc;
            uint8_t* dst = reinterpret_cast<uint8_t*>(pool) + tok * D;
            for (int d = 4 * lane; d < D; d += 128) {
                uint32_t w = 0;
#pragma unroll
                for (int e = 0; e < 4; ++e) w |= (uint32_t)f32_to_e4m3(vals[d + e] * inv) << (8 * e);
                if (a.wide) *reinterpret_cast<uint32_t*>(dst + d) = w;
                else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) dst[d + e] = (uint8_t)(w >> (8 * e));
                }
            }
            if (lane == 0) *scale = sc;
        }
    }
}

}  // namespace ps

PS_API int ps_attn_prep(const void* qkv, int ld_qkv, int rows, int Hq, int Hkv, int D, int rotary_dim,
                        const void* q_norm_w, const void* k_norm_w, float eps, const void* inv_freq,
                        const void* row_slot, const void* row_pos, void* q_out, void* k_pool, void* v_pool,
                        void* k_scale, void* v_scale, const void* block_table, int max_blocks, int page_tokens,
                        int num_pages, int kv_fp8, void* status, cudaStream_t stream) {
    using namespace ps;
    if (D > 512 || (D & 63) || rotary_dim > D || rows <= 0) return (int)cudaErrorInvalidValue;
    AttnPrepArgs a;
    a.qkv = (const __nv_bfloat16*)qkv; a.ld_qkv = ld_qkv; a.rows = rows; a.Hq = Hq; a.Hkv = Hkv; a.D = D;
    a.rotary_dim = rotary_dim; a.q_norm_w = (const __nv_bfloat16*)q_norm_w; a.k_norm_w = (const __nv_bfloat16*)k_norm_w;
    a.eps = eps; a.inv_freq = (const double*)inv_freq; a.row_slot = (const int*)row_slot; a.row_pos = (const int*)row_pos;
    a.q_out = (__nv_bfloat16*)q_out; a.k_pool = k_pool; a.v_pool = v_pool; a.k_scale = (float*)k_scale;
    a.v_scale = (float*)v_scale; a.block_table = (const int*)block_table; a.max_blocks = max_blocks;
    a.page_tokens = page_tokens; a.num_pages = num_pages; a.kv_fp8 = kv_fp8; a.status = (uint32_t*)status;
    a.pairs = ld_qkv % 2 == 0 && (uintptr_t)qkv % 4 == 0;
    a.wide = ((uintptr_t)q_out | (uintptr_t)k_pool | (uintptr_t)v_pool) % 4 == 0;
    // many rows: one CTA per row; few: the heads over several, so that the row does not wait for its warps' second round
    const int ctas = rows >= 64 ? 1 : (Hq + 2 * Hkv + kPrepWarps - 1) / kPrepWarps;
    return launch_pdl(attn_prep_kernel, dim3(ctas, rows), dim3(kPrepWarps * 32), (size_t)rotary_dim * sizeof(double), stream, a);
}
