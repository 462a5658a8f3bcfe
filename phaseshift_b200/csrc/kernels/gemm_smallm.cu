// Batched-decode GEMM (2 <= M <= 64 rows) on resident bf16 weights: out[M,N] = epilogue(A[M,K] . W[N,K]^T).
//
// In this regime the problem is a stream over W.  The operands are swapped relative to the prefill GEMM:
// 128 WEIGHT rows are the M side of `tcgen05.mma` and the few batch rows the N side (16, 32 or 64), so every
// byte a TMA stage brings into shared memory is weight data (16 KB per stage, ~100 KB in flight per CTA, two
// CTAs per SM).  K is split across CTAs so that even N = 5120 yields a few hundred CTAs; each writes fp32
// partial sums [split, M, N] and a second tiny kernel adds the splits in a fixed order (deterministic) and
// applies the residual / SwiGLU / dtype epilogue.  Accumulators live in tensor memory; epilogue warps read
// them with `tcgen05.ld` (lane = weight row, column = batch row), so the partial stores are coalesced.
// The tensor core drops what falls below an accumulator's last bit, so the error grows with the number of products added to one
// accumulator: a CTA with more than kSmRun k-iterations keeps two, one for either half of its run of K, and adds them in 32 bits (shorter
// runs do with one: with two, 8 rows took 0.15 us longer per product).  With one accumulator a run of 80
// k-iterations (34816 x 5120) was 5.6e-6 off 64 bits, one of 20 (18432 x 2560) 1.3e-6; with two 2.7e-6 and 6.0e-7.
// All mbarrier waits are bounded; a timeout sets PS_DEV_WAIT_TIMEOUT, frees the tensor memory and returns.
//
// A decoding step is a chain of about five such products per layer, 3 to 15 us of weights each, so what lies between them counts: all
// kernels here are launched programmatically, the product asks for its first 128 KB of weights per SM before its rows exist, and the
// reduction of a residual product norms the rows for the next one (gemm_smallm_norm_kernel).
// May a product that starts early hold what its predecessors need?  It takes up to 128 columns of tensor memory and 97 KB; a predecessor
// that wants more than what is left (512 columns or 200 KB: attention, CTA-pair and block-scaled GEMMs) has it before it lets its
// successors start, or fills the SM by its shared memory, so that both are never resident together.
//
// The reference serves this regime with its RowBlock2/4/8 WMMA kernels (src/phaseshift/models/qwen35/
// kernels/optimized/linear/psq4.hip:221-349); here it runs from a bf16 expansion that 180 GB of HBM can
// afford to keep resident next to the block-quantised weights.
#include "ps_tcgen05.cuh"

namespace ps {

constexpr int kSmBM = 128, kSmBK = 64, kSmThreads = 192, kSmRun = 8;

struct SmallMArgs {
    int M, N, K;
    int nb;                 // MMA N: batch rows padded to 16 / 32 / 64
    int x_box_rows;         // rows fetched per X tile (multiple of 8)
    int iters_per_split;    // k-iterations (of 64) per split
    int splits;
    float* partial;         // [splits, M, ld] fp32
    int ld;
    uint32_t* status;
    long long budget;       // clock-cycle budget of every mbarrier wait
};

template <int STAGES>
__global__ void __launch_bounds__(kSmThreads, 2)
gemm_smallm_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const SmallMArgs g) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    constexpr int kWBytes = kSmBM * kSmBK * 2;                 // 16 KB of weights per stage
    const int x_tile_bytes = g.nb * kSmBK * 2;                  // smem footprint of the X tile (all nb rows)
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char* sW = smem;
    unsigned char* sX = smem + STAGES * kWBytes;                // each X stage is 64 rows x 128 B = 8 KB apart
    constexpr int kXStride = 64 * kSmBK * 2;
    __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int s_abort, s_issued, s_consumed;      // stages handed to TMA / waited for by the MMA thread

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile_n = blockIdx.x, split = blockIdx.y;
    const int total_iters = (g.K + kSmBK - 1) / kSmBK;
    const int it0 = split * g.iters_per_split;
    const int k_iters = min(g.iters_per_split, total_iters - it0);
    const int x_bytes = g.x_box_rows * kSmBK * 2;
    // k-iterations of the first accumulator; the rest go to the second, which runs of up to kSmRun do without
    const int first_run = k_iters > kSmRun ? (k_iters + 1) / 2 : k_iters;
    const uint32_t acc_cols = g.nb <= 32 ? 32 : 64;

    cudaTriggerProgrammaticLaunchCompletion();
    // rows of the X tile beyond the fetched box must read as zero
    for (int i = threadIdx.x; i < STAGES * kXStride / 16; i += kSmThreads) reinterpret_cast<uint4*>(sX)[i] = make_uint4(0, 0, 0, 0);
    tc::fence_proxy_async_smem();
    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { tc::mbar_init(&full_bar[s], 1); tc::mbar_init(&empty_bar[s], 1); }
        tc::mbar_init(&acc_bar, 1);
        tc::fence_barrier_init();
        s_abort = 0; s_issued = 0; s_consumed = 0;
        tc::tma_prefetch_desc(&map_w);
        tc::tma_prefetch_desc(&map_x);
    }
    if (warp == 1) {
        tc::tmem_alloc(&tmem_base_slot, 2 * acc_cols);        // two accumulators of up to 64 fp32 columns x 128 lanes
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem_acc = tmem_base_slot;
    (void)x_tile_bytes;

    if (warp == 0) {
        if (k_iters > 0 && tc::elect_one()) {
            // the first weights are on their way before the kernel that writes the rows is done
            const int early = min(k_iters, STAGES);
            for (int it = 0; it < early; ++it) {
                tc::mbar_expect_tx(&full_bar[it], kWBytes + x_bytes);
                tc::tma_load_2d(sW + it * kWBytes, &map_w, (it0 + it) * kSmBK, tile_n * kSmBM, &full_bar[it]);
            }
            cudaGridDependencySynchronize();
            for (int it = 0; it < k_iters; ++it) {
                const int s = it % STAGES;
                if (it >= STAGES) {
                    if (!tc::mbar_wait(&empty_bar[s], ((uint32_t)(it / STAGES) & 1u) ^ 1u, g.budget)) { atomicExch(&s_abort, 1); break; }
                    tc::mbar_expect_tx(&full_bar[s], kWBytes + x_bytes);
                    tc::tma_load_2d(sW + s * kWBytes, &map_w, (it0 + it) * kSmBK, tile_n * kSmBM, &full_bar[s]);
                }
                tc::tma_load_2d(sX + s * kXStride, &map_x, (it0 + it) * kSmBK, 0, &full_bar[s]);
                s_issued = it + 1;
            }
        }
    } else if (warp == 1) {
        if (tc::elect_one()) {
            const uint32_t idesc = tc::idesc_bf16_f32(kSmBM, g.nb);
            bool ok = true;
            cudaGridDependencySynchronize();             // the waits below are for this kernel's copies, not for its predecessor
            for (int it = 0; it < k_iters && ok; ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                if (!tc::mbar_wait(&full_bar[s], ph, g.budget)) { atomicExch(&s_abort, 1); ok = false; break; }
                s_consumed = it + 1;
                tc::fence_after_sync();
                const uint32_t w_addr = tc::smem_u32(sW + s * kWBytes), x_addr = tc::smem_u32(sX + s * kXStride);
                const uint32_t acc = it < first_run ? tmem_acc : tmem_acc + acc_cols;
                const bool begun = it > 0 && it != first_run;
#pragma unroll
                for (int kk = 0; kk < kSmBK / 16; ++kk)
                    tc::mma_bf16_ss(acc, tc::smem_desc_sw128(w_addr + kk * 32), tc::smem_desc_sw128(x_addr + kk * 32), idesc,
                                    (begun || kk > 0) ? 1u : 0u);
                tc::mma_commit(&empty_bar[s]);
            }
            tc::mma_commit(&acc_bar);
        }
    } else {
        // epilogue warps 2..5 -> TMEM lane quadrant (warp % 4); lane = weight row, column = batch row
        cudaGridDependencySynchronize();                 // the previous product's sums have been read
        const int quad = warp & 3;
        const bool done = k_iters > 0 ? tc::mbar_wait(&acc_bar, 0, g.budget) : true;
        tc::fence_after_sync();
        const int n = tile_n * kSmBM + quad * 32 + lane;
        if (done && s_abort == 0) {
            float* dst = g.partial + (size_t)split * g.M * g.ld;
            for (int c0 = 0; c0 < g.nb; c0 += 32) {
                uint32_t r[32];
                const uint32_t at = tmem_acc + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0;
                if (k_iters > first_run) {
                    uint32_t q[32];
                    tc::tmem_ld_32x32(at, r);
                    tc::tmem_ld_32x32(at + acc_cols, q);
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(q[j]));
                } else if (k_iters > 0) {
                    tc::tmem_ld_32x32(at, r);
                    tc::tmem_ld_wait();
                } else {
#pragma unroll
                    for (int j = 0; j < 32; ++j) r[j] = 0u;
                }
                if (n < g.N) {
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (c0 + j < g.M) dst[(size_t)(c0 + j) * g.ld + n] = __uint_as_float(r[j]);
                }
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (s_abort != 0 && threadIdx.x == 0) {
        set_status(g.status, PS_DEV_WAIT_TIMEOUT);
        // copies still in flight get a bounded chance to land before the shared memory goes back to the next CTA
        const long long b = g.budget < 4000000ll ? g.budget : 4000000ll;
        for (int c = s_consumed; c < s_issued; ++c) tc::mbar_wait(&full_bar[c % STAGES], (uint32_t)((c / STAGES) & 1), b);
    }
    __syncthreads();
    if (warp == 1) {
        tc::fence_after_sync();
        tc::tmem_dealloc(tmem_acc, 2 * acc_cols);
    }
}

struct SmallMReduceArgs {
    const float* partial; int splits, M, N;
    int epilogue;            // 0 store, 1 residual, 2 / 3 / 5 SwiGLU / ReGLU / GeGLU on interleaved (gate, up) columns, 4 tanh-gelu
    const __nv_bfloat16* residual; int ld_res;
    void* out; int ldo; int out_f32;
    const __nv_bfloat16* norm_w; float eps; __nv_bfloat16* normed; int ld_normed;      // gemm_smallm_norm_kernel
};

// Sum of the splits of four neighbouring columns (c a multiple of 4) of row m, in ascending order; F loads in flight (their latency is
// most of a reduction: with four, fourteen splits took four round trips to L2).
template <int F>
__device__ __forceinline__ float4 smallm_sum4(const SmallMReduceArgs& a, int m, int c) {
    const float4* p = reinterpret_cast<const float4*>(a.partial + (size_t)m * a.N + c);
    const size_t step = (size_t)a.M * a.N / 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s = 0; s < a.splits; s += F) {
        float4 q[F];
#pragma unroll
        for (int i = 0; i < F; ++i) if (s + i < a.splits) q[i] = p[(s + i) * step];
#pragma unroll
        for (int i = 0; i < F; ++i) if (s + i < a.splits) { v.x += q[i].x; v.y += q[i].y; v.z += q[i].z; v.w += q[i].w; }
    }
    return v;
}
__device__ __forceinline__ float smallm_gated(const SmallMReduceArgs& a, float g, float u) {
    const float gt = bf16_to_f32(f32_to_bf16(g)), up = bf16_to_f32(f32_to_bf16(u));
    return (a.epilogue == 3 ? fmaxf(gt, 0.f) : a.epilogue == 5 ? gelu_tanh_f(gt) : silu_f(gt)) * up;
}

// One thread per four output columns (N a multiple of 4, rows of `out` and the residual 16- / 8-byte aligned).
template <int F>
__global__ void gemm_smallm_reduce4_kernel(const SmallMReduceArgs a) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int quads = a.N >> 2;
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= a.M * quads) return;
    const int m = id / quads, c = (id - m * quads) * 4;
    float4 v = smallm_sum4<F>(a, m, c);
    if (a.epilogue == 2 || a.epilogue == 3 || a.epilogue == 5) {
        *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)m * a.ldo + (c >> 1)) =
            f32x2_to_bf16x2_bits(smallm_gated(a, v.x, v.y), smallm_gated(a, v.z, v.w));
        return;
    }
    if (a.epilogue == 1) {
        const uint2 rb = *reinterpret_cast<const uint2*>(a.residual + (size_t)m * a.ld_res + c);
        const float2 r0 = bf16x2_bits_to_f32x2(rb.x), r1 = bf16x2_bits_to_f32x2(rb.y);
        v.x = bf16_to_f32(f32_to_bf16(v.x)) + r0.x; v.y = bf16_to_f32(f32_to_bf16(v.y)) + r0.y;
        v.z = bf16_to_f32(f32_to_bf16(v.z)) + r1.x; v.w = bf16_to_f32(f32_to_bf16(v.w)) + r1.y;
    }
    if (a.epilogue == 4) { v.x = gelu_tanh_f(v.x); v.y = gelu_tanh_f(v.y); v.z = gelu_tanh_f(v.z); v.w = gelu_tanh_f(v.w); }
    if (a.out_f32) *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + (size_t)m * a.ldo + c) = v;
    else *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)m * a.ldo + c) =
        make_uint2(f32x2_to_bf16x2_bits(v.x, v.y), f32x2_to_bf16x2_bits(v.z, v.w));
}

// Residual epilogue and the next projection's RMSNorm (scale 1 + w) in one launch: the four CTAs of a cluster share a row, exchange
// their sums of squares through distributed shared memory and write the new residual and its normed row.  Replaces a reduction
// and a norm launch (2.9 + 6.5 us for 8 rows of 2560); with the early weights above, a step of 8 rows through 8 layers of 2560 x 9216
// went from 1190 to 931 us, one of 32 rows through 4 layers of 5120 x 17408 from 2010 to 1780.  What bounds it: latency.  The sums are
// written to the others instead of read from them: no CTA has to stay for a last cluster barrier (8 rows of 2560: 4.4 -> 4.3 us).
constexpr int kSmNormCtas = 4, kSmNormThreads = 256, kSmNormItems = 4;       // rows of up to 4 * 4 * 4 * 256 columns
__global__ void __cluster_dims__(kSmNormCtas, 1, 1) __launch_bounds__(kSmNormThreads) gemm_smallm_norm_kernel(const SmallMReduceArgs a) {
    __shared__ float red[32], s_part[kSmNormCtas];
    tc::cluster_arrive();            // (the others have started when they are written to)
    const int m = blockIdx.x / kSmNormCtas, per = (a.N / 4 + kSmNormCtas - 1) / kSmNormCtas;
    const uint32_t rank = tc::cluster_ctarank();
    const int first = (int)rank * per, last = min(first + per, a.N / 4);         // this CTA's groups of four columns
    cudaTriggerProgrammaticLaunchCompletion();
    uint2 w[kSmNormItems];
#pragma unroll
    for (int j = 0; j < kSmNormItems; ++j) {
        const int i = first + threadIdx.x + j * kSmNormThreads;
        w[j] = i < last ? __ldg(reinterpret_cast<const uint2*>(a.norm_w) + i) : make_uint2(0, 0);
    }
    cudaGridDependencySynchronize();
    float4 x[kSmNormItems];
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < kSmNormItems; ++j) {
        const int i = first + threadIdx.x + j * kSmNormThreads, c = 4 * i;
        x[j] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i >= last) continue;
        const float4 v = smallm_sum4<8>(a, m, c);
        const uint2 rb = *reinterpret_cast<const uint2*>(a.residual + (size_t)m * a.ld_res + c);
        const float2 r0 = bf16x2_bits_to_f32x2(rb.x), r1 = bf16x2_bits_to_f32x2(rb.y);
        const uint2 o = make_uint2(f32x2_to_bf16x2_bits(bf16_to_f32(f32_to_bf16(v.x)) + r0.x, bf16_to_f32(f32_to_bf16(v.y)) + r0.y),
                                   f32x2_to_bf16x2_bits(bf16_to_f32(f32_to_bf16(v.z)) + r1.x, bf16_to_f32(f32_to_bf16(v.w)) + r1.y));
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)m * a.ldo + c) = o;
        const float2 x0 = bf16x2_bits_to_f32x2(o.x), x1 = bf16x2_bits_to_f32x2(o.y);
        x[j] = make_float4(x0.x, x0.y, x1.x, x1.y);
        ss += x0.x * x0.x + x0.y * x0.y + x1.x * x1.x + x1.y * x1.y;
    }
    ss = block_sum(ss, red);
    // every CTA puts its sum into all of them, so that nobody reads from one that may have left
    tc::cluster_wait();
    if (threadIdx.x < kSmNormCtas) tc::cluster_store_f32(&s_part[rank], threadIdx.x, ss);
    tc::cluster_sync();
    ss = 0.f;
#pragma unroll
    for (int r = 0; r < kSmNormCtas; ++r) ss += s_part[r];
    const float inv = rsqrtf(ss / (float)a.N + a.eps);
#pragma unroll
    for (int j = 0; j < kSmNormItems; ++j) {
        const int i = first + threadIdx.x + j * kSmNormThreads;
        if (i >= last) continue;
        const float2 w0 = bf16x2_bits_to_f32x2(w[j].x), w1 = bf16x2_bits_to_f32x2(w[j].y);
        *reinterpret_cast<uint2*>(a.normed + (size_t)m * a.ld_normed + 4 * i) =
            make_uint2(f32x2_to_bf16x2_bits(x[j].x * inv * (1.f + w0.x), x[j].y * inv * (1.f + w0.y)),
                       f32x2_to_bf16x2_bits(x[j].z * inv * (1.f + w1.x), x[j].w * inv * (1.f + w1.y)));
    }
}

// Any even N and any alignment: one thread per output pair (two neighbouring columns); splits are added in ascending order.
__global__ void gemm_smallm_reduce_kernel(const SmallMReduceArgs a) {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    const int pairs = a.N >> 1;
    const long long id = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= (long long)a.M * pairs) return;
    const int m = (int)(id / pairs), c = (int)(id % pairs) * 2;
    float v0 = 0.f, v1 = 0.f;
    for (int s = 0; s < a.splits; ++s) {
        const float2 p = *reinterpret_cast<const float2*>(a.partial + ((size_t)s * a.M + m) * a.N + c);
        v0 += p.x; v1 += p.y;
    }
    if (a.epilogue == 2 || a.epilogue == 3 || a.epilogue == 5) {
        reinterpret_cast<__nv_bfloat16*>(a.out)[(size_t)m * a.ldo + (c >> 1)] = f32_to_bf16(smallm_gated(a, v0, v1));
        return;
    }
    if (a.epilogue == 1) {
        const float2 rs = bf16x2_bits_to_f32x2(*reinterpret_cast<const uint32_t*>(a.residual + (size_t)m * a.ld_res + c));
        v0 = bf16_to_f32(f32_to_bf16(v0)) + rs.x;
        v1 = bf16_to_f32(f32_to_bf16(v1)) + rs.y;
    }
    if (a.epilogue == 4) { v0 = gelu_tanh_f(v0); v1 = gelu_tanh_f(v1); }
    if (a.out_f32) *reinterpret_cast<float2*>(reinterpret_cast<float*>(a.out) + (size_t)m * a.ldo + c) = make_float2(v0, v1);
    else *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(a.out) + (size_t)m * a.ldo + c) = f32x2_to_bf16x2_bits(v0, v1);
}

typedef CUresult (*SmEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static SmEncodeFn sm_encode_fn() {
    static SmEncodeFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<SmEncodeFn>(p);
    }
    return fn;
}

static int sm_map_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
    SmEncodeFn enc = sm_encode_fn();
    if (enc == nullptr) return (int)cudaErrorNotSupported;
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kSmBK, box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS
               ? 0 : (int)cudaErrorInvalidValue;
}

}  // namespace ps

// Number of K splits the launcher will use (the caller sizes `partial` = splits * M * N floats with it).
PS_API int ps_gemm_smallm_splits(int N, int K) {
    const int tiles = (N + ps::kSmBM - 1) / ps::kSmBM;
    const int iters = (K + ps::kSmBK - 1) / ps::kSmBK;
    // as many CTAs as fit at once, two on each SM (296 here): a few more than that and the step waits for a second round of them (with
    // the count rounded up instead, 18432 x 2560 ran as 432 CTAs and 2560 x 9216 as 300: steps of 8, 12 and 32 rows took 858, 983 and
    // 1456 us, with this rule 797, 922 and 1384)
    int splits = 2 * ps::sm_count() / tiles;
    const int max_splits = iters / 4 > 0 ? iters / 4 : 1;   // at least 4 k-iterations (64 KB of weights) per CTA
    if (splits > max_splits) splits = max_splits;
    if (splits < 1) splits = 1;
    if (splits > 16) splits = 16;
    const int per = (iters + splits - 1) / splits;
    return (iters + per - 1) / per;                         // drop empty trailing splits
}

// out[M,N] = epilogue(A[M,K] . W[N,K]^T) for 1 <= M <= 64; A, W bf16 row-major (lda, ldw multiples of 8,
// 16-byte aligned bases), N even, `partial` = ps_gemm_smallm_splits(N, K) * M * N floats of scratch (16-byte aligned; none for one
// run of K stored in 32 bits, whose sums are the output).
// With `norm_w` (residual epilogue, bf16 output): `normed` [M, N] bf16 receives out / rms(out) * (1 + norm_w) as well; N a multiple of
// 4, at most ps_gemm_smallm_norm_cols(), and 8-byte aligned rows of out, residual, norm_w and normed.
PS_API int ps_gemm_smallm_norm_cols() { return 16 * ps::kSmNormItems * ps::kSmNormThreads; }

PS_API int ps_gemm_smallm_normed(const void* a, int lda, const void* w, int ldw, int M, int N, int K, int epilogue, const void* residual,
                                 int ld_res, void* out, int ldo, int out_f32, const void* norm_w, float eps, void* normed, int ld_normed,
                                 void* partial, void* status, cudaStream_t stream) {
    using namespace ps;
    if (M < 1 || M > 64 || N <= 0 || (N & 1) || K <= 0 || (K % 8) || (lda % 8) || (ldw % 8) || ((uintptr_t)a % 16) ||
        ((uintptr_t)w % 16))
        return (int)cudaErrorInvalidValue;
    const bool gated = epilogue == 2 || epilogue == 3 || epilogue == 5;
    if (gated && out_f32) return (int)cudaErrorInvalidValue;
    auto rows8 = [](const void* p, int ld) { return (uintptr_t)p % 8 == 0 && ld % 4 == 0; };       // bf16 rows in 8-byte pieces
    if (norm_w != nullptr && (epilogue != 1 || out_f32 || N % 4 || N > ps_gemm_smallm_norm_cols() || (uintptr_t)norm_w % 8 || !rows8(out, ldo) ||
                              !rows8(residual, ld_res) || !rows8(normed, ld_normed)))
        return (int)cudaErrorInvalidValue;
    SmallMArgs g;
    g.M = M; g.N = N; g.K = K;
    g.nb = M <= 16 ? 16 : (M <= 32 ? 32 : 64);
    g.x_box_rows = (M + 7) / 8 * 8;
    g.splits = ps_gemm_smallm_splits(N, K);
    const int iters = (K + kSmBK - 1) / kSmBK;
    g.iters_per_split = (iters + g.splits - 1) / g.splits;
    const bool direct = g.splits == 1 && epilogue == 0 && out_f32;
    if (!direct && partial == nullptr) return (int)cudaErrorInvalidValue;
    g.partial = direct ? (float*)out : (float*)partial; g.ld = direct ? ldo : N; g.status = (uint32_t*)status; g.budget = g_ps_wait_budget_cycles;
    CUtensorMap map_w, map_x;
    int err = sm_map_2d(&map_w, w, (uint64_t)N, (uint64_t)K, (uint64_t)ldw, kSmBM);
    if (err) return err;
    err = sm_map_2d(&map_x, a, (uint64_t)M, (uint64_t)K, (uint64_t)lda, (uint32_t)g.x_box_rows);
    if (err) return err;
    constexpr int STAGES = 4;
    const size_t smem = (size_t)STAGES * (kSmBM * kSmBK * 2 + 64 * kSmBK * 2) + 1024;       // 4 x 24 KB + alignment slack
    static bool attr_set = false;
    if (!attr_set) {
        cudaFuncSetAttribute(gemm_smallm_kernel<STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(gemm_smallm_kernel<STAGES>, cudaFuncAttributePreferredSharedMemoryCarveout, (int)cudaSharedmemCarveoutMaxShared);
        attr_set = true;
    }
    dim3 grid((N + kSmBM - 1) / kSmBM, g.splits);
    err = launch_pdl(gemm_smallm_kernel<STAGES>, grid, dim3(kSmThreads), smem, stream, map_w, map_x, g);
    if (err || direct) return err;
    SmallMReduceArgs r;
    r.partial = g.partial; r.splits = g.splits; r.M = M; r.N = N; r.epilogue = epilogue;
    r.residual = (const __nv_bfloat16*)residual; r.ld_res = ld_res; r.out = out; r.ldo = ldo; r.out_f32 = out_f32;
    r.norm_w = (const __nv_bfloat16*)norm_w; r.eps = eps; r.normed = (__nv_bfloat16*)normed; r.ld_normed = ld_normed;
    if (norm_w != nullptr) return launch_pdl(gemm_smallm_norm_kernel, dim3(M * kSmNormCtas), dim3(kSmNormThreads), 0, stream, r);
    // With more than two CTAs for an SM, registers for loads that no split has cost occupancy (two splits, 34816 x 5120, 24 / 64 rows: room for eight
    // 120.3 / 133.5 us, for two 116.8 / 129.4; three splits, 12352 x 2560, 32 rows: 13.85 and, for four, 13.58; 16 rows: 12.97 and 13.18).
    const int ctas = (M * (N >> 2) + 255) / 256, f = ctas <= 2 * sm_count() || g.splits > 4 ? 8 : g.splits > 2 ? 4 : 2;
    if (N % 4 == 0 && (uintptr_t)partial % 16 == 0 && (epilogue != 1 || rows8(residual, ld_res)) &&
        (gated ? (uintptr_t)out % 4 == 0 && ldo % 2 == 0 : out_f32 ? (uintptr_t)out % 16 == 0 && ldo % 4 == 0 : rows8(out, ldo)))
        return launch_pdl(f == 2 ? gemm_smallm_reduce4_kernel<2> : f == 4 ? gemm_smallm_reduce4_kernel<4> : gemm_smallm_reduce4_kernel<8>,
                          dim3((unsigned)ctas), dim3(256), 0, stream, r);
    const long long n = (long long)M * (N >> 1);
    return launch_pdl(gemm_smallm_reduce_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, r);
}
