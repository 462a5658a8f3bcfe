// Gated DeltaNet, row-sequential form: one launch covers the whole mixer between in_proj and out_proj.
//
// Per (sequence, value head) CTA, for each of the sequence's rows in order:
//   causal depthwise conv (kernel 4) + SiLU on this head's q/k/v channels, L2-normalise q (scaled by
//   Dk^-0.5) and k, beta = sigmoid(b), d = exp(-exp(A_log) * softplus(a + dt_bias)),
//   kv = (d S)^T k, delta = (v - kv) beta, S = d S + k (x) delta, o = S^T q,
//   out = RMSNorm_direct(o; w) * SiLU(z)  -> bf16.
// The fp32 state tile S[Dk, Dv] lives in registers for the whole launch, so decode reads and writes the
// state exactly once.  The reference spreads this over conv1d, silu, l2-normalise, scale, recurrence,
// per-group RMSNorm, silu and mul dispatches (src/phaseshift/models/qwen35/model/lower_to_primitives.cpp:
// 704-808; math in kernels/correctness/detail/gdn.inc:5-166).
//
// A row's arithmetic never depends on how many rows the launch carries, so verifying 1+K speculative
// rows reproduces K+1 single-row decodes bit for bit (the job of the reference's decode_rows_exact
// kernels, gdn/recurrence.hip:922-1190).  For speculative rollback the launch can write the new state
// to a second buffer and log (k, delta, d) per row; `ps_gdn_replay` re-applies an accepted prefix of
// that log to the untouched old state (the reference's compact-log commit, recurrence.hip:812-920).
//
// Conv history: [slots, Hv, ring, 2*Dk + Dv] bf16, slot (pos % ring) holds the pre-conv input of
// position pos.  Each value head keeps a private copy of its key head's q/k channels, so CTAs never
// share history and no ordering between them is needed; rolling back is just re-using an older pos.
#include "ps_common.cuh"

namespace ps {

struct GdnSeqDesc { int row_start; int n_rows; int slot; int pos_start; };

struct GdnArgs {
    const __nv_bfloat16* proj; int ld_proj;     // [rows, ld]: [q(Hk*Dk) | k(Hk*Dk) | v(Hv*Dv) | z(Hv*Dv) | b(Hv) | a(Hv)]
    int Hk, Hv;
    const __nv_bfloat16* conv_w;                // [2*Hk*Dk + Hv*Dv, 4]; tap 3 multiplies the current input
    const float* A_log; const float* dt_bias;   // [Hv]
    const __nv_bfloat16* norm_w; float eps;     // [Dv]
    __nv_bfloat16* conv_state; int ring;
    const float* state_in; float* state_out;    // [slots, Hv, Dk, Dv]
    const GdnSeqDesc* seqs;
    __nv_bfloat16* out;                         // [rows, Hv*Dv]
    float* log_k; float* log_delta; float* log_d;   // optional: [rows, Hv, Dk], [rows, Hv, Dv], [rows, Hv]
    // optional in-kernel beta/decay projections: b = xn . ba_w[h], a = xn . ba_w[Hv + h] (bf16 weights);
    // when null the kernel reads b and a from `proj`
    const __nv_bfloat16* ba_w; const __nv_bfloat16* xn; int ba_k;
    int max_rows;                               // sequences with more rows in this step belong to the chunked kernels
};

// Sums over a CTA's warps: what warp_sum gives of the warps' sums in the first lanes (absent ones are 0).
__device__ __forceinline__ float gdn_sum4(const float* p) { return (p[0] + p[2]) + (p[1] + p[3]); }
__device__ __forceinline__ float gdn_sum8(const float* p) { return ((p[0] + p[4]) + (p[2] + p[6])) + ((p[1] + p[5]) + (p[3] + p[7])); }

// A CTA is a chain of loads, sums and barriers, most of it latency; with many sequences the chip holds two CTAs per SM and a launch
// takes as many such chains as there are rounds of them.  So what the predecessor has not written -- state, history, weights -- is
// loaded before the wait for it, a thread keeps its channels' convolution in registers, and three barriers are left of eight: after the
// channels and the warps' sums, after the pass over the state, after Delta.  One row through 32 heads of 128: 11.2 -> 7.7 us, 12
// sequences 21.3 -> 14.7; 32 sequences through 48 heads 63 -> 42.7 (the state alone, read and written once, takes 31 of measured).
template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) gdn_rows_kernel(const GdnArgs a) {
    constexpr int CG = DV / 4;          // column groups of 4 consecutive columns
    constexpr int RG = 256 / CG;        // row groups
    constexpr int R = DK / RG;          // rows per thread
    constexpr int CH = 2 * DK + DV;     // conv channels owned by this head
    constexpr int NC = (CH + 255) / 256, G = DK / 32;
    static_assert(2 * DK <= 256 && G <= 4 && DV <= 128, "a warp holds 32 channels of q or of k");
    __shared__ float s_q[DK], s_k[DK], s_v[DV], s_sum[5][8], s_ss[4];     // sums of the warps: q.q, k.k, b, a, q.k; o.o
    __shared__ __align__(16) float s_part[RG][DV], s_partq[RG][DV];      // float4 accesses
    __shared__ __align__(16) float s_vec[DV];

    const int h = blockIdx.x;
    const GdnSeqDesc sd = a.seqs[blockIdx.y];
    if (sd.n_rows <= 0 || sd.n_rows > a.max_rows) return;
    PS_CHECK(PS_SLOT_OK(sd.slot) && PS_ROWS_OK(sd.row_start, sd.n_rows) && sd.pos_start >= 0);
    const int hk = h / (a.Hv / a.Hk);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, cg = t % CG, rg = t / CG;
    const int q_off = hk * DK, k_off = a.Hk * DK + hk * DK, v_off = 2 * a.Hk * DK + h * DV;
    const int z_off = 2 * a.Hk * DK + a.Hv * DV + h * DV;
    const int b_off = 2 * a.Hk * DK + 2 * a.Hv * DV + h, a_off = b_off + a.Hv;

    cudaTriggerProgrammaticLaunchCompletion();
    // ---- what was last written by an earlier step, not by the stream predecessor
    float S[R][4];
    {
        const float* sp = a.state_in + ((size_t)sd.slot * a.Hv + h) * DK * DV;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(sp + (size_t)(rg + RG * r) * DV + cg * 4);
            S[r][0] = v.x; S[r][1] = v.y; S[r][2] = v.z; S[r][3] = v.w;
        }
    }
    __nv_bfloat16* hist = a.conv_state + ((size_t)sd.slot * a.Hv + h) * a.ring * CH;
    uint2 taps[NC];                      // the channel's four weights
    __nv_bfloat16 past[NC][3];           // x_{t-1}, x_{t-2}, x_{t-3}
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const int c = t + 256 * n;
        taps[n] = make_uint2(0u, 0u);
#pragma unroll
        for (int j = 0; j < 3; ++j) past[n][j] = __float2bfloat16(0.f);
        if (c < CH) {
            const int gc = c < DK ? q_off + c : (c < 2 * DK ? k_off + (c - DK) : v_off + (c - 2 * DK));
            taps[n] = __ldg(reinterpret_cast<const uint2*>(a.conv_w + (size_t)gc * 4));
#pragma unroll
            for (int j = 1; j <= 3; ++j)
                if (sd.pos_start - j >= 0) past[n][j - 1] = hist[(size_t)((sd.pos_start - j) % a.ring) * CH + c];
        }
    }
    const float neg_expA = -__expf(a.A_log[h]);
    const float dtb = a.dt_bias[h];
    const float nw = t < DV ? bf16_to_f32(a.norm_w[t]) : 0.f;
    if (t < 8) { s_sum[0][t] = s_sum[1][t] = s_sum[4][t] = 0.f; }
    if (t < 4) s_ss[t] = 0.f;
    __syncthreads();
    cudaGridDependencySynchronize();

    for (int r_i = 0; r_i < sd.n_rows; ++r_i) {
        const int row = sd.row_start + r_i, pos = sd.pos_start + r_i;
        const __nv_bfloat16* pr = a.proj + (size_t)row * a.ld_proj;
        __nv_bfloat16 x[NC];
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int c = t + 256 * n, gc = c < DK ? q_off + c : (c < 2 * DK ? k_off + (c - DK) : v_off + (c - 2 * DK));
            x[n] = c < CH ? pr[gc] : __float2bfloat16(0.f);
        }
        const __nv_bfloat16 zb = t < DV ? pr[z_off + t] : __float2bfloat16(0.f);
        float b_in = 0.f, a_in = 0.f;
        if (a.ba_w == nullptr) { b_in = bf16_to_f32(pr[b_off]); a_in = bf16_to_f32(pr[a_off]); }
        else {
            // beta / decay input projections
            const __nv_bfloat16* xr = a.xn + (size_t)row * a.ba_k;
            const __nv_bfloat16* wb = a.ba_w + (size_t)h * a.ba_k;
            const __nv_bfloat16* wa = a.ba_w + (size_t)(a.Hv + h) * a.ba_k;
            float sb = 0.f, sa = 0.f;
            for (int i = t * 2; i < a.ba_k; i += 512) {
                const float2 xv = bf16x2_bits_to_f32x2(*reinterpret_cast<const uint32_t*>(xr + i));
                const float2 bv = bf16x2_bits_to_f32x2(__ldg(reinterpret_cast<const uint32_t*>(wb + i)));
                const float2 av = bf16x2_bits_to_f32x2(__ldg(reinterpret_cast<const uint32_t*>(wa + i)));
                sb = fmaf(xv.x, bv.x, sb); sb = fmaf(xv.y, bv.y, sb);
                sa = fmaf(xv.x, av.x, sa); sa = fmaf(xv.y, av.y, sa);
            }
            sb = warp_sum(sb); sa = warp_sum(sa);
            if (lane == 0) { s_sum[2][warp] = sb; s_sum[3][warp] = sa; }
        }
        // ---- conv + SiLU for this thread's channels, whose history nobody else reads
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int c = t + 256 * n;
            const float2 w01 = bf16x2_bits_to_f32x2(taps[n].x), w23 = bf16x2_bits_to_f32x2(taps[n].y);
            float y = w01.x * bf16_to_f32(past[n][2]);
            y = fmaf(w01.y, bf16_to_f32(past[n][1]), y);
            y = fmaf(w23.x, bf16_to_f32(past[n][0]), y);
            y = fmaf(w23.y, bf16_to_f32(x[n]), y);
            y = silu_f(y);
            past[n][2] = past[n][1]; past[n][1] = past[n][0]; past[n][0] = x[n];
            if (c < CH) {
                hist[(size_t)(pos % a.ring) * CH + c] = x[n];
                if (c < DK) s_q[c] = y; else if (c < 2 * DK) s_k[c - DK] = y; else s_v[c - 2 * DK] = y;
            }
            if (n == 0 && warp < 2 * G) {
                const float sq = warp_sum(y * y);
                if (lane == 0) s_sum[warp < G ? 0 : 1][warp < G ? warp : warp - G] = sq;
            }
        }
        __syncthreads();
        if (t < DK) {
            const float qk = warp_sum(s_q[t] * s_k[t]);               // (read after the next barrier)
            if (lane == 0) s_sum[4][warp] = qk;
        }
        const float qn = rsqrtf(gdn_sum4(s_sum[0]) + 1e-6f) * rsqrtf((float)DK);
        const float kn = rsqrtf(gdn_sum4(s_sum[1]) + 1e-6f);
        if (a.ba_w != nullptr) { b_in = bf16_to_f32(f32_to_bf16(gdn_sum8(s_sum[2]))); a_in = bf16_to_f32(f32_to_bf16(gdn_sum8(s_sum[3]))); }
        const float beta = sigmoid_f(b_in);
        const float gate = neg_expA * softplus_f(a_in + dtb);
        const float d = __expf(gate);
        // ---- one pass over the state: S <- d S, partial sums of S^T k and S^T q (both of the decayed old state)
        float kreg[R], qreg[R];
#pragma unroll
        for (int r = 0; r < R; ++r) { kreg[r] = s_k[rg + RG * r] * kn; qreg[r] = s_q[rg + RG * r] * qn; }
        float p[4] = {0.f, 0.f, 0.f, 0.f}, pq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int c = 0; c < 4; ++c) { S[r][c] *= d; p[c] = fmaf(S[r][c], kreg[r], p[c]); pq[c] = fmaf(S[r][c], qreg[r], pq[c]); }
        }
        *reinterpret_cast<float4*>(&s_part[rg][cg * 4]) = make_float4(p[0], p[1], p[2], p[3]);
        *reinterpret_cast<float4*>(&s_partq[rg][cg * 4]) = make_float4(pq[0], pq[1], pq[2], pq[3]);
        if (a.log_k) {
            for (int i = t; i < DK; i += 256) a.log_k[((size_t)row * a.Hv + h) * DK + i] = s_k[i] * kn;
            if (t == 0) a.log_d[(size_t)row * a.Hv + h] = d;
        }
        __syncthreads();
        // delta = beta (v - S^T k);  o = S_new^T q = S^T q + (k.q) delta   with S_new = S + k delta^T
        float ov = 0.f;
        if (t < DV) {
            float kv = 0.f, qv = 0.f;
#pragma unroll
            for (int g = 0; g < RG; ++g) { kv += s_part[g][t]; qv += s_partq[g][t]; }
            const float kq = gdn_sum4(s_sum[4]) * qn * kn;            // k . q of the normalised vectors
            const float delta = (s_v[t] - kv) * beta;
            s_vec[t] = delta;
            ov = fmaf(kq, delta, qv);
            if (a.log_delta) a.log_delta[((size_t)row * a.Hv + h) * DV + t] = delta;
            const float sq = warp_sum(ov * ov);
            if (lane == 0) s_ss[warp] = sq;
        }
        __syncthreads();
        if (t < DV) {
            const float inv = rsqrtf(gdn_sum4(s_ss) / (float)DV + a.eps);
            const float y = ov * inv * nw;
            a.out[(size_t)row * (a.Hv * DV) + h * DV + t] = f32_to_bf16(y * silu_f(bf16_to_f32(zb)));
        }
        // ---- S += k (x) delta (registers only)
        {
            const float4 dl = *reinterpret_cast<const float4*>(&s_vec[cg * 4]);
            const float dlr[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int c = 0; c < 4; ++c) S[r][c] = fmaf(kreg[r], dlr[c], S[r][c]);
            }
        }
        if (r_i + 1 < sd.n_rows) __syncthreads();      // the row's vectors and sums are rewritten by the next one
    }
    {
        float* sp = a.state_out + ((size_t)sd.slot * a.Hv + h) * DK * DV;
#pragma unroll
        for (int r = 0; r < R; ++r)
            *reinterpret_cast<float4*>(sp + (size_t)(rg + RG * r) * DV + cg * 4) =
                make_float4(S[r][0], S[r][1], S[r][2], S[r][3]);
    }
}

// The same for sequences with several rows in the step (the rows of a drafted block, short prompts): what does not depend on the state --
// convolution, norms, gates -- is prepared for eight rows at once, a warp per row, and the head norm and the gate follow for all eight;
// between them a row costs the pass over the state and two barriers instead of four.  Every sum is formed in the order of the kernel
// above, so rows have the same bits in both.  A single row takes longer here, hence two kernels.  Eight rows through 32 heads of 128:
// 21.3 -> 13.8 us with all rows' inputs and gates in flight together (a thread per channel before: a chain of loads for each row).
constexpr int kManyRows = 8;
template <int DK, int DV>
__global__ void __launch_bounds__(256, 2) gdn_rows_many_kernel(const GdnArgs a) {
    constexpr int CG = DV / 4, RG = 256 / CG, R = DK / RG, CH = 2 * DK + DV, NC = (CH + 255) / 256;
    static_assert(DK % 32 == 0 && DV % 32 == 0, "a warp sums a row's channels in whole groups of 32");
    __shared__ float s_qk[kManyRows][2 * DK], s_v[kManyRows][DV], s_o[kManyRows][DV];
    __shared__ float s_row[kManyRows][5];                                // factors of q and k, k . q, beta, decay
    __shared__ float s_ba[kManyRows][2][8];                              // beta and decay projections: sums of the warps
    __shared__ __align__(16) float s_part[RG][DV], s_partq[RG][DV];      // float4 accesses
    __shared__ __align__(16) float s_vec[DV];

    const int h = blockIdx.x;
    const GdnSeqDesc sd = a.seqs[blockIdx.y];
    if (sd.n_rows <= 0 || sd.n_rows > a.max_rows) return;
    PS_CHECK(PS_SLOT_OK(sd.slot) && PS_ROWS_OK(sd.row_start, sd.n_rows) && sd.pos_start >= 0);
    const int hk = h / (a.Hv / a.Hk);
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31, cg = t % CG, rg = t / CG;
    const int q_off = hk * DK, k_off = a.Hk * DK + hk * DK, v_off = 2 * a.Hk * DK + h * DV;
    const int z_off = 2 * a.Hk * DK + a.Hv * DV + h * DV;
    const int b_off = 2 * a.Hk * DK + 2 * a.Hv * DV + h, a_off = b_off + a.Hv;

    cudaTriggerProgrammaticLaunchCompletion();
    float S[R][4];
    {
        // the recurrent state was last written by an earlier step, not by the stream predecessor
        const float* sp = a.state_in + ((size_t)sd.slot * a.Hv + h) * DK * DV;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float4 v = *reinterpret_cast<const float4*>(sp + (size_t)(rg + RG * r) * DV + cg * 4);
            S[r][0] = v.x; S[r][1] = v.y; S[r][2] = v.z; S[r][3] = v.w;
        }
    }
    auto channel = [&](int c) { return c < DK ? q_off + c : (c < 2 * DK ? k_off + (c - DK) : v_off + (c - 2 * DK)); };
    __nv_bfloat16* hist = a.conv_state + ((size_t)sd.slot * a.Hv + h) * a.ring * CH;
    uint2 taps[NC];                      // the four weights of this thread's channels
    __nv_bfloat16 past[NC][3];           // x_{t-1}, x_{t-2}, x_{t-3}
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const int c = t + 256 * n;
        taps[n] = c < CH ? __ldg(reinterpret_cast<const uint2*>(a.conv_w + (size_t)channel(c) * 4)) : make_uint2(0u, 0u);
#pragma unroll
        for (int j = 1; j <= 3; ++j)
            past[n][j - 1] = c < CH && sd.pos_start - j >= 0 ? hist[(size_t)((sd.pos_start - j) % a.ring) * CH + c] : __float2bfloat16(0.f);
    }
    cudaGridDependencySynchronize();
    const float neg_expA = -__expf(a.A_log[h]);
    const float dtb = a.dt_bias[h];

    for (int first = 0; first < sd.n_rows; first += kManyRows) {
        const int nb = min(kManyRows, sd.n_rows - first);
        if (a.ba_w != nullptr) {
            // beta / decay input projections of all rows at once: a thread has its columns' weights for every row (a warp per row read them
            // row by row, 5120 columns of two rows of weights in 80 round trips: eight rows through 48 heads 30.8 us, 16.8 now; four 27.3 and 12.4)
            const __nv_bfloat16* xr = a.xn + (size_t)(sd.row_start + first) * a.ba_k;
            const __nv_bfloat16* wb = a.ba_w + (size_t)h * a.ba_k;
            const __nv_bfloat16* wa = a.ba_w + (size_t)(a.Hv + h) * a.ba_k;
            float sb[kManyRows] = {}, sa[kManyRows] = {};
            for (int i = t * 2; i < a.ba_k; i += 512) {
                const float2 bv = bf16x2_bits_to_f32x2(__ldg(reinterpret_cast<const uint32_t*>(wb + i)));
                const float2 av = bf16x2_bits_to_f32x2(__ldg(reinterpret_cast<const uint32_t*>(wa + i)));
                uint32_t x2[kManyRows];
#pragma unroll
                for (int r = 0; r < kManyRows; ++r) x2[r] = r < nb ? *reinterpret_cast<const uint32_t*>(xr + (size_t)r * a.ba_k + i) : 0u;
#pragma unroll
                for (int r = 0; r < kManyRows; ++r) {
                    const float2 xv = bf16x2_bits_to_f32x2(x2[r]);
                    sb[r] = fmaf(xv.x, bv.x, sb[r]); sb[r] = fmaf(xv.y, bv.y, sb[r]);
                    sa[r] = fmaf(xv.x, av.x, sa[r]); sa[r] = fmaf(xv.y, av.y, sa[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < kManyRows; ++r) {
                if (r >= nb) break;
                const float b_w = warp_sum(sb[r]), a_w = warp_sum(sa[r]);
                if (lane == 0) { s_ba[r][0][warp] = b_w; s_ba[r][1][warp] = a_w; }
            }
        }
        // ---- conv + SiLU for this thread's channels, whose history nobody else reads: all rows' inputs are in flight together
        __nv_bfloat16 x[NC][kManyRows];
#pragma unroll
        for (int n = 0; n < NC; ++n)
#pragma unroll
            for (int r = 0; r < kManyRows; ++r) {
                const int c = t + 256 * n;
                x[n][r] = c < CH && r < nb ? a.proj[(size_t)(sd.row_start + first + r) * a.ld_proj + channel(c)] : __float2bfloat16(0.f);
            }
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int c = t + 256 * n;
            const float2 w01 = bf16x2_bits_to_f32x2(taps[n].x), w23 = bf16x2_bits_to_f32x2(taps[n].y);
#pragma unroll
            for (int r = 0; r < kManyRows; ++r) {
                float y = w01.x * bf16_to_f32(past[n][2]);
                y = fmaf(w01.y, bf16_to_f32(past[n][1]), y);
                y = fmaf(w23.x, bf16_to_f32(past[n][0]), y);
                y = fmaf(w23.y, bf16_to_f32(x[n][r]), y);
                y = silu_f(y);
                past[n][2] = past[n][1]; past[n][1] = past[n][0]; past[n][0] = x[n][r];
                if (c < CH && r < nb) {
                    if (c < 2 * DK) s_qk[r][c] = y; else s_v[r][c - 2 * DK] = y;
                    // history of the sequence's last rows
                    if (first + r + a.ring >= sd.n_rows) hist[(size_t)((sd.pos_start + first + r) % a.ring) * CH + c] = x[n][r];
                }
            }
        }
        __syncthreads();
        // ---- L2 norms, k.q, gates and (optionally) the beta / decay input projections of row `warp`
        if (warp < nb) {
            const int row = sd.row_start + first + warp;
            const __nv_bfloat16* pr = a.proj + (size_t)row * a.ld_proj;
            const float *q = s_qk[warp], *k = s_qk[warp] + DK;
            float part[5] = {0.f, 0.f, 0.f, 0.f, 0.f};                  // lane w: the sum of warp w of the kernel above
#pragma unroll
            for (int w = 0; w < DK / 32; ++w) {
                const float qv = q[32 * w + lane], kv = k[32 * w + lane];
                const float qq = warp_sum(qv * qv), kk = warp_sum(kv * kv), qk = warp_sum(qv * kv);
                if (lane == w) { part[0] = qq; part[1] = kk; part[4] = qk; }
            }
            if (a.ba_w != nullptr && lane < 8) { part[2] = s_ba[warp][0][lane]; part[3] = s_ba[warp][1][lane]; }
#pragma unroll
            for (int i = 0; i < 5; ++i) part[i] = warp_sum(part[i]);
            const float qn = rsqrtf(part[0] + 1e-6f) * rsqrtf((float)DK), kn = rsqrtf(part[1] + 1e-6f);
            const float b_in = a.ba_w != nullptr ? bf16_to_f32(f32_to_bf16(part[2])) : bf16_to_f32(pr[b_off]);
            const float a_in = a.ba_w != nullptr ? bf16_to_f32(f32_to_bf16(part[3])) : bf16_to_f32(pr[a_off]);
            const float gate = neg_expA * softplus_f(a_in + dtb), d = __expf(gate);
            if (lane == 0) { s_row[warp][0] = qn; s_row[warp][1] = kn; s_row[warp][2] = part[4] * qn * kn; s_row[warp][3] = sigmoid_f(b_in); s_row[warp][4] = d; }
            if (a.log_k) {
                for (int i = lane; i < DK; i += 32) a.log_k[((size_t)row * a.Hv + h) * DK + i] = k[i] * kn;
                if (lane == 0) a.log_d[(size_t)row * a.Hv + h] = d;
            }
        }
        __nv_bfloat16 z[DV / 32], nw[DV / 32];                          // of the head norm and gate of row `warp`
#pragma unroll
        for (int w = 0; w < DV / 32; ++w) {
            z[w] = warp < nb ? a.proj[(size_t)(sd.row_start + first + warp) * a.ld_proj + z_off + 32 * w + lane] : __float2bfloat16(0.f);
            nw[w] = a.norm_w[32 * w + lane];
        }
        __syncthreads();
        // ---- row after row: one pass over the state each
        for (int r = 0; r < nb; ++r) {
            const float qn = s_row[r][0], kn = s_row[r][1], kq = s_row[r][2], beta = s_row[r][3], d = s_row[r][4];
            float kreg[R], qreg[R];
#pragma unroll
            for (int j = 0; j < R; ++j) { kreg[j] = s_qk[r][DK + rg + RG * j] * kn; qreg[j] = s_qk[r][rg + RG * j] * qn; }
            float p[4] = {0.f, 0.f, 0.f, 0.f}, pq[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int j = 0; j < R; ++j) {
#pragma unroll
                for (int c = 0; c < 4; ++c) { S[j][c] *= d; p[c] = fmaf(S[j][c], kreg[j], p[c]); pq[c] = fmaf(S[j][c], qreg[j], pq[c]); }
            }
            *reinterpret_cast<float4*>(&s_part[rg][cg * 4]) = make_float4(p[0], p[1], p[2], p[3]);
            *reinterpret_cast<float4*>(&s_partq[rg][cg * 4]) = make_float4(pq[0], pq[1], pq[2], pq[3]);
            __syncthreads();
            if (t < DV) {
                float kv = 0.f, qv = 0.f;
#pragma unroll
                for (int g = 0; g < RG; ++g) { kv += s_part[g][t]; qv += s_partq[g][t]; }
                const float delta = (s_v[r][t] - kv) * beta;
                s_vec[t] = delta;
                s_o[r][t] = fmaf(kq, delta, qv);
                if (a.log_delta) a.log_delta[((size_t)(sd.row_start + first + r) * a.Hv + h) * DV + t] = delta;
            }
            __syncthreads();
            const float4 dl = *reinterpret_cast<const float4*>(&s_vec[cg * 4]);
            const float dlr[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
            for (int j = 0; j < R; ++j) {
#pragma unroll
                for (int c = 0; c < 4; ++c) S[j][c] = fmaf(kreg[j], dlr[c], S[j][c]);
            }
        }
        // ---- head norm and gate of row `warp`
        if (warp < nb) {
            const int row = sd.row_start + first + warp;
            float part = 0.f;
#pragma unroll
            for (int w = 0; w < DV / 32; ++w) {
                const float o = s_o[warp][32 * w + lane], sq = warp_sum(o * o);
                if (lane == w) part = sq;
            }
            const float inv = rsqrtf(warp_sum(part) / (float)DV + a.eps);
#pragma unroll
            for (int w = 0; w < DV / 32; ++w) {
                const int i = 32 * w + lane;
                const float y = s_o[warp][i] * inv * bf16_to_f32(nw[w]);
                a.out[(size_t)row * (a.Hv * DV) + h * DV + i] = f32_to_bf16(y * silu_f(bf16_to_f32(z[w])));
            }
        }
        __syncthreads();      // the rows' vectors are rewritten by the next ones
    }
    {
        float* sp = a.state_out + ((size_t)sd.slot * a.Hv + h) * DK * DV;
#pragma unroll
        for (int r = 0; r < R; ++r)
            *reinterpret_cast<float4*>(sp + (size_t)(rg + RG * r) * DV + cg * 4) =
                make_float4(S[r][0], S[r][1], S[r][2], S[r][3]);
    }
}

struct GdnReplayArgs {
    float* state; int Hv;            // [slots, Hv, Dk, Dv]: old state, updated in place
    const GdnSeqDesc* seqs;          // n_rows = number of accepted rows to re-apply
    const float* log_k; const float* log_delta; const float* log_d;
};

// Re-apply S = d S + k (x) delta for the accepted rows; same expression order as the forward pass.
template <int DK, int DV>
__global__ void __launch_bounds__(256) gdn_replay_kernel(const GdnReplayArgs a) {
    constexpr int CG = DV / 4, RG = 256 / CG, R = DK / RG;
    const int h = blockIdx.x;
    const GdnSeqDesc sd = a.seqs[blockIdx.y];
    if (sd.n_rows <= 0) return;
    PS_CHECK(PS_SLOT_OK(sd.slot) && PS_ROWS_OK(sd.row_start, sd.n_rows));
    const int t = threadIdx.x, cg = t % CG, rg = t / CG;
    float* sp = a.state + ((size_t)sd.slot * a.Hv + h) * DK * DV;
    float S[R][4];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float4 v = *reinterpret_cast<const float4*>(sp + (size_t)(rg + RG * r) * DV + cg * 4);
        S[r][0] = v.x; S[r][1] = v.y; S[r][2] = v.z; S[r][3] = v.w;
    }
    for (int r_i = 0; r_i < sd.n_rows; ++r_i) {
        const size_t rh = (size_t)(sd.row_start + r_i) * a.Hv + h;
        const float d = a.log_d[rh];
        const float4 dl = *reinterpret_cast<const float4*>(a.log_delta + rh * DV + cg * 4);
        const float dlr[4] = {dl.x, dl.y, dl.z, dl.w};
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const float k = a.log_k[rh * DK + rg + RG * r];
#pragma unroll
            for (int c = 0; c < 4; ++c) { S[r][c] *= d; S[r][c] = fmaf(k, dlr[c], S[r][c]); }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        *reinterpret_cast<float4*>(sp + (size_t)(rg + RG * r) * DV + cg * 4) = make_float4(S[r][0], S[r][1], S[r][2], S[r][3]);
}

}  // namespace ps

PS_DEFINE_LIMITS_SETTER(gdn_recurrent)

namespace ps {
static int gdn_rows(bool many, const void* proj, int ld_proj, int Hk, int Hv, int Dk, int Dv, const void* conv_w,
                       const void* A_log, const void* dt_bias, const void* norm_w, float eps, void* conv_state,
                       int ring, const void* state_in, void* state_out, const void* seqs, int n_seqs, void* out,
                       void* log_k, void* log_delta, void* log_d, const void* ba_w, const void* xn, int ba_k, int max_rows,
                       cudaStream_t stream) {
    if (n_seqs <= 0 || Hk <= 0 || (Hv % Hk) || ring < 4) return (int)cudaErrorInvalidValue;
    GdnArgs a;
    a.proj = (const __nv_bfloat16*)proj; a.ld_proj = ld_proj; a.Hk = Hk; a.Hv = Hv;
    a.conv_w = (const __nv_bfloat16*)conv_w; a.A_log = (const float*)A_log; a.dt_bias = (const float*)dt_bias;
    a.norm_w = (const __nv_bfloat16*)norm_w; a.eps = eps; a.conv_state = (__nv_bfloat16*)conv_state; a.ring = ring;
    a.state_in = (const float*)state_in; a.state_out = (float*)state_out; a.seqs = (const GdnSeqDesc*)seqs;
    a.out = (__nv_bfloat16*)out; a.log_k = (float*)log_k; a.log_delta = (float*)log_delta; a.log_d = (float*)log_d;
    a.ba_w = (const __nv_bfloat16*)ba_w; a.xn = (const __nv_bfloat16*)xn; a.ba_k = ba_k;
    a.max_rows = max_rows > 0 ? max_rows : 0x7fffffff;
    if (ba_w != nullptr && (ba_k & 1)) return (int)cudaErrorInvalidValue;
    dim3 grid(Hv, n_seqs);
    if (Dk == 128 && Dv == 128) return launch_pdl(many ? gdn_rows_many_kernel<128, 128> : gdn_rows_kernel<128, 128>, grid, dim3(256), 0, stream, a);
    if (Dk == 64 && Dv == 64) return launch_pdl(many ? gdn_rows_many_kernel<64, 64> : gdn_rows_kernel<64, 64>, grid, dim3(256), 0, stream, a);
    return (int)cudaErrorInvalidValue;
}
}  // namespace ps

// Contract of both entries: the kernel may load the recurrent state (`state_in`) and the convolution history (`conv_state`) of its slots,
// and the layer's weights, BEFORE its stream predecessor has finished (programmatic dependent launch).  Nothing that may still run
// then may write them.  A kernel between two launches on one slot is not enough to order them if it lets its successor start before it
// has waited itself, as the few-row GEMM and the streaming projection do; a copy, an ordinary launch, a kernel that waits first or the
// end of a graph is.  Inside the engine every step begins with the copy of its descriptors, or is a graph of its own, and has each
// layer's mixer once per slot.  A caller that runs two launches back to back puts one of these between them, or sets PS_PDL=0.
PS_API int ps_gdn_rows(const void* proj, int ld_proj, int Hk, int Hv, int Dk, int Dv, const void* conv_w,
                       const void* A_log, const void* dt_bias, const void* norm_w, float eps, void* conv_state,
                       int ring, const void* state_in, void* state_out, const void* seqs, int n_seqs, void* out,
                       void* log_k, void* log_delta, void* log_d, const void* ba_w, const void* xn, int ba_k, int max_rows,
                       cudaStream_t stream) {
    return ps::gdn_rows(false, proj, ld_proj, Hk, Hv, Dk, Dv, conv_w, A_log, dt_bias, norm_w, eps, conv_state, ring, state_in, state_out, seqs, n_seqs, out, log_k,
                        log_delta, log_d, ba_w, xn, ba_k, max_rows, stream);
}

// The same results and the same contract, sooner where sequences have several rows.
PS_API int ps_gdn_rows_many(const void* proj, int ld_proj, int Hk, int Hv, int Dk, int Dv, const void* conv_w,
                       const void* A_log, const void* dt_bias, const void* norm_w, float eps, void* conv_state,
                       int ring, const void* state_in, void* state_out, const void* seqs, int n_seqs, void* out,
                       void* log_k, void* log_delta, void* log_d, const void* ba_w, const void* xn, int ba_k, int max_rows,
                       cudaStream_t stream) {
    return ps::gdn_rows(true, proj, ld_proj, Hk, Hv, Dk, Dv, conv_w, A_log, dt_bias, norm_w, eps, conv_state, ring, state_in, state_out, seqs, n_seqs, out, log_k,
                        log_delta, log_d, ba_w, xn, ba_k, max_rows, stream);
}

PS_API int ps_gdn_replay(void* state, int Hv, int Dk, int Dv, const void* seqs, int n_seqs, const void* log_k,
                         const void* log_delta, const void* log_d, cudaStream_t stream) {
    using namespace ps;
    if (n_seqs <= 0) return (int)cudaErrorInvalidValue;
    GdnReplayArgs a;
    a.state = (float*)state; a.Hv = Hv; a.seqs = (const GdnSeqDesc*)seqs;
    a.log_k = (const float*)log_k; a.log_delta = (const float*)log_delta; a.log_d = (const float*)log_d;
    dim3 grid(Hv, n_seqs);
    if (Dk == 128 && Dv == 128) gdn_replay_kernel<128, 128><<<grid, 256, 0, stream>>>(a);
    else if (Dk == 64 && Dv == 64) gdn_replay_kernel<64, 64><<<grid, 256, 0, stream>>>(a);
    else return (int)cudaErrorInvalidValue;
    return PS_LAUNCH_CHECK();
}
