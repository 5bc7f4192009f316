// Shared expert (dense bf16 SwiGLU) and its sigmoid gate.
//
// Reference behaviour (src/models/qwen3_6/forward.rs:684-714 with the bf16 projection of
// :162-179, :727-742; device form src/infrastructure/cuda_linear.rs:391-450 and
// src/models/qwen3_6/forward_cudarc.rs:1541-1561):
//   ic1 = gate_up_s x            [2*SI]
//   ic2 = silu(ic1[:SI]) * ic1[SI:]
//   shared = down_s ic2          [H]
//   se_gate = sigmoid(x . shared_gate)
// f32 accumulation throughout.
#include "kernels.cuh"

namespace ftm {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kTokTile = 8;  // tokens per CTA, activations staged in shared memory as f32

// dot of one bf16 weight row with kTokTile activation rows held in shared memory
template <int NT>
__device__ __forceinline__ void row_dots(const __nv_bfloat16* __restrict__ wrow, const float* __restrict__ xs,
                                         int K, int lane, float (&acc)[NT]) {
#pragma unroll
    for (int t = 0; t < NT; t++) acc[t] = 0.f;
    for (int k = lane * 8; k < K; k += 32 * 8) {
        uint4 wv = *reinterpret_cast<const uint4*>(wrow + k);
        float w[8];
        float2 p;
        p = bf16x2_to_f32(wv.x); w[0] = p.x; w[1] = p.y;
        p = bf16x2_to_f32(wv.y); w[2] = p.x; w[3] = p.y;
        p = bf16x2_to_f32(wv.z); w[4] = p.x; w[5] = p.y;
        p = bf16x2_to_f32(wv.w); w[6] = p.x; w[7] = p.y;
#pragma unroll
        for (int t = 0; t < NT; t++) {
            const float4 a = *reinterpret_cast<const float4*>(xs + (size_t)t * K + k);
            const float4 b = *reinterpret_cast<const float4*>(xs + (size_t)t * K + k + 4);
            acc[t] += a.x * w[0] + a.y * w[1] + a.z * w[2] + a.w * w[3] + b.x * w[4] + b.y * w[5] +
                      b.z * w[6] + b.w * w[7];
        }
    }
#pragma unroll
    for (int t = 0; t < NT; t++) acc[t] = warp_sum(acc[t]);
}

// grid (ceil(T / kTokTile), SI / rows_per_cta).  K = hidden must be a multiple of 8.
__global__ void __launch_bounds__(kThreads)
shared_phase1_kernel(const __nv_bfloat16* __restrict__ x, int tokens, int H, int SI,
                     const __nv_bfloat16* __restrict__ gate_up, const __nv_bfloat16* __restrict__ shared_gate,
                     int rows_per_cta, float* __restrict__ ic2s, float* __restrict__ se_gate) {
    extern __shared__ float xs[];  // [kTokTile][H]
    const int t0 = blockIdx.x * kTokTile;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < kTokTile * H; i += kThreads) {
        int t = t0 + i / H;
        xs[i] = (t < tokens) ? __bfloat162float(x[(size_t)t * H + i % H]) : 0.f;
    }
    __syncthreads();
    const int n0 = blockIdx.y * rows_per_cta;
    float ag[kTokTile], au[kTokTile];
    for (int i = warp; i < rows_per_cta && n0 + i < SI; i += kWarps) {
        const int n = n0 + i;
        row_dots<kTokTile>(gate_up + (size_t)n * H, xs, H, lane, ag);
        row_dots<kTokTile>(gate_up + (size_t)(SI + n) * H, xs, H, lane, au);
        if (lane == 0) {
#pragma unroll
            for (int t = 0; t < kTokTile; t++)
                if (t0 + t < tokens) ic2s[(size_t)(t0 + t) * SI + n] = (ag[t] / (1.0f + expf(-ag[t]))) * au[t];
        }
    }
    // the first row-tile also produces the sigmoid gate
    if (blockIdx.y == 0 && warp == 0) {
        row_dots<kTokTile>(shared_gate, xs, H, lane, ag);
        if (lane == 0) {
#pragma unroll
            for (int t = 0; t < kTokTile; t++)
                if (t0 + t < tokens) se_gate[t0 + t] = 1.0f / (1.0f + expf(-ag[t]));
        }
    }
}

// grid (ceil(T / kTokTile), H / rows_per_cta)
__global__ void __launch_bounds__(kThreads)
shared_phase2_kernel(const float* __restrict__ ic2s, int tokens, int H, int SI,
                     const __nv_bfloat16* __restrict__ down, int rows_per_cta, float* __restrict__ shared_out) {
    extern __shared__ float xs[];  // [kTokTile][SI]
    const int t0 = blockIdx.x * kTokTile;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    for (int i = threadIdx.x; i < kTokTile * SI; i += kThreads) {
        int t = t0 + i / SI;
        xs[i] = (t < tokens) ? ic2s[(size_t)t * SI + i % SI] : 0.f;
    }
    __syncthreads();
    const int d0 = blockIdx.y * rows_per_cta;
    float a[kTokTile];
    for (int i = warp; i < rows_per_cta && d0 + i < H; i += kWarps) {
        const int d = d0 + i;
        row_dots<kTokTile>(down + (size_t)d * SI, xs, SI, lane, a);
        if (lane == 0) {
#pragma unroll
            for (int t = 0; t < kTokTile; t++)
                if (t0 + t < tokens) shared_out[(size_t)(t0 + t) * H + d] = a[t];
        }
    }
}

// ---- tensor-core variant for small batches --------------------------------------------------
// The weights are the A operand of mma.sync.m16n8k16 (16 rows x 16 k, bf16), the tokens the N
// dimension (eight per tile).  A lane reads 16 contiguous bytes of a weight row (eight k) and the
// same eight k of its token row; the k slots of two MMAs are fed from those eight k in order, for
// both operands alike, so any assignment is consistent.  Each weight byte is read once.

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Partial products of one warp: rows (row_lo + g8, row_hi + g8) x tokens [tok0, tok0 + 8*NT) over the k of [k_begin,
// k_end), 32 k per step, SB steps at a time: the weight rows of a block of steps are all asked for before the first
// is used (for a decode batch these kernels are one cold read of a few KB per warp, so they cost its latency: asking
// for two steps at a time took 9.5 us per kernel), the tokens' rows UB steps at a time (they come from L2).
template <int NT, int SB, int UB>
__device__ __forceinline__ void load_rows(uint4 (&lo)[SB], uint4 (&hi)[SB], const __nv_bfloat16* __restrict__ w_lo,
                                          const __nv_bfloat16* __restrict__ w_hi, int k, int k_end) {
#pragma unroll
    for (int i = 0; i < SB; i++)
        if (k + i * 32 < k_end) {
            lo[i] = *reinterpret_cast<const uint4*>(w_lo + k + i * 32);
            hi[i] = *reinterpret_cast<const uint4*>(w_hi + k + i * 32);
        }
}
template <int NT, int SB, int UB>
__device__ __forceinline__ void mma_rows(const uint4 (&lo)[SB], const uint4 (&hi)[SB], const __nv_bfloat16* x,
                                         int ldx, int tok0, int tokens, int k, int k_end, int g8, float (&acc)[NT][4]) {
    const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int i0 = 0; i0 < SB; i0 += UB) {
        uint4 b[UB][NT];
#pragma unroll
        for (int i = 0; i < UB; i++)
#pragma unroll
            for (int n = 0; n < NT; n++) {
                const int t = tok0 + n * 8 + g8, kk = k + (i0 + i) * 32;
                b[i][n] = (t < tokens && kk < k_end) ? *reinterpret_cast<const uint4*>(x + (size_t)t * ldx + kk) : zero;
            }
#pragma unroll
        for (int i = 0; i < UB; i++)
            if (k + (i0 + i) * 32 < k_end) {
                const uint4 &l = lo[i0 + i], &h = hi[i0 + i];
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    mma_bf16_16816(acc[n], l.x, h.x, l.y, h.y, b[i][n].x, b[i][n].y);
                    mma_bf16_16816(acc[n], l.z, h.z, l.w, h.w, b[i][n].z, b[i][n].w);
                }
            }
    }
}

// phase 1: grid (SI / 8 + NT, ceil(T / (8 * NT))); 8 warps split K; rows = 8 gate rows + the 8 matching up rows.  The last NT
// CTAs of a token tile produce its sigmoid gates, one token per warp.  (A ninth warp of every CTA did them: 288 threads of
// 130 registers leave one CTA per SM, and from 129 tokens on a router beside it waited for a second round.  Eight warps
// of at most 128 registers are two CTAs per SM.)
template <int NT>
__global__ void __launch_bounds__(256, 2)
shared_phase1_mma_kernel(const __nv_bfloat16* __restrict__ x, int tokens, int H, int SI,
                         const __nv_bfloat16* __restrict__ gate_up, const __nv_bfloat16* __restrict__ shared_gate,
                         __nv_bfloat16* __restrict__ ic2b, float* __restrict__ se_gate) {
    constexpr int SB = NT == 8 ? 4 : 8, UB = NT == 8 ? 1 : 4;
    __shared__ float red[8][NT][32][4];
    pdl_launch_dependents();
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g8 = lane >> 2, t4 = lane & 3;
    const int pair0 = blockIdx.x * 8, tok0 = blockIdx.y * (8 * NT);
    if (blockIdx.x >= SI / 8) {
        const int t = tok0 + (blockIdx.x - SI / 8) * 8 + warp;
        if (t >= tokens) return;
        float a = 0.f;
#pragma unroll 8
        for (int k = lane * 8; k < H; k += 256) {
            const uint4 wv = *reinterpret_cast<const uint4*>(shared_gate + k);
            const uint4 xv = *reinterpret_cast<const uint4*>(x + (size_t)t * H + k);
            const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w}, xx[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const float2 w2 = bf16x2_to_f32(ww[q]), x2 = bf16x2_to_f32(xx[q]);
                a += w2.x * x2.x + w2.y * x2.y;
            }
        }
        a = warp_sum(a);
        if (lane == 0) se_gate[t] = 1.0f / (1.0f + expf(-a));
        return;
    }
    const int kper = H / 8, k_end = (warp + 1) * kper;
    const __nv_bfloat16 *w_lo = gate_up + (size_t)(pair0 + g8) * H, *w_hi = gate_up + (size_t)(SI + pair0 + g8) * H;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[n][q] = 0.f;
    for (int k = warp * kper + t4 * 8; k < k_end; k += SB * 32) {
        uint4 lo[SB], hi[SB];
        load_rows<NT, SB, UB>(lo, hi, w_lo, w_hi, k, k_end);
        mma_rows<NT, SB, UB>(lo, hi, x, H, tok0, tokens, k, k_end, g8, acc);
    }
#pragma unroll
    for (int n = 0; n < NT; n++)
        *reinterpret_cast<float4*>(red[warp][n][lane]) = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
    __syncthreads();
    // warp n finishes token tile n: sum the K partials, silu(gate) * up
    if (warp < NT) {
        const int n = warp;
        float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int w = 0; w < 8; w++) {
            const float4 v = *reinterpret_cast<const float4*>(red[w][n][lane]);
            c[0] += v.x; c[1] += v.y; c[2] += v.z; c[3] += v.w;
        }
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int t = tok0 + n * 8 + 2 * t4 + q;
            if (t < tokens) {
                // ic2 leaves as a bf16 pair hi + lo (16 significant bits), two planes [tokens, SI]
                const float g = c[q], u = c[2 + q];
                const float v = (g / (1.0f + expf(-g))) * u;
                const __nv_bfloat16 hi = __float2bfloat16_rn(v);
                ic2b[(size_t)t * SI + pair0 + g8] = hi;
                ic2b[(size_t)(tokens + t) * SI + pair0 + g8] = __float2bfloat16_rn(v - __bfloat162float(hi));
            }
        }
    }
}

// phase 2: grid (H / 16, ceil(T / (8 * NT))); 2 warps split K = SI.  Launched behind phase 1 with programmatic dependent
// launch: the weight rows (which phase 1 does not write) are asked for before its result is waited for.
template <int NT>
__global__ void __launch_bounds__(64)
shared_phase2_mma_kernel(const __nv_bfloat16* ic2b, int tokens, int H, int SI,
                         const __nv_bfloat16* __restrict__ down, float* __restrict__ shared_out) {
    constexpr int SB = NT == 8 ? 4 : 8, UB = NT == 8 ? 1 : 4;
    __shared__ float red[NT][32][4];
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g8 = lane >> 2, t4 = lane & 3;
    const int d0 = blockIdx.x * 16, tok0 = blockIdx.y * (8 * NT);
    const int kper = SI / 2, k0 = warp * kper + t4 * 8, k_end = (warp + 1) * kper;
    const __nv_bfloat16 *w_lo = down + (size_t)(d0 + g8) * SI, *w_hi = down + (size_t)(d0 + 8 + g8) * SI;
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[n][q] = 0.f;
    uint4 lo[SB], hi[SB];
    load_rows<NT, SB, UB>(lo, hi, w_lo, w_hi, k0, k_end);
    pdl_wait();
    for (int plane = 0; plane < 2; plane++) {      // the hi plane of ic2, then the lo plane
        const __nv_bfloat16* const xp = ic2b + (size_t)plane * tokens * SI;
        for (int k = k0; k < k_end; k += SB * 32) {
            if (k != k0 || (plane && kper > SB * 32)) load_rows<NT, SB, UB>(lo, hi, w_lo, w_hi, k, k_end);
            mma_rows<NT, SB, UB>(lo, hi, xp, SI, tok0, tokens, k, k_end, g8, acc);
        }
    }
    if (warp == 1) {
#pragma unroll
        for (int n = 0; n < NT; n++)
            *reinterpret_cast<float4*>(red[n][lane]) = make_float4(acc[n][0], acc[n][1], acc[n][2], acc[n][3]);
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int n = 0; n < NT; n++) {
            const float4 v = *reinterpret_cast<const float4*>(red[n][lane]);
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const int t = tok0 + n * 8 + 2 * t4 + q;
                if (t < tokens) {
                    shared_out[(size_t)t * H + d0 + g8] = acc[n][q] + (q ? v.y : v.x);
                    shared_out[(size_t)t * H + d0 + 8 + g8] = acc[n][2 + q] + (q ? v.w : v.z);
                }
            }
        }
    }
}

// NT: token tiles of eight per CTA
template <int NT>
void launch_mma(const __nv_bfloat16* x, int tokens, int H, int SI, const __nv_bfloat16* gate_up, const __nv_bfloat16* down,
                const __nv_bfloat16* shared_gate, __nv_bfloat16* ic2b, float* shared_out, float* se_gate, const Ctx& c) {
    const int tiles = (tokens + 8 * NT - 1) / (8 * NT);
    c.begin(K_SHARED_PHASE1);
    shared_phase1_mma_kernel<NT><<<dim3(SI / 8 + NT, tiles), 256, 0, c.s>>>(x, tokens, H, SI, gate_up, shared_gate, ic2b, se_gate);
    c.end();
    c.begin(K_SHARED_PHASE2);
    launch_pdl(shared_phase2_mma_kernel<NT>, dim3(H / 16, tiles), dim3(64), 0, c.s, (const __nv_bfloat16*)ic2b, tokens, H, SI, down,
               shared_out);
    c.end();
}

}  // namespace

int launch_shared_expert(const __nv_bfloat16* x, int tokens, int hidden, int shared_inter,
                         const __nv_bfloat16* gate_up, const __nv_bfloat16* down,
                         const __nv_bfloat16* shared_gate, float* ic2s, float* shared_out, float* se_gate,
                         int32_t* err, const Ctx& c) {
    if (shared_umma_supported(tokens, hidden, shared_inter)) {
        const int n = launch_shared_umma(x, tokens, hidden, shared_inter, gate_up, down, shared_gate,
                                         reinterpret_cast<__nv_bfloat16*>(ic2s), shared_out, se_gate, err, c);
        if (n >= 0) return n;
    }
    // tensor-core path: K splits must be multiples of 32
    if (hidden % 256 == 0 && shared_inter % 64 == 0 && hidden % 16 == 0 && shared_inter % 8 == 0) {
        __nv_bfloat16* ic2b = reinterpret_cast<__nv_bfloat16*>(ic2s);
        // up to 8, 16 and 64 tokens per CTA: the tiles a small batch does not fill cost MMAs and registers, and a weight row
        // is read once per CTA.  (Four tiles, for 17 to 32 tokens, were slower than eight: 32 tokens 22.8 us against 13.9,
        // with a shared expert of 2048 78.8 against 43.3.)
        auto* const launch = tokens <= 8 ? launch_mma<1> : tokens <= 16 ? launch_mma<2> : launch_mma<8>;
        launch(x, tokens, hidden, shared_inter, gate_up, down, shared_gate, ic2b, shared_out, se_gate, c);
        return 2;
    }
    const int ttiles = (tokens + kTokTile - 1) / kTokTile;
    const int r1 = 16, r2 = 64;
    size_t sm1 = (size_t)kTokTile * hidden * sizeof(float), sm2 = (size_t)kTokTile * shared_inter * sizeof(float);
    static PerDeviceOnce once1, once2;
    allow_dyn_smem(once1, shared_phase1_kernel, 200 * 1024);
    allow_dyn_smem(once2, shared_phase2_kernel, 200 * 1024);
    dim3 g1(ttiles, (shared_inter + r1 - 1) / r1);
    c.begin(K_SHARED_PHASE1);
    shared_phase1_kernel<<<g1, kThreads, sm1, c.s>>>(x, tokens, hidden, shared_inter, gate_up, shared_gate, r1, ic2s,
                                                     se_gate);
    c.end();
    dim3 g2(ttiles, (hidden + r2 - 1) / r2);
    c.begin(K_SHARED_PHASE2);
    shared_phase2_kernel<<<g2, kThreads, sm2, c.s>>>(ic2s, tokens, hidden, shared_inter, down, r2, shared_out);
    c.end();
    return 2;
}

}  // namespace ftm
