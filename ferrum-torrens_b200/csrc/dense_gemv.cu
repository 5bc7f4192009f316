// Dense NVFP4 GEMV for the decode tail (the lm_head): c[m, n] = global[n] * sum_k a[m, k] * W[n, k].
//
// Reference: python/ferrum_kernel/linear.py:41-150 (`_nvfp4_dense_gemv_kernel`, oracle
// `nvfp4_dense_gemv_reference`), launcher src/infrastructure/cuda_linear.rs:48-175 (`DenseGemv::gemv`).
// The weight is the engine's K-MAJOR resident bank, exactly as that launcher takes it:
//   packed [K/8, N] int32   word (w, n) holds the eight e2m1 codes k = 8w .. 8w+7 of row n, nibble j -> k = 8w + j
//   scale  [K/16, N] uint8  e4m3 block scale of block b of row n at (b, n)
//   global [N] f16
// 248 320 x 2048 is 254 MB of packed bytes and 32 MB of scales, streamed once per step: a pure
// HBM-bandwidth kernel.  Three kernels: two share the fragment mapping below and serve sixteen tokens per pass, a
// register-streaming one (any N % 4, K % 32) and, for N % 16 == 0, K % 256 == 0 and N >= 672, one fed by tiled TMA through a
// shared-memory ring, which is the one the lm_head takes (2.3 times the rate of the first on that shape); the third, for
// more tokens, runs on the 5th-generation tensor cores, up to 64 tokens per pass.
//
// Work item: 32 consecutive rows (n) x one half of K.  In a K-major bank four consecutive rows of one k-word
// are 16 contiguous bytes, so lane (g8, t4) of a warp loads, per step, k-word 4*s + t4 of rows
// n0 + 4*g8 .. + 3 with ONE 128-bit load (a warp-wide load is four full 128-byte lines) and the four rows'
// block scales with one 32-bit load.  Which actual row sits in which row of an MMA tile is free, as long as
// the four lanes of a quad agree, so the quad's rows (+0, +1) form one m16n8k16 tile and (+2, +3) another:
//   A (16 rows x 16 k)  row g8 = actual row n0 + 4*g8 (+2), row g8 + 8 = actual row n0 + 4*g8 + 1 (+3);
//                       the quad's four lanes supply k slots {2t, 2t+1, 2t+8, 2t+9} from half of their word
//   B (16 k x 8 tokens) the same eight k of the lane's word for token g8: one 128-bit shared load from the
//                       token's f16 row in natural k order
// Every word is converted with the hardware e2m1x2 -> f16x2 conversion, multiplied by its row's block
// scale (exact in f16) and used by two MMAs per row pair, f32 accumulate.  The two K halves of a row meet
// in `c` by atomic add (c is cleared first; two partial sums commute, so the result is deterministic).
// Loads run kPre steps ahead in a rotating register buffer; nothing waits on a barrier.
#include "kernels.cuh"
#include "umma.cuh"

namespace ftm {

namespace {

constexpr int kDgWarps = 8;
constexpr int kDgPre = 8;        // steps in flight per warp
constexpr int kDgTileRows = 32;

struct DenseArgs {
    const void* a;           // [M, K] bf16 or f32
    int a_dtype;
    const uint32_t* packed;  // [K/8, N]
    const uint8_t* scale;    // [K/16, N]
    const uint16_t* global;  // [N]
    float* c;                // [M, N]; cleared before a launch that splits K (not for the tensor-memory kernel)
    int M, N, K, tok0, ntok, splits;
    int32_t* err;
};

__device__ __forceinline__ uint4 ldg_stream128(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ldg_u32(const void* p) {
    uint32_t v;
    asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void e2m1x8_to_f16x2(uint32_t w, uint32_t (&q)[4]) {
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "mov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\t"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n\t"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n\t"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3])
        : "r"(w));
}
__device__ __forceinline__ uint32_t hmul2_f16(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                        uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT token tiles of 8; dynamic shared memory: the tokens' f16 rows (padded by 64 bytes so that the eight
// token rows of a 128-bit fragment load fall into different banks) and their power-of-two scales
template <int NT>
__global__ void __launch_bounds__(kDgWarps * 32, 2) dense_gemv_kernel(DenseArgs a) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int K = a.K, N = a.N;
    const int rsx = K * 2 + 64;
    float* const s_xscale = reinterpret_cast<float*>(smem + (size_t)8 * NT * rsx);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g8 = lane >> 2, t4 = lane & 3;

    // ---- the activations: warp w converts tokens w, w + 8, .. ----
    for (int tk = warp; tk < 8 * NT; tk += kDgWarps) {
        __half* const xrow = reinterpret_cast<__half*>(smem + (size_t)tk * rsx);
        if (tk >= a.ntok) {      // unused token rows read as zero
            for (int k = lane * 8; k < K; k += 256) *reinterpret_cast<uint4*>(xrow + k) = make_uint4(0, 0, 0, 0);
            if (lane == 0) s_xscale[tk] = 0.f;
            continue;
        }
        const size_t row = (size_t)(a.tok0 + tk) * K;
        float m = 0.f;
        for (int k = lane; k < K; k += 32) m = fmaxf(m, fabsf(load_act(a.a, a.a_dtype, row + k)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float inv, sc;
        f16_row_scale(m, inv, sc);
        for (int k = lane * 2; k < K; k += 64) {
            const float v0 = load_act(a.a, a.a_dtype, row + k), v1 = load_act(a.a, a.a_dtype, row + k + 1);
            *reinterpret_cast<__half2*>(xrow + k) = __floats2half2_rn(v0 * inv, v1 * inv);
        }
        if (lane == 0) s_xscale[tk] = sc;
    }
    __syncthreads();

    const int tiles = (N + kDgTileRows - 1) / kDgTileRows;
    const int steps = K / (32 * a.splits);        // 32 k (four k-words) per step
    const long long items = (long long)tiles * a.splits;
    const long long stride = (long long)gridDim.x * kDgWarps;
    for (long long it = (long long)blockIdx.x * kDgWarps + warp; it < items; it += stride) {
        // items that run at the same time cover neighbouring rows of the same k-words: the bank is read in
        // wide contiguous stripes
        const int split = (int)(it / tiles), tile = (int)(it % tiles);
        const int n = tile * kDgTileRows + 4 * g8;           // this lane's four rows
        const bool live = n < N;                             // N is a multiple of 4: a quad is in or out
        const int kw0 = split * steps * 4 + t4;              // this lane's k-word of step 0
        const uint32_t* const pp = a.packed + (size_t)kw0 * N + n;
        const uint8_t* const sp = a.scale + (size_t)(kw0 >> 1) * N + n;
        uint4 wb[kDgPre];
        uint32_t sb[kDgPre];
        auto fetch = [&](int s, int sl) {
            if (live) {
                wb[sl] = ldg_stream128(pp + (size_t)s * 4 * N);
                sb[sl] = ldg_u32(sp + (size_t)s * 2 * N);     // k-word 4s + t4 lies in block 2s + (t4 >> 1)
            } else {
                wb[sl] = make_uint4(0, 0, 0, 0);
                sb[sl] = 0;
            }
        };
#pragma unroll
        for (int p = 0; p < kDgPre; p++)
            if (p < steps) fetch(p, p);
        float acc[NT][2][2][4];
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int pr = 0; pr < 2; pr++)
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < 4; r++) acc[nt][pr][h][r] = 0.f;
        const uint8_t* const xa = smem + (size_t)g8 * rsx + (size_t)kw0 * 16;
        for (int s0 = 0; s0 < steps; s0 += kDgPre) {
#pragma unroll
            for (int sl = 0; sl < kDgPre; sl++) {
                const int s = s0 + sl;
                if (s < steps) {
                    const uint4 w4 = wb[sl];
                    const uint32_t sc4 = sb[sl];
                    if (s + kDgPre < steps) fetch(s + kDgPre, sl);
                    // four rows' block scales -> f16x2 with the scale in both halves
                    uint32_t h01, h23;
                    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h01) : "h"((uint16_t)sc4));
                    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h23) : "h"((uint16_t)(sc4 >> 16)));
                    const uint32_t sr[4] = {__byte_perm(h01, h01, 0x1010), __byte_perm(h01, h01, 0x3232),
                                            __byte_perm(h23, h23, 0x1010), __byte_perm(h23, h23, 0x3232)};
                    const uint32_t wr[4] = {w4.x, w4.y, w4.z, w4.w};
                    uint32_t q[4][4];
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        e2m1x8_to_f16x2(wr[r], q[r]);
#pragma unroll
                        for (int e = 0; e < 4; e++) q[r][e] = hmul2_f16(q[r][e], sr[r]);
                    }
#pragma unroll
                    for (int nt = 0; nt < NT; nt++) {
                        const uint4 xb = *reinterpret_cast<const uint4*>(xa + (size_t)nt * 8 * rsx + (size_t)s * 64);
#pragma unroll
                        for (int pr = 0; pr < 2; pr++) {
                            // k slots (2t, 2t+1 | 2t+8, 2t+9) <- the word's k (0,1 | 2,3), then (4,5 | 6,7)
                            mma_f16(acc[nt][pr][0], q[2 * pr][0], q[2 * pr + 1][0], q[2 * pr][1], q[2 * pr + 1][1], xb.x, xb.y);
                            mma_f16(acc[nt][pr][1], q[2 * pr][2], q[2 * pr + 1][2], q[2 * pr][3], q[2 * pr + 1][3], xb.z, xb.w);
                        }
                    }
                }
            }
        }
        // ---- epilogue: tile rows g8 / g8 + 8 are actual rows n + 2*pr / n + 2*pr + 1; tokens 2*t4, 2*t4 + 1 ----
        if (live) {
#pragma unroll
            for (int pr = 0; pr < 2; pr++) {
                const float g0 = f16_global_to_f32(a.global[n + 2 * pr]), g1 = f16_global_to_f32(a.global[n + 2 * pr + 1]);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
#pragma unroll
                    for (int cc = 0; cc < 2; cc++) {
                        const int tok = nt * 8 + 2 * t4 + cc;
                        if (tok < a.ntok) {
                            const float ts = s_xscale[tok];
                            float* const dst = a.c + (size_t)(a.tok0 + tok) * N + n + 2 * pr;
                            const float v0 = ((acc[nt][pr][0][cc] + acc[nt][pr][1][cc]) * ts) * g0;
                            const float v1 = ((acc[nt][pr][0][2 + cc] + acc[nt][pr][1][2 + cc]) * ts) * g1;
                            if (a.splits > 1) {
                                atomicAdd(dst, v0);
                                atomicAdd(dst + 1, v1);
                            } else {
                                dst[0] = v0;
                                dst[1] = v1;
                            }
                        }
                    }
                }
            }
        }
    }
}


// ---- the same GEMV fed by TMA ------------------------------------------------------------------
// The register-streaming kernel above keeps few bytes in flight per SM for a bank whose k-word rows lie
// N * 4 bytes apart, and reaches a third of the HBM rate.  Here a CTA owns 672 consecutive rows and one half
// of K, and a producer warp brings, per stage of sixteen k-words, three boxes of [16 k-words x 232 rows] packed
// words and three boxes of [8 blocks x 224 rows] block scales into a ring of shared-memory stages (tiled TMA,
// one mbarrier per stage: six copy instructions per 50 KB; bulk copies of single 2 KB runs spent their time
// on the per-copy cost).  The 232-row box over-fetches eight rows so that its rows sit at a pitch of 928
// bytes, which puts the four k-words a quad reads into different banks.  Twenty-one consumer warps of 32 rows
// each read their fragments from there: the same lane -> (rows, k-word) map, the same conversions and MMAs
// as above.  The two K halves of a row meet in `c` by atomic add, as above (two partial sums commute).
constexpr int kTmBoxRows = 232;              // rows a weight box fetches
constexpr int kTmUseRows = 224;              // rows of it that are used: seven groups of 32
constexpr int kTmBoxes = 3;
constexpr int kTmTileRows = kTmBoxes * kTmUseRows;
constexpr int kTmWarps = kTmTileRows / 32;   // 21 consumer warps (the lm_head's 248 320 rows are 370 tiles: with the two
                                             // K halves 740 items, five for each of 148 CTAs)
constexpr int kTmKw = 16;                    // k-words per stage: four MMA steps
constexpr int kTmStages = 3;
constexpr int kTmWBoxBytes = kTmKw * kTmBoxRows * 4;
constexpr int kTmSBoxBytes = (kTmKw / 2) * kTmUseRows;
constexpr int kTmStageBytes = kTmBoxes * (kTmWBoxBytes + kTmSBoxBytes);
static_assert(kTmWBoxBytes % 128 == 0 && kTmSBoxBytes % 128 == 0, "TMA destinations are 128-byte aligned");

struct DenseMaps {
    CUtensorMap packed, scale;
    CUtensorMap x;      // bf16 activations (tensor-memory kernel)
};

template <int NT>
__global__ void __launch_bounds__((kTmWarps + 1) * 32, 1)
dense_gemv_tma_kernel(const __grid_constant__ DenseMaps maps, DenseArgs a) {
    using namespace umma;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~(uintptr_t)127);
    const int K = a.K, N = a.N;
    const int rsx = K * 2 + 64;
    uint8_t* const ring = smem;                                                    // [kTmStages][kTmStageBytes]
    uint8_t* const xrows = smem + (size_t)kTmStages * kTmStageBytes;               // [8 * NT][rsx]
    float* const s_xscale = reinterpret_cast<float*>(xrows + (size_t)8 * NT * rsx);
    uint64_t* const bars = reinterpret_cast<uint64_t*>(s_xscale + 8 * NT);         // full[stages], empty[stages]
    volatile int* const s_abort = reinterpret_cast<volatile int*>(bars + 2 * kTmStages);
    const uint32_t bar0 = smem_u32(bars);
    auto FULL = [&](int s) { return bar0 + 8u * s; };
    auto EMPTY = [&](int s) { return bar0 + 8u * (kTmStages + s); };
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int g8 = lane >> 2, t4 = lane & 3;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kTmStages; s++) {
            mbar_init(FULL(s), 1);
            mbar_init(EMPTY(s), kTmWarps);
        }
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();     // the barriers are initialised

    const int tiles = (N + kTmTileRows - 1) / kTmTileRows;
    const int stages_per_item = K / (8 * kTmKw * 2);      // half of K, sixteen k-words per stage
    const int items = tiles * 2;

    if (warp == kTmWarps) {
        // ===================== producer: one elected lane issues the four copies of a stage ===========
        uint32_t it = 0;
        for (int item = blockIdx.x; item < items && !*s_abort; item += gridDim.x) {
            const int split = item / tiles, n0 = (item % tiles) * kTmTileRows;
            bool ok = true;
            for (int s = 0; s < stages_per_item && ok; s++, it++) {
                const int st = it % kTmStages;
                ok = mbar_wait_warp(EMPTY(st), ((it / kTmStages) & 1) ^ 1, s_abort, a.err);
                if (!ok) break;
                if (elect_one()) {
                    const int kw = (split * stages_per_item + s) * kTmKw;
                    const uint32_t dst = smem_u32(ring + (size_t)st * kTmStageBytes);
                    // rows past N read as zero and count like the others
                    mbar_expect_tx(FULL(st), kTmStageBytes);
#pragma unroll
                    for (int b = 0; b < kTmBoxes; b++) {
                        tma_load_2d(dst + b * kTmWBoxBytes, &maps.packed, n0 + b * kTmUseRows, kw, FULL(st));
                        tma_load_2d(dst + kTmBoxes * kTmWBoxBytes + b * kTmSBoxBytes, &maps.scale, n0 + b * kTmUseRows, kw / 2, FULL(st));
                    }
                }
                __syncwarp();
            }
            if (!ok) break;
        }
        return;
    }

    // ===================== consumers: warp w owns rows 32 w .. 32 w + 31 of the tile ====================
    // ---- the activations (as in the kernel above): consumer warp w converts tokens w, w + 21, .. while the
    // producer already fills the ring ----
    for (int tk = warp; tk < 8 * NT; tk += kTmWarps) {
        __half* const xrow = reinterpret_cast<__half*>(xrows + (size_t)tk * rsx);
        if (tk >= a.ntok) {
            for (int k = lane * 8; k < K; k += 256) *reinterpret_cast<uint4*>(xrow + k) = make_uint4(0, 0, 0, 0);
            if (lane == 0) s_xscale[tk] = 0.f;
            continue;
        }
        const size_t row = (size_t)(a.tok0 + tk) * K;
        float m = 0.f;
#pragma unroll 16
        for (int k = lane; k < K; k += 32) m = fmaxf(m, fabsf(load_act(a.a, a.a_dtype, row + k)));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        float inv, sc;
        f16_row_scale(m, inv, sc);
#pragma unroll 8
        for (int k = lane * 2; k < K; k += 64) {
            const float v0 = load_act(a.a, a.a_dtype, row + k), v1 = load_act(a.a, a.a_dtype, row + k + 1);
            *reinterpret_cast<__half2*>(xrow + k) = __floats2half2_rn(v0 * inv, v1 * inv);
        }
        if (lane == 0) s_xscale[tk] = sc;
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kTmWarps * 32) : "memory");     // the consumer warps only

    const int box = warp / 7, rbox = (warp % 7) * 32 + 4 * g8;     // this lane's four rows inside its box
    const uint32_t woff = box * kTmWBoxBytes + rbox * 4;
    const uint32_t soff = kTmBoxes * kTmWBoxBytes + box * kTmSBoxBytes + rbox;
    uint32_t it = 0;
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const int split = item / tiles, n0 = (item % tiles) * kTmTileRows;
        float acc[NT][2][2][4];      // [token tile][row pair][k half][fragment]
#pragma unroll
        for (int nt = 0; nt < NT; nt++)
#pragma unroll
            for (int pr = 0; pr < 2; pr++)
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int r = 0; r < 4; r++) acc[nt][pr][h][r] = 0.f;
        const uint8_t* const xa = xrows + (size_t)g8 * rsx + ((size_t)split * stages_per_item * kTmKw + t4) * 16;
        bool ok = true;
        for (int s = 0; s < stages_per_item; s++, it++) {
            const int st = it % kTmStages;
            ok = mbar_wait_warp(FULL(st), (it / kTmStages) & 1, s_abort, a.err);
            if (!ok) break;
            const uint8_t* const sp = ring + (size_t)st * kTmStageBytes;
#pragma unroll
            for (int j = 0; j < kTmKw / 4; j++) {
                const uint4 w4 = *reinterpret_cast<const uint4*>(sp + woff + (4 * j + t4) * (kTmBoxRows * 4));
                const uint32_t sc4 = *reinterpret_cast<const uint32_t*>(sp + soff + (2 * j + (t4 >> 1)) * kTmUseRows);
                uint32_t h01, h23;
                asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h01) : "h"((uint16_t)sc4));
                asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h23) : "h"((uint16_t)(sc4 >> 16)));
                const uint32_t sr[4] = {__byte_perm(h01, h01, 0x1010), __byte_perm(h01, h01, 0x3232),
                                        __byte_perm(h23, h23, 0x1010), __byte_perm(h23, h23, 0x3232)};
                const uint32_t wr[4] = {w4.x, w4.y, w4.z, w4.w};
                uint32_t q[4][4];
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    e2m1x8_to_f16x2(wr[r], q[r]);
#pragma unroll
                    for (int e = 0; e < 4; e++) q[r][e] = hmul2_f16(q[r][e], sr[r]);
                }
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
                    const uint4 xb = *reinterpret_cast<const uint4*>(xa + (size_t)nt * 8 * rsx + (size_t)(s * (kTmKw / 4) + j) * 64);
#pragma unroll
                    for (int pr = 0; pr < 2; pr++) {
                        mma_f16(acc[nt][pr][0], q[2 * pr][0], q[2 * pr + 1][0], q[2 * pr][1], q[2 * pr + 1][1], xb.x, xb.y);
                        mma_f16(acc[nt][pr][1], q[2 * pr][2], q[2 * pr + 1][2], q[2 * pr][3], q[2 * pr + 1][3], xb.z, xb.w);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(EMPTY(st));
        }
        if (!ok) break;
        // ---- epilogue: as above; rows past N of the last tile read as zero and are not stored ----
        const int n = n0 + box * kTmUseRows + rbox;
        if (n < N) {
#pragma unroll
            for (int pr = 0; pr < 2; pr++) {
                const float g0 = f16_global_to_f32(a.global[n + 2 * pr]), g1 = f16_global_to_f32(a.global[n + 2 * pr + 1]);
#pragma unroll
                for (int nt = 0; nt < NT; nt++) {
#pragma unroll
                    for (int cc = 0; cc < 2; cc++) {
                        const int tok = nt * 8 + 2 * t4 + cc;
                        if (tok < a.ntok) {
                            const float ts = s_xscale[tok];
                            float* const dst = a.c + (size_t)(a.tok0 + tok) * N + n + 2 * pr;
                            atomicAdd(dst, ((acc[nt][pr][0][cc] + acc[nt][pr][1][cc]) * ts) * g0);
                            atomicAdd(dst + 1, ((acc[nt][pr][0][2 + cc] + acc[nt][pr][1][2 + cc]) * ts) * g1);
                        }
                    }
                }
            }
        }
    }
}

template <int NT>
size_t tma_smem(int K) {
    return 128 + (size_t)kTmStages * kTmStageBytes + (size_t)8 * NT * (K * 2 + 64) + 8 * NT * sizeof(float) + 2 * kTmStages * 8 + 16;
}
template <int NT>
void launch_tma(const DenseMaps& maps, const DenseArgs& a, int sm_count, cudaStream_t s) {
    static PerDeviceOnce once;
    allow_dyn_smem(once, dense_gemv_tma_kernel<NT>, 222 * 1024);
    dense_gemv_tma_kernel<NT><<<sm_count, (kTmWarps + 1) * 32, tma_smem<NT>(a.K), s>>>(maps, a);
}

// [rows, inner] matrix of `esize`-byte elements, row-major, box = box_inner x box_rows
bool make_plain_map(CUtensorMap* map, CUtensorMapDataType type, int esize, const void* base, size_t inner, size_t rows,
                    int box_inner, int box_rows, CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_NONE) {
    umma::EncodeTiledFn fn = umma::encode_tiled();
    if (!fn) return false;
    cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)inner * esize};
    cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return fn(map, type, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// ---- the same product on the 5th-generation tensor cores, for more than kUmmaMinTok tokens ------------
// The kernels above serve sixteen tokens per pass over the bank and are bound by their conversions and the
// mma.sync rate from there on (95 us a pass at 248 320 x 2048), so 64 tokens were four passes (408 us).  Here one pass
// serves up to 64: the dequantised weights are the A operand in tensor memory (one lane per weight row, as in the
// grouped GEMM of prefill_umma.cu), the tokens are the B operand in shared memory, f32 accumulators in tensor memory.
// Unit = 256 rows (two tiles of 128) x the whole of K, persistent CTAs of 24 warps:
//   warp 0        TMA: [32 k-words x 128 rows] packed words and [16 blocks x 128 rows] block scales into a raw ring.
//                 The bank is K-major, so a k-word of a tile is one 512-byte run and lane = row reads it without
//                 bank conflicts
//   warps 1, 3    tcgen05.mma issuers, one per row tile (M = 128, N = tokens rounded up to 16)
//   warp 2        TMA: tiles of 64 tokens x 64 k of bf16 activations (they stay in L2), 128-byte swizzle
//   warps 4..7    rewrite every such tile in place as f16, scaled per token by a power of two (exact).  Converting the
//                 activations again for every unit costs these four warps less time than the unit takes, and needs
//                 no scratch buffer that calls on two streams would share.  f32 activations they read themselves
//   warps 8..15   two dequantiser sets, two weight buffers each
//   warps 16..23  epilogue, one set per row tile: sums the accumulators, applies token scale and row global,
//                 stores whole rows (no K split: nothing to clear, no atomics)
// Consecutive 64-k steps go to different accumulators in turn (two for 64 tokens, four for 32), summed in f32 by the
// epilogue: the chain of one accumulator stays short, as in the kernels above.
// Every mbarrier wait is bounded; a wait that gives up raises the error flag and the CTA drains.
// Seventeen tokens would be two passes of the kernels above; sixteen are one pass of either.  248 320 rows, cold: 99.4 us above
// and 96.7 here for sixteen tokens, 90.8 and 101.7 for nine.  Smaller banks lean further to this side (75 776 rows 45.8 and
// 30.9, 8192 rows 26.3 and 16.4 for sixteen), which the border does not use yet.
constexpr int kUmmaMinTok = 16;
constexpr int kUmThreads = 768;
constexpr int kUmTok = 64;                     // most tokens per pass
constexpr int kUmXStages = 8, kUmRawStages = 6;
constexpr int kUmXBytes = kUmTok * 128;        // 64 tokens x 64 k f16
constexpr int kUmPackedBytes = 32 * 128 * 4, kUmScaleBytes = 16 * 128;
constexpr int kUmRawBytes = kUmPackedBytes + kUmScaleBytes;
constexpr int kUmWBufs = 4, kUmWCols = 64;     // dequantised chunks of 128 k in tensor memory
constexpr int kUmAccCol0 = kUmWBufs * kUmWCols, kUmAccCols = 128;   // accumulator columns of one row tile
constexpr size_t kUmSmem = 1024 + (size_t)kUmXStages * kUmXBytes + (size_t)kUmRawStages * kUmRawBytes + 48 * 8 + kUmTok * 4 + 64;

template <bool F32>
__global__ void __launch_bounds__(kUmThreads, 1)
dense_gemv_umma_kernel(const __grid_constant__ DenseMaps maps, DenseArgs a) {
    using namespace umma;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* const smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* const x_tiles = smem;
    uint8_t* const raw_ring = smem + kUmXStages * kUmXBytes;
    uint64_t* const bars = reinterpret_cast<uint64_t*>(raw_ring + kUmRawStages * kUmRawBytes);
    float* const s_scale = reinterpret_cast<float*>(bars + 48);     // per token: the power of two its row was divided by
    uint32_t* const s_tmem = reinterpret_cast<uint32_t*>(s_scale + kUmTok);
    volatile int* const s_abort = reinterpret_cast<volatile int*>(s_tmem + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto X_FULL = [&](int s) { return bar0 + 8u * s; };
    auto X_EMPTY = [&](int s) { return bar0 + 8u * (8 + s); };
    auto RAW_FULL = [&](int s) { return bar0 + 8u * (16 + s); };
    auto RAW_EMPTY = [&](int s) { return bar0 + 8u * (22 + s); };
    auto W_READY = [&](int s) { return bar0 + 8u * (28 + s); };
    auto W_FREE = [&](int s) { return bar0 + 8u * (32 + s); };
    const uint32_t ACC_FULL = bar0 + 8u * 36, ACC_EMPTY = bar0 + 8u * 37;
    auto XRAW_FULL = [&](int s) { return bar0 + 8u * (38 + s); };
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kUmXStages; s++) {
            mbar_init(XRAW_FULL(s), 1);
            mbar_init(X_FULL(s), 4);
            mbar_init(X_EMPTY(s), 2);
        }
        for (int s = 0; s < kUmRawStages; s++) {
            mbar_init(RAW_FULL(s), 1);
            mbar_init(RAW_EMPTY(s), 8);       // two pieces x four warps
        }
        for (int s = 0; s < kUmWBufs; s++) {
            mbar_init(W_READY(s), 4);
            mbar_init(W_FREE(s), 1);
        }
        mbar_init(ACC_FULL, 2);
        mbar_init(ACC_EMPTY, 8);
        *s_abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(s_tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *s_tmem;

    const int K = a.K, N = a.N;
    const int chunks = K / 128, items_per_unit = 2 * chunks;    // (chunk, row tile) pieces; chunks is even
    const int n_units = (N + 255) / 256;
    const int n_pad = (a.ntok + 15) & ~15;
    const int splits = n_pad <= 32 ? 4 : 2, acc_stride = kUmAccCols / splits;

    if (warp != 0) {
        // the power of two of every token (the weight producer is already at work): largest magnitude into [2^14, 2^15)
        for (int tk = warp - 1; tk < a.ntok; tk += kUmThreads / 32 - 1) {
            const size_t row = (size_t)(a.tok0 + tk) * K;
            float m = 0.f;
#pragma unroll 8
            for (int k = lane * (F32 ? 4 : 8); k < K; k += F32 ? 128 : 256) {
                if (F32) {
                    const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(a.a) + row + k);
                    m = fmaxf(fmaxf(fmaxf(m, fabsf(v.x)), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
                } else {
                    const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(a.a) + row + k);
                    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float2 f = bf16x2_to_f32(w[q]);
                        m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
                    }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            float inv, sc;
            f16_row_scale(m, inv, sc);
            if (lane == 0) s_scale[tk] = sc;
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kUmThreads - 32) : "memory");
    }

    if (warp == 0) {
        // ===================== packed weights and block scales =======================================
        uint32_t it = 0;
        for (int u = blockIdx.x; u < n_units && !*s_abort; u += gridDim.x) {
            bool ok = true;
            for (int q = 0; q < chunks && ok; q++, it++) {     // a stage = two chunks (256 k) of one row tile
                const int cp = q >> 1, r = q & 1, st = it % kUmRawStages;
                ok = mbar_wait_warp(RAW_EMPTY(st), ((it / kUmRawStages) & 1) ^ 1, s_abort, a.err);
                if (!ok) break;
                if (elect_one()) {
                    const uint32_t dst = smem_u32(raw_ring + (size_t)st * kUmRawBytes);
                    mbar_expect_tx(RAW_FULL(st), kUmRawBytes);      // rows past N read as zero and count like the others
                    tma_load_2d(dst, &maps.packed, u * 256 + r * 128, cp * 32, RAW_FULL(st));
                    tma_load_2d(dst + kUmPackedBytes, &maps.scale, u * 256 + r * 128, cp * 16, RAW_FULL(st));
                }
                __syncwarp();
            }
            if (!ok) break;
        }
    } else if (warp == 2) {
        // ===================== bf16 activation tiles ================================================
        if constexpr (!F32) {
            uint32_t it = 0;
            for (int u = blockIdx.x; u < n_units && !*s_abort; u += gridDim.x) {
                bool ok = true;
                for (int ks = 0; ks < K / 64; ks++, it++) {
                    const int st = it % kUmXStages;
                    ok = mbar_wait_warp(X_EMPTY(st), ((it / kUmXStages) & 1) ^ 1, s_abort, a.err);
                    if (!ok) break;
                    if (elect_one()) {
                        mbar_expect_tx(XRAW_FULL(st), kUmXBytes);      // rows past the last token read as zero
                        tma_load_2d(smem_u32(x_tiles + (size_t)st * kUmXBytes), &maps.x, ks * 64, a.tok0, XRAW_FULL(st));
                    }
                    __syncwarp();
                }
                if (!ok) break;
            }
        }
    } else if (warp == 1 || warp == 3) {
        // ===================== MMA issuers (see the grouped GEMM for the looks ahead) ================
        const int r = warp >> 1;
        const uint32_t idesc = (1u << 4) | ((uint32_t)(128 >> 4) << 24) | ((uint32_t)(n_pad >> 3) << 17);
        const uint32_t d_tmem = tmem_base + kUmAccCol0 + r * kUmAccCols;
        uint32_t it = 0, item = r, unit_i = 0;
        bool x_seen = false, w_seen = false;
        for (int u = blockIdx.x; u < n_units && !*s_abort; u += gridDim.x, unit_i++) {
            bool ok = mbar_wait_warp(ACC_EMPTY, (unit_i & 1) ^ 1, s_abort, a.err);
            for (int ks = 0; ks < 2 * chunks && ok; ks++, it++) {
                const int h = ks & 1, wb = item % kUmWBufs, st = it % kUmXStages;
                if (h == 0 && !w_seen) ok = mbar_wait_warp(W_READY(wb), (item / kUmWBufs) & 1, s_abort, a.err);
                if (!ok) break;
                if (!x_seen) ok = mbar_wait_warp(X_FULL(st), (it / kUmXStages) & 1, s_abort, a.err);
                if (!ok) break;
                {
                    const uint32_t it1 = it + 1;
                    x_seen = __all_sync(0xffffffffu, mbar_test_wait(X_FULL(it1 % kUmXStages), (it1 / kUmXStages) & 1));
                    if (h == 1) {
                        const uint32_t item1 = item + 2;
                        w_seen = __all_sync(0xffffffffu, mbar_test_wait(W_READY(item1 % kUmWBufs), (item1 / kUmWBufs) & 1));
                    }
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t w_addr = tmem_base + wb * kUmWCols;
                const uint64_t xdesc = umma_desc(smem_u32(x_tiles + (size_t)st * kUmXBytes));
                const uint32_t d = d_tmem + (ks & (splits - 1)) * acc_stride;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 4; kk++)
                        umma_f16_ts(d, w_addr + (h * 4 + kk) * 8, xdesc + kk * 2, idesc, (ks >= splits || kk > 0) ? 1u : 0u);
                    umma_commit(X_EMPTY(st));
                    if (h == 1) umma_commit(W_FREE(wb));
                }
                __syncwarp();
                if (h == 1) item += 2;
            }
            if (!ok) break;
            if (elect_one()) umma_commit(ACC_FULL);
            __syncwarp();
        }
    } else if (warp >= 4 && warp < 8) {
        // ===================== activations: two threads per token, 32 k each ==========================
        const int tid = threadIdx.x - 128, tok = tid >> 1, half = tid & 1;
        const bool live = tok < a.ntok, in_tile = tok < n_pad;      // (a row past this pass's may be another's: its factor is 0)
        const int steps = K / 64;
        const float inv = live ? 1.0f / s_scale[tok] : 0.f;       // a power of two: exact
        const float* const src = reinterpret_cast<const float*>(a.a) + (size_t)(a.tok0 + (live ? tok : 0)) * K + half * 32;
        float4 buf[F32 ? 8 : 1];      // f32: the next step's 32 k, loaded a step ahead
        auto load = [&](int ks) {
#pragma unroll
            for (int v = 0; v < 8; v++)
                buf[v] = live ? *reinterpret_cast<const float4*>(src + (size_t)ks * 64 + v * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        uint32_t it = 0;
        for (int u = blockIdx.x; u < n_units && !*s_abort; u += gridDim.x) {
            bool ok = true;
            if constexpr (F32) load(0);
            for (int ks = 0; ks < steps; ks++, it++) {
                const int st = it % kUmXStages;
                uint8_t* const row = x_tiles + (size_t)st * kUmXBytes + tok * 128;
                __half2 h2[16];
                if constexpr (F32) {
#pragma unroll
                    for (int v = 0; v < 8; v++) {
                        h2[2 * v] = __floats2half2_rn(buf[v].x * inv, buf[v].y * inv);
                        h2[2 * v + 1] = __floats2half2_rn(buf[v].z * inv, buf[v].w * inv);
                    }
                    if (ks + 1 < steps) load(ks + 1);
                    ok = mbar_wait_warp(X_EMPTY(st), ((it / kUmXStages) & 1) ^ 1, s_abort, a.err);
                    if (!ok) break;
                } else {
                    ok = mbar_wait_warp(XRAW_FULL(st), (it / kUmXStages) & 1, s_abort, a.err);
                    if (!ok) break;
                    if (in_tile) {
#pragma unroll
                        for (int j = 0; j < 4; j++) {
                            const uint4 v = *reinterpret_cast<const uint4*>(row + (((half * 4 + j) ^ (tok & 7)) << 4));
                            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                const float2 f = bf16x2_to_f32(w[q]);
                                h2[4 * j + q] = __floats2half2_rn(f.x * inv, f.y * inv);
                            }
                        }
                    }
                }
                if (in_tile) {
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        *reinterpret_cast<uint4*>(row + (((half * 4 + j) ^ (tok & 7)) << 4)) =
                            make_uint4(*reinterpret_cast<uint32_t*>(&h2[4 * j]), *reinterpret_cast<uint32_t*>(&h2[4 * j + 1]),
                                       *reinterpret_cast<uint32_t*>(&h2[4 * j + 2]), *reinterpret_cast<uint32_t*>(&h2[4 * j + 3]));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the tensor core reads what this thread stored
                mbar_arrive_warp(X_FULL(st));
            }
            if (!ok) break;
        }
    } else if (warp >= 8 && warp < 16) {
        // ===================== dequantisers: raw ring -> f16 weights in tensor memory ================
        const int quarter = warp & 3, set = (warp - 8) >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t tlane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        uint32_t item0 = 0, stage0 = 0;
        for (int u = blockIdx.x; u < n_units && !*s_abort; u += gridDim.x, item0 += items_per_unit, stage0 += chunks) {
            bool ok = true;
            for (int w = set; w < items_per_unit; w += 2) {
                const uint32_t item = item0 + w;
                const int c = w >> 1;
                const uint32_t stage = stage0 + 2 * (c >> 1) + (w & 1);
                const int st = stage % kUmRawStages;
                ok = mbar_wait_warp(RAW_FULL(st), (stage / kUmRawStages) & 1, s_abort, a.err);
                if (!ok) break;
                const int wb = item % kUmWBufs;
                const uint32_t taddr = tlane + wb * kUmWCols;
                const uint8_t* const rp = raw_ring + (size_t)st * kUmRawBytes + (c & 1) * 16 * 512 + row * 4;
                const uint8_t* const sp = raw_ring + (size_t)st * kUmRawBytes + kUmPackedBytes + (c & 1) * 8 * 128 + row;
                // 32 k (four k-words, two block scales) -> 16 columns
                auto convert = [&](int g, uint32_t (&r)[16]) {
                    const uint32_t two = (uint32_t)sp[(2 * g) * 128] | ((uint32_t)sp[(2 * g + 1) * 128] << 8);
                    uint32_t h2;
                    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"((uint16_t)two));
                    const uint32_t s0 = __byte_perm(h2, h2, 0x1010), s1 = __byte_perm(h2, h2, 0x3232);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uint32_t q[4];
                        e2m1x8_to_f16x2(*reinterpret_cast<const uint32_t*>(rp + (4 * g + j) * 512), q);
#pragma unroll
                        for (int e = 0; e < 4; e++) r[4 * j + e] = hmul2_f16(q[e], (j < 2) ? s0 : s1);
                    }
                };
                uint32_t r0[16], r1[16];
                convert(0, r0);
                convert(1, r1);
                ok = mbar_wait_warp(W_FREE(wb), ((item / kUmWBufs) & 1) ^ 1, s_abort, a.err);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                tmem_st16(taddr, r0);
                tmem_st16(taddr + 16, r1);
                convert(2, r0);
                tmem_st16(taddr + 32, r0);
                convert(3, r1);
                tmem_st16(taddr + 48, r1);
                mbar_arrive_warp(RAW_EMPTY(st));
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive_warp(W_READY(wb));
            }
            if (!ok) break;
        }
    } else if (warp >= 16) {
        // ===================== epilogue: one thread = one weight row, a column = one token =============
        const int quarter = warp & 3, r = (warp - 16) >> 2;
        uint32_t unit_i = 0;
        for (int u = blockIdx.x; u < n_units && !*s_abort; u += gridDim.x, unit_i++) {
            const int n = u * 256 + r * 128 + quarter * 32 + lane;
            const float gl = n < N ? f16_global_to_f32(a.global[n]) : 0.f;
            if (!mbar_wait_warp(ACC_FULL, unit_i & 1, s_abort, a.err)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + kUmAccCol0 + r * kUmAccCols;
#pragma unroll 1
            for (int c0 = 0; c0 < a.ntok; c0 += 16) {
                float v[16], v1[16];
                tmem_ld16(taddr + c0, v);
                tmem_ld16(taddr + acc_stride + c0, v1);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] += v1[j];
                if (splits == 4) {
                    float v2[16];
                    tmem_ld16(taddr + 2 * acc_stride + c0, v1);
                    tmem_ld16(taddr + 3 * acc_stride + c0, v2);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] += v1[j] + v2[j];
                }
                if (n < N) {
                    float* const dst = a.c + (size_t)(a.tok0 + c0) * N + n;
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        if (c0 + j < a.ntok) dst[(size_t)j * N] = (v[j] * s_scale[c0 + j]) * gl;
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive_warp(ACC_EMPTY);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
}

template <bool F32>
void launch_umma(const DenseMaps& maps, const DenseArgs& a, int sm_count, cudaStream_t s) {
    static PerDeviceOnce once;
    allow_dyn_smem(once, dense_gemv_umma_kernel<F32>, kUmSmem);
    dense_gemv_umma_kernel<F32><<<sm_count, kUmThreads, kUmSmem, s>>>(maps, a);
}

template <int NT>
void launch_one(const DenseArgs& a, int sm_count, cudaStream_t s) {
    const size_t smem = (size_t)8 * NT * (a.K * 2 + 64) + 8 * NT * sizeof(float) + 16;
    static PerDeviceOnce once;
    allow_dyn_smem(once, dense_gemv_kernel<NT>, 100 * 1024);
    dense_gemv_kernel<NT><<<sm_count * 2, kDgWarps * 32, smem, s>>>(a);
}

}  // namespace

bool dense_gemv_supported(int N, int K) {
    // 16-byte loads of four rows, 32 k per step, the token rows of at most sixteen tokens in shared memory
    return N > 0 && K > 0 && N % 4 == 0 && K % 32 == 0 && (size_t)16 * (K * 2 + 64) + 256 <= 100 * 1024;
}

int launch_dense_gemv(const void* a, int a_dtype, const uint32_t* packed, const uint8_t* scale, const uint16_t* global,
                      int M, int N, int K, float* c, int sm_count, int32_t* err, const Ctx& ctx) {
    DenseArgs d{};
    d.a = a; d.a_dtype = a_dtype; d.packed = packed; d.scale = scale; d.global = global; d.c = c;
    d.M = M; d.N = N; d.K = K; d.err = err;
    // TMA wants the rows of both matrices 16-byte aligned (N % 16 for the scales) and whole stages per K half
    DenseMaps maps;
    const bool tma = N % 16 == 0 && K % 256 == 0 && N >= kTmTileRows && (reinterpret_cast<uintptr_t>(packed) & 15) == 0 &&
                     (reinterpret_cast<uintptr_t>(scale) & 15) == 0 && tma_smem<2>(K) <= 222 * 1024 &&
                     make_plain_map(&maps.packed, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, packed, (size_t)N, (size_t)K / 8, kTmBoxRows, kTmKw) &&
                     make_plain_map(&maps.scale, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, scale, (size_t)N, (size_t)K / 16, kTmUseRows, kTmKw / 2);
    d.splits = (tma || K % 64 == 0) ? 2 : 1;
    // More tokens than one pass of the kernels above serves: the tensor-memory kernel, under their alignment rules for
    // the bank (its units are 256 rows) and with activations that can be read 16 bytes at a time.  A remainder of up to
    // kUmmaMinTok tokens after passes of 64 goes to the kernels above.
    DenseMaps umaps;
    const bool umma = M > kUmmaMinTok && N % 16 == 0 && K % 256 == 0 && N >= 256 && (reinterpret_cast<uintptr_t>(packed) & 15) == 0 &&
                      (reinterpret_cast<uintptr_t>(scale) & 15) == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0 &&
                      make_plain_map(&umaps.packed, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, packed, (size_t)N, (size_t)K / 8, 128, 32) &&
                      make_plain_map(&umaps.scale, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, scale, (size_t)N, (size_t)K / 16, 128, 16) &&
                      (a_dtype == 1 || make_plain_map(&umaps.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, a, (size_t)K, (size_t)M, 64, kUmTok,
                                                      CU_TENSOR_MAP_SWIZZLE_128B));
    int launches = 0, t0 = 0;
    ctx.begin(K_DENSE_GEMV);
    for (; umma && M - t0 > kUmmaMinTok; t0 += kUmTok) {
        d.tok0 = t0;
        d.ntok = (M - t0 < kUmTok) ? M - t0 : kUmTok;
        if (a_dtype == 1)
            launch_umma<true>(umaps, d, sm_count, ctx.s);
        else
            launch_umma<false>(umaps, d, sm_count, ctx.s);
        launches++;
    }
    // the K halves of the kernels above add into c
    if (t0 < M && d.splits > 1) cudaMemsetAsync(c + (size_t)t0 * N, 0, (size_t)(M - t0) * N * sizeof(float), ctx.s);
    // sixteen tokens per pass over the weights (the decode tail runs at one token per sequence)
    for (; t0 < M; t0 += 16) {
        d.tok0 = t0;
        d.ntok = (M - t0 < 16) ? M - t0 : 16;
        if (tma) {
            if (d.ntok <= 8)
                launch_tma<1>(maps, d, sm_count, ctx.s);
            else
                launch_tma<2>(maps, d, sm_count, ctx.s);
        } else if (d.ntok <= 8) {
            launch_one<1>(d, sm_count, ctx.s);
        } else {
            launch_one<2>(d, sm_count, ctx.s);
        }
        launches++;
    }
    ctx.end();
    return launches;
}

}  // namespace ftm
