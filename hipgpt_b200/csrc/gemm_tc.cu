// The projections either side of attention on the Blackwell tensor pipe (tcgen05 + TMEM) with fp32-grade results:
//   C[M][K] = A[M][N] B[N][K] (+ bias[K]),  the reference's argument order, N the inner dimension
// (HipGPT launch_matmul / launch_matmul_add_bias, src/hip_kernels.cpp:69-154; callers src/transformer_layer.cpp:217,220).
// The exact mode (one accumulator per output, inner index ascending, FMA: bit-identical to the reference's order) is
// hipgpt_matmul in layer_ops.cu; this is the fast mode: same operands, same output, 1e-5 instead of identical bits.
//
// Arithmetic (the scheme of the tiled attention kernel): every fp32 operand x is scaled by a power of two (exact) and cut
// into hi (its 11 leading bits, exact in fp16) and lo = x - hi (rounded to fp16's 11 bits); a*b = a_hi*b_hi + a_hi*b_lo +
// a_lo*b_hi as kind::f16 products with fp32 accumulation in the tensor core, the dropped a_lo*b_lo is 2^-22 relative.
// Scales: one per row of A (range_scale of the row's largest magnitude) and one for the whole of B; both leave in the
// epilogue.  An element of B more than 2^-20 below B's largest magnitude keeps fewer bits (its lo part becomes a
// subnormal fp16); the exact mode is there for such operands.
//
// Four kernels per call:
//   gemm_amax_kernel     largest |B|  (B is at most a few MB here: one pass)
//   gemm_pack_a_kernel   A -> per (128-row tile, 64-deep slice) the shared-memory image of a K-major operand stage with
//                        128-byte swizzle: a block of A_hi rows and a block of A_lo rows (fp16); row scales to a vector
//   gemm_pack_b_kernel   B -> per (64-deep slice, 128-column tile) the image of an N-major operand stage without
//                        swizzle, columns [B_hi (128) | B_lo (128)]
//   gemm_tc_kernel       one block per SM, 128 x 128 output tiles in turn: a producer warp fetches whole stages with bulk
//                        copies (three stages of 64 KB in flight, running on into the next tile), an issuing warp forms
//                        A_hi [B_hi | B_lo] (N = 256) and A_lo B_hi (N = 128, onto the second half) for every slice, 8
//                        instructions per slice, into one of two accumulators of 256 TMEM columns; eight warps (thread =
//                        output row = TMEM lane; two share the columns of a row) add the halves, take the scales out, add
//                        the bias and store one tile while the products of the next one run.
// Where the time of a small product goes (1407 x 512 x 1536, marks in an instrumented copy, us after A's images are there): first
// stage landed 0.8 (1.3 with B's part asked for only then), eight slices 4.0 (64 KB each at 64 bytes per clock and SM), last product 0.7, output
// 1.5 (4.0 with four warps and the bias asked for piece by piece behind the products).
// Rows, columns and depth beyond the matrices are zeros in the images; stores are bounded by M and K.
// Every wait is bounded: on expiry the block records a status code, skips its stores, lets what is on its way land, frees its TMEM
// and returns; the blocks that share its tile store none of it.
#include "stream_workspace.hpp"
#include "tc_primitives.cuh"

#include <math.h>

namespace hipgpt {
namespace {

constexpr int kTM = 128, kTN = 128, kTK = 64;     // output tile and depth of a slice
constexpr int kStages = 3;
constexpr int kABlk = kTM * 128;                  // bytes of one block of an A stage: 128 rows of 64 fp16
constexpr int kAStage = 2 * kABlk;                // [A_hi | A_lo]
constexpr int kBStage = kTK * 2 * kTN * 2;        // 64 deep x [B_hi (128) | B_lo (128)] fp16
constexpr int kGroupStride = 2 * kTN * 16;        // bytes between groups of 8 reduction rows of a B stage (32 column blocks of 128 bytes)
constexpr int kEpiWarps = 8;                      // two per quarter of the rows, each half of the columns
constexpr int kGemmThreads = 32 * (kEpiWarps + 2);        // and a producer warp, an issuing warp
constexpr int kTmemCols = 512;                    // two accumulators of [A_hi B_hi (128) | corrections (128)]
constexpr size_t kGemmSmem = (size_t)kStages * (kAStage + kBStage) + 1024;

__device__ int g_gemm_status = 0;

__device__ __forceinline__ float pow2_scale(float amax)
{
    // the power of two that brings `amax` into [2^14, 2^15); 1 for zero, infinite or NaN input
    if (!(amax > 0.0f && amax <= 3.0e38f)) return 1.0f;
    const int e = (int)((__float_as_uint(amax) >> 23) & 0xffu) - 127;
    int sh = 14 - e;
    sh = sh > 126 ? 126 : (sh < -126 ? -126 : sh);
    return __uint_as_float((uint32_t)(127 + sh) << 23);
}
__device__ __forceinline__ float pow2_inverse(float p) { return __uint_as_float(0x7F000000u - __float_as_uint(p)); }

// largest |x| of n floats -> *out (zeroed before the launch; non-negative floats order like their bit patterns)
__global__ void __launch_bounds__(256) gemm_amax_kernel(const float *__restrict__ x, size_t n, float *out)
{
    dependents_may_start();
    float m = 0.0f;
    const size_t tid = (size_t)blockIdx.x * 256 + threadIdx.x, nthr = (size_t)gridDim.x * 256;
    if ((reinterpret_cast<uintptr_t>(x) & 15) == 0) {
        const size_t n4 = n / 4;
        for (size_t i = tid; i < n4; i += nthr) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(x) + i);
            m = fmaxf(m, fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(a.w))));
        }
        for (size_t i = 4 * n4 + tid; i < n; i += nthr) m = fmaxf(m, fabsf(__ldg(x + i)));
    } else {
        for (size_t i = tid; i < n; i += nthr) m = fmaxf(m, fabsf(__ldg(x + i)));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0 && m > 0.0f) atomicMax(reinterpret_cast<unsigned *>(out), __float_as_uint(m));
}

// One warp per row of A (rows up to the padded count: rows past M are zeros).  A lane owns runs of 8 consecutive values
// (one 16-byte chunk of fp16).  Image: stage (mt, kt) at ((mt * KT + kt) * kAStage); block 0 = hi, block 1 = lo; row r,
// chunk c at r * 128 + ((c ^ (r & 7)) * 16).
// With ln_g / ln_b given, the row is layer-normalised first (mean and variance over its N values, eps 1e-5, times gamma
// plus beta: launch_layer_norm_forward, src/hip_kernels.cpp:757-848, to rounding), so that LN + projection of the
// reference's block (src/transformer_layer.cpp:240-241, 246-247) need no pass over memory of their own.
// NV > 0: the row (at most 256 NV values) stays in registers from its one read to the stores; 0: it is read again for every sweep.
template <int NV>
__global__ void __launch_bounds__(128) gemm_pack_a_kernel(const float *__restrict__ A, uint8_t *__restrict__ img, float *__restrict__ row_inv,
                                                           int M, int N, int KT, const float *__restrict__ ln_g, const float *__restrict__ ln_b)
{
    // overlapped launch: placed while the kernel before it drains; waiting for it here also orders the product kernel,
    // which waits for this one, after everything before
    dependency_wait();
    dependents_may_start();
    const int lane = threadIdx.x & 31;
    const int m = blockIdx.x * 4 + (threadIdx.x >> 5);
    const bool live = m < M;
    const float *row = A + (size_t)(live ? m : 0) * N;
    const bool vec = (N & 3) == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    const bool ln_vec = ((reinterpret_cast<uintptr_t>(ln_g) | reinterpret_cast<uintptr_t>(ln_b)) & 15) == 0;
    auto load8 = [&](const float *p, int k0, bool wide, float (&v)[8]) {          // values past N: zeros
        if (wide && k0 + 8 <= N) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(p + k0)), b = __ldg(reinterpret_cast<const float4 *>(p + k0) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = k0 + j < N ? __ldg(p + k0 + j) : 0.0f;
        }
    };
    auto raw8 = [&](int k0, float (&v)[8]) {
        if (live) load8(row, k0, vec, v);
        else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = 0.0f;
        }
    };
    const int depth = KT * kTK;
    // Gamma and beta come with the row, 16 bytes at a time, and wait in registers where the row is short: as 16 loads of 4 bytes per run of eight
    // behind the statistics they made the two normalised packings of a block (1407 rows, E=512) 4 of its 86 us longer.  (Four warps to a long row: 82 -> 88.)
    constexpr bool kHoldLn = NV > 0 && NV <= 2;
    float held[NV > 0 ? NV : 1][8], gm[kHoldLn ? NV : 1][8], bt[kHoldLn ? NV : 1][8];
    if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) raw8(lane * 8 + 256 * i, held[i]);
    }
    if constexpr (kHoldLn) {
        if (ln_g) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                load8(ln_g, lane * 8 + 256 * i, ln_vec, gm[i]);
                load8(ln_b, lane * 8 + 256 * i, ln_vec, bt[i]);
            }
        }
    }
    // f(i, k0, values) for this lane's runs of eight
    auto sweep = [&](auto f) {
        if constexpr (NV > 0) {
#pragma unroll
            for (int i = 0; i < NV; ++i) f(i, lane * 8 + 256 * i, held[i]);
        } else {
            for (int k0 = lane * 8; k0 < depth; k0 += 256) {
                float v[8];
                raw8(k0, v);
                f(0, k0, v);
            }
        }
    };
    auto over_row = [&](float x, auto op) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = op(x, __shfl_xor_sync(0xffffffffu, x, o));
        return x;
    };
    auto add = [](float x, float y) { return x + y; };
    float mean = 0.0f, rstd = 1.0f;
    if (ln_g) {
        float sum = 0.0f;
        sweep([&](int, int, float (&v)[8]) {
#pragma unroll
            for (int j = 0; j < 8; ++j) sum += v[j];             // values past N are zeros
        });
        mean = over_row(sum, add) / (float)N;
        float var = 0.0f;
        sweep([&](int, int k0, float (&v)[8]) {
#pragma unroll
            for (int j = 0; j < 8; ++j) { const float d = (k0 + j < N) ? v[j] - mean : 0.0f; var = fmaf(d, d, var); }
        });
        rstd = 1.0f / sqrtf(over_row(var, add) / (float)N + 1e-5f);
    }
    auto normalised = [&](int i, int k0, float (&v)[8]) {
        if (ln_g) {
            float g8[8], b8[8];
            if constexpr (!kHoldLn) {
                load8(ln_g, k0, ln_vec, g8);
                load8(ln_b, k0, ln_vec, b8);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float g = kHoldLn ? gm[i][j] : g8[j], b = kHoldLn ? bt[i][j] : b8[j];      // (zeros past N)
                v[j] = live && k0 + j < N ? g * (v[j] - mean) * rstd + b : 0.0f;
            }
        }
    };
    float amax = 0.0f;
    sweep([&](int i, int k0, float (&v)[8]) {
        normalised(i, k0, v);                                    // (held in registers: normalised in place)
#pragma unroll
        for (int j = 0; j < 8; ++j) amax = fmaxf(amax, fabsf(v[j]));
    });
    const float s = pow2_scale(over_row(amax, [](float x, float y) { return fmaxf(x, y); }));
    if (lane == 0) row_inv[m] = pow2_inverse(s);
    const int mt = m / kTM, r = m % kTM;
    sweep([&](int i, int k0, float (&v)[8]) {
        if (NV > 0 && k0 >= depth) return;
        if constexpr (NV == 0) normalised(i, k0, v);
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = v[2 * j] * s, b = v[2 * j + 1] * s;
            const float ah = tf32_hi(a), bh = tf32_hi(b);
            hi[j] = pack_f16(ah, bh);
            lo[j] = pack_f16(a - ah, b - bh);
        }
        const int kt = k0 / kTK, c = (k0 % kTK) >> 3;
        uint8_t *stage = img + ((size_t)mt * KT + kt) * kAStage;
        *reinterpret_cast<uint4 *>(stage + sw128(r, c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4 *>(stage + kABlk + sw128(r, c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    });
}

// One block per 8 reduction rows of a (64-deep slice kt, 128-column tile nt) of B [N][K] (N inner, K the output width).
// A thread owns 8 consecutive columns of one reduction row.  Image: stage (nt, kt) at ((nt * KT + kt) * kBStage); reduction row r,
// column block cb (8 columns of [B_hi (128) | B_lo (128)]) at (r / 8) * kGroupStride + cb * 128 + (r % 8) * 16.
__global__ void __launch_bounds__(128) gemm_pack_b_kernel(const float *__restrict__ B, const float *__restrict__ amax, uint8_t *__restrict__ img,
                                                           int N, int K, int KT)
{
    dependency_wait();                               // the largest magnitude has been found
    dependents_may_start();
    const int kt = blockIdx.x >> 3, pass = blockIdx.x & 7, nt = blockIdx.y;
    const float s = pow2_scale(*amax);
    const int cb = threadIdx.x & 15, r0 = threadIdx.x >> 4;      // 16 threads cover the 128 columns of a row, 8 rows per block
    const bool vec = (K & 3) == 0 && (reinterpret_cast<uintptr_t>(B) & 15) == 0;
    uint8_t *stage = img + ((size_t)nt * KT + kt) * kBStage;
    {
        const int r = r0 + 8 * pass;
        const int n = kt * kTK + r, c0 = nt * kTN + 8 * cb;
        float v[8];
        if (n < N && vec && c0 + 8 <= K) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(B + (size_t)n * K + c0)), b = __ldg(reinterpret_cast<const float4 *>(B + (size_t)n * K + c0) + 1);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = (n < N && c0 + j < K) ? __ldg(B + (size_t)n * K + c0 + j) : 0.0f;
        }
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float a = v[2 * j] * s, b = v[2 * j + 1] * s;
            const float ah = tf32_hi(a), bh = tf32_hi(b);
            hi[j] = pack_f16(ah, bh);
            lo[j] = pack_f16(a - ah, b - bh);
        }
        uint8_t *dst = stage + (r >> 3) * kGroupStride + (r & 7) * 16;
        *reinterpret_cast<uint4 *>(dst + cb * 128) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4 *>(dst + (16 + cb) * 128) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
}

__device__ __noinline__ bool gemm_wait_slow(uint64_t *bar, uint32_t parity, int site, volatile int *abort_flag, int expire)
{
    if (!expires_now(expire, site) && mbar_wait(bar, parity)) return true;
    *abort_flag = 1;
    atomicCAS(&g_gemm_status, 0, site);
    linger();
    return false;
}

// KS > 1: the slices of a tile are shared by the KS blocks of a cluster (each one tile, no second one), for products with too few
// tiles for the SMs: a block fetches 64 KB per slice at what L2 gives one SM, about 80 GB/s, so 32 slices on 44 SMs took 25 us.
// The blocks' partial sums meet in shared memory: the tile's columns are dealt out in pieces of 32, every block stores what it
// has of the others' pieces into their (now idle) operand stages and adds up its own, in rank order.
constexpr int kMostSplit = 4;
template <int KS>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_tc_kernel(const uint8_t *__restrict__ aimg, const uint8_t *__restrict__ bimg, const float *__restrict__ row_inv, const float *__restrict__ b_amax,
               const float *__restrict__ bias, float *__restrict__ C, int M, int K, int KT, int NT, int ntiles, int expire)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *base = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *a_s = base;                              // [stage][A_hi block | A_lo block]
    uint8_t *b_s = base + kStages * kAStage;          // [stage][64 deep][B_hi | B_lo]
    __shared__ uint64_t full[kStages], empty[kStages], acc_full[2], acc_empty[2];
    __shared__ __align__(16) float epi[kEpiWarps][32 * 32];  // per epilogue warp: a 32 x 32 piece of the output on its way out
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);      // warp-uniform for the compiler

    if (tid == 0) {
        abort_flag = 0;
        for (int i = 0; i < kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&acc_full[i], 1); mbar_init(&acc_empty[i], kEpiWarps); }
    }
    __syncthreads();
    // site codes in the status word: 1 stage landed, 2 stage free, 3 accumulator complete, 4 accumulator drained
    bool seen = true;                                // what this thread waited for last has come (for who asks for copies then)
    auto wait = [&](uint64_t *bar, uint32_t parity, int site) {
        const int gone = abort_flag;                 // (before the test, and not in its way)
        const bool done = mbar_test(bar, parity);
        seen = !gone;
        if (!gone && !done) seen = gemm_wait_slow(bar, parity, site, &abort_flag, expire);
    };
    // The block takes output tiles blockIdx.x, + gridDim.x, ... (column tile fastest: blocks that run side by side share
    // the rows of A).  Stages are counted through all tiles (g), accumulators alternate between two halves of TMEM, so
    // the copies of the next tile and its products run while the eight epilogue warps drain the tile before it.
    int rank = 0;
    if constexpr (KS > 1) asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int kt0 = rank * KT / KS, kt1 = (rank + 1) * KT / KS, first = (int)blockIdx.x / KS, stride = (int)gridDim.x / KS;

    if (warp == kEpiWarps) {
        // ---- producer: whole stages by bulk copies ----
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        dependents_may_start();
        // What the kernel that packs A does not write is asked for before it has completed: it let this kernel in behind its own wait, so
        // B's images (and magnitude, and the bias) are older.
        auto ask_b = [&](int s, int nt, int kt) {
            mbar_arrive_expect_tx(&full[s], (uint32_t)(kAStage + kBStage));
            const uint8_t *bsrc = bimg + ((size_t)nt * KT + kt) * kBStage;
            bulk_load(b_s + s * kBStage, bsrc, kBStage / 2, &full[s]);
            bulk_load(b_s + s * kBStage + kBStage / 2, bsrc + kBStage / 2, kBStage / 2, &full[s]);
        };
        int early = 0;
        for (int t = first, kt = kt0; early < kStages && t < ntiles; ++early) {
            if (lane == 0) ask_b(early, t % NT, kt);
            if (++kt == kt1) { kt = kt0; t += stride; }
        }
        dependency_wait();                            // A's images are there
        tc_fence_before();
        __syncthreads();                              // TMEM allocated
        int g = 0;
        for (int t = first; t < ntiles; t += stride) {
            const int nt = t % NT, mt = t / NT;
            for (int kt = kt0; kt < kt1; ++kt, ++g) {
                const int s = g % kStages;
                if (g >= kStages) wait(&empty[s], (uint32_t)((g / kStages - 1) & 1), 2);     // the products that read the stage have completed
                if (lane == 0 && seen) {
                    if (g >= early) ask_b(s, nt, kt);
                    const uint8_t *asrc = aimg + ((size_t)mt * KT + kt) * kAStage;
                    bulk_load(a_s + s * kAStage, asrc, kABlk, &full[s]);
                    bulk_load(a_s + s * kAStage + kABlk, asrc + kABlk, kABlk, &full[s]);
                }
                __syncwarp();
            }
        }
        __syncwarp();
        if (abort_flag) linger();
        if constexpr (KS > 1) { cluster_sync(); cluster_sync(); }
        tc_fence_before();
        __syncthreads();                              // the last output has been read from TMEM
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base_slot), "r"(kTmemCols) : "memory");
        return;
    }
    if (warp == kEpiWarps + 1) {
        // ---- issuing warp: stays converged, elects the lane per instruction ----
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        const uint32_t tmem = tmem_base_slot;
        constexpr uint32_t id_wide = idesc_f16(kTM, 2 * kTN) | (1u << 16);       // A_hi x [B_hi | B_lo], B N-major
        constexpr uint32_t id_half = idesc_f16(kTM, kTN) | (1u << 16);           // A_lo x B_hi
        int g = 0, i = 0;
        for (int t = first; t < ntiles; t += stride, ++i) {
            const uint32_t acc = tmem + (uint32_t)((i & 1) * 2 * kTN);
            if (i >= 2) wait(&acc_empty[i & 1], (uint32_t)((i / 2 - 1) & 1), 4);             // the epilogue has read this half's previous tile
            tc_fence_after();
            for (int kt = kt0; kt < kt1; ++kt, ++g) {
                const int s = g % kStages;
                wait(&full[s], (uint32_t)((g / kStages) & 1), 1);
                tc_fence_after();
                const uint64_t da_hi = make_desc(smem_u32(a_s + s * kAStage), 16, 1024, 2);
                const uint64_t da_lo = make_desc(smem_u32(a_s + s * kAStage + kABlk), 16, 1024, 2);
                // N-major B without swizzle: lbo = bytes between groups of 8 reduction rows, sbo = bytes between blocks of 8 columns
                const uint64_t db = make_desc(smem_u32(b_s + s * kBStage), kGroupStride, 128, 0);
#pragma unroll
                for (int k = 0; k < kTK / 16; ++k)    // 16 deep = 32 bytes of an A row = two groups of B
                    if (elect_one()) mma_h_ss(acc, da_hi + (uint64_t)(2 * k), db + (uint64_t)(k * 2 * (kGroupStride >> 4)), id_wide, (kt > kt0 || k) ? 1u : 0u);
#pragma unroll
                for (int k = 0; k < kTK / 16; ++k)
                    if (elect_one()) mma_h_ss(acc + kTN, da_lo + (uint64_t)(2 * k), db + (uint64_t)(k * 2 * (kGroupStride >> 4)), id_half, 1u);
                if (elect_one()) tc_commit(&empty[s]);
            }
            if (elect_one()) tc_commit(&acc_full[i & 1]);
        }
        __syncwarp();
        if (abort_flag) linger();
        if constexpr (KS > 1) { cluster_sync(); cluster_sync(); }
        tc_fence_before();
        __syncthreads();
        return;
    }

    // ---- epilogue warps: thread = output row = TMEM lane ----
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const float b_inv = pow2_inverse(pow2_scale(__ldg(b_amax)));
    const bool vec = (K & 3) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
    const int quarter = warp & 3, half = warp >> 2;   // its rows; its pieces of 32 columns: half, half + 2
    const int ch = lane & 7;                          // of a piece it stores columns 4 ch ... 4 ch + 3
    int i = 0;
    for (int t = first; t < ntiles; t += stride, ++i) {
        const int nt = t % NT, mt = t / NT;
        const int r = quarter * 32 + lane, m = mt * kTM + r;
        const uint32_t lane_base = tmem_base_slot + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((i & 1) * 2 * kTN);
        const float unscale = (m < M ? __ldg(row_inv + m) : 0.0f) * b_inv;
        // the bias is on its way while the products run: asked for behind them, piece by piece, it cost 2.8 us per tile
        float4 bias4[2] = {make_float4(0.f, 0.f, 0.f, 0.f), make_float4(0.f, 0.f, 0.f, 0.f)};
        if (bias) {
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const int col = nt * kTN + 32 * (half + 2 * p) + 4 * ch;
                bias4[p] = make_float4(col < K ? __ldg(bias + col) : 0.0f, col + 1 < K ? __ldg(bias + col + 1) : 0.0f,
                                       col + 2 < K ? __ldg(bias + col + 2) : 0.0f, col + 3 < K ? __ldg(bias + col + 3) : 0.0f);
            }
        }
        wait(&acc_full[i & 1], (uint32_t)((i / 2) & 1), 3);
        tc_fence_after();
        const int c_base = nt * kTN;
        bool live = !abort_flag;
        // 32 columns at a time; the warp turns its 32 x 32 piece through shared memory (16-byte chunk c of row r at
        // r * 128 + ((c ^ (r & 7)) * 16)) so that a store instruction writes four rows of 128 contiguous bytes instead
        // of 32 rows of 16
        uint8_t *tb = reinterpret_cast<uint8_t *>(epi[warp]);
        // (KS > 1) piece c of the columns belongs to block c * KS / 4; what block q has of it lies in the owner's stages, q's place
        // among the others first: [place][piece of the owner's (at most 2)][column / 4][row] of 16 bytes
        auto parked = [&](int q, int owner, int c) {
            const int place = q < owner ? q : q - 1, lc = c - (owner * 4 + KS - 1) / KS;
            return (uint32_t)((place * 2 + lc) * (8 * kTM * 16) + r * 16);
        };
        if constexpr (KS > 1) {
            cluster_sync();                           // every block of the cluster is done with its operand stages, and with its waits
            // a tile whose sum is unfinished in one block is stored by none (the loads are used behind the exchange)
            uint32_t gone[KS];
#pragma unroll
            for (int q = 0; q < KS; ++q)
                asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.b32 %0, [a];\n\t}"
                             : "=r"(gone[q]) : "r"(smem_u32(const_cast<const int *>(&abort_flag))), "r"(q) : "memory");
#pragma unroll 1
            for (int c = half; c < 4; c += 2) {
                const int owner = c * KS / 4;
                if (owner == rank) continue;
                float a[32], b[32];
                tmem_ld32(lane_base + 32 * c, a);
                tmem_ld32(lane_base + kTN + 32 * c, b);
                tmem_wait_ld();
                uint32_t dst;
                asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_u32(base) + parked(rank, owner, c)), "r"(owner));
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(dst + j * (kTM * 16)), "f"(a[4 * j] + b[4 * j]), "f"(a[4 * j + 1] + b[4 * j + 1]),
                                 "f"(a[4 * j + 2] + b[4 * j + 2]), "f"(a[4 * j + 3] + b[4 * j + 3]) : "memory");
            }
#pragma unroll
            for (int q = 0; q < KS; ++q) live = live && gone[q] == 0;
            cluster_sync();
        }
#pragma unroll (KS > 1 ? 1 : 2)
        for (int p = 0; p < 2; ++p) {
            const int c0 = 32 * (half + 2 * p);
            if (KS > 1 && (c0 / 32) * KS / 4 != rank) continue;
            float a[32], b[32];
            tmem_ld32(lane_base + c0, a);             // A_hi B_hi
            tmem_ld32(lane_base + kTN + c0, b);       // the correction terms
            tmem_wait_ld();
            if constexpr (KS > 1) {
#pragma unroll
                for (int x = 0; x < 32; ++x) { b[x] += a[x]; a[x] = 0.0f; }                  // b: this block's share
#pragma unroll
                for (int q = 0; q < KS; ++q) {
                    const uint8_t *src = base + (q == rank ? 0 : parked(q, rank, c0 / 32));
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float4 y = q == rank ? make_float4(b[4 * j], b[4 * j + 1], b[4 * j + 2], b[4 * j + 3])
                                                   : *reinterpret_cast<const float4 *>(src + j * (kTM * 16));
                        a[4 * j] += y.x; a[4 * j + 1] += y.y; a[4 * j + 2] += y.z; a[4 * j + 3] += y.w;
                    }
                }
#pragma unroll
                for (int x = 0; x < 32; ++x) b[x] = 0.0f;
            }
            if (c_base + c0 >= K) continue;           // warp-uniform: a tile past the last column
#pragma unroll
            for (int j4 = 0; j4 < 8; ++j4) {
                float o[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) o[j] = (a[4 * j4 + j] + b[4 * j4 + j]) * unscale;     // (a power of two)
                *reinterpret_cast<float4 *>(tb + lane * 128 + ((j4 ^ (lane & 7)) << 4)) = make_float4(o[0], o[1], o[2], o[3]);
            }
            __syncwarp();
            const int col = c_base + c0 + 4 * ch;
            const float4 bp = p ? bias4[1] : bias4[0];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int rr = 4 * i + (lane >> 3);
                const int mrow = mt * kTM + quarter * 32 + rr;
                float4 val = *reinterpret_cast<const float4 *>(tb + rr * 128 + ((ch ^ (rr & 7)) << 4));
                val.x += bp.x; val.y += bp.y; val.z += bp.z; val.w += bp.w;
                if (live && mrow < M) {
                    float *dst = C + (size_t)mrow * K + col;
                    if (vec && col + 4 <= K) {
                        *reinterpret_cast<float4 *>(dst) = val;
                    } else {
                        if (col < K) dst[0] = val.x;
                        if (col + 1 < K) dst[1] = val.y;
                        if (col + 2 < K) dst[2] = val.z;
                        if (col + 3 < K) dst[3] = val.w;
                    }
                }
            }
            __syncwarp();                             // the piece is out before the next one is staged
        }
        // this half of TMEM may take the tile after next
        tc_fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[i & 1])) : "memory");
    }
    tc_fence_before();
    __syncthreads();
}

StreamWorkspace g_gemm;                              // the packed operands of a call

}  // namespace

void gemm_tc_release_scratch() { g_gemm.release(); }

int gemm_tc_status_fetch(int *status)
{
    int v = 0;
    const cudaError_t e = cudaMemcpyFromSymbol(&v, g_gemm_status, sizeof(v));
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    if (v) { const int zero = 0; cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(zero)); }
    *status = v;
    return HIPGPT_OK;
}

namespace {

int set_gemm_attr(int dev)
{
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e = once_per_device(done, dev, [] {
        cudaError_t r = cudaSuccess;
        for (auto kern : {gemm_tc_kernel<1>, gemm_tc_kernel<2>, gemm_tc_kernel<3>, gemm_tc_kernel<4>})
            if (r == cudaSuccess) r = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
        return r;
    });
    return e == cudaSuccess ? HIPGPT_OK : fail(HIPGPT_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
}

// How many clusters of `ks` blocks of the product kernel the device holds at the same time (a property of the device: asked for once on each)
int clusters_at_once(int dev, int ks)
{
    static std::atomic<int> known[64][kMostSplit + 1];
    std::atomic<int> *cell = dev >= 0 && dev < 64 ? &known[dev][ks] : nullptr;
    if (cell && cell->load(std::memory_order_relaxed) > 0) return cell->load(std::memory_order_relaxed);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3((unsigned)(ks * 148));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = kGemmSmem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, ks == 2 ? gemm_tc_kernel<2> : ks == 3 ? gemm_tc_kernel<3> : gemm_tc_kernel<4>, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    if (cell) cell->store(n, std::memory_order_relaxed);
    return n;
}

// B -> its stage images and its largest magnitude (three launches on `st`; the first is a plain one, so everything
// enqueued before has completed when the images are written)
int pack_b(const float *B, int N, int K, uint8_t *bimg, float *b_amax, cudaStream_t st)
{
    const int NT = (K + kTN - 1) / kTN, KT = (N + kTK - 1) / kTK;
    cudaError_t e = cudaMemsetAsync(b_amax, 0, sizeof(float), st);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    const size_t nb = (size_t)N * K;
    size_t ablocks = (nb + 256 * 4 - 1) / (256 * 4);
    if (ablocks > 1184) ablocks = 1184;
    gemm_amax_kernel<<<(unsigned)ablocks, 256, 0, st>>>(B, nb, b_amax);
    int rc = check_launch("gemm_amax_kernel");
    if (rc != HIPGPT_OK) return rc;
    e = launch_overlapped(gemm_pack_b_kernel, dim3((unsigned)(KT * (kTK / 8)), (unsigned)NT), dim3(128), 0, st, B, (const float *)b_amax, bimg, N, K, KT);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "gemm_pack_b_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("gemm_pack_b_kernel");
}

// A -> its stage images, then the product kernel, with B's images given
int pack_a_and_multiply(const float *A, const uint8_t *bimg, const float *b_amax, const float *bias, float *C, int M, int N, int K,
                        uint8_t *aimg, float *row_inv, int dev, cudaStream_t st, const float *ln_g = nullptr, const float *ln_b = nullptr)
{
    const int MT = (M + kTM - 1) / kTM, NT = (K + kTN - 1) / kTN, KT = (N + kTK - 1) / kTK;
    cudaError_t e;
    const auto pack = KT <= 4 ? gemm_pack_a_kernel<1> : KT <= 8 ? gemm_pack_a_kernel<2> : KT <= 16 ? gemm_pack_a_kernel<4> : KT <= 32 ? gemm_pack_a_kernel<8> : gemm_pack_a_kernel<0>;
    e = launch_overlapped(pack, dim3((unsigned)(MT * kTM / 4)), dim3(128), 0, st, A, aimg, row_inv, M, N, KT, ln_g, ln_b);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "gemm_pack_a_kernel launch: %s", cudaGetErrorString(e));
    int rc = check_launch("gemm_pack_a_kernel");
    if (rc != HIPGPT_OK) return rc;
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
    const long long ntiles = (long long)MT * NT;
    if (ntiles > 2147483647LL) return fail(HIPGPT_ERR_BAD_ARG, "%lld output tiles are too many", ntiles);
    // Too few tiles: the slices of a tile on up to four SMs, two slices each at least, and as many clusters at
    // the same time as there are tiles: one that waits for another costs the whole product again (148 SMs in clusters of four are 33 clusters, not 37:
    // 1152 x 2048 x 512, 36 tiles, 23.9 -> 17.7 us; 640 x 1024 x 896, 35 tiles, 17.7 -> 13.0).
    // A sixteenth of the places stays free where the block more does not pay for the last ones (us back to back):
    //   threes of fewer than 16 slices: the last places are found only when the SMs come free in the right order, of 45 that fit 43 - 45 tiles waited
    //     (44 tiles: 8 slices 9.8, threes 12.7; 12 slices 12.0, 14.2; a block of 1407 rows, E=512 81.9 -> 80.1 with this);
    //   pairs of fewer than 8 slices: one block alone is the faster (72 tiles: 4 slices 7.9, pairs 8.8; 6 slices 9.5, 9.7; 8 slices 10.6, 10.3; 12 slices 13.5, 12.6).
    // Fours leave none (33 tiles: 8 slices 10.05, threes 10.3; 31 tiles, 12 slices 12.3, 12.7).
    // Fewer blocks per tile than this would often be faster (32 tiles of 16 slices in pairs 12.2, fours 13.0; 44 of 32 in pairs 17.9, threes 18.8; fewer than 8
    // slices alone), but the sum that one block keeps in TMEM is then longer and its error larger: 6.2e-7 instead of 3.4e-7 of the result's norm for
    // 6 slices alone instead of on three blocks, 1.37e-6 instead of 0.97e-6 for 32 on two.
    auto leaves_some = [&](int n) { return (n == 3 && KT < 16) || (n == 2 && KT < 8); };
    int ks = 1;
    while (ks < kMostSplit && ntiles * (ks + 1) <= sms && KT >= 2 * (ks + 1) && ntiles * 16 <= (leaves_some(ks + 1) ? 15LL : 16LL) * clusters_at_once(dev, ks + 1)) ++ks;
    const unsigned grid = ks > 1 ? (unsigned)(ntiles * ks) : (unsigned)(ntiles < sms ? ntiles : sms);      // ks = 1: one block per SM, each takes tiles in turn
    const auto kern = ks == 1 ? gemm_tc_kernel<1> : ks == 2 ? gemm_tc_kernel<2> : ks == 3 ? gemm_tc_kernel<3> : gemm_tc_kernel<4>;
    e = launch_overlapped_clusters(kern, ks, dim3(grid), dim3(kGemmThreads), kGemmSmem, st, (const uint8_t *)aimg, bimg,
                                   (const float *)row_inv, b_amax, bias, C, M, K, KT, NT, (int)ntiles, take_expiry(500));
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "gemm_tc_kernel launch: %s", cudaGetErrorString(e));
    return check_launch("gemm_tc_kernel");
}

}  // namespace

// C[M][K] = A[M][N] B[N][K] (+ bias), fp32-grade on the tensor pipe.  C must not alias A or B.
int launch_matmul_tc(const float *A, const float *B, const float *bias, float *C, int M, int N, int K, cudaStream_t st, const float *ln_g, const float *ln_b)
{
    const int MT = (M + kTM - 1) / kTM, NT = (K + kTN - 1) / kTN, KT = (N + kTK - 1) / kTK;
    if (MT > 65535) return fail(HIPGPT_ERR_BAD_ARG, "M = %d is beyond %d rows per call", M, 65535 * kTM);
    if (KT == 0) return fail(HIPGPT_ERR_BAD_ARG, "an inner dimension of 0");
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    const size_t abytes = (size_t)MT * KT * kAStage, bbytes = (size_t)NT * KT * kBStage, rbytes = ((size_t)MT * kTM * sizeof(float) + 255) & ~(size_t)255;
    StreamWorkspace::Lease ws;
    int rc = g_gemm.enter(st, abytes + bbytes + rbytes + 256, &ws);
    if (rc != HIPGPT_OK) return rc;
    uint8_t *scratch = ws.get(), *aimg = scratch, *bimg = scratch + abytes;
    float *row_inv = reinterpret_cast<float *>(scratch + abytes + bbytes), *b_amax = reinterpret_cast<float *>(scratch + abytes + bbytes + rbytes);
    rc = set_gemm_attr(dev);
    if (rc == HIPGPT_OK) rc = pack_b(B, N, K, bimg, b_amax, st);
    if (rc != HIPGPT_OK) return rc;
    return pack_a_and_multiply(A, bimg, b_amax, bias, C, M, N, K, aimg, row_inv, dev, st, ln_g, ln_b);
}

// ---- a right-hand side packed once (the weights of a layer) and used by many products ---------------------------
struct PackedB {
    int dev, N, K;
    uint8_t *bimg;
    float *b_amax;
};

int matmul_tc_prepare(const float *B, int N, int K, PackedB **out, cudaStream_t st)
{
    const int NT = (K + kTN - 1) / kTN, KT = (N + kTK - 1) / kTK;
    if (KT == 0 || NT == 0) return fail(HIPGPT_ERR_BAD_ARG, "an empty right-hand side: N=%d K=%d", N, K);
    PackedB *p = new PackedB{0, N, K, nullptr, nullptr};
    cudaError_t e = cudaGetDevice(&p->dev);
    const size_t bbytes = (size_t)NT * KT * kBStage;
    if (e == cudaSuccess) e = cudaMalloc(&p->bimg, bbytes + 256);
    if (e != cudaSuccess) { delete p; return fail(HIPGPT_ERR_CUDA, "cudaMalloc(%zu) for the packed right-hand side: %s", bbytes + 256, cudaGetErrorString(e)); }
    p->b_amax = reinterpret_cast<float *>(p->bimg + bbytes);
    const int rc = pack_b(B, N, K, p->bimg, p->b_amax, st);
    if (rc != HIPGPT_OK) { cudaFree(p->bimg); delete p; return rc; }
    *out = p;
    return HIPGPT_OK;
}

void matmul_tc_release(PackedB *p)
{
    if (!p) return;
    cudaFree(p->bimg);                               // waits for the kernels that read it
    delete p;
}

int launch_matmul_tc_prepared(const float *A, const PackedB *b, const float *bias, float *C, int M, cudaStream_t st, const float *ln_g, const float *ln_b)
{
    const int N = b->N, K = b->K;
    const int MT = (M + kTM - 1) / kTM, KT = (N + kTK - 1) / kTK;
    if (MT > 65535) return fail(HIPGPT_ERR_BAD_ARG, "M = %d is beyond %d rows per call", M, 65535 * kTM);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
    if (dev != b->dev) return fail(HIPGPT_ERR_BAD_ARG, "the right-hand side was packed on device %d, the current device is %d", b->dev, dev);
    const size_t abytes = (size_t)MT * KT * kAStage, rbytes = ((size_t)MT * kTM * sizeof(float) + 255) & ~(size_t)255;
    StreamWorkspace::Lease ws;
    int rc = g_gemm.enter(st, abytes + rbytes, &ws);
    if (rc != HIPGPT_OK) return rc;
    uint8_t *scratch = ws.get();
    rc = set_gemm_attr(dev);
    if (rc != HIPGPT_OK) return rc;
    return pack_a_and_multiply(A, b->bimg, b->b_amax, bias, C, M, N, K, scratch, reinterpret_cast<float *>(scratch + abytes), dev, st, ln_g, ln_b);
}

}  // namespace hipgpt
