// Attention backward on the Blackwell tensor pipe (tcgen05 + TMEM), head_dim 32 or 64, any sequence length, with the accuracy of
// fp32 sums over the range that is stated below.  Same contract as attn_bwd.cu (HipGPT src/hip_kernels.cpp:1162-1272), which keeps every other head_dim:
//     vd_ij = g_i . V_j            w_i  = sum_j P_ij vd_ij        ds_ij = P_ij (vd_ij - w_i)
//     dQ_i  = c sum_j ds_ij K_j    dK_j = c sum_i ds_ij Q_i       dV_j  = sum_i P_ij g_i
//
// Arithmetic.  An fp32 number, brought near 2^14 by a power of two, is the sum of two fp16 numbers to 2^-23 of it.  A product of two
// such sums is formed from three products of the pieces, lo hi, hi lo, hi hi, which the tensor core multiplies exactly and adds in
// fp32 (lo lo, below 2^-22 of the product, where it comes in the same instruction).  The tensor core truncates where it adds to its
// accumulator; what that takes on the average is given back at the end.  Before, three bf16 pieces and six products: twice the instructions and half as
// many bytes more per operand (B=3 H=12 S=777 D=64 causal 117 -> 79 us), and the relative error of the gradients against float64 no smaller where P is formed here:
// 2.8, 3.1, 2.6e-7 then and 2.1, 2.3, 1.9e-7 now (dQ, dK, dV).  Stored probabilities are exact, and so is dO: there two pieces' 23 bits
// showed in dV (1.11 -> 1.17e-7 at B=2 H=16 S=1024 D=64, 0.90 -> 0.97e-7 at S=200), so that this one product keeps three bf16 pieces and six products
// (1.11 and 0.90e-7; 143 -> 165 us and 28.2 -> 29.5).  dQ and dK are 1.60 and 1.57e-7 there, 1.73 and 1.78e-7 with six products throughout (208 us).
// Powers of two: one per 64-row tile for Q, K, V and dO, kept beside the images; for P and ds, which are formed in fp32 in registers,
// one per thread (32 columns of a row or key of a tile).  An accumulator holds one tile and one half of its columns, and the factors leave
// where the workers add it to the running sum; those of a tile's scores go into the multiply-adds that form P and ds.  The low piece is kept 2^12 times too
// large (the tensor core brings the accumulator down by as much between the products), so that a value keeps its 23 bits down to 2^-29 of the largest of its
// tile, and below that what the largest leaves of it: 2^-52 of that one.  (With both pieces at one scale: 2^-15 and 2^-39; a row of dO 2^-30 below its
// neighbours gave nine bits of dQ.  The times are the same: B=3 H=12 S=777 D=64 causal 79.0 -> 79.6 us.)
//
// Three kernels per group of batches:
//   bwd_pack_kernel   Q, K, V, dO -> their pieces, once per call, in the order in which shared memory holds an operand: 8 x 8 core
//                     matrices of 128 bytes, [8-row block][piece][8-column block].  The same bytes serve as a K-major operand (rows =
//                     M or N) and as an N-major one (rows = the reduction), so a tile is fetched with one bulk copy and used for
//                     both products in which it takes part.  Rows up to the next multiple of 128 are zeros.
//   bwd_rows_kernel   128 query rows per block (TMEM lane = row), 64-key tiles.  First sweep: S = Q K^T (where P is not given) and
//                     dP = dO V^T; per row the maximum and sum of exponentials and w_i.  Second sweep: S and dP again, ds to TMEM as
//                     the A operand, dQ += ds K.
//   bwd_cols_kernel   128 keys per block (lane = key), 64-query tiles: S^T = K Q^T, dP^T = V dO^T, P^T and ds^T to TMEM as A operands,
//                     dV += P^T dO, dK += ds^T Q, queries ascending.
// Nothing is added atomically: each output has one owner and a fixed order, results are the same bits on every run.
//
// Eight worker warps (two per TMEM lane quarter, each 32 of the tile's 64 columns) and two issuing warps, which also fetch and
// issue side by side.  Two score buffers in TMEM: the products of tile i + 1 run while the workers are at tile i.  Every wait is bounded: on expiry the
// block raises a flag that cuts later waits short, records a status code, skips its stores, lets what is on its way land, frees its
// TMEM and returns.
#include "attn_bwd_pieces.cuh"
#include "stream_workspace.hpp"
#include "tma_host.cuh"

#include <math.h>
#include <type_traits>

namespace hipgpt {
namespace {

constexpr int kWorkerWarps = 8;
constexpr int kThreads = kWorkerWarps * 32 + 64;
constexpr uint32_t kTmemCols = 512;

__device__ int g_bwd_status = 0;

__device__ __noinline__ bool bwd_wait_slow(uint64_t *bar, uint32_t parity, int site, volatile int *abort_flag, int expire)
{
    if (!expires_now(expire, site) && mbar_wait(bar, parity)) return true;
    *abort_flag = 1;
    atomicCAS(&g_bwd_status, 0, site);
    linger();
    return false;
}

// ---- the pieces of the four planes ---------------------------------------------------------------------
// A block takes a 64-row tile of a head in one plane, a warp 8 of its rows: lane = (column block of 8) * 8 + row, so that it reads 8 whole lines and
// writes core matrices of 128 contiguous bytes per piece.  fac: [plane][tile], what an image is multiplied by to give the plane.  The tile's
// largest magnitude counts finite values only: an infinity becomes NaN in its own row and the tile's other rows keep their scale.
// exact_g: where dO's three bf16 pieces go, for dV of stored probabilities.  Bound by memory: 4 bytes read and 4 written per element (dO's: 10).
template <int D>
__global__ void __launch_bounds__(256)
bwd_pack_kernel(const float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v, const float *__restrict__ g,
                uint8_t *__restrict__ img, size_t img_bytes, float *__restrict__ fac, uint8_t *__restrict__ exact_g, int S, int nt, int E, int H)
{
    constexpr int PARTS = D / 32;
    __shared__ uint32_t red[8];
    dependency_wait();
    dependents_may_start();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = (int)blockIdx.x % nt, bh = (int)blockIdx.x / nt;
    const int r = lane & 7, row = t * kTile + warp * 8 + r;
    const float *src = blockIdx.y == 0 ? q : blockIdx.y == 1 ? k : blockIdx.y == 2 ? v : g;
    float4 x[PARTS][2];
    uint32_t mx = 0;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
        x[p][0] = x[p][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < S) {
            const float4 *at = reinterpret_cast<const float4 *>(src + ((size_t)(bh / H) * S + row) * E + (size_t)(bh % H) * D + p * 32 + (lane >> 3) * 8);
            x[p][0] = __ldg(at);
            x[p][1] = __ldg(at + 1);
        }
    }
#pragma unroll
    for (int p = 0; p < PARTS; ++p)
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const uint32_t m = __float_as_uint(reinterpret_cast<const float *>(&x[p][c])[u]) & 0x7fffffffu;
                mx = m < 0x7f800000u ? max(mx, m) : mx;
            }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) red[warp] = mx;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i) mx = max(mx, red[i]);
    const uint32_t e = range_exponent(mx);
    const float up = range_up(e);
    if (threadIdx.x == 0) fac[(size_t)blockIdx.y * gridDim.x + blockIdx.x] = range_down(e);
    uint8_t *dst = img + blockIdx.y * img_bytes + (size_t)blockIdx.x * Img<D>::kTileBytes + warp * Img<D>::kBlock + (lane >> 3) * 128 + r * 16;
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
        uint4 h, l;
        cut2(make_float2(x[p][0].x * up, x[p][0].y * up), h.x, l.x);
        cut2(make_float2(x[p][0].z * up, x[p][0].w * up), h.y, l.y);
        cut2(make_float2(x[p][1].x * up, x[p][1].y * up), h.z, l.z);
        cut2(make_float2(x[p][1].z * up, x[p][1].w * up), h.w, l.w);
        *reinterpret_cast<uint4 *>(dst + p * 512) = h;
        *reinterpret_cast<uint4 *>(dst + p * 512 + Img<D>::kPiece) = l;
    }
    if (exact_g && blockIdx.y == 3) {
        dst = exact_g + (size_t)blockIdx.x * kTileBytes3<D> + warp * kBlock3<D> + (lane >> 3) * 128 + r * 16;
#pragma unroll
        for (int p = 0; p < PARTS; ++p) {
            uint4 pc[3];
            cut3(make_float2(x[p][0].x, x[p][0].y), pc[0].x, pc[1].x, pc[2].x);
            cut3(make_float2(x[p][0].z, x[p][0].w), pc[0].y, pc[1].y, pc[2].y);
            cut3(make_float2(x[p][1].x, x[p][1].y), pc[0].z, pc[1].z, pc[2].z);
            cut3(make_float2(x[p][1].z, x[p][1].w), pc[0].w, pc[1].w, pc[2].w);
#pragma unroll
            for (int z = 0; z < 3; ++z) *reinterpret_cast<uint4 *>(dst + p * 512 + z * Img<D>::kPiece) = pc[z];
        }
    }
}

// ---- the products, issued by one converged warp that elects the lane per instruction ---------------------
// D[tmem] (128 x 64) = A B^T over the head dimension; A: 128 rows, B: 64 rows, both images read K-major.
template <int D>
__device__ __forceinline__ void issue_scores(uint32_t d_tmem, uint32_t a_smem, uint32_t b_smem)
{
    const uint64_t a = make_desc(a_smem, 128, Img<D>::kBlock, 0), b = make_desc(b_smem, 128, Img<D>::kBlock, 0);
    constexpr uint32_t id = idesc_f16(kLanes, kTile);
    constexpr int PA[3] = {1, 0, 0}, PB[3] = {0, 1, 0};      // small terms first
#pragma unroll
    for (int p = 0; p < 3; ++p)
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            const uint64_t da = a + (uint64_t)((PA[p] * (D / 8) + 2 * k) * 8), db = b + (uint64_t)((PB[p] * (D / 8) + 2 * k) * 8);
            if (elect_one()) {
                if (p == 2 && k == 0) mma_h_ss_down<kLowShift>(d_tmem, da, db, id);
                else mma_h_ss(d_tmem, da, db, id, (p | k) ? 1u : 0u);
            }
        }
}

// acc[tmem] (128 x D) = A B over rows [32 hf, 32 hf + 32) of B's image, read N-major; A: two pieces in TMEM, 16 columns each, hi first.
// WIDE: acc is 2 D columns, the second half collects the products with B's lo pieces, 2^12 times (wider instructions, fewer of them).  The
// small products come first: the tensor core truncates where it adds to its accumulator, so the accumulator should be small
// while they are added, and it starts anew for every tile (the workers add the tiles up in registers).  One accumulator over all
// tiles was 10 times farther from float64 at S = 777.
// LOLO: lo x lo too (WIDE has it in any case), for stored probabilities, which are exact: without it dQ was 1.66e-7 instead of 1.60e-7 from float64 at S = 1024, D = 64, about 1 us less of 165;
// probabilities formed again carry more than it takes away.
template <int D, bool WIDE, bool LOLO>
__device__ __forceinline__ void issue_accumulate(uint32_t acc, uint32_t a_tmem, uint32_t b_smem, int hf)
{
    const uint64_t b = make_desc(b_smem, Img<D>::kBlock, 128, 0) + (uint64_t)(hf * 4 * (Img<D>::kBlock >> 4));
    constexpr uint32_t id = idesc_f16(kLanes, WIDE ? 2 * D : D) | (1u << 16);
    enum { kFresh, kDown, kMore };                   // how a product finds the accumulator
    auto product = [&](int pa, int pb, int start) {
#pragma unroll
        for (int ks = 0; ks < 2; ++ks) {
            const uint64_t bk = b + (uint64_t)(ks * 2 * (Img<D>::kBlock >> 4) + pb * (Img<D>::kPiece >> 4));
            const uint32_t ak = a_tmem + 16 * pa + 8 * ks;
            if (elect_one()) {
                if (start == kDown && ks == 0) mma_h_ts_down<kLowShift>(acc, ak, bk, id);
                else mma_h_ts(acc, ak, bk, id, (start == kFresh && ks == 0) ? 0u : 1u);
            }
        }
    };
    if (!WIDE && LOLO) product(1, 1, kFresh);
    product(1, 0, WIDE || !LOLO ? kFresh : kDown);   // lo x hi (WIDE: lo x [hi | lo])
    if (!WIDE) product(0, 1, kMore);                 // hi x lo
    product(0, 0, kDown);                            // hi x hi (WIDE: hi x [hi | lo])
}

// acc[tmem] (128 x D) = A B over the 64 rows of B's image of three pieces, read N-major; A: three pieces in TMEM, 32 columns each
template <int D>
__device__ __forceinline__ void issue_exact(uint32_t acc, uint32_t a_tmem, uint32_t b_smem)
{
    const uint64_t b = make_desc(b_smem, kBlock3<D>, 128, 0);
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
            if (elect_one())
                mma_h_ts(acc, a_tmem + 32 * kExactA[p] + 8 * ks, b + (uint64_t)(ks * 2 * (kBlock3<D> >> 4) + kExactB[p] * (Img<D>::kPiece >> 4)), idesc_bf16(kLanes, D, 1), p + ks > 0 ? 1u : 0u);
}

// 32 numbers of a row (or key), scaled by a power of two of their own -> their two pieces in 32 TMEM columns, hi first.  Returns one
// over the factor.
__device__ __forceinline__ float store_pieces(const float (&x)[32], uint32_t addr)
{
    float m4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 32; c += 2) m4[(c >> 1) & 3] = max3(m4[(c >> 1) & 3], fabsf(x[c]), fabsf(x[c + 1]));
    const uint32_t e = range_exponent(__float_as_uint(max3(fmaxf(m4[0], m4[1]), m4[2], m4[3])));
    const float up = range_up(e);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t h[8], l[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) cut2(fmul2(make_float2(x[16 * half + 2 * c], x[16 * half + 2 * c + 1]), make_float2(up, up)), h[c], l[c]);
        tmem_st8_u32(addr + 8 * half, h);
        tmem_st8_u32(addr + 16 + 8 * half, l);
    }
    return range_down(e);
}

// 32 probabilities of a key (half of a tile's queries) -> their three pieces, 32 TMEM columns apart, 16 columns each
__device__ __forceinline__ void store_exact(const float (&x)[32], uint32_t addr)
{
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t pc[3][8];
#pragma unroll
        for (int c = 0; c < 8; ++c) cut3(make_float2(x[16 * half + 2 * c], x[16 * half + 2 * c + 1]), pc[0][c], pc[1][c], pc[2][c]);
#pragma unroll
        for (int z = 0; z < 3; ++z) tmem_st8_u32(addr + 32 * z + 8 * half, pc[z]);
    }
}
// Adds a tile's accumulator of the exact products (this thread's D / 2 columns of its key) to the running sum
template <int D>
__device__ __forceinline__ void add_exact(uint32_t acc, int hf, float (&o)[D / 2])
{
#pragma unroll
    for (int c0 = 0; c0 < D / 2; c0 += 16) {
        float a[16];
        tmem_ld16(acc + hf * (D / 2) + c0, a);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; ++c) o[c0 + c] += a[c];
    }
}

// Adds a tile's two accumulators (one per half of its columns; this thread's D / 2 columns of its row) times their factors to the running sum
template <int D, bool WIDE>
__device__ __forceinline__ void add_tile(uint32_t acc, int hf, float f0, float f1, float (&o)[D / 2])
{
    constexpr int kAcc = WIDE ? 2 * D : D;
#pragma unroll
    for (int c0 = 0; c0 < D / 2; c0 += 16) {
        float a[2][16], b[2][16];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            tmem_ld16(acc + u * kAcc + hf * (D / 2) + c0, a[u]);
            if (WIDE) tmem_ld16(acc + u * kAcc + D + hf * (D / 2) + c0, b[u]);
        }
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
            float2 y[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                y[u] = make_float2(a[u][c], a[u][c + 1]);
                if (WIDE) y[u] = ffma2(make_float2(b[u][c], b[u][c + 1]), make_float2(kLowDown, kLowDown), y[u]);
            }
            // (the halves first: one addition to the long sum per tile)
            const float2 t = fadd2(make_float2(o[c0 + c], o[c0 + c + 1]), ffma2(y[1], make_float2(f1, f1), fmul2(y[0], make_float2(f0, f0))));
            o[c0 + c] = t.x;
            o[c0 + c + 1] = t.y;
        }
    }
}

// The tensor core cuts off, towards zero, what does not fit where it adds to its accumulator: results come out smaller by so much on the
// average, whatever the sizes (measured against float64: 5.1 - 5.5e-8 behind the one product of dV, 1.2 - 1.4e-7 behind the two of dQ and dK).
// It is given back with the last multiplication.
constexpr float kSumLoss = 5.4e-8f, kScoreLoss = 1.3e-7f;

// A warp's 32 rows x D / 2 results leave in whole lines: through shared memory (boxes of 32 x 32, 16-byte pieces permuted by the row; at head_dim
// 32 the two warps of a quarter share one), then a row of 128 bytes per eight lanes.  A thread's own stores touched 32 lines
// each (1.2 us at the end of a 10.7 us block of columns).  dst: the head's first column of the warp's first row.
template <int D>
__device__ __forceinline__ void store_out(const float (&o)[D / 2], int warp, int lane, float scale, float loss, uint8_t *stage, float *dst, int E, int nrows, bool off)
{
    const int wq = warp & 3, hf = warp >> 2;
    uint8_t *box = stage + (D == 64 ? warp : wq) * 4096;
#pragma unroll
    for (int c = 0; c < D / 8; ++c) {
        float4 x = make_float4(o[4 * c] * scale, o[4 * c + 1] * scale, o[4 * c + 2] * scale, o[4 * c + 3] * scale);
        if (loss != 0.0f) { x.x = fmaf(x.x, loss, x.x); x.y = fmaf(x.y, loss, x.y); x.z = fmaf(x.z, loss, x.z); x.w = fmaf(x.w, loss, x.w); }
        *reinterpret_cast<float4 *>(box + sw128(lane, D == 64 ? c : hf * 4 + c)) = x;
    }
    if (D == 64) __syncwarp();
    else asm volatile("bar.sync %0, 64;" ::"r"(2 + wq) : "memory");
    constexpr int kRows = D == 64 ? 32 : 16;
#pragma unroll
    for (int i = 0; i < kRows / 4; ++i) {
        const int r = (D == 64 ? 0 : hf * 16) + 4 * i + (lane >> 3);
        const float4 v = *reinterpret_cast<const float4 *>(box + sw128(r, lane & 7));
        if (r < nrows && !off) *reinterpret_cast<float4 *>(dst + (size_t)r * E + (D == 64 ? hf * 32 : 0) + (lane & 7) * 4) = v;
    }
}

// ---- rows: maximum and sum, w, dQ --------------------------------------------------------------------------
// STORED: where the probabilities come from.  0: formed again from Q and K.  1: the caller's, one tile ahead through registers
// (rows that TMA cannot address: S not a multiple of four).  2: the caller's, by TMA into a ring of tiles: a tile of
// the first sweep took 1.2 us, which was the latency of the loads one tile ahead; no registers and no turning are needed
// either (B=32 H=8 S=256 D=32: 109.9 -> 102.5 us, B=2 H=16 S=1024 D=64: 258 -> 212).
constexpr int kPTile = kLanes * kTile * 4;           // bytes of a tile of probabilities
template <int STORED>
using PMap = std::conditional_t<STORED == 2, CUtensorMap, int>;
template <int D>
constexpr int kPStages = D == 32 ? 3 : 2;

// A worker writes the factor of its piece of tile i beside tile i and reads that of both halves when tile i + 1 is under way.  The other half's
// worker may be as far as tile i + 2 then (whose scores are formed before tile i + 1 has been handed over), not i + 3.
constexpr int kDownSlots = 4;

template <int D, int STORED>
struct RowsCfg {
    static constexpr int kKStages = D == 64 && STORED ? 3 : 4;           // what 227 KB hold beside Q, dO and the probabilities
    static constexpr int kVStages = kKStages;
    static constexpr int kResident = (STORED ? 1 : 2) * 2 * Img<D>::kTileBytes;      // dO and, to form P again, Q: 128 rows each
    // 1: per warp 32 rows x 32 probabilities on their way to their rows
    static constexpr int kStage = STORED == 2 ? kPStages<D> * kPTile : STORED == 1 ? kWorkerWarps * 4096 : 0;
    static constexpr size_t kSmem = (STORED == 2 ? 1024 : 0) + (size_t)kResident + (kKStages + kVStages) * Img<D>::kTileBytes + kStage;
    static constexpr bool kWide = D == 32;                               // an accumulator has 64 columns
    static constexpr uint32_t kColAcc = 4 * kTile;                       // after two buffers of S and dP: an accumulator per half tile
};

template <int D, bool CAUSAL, int STORED>
__global__ void __launch_bounds__(kThreads, 1)
bwd_rows_kernel(const uint8_t *__restrict__ img, size_t img_bytes, const float *fac, const float *__restrict__ P, float *__restrict__ dQ,
                float *__restrict__ stat, size_t nstat, int S, int Spad, int E, int H, int nblk, float c, const __grid_constant__ PMap<STORED> p_map, int expire)
{
    using C = RowsCfg<D, STORED>;
    constexpr int TB = Img<D>::kTileBytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *p_s = STORED == 2 ? reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023) : smem_raw;
    uint8_t *q_s = p_s + C::kStage, *g_s = q_s + (STORED ? 0 : 2 * TB), *k_s = g_s + 2 * TB, *v_s = k_s + C::kKStages * TB;
    __shared__ uint64_t res_full, k_full[C::kKStages], v_full[C::kVStages], sd_full[2], ready[2], acc_done[2], p_full[STORED == 2 ? kPStages<D> : 1];
    __shared__ float comb[2][STORED ? 1 : 3][kLanes];           // w and, where P is formed again, maximum and sum of each half row
    __shared__ float down_s[kDownSlots][2][kLanes];             // a tile's factors: [half][row]
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    // with the mask the longest blocks of all heads come first; else a head's blocks run side by side
    const int nbh = (int)gridDim.x / nblk;
    const int bh = CAUSAL ? (int)blockIdx.x % nbh : (int)blockIdx.x / nblk;
    const int blk = CAUSAL ? nblk - 1 - (int)blockIdx.x / nbh : (int)blockIdx.x % nblk;
    const int b = bh / H, h = bh % H, q0 = blk * kLanes;
    const int kend = CAUSAL ? min(S, q0 + kLanes) : S;
    const int nk = (kend + kTile - 1) / kTile;       // key tiles of a sweep
    const int total = 2 * nk;

    if (tid == 0) {
        abort_flag = 0;
        mbar_init(&res_full, 1);
        for (int i = 0; i < C::kKStages; ++i) mbar_init(&k_full[i], 1);
        for (int i = 0; i < C::kVStages; ++i) mbar_init(&v_full[i], 1);
        if (STORED == 2) for (int i = 0; i < kPStages<D>; ++i) mbar_init(&p_full[i], 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&sd_full[i], 2); mbar_init(&ready[i], kWorkerWarps); mbar_init(&acc_done[i], 2); }      // (commits: one per issuing warp)
    }
    if (warp == kWorkerWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    dependency_wait();
    dependents_may_start();                          // the columns' blocks take the SMs that run out of rows, up to where they need w
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;
    // site codes: 1 resident operands, 2 K tile, 3 V tile, 4 scores, 5 workers at a tile, 6 accumulation, 7 probabilities
    bool seen = true;                                // what this thread waited for last has come (for who asks for copies then)
    auto wait = [&](uint64_t *bar, uint32_t parity, int site) {
        const int gone = abort_flag;                 // (before the test, and not in its way)
        const bool done = mbar_test(bar, parity);
        seen = !gone;
        if (!gone && !done) seen = bwd_wait_slow(bar, parity, site, &abort_flag, expire);
    };

    if (warp >= kWorkerWarps) {
        // the first issuing warp has K: S = Q K^T and half of the accumulation; the second V: dP = dO V^T and the other half
        const bool first = warp == kWorkerWarps;
        const uint8_t *q_img = img + (size_t)bh * Spad * (Img<D>::kBlock / 8) + (size_t)q0 * (Img<D>::kBlock / 8);
        const uint8_t *k_img = img + img_bytes + (size_t)bh * Spad * (Img<D>::kBlock / 8);
        const uint8_t *v_img = k_img + img_bytes, *g_img = q_img + 3 * img_bytes;
        // with the probabilities given K takes part in the second sweep only: its ring starts there
        const int k_first = STORED ? nk : 0;
        auto k_slot = [&](int i) { return (i - k_first) % C::kKStages; };
        auto k_phase = [&](int i) { return (uint32_t)(((i - k_first) / C::kKStages) & 1); };
        auto fetch_k = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &k_full[k_slot(i)];
                mbar_arrive_expect_tx(bar, TB);
                bulk_load(k_s + k_slot(i) * TB, k_img + (size_t)(i % nk) * TB, TB, bar);
            }
            __syncwarp();
        };
        auto fetch_v = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &v_full[i % C::kVStages];
                mbar_arrive_expect_tx(bar, TB);
                bulk_load(v_s + (i % C::kVStages) * TB, v_img + (size_t)(i % nk) * TB, TB, bar);
            }
            __syncwarp();
        };
        // 128 rows x 64 probabilities in two boxes of 32 columns (rows and columns past S arrive as zeros)
        auto fetch_p = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &p_full[i % kPStages<D>];
                uint8_t *dst = p_s + (i % kPStages<D>) * kPTile;
                mbar_arrive_expect_tx(bar, kPTile);
                tma_load_3d(dst, &p_map, (i % nk) * kTile, q0, bh, bar);
                tma_load_3d(dst + kPTile / 2, &p_map, (i % nk) * kTile + 32, q0, bh, bar);
            }
            __syncwarp();
        };
        if (first) {
            if (lane == 0) {
                mbar_arrive_expect_tx(&res_full, (STORED ? 2 : 4) * TB);
                if (!STORED) bulk_load(q_s, q_img, 2 * TB, &res_full);
                bulk_load(g_s, g_img, 2 * TB, &res_full);
            }
            __syncwarp();
            if (STORED == 2) for (int i = 0; i < kPStages<D>; ++i) fetch_p(i);
            for (int i = 0; i < C::kKStages; ++i) fetch_k(k_first + i);
        } else {
            for (int i = 0; i < C::kVStages; ++i) fetch_v(i);
        }
        auto issue_sd = [&](int i) {
            const uint32_t d = tmem + (uint32_t)((i & 1) * 2 * kTile);
            if (first && STORED) {
                // No product of its own, but the workers wait for this warp's word all the same: it must not fall two tiles behind them in
                // the first sweep, where a ring of three tiles of probabilities would let them.  The phase of `ready` that it
                // looks for would then have come and gone twice, for the tile after too, and it would wait for a third that needs its next copy.
                if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&sd_full[i & 1])) : "memory");
                __syncwarp();
                return;
            }
            if (first) {
                wait(&k_full[k_slot(i)], k_phase(i), 2);
                tc_fence_after();
                issue_scores<D>(d, smem_u32(q_s), smem_u32(k_s + k_slot(i) * TB));
            } else {
                wait(&v_full[i % C::kVStages], (uint32_t)((i / C::kVStages) & 1), 3);
                tc_fence_after();
                issue_scores<D>(d + kTile, smem_u32(g_s), smem_u32(v_s + (i % C::kVStages) * TB));
            }
            if (elect_one()) tc_commit(&sd_full[i & 1]);
        };
        wait(&res_full, 0, 1);
        tc_fence_after();
        issue_sd(0);
        for (int i = 0; i < total; ++i) {
            // the buffer of scores i + 1 is free once the workers (first sweep) or the accumulation (second) have read it
            if (i - 1 >= nk) {
                wait(&acc_done[(i - 1) & 1], (uint32_t)(((i - 1 - nk) >> 1) & 1), 6);
                if (first) fetch_k(i - 1 + C::kKStages);
            }
            if (i + 1 < total) issue_sd(i + 1);
            wait(&ready[i & 1], (uint32_t)((i >> 1) & 1), 5);
            tc_fence_after();
            if (STORED == 2 && first) fetch_p(i + kPStages<D>);      // the workers have read tile i of the probabilities
            if (!first) fetch_v(i + C::kVStages);    // the scores of tile i have been read, so the products that read V have completed
            if (i < nk) {
                if (!STORED && first) fetch_k(i + C::kKStages);
            } else {
                wait(&k_full[k_slot(i)], k_phase(i), 2);
                tc_fence_after();
                const uint32_t s0 = tmem + (uint32_t)((i & 1) * 2 * kTile), kt = smem_u32(k_s + k_slot(i) * TB);
                const int half = first ? 0 : 1;
                issue_accumulate<D, C::kWide, STORED != 0>(tmem + C::kColAcc + 64 * half, s0 + 32 * half, kt, half);
                if (elect_one()) tc_commit(&acc_done[i & 1]);
            }
        }
        __syncwarp();
        if (abort_flag) linger();
        tc_fence_before();
        __syncthreads();
        if (first) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        return;
    }

    // ---- workers: thread = query row, half of the tile's columns ----
    const int wq = warp & 3, hf = warp >> 2;
    const int rloc = wq * 32 + lane, row = q0 + rloc;
    const uint32_t lane_base = tmem + ((uint32_t)(wq * 32) << 16);
    const float cl2 = c * kLog2e;
    auto arrive = [&](uint64_t *bar) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
    };
    // The stored probabilities of this thread's row.  1: a warp reads 32 rows x 32 columns a row per load, and turns them to their
    // rows through shared memory (16-byte pieces, permuted by the row: no bank conflicts).
    const float *p_rows = STORED == 1 ? P + ((size_t)bh * S + q0 + wq * 32) * S : nullptr;
    float pf[STORED == 1 ? 32 : 1];
    auto fetch_p = [&](int i) {
        const int j0 = (i % nk) * kTile + hf * 32;
        // (a lane past S reads its neighbour's column: dP is zero there, and ds is set to zero)
        const float *src = p_rows + min(j0 + lane, S - 1);
        if (q0 + wq * 32 + 32 <= S) {
#pragma unroll
            for (int r = 0; r < 32; ++r, src += S) pf[STORED == 1 ? r : 0] = __ldg(src);
        } else {
#pragma unroll
            for (int r = 0; r < 32; ++r, src += S) pf[STORED == 1 ? r : 0] = q0 + wq * 32 + r < S ? __ldg(src) : 0.0f;
        }
    };
    auto take_p = [&](int i, float (&p)[32]) {
        const uint8_t *src = p_s + (i % kPStages<D>) * kPTile + hf * (kPTile / 2);
        int r0 = rloc;
        if (STORED == 2) {
            wait(&p_full[i % kPStages<D>], (uint32_t)((i / kPStages<D>) & 1), 7);
        } else {
            uint8_t *turn = p_s + warp * 4096;
            __syncwarp();
#pragma unroll
            for (int r = 0; r < 32; ++r) *reinterpret_cast<float *>(turn + sw128(r, lane >> 2) + (lane & 3) * 4) = pf[STORED == 1 ? r : 0];
            __syncwarp();
            src = turn;
            r0 = lane;
        }
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) *reinterpret_cast<float4 *>(&p[ch * 4]) = *reinterpret_cast<const float4 *>(src + sw128(r0, ch));
    };

    float m = -INFINITY, l = 0.0f, w = 0.0f, rinv = 1.0f;
    float o[D / 2];
#pragma unroll
    for (int x = 0; x < D / 2; ++x) o[x] = 0.0f;
    auto add_dq = [&](int i) {                       // tile i of the second sweep has been accumulated
        wait(&acc_done[i & 1], (uint32_t)(((i - nk) >> 1) & 1), 6);
        tc_fence_after();
        add_tile<D, C::kWide>(lane_base + C::kColAcc, hf, down_s[i % kDownSlots][0][rloc], down_s[i % kDownSlots][1][rloc], o);
    };
    // factors: of this row's Q (with the exponent's) and dO, and of 32 tiles of K and V, one per lane
    const size_t ntile = (size_t)nbh * (Spad / kTile), tile0 = (size_t)bh * (Spad / kTile);
    const float q_fac = STORED ? 0.0f : cl2 * fac[tile0 + row / kTile], g_fac = fac[3 * ntile + tile0 + row / kTile];
    float k_facs = 0.0f, v_facs = 0.0f;
    if (STORED == 1) fetch_p(0);
    for (int i = 0; i < total; ++i) {
        const uint32_t s_addr = lane_base + (uint32_t)((i & 1) * 2 * kTile) + hf * 32, dp_addr = s_addr + kTile;
        const int kt = i < nk ? i : i - nk, j0 = kt * kTile + hf * 32;
        const int nvalid = min(S - j0, CAUSAL ? row - j0 + 1 : 32);      // columns of this row that count
        if ((kt & 31) == 0) {
            const size_t at = tile0 + min(kt + lane, Spad / kTile - 1);
            k_facs = fac[ntile + at];
            v_facs = fac[2 * ntile + at];
        }
        const float k_fac = __shfl_sync(0xffffffffu, k_facs, kt & 31), dp_fac = fminf(g_fac * __shfl_sync(0xffffffffu, v_facs, kt & 31), kFacMost);
        const float s_fac = fminf(fmaxf(q_fac * k_fac, 1e-37f), kFacMost);        // (never zero: a hidden score is -inf, and times the factor it stays that)
        const float2 dp2 = make_float2(dp_fac, dp_fac), s2 = make_float2(s_fac, s_fac);
        float s[32], dp[32];
        if (i == nk) {
            // the first sweep is over: join the two halves of each row
            comb[hf][0][rloc] = w;
            if constexpr (!STORED) { comb[hf][1][rloc] = m; comb[hf][2][rloc] = l; }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const float w2 = comb[hf ^ 1][0][rloc];
            if constexpr (STORED) {
                w = hf == 0 ? w + w2 : w2 + w;
            } else {
                const float m2 = comb[hf ^ 1][1][rloc], l2 = comb[hf ^ 1][2][rloc];
                const float mn = fmaxf(fmaxf(m, m2), -1e30f);
                const float a1 = ex2_approx(m - mn), a2 = ex2_approx(m2 - mn);
                const float la = l * a1, lb = l2 * a2, wa = w * a1, wb = w2 * a2;
                l = hf == 0 ? la + lb : lb + la;
                rinv = 1.0f / fmaxf(l, 1e-30f);
                w = (hf == 0 ? wa + wb : wb + wa) * rinv;
                m = mn;
            }
            if (hf == 0) {                           // rows past S: a probability of 0 for every key
                // after a wait that ran out: NaN, so that no block of columns makes a result of what the buffer held before
                const bool lost = abort_flag;
                float *at = stat + (size_t)bh * Spad + row;
                at[0] = lost ? NAN : row < S ? w : 0.0f;
                if (!STORED) { at[nstat] = lost ? NAN : row < S ? m : 0.0f; at[2 * nstat] = lost ? NAN : row < S ? rinv : 0.0f; }
            }
        }
        if (STORED) {
            take_p(i, s);
            if (STORED == 1 && i + 1 < total) fetch_p(i + 1);       // in flight during this tile
        }
        wait(&sd_full[i & 1], (uint32_t)((i >> 1) & 1), 4);
        tc_fence_after();
        if (!STORED) tmem_ld32(s_addr, s);
        tmem_ld32(dp_addr, dp);
        tmem_wait_ld();
        if (i < nk) {
            arrive(&ready[i & 1]);
            if (STORED) {
                float2 ws[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                for (int x = 0; x < 32; x += 2) {
                    if (CAUSAL) { s[x] = x < nvalid ? s[x] : 0.0f; s[x + 1] = x + 1 < nvalid ? s[x + 1] : 0.0f; }
                    ws[(x >> 1) & 1] = ffma2(make_float2(s[x], s[x + 1]), make_float2(dp[x], dp[x + 1]), ws[(x >> 1) & 1]);
                }
                w = fmaf((ws[0].x + ws[0].y) + (ws[1].x + ws[1].y), dp_fac, w);
            } else if (nvalid > 0) {
                float mx = -INFINITY;
                if (nvalid < 32) {
#pragma unroll
                    for (int x = 0; x < 32; ++x) s[x] = x < nvalid ? s[x] : -INFINITY;
                }
#pragma unroll
                for (int x = 0; x < 32; x += 2) mx = max3(mx, s[x], s[x + 1]);
                const float mn = fmaxf(m, mx * s_fac), alpha = ex2_approx(m - mn);
                m = mn;
                float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, ws[2] = {ls[0], ls[0]};
#pragma unroll
                for (int x = 0; x < 32; x += 2) {
                    const float2 t = ffma2(make_float2(s[x], s[x + 1]), s2, make_float2(-mn, -mn));
                    const float2 e = make_float2(ex2_approx(t.x), ex2_approx(t.y));
                    ls[(x >> 1) & 1] = fadd2(ls[(x >> 1) & 1], e);
                    ws[(x >> 1) & 1] = ffma2(e, make_float2(dp[x], dp[x + 1]), ws[(x >> 1) & 1]);
                }
                l = fmaf(l, alpha, (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y));
                w = fmaf(w, alpha, ((ws[0].x + ws[0].y) + (ws[1].x + ws[1].y)) * dp_fac);
            }
        } else {
#pragma unroll
            for (int x = 0; x < 32; x += 2) {
                float2 p = make_float2(s[x], s[x + 1]);
                if (!STORED) {
                    p = ffma2(p, s2, make_float2(-m, -m));         // (1 / l leaves with the row of dQ)
                    p = make_float2(ex2_approx(p.x), ex2_approx(p.y));
                }
                const float2 d = fmul2(p, ffma2(make_float2(dp[x], dp[x + 1]), dp2, make_float2(-w, -w)));
                dp[x] = d.x;
                dp[x + 1] = d.y;
            }
            if (nvalid < 32) {
#pragma unroll
                for (int x = 0; x < 32; ++x) dp[x] = x < nvalid ? dp[x] : 0.0f;
            }
            down_s[i % kDownSlots][hf][rloc] = store_pieces(dp, s_addr) * k_fac;
            if (i > nk) add_dq(i - 1);
            tmem_wait_st();
            arrive(&ready[i & 1]);
        }
    }
    add_dq(total - 1);
    // (through the K tiles' memory: the last product has read it)
    const int row0 = q0 + wq * 32;
    store_out<D>(o, warp, lane, c * rinv, kScoreLoss, k_s, dQ + ((size_t)b * S + row0) * E + (size_t)h * D, E, S - row0, abort_flag);
    tc_fence_before();
    __syncthreads();
}

// ---- columns: dK, dV -----------------------------------------------------------------------------------
template <int D, int STORED>
struct ColsCfg {
    // dV of stored probabilities, which are exact, as dO is: three bf16 pieces hold all 24 bits of both (two fp16 ones hold 23: dV was 0.97e-7 instead of
    // 0.90e-7 from float64 at S = 200 D = 64).  A tile pair then comes with dO's three pieces too, and P^T's take 96 columns.
    static constexpr int kStages = !STORED ? 4 : D == 64 ? 2 : 3;        // (Q, dO) tile pairs
    static constexpr int kPair = 2 * Img<D>::kTileBytes + (STORED ? kTileBytes3<D> : 0);
    static constexpr int kResident = (STORED ? 1 : 2) * 2 * Img<D>::kTileBytes;      // V and, to form P again, K: 128 rows each
    static constexpr int kStage = STORED == 2 ? kPStages<D> * kPTile : 0;
    static constexpr size_t kSmem = (STORED == 2 ? 1024 : 0) + (size_t)kResident + kStages * kPair + kStage;
    static constexpr uint32_t kColD = STORED ? 96 : kTile, kBuf = kColD + kTile;      // S^T and, from kColD on, dP^T, then the pieces of P^T and ds^T
    static constexpr uint32_t kColV = 2 * kBuf, kColK = kColV + (STORED ? 64 : 128);  // an accumulator per half tile; one per tile for the exact products
    static constexpr bool kWide = D == 32;                               // an accumulator has 64 columns
    // (a tile's w, maxima and sums come by bulk copy, tiles ahead: the workers' own loads stood between the scores and ds, 0.3 us per tile of
    // 1.4, 1.4 in a block's first at D = 32 with stored probabilities)
};

template <int D, bool CAUSAL, int STORED>
__global__ void __launch_bounds__(kThreads, 1)
bwd_cols_kernel(const uint8_t *__restrict__ img, size_t img_bytes, const float *fac, const float *__restrict__ P, float *__restrict__ dK, float *__restrict__ dV,
                const float *__restrict__ stat, size_t nstat, int S, int Spad, int E, int H, int nblk, float c, const __grid_constant__ PMap<STORED> p_map, int expire)
{
    using C = ColsCfg<D, STORED>;
    constexpr int TB = Img<D>::kTileBytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *p_s = STORED == 2 ? reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023) : smem_raw;
    uint8_t *k_s = p_s + C::kStage, *v_s = k_s + (STORED ? 0 : 2 * TB), *t_s = v_s + 2 * TB;     // t_s: [stage][Q tile | dO tile | its three pieces]
    __shared__ __align__(16) float rows_s[C::kStages][STORED ? 1 : 3][kTile];        // w and, to form P again, maximum and 1 / sum of a tile's queries
    __shared__ float down_s[kDownSlots][2][2][kLanes];                   // a tile's factors: [dV, dK][half][key]
    __shared__ uint64_t res_full, full[C::kStages], w_full[C::kStages], sd_full[2], ready[2], acc_done[2], p_full[STORED == 2 ? kPStages<D> : 1];
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile int abort_flag;

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int nbh = (int)gridDim.x / nblk;           // with the mask the first key block of a head is the longest
    const int bh = CAUSAL ? (int)blockIdx.x % nbh : (int)blockIdx.x / nblk, blk = CAUSAL ? (int)blockIdx.x / nbh : (int)blockIdx.x % nblk;
    const int b = bh / H, h = bh % H, k0 = blk * kLanes;
    const int t0 = CAUSAL ? k0 / kTile : 0;          // the first query that sees key j is query j
    const int total = (S + kTile - 1) / kTile - t0;

    if (tid == 0) {
        abort_flag = 0;
        mbar_init(&res_full, 1);
        for (int i = 0; i < C::kStages; ++i) { mbar_init(&full[i], 1); mbar_init(&w_full[i], 1); }
        if (STORED == 2) for (int i = 0; i < kPStages<D>; ++i) mbar_init(&p_full[i], 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&sd_full[i], STORED ? 1 : 2); mbar_init(&ready[i], kWorkerWarps); mbar_init(&acc_done[i], 2); }      // (commits: one per issuing warp)
    }
    if (warp == kWorkerWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // No wait for the kernel before yet: the probabilities and the images are older than that one (it waited for the
    // packing before it let this one start); who reads the rows' statistics waits for it.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;
    // site codes: 11 resident operands, 12 tile pair, 14 scores, 15 workers at a tile, 16 accumulation, 17 probabilities, 18 rows' statistics
    bool seen = true;                                // what this thread waited for last has come (for who asks for copies then)
    auto wait = [&](uint64_t *bar, uint32_t parity, int site) {
        const int gone = abort_flag;                 // (before the test, and not in its way)
        const bool done = mbar_test(bar, parity);
        seen = !gone;
        if (!gone && !done) seen = bwd_wait_slow(bar, parity, site, &abort_flag, expire);
    };

    if (warp >= kWorkerWarps) {
        // the first issuing warp: S^T = K Q^T and dV; the second: dP^T = V dO^T and dK
        const bool first = warp == kWorkerWarps;
        const uint8_t *q_img = img + (size_t)bh * Spad * (Img<D>::kBlock / 8);
        const uint8_t *k_img = q_img + img_bytes + (size_t)k0 * (Img<D>::kBlock / 8), *v_img = k_img + img_bytes, *g_img = q_img + 3 * img_bytes;
        const uint8_t *g3_img = img + 4 * img_bytes + (size_t)bh * (Spad / kTile) * kTileBytes3<D>;
        auto fetch = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &full[i % C::kStages];
                uint8_t *dst = t_s + (i % C::kStages) * C::kPair;
                mbar_arrive_expect_tx(bar, C::kPair);
                bulk_load(dst, q_img + (size_t)(t0 + i) * TB, TB, bar);
                bulk_load(dst + TB, g_img + (size_t)(t0 + i) * TB, TB, bar);
                if (STORED) bulk_load(dst + 2 * TB, g3_img + (size_t)(t0 + i) * kTileBytes3<D>, kTileBytes3<D>, bar);
            }
            __syncwarp();
        };
        // 64 queries x 128 probabilities in four boxes of 32 columns (a box per lane quarter)
        auto fetch_p = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &p_full[i % kPStages<D>];
                uint8_t *dst = p_s + (i % kPStages<D>) * kPTile;
                mbar_arrive_expect_tx(bar, kPTile);
                for (int u = 0; u < 4; ++u) tma_load_3d(dst + u * (kPTile / 4), &p_map, k0 + 32 * u, (t0 + i) * kTile, bh, bar);
            }
            __syncwarp();
        };
        if (first) {
            if (lane == 0) {
                mbar_arrive_expect_tx(&res_full, (STORED ? 2 : 4) * TB);
                if (!STORED) bulk_load(k_s, k_img, 2 * TB, &res_full);
                bulk_load(v_s, v_img, 2 * TB, &res_full);
            }
            __syncwarp();
            if (STORED == 2) {
                for (int i = 0; i < C::kStages; ++i) {
                    fetch(i);
                    if (i < kPStages<D>) fetch_p(i);
                }
            } else {
                for (int i = 0; i < C::kStages; ++i) fetch(i);
            }
        }
        auto fetch_w = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &w_full[i % C::kStages];
                const size_t at = (size_t)bh * Spad + (size_t)(t0 + i) * kTile;
                mbar_arrive_expect_tx(bar, (STORED ? 1 : 3) * kTile * 4);
                for (int u = 0; u < (STORED ? 1 : 3); ++u) bulk_load(rows_s[i % C::kStages][u], stat + u * nstat + at, kTile * 4, bar);
            }
            __syncwarp();
        };
        auto issue_sd = [&](int i) {
            if (STORED && first) return;
            const uint32_t d = tmem + (uint32_t)(i & 1) * C::kBuf, t = smem_u32(t_s + (i % C::kStages) * C::kPair);
            wait(&full[i % C::kStages], (uint32_t)((i / C::kStages) & 1), 12);
            tc_fence_after();
            if (first) issue_scores<D>(d, smem_u32(k_s), t);
            else issue_scores<D>(d + C::kColD, smem_u32(v_s), t + TB);
            if (elect_one()) tc_commit(&sd_full[i & 1]);
        };
        wait(&res_full, 0, 11);
        tc_fence_after();
        issue_sd(0);
        if (!first) {
            dependency_wait();
            for (int i = 0; i < C::kStages; ++i) fetch_w(i);
        }
        for (int i = 0; i < total; ++i) {
            if (i >= 1) {                            // tile i - 1 has been accumulated: its stage and its buffer are free
                wait(&acc_done[(i - 1) & 1], (uint32_t)(((i - 1) >> 1) & 1), 16);
                if (first) fetch(i - 1 + C::kStages);
            }
            if (i + 1 < total) issue_sd(i + 1);
            if (STORED && first) wait(&full[i % C::kStages], (uint32_t)((i / C::kStages) & 1), 12);
            wait(&ready[i & 1], (uint32_t)((i >> 1) & 1), 15);
            tc_fence_after();
            if (STORED == 2 && first) fetch_p(i + kPStages<D>);      // the workers have read tile i of the probabilities
            if (!first) fetch_w(i + C::kStages);     // ... and its rows' statistics
            const uint32_t s0 = tmem + (uint32_t)(i & 1) * C::kBuf, t = smem_u32(t_s + (i % C::kStages) * C::kPair);
            if (STORED && first)
                issue_exact<D>(tmem + C::kColV, s0, t + 2 * TB);
            else
                for (int half = 0; half < 2; ++half)
                    issue_accumulate<D, C::kWide, STORED != 0>(tmem + (first ? C::kColV : C::kColK) + 64 * half, s0 + (first ? 0 : C::kColD) + 32 * half, first ? t + TB : t, half);
            if (elect_one()) tc_commit(&acc_done[i & 1]);
        }
        __syncwarp();
        if (abort_flag) linger();
        tc_fence_before();
        __syncthreads();
        if (first) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        return;
    }

    // ---- workers: thread = key, half of the tile's queries ----
    const int wq = warp & 3, hf = warp >> 2;
    const int rloc = wq * 32 + lane, key = k0 + rloc;
    const uint32_t lane_base = tmem + ((uint32_t)(wq * 32) << 16);
    const float cl2 = c * kLog2e;
    auto arrive = [&](uint64_t *bar) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
    };
    float pn[STORED == 1 ? 32 : 1];                  // stored probabilities of the tile ahead: a query's are contiguous over the keys (lanes)
    auto fetch_p = [&](int i) {
        const int qb = (t0 + i) * kTile + hf * 32;
        // a lane past S reads its neighbour's key (its results go nowhere): no load depends on the lane, and in a full tile none
        // on the query either (loads behind conditions took 3500 cycles per tile to issue)
        const float *src = P + ((size_t)bh * S + qb) * S + min(key, S - 1);
        if (qb + 32 <= S) {
#pragma unroll
            for (int x = 0; x < 32; ++x, src += S) pn[STORED == 1 ? x : 0] = __ldg(src);
        } else {
#pragma unroll
            for (int x = 0; x < 32; ++x, src += S) pn[STORED == 1 ? x : 0] = qb + x < S ? __ldg(src) : 0.0f;
        }
    };
    float ok[D / 2], ov[D / 2];
#pragma unroll
    for (int x = 0; x < D / 2; ++x) ok[x] = ov[x] = 0.0f;
    auto add_dkv = [&](int i) {                      // tile i has been accumulated
        wait(&acc_done[i & 1], (uint32_t)((i >> 1) & 1), 16);
        tc_fence_after();
        if (STORED) add_exact<D>(lane_base + C::kColV, hf, ov);
        else add_tile<D, C::kWide>(lane_base + C::kColV, hf, down_s[i % kDownSlots][0][0][rloc], down_s[i % kDownSlots][0][1][rloc], ov);
        add_tile<D, C::kWide>(lane_base + C::kColK, hf, down_s[i % kDownSlots][1][0][rloc], down_s[i % kDownSlots][1][1][rloc], ok);
    };
    // factors: of this key's K (with the exponent's) and V, and of 32 tiles of Q and dO, one per lane
    const size_t ntile = (size_t)nbh * (Spad / kTile), tile0 = (size_t)bh * (Spad / kTile);
    const float k_fac = STORED ? 0.0f : cl2 * fac[ntile + tile0 + key / kTile], v_fac = fac[2 * ntile + tile0 + key / kTile];
    float q_facs = 0.0f, g_facs = 0.0f;
    if (STORED == 1) fetch_p(0);
    for (int i = 0; i < total; ++i) {
        const uint32_t s_addr = lane_base + (uint32_t)(i & 1) * C::kBuf + hf * 32, dp_addr = s_addr + C::kColD;
        const int qb = (t0 + i) * kTile + hf * 32;
        if ((i & 31) == 0) {
            const size_t ft = tile0 + min(t0 + i + lane, Spad / kTile - 1);
            q_facs = fac[ft];
            g_facs = fac[3 * ntile + ft];
        }
        const float q_fac = __shfl_sync(0xffffffffu, q_facs, i & 31), g_fac = __shfl_sync(0xffffffffu, g_facs, i & 31);
        const float s_fac = fminf(k_fac * q_fac, kFacMost), dp_fac = fminf(v_fac * g_fac, kFacMost);
        const float2 s2 = make_float2(s_fac, s_fac), dp2 = make_float2(dp_fac, dp_fac);
        const float *wrow = rows_s[i % C::kStages][0] + hf * 32;
        const bool mask = CAUSAL && qb < k0 + wq * 32 + 31;              // some lane of the warp has a key after some query
        float p[32], d[32];
        if (STORED == 1) {
#pragma unroll
            for (int x = 0; x < 32; ++x) p[x] = pn[STORED == 1 ? x : 0];
            if (i + 1 < total) fetch_p(i + 1);       // in flight during this tile
        }
        if (STORED == 2) {
            wait(&p_full[i % kPStages<D>], (uint32_t)((i / kPStages<D>) & 1), 17);
            const uint8_t *src = p_s + (i % kPStages<D>) * kPTile + wq * (kPTile / 4) + (lane & 3) * 4;
#pragma unroll
            for (int x = 0; x < 32; ++x) p[x] = *reinterpret_cast<const float *>(src + sw128(hf * 32 + x, lane >> 2));
        }
        wait(&sd_full[i & 1], (uint32_t)((i >> 1) & 1), 14);
        tc_fence_after();
        if (!STORED) tmem_ld32(s_addr, p);
        tmem_ld32(dp_addr, d);
        tmem_wait_ld();
        wait(&w_full[i % C::kStages], (uint32_t)((i / C::kStages) & 1), 18);
        if (!STORED) {
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
                // (the maximum and 1 / sum apart: the exponent of a probability that counts is then near zero and its rounding small)
                const float4 mx = *reinterpret_cast<const float4 *>(wrow + kTile + x), ri = *reinterpret_cast<const float4 *>(wrow + 2 * kTile + x);
                const float2 a = ffma2(make_float2(p[x], p[x + 1]), s2, make_float2(-mx.x, -mx.y));
                const float2 e = ffma2(make_float2(p[x + 2], p[x + 3]), s2, make_float2(-mx.z, -mx.w));
                const float2 pa = fmul2(make_float2(ex2_approx(a.x), ex2_approx(a.y)), make_float2(ri.x, ri.y));       // rows past S: 1 / sum is 0
                const float2 pe = fmul2(make_float2(ex2_approx(e.x), ex2_approx(e.y)), make_float2(ri.z, ri.w));
                p[x] = pa.x; p[x + 1] = pa.y; p[x + 2] = pe.x; p[x + 3] = pe.y;
            }
        }
        if (mask) {
#pragma unroll
            for (int x = 0; x < 32; ++x) p[x] = key <= qb + x ? p[x] : 0.0f;
        }
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
            const float4 w4 = *reinterpret_cast<const float4 *>(wrow + x);
            const float2 a = fmul2(make_float2(p[x], p[x + 1]), ffma2(make_float2(d[x], d[x + 1]), dp2, make_float2(-w4.x, -w4.y)));
            const float2 e = fmul2(make_float2(p[x + 2], p[x + 3]), ffma2(make_float2(d[x + 2], d[x + 3]), dp2, make_float2(-w4.z, -w4.w)));
            d[x] = a.x; d[x + 1] = a.y; d[x + 2] = e.x; d[x + 3] = e.y;
        }
        if (STORED) store_exact(p, s_addr - hf * 16);
        else down_s[i % kDownSlots][0][hf][rloc] = store_pieces(p, s_addr) * g_fac;
        down_s[i % kDownSlots][1][hf][rloc] = store_pieces(d, dp_addr) * q_fac;
        if (i > 0) add_dkv(i - 1);
        tmem_wait_st();
        arrive(&ready[i & 1]);
    }
    add_dkv(total - 1);
    // (through the tiles' memory: the last products have read it)
    const int row0 = k0 + wq * 32;
    const size_t dst = ((size_t)b * S + row0) * E + (size_t)h * D;
    store_out<D>(ov, warp, lane, 1.0f, STORED ? 0.0f : kSumLoss, t_s, dV + dst, E, S - row0, abort_flag);
    store_out<D>(ok, warp, lane, c, kScoreLoss, t_s + TB * 2, dK + dst, E, S - row0, abort_flag);
    tc_fence_before();
    __syncthreads();
}

StreamWorkspace g_bwd_ws;

template <int D, bool CAUSAL, int STORED>
int launch_cfg(const float *g, const float *q, const float *k, const float *v, const float *probs, float *dq, float *dk, float *dv,
               int B, int S, int E, int H, cudaStream_t st)
{
    auto rows = bwd_rows_kernel<D, CAUSAL, STORED>;
    auto cols = bwd_cols_kernel<D, CAUSAL, STORED>;
    constexpr size_t rows_smem = RowsCfg<D, STORED>::kSmem, cols_smem = ColsCfg<D, STORED>::kSmem;
    static_assert(rows_smem + ((STORED ? 1 : 3) + kDownSlots) * 2 * kLanes * 4 + 256 <= 232448 &&
                  cols_smem + ColsCfg<D, STORED>::kStages * (STORED ? 1 : 3) * kTile * 4 + kDownSlots * 4 * kLanes * 4 + 512 <= 232448 && ColsCfg<D, STORED>::kColK + 128 <= kTmemCols, "shared memory of a block");
    cudaError_t e = cudaFuncSetAttribute(rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cols_smem);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    const int nblk = (S + kLanes - 1) / kLanes, Spad = nblk * kLanes;
    // groups of batches whose images (4 bytes per element, 6 more for dO's three pieces) stay in L2 between the kernels that write and read them
    const size_t per_batch = (size_t)H * Spad * D * (STORED ? 22 : 16);
    long long gb = (long long)((64u << 20) / per_batch);
    gb = gb < 1 ? 1 : gb > B ? B : gb;
    while (gb > 1 && gb * H * (long long)(Spad / kTile) > 2000000000LL) gb /= 2;
    const size_t img_bytes = (size_t)gb * H * Spad * D * 4, exact_bytes = STORED ? img_bytes / 2 * 3 : 0, nstat = (size_t)gb * H * Spad;
    StreamWorkspace::Lease ws;
    int rc = g_bwd_ws.enter(st, 4 * img_bytes + exact_bytes + ((STORED ? 1 : 3) * nstat + 4 * (nstat / kTile)) * sizeof(float), &ws);
    if (rc != HIPGPT_OK) return rc;
    uint8_t *img = ws.get();
    // beside the images: w and, where P is formed again, maximum and 1 / sum of the rows; the tiles' factors
    float *stat = reinterpret_cast<float *>(img + 4 * img_bytes + exact_bytes), *fac = stat + (STORED ? 1 : 3) * nstat;
    const float c = 1.0f / sqrtf((float)D);
    const int expire = take_expiry(600);
    for (long long b0 = 0; b0 < B; b0 += gb) {
        const int nb = (int)(B - b0 < gb ? B - b0 : gb);
        const size_t off = (size_t)b0 * S * E;
        const float *p = STORED ? probs + (size_t)b0 * H * S * S : nullptr;
        e = launch_overlapped(bwd_pack_kernel<D>, dim3((unsigned)(nb * H * (Spad / kTile)), 4), dim3(256), 0, st, q + off, k + off, v + off, g + off, img, img_bytes, fac, STORED ? img + 4 * img_bytes : (uint8_t *)nullptr, S, Spad / kTile, E, H);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_pack_kernel launch: %s", cudaGetErrorString(e));
        PMap<STORED> rows_map = {}, cols_map = {};
        if constexpr (STORED == 2) {
            rc = tma_plane_map(&rows_map, p, nb * H, S, S, kLanes, CU_TENSOR_MAP_SWIZZLE_128B);
            if (rc == HIPGPT_OK) rc = tma_plane_map(&cols_map, p, nb * H, S, S, kTile, CU_TENSOR_MAP_SWIZZLE_128B);
            if (rc != HIPGPT_OK) return rc;
        }
        const dim3 grid((unsigned)(nb * H * nblk));
        e = launch_overlapped(rows, grid, dim3(kThreads), rows_smem, st, (const uint8_t *)img, img_bytes, (const float *)fac, p, dq + off, stat, nstat, S, Spad, E, H, nblk, c, rows_map, (expire & 255) <= 10 ? expire : 0);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_rows_kernel launch: %s", cudaGetErrorString(e));
        e = launch_overlapped(cols, grid, dim3(kThreads), cols_smem, st, (const uint8_t *)img, img_bytes, (const float *)fac, p, dk + off, dv + off, (const float *)stat, nstat,
                              S, Spad, E, H, nblk, c, cols_map, (expire & 255) > 10 ? expire : 0);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_cols_kernel launch: %s", cudaGetErrorString(e));
    }
    return HIPGPT_OK;
}

}  // namespace

// head_dim 32 / 64 on 16-byte aligned planes
bool mha_backward_tc_supports(const void *g, const void *q, const void *k, const void *v, const void *probs, const void *dq, const void *dk,
                              const void *dv, int B, int S, int E, int H)
{
    const int D = E / H;
    if (D != 32 && D != 64) return false;
    if ((long long)H * ((S + 127) / 128) * 16 * (D / 32) > 2000000000LL || (long long)B * H > 65535) return false;
    uintptr_t all = 0;
    for (const void *p : {g, q, k, v, probs, dq, dk, dv}) all |= reinterpret_cast<uintptr_t>(p);
    return (all & 15) == 0;
}

int launch_mha_backward_tc(const float *g, const float *q, const float *k, const float *v, const float *probs, float *dq, float *dk, float *dv,
                           int B, int S, int E, int H, int causal, cudaStream_t st)
{
    if (mha_backward_head_supports(E / H, S)) return launch_mha_backward_head(g, q, k, v, probs, dq, dk, dv, B, S, E, H, causal, st);
    // probabilities whose rows TMA can address (the pointer is 16-byte aligned)
    const int stored = !probs ? 0 : (S & 3) == 0 && tma_encode_fn() != nullptr ? 2 : 1;
    auto go = [&](auto launch) { return launch(g, q, k, v, probs, dq, dk, dv, B, S, E, H, st); };
    auto pick = [&](auto l0, auto l1, auto l2) { return stored == 0 ? go(l0) : stored == 1 ? go(l1) : go(l2); };
    if (E / H == 64)
        return causal ? pick(launch_cfg<64, true, 0>, launch_cfg<64, true, 1>, launch_cfg<64, true, 2>) : pick(launch_cfg<64, false, 0>, launch_cfg<64, false, 1>, launch_cfg<64, false, 2>);
    return causal ? pick(launch_cfg<32, true, 0>, launch_cfg<32, true, 1>, launch_cfg<32, true, 2>) : pick(launch_cfg<32, false, 0>, launch_cfg<32, false, 1>, launch_cfg<32, false, 2>);
}

void mha_backward_tc_release() { g_bwd_ws.release(); }

int mha_backward_tc_status_fetch(int *status)
{
    int s = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&s, g_bwd_status, sizeof(int));
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    if (s != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_bwd_status, &zero, sizeof(int));
    }
    *status = s;
    return HIPGPT_OK;
}

}  // namespace hipgpt
