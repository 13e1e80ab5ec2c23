// Attention backward on the Blackwell tensor pipe (tcgen05 + TMEM), head_dim 32 or 64, any sequence length, with the accuracy of
// fp32 products.  Same contract as attn_bwd.cu (HipGPT src/hip_kernels.cpp:1162-1272), which keeps every other head_dim:
//     vd_ij = g_i . V_j            w_i  = sum_j P_ij vd_ij        ds_ij = P_ij (vd_ij - w_i)
//     dQ_i  = c sum_j ds_ij K_j    dK_j = c sum_i ds_ij Q_i       dV_j  = sum_i P_ij g_i
//
// Arithmetic.  An fp32 number is the sum of three bf16 numbers (8 bits each, the exponent range of fp32: no scaling, any magnitude).
// A product of two such sums is formed from six products of the pieces, hi hi, hi mid, mid hi, mid mid, hi lo, lo hi, which the
// tensor core multiplies exactly and adds in fp32; what is dropped (mid lo, lo mid, lo lo) is below 2^-24 of the product, the
// rounding of an fp32 product.  P and ds, formed in fp32 in registers, are cut the same way before they become operands.
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
#include "stream_workspace.hpp"
#include "tc_primitives.cuh"
#include "tma_host.cuh"

#include <math.h>
#include <type_traits>

namespace hipgpt {
namespace {

constexpr int kLanes = 128;            // rows (or keys) per block = TMEM lanes
constexpr int kTile = 64;              // columns per tile
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

// Sizes of an operand image, in bytes.
template <int D>
struct Img {
    static constexpr int kPiece = (D / 8) * 128;     // one piece of an 8-row block
    static constexpr int kBlock = 3 * kPiece;        // an 8-row block
    static constexpr int kTileBytes = (kTile / 8) * kBlock;     // 64 rows
};

// Two fp32 numbers -> three words of two bf16 each whose sums are the numbers (to 2^-25 of them)
__device__ __forceinline__ void cut3(float x, float y, uint32_t &h, uint32_t &m, uint32_t &l)
{
    h = pack_bf16(x, y);
    const float2 r = fadd2(make_float2(x, y), make_float2(-__uint_as_float(h << 16), -__uint_as_float(h & 0xffff0000u)));
    m = pack_bf16(r.x, r.y);
    const float2 s = fadd2(r, make_float2(-__uint_as_float(m << 16), -__uint_as_float(m & 0xffff0000u)));
    l = pack_bf16(s.x, s.y);
}

// ---- the pieces of the four planes ---------------------------------------------------------------------
// A warp takes 8 rows x 32 columns: lane = (column block of 8) * 8 + row, so that it reads 8 whole lines and writes four core
// matrices of 128 contiguous bytes per piece.  Bound by memory: 4 bytes read and 6 written per element.
template <int D>
__global__ void __launch_bounds__(256)
bwd_pack_kernel(const float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v, const float *__restrict__ g,
                uint8_t *__restrict__ img, size_t img_bytes, int S, int Spad, int E, int H, int tasks)
{
    constexpr int PARTS = D / 32;
    dependency_wait();
    dependents_may_start();
    const int task = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (task >= tasks) return;
    const int part = task % PARTS, rb = (task / PARTS) % (Spad / 8), bh = task / PARTS / (Spad / 8);
    const int r = lane & 7, cb = part * 4 + (lane >> 3), row = rb * 8 + r;
    const float *src = blockIdx.y == 0 ? q : blockIdx.y == 1 ? k : blockIdx.y == 2 ? v : g;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (row < S) {
        const float4 *p = reinterpret_cast<const float4 *>(src + ((size_t)(bh / H) * S + row) * E + (size_t)(bh % H) * D + cb * 8);
        a = __ldg(p);
        b = __ldg(p + 1);
    }
    uint4 h, m, l;
    cut3(a.x, a.y, h.x, m.x, l.x);
    cut3(a.z, a.w, h.y, m.y, l.y);
    cut3(b.x, b.y, h.z, m.z, l.z);
    cut3(b.z, b.w, h.w, m.w, l.w);
    uint8_t *dst = img + blockIdx.y * img_bytes + ((size_t)bh * (Spad / 8) + rb) * Img<D>::kBlock + cb * 128 + r * 16;
    *reinterpret_cast<uint4 *>(dst) = h;
    *reinterpret_cast<uint4 *>(dst + Img<D>::kPiece) = m;
    *reinterpret_cast<uint4 *>(dst + 2 * Img<D>::kPiece) = l;
}

// ---- the products, issued by one converged warp that elects the lane per instruction ---------------------
// D[tmem] (128 x 64) = A B^T over the head dimension; A: 128 rows, B: 64 rows, both images read K-major.
template <int D>
__device__ __forceinline__ void issue_scores(uint32_t d_tmem, uint32_t a_smem, uint32_t b_smem)
{
    const uint64_t a = make_desc(a_smem, 128, Img<D>::kBlock, 0), b = make_desc(b_smem, 128, Img<D>::kBlock, 0);
    constexpr uint32_t id = idesc_bf16(kLanes, kTile, 0);
    constexpr int PA[6] = {0, 2, 1, 1, 0, 0}, PB[6] = {2, 0, 1, 0, 1, 0};        // small terms first
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            const uint64_t da = a + (uint64_t)((PA[p] * (D / 8) + 2 * k) * 8), db = b + (uint64_t)((PB[p] * (D / 8) + 2 * k) * 8);
            if (elect_one()) mma_h_ss(d_tmem, da, db, id, (p | k) ? 1u : 0u);
        }
}

// acc[tmem] (128 x D) = A B over rows [16 KS0, 16 KS1) of B's image, read N-major; A: three pieces in TMEM, the piece `p` of the columns
// [32 hf, 32 hf + 32) packed in 16 columns at a_col(p, hf).  WIDE: acc is 2 D columns, the second half collects the products with
// B's mid and lo pieces (wider instructions, fewer of them).  The small products come first: the tensor core truncates where
// it adds to its accumulator, so the accumulator should be small while they are added, and it starts anew for every tile (the
// workers add the tiles up in registers).  One accumulator over all tiles was 10 times farther from float64 at S = 777.
template <int D, bool WIDE, int KS0, int KS1, typename ACol>
__device__ __forceinline__ void issue_accumulate(uint32_t acc, ACol a_col, uint32_t b_smem)
{
    const uint64_t b = make_desc(b_smem, Img<D>::kBlock, 128, 0);
    constexpr uint32_t id1 = idesc_bf16(kLanes, D, 1), id2 = idesc_bf16(kLanes, 2 * D, 1);
    auto product = [&](int pa, int pb, int d, uint32_t id, bool fresh) {
#pragma unroll
        for (int ks = KS0; ks < KS1; ++ks) {
            const uint64_t bk = b + (uint64_t)(ks * 2 * (Img<D>::kBlock >> 4) + pb * (Img<D>::kPiece >> 4));
            if (elect_one()) mma_h_ts(acc + d, a_col(pa, ks >> 1) + (ks & 1) * 8, bk, id, (fresh && ks == KS0) ? 0u : 1u);
        }
    };
    if (WIDE) {
        product(1, 0, 0, id2, true);                 // mid x [hi | mid]
        product(2, 0, 0, id1, false);                // lo x hi
        product(0, 2, D, id1, false);                // hi x lo
        product(0, 0, 0, id2, false);                // hi x [hi | mid]
    } else {
        product(0, 2, 0, id1, true);
        product(2, 0, 0, id1, false);
        product(1, 1, 0, id1, false);
        product(0, 1, 0, id1, false);
        product(1, 0, 0, id1, false);
        product(0, 0, 0, id1, false);
    }
}

// 32 numbers of a row (or key) -> their three pieces at the given TMEM columns
__device__ __forceinline__ void store_pieces(const float (&x)[32], uint32_t hi, uint32_t mid, uint32_t lo)
{
    uint32_t h[16], m[16], l[16];
#pragma unroll
    for (int c = 0; c < 16; ++c) cut3(x[2 * c], x[2 * c + 1], h[c], m[c], l[c]);
    tmem_st16_u32(hi, h);
    tmem_st16_u32(mid, m);
    tmem_st16_u32(lo, l);
}

// Adds a tile's accumulator (this thread's D / 2 columns of its row) to the running sum
template <int D, bool WIDE>
__device__ __forceinline__ void add_tile(uint32_t acc, int hf, float (&o)[D / 2])
{
#pragma unroll
    for (int c0 = 0; c0 < D / 2; c0 += 16) {
        float a[16], b[16];
        tmem_ld16(acc + hf * (D / 2) + c0, a);
        if (WIDE) tmem_ld16(acc + D + hf * (D / 2) + c0, b);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; c += 2) {
            float2 t = make_float2(a[c], a[c + 1]);
            if (WIDE) t = fadd2(t, make_float2(b[c], b[c + 1]));
            t = fadd2(make_float2(o[c0 + c], o[c0 + c + 1]), t);
            o[c0 + c] = t.x;
            o[c0 + c + 1] = t.y;
        }
    }
}

// A warp's 32 rows x D / 2 results leave in whole lines: through shared memory (boxes of 32 x 32, 16-byte pieces permuted by the row; at head_dim
// 32 the two warps of a quarter share one), then a row of 128 bytes per eight lanes.  A thread's own stores touched 32 lines
// each (1.2 us at the end of a 10.7 us block of columns).  dst: the head's first column of the warp's first row.
template <int D>
__device__ __forceinline__ void store_out(const float (&o)[D / 2], int warp, int lane, float scale, uint8_t *stage, float *dst, int E, int nrows, bool off)
{
    const int wq = warp & 3, hf = warp >> 2;
    uint8_t *box = stage + (D == 64 ? warp : wq) * 4096;
#pragma unroll
    for (int c = 0; c < D / 8; ++c)
        *reinterpret_cast<float4 *>(box + sw128(lane, D == 64 ? c : hf * 4 + c)) = make_float4(o[4 * c] * scale, o[4 * c + 1] * scale, o[4 * c + 2] * scale, o[4 * c + 3] * scale);
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

// ---- rows: log-sum-exp, w, dQ --------------------------------------------------------------------------
// STORED: where the probabilities come from.  0: formed again from Q and K.  1: the caller's, one tile ahead through registers
// (rows that TMA cannot address: S not a multiple of four).  2: the caller's, by TMA into a ring of tiles: a tile of
// the first sweep took 1.2 us, which was the latency of the loads one tile ahead; no registers and no turning are needed
// either (B=32 H=8 S=256 D=32: 109.9 -> 102.5 us, B=2 H=16 S=1024 D=64: 258 -> 212).
constexpr int kPTile = kLanes * kTile * 4;           // bytes of a tile of probabilities
template <int STORED>
using PMap = std::conditional_t<STORED == 2, CUtensorMap, int>;
template <int D>
constexpr int kPStages = D == 32 ? 3 : 2;

template <int D, int STORED>
struct RowsCfg {
    static constexpr int kKStages = D == 32 ? 4 : (STORED ? 2 : 3);      // what 227 KB hold beside Q, dO and the probabilities
    static constexpr int kVStages = D == 32 ? 4 : 2;
    static constexpr int kResident = (STORED ? 1 : 2) * 2 * Img<D>::kTileBytes;      // dO and, to form P again, Q: 128 rows each
    // 1: per warp 32 rows x 32 probabilities on their way to their rows
    static constexpr int kStage = STORED == 2 ? kPStages<D> * kPTile : STORED == 1 ? kWorkerWarps * 4096 : 0;
    static constexpr size_t kSmem = (STORED == 2 ? 1024 : 0) + (size_t)kResident + (kKStages + kVStages) * Img<D>::kTileBytes + kStage;
    static constexpr uint32_t kColAcc = 4 * kTile;                       // after two buffers of S and dP: two accumulators of 2 D columns
};

template <int D, bool CAUSAL, int STORED>
__global__ void __launch_bounds__(kThreads, 1)
bwd_rows_kernel(const uint8_t *__restrict__ img, size_t img_bytes, const float *__restrict__ P, float *__restrict__ dQ,
                float *__restrict__ lse_out, float *__restrict__ w_out, int S, int Spad, int E, int H, int nblk, float c, const __grid_constant__ PMap<STORED> p_map, int expire)
{
    using C = RowsCfg<D, STORED>;
    constexpr int TB = Img<D>::kTileBytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *p_s = STORED == 2 ? reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023) : smem_raw;
    uint8_t *q_s = p_s + C::kStage, *g_s = q_s + (STORED ? 0 : 2 * TB), *k_s = g_s + 2 * TB, *v_s = k_s + C::kKStages * TB;
    __shared__ uint64_t res_full, k_full[C::kKStages], v_full[C::kVStages], sd_full[2], ready[2], acc_done[2], p_full[STORED == 2 ? kPStages<D> : 1];
    __shared__ float comb[2][STORED ? 1 : 3][kLanes];           // w and, where P is formed again, maximum and sum of each half row
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
        for (int i = 0; i < 2; ++i) { mbar_init(&sd_full[i], STORED ? 1 : 2); mbar_init(&ready[i], kWorkerWarps); mbar_init(&acc_done[i], 2); }      // (commits: one per issuing warp)
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
    // the workers' wait: without stored probabilities they are short of registers (B=3 H=12 S=777 D=64 causal: 114.4 us with the wait above)
    auto wait_w = [&](uint64_t *bar, uint32_t parity, int site) {
        if (STORED) return wait(bar, parity, site);
        if (abort_flag || mbar_test(bar, parity)) return;
        bwd_wait_slow(bar, parity, site, &abort_flag, expire);
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
            if (first) {
                if (STORED) return;
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
                auto a_col = [&](int p, int hf) { return p == 2 ? s0 + kTile + 32 * hf : s0 + 32 * hf + 16 * p; };
                if (first) issue_accumulate<D, true, 0, 2>(tmem + C::kColAcc, a_col, kt);
                else issue_accumulate<D, true, 2, 4>(tmem + C::kColAcc + 2 * D, a_col, kt);
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
            wait_w(&p_full[i % kPStages<D>], (uint32_t)((i / kPStages<D>) & 1), 7);
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

    float m = -INFINITY, l = 0.0f, w = 0.0f, lse = 0.0f;
    float o[D / 2];
#pragma unroll
    for (int x = 0; x < D / 2; ++x) o[x] = 0.0f;
    auto add_dq = [&](int i) {                       // tile i of the second sweep has been accumulated
        wait_w(&acc_done[i & 1], (uint32_t)(((i - nk) >> 1) & 1), 6);
        tc_fence_after();
        add_tile<D, true>(lane_base + C::kColAcc, hf, o);
        add_tile<D, true>(lane_base + C::kColAcc + 2 * D, hf, o);
    };
    if (STORED == 1) fetch_p(0);
    for (int i = 0; i < total; ++i) {
        const uint32_t s_addr = lane_base + (uint32_t)((i & 1) * 2 * kTile) + hf * 32, dp_addr = s_addr + kTile;
        const int j0 = (i % nk) * kTile + hf * 32;
        const int nvalid = min(S - j0, CAUSAL ? row - j0 + 1 : 32);      // columns of this row that count
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
                w = (hf == 0 ? wa + wb : wb + wa) / fmaxf(l, 1e-30f);
                lse = mn + log2f(fmaxf(l, 1e-30f));
            }
            if (hf == 0) {                           // rows past S: a probability of 0 for every key
                // after a wait that ran out: NaN, so that no block of columns makes a result of what the buffer held before
                const bool lost = abort_flag;
                if (!STORED) lse_out[(size_t)bh * Spad + row] = lost ? NAN : row < S ? lse : 1e30f;
                w_out[(size_t)bh * Spad + row] = lost ? NAN : row < S ? w : 0.0f;
            }
        }
        if (STORED) {
            take_p(i, s);
            if (STORED == 1 && i + 1 < total) fetch_p(i + 1);       // in flight during this tile
        }
        wait_w(&sd_full[i & 1], (uint32_t)((i >> 1) & 1), 4);
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
                w += (ws[0].x + ws[0].y) + (ws[1].x + ws[1].y);
            } else if (nvalid > 0) {
                float mx = -INFINITY;
                if (nvalid < 32) {
#pragma unroll
                    for (int x = 0; x < 32; ++x) s[x] = x < nvalid ? s[x] : -INFINITY;
                }
#pragma unroll
                for (int x = 0; x < 32; x += 2) mx = max3(mx, s[x], s[x + 1]);
                const float mn = fmaxf(m, mx * cl2), alpha = ex2_approx(m - mn);
                m = mn;
                float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, ws[2] = {ls[0], ls[0]};
#pragma unroll
                for (int x = 0; x < 32; x += 2) {
                    const float2 t = ffma2(make_float2(s[x], s[x + 1]), make_float2(cl2, cl2), make_float2(-mn, -mn));
                    const float2 e = make_float2(ex2_approx(t.x), ex2_approx(t.y));
                    ls[(x >> 1) & 1] = fadd2(ls[(x >> 1) & 1], e);
                    ws[(x >> 1) & 1] = ffma2(e, make_float2(dp[x], dp[x + 1]), ws[(x >> 1) & 1]);
                }
                l = fmaf(l, alpha, (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y));
                w = fmaf(w, alpha, (ws[0].x + ws[0].y) + (ws[1].x + ws[1].y));
            }
        } else {
#pragma unroll
            for (int x = 0; x < 32; x += 2) {
                float2 p = make_float2(s[x], s[x + 1]);
                if (!STORED) {
                    p = ffma2(p, make_float2(cl2, cl2), make_float2(-lse, -lse));
                    p = make_float2(ex2_approx(p.x), ex2_approx(p.y));
                }
                const float2 d = fadd2(make_float2(dp[x], dp[x + 1]), make_float2(-w, -w));
                dp[x] = p.x * d.x;
                dp[x + 1] = p.y * d.y;
            }
            if (nvalid < 32) {
#pragma unroll
                for (int x = 0; x < 32; ++x) dp[x] = x < nvalid ? dp[x] : 0.0f;
            }
            store_pieces(dp, s_addr, s_addr + 16, dp_addr);
            if (i > nk) add_dq(i - 1);
            tmem_wait_st();
            arrive(&ready[i & 1]);
        }
    }
    add_dq(total - 1);
    // (through the K tiles' memory: the last product has read it)
    const int row0 = q0 + wq * 32;
    store_out<D>(o, warp, lane, c, k_s, dQ + ((size_t)b * S + row0) * E + (size_t)h * D, E, S - row0, abort_flag);
    tc_fence_before();
    __syncthreads();
}

// ---- columns: dK, dV -----------------------------------------------------------------------------------
template <int D, int STORED>
struct ColsCfg {
    static constexpr int kStages = D == 32 ? 4 : 2;                      // (Q, dO) tile pairs
    static constexpr int kResident = (STORED ? 1 : 2) * 2 * Img<D>::kTileBytes;      // V and, to form P again, K: 128 rows each
    static constexpr int kStage = STORED == 2 ? kPStages<D> * kPTile : 0;
    static constexpr size_t kSmem = (STORED == 2 ? 1024 : 0) + (size_t)kResident + kStages * 2 * Img<D>::kTileBytes + kStage;
    static constexpr uint32_t kBuf = 3 * kTile;                          // S^T, dP^T and room: six pieces take 192 columns
    static constexpr uint32_t kColV = 2 * kBuf, kColK = kColV + 64;
    static constexpr bool kWide = D == 32;                               // 64 columns per accumulator
    // w and lse by bulk copy, tiles ahead, or by the workers' loads: those stand between the scores and ds (0.3 us per tile of 1.4, 1.4 in
    // a block's first at D = 32 with stored probabilities: 100.7 -> 97.8 us at B=32 H=8 S=256), but where the rest of a tile is short
    // and a block has a tile or two the copy's longer way costs more (D = 32 without them, S = 64: 17.1 against 17.5 us)
    static constexpr bool kRowsAhead = STORED != 0 || D == 64;
};

template <int D, bool CAUSAL, int STORED>
__global__ void __launch_bounds__(kThreads, 1)
bwd_cols_kernel(const uint8_t *__restrict__ img, size_t img_bytes, const float *__restrict__ P, float *__restrict__ dK, float *__restrict__ dV,
                const float *__restrict__ lse_in, const float *__restrict__ w_in, int S, int Spad, int E, int H, int nblk, float c, const __grid_constant__ PMap<STORED> p_map, int expire)
{
    using C = ColsCfg<D, STORED>;
    constexpr int TB = Img<D>::kTileBytes;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *p_s = STORED == 2 ? reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023) : smem_raw;
    uint8_t *k_s = p_s + C::kStage, *v_s = k_s + (STORED ? 0 : 2 * TB), *t_s = v_s + 2 * TB;     // t_s: [stage][Q tile | dO tile]
    __shared__ __align__(16) float rows_s[C::kStages][2][kTile];         // w and, to form P again, lse of a tile's queries
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
    // packing before it let this one start); who reads w and lse waits for it.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_slot;
    // site codes: 11 resident operands, 12 tile pair, 14 scores, 15 workers at a tile, 16 accumulation, 17 probabilities, 18 w and lse
    bool seen = true;                                // what this thread waited for last has come (for who asks for copies then)
    auto wait = [&](uint64_t *bar, uint32_t parity, int site) {
        const int gone = abort_flag;                 // (before the test, and not in its way)
        const bool done = mbar_test(bar, parity);
        seen = !gone;
        if (!gone && !done) seen = bwd_wait_slow(bar, parity, site, &abort_flag, expire);
    };
    // the workers' wait: without stored probabilities they are short of registers (B=3 H=12 S=777 D=64 causal: 114.4 us with the wait above)
    auto wait_w = [&](uint64_t *bar, uint32_t parity, int site) {
        if (STORED) return wait(bar, parity, site);
        if (abort_flag || mbar_test(bar, parity)) return;
        bwd_wait_slow(bar, parity, site, &abort_flag, expire);
    };

    if (warp >= kWorkerWarps) {
        // the first issuing warp: S^T = K Q^T and dV; the second: dP^T = V dO^T and dK
        const bool first = warp == kWorkerWarps;
        const uint8_t *q_img = img + (size_t)bh * Spad * (Img<D>::kBlock / 8);
        const uint8_t *k_img = q_img + img_bytes + (size_t)k0 * (Img<D>::kBlock / 8), *v_img = k_img + img_bytes, *g_img = q_img + 3 * img_bytes;
        auto fetch = [&](int i) {
            if (lane == 0 && i < total && seen) {
                uint64_t *bar = &full[i % C::kStages];
                uint8_t *dst = t_s + (i % C::kStages) * 2 * TB;
                mbar_arrive_expect_tx(bar, 2 * TB);
                bulk_load(dst, q_img + (size_t)(t0 + i) * TB, TB, bar);
                bulk_load(dst + TB, g_img + (size_t)(t0 + i) * TB, TB, bar);
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
                mbar_arrive_expect_tx(bar, (STORED ? 1 : 2) * kTile * 4);
                bulk_load(rows_s[i % C::kStages][0], w_in + at, kTile * 4, bar);
                if (!STORED) bulk_load(rows_s[i % C::kStages][1], lse_in + at, kTile * 4, bar);
            }
            __syncwarp();
        };
        auto issue_sd = [&](int i) {
            if (STORED && first) return;
            const uint32_t d = tmem + (uint32_t)(i & 1) * C::kBuf, t = smem_u32(t_s + (i % C::kStages) * 2 * TB);
            wait(&full[i % C::kStages], (uint32_t)((i / C::kStages) & 1), 12);
            tc_fence_after();
            if (first) issue_scores<D>(d, smem_u32(k_s), t);
            else issue_scores<D>(d + kTile, smem_u32(v_s), t + TB);
            if (elect_one()) tc_commit(&sd_full[i & 1]);
        };
        wait(&res_full, 0, 11);
        tc_fence_after();
        issue_sd(0);
        if (!first && C::kRowsAhead) {
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
            if (!first && C::kRowsAhead) fetch_w(i + C::kStages);                     // ... and its w and lse
            const uint32_t s0 = tmem + (uint32_t)(i & 1) * C::kBuf, t = smem_u32(t_s + (i % C::kStages) * 2 * TB);
            auto p_col = [&](int p, int hf) { return p == 2 ? s0 + kTile + 32 * hf : s0 + 32 * hf + 16 * p; };
            auto ds_col = [&](int p, int hf) { return p == 0 ? s0 + kTile + 32 * hf + 16 : s0 + 2 * kTile + 32 * hf + 16 * (p - 1); };
            if (first) issue_accumulate<D, C::kWide, 0, 4>(tmem + C::kColV, p_col, t + TB);
            else issue_accumulate<D, C::kWide, 0, 4>(tmem + C::kColK, ds_col, t);
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
        wait_w(&acc_done[i & 1], (uint32_t)((i >> 1) & 1), 16);
        tc_fence_after();
        add_tile<D, C::kWide>(lane_base + C::kColV, hf, ov);
        add_tile<D, C::kWide>(lane_base + C::kColK, hf, ok);
    };
    if (STORED == 1) fetch_p(0);
    if (!C::kRowsAhead) dependency_wait();
    for (int i = 0; i < total; ++i) {
        const uint32_t s_addr = lane_base + (uint32_t)(i & 1) * C::kBuf + hf * 32, dp_addr = s_addr + kTile, room = s_addr + 2 * kTile;
        const int qb = (t0 + i) * kTile + hf * 32;
        const size_t at = (size_t)bh * Spad + qb;
        const float *wrow = C::kRowsAhead ? rows_s[i % C::kStages][0] + hf * 32 : w_in + at, *lrow = C::kRowsAhead ? rows_s[i % C::kStages][1] + hf * 32 : lse_in + at;
        const bool mask = CAUSAL && qb < k0 + wq * 32 + 31;              // some lane of the warp has a key after some query
        float p[32], d[32];
        if (STORED == 1) {
#pragma unroll
            for (int x = 0; x < 32; ++x) p[x] = pn[STORED == 1 ? x : 0];
            if (i + 1 < total) fetch_p(i + 1);       // in flight during this tile
        }
        if (STORED == 2) {
            wait_w(&p_full[i % kPStages<D>], (uint32_t)((i / kPStages<D>) & 1), 17);
            const uint8_t *src = p_s + (i % kPStages<D>) * kPTile + wq * (kPTile / 4) + (lane & 3) * 4;
#pragma unroll
            for (int x = 0; x < 32; ++x) p[x] = *reinterpret_cast<const float *>(src + sw128(hf * 32 + x, lane >> 2));
        }
        wait_w(&sd_full[i & 1], (uint32_t)((i >> 1) & 1), 14);
        tc_fence_after();
        if (!STORED) tmem_ld32(s_addr, p);
        tmem_ld32(dp_addr, d);
        tmem_wait_ld();
        if (C::kRowsAhead) wait_w(&w_full[i % C::kStages], (uint32_t)((i / C::kStages) & 1), 18);
        if (!STORED) {
#pragma unroll
            for (int x = 0; x < 32; x += 4) {
                const float4 ls = *reinterpret_cast<const float4 *>(lrow + x);       // rows past S: a probability of 0
                float2 a = ffma2(make_float2(p[x], p[x + 1]), make_float2(cl2, cl2), make_float2(-ls.x, -ls.y));
                float2 e = ffma2(make_float2(p[x + 2], p[x + 3]), make_float2(cl2, cl2), make_float2(-ls.z, -ls.w));
                p[x] = ex2_approx(a.x); p[x + 1] = ex2_approx(a.y); p[x + 2] = ex2_approx(e.x); p[x + 3] = ex2_approx(e.y);
            }
        }
        if (mask) {
#pragma unroll
            for (int x = 0; x < 32; ++x) p[x] = key <= qb + x ? p[x] : 0.0f;
        }
#pragma unroll
        for (int x = 0; x < 32; x += 4) {
            const float4 w4 = *reinterpret_cast<const float4 *>(wrow + x);
            d[x] = p[x] * (d[x] - w4.x); d[x + 1] = p[x + 1] * (d[x + 1] - w4.y);
            d[x + 2] = p[x + 2] * (d[x + 2] - w4.z); d[x + 3] = p[x + 3] * (d[x + 3] - w4.w);
        }
        store_pieces(p, s_addr, s_addr + 16, dp_addr);
        store_pieces(d, dp_addr + 16, room, room + 16);
        if (i > 0) add_dkv(i - 1);
        tmem_wait_st();
        arrive(&ready[i & 1]);
    }
    add_dkv(total - 1);
    // (through the tiles' memory: the last products have read it)
    const int row0 = k0 + wq * 32;
    const size_t dst = ((size_t)b * S + row0) * E + (size_t)h * D;
    store_out<D>(ov, warp, lane, 1.0f, t_s, dV + dst, E, S - row0, abort_flag);
    store_out<D>(ok, warp, lane, c, t_s + TB * 2, dK + dst, E, S - row0, abort_flag);
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
    static_assert(rows_smem + (STORED ? 1 : 3) * 2 * kLanes * 4 + 256 <= 232448 && cols_smem + ColsCfg<D, STORED>::kStages * 2 * kTile * 4 + 512 <= 232448, "shared memory of a block");
    cudaError_t e = cudaFuncSetAttribute(rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rows_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cols_smem);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    const int nblk = (S + kLanes - 1) / kLanes, Spad = nblk * kLanes;
    // groups of batches whose images (6 bytes per element) stay in L2 between the kernels that write and read them
    const size_t per_batch = (size_t)4 * H * Spad * D * 6;
    long long gb = (long long)((96u << 20) / per_batch);
    gb = gb < 1 ? 1 : gb > B ? B : gb;
    while (gb > 1 && gb * H * (long long)(Spad / 8) * (D / 32) > 2000000000LL) gb /= 2;
    const size_t img_bytes = (size_t)gb * H * Spad * D * 6, stat = (size_t)gb * H * Spad;
    StreamWorkspace::Lease ws;
    int rc = g_bwd_ws.enter(st, 4 * img_bytes + 2 * stat * sizeof(float), &ws);
    if (rc != HIPGPT_OK) return rc;
    uint8_t *img = ws.get();
    float *lse = reinterpret_cast<float *>(img + 4 * img_bytes), *w = lse + stat;
    const float c = 1.0f / sqrtf((float)D);
    const int expire = take_expiry(600);
    for (long long b0 = 0; b0 < B; b0 += gb) {
        const int nb = (int)(B - b0 < gb ? B - b0 : gb);
        const size_t off = (size_t)b0 * S * E;
        const float *p = STORED ? probs + (size_t)b0 * H * S * S : nullptr;
        const int tasks = nb * H * (Spad / 8) * (D / 32);
        e = launch_overlapped(bwd_pack_kernel<D>, dim3((unsigned)((tasks + 7) / 8), 4), dim3(256), 0, st, q + off, k + off, v + off, g + off, img, img_bytes, S, Spad, E, H, tasks);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_pack_kernel launch: %s", cudaGetErrorString(e));
        PMap<STORED> rows_map = {}, cols_map = {};
        if constexpr (STORED == 2) {
            rc = tma_plane_map(&rows_map, p, nb * H, S, S, kLanes, CU_TENSOR_MAP_SWIZZLE_128B);
            if (rc == HIPGPT_OK) rc = tma_plane_map(&cols_map, p, nb * H, S, S, kTile, CU_TENSOR_MAP_SWIZZLE_128B);
            if (rc != HIPGPT_OK) return rc;
        }
        const dim3 grid((unsigned)(nb * H * nblk));
        e = launch_overlapped(rows, grid, dim3(kThreads), rows_smem, st, (const uint8_t *)img, img_bytes, p, dq + off, lse, w, S, Spad, E, H, nblk, c, rows_map, (expire & 255) <= 10 ? expire : 0);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_rows_kernel launch: %s", cudaGetErrorString(e));
        e = launch_overlapped(cols, grid, dim3(kThreads), cols_smem, st, (const uint8_t *)img, img_bytes, p, dk + off, dv + off, (const float *)lse,
                              (const float *)w, S, Spad, E, H, nblk, c, cols_map, (expire & 255) > 10 ? expire : 0);
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
