// Attention backward, a whole head at a time: head_dim 32 with S <= 256, head_dim 64 with S <= 128.  Same contract and the same
// arithmetic of pieces as attn_bwd_tc.cu, which keeps the longer contexts.
//
// There a call is three kernels: the operands are cut into pieces in one pass over memory, the rows' kernel reads the
// probabilities twice and forms g V^T twice, the columns' kernel reads and forms them once more, and both go from 64-column tile to
// 64-column tile with two products between, each a chain of waits (1.1 - 1.4 us per tile of B=32 H=8 S=256 D=32).  Where a head's operands fit
// shared memory one kernel does it all: 128 queries per block, all keys of the head, the two blocks of a head of more
// than 128 rows as a cluster.  Everything a block needs is on the SM at once:
//   operands       as pieces (attn_bwd_pieces.cuh), cut by the workers on the way from memory: g and Q of the block's rows, K and V of the head
//   P              128 x 256 fp32 (from memory, by TMA; or formed here), 128 KB
//   dP = g V^T     256 columns of TMEM, formed once
//   ds             as pieces in P's place, where they serve both products: read K-major for dQ = ds K, M-major for dK = ds^T Q
//   dV             formed probabilities: their two pieces take P's place first, and ds waits in dP's in fp32 until they have been read.
//                  Stored ones, which are exact: as in attn_bwd_tc.cu, from three bf16 pieces, when all else has been done: the block's keys, all queries.
// so that the sweeps of the workers (w; ds and P's pieces; ds's pieces) run over whole rows with no product to wait for inside.
// The pieces of P and ds are cut by one power of two per tile of 64 queries x 64 keys, which can leave with a row of dQ's sums (kept per tile of keys) and with
// one of dV's and dK's (kept per 64 queries): P's from its largest there, ds's from an upper bound by row (largest P |dP|, and largest P times |w|).
// The bound is no estimate: where a row has all its weight on one key it is 2 |w| and ds near zero.  The pieces' range (attn_bwd_pieces.cuh) is what covers that.
// The queries of the other block contribute to this block's keys: their sums come through distributed shared memory at the end.
//
// Measured, us, three kernels -> one: B=32 H=8 S=256 D=32 with stored probabilities 94.9 -> 74.9, causal without 80.9 -> 69.8; S=161 (probabilities that TMA cannot
// address) 84.7 -> 85.4, causal without 69.1 -> 59.8; B=16 H=12 S=128 D=32 stored 31.2 -> 25.4; B=64 H=12 S=35 82.0 -> 61.9; D=64: B=32 H=8 S=128 stored 46.2 -> 36.3, causal
// without 46.2 -> 33.0; B=9 H=16 S=101 27.2 -> 19.9.  But for odd lengths just above 128 at D=32, where both are the same, the one is faster throughout.
// Relative error of the gradients against float64: 1.45, 1.40, 0.90e-7 (dQ, dK, dV) at the first, 1.34, 1.40, 0.83e-7 at B=8 H=8 S=128 D=64 stored; three bf16
// pieces and six products throughout: 1.47, 1.68, 0.94e-7 and 1.41, 1.63, 0.83e-7.  (dV of two fp16 pieces: 1.03 and 0.95e-7; 69.0 us at the first.)
// What bounds it: a block takes about 32000 cycles at the first shape, 3.5 rounds of them.  9700 until its operands are cut and g V^T is there (224 KB come in at
// 64 bytes per clock; the cut is bound by the instructions of conversion), 4500 for w and the scales, 5300 for ds and its pieces, 4300 for the products with
// them and the other block's sums, 6000 for dV (900 dO's pieces, 900 per tile of probabilities, the last product), 1700 for the output.
// Steps, B=32 H=8 S=256 D=32 stored: eight worker warps 76.7, sixteen 72.9; operands as whole sectors, two issuing warps, no stall between the reading of a tile's
// probabilities and the writing of its pieces 64.3; scales per 64 x 64 instead of per 64 x 256, for keys of little probability, 69.0; dV exact 77.3; its
// probabilities' next tile read while the pieces of one are on their way, the other gradients got ready during its last products, a tile's exponents read at once 74.9.
#include "attn_bwd_pieces.cuh"
#include "tma_host.cuh"

#include <math.h>

namespace hipgpt {
namespace {

constexpr int kWorkerWarps = 16;
constexpr int kThreads = kWorkerWarps * 32 + 64;
constexpr int kCols = 16;                // of a tile's 64 columns, per thread
constexpr uint32_t kTmemCols = 512;
// What the tensor core's truncation takes from the results on the average (attn_bwd_tc.cu), given back with the last multiplication
constexpr float kSumLoss = 7.3e-8f, kScoreLoss = 1.65e-7f, kScoreLoss32 = 1.3e-7f;      // the last: accumulators of 32

__device__ int g_bwd_head_status = 0;

__device__ __noinline__ bool head_wait_slow(uint64_t *bar, uint32_t parity, int site, volatile int *abort_flag, int expire)
{
    if (!expires_now(expire, site) && mbar_wait(bar, parity)) return true;
    *abort_flag = 1;
    atomicCAS(&g_bwd_head_status, 0, site);
    linger();
    return false;
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void peer_store4(uint32_t addr, float a, float b, float c, float d)
{
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}

// The pieces of P and of ds, [8 keys][piece][8 queries] core matrices of 128 bytes: 16 of them along the queries.
constexpr int kPiecePart = 16 * 128, kKeys8 = 2 * kPiecePart, kGroup = 4 * kKeys8;          // a piece of 8 keys, 8 keys, 32 keys

// NB: blocks of a head
template <int D, int NB>
struct HeadCfg {
    static constexpr int TB = Img<D>::kTileBytes;
    static constexpr int kP = NB * 4 * kGroup;                           // probabilities, then their pieces, then those of ds
    static constexpr int kG = kP, kQ = kG + 2 * TB, kV = kQ + 2 * TB, kK = kV + NB * 2 * TB, kSmall = kK + NB * 2 * TB;
    static constexpr size_t kSmem = 1024 + kSmall + 1024;
    static constexpr bool kWide = D == 32;                               // products with [hi | lo] at once, accumulators of 64 columns either way
    static constexpr int kTiles = 2 * NB;                                // of 64 keys
    // columns of TMEM: dP (ds, dQ's sums of a tile); scores, then the sums of dV and dK, [block of keys][64 queries]
    static constexpr int kColAcc = 256, kColK = D == 32 ? 0 : 128, kColQ2 = 384;
    // tiles of 64 rows of the planes
    // dV of stored probabilities: g's image as three bf16 pieces, in V's and K's place (behind what the other block sends); pieces of P in TMEM, 96 columns per 64 queries, then sums
    static constexpr int kExactG = kV + (NB > 1 ? 16384 : 0), kCols3 = 96;
    static constexpr uint32_t kCol3 = kTiles * kCols3;
    static_assert(kExactG + NB * 16 * kBlock3<D> <= kSmall && kCol3 + kTiles * D <= kTmemCols, "");
    static constexpr int tG = 0, tV = 2, tQ = 2 + kTiles, tK = 4 + kTiles, kAll = 4 + 2 * kTiles;
};

// The small things behind the operands
template <int NB>
struct HeadSmall {
    uint64_t p_full[2 * NB], p3_full[NB], p3_ready[2 * NB], v3_done, scores, asked, cut[2], p_read[NB], p_ready[NB], v_done[NB], d_ready[NB], k_done[NB];
    alignas(16) uint32_t largest[4 + 4 * NB][8];                // of a tile's rows that a warp has
    float fac[4 + 4 * NB];
    alignas(16) uint32_t group_p[2][4], group_d[2][4];          // of a tile of 64 queries (first index) x 64 keys: P's largest, ds's bound
    uint32_t tmem_base;
    volatile int abort_flag, peer_gone;
};

template <int D, bool CAUSAL, bool STORED, int NB>
__global__ void __launch_bounds__(kThreads, 1)
bwd_head_kernel(const float *q, const float *k, const float *v, const float *g, const float *P, float *dQ, float *dK, float *dV,
                int S, int E, int H, float c, int by_tma, int ahead, const __grid_constant__ CUtensorMap p_map, int expire)
{
    using C = HeadCfg<D, NB>;
    // One block per head and stored probabilities, whose dV takes no columns yet: a tile's dQ from two accumulators of 32 keys, so that less is truncated
    // (B=8 H=8: dQ 1.42 -> 1.34e-7 at S = 128 D = 64, 1.39 -> 1.28e-7 at S = 64 D = 32, where three bf16 pieces gave 1.41 and 1.38; 35.4 -> 36.1 us at B=32 H=8 S=128 D=64)
    constexpr bool kHalves = STORED && NB == 1;
    constexpr int kColK = STORED ? 0 : C::kColK;
    constexpr int TB = C::TB;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t *p_s = sm, *g_s = sm + C::kG, *q_s = sm + C::kQ, *v_s = sm + C::kV, *k_s = sm + C::kK;
    using Small = HeadSmall<NB>;
    Small &sh = *reinterpret_cast<Small *>(sm + C::kSmall);
    static_assert(sizeof(Small) <= 1024 && C::kSmem <= 232448, "shared memory of a block");

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int blk = NB > 1 ? (int)blockIdx.x % NB : 0, bh = (int)blockIdx.x / NB;
    const int b = bh / H, h = bh % H, q0 = blk * kLanes, next = (int)blockIdx.x + ahead;
    const int nkb = CAUSAL ? blk + 1 : NB;           // blocks of 128 keys that these queries see
    const int ntile = (min(S, nkb * kLanes) + kTile - 1) / kTile;
    const int qb0 = CAUSAL ? blk : 0, nqb = (S + kLanes - 1) / kLanes, nq = (S + kTile - 1) / kTile;      // blocks and tiles of queries that see these keys: from qb0, 2 qb0 on
    auto block_at = [&](int i) { return nkb == 1 ? 0 : i == 0 ? blk ^ 1 : blk; };         // the other block's keys first: their sums have a way to go
    // the block of keys whose place the probabilities of query block j take later on
    auto place = [&](int j) { return nkb == 1 ? j - qb0 : block_at(j - qb0); };

    if (tid == 0) {
        sh.abort_flag = 0;
        sh.peer_gone = 0;
        for (int t = 0; t < 2 * NB; ++t) sh.group_p[0][t] = sh.group_p[1][t] = sh.group_d[0][t] = sh.group_d[1][t] = 0;
        for (int i = 0; i < 2 * NB; ++i) { mbar_init(&sh.p_full[i], 1); mbar_init(&sh.p3_ready[i], kWorkerWarps); }
        for (int i = 0; i < NB; ++i) mbar_init(&sh.p3_full[i], 1);
        mbar_init(&sh.v3_done, 2);
        mbar_init(&sh.scores, 2);                    // (commits: one per issuing warp)
        for (int i = 0; i < 2; ++i) mbar_init(&sh.cut[i], kWorkerWarps);
        mbar_init(&sh.asked, kWorkerWarps);
        for (int i = 0; i < NB; ++i) { mbar_init(&sh.p_read[i], kWorkerWarps); mbar_init(&sh.p_ready[i], kWorkerWarps); mbar_init(&sh.v_done[i], 2); mbar_init(&sh.d_ready[i], kWorkerWarps); mbar_init(&sh.k_done[i], 2); }
    }
    if (warp == kWorkerWarps) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh.tmem_base;
    dependency_wait();
    dependents_may_start();
    // site codes: 21 operands asked for or cut, 22 probabilities, 23 scores, 24 workers' pieces, 25 dV, 26 dQ and dK, 27 probabilities read
    auto wait = [&](uint64_t *bar, uint32_t parity, int site) {
        const int gone = sh.abort_flag;              // (before the test, and not in its way)
        const bool done = mbar_test(bar, parity);
        if (!gone && !done) head_wait_slow(bar, parity, site, &sh.abort_flag, expire);
    };

    if (warp >= kWorkerWarps) {
        // ---- two warps that issue side by side; the first fetches the probabilities ----
        const int mine = warp - kWorkerWarps;
        if (STORED && by_tma && mine == 0) {
            wait(&sh.asked, 0, 21);                  // (the operands are needed first)
            if (lane == 0)
                for (int t = 0; t < ntile; ++t) {
                    mbar_arrive_expect_tx(&sh.p_full[t], 2 * kGroup);
                    for (int u = 0; u < 2; ++u) tma_load_3d(p_s + (2 * t + u) * kGroup, &p_map, t * kTile + 32 * u, q0, bh, &sh.p_full[t]);
                }
            __syncwarp();
        }
        // (128 x 128) = A B^T over the head dimension, both images read K-major
        auto scores = [&](uint32_t d, const uint8_t *as, const uint8_t *bs) {
            const uint64_t da = make_desc(smem_u32(as), 128, Img<D>::kBlock, 0), db = make_desc(smem_u32(bs), 128, Img<D>::kBlock, 0);
            constexpr uint32_t id = idesc_f16(kLanes, kLanes);
            constexpr int PA[4] = {1, 1, 0, 0}, PB[4] = {1, 0, 1, 0};    // small terms first; the smallest where the probabilities, stored, are exact
#pragma unroll
            for (int p = STORED ? 0 : 1; p < 4; ++p)
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks)
                    if (elect_one()) {
                        const uint64_t ak = da + (uint64_t)((PA[p] * (D / 8) + 2 * ks) * 8), bk = db + (uint64_t)((PB[p] * (D / 8) + 2 * ks) * 8);
                        if (ks == 0 && (p == 3 || (STORED && p == 1))) mma_h_ss_down<kLowShift>(d, ak, bk, id);
                        else mma_h_ss(d, ak, bk, id, p > (STORED ? 0 : 1) || ks > 0 ? 1u : 0u);
                    }
        };
        // acc (128 x D; WIDE: 2 D, the products with B's lo pieces apart) = A B over 64 rows of B's image, read N-major.  da: the descriptor of A's hi
        // pieces; a_step: 16 reductions on, in 16 bytes; id: A K- or M-major.  The small products first, a fresh accumulator per 64.
        auto sums = [&](uint32_t acc, uint64_t da, int a_step, uint32_t id, const uint8_t *bs, int from = 0, int to = 4) {
            const uint64_t db = make_desc(smem_u32(bs), Img<D>::kBlock, 128, 0);
            enum { kFresh, kDown, kMore };           // how a product finds the accumulator
            auto product = [&](int pa, int pb, int start) {
#pragma unroll
                for (int ks = 0; ks < 4; ++ks)
                    if (ks >= from && ks < to && elect_one()) {
                        const uint64_t ak = da + (uint64_t)(pa * (kPiecePart >> 4) + ks * a_step), bk = db + (uint64_t)(ks * 2 * (Img<D>::kBlock >> 4) + pb * (Img<D>::kPiece >> 4));
                        if (start == kDown && ks == from) mma_h_ss_down<kLowShift>(acc, ak, bk, id);
                        else mma_h_ss(acc, ak, bk, id, start == kFresh && ks == from ? 0u : 1u);
                    }
            };
            if (!C::kWide && STORED) product(1, 1, kFresh);      // (WIDE has it in any case.  Formed probabilities carry more than it takes away)
            product(1, 0, C::kWide || !STORED ? kFresh : kDown);
            if (!C::kWide) product(0, 1, kMore);
            product(0, 0, kDown);
        };
        constexpr uint32_t id_sums = idesc_f16(kLanes, C::kWide ? 2 * D : D) | (1u << 16);
        // the M-major image of 128 keys: A of dV and dK
        auto keys_desc = [&](int kb, int u) { return make_desc(smem_u32(p_s + kb * 16 * kKeys8 + u * 8 * 128), 128, kKeys8, 0); };
        wait(&sh.cut[0], 0, 21);
        tc_fence_after();
        for (int kb = 0; kb < nkb; ++kb)
            if ((kb & 1) == mine) scores(tmem + kb * kLanes, g_s, v_s + kb * 2 * TB);
        if (!STORED) {
            wait(&sh.cut[1], 0, 21);
            tc_fence_after();
            for (int kb = 0; kb < nkb; ++kb)
                if ((kb & 1) != mine) scores(tmem + C::kColAcc + kb * kLanes, q_s, k_s + kb * 2 * TB);
        }
        if (elect_one()) tc_commit(&sh.scores);
        if (STORED) wait(&sh.cut[1], 0, 21);
        if (NB > 1) cluster_arrive();
        for (int i = 0; i < (STORED ? 0 : nkb); ++i) {
            const int kb = block_at(i);
            wait(&sh.p_ready[i], 0, 24);
            tc_fence_after();
            sums(tmem + C::kColAcc + kb * 128 + 64 * mine, keys_desc(kb, mine), 256 >> 4, id_sums | (1u << 15), g_s + mine * TB);
            if (elect_one()) tc_commit(&sh.v_done[i]);
        }
        for (int i = 0; i < nkb; ++i) {
            const int kb = block_at(i);
            wait(&sh.d_ready[i], 0, 24);
            tc_fence_after();
            sums(tmem + C::kColAcc + kColK + kb * 128 + 64 * mine, keys_desc(kb, mine), 256 >> 4, id_sums | (1u << 15), q_s + mine * TB);
            const int t = 2 * kb + mine;
            if (t < ntile) {
                const uint64_t da = make_desc(smem_u32(p_s + t * 2 * kGroup), kKeys8, 128, 0);
                sums(tmem + t * kTile, da, 2 * kKeys8 >> 4, id_sums, k_s + t * TB, 0, kHalves ? 2 : 4);
                if (kHalves) sums(tmem + C::kColQ2 + t * kTile, da, 2 * kKeys8 >> 4, id_sums, k_s + t * TB, 2, 4);
            }
            if (elect_one()) tc_commit(&sh.k_done[i]);
        }
        if (NB > 1) {                                // (before the workers are needed again: theirs wait for these arrivals too)
            cluster_wait();
            cluster_arrive();
        }
        if constexpr (STORED) {
            for (int i = 0; i < nkb; ++i) {          // a block of keys' pieces have been read: a block of queries' probabilities take their place
                wait(&sh.k_done[i], 0, 26);
                if (by_tma && mine == 0 && lane == 0 && !sh.abort_flag)
                    for (int j = qb0 + i; j < (i + 1 < nkb ? min(qb0 + i + 1, nqb) : nqb); ++j) {
                        mbar_arrive_expect_tx(&sh.p3_full[j], 4 * kGroup);
                        for (int x = 0; x < 4; ++x) tma_load_3d(p_s + (4 * place(j) + x) * kGroup, &p_map, q0 + 32 * x, j * kLanes, bh, &sh.p3_full[j]);
                    }
                __syncwarp();
            }
            for (int t = 2 * qb0 + mine; t < nq; t += 2) {
                wait(&sh.p3_ready[t], 0, 24);
                tc_fence_after();
                const uint64_t db = make_desc(smem_u32(sm + C::kExactG + t * 8 * kBlock3<D>), kBlock3<D>, 128, 0);
#pragma unroll
                for (int p = 0; p < 6; ++p)
#pragma unroll
                    for (int ks = 0; ks < 4; ++ks)
                        if (elect_one()) mma_h_ts(tmem + C::kCol3 + t * D, tmem + t * C::kCols3 + kExactA[p] * 32 + ks * 8, db + (uint64_t)(ks * 2 * (kBlock3<D> >> 4) + kExactB[p] * (Img<D>::kPiece >> 4)), idesc_bf16(kLanes, D, 1), p + ks > 0 ? 1u : 0u);
            }
            if (elect_one()) tc_commit(&sh.v3_done);
        }
        __syncwarp();
        if (sh.abort_flag) linger();
        if (NB > 1) cluster_wait();
        tc_fence_before();
        __syncthreads();
        if (mine == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
        return;
    }

    // ---- workers: thread = query row (later: key), 16 of the 64 columns of a tile; four warps to a lane quarter ----
    const int wq = warp & 3, cf = warp >> 2;
    const int rloc = wq * 32 + lane, row = q0 + rloc, u = wq >> 1;       // u: which 64 rows
    const uint32_t lane_base = tmem + ((uint32_t)(wq * 32) << 16), my_tile = lane_base + cf * kCols;
    auto arrive = [&](uint64_t *bar) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
    };
    auto meet = [] { asm volatile("bar.sync 1, 512;" ::: "memory"); };

    // The operands: a warp takes eight rows of one of two tiles of 64, lane = (column block of 8) * 8 + row (whole lines in, core matrices of 128
    // bytes out); everything is asked for at once.
    {
        constexpr int PARTS = D / 32, PAIRS = C::kAll / 2;
        const int second = warp >> 3, r8 = warp * 8 + (lane & 7), col = (lane >> 3) * 8;
        float4 x[PAIRS][PARTS][2];
        // whole sectors where the planes allow it: as two halves each was asked for twice
        const bool sectors = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(g)) & 31) == 0;
#pragma unroll
        for (int t = 0; t < PAIRS; ++t) {
            const bool keys = (2 * t >= C::tV && 2 * t < C::tQ) || 2 * t >= C::tK;
            const float *src = 2 * t < C::tV ? g : 2 * t < C::tQ ? v : 2 * t < C::tK ? q : k;
            const int at = (keys ? (2 * t - (2 * t >= C::tK ? C::tK : C::tV)) * kTile : q0) + r8;
            const bool here = at < S && (!keys || at < nkb * kLanes);
            const float4 *p4 = reinterpret_cast<const float4 *>(src + ((size_t)b * S + at) * E + (size_t)h * D + col);
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                x[t][p][0] = x[t][p][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (here && sectors) {
                    load_sector(p4 + 8 * p, x[t][p][0], x[t][p][1]);
                } else if (here) {
                    x[t][p][0] = p4[8 * p];
                    x[t][p][1] = p4[8 * p + 1];
                }
            }
        }
        arrive(&sh.asked);
        // a tile's largest finite magnitude: an infinity becomes NaN in its own row and the tile's other rows keep their scale
#pragma unroll
        for (int t = 0; t < PAIRS; ++t) {
            float mx = 0.0f;
#pragma unroll
            for (int p = 0; p < PARTS; ++p)
#pragma unroll
                for (int i = 0; i < 2; ++i) mx = max3(max3(mx, fabsf(x[t][p][i].x), fabsf(x[t][p][i].y)), fabsf(x[t][p][i].z), fabsf(x[t][p][i].w));
            uint32_t bits = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
            if (bits >= 0x7f800000u) {
                uint32_t fin = 0;
#pragma unroll
                for (int p = 0; p < PARTS; ++p)
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const uint32_t m = __float_as_uint(reinterpret_cast<const float *>(x[t][p])[i]) & 0x7fffffffu;
                        fin = m < 0x7f800000u ? max(fin, m) : fin;
                    }
                bits = __reduce_max_sync(0xffffffffu, fin);
            }
            if (lane == 0) sh.largest[2 * t + second][warp & 7] = bits;
        }
        meet();
#pragma unroll
        for (int t = 0; t < PAIRS; ++t) {
            const uint4 a = *reinterpret_cast<const uint4 *>(&sh.largest[2 * t + second][0]), z = *reinterpret_cast<const uint4 *>(&sh.largest[2 * t + second][4]);
            const uint32_t e = range_exponent(max(max(max(a.x, a.y), max(a.z, a.w)), max(max(z.x, z.y), max(z.z, z.w))));
            const float up = range_up(e);
            if ((warp & 7) == 0 && lane == 0) sh.fac[2 * t + second] = range_down(e);
            uint8_t *img = 2 * t < C::tV ? g_s : 2 * t < C::tQ ? v_s + (2 * t - C::tV) * TB : 2 * t < C::tK ? q_s : k_s + (2 * t - C::tK) * TB;
            img += warp * Img<D>::kBlock + (lane >> 3) * 128 + (lane & 7) * 16;
#pragma unroll
            for (int p = 0; p < PARTS; ++p) {
                const float *xs = reinterpret_cast<const float *>(x[t][p]);
                uint4 hi, lo;
                cut2(fmul2(make_float2(xs[0], xs[1]), make_float2(up, up)), hi.x, lo.x);
                cut2(fmul2(make_float2(xs[2], xs[3]), make_float2(up, up)), hi.y, lo.y);
                cut2(fmul2(make_float2(xs[4], xs[5]), make_float2(up, up)), hi.z, lo.z);
                cut2(fmul2(make_float2(xs[6], xs[7]), make_float2(up, up)), hi.w, lo.w);
                *reinterpret_cast<uint4 *>(img + p * 512) = hi;
                *reinterpret_cast<uint4 *>(img + p * 512 + Img<D>::kPiece) = lo;
            }
            if (2 * t + 2 == C::tQ || t == PAIRS - 1) {
                proxy_fence();
                arrive(&sh.cut[2 * t + 2 == C::tQ ? 0 : 1]);
            }
        }
    }
    // probabilities whose rows TMA cannot address: a warp reads two rows of 16 at a time into the places that TMA would have used
    const int own = (cf >> 1) * kGroup + rloc * 128;  // (+ tile) this row's probabilities, 16-byte pieces permuted by the row
    if (STORED && !by_tma) {
        const float *p_rows = P + ((size_t)bh * S + q0 + wq * 32) * S;
        const int last = S - 1 - q0 - wq * 32;       // a row or column past S repeats the last one: g and V, K are zero there
        for (int t = 0; t < ntile; ++t) {
            const float *src = p_rows + min(t * kTile + cf * kCols + (lane & 15), S - 1);
            uint8_t *dst = p_s + 2 * t * kGroup + (cf >> 1) * kGroup + wq * 4096 + (lane & 3) * 4;
            float x[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) x[r] = src[(ptrdiff_t)min(2 * r + (lane >> 4), last) * S];
#pragma unroll
            for (int r = 0; r < 16; ++r) *reinterpret_cast<float *>(dst + sw128(2 * r + (lane >> 4), (cf & 1) * 4 + ((lane & 15) >> 2))) = x[r];
        }
        __syncwarp();
    }
    // what the block that follows on this SM will read is asked into L2 (memory is idle while this one computes)
    if (next < (int)gridDim.x) {
        const int nblk = NB > 1 ? next % NB : 0, nbh = next / NB;
        const int what = tid >> 7;                   // 128 threads to a plane: g and Q of its rows, K and V of its head
        const float *src = (what == 0 ? g : what == 1 ? q : what == 2 ? v : k) + (size_t)(nbh / H) * S * E + (size_t)(nbh % H) * D;
        for (int r = (what < 2 ? nblk * kLanes : 0) + (tid & 127); r < min(S, what < 2 ? (nblk + 1) * kLanes : S); r += kLanes)
            for (int x = 0; x < D; x += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(src + (size_t)r * E + x));
        if (STORED && by_tma && tid == 0) {
            const int rows = min(kLanes, S - nblk * kLanes);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(P + ((size_t)nbh * S + nblk * kLanes) * S), "r"(rows * S * 4));
        }
    }
    meet();                                          // (the factors; from here on V's image, once dP is there, serves the exchanges)
    auto read_p = [&](int t, float (&p)[kCols]) {
#pragma unroll
        for (int ch = 0; ch < 4; ++ch)
            *reinterpret_cast<float4 *>(&p[ch * 4]) = *reinterpret_cast<const float4 *>(p_s + 2 * t * kGroup + own + ((((cf & 1) * 4 + ch) ^ (rloc & 7)) << 4));
    };
    auto count = [&](int t) { const int j0 = t * kTile + cf * kCols; return min(S - j0, CAUSAL ? row - j0 + 1 : kCols); };     // columns of this row that count
    auto mask = [&](float (&x)[kCols], int nvalid, float hidden) {
        if (nvalid < kCols) {
#pragma unroll
            for (int i = 0; i < kCols; ++i) x[i] = i < nvalid ? x[i] : hidden;
        }
    };
    float (*comb)[4][kLanes] = reinterpret_cast<float (*)[4][kLanes]>(v_s);          // [what][columns' quarter][row]
    const float g_fac = sh.fac[C::tG + u], q_fac = STORED ? 0.0f : c * kLog2e * sh.fac[C::tQ + u];
    wait(&sh.scores, 0, 23);
    tc_fence_after();

    // First sweep: maximum and sum of the exponentials (where P is formed here), w, and the largest P and P |dP| of the row
    float m = -INFINITY, l = 0.0f, w = 0.0f, rinv = 1.0f, most_p[C::kTiles], most_d[C::kTiles];
    if (!STORED) {
        for (int t = 0; t < ntile; ++t) {
            const int nvalid = count(t);
            const float s_fac = fminf(fmaxf(q_fac * sh.fac[C::tK + t], 1e-37f), kFacMost);        // (never zero: a hidden score is -inf, and times the factor it stays that)
            float s[kCols];
            tmem_ld16(my_tile + C::kColAcc + t * kTile, s);
            tmem_wait_ld();
            mask(s, nvalid, -INFINITY);
            float mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < kCols; i += 2) mx = max3(mx, s[i], s[i + 1]);
            m = fmaxf(m, mx * s_fac);
        }
        comb[0][cf][rloc] = m;
        meet();
        m = fmaxf(fmaxf(fmaxf(comb[0][0][rloc], comb[0][1][rloc]), fmaxf(comb[0][2][rloc], comb[0][3][rloc])), -1e30f);
    }
#pragma unroll
    for (int t = 0; t < C::kTiles; ++t) {
        most_p[t] = most_d[t] = 0.0f;
        if (t >= ntile) continue;
        const int nvalid = count(t);
        const float dp_fac = fminf(g_fac * sh.fac[C::tV + t], kFacMost);
        float p[kCols], dp[kCols];
        if (STORED && by_tma) wait(&sh.p_full[t], 0, 22);
        if (STORED) read_p(t, p);
        if (!STORED) tmem_ld16(my_tile + C::kColAcc + t * kTile, p);
        tmem_ld16(my_tile + t * kTile, dp);
        tmem_wait_ld();
        float2 ls[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, ws[2] = {ls[0], ls[0]};
        float mp[2] = {0.0f, 0.0f}, md[2] = {0.0f, 0.0f};
        if (STORED) {
            mask(p, nvalid, 0.0f);
        } else {
            const float s_fac = fminf(fmaxf(q_fac * sh.fac[C::tK + t], 1e-37f), kFacMost);
            mask(p, nvalid, -INFINITY);
#pragma unroll
            for (int i = 0; i < kCols; i += 2) {
                const float2 x = ffma2(make_float2(p[i], p[i + 1]), make_float2(s_fac, s_fac), make_float2(-m, -m));
                p[i] = ex2_approx(x.x);
                p[i + 1] = ex2_approx(x.y);
                ls[(i >> 1) & 1] = fadd2(ls[(i >> 1) & 1], make_float2(p[i], p[i + 1]));
            }
#pragma unroll
            for (int ch = 0; ch < 4; ++ch)
                *reinterpret_cast<float4 *>(p_s + 2 * t * kGroup + own + ((((cf & 1) * 4 + ch) ^ (rloc & 7)) << 4)) = make_float4(p[4 * ch], p[4 * ch + 1], p[4 * ch + 2], p[4 * ch + 3]);
            l += (ls[0].x + ls[0].y) + (ls[1].x + ls[1].y);
        }
#pragma unroll
        for (int i = 0; i < kCols; i += 2) {
            const int z = (i >> 1) & 1;
            const float2 pp = make_float2(p[i], p[i + 1]), dd = make_float2(dp[i], dp[i + 1]), pd = fmul2(pp, dd);
            ws[z] = ffma2(pp, dd, ws[z]);
            mp[z] = max3(mp[z], fabsf(pp.x), fabsf(pp.y));
            md[z] = max3(md[z], fabsf(pd.x), fabsf(pd.y));
        }
        w = fmaf((ws[0].x + ws[0].y) + (ws[1].x + ws[1].y), dp_fac, w);
        most_p[t] = fmaxf(mp[0], mp[1]);
        most_d[t] = fmaxf(md[0], md[1]) * dp_fac;
    }
    {
        comb[1][cf][rloc] = w;
        if (!STORED) comb[2][cf][rloc] = l;
        meet();
        w = (comb[1][0][rloc] + comb[1][1][rloc]) + (comb[1][2][rloc] + comb[1][3][rloc]);
        if (!STORED) {
            rinv = 1.0f / fmaxf((comb[2][0][rloc] + comb[2][1][rloc]) + (comb[2][2][rloc] + comb[2][3][rloc]), 1e-30f);
            w *= rinv;
        }
        // (finite ones only; whatever is in a row with an infinity or a NaN stays in it)
#pragma unroll
        for (int t = 0; t < C::kTiles; ++t) {
            if (t >= ntile) break;
            uint32_t bp = __float_as_uint(most_p[t] * rinv), bd = __float_as_uint(fmaf(most_p[t], fabsf(w), most_d[t]) * rinv);
            if (!STORED) bp = __reduce_max_sync(0xffffffffu, bp < 0x7f800000u ? bp : 0u);
            bd = __reduce_max_sync(0xffffffffu, bd < 0x7f800000u ? bd : 0u);
            if (lane == 0 && !STORED) atomicMax(&sh.group_p[u][t], bp);
            if (lane == 0) atomicMax(&sh.group_d[u][t], bd);
        }
        meet();
    }
    if (NB > 1) cluster_arrive();                    // V's image is this block's no longer: the other one's sums may come
    // exponents of a tile: of its probabilities (those that are formed: at most 1) and of its ds
    auto e_p = [&](int t, int y) { return range_exponent(sh.group_p[y][t]); };
    auto e_d = [&](int t, int y) { return range_exponent(sh.group_d[y][t]); };

    // Second sweep: ds, scaled, in fp32 in dP's place; P's pieces in P's.  A block of keys' probabilities are read first: eight warps share the memory
    // that each of them then writes its pieces to (a meeting per tile, between reading and writing it, kept them all in the same step: 1300 cycles per tile).
    const int at_piece = cf * 2 * kKeys8 + (rloc >> 3) * 128 + (rloc & 7) * 16;
    auto store_pieces = [&](int t, const float (&x)[kCols], auto before) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) cut2(make_float2(x[2 * i], x[2 * i + 1]), hi[i], lo[i]);
        before();
        uint8_t *at = p_s + 2 * t * kGroup + at_piece;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            *reinterpret_cast<uint4 *>(at + i * kKeys8) = make_uint4(hi[4 * i], hi[4 * i + 1], hi[4 * i + 2], hi[4 * i + 3]);
            *reinterpret_cast<uint4 *>(at + i * kKeys8 + kPiecePart) = make_uint4(lo[4 * i], lo[4 * i + 1], lo[4 * i + 2], lo[4 * i + 3]);
        }
    };
    const uint4 all_p = STORED ? make_uint4(0, 0, 0, 0) : *reinterpret_cast<const uint4 *>(sh.group_p[u]), all_d = *reinterpret_cast<const uint4 *>(sh.group_d[u]);
    auto of_tile = [](const uint4 &v, int kb, int y) { return range_exponent(NB == 1 || kb == 0 ? (y ? v.y : v.x) : (y ? v.w : v.z)); };
    float p[2][kCols];
    auto read_block = [&](int i) {
        const int t = 2 * block_at(i);
        read_p(t, p[0]);
        if (t + 1 < ntile) read_p(t + 1, p[1]);
        arrive(&sh.p_read[i]);
    };
    read_block(0);
    for (int i = 0; i < nkb; ++i) {
        const int kb = block_at(i);
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const int t = 2 * kb + y;
            if (t >= ntile) break;
            const uint32_t ep = STORED ? 0u : of_tile(all_p, kb, y);
            const float up_d = range_up(of_tile(all_d, kb, y)), up_row = rinv * range_up(ep), ratio = STORED ? 1.0f : up_d * range_down(ep);
            const float dp_up = fminf(g_fac * sh.fac[C::tV + t], kFacMost) * ratio, w_up = w * ratio;
            float dp[kCols];
            tmem_ld16(my_tile + t * kTile, dp);
            if (STORED) mask(p[y], count(t), 0.0f);
            if (!STORED)
#pragma unroll
                for (int x = 0; x < kCols; x += 2) { const float2 z = fmul2(make_float2(p[y][x], p[y][x + 1]), make_float2(up_row, up_row)); p[y][x] = z.x; p[y][x + 1] = z.y; }
            tmem_wait_ld();
#pragma unroll
            for (int x = 0; x < kCols; x += 2) {
                float2 d = fmul2(make_float2(p[y][x], p[y][x + 1]), ffma2(make_float2(dp[x], dp[x + 1]), make_float2(dp_up, dp_up), make_float2(-w_up, -w_up)));
                if (STORED) d = fmul2(d, make_float2(up_d, up_d));       // (last: whatever the probabilities are, this is at most 2^15)
                dp[x] = d.x;
                dp[x + 1] = d.y;
            }
            if (!STORED) tmem_st16(my_tile + t * kTile, dp);
            store_pieces(t, STORED ? dp : p[y], [&] { if (y == 0) wait(&sh.p_read[i], 0, 27); });
        }
        if (i + 1 < nkb) read_block(i + 1);
        if (!STORED) tmem_wait_st();
        proxy_fence();
        tc_fence_before();
        arrive(STORED ? &sh.d_ready[i] : &sh.p_ready[i]);
    }

    // Third sweep: ds's pieces in the place of P's.  Between: this thread's columns of its key's row of dV
    constexpr int OC = D / 4;                        // columns of an output row per thread
    auto load_acc = [&](uint32_t at, float (&x)[OC]) {
        if constexpr (OC == 8) tmem_ld8(at, x);
        else tmem_ld16(at, x);
    };
    // sums over the two 64's of queries: accumulators times their factors (this thread's key is in tile 2 kb + u)
    auto key_sums = [&](uint32_t acc, float f0, float f1, float (&o)[OC]) {
        float a[2][OC], z[2][OC];
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            load_acc(acc + y * 64 + cf * OC, a[y]);
            if (C::kWide) load_acc(acc + y * 64 + D + cf * OC, z[y]);
        }
        tmem_wait_ld();
#pragma unroll
        for (int x = 0; x < OC; ++x) {
            if (C::kWide) { a[0][x] = fmaf(z[0][x], kLowDown, a[0][x]); a[1][x] = fmaf(z[1][x], kLowDown, a[1][x]); }
            o[x] = fmaf(a[1][x], f1, a[0][x] * f0);
        }
    };
    const int recv = cf * 2 * kLanes * 16 + rloc * 16;                   // [dV, dK][quarter][16 bytes][key]
    auto send = [&](const float (&o)[OC], int what) {
        if constexpr (NB > 1) {
            const uint32_t to = peer_addr(smem_u32(v_s) + recv + what * 16384, blk ^ 1);
#pragma unroll
            for (int x = 0; x < 2; ++x) peer_store4(to + x * (kLanes * 16), o[4 * x], o[4 * x + 1], o[4 * x + 2], o[4 * x + 3]);
        }
    };
    auto receive = [&](float (&o)[OC], int what) {
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const float4 y = *reinterpret_cast<const float4 *>(v_s + what * 16384 + recv + x * (kLanes * 16));
            o[4 * x] += y.x; o[4 * x + 1] += y.y; o[4 * x + 2] += y.z; o[4 * x + 3] += y.w;
        }
    };
    float ov[OC], ok[OC], oq[OC];
#pragma unroll
    for (int x = 0; x < OC; ++x) ov[x] = 0.0f;
    bool joined = NB == 1;                           // the other block has said that its V is free
    for (int i = 0; i < (STORED ? 0 : nkb); ++i) {
        const int kb = block_at(i);
        wait(&sh.v_done[i], 0, 25);
        tc_fence_after();
        for (int t = 2 * kb; t < min(2 * kb + 2, ntile); ++t) {
            float d[kCols];
            tmem_ld16(my_tile + t * kTile, d);
            tmem_wait_ld();
            store_pieces(t, d, [] {});
        }
        key_sums(lane_base + C::kColAcc + kb * 128, range_down(e_p(2 * kb + u, 0)) * sh.fac[C::tG], range_down(e_p(2 * kb + u, 1)) * sh.fac[C::tG + 1], ov);
        proxy_fence();
        tc_fence_before();
        arrive(&sh.d_ready[i]);
        if (kb != blk) {
            if (!joined) cluster_wait();
            joined = true;
            send(ov, 0);
        }
    }
    // dK; dQ from the tiles' sums, a block of keys after the other
#pragma unroll
    for (int x = 0; x < OC; ++x) oq[x] = 0.0f;
    for (int i = 0; i < nkb; ++i) {
        const int kb = block_at(i);
        wait(&sh.k_done[i], 0, 26);
        tc_fence_after();
        key_sums(lane_base + C::kColAcc + kColK + kb * 128, range_down(e_d(2 * kb + u, 0)) * sh.fac[C::tQ], range_down(e_d(2 * kb + u, 1)) * sh.fac[C::tQ + 1], ok);
        if (NB > 1 && i == 0) {                      // (every block takes both steps of the cluster's barrier twice)
            if (!joined) cluster_wait();
            if (kb != blk) {
                send(ok, STORED ? 0 : 1);
                // a warp that has seen a wait run out, its own or one that its sums depend on, says so
                if (lane == 0 && sh.abort_flag) {
                    const uint32_t gone = peer_addr(smem_u32(const_cast<int *>(&sh.peer_gone)), blk ^ 1);
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(gone), "r"(1) : "memory");
                }
            }
            cluster_arrive();
        }
        float a[2][OC], z[2][OC];
        auto load_q = [&](uint32_t col) {
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                if (2 * kb + y >= ntile) break;
                load_acc(lane_base + col + (2 * kb + y) * kTile + cf * OC, a[y]);
                if (C::kWide) load_acc(lane_base + col + (2 * kb + y) * kTile + D + cf * OC, z[y]);
            }
            tmem_wait_ld();
        };
        load_q(0);
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            if (2 * kb + y >= ntile) break;
            const float f = range_down(e_d(2 * kb + y, u)) * sh.fac[C::tK + 2 * kb + y];
#pragma unroll
            for (int x = 0; x < OC; ++x) oq[x] = fmaf(C::kWide ? fmaf(z[y][x], kLowDown, a[y][x]) : a[y][x], f, oq[x]);
        }
        if (kHalves) {
            load_q(C::kColQ2);
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                if (2 * kb + y >= ntile) break;
                const float f = range_down(e_d(2 * kb + y, u)) * sh.fac[C::tK + 2 * kb + y];
#pragma unroll
                for (int x = 0; x < OC; ++x) oq[x] = fmaf(C::kWide ? fmaf(z[y][x], kLowDown, a[y][x]) : a[y][x], f, oq[x]);
            }
        }
    }
    // 32 rows x 32 columns leave in whole lines: through shared memory (16-byte pieces permuted by the row), then a row of 128 bytes per eight lanes
    const int row0 = q0 + wq * 32;
    auto stage_rows = [&](const float (&o)[OC], float scale, float loss, uint8_t *stage) {
        uint8_t *box = stage + (D == 64 ? wq * 2 + (cf >> 1) : wq) * 4096;
#pragma unroll
        for (int i = 0; i < OC / 4; ++i) {
            float4 x = make_float4(o[4 * i] * scale, o[4 * i + 1] * scale, o[4 * i + 2] * scale, o[4 * i + 3] * scale);
            if (loss != 0.0f) { x.x = fmaf(x.x, loss, x.x); x.y = fmaf(x.y, loss, x.y); x.z = fmaf(x.z, loss, x.z); x.w = fmaf(x.w, loss, x.w); }
            *reinterpret_cast<float4 *>(box + sw128(lane, D == 64 ? (cf & 1) * 4 + i : cf * 2 + i)) = x;
        }
    };
    auto store_rows = [&](const uint8_t *stage, float *dst, bool off) {
        const uint8_t *box = stage + (D == 64 ? wq * 2 + (cf >> 1) : wq) * 4096;
        if (D == 64) asm volatile("bar.sync %0, 64;" ::"r"(4 + wq * 2 + (cf >> 1)) : "memory");
        else asm volatile("bar.sync %0, 128;" ::"r"(4 + wq) : "memory");
        constexpr int kRows = D == 64 ? 16 : 8;
#pragma unroll
        for (int i = 0; i < kRows / 4; ++i) {
            const int r = (D == 64 ? (cf & 1) : cf) * kRows + 4 * i + (lane >> 3);
            const float4 x = *reinterpret_cast<const float4 *>(box + sw128(r, lane & 7));
            if (row0 + r < S && !off) *reinterpret_cast<float4 *>(dst + ((size_t)b * S + row0 + r) * E + (size_t)h * D + (D == 64 ? (cf >> 1) * 32 : 0) + (lane & 7) * 4) = x;
        }
    };
    tc_fence_before();
    meet();                                          // the products have been waited for by all: their operands' memory is free
    tc_fence_after();
    // dV of stored probabilities, which are exact, as dO is: three bf16 pieces hold all 24 bits of both, and nothing depends on their magnitudes.  The block's
    // keys, all queries; the probabilities come a second time (from L2), turned: lane = key, 16 queries of a tile.
    if constexpr (STORED) {
        constexpr int PARTS = D / 32;
        float4 x3[NB][PARTS][2];
#pragma unroll
        for (int i = 0; i < NB; ++i) {
            const int at = i * kLanes + warp * 8 + (lane & 7);
            const float4 *g4 = reinterpret_cast<const float4 *>(g + ((size_t)b * S + at) * E + (size_t)h * D + (lane >> 3) * 8);
#pragma unroll
            for (int y = 0; y < PARTS; ++y) {
                x3[i][y][0] = x3[i][y][1] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i >= qb0 && at < S) { x3[i][y][0] = g4[8 * y]; x3[i][y][1] = g4[8 * y + 1]; }
            }
        }
#pragma unroll
        for (int i = 0; i < NB; ++i)
#pragma unroll
            for (int y = 0; y < PARTS; ++y) {
                uint8_t *at = sm + C::kExactG + (i * 16 + warp) * kBlock3<D> + (lane >> 3) * 128 + (lane & 7) * 16 + y * 512;
                uint4 pc[3];
                cut3(make_float2(x3[i][y][0].x, x3[i][y][0].y), pc[0].x, pc[1].x, pc[2].x);
                cut3(make_float2(x3[i][y][0].z, x3[i][y][0].w), pc[0].y, pc[1].y, pc[2].y);
                cut3(make_float2(x3[i][y][1].x, x3[i][y][1].y), pc[0].z, pc[1].z, pc[2].z);
                cut3(make_float2(x3[i][y][1].z, x3[i][y][1].w), pc[0].w, pc[1].w, pc[2].w);
#pragma unroll
                for (int z = 0; z < 3; ++z) *reinterpret_cast<uint4 *>(at + z * Img<D>::kPiece) = pc[z];
            }
        proxy_fence();
        float pt[16];
        auto fetch = [&](int t) {                    // this thread's 16 queries of tile t
            const int q16 = t * kTile + cf * 16;
            if (by_tma) {
                if ((t & 1) == 0) wait(&sh.p3_full[t >> 1], 0, 22);
                const uint8_t *src = p_s + (4 * place(t >> 1) + wq) * kGroup + (lane & 3) * 4;
#pragma unroll
                for (int i = 0; i < 16; ++i) pt[i] = *reinterpret_cast<const float *>(src + sw128((t & 1) * kTile + cf * 16 + i, lane >> 2));
            } else {
                // (a lane past S reads its neighbour's key: its results go nowhere)
                const float *src = P + ((size_t)bh * S + q16) * S + min(row, S - 1);
#pragma unroll
                for (int i = 0; i < 16; ++i) pt[i] = q16 + i < S ? src[(size_t)i * S] : 0.0f;
            }
        };
        fetch(2 * qb0);
#pragma unroll
        for (int n = 0; n < C::kTiles; ++n) {
            const int t = 2 * qb0 + n;
            if (t >= nq) break;
            if (CAUSAL) {
#pragma unroll
                for (int i = 0; i < 16; ++i) pt[i] = row <= t * kTile + cf * 16 + i ? pt[i] : 0.0f;
            }
            uint32_t pc[3][8];
#pragma unroll
            for (int i = 0; i < 8; ++i) cut3(make_float2(pt[2 * i], pt[2 * i + 1]), pc[0][i], pc[1][i], pc[2][i]);
#pragma unroll
            for (int z = 0; z < 3; ++z) tmem_st8_u32(lane_base + t * C::kCols3 + 32 * z + 8 * cf, pc[z]);
            if (t + 1 < nq) fetch(t + 1);            // (while the pieces are on their way)
            tmem_wait_st();
            tc_fence_before();
            arrive(&sh.p3_ready[t]);
        }
        // (while the last products run: the other gradients are got ready.  Nothing is stored before it is known that no wait has run out)
        stage_rows(oq, c, kHalves ? kScoreLoss32 : kScoreLoss, q_s);
        if (NB > 1) {
            cluster_wait();
            if (!CAUSAL || blk == 0) receive(ok, 0);
        }
        stage_rows(ok, c, kScoreLoss, g_s);
        wait(&sh.v3_done, 0, 25);
        tc_fence_after();
#pragma unroll
        for (int t = 0; t < C::kTiles; ++t) {
            if (t < 2 * qb0 || t >= nq) continue;
            float a[OC];
            load_acc(lane_base + C::kCol3 + t * D + cf * OC, a);
            tmem_wait_ld();
#pragma unroll
            for (int i = 0; i < OC; ++i) ov[i] += a[i];
        }
        meet();                                      // (who has not seen a wait run out: the last word on it)
    }
    bool off = sh.abort_flag;
    if constexpr (STORED) {
        store_rows(q_s, dQ, off);
        store_rows(g_s, dK, off || sh.peer_gone);
        stage_rows(ov, 1.0f, 0.0f, p_s);
        store_rows(p_s, dV, off);
    } else {
        stage_rows(oq, c, kScoreLoss, q_s);
        store_rows(q_s, dQ, off);
        if (NB > 1) {
            cluster_wait();
            if (!CAUSAL || blk == 0) { receive(ov, 0); receive(ok, 1); }
            off = off || sh.peer_gone;
        }
        stage_rows(ov, 1.0f, kSumLoss, g_s);
        store_rows(g_s, dV, off);
        stage_rows(ok, c, kScoreLoss, k_s);
        store_rows(k_s, dK, off);
    }
    tc_fence_before();
    __syncthreads();
}

template <int D, bool CAUSAL, bool STORED, int NB>
int launch_head(const float *g, const float *q, const float *k, const float *v, const float *probs, float *dq, float *dk, float *dv,
                int B, int S, int E, int H, cudaStream_t st)
{
    auto kern = bwd_head_kernel<D, CAUSAL, STORED, NB>;
    constexpr size_t smem = HeadCfg<D, NB>::kSmem;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    CUtensorMap map = {};
    const int by_tma = STORED && (S & 3) == 0 && tma_encode_fn() != nullptr;
    if (by_tma) {
        const int rc = tma_plane_map(&map, probs, B * H, S, S, kLanes, CU_TENSOR_MAP_SWIZZLE_128B);
        if (rc != HIPGPT_OK) return rc;
    }
    int dev = 0, ahead = 0;                          // one block per SM: that many on is the one that follows
    e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&ahead, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_head_kernel: %s", cudaGetErrorString(e));
    const int expire = take_expiry(600);
    e = launch_overlapped_clusters(kern, NB, dim3((unsigned)(B * H * NB)), dim3(kThreads), smem, st, q, k, v, g, probs, dq, dk, dv, S, E, H, 1.0f / sqrtf((float)D), by_tma, ahead, map, expire);
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "bwd_head_kernel launch: %s", cudaGetErrorString(e));
    return HIPGPT_OK;
}

}  // namespace

// (what mha_backward_tc_supports takes, with a head that fits)
bool mha_backward_head_supports(int D, int S) { return D == 32 ? S <= 256 : S <= 128; }

int launch_mha_backward_head(const float *g, const float *q, const float *k, const float *v, const float *probs, float *dq, float *dk, float *dv,
                             int B, int S, int E, int H, int causal, cudaStream_t st)
{
    auto go = [&](auto launch) { return launch(g, q, k, v, probs, dq, dk, dv, B, S, E, H, st); };
#define HIPGPT_HEAD(D, NB) (causal ? probs ? go(launch_head<D, true, true, NB>) : go(launch_head<D, true, false, NB>) : probs ? go(launch_head<D, false, true, NB>) : go(launch_head<D, false, false, NB>))
    if (E / H == 64) return HIPGPT_HEAD(64, 1);
    return S <= kLanes ? HIPGPT_HEAD(32, 1) : HIPGPT_HEAD(32, 2);
#undef HIPGPT_HEAD
}

int mha_backward_head_status_fetch(int *status)
{
    int s = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&s, g_bwd_head_status, sizeof(int));
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaMemcpyFromSymbol: %s", cudaGetErrorString(e));
    if (s != 0) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_bwd_head_status, &zero, sizeof(int));
    }
    *status = s;
    return HIPGPT_OK;
}

}  // namespace hipgpt
