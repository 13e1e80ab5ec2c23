// Greedy generation with HipGPT's model shape, KV-cache form, by clusters of sixteen blocks (sm_100a).
//
// The same arithmetic as the launches of gpt_decode.cu, bit for bit: matmuls accumulate 16 segments of the inner dimension k
// ascending with fused multiply-add and add the partial sums in order, layer norms are 32 lane-strided sums joined by a butterfly,
// the attention is split over the context as attn_decode.cu splits it and merged in its order.
//
// What bounds a token step is a chain of small products: 4 per layer, each needing all of the one before it, with a few KB of
// activations between them and 30 MB of weights beside them.  As 52 launches a step of the default model took 320 us, nearly all
// of it launch gaps, L2 round trips and weights fetched only when a kernel had started.  Here one launch runs all steps, and
// sequences, which do not depend on one another, are dealt out to clusters:
//   * A cluster owns `rows` sequences and runs every layer for them.  A block owns a sixteenth of the columns of every matrix.
//     The activations are replicated: each block keeps whole rows in its shared memory, and the block that finishes four columns
//     stores them into all sixteen with st.async, which counts the bytes on the receiver's mbarrier.  A hop from product to product
//     is therefore one such store and one barrier inside the block: no barrier over the cluster, nothing through L2.
//   * A block's weights are laid out once in the order in which a step reads them and arrive through a ring in shared memory by
//     bulk copies that run up to a layer ahead of the arithmetic; they do not depend on activations, so nothing waits for them.
//   * The feed-forward's inner row does not leave its block: a block's columns of the first matrix are a segment of the second one's inner
//     dimension, so it multiplies them on and sends partial sums to the columns' owners.
//   * Elsewhere warp s owns segment s of the inner dimension (lanes: columns), so a layer norm needs no barrier either: every warp forms
//     the row's statistics and normalises the part that it multiplies.
//   * Keys and values of older positions are asked for while the projection of the new one is on its way between the blocks.
//   * The logits are formed where an id is picked from them: not at prompt positions before the last.
// Buffers are received into once per layer (or step); a sender can be at most one product ahead of the slowest receiver, because
// each product needs the columns of all blocks, so a buffer is never overwritten while it is read.
// Waits on mbarriers are bounded: on expiry the block raises a flag that cuts its later waits short and sets the error word, goes on
// without waiting to the end of the step (or of four layers) and sends nothing after it; the other blocks' waits then run
// out too, and all meet at the barriers of the remaining steps and leave.  (A barrier whose phase has not been seen complete is not
// opened again, and the bytes that nobody waits for stay within eight layers' worth, at most 90 KB each: an mbarrier counts 2^20.)
//
// Measured at the default model (E=256 L=8 H=8 V=5000), batch 8: 64 us per step (the replayed graph: 184), batch 3: 57.  A layer of
// 7.6 us: the hops (450 - 700 ns from the last store to the first read, five of them), attention 1.2, the two layer norms 0.35 each, a product's
// multiply-adds 0.15 - 0.5.  Besides, the shared memory's width is in the chain wherever all warps read at once (192 KB of weights are 1536 cycles of a
// layer): sums column by column, weights that no two lanes read twice and QKV's weights asked for before their activations took a step from 72 to 66 us
// (B=7 E=192 L=5, 67 positions and more: 5268 -> 4723 us a request).  Sizes are template parameters because the chain is
// bound by the instructions of single warps: with sizes read from the plan a step took 143 us.
#include "gpt_cluster.cuh"
#include "tc_primitives.cuh"

#include <math.h>

namespace hipgpt {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps = 16;
constexpr int kMostSlots = 24;
constexpr int kSmemMost = 232448 - 1024;
constexpr int kLayersChecked = 4;                // layers between two looks at whether a wait has run out
constexpr int kAhead = 4;                        // key / value rows per lane asked for ahead of the projection

// 16 or 8 bytes into a block of the cluster, counted on the mbarrier there
__device__ __forceinline__ void send4(uint32_t addr, uint32_t bar, float4 v)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(addr), "r"(__float_as_uint(v.x)), "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w)), "r"(bar) : "memory");
}
__device__ __forceinline__ void send2(uint32_t addr, uint32_t bar, uint32_t x, uint32_t y)
{
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];" ::"r"(addr), "r"(x), "r"(y), "r"(bar) : "memory");
}

// What the waits of a block share
struct Waits {
    volatile int gone;                               // a wait has run out: later ones are cut short
    int *err;
    long long limit;                                 // SM cycles
    const uint64_t *expire;                          // test hook: the barrier whose wait runs out at once
};
// The polling part of a wait, out of line: the kernel's code should stay in the instruction cache.  1: it, or one before it, has run out.
__device__ __noinline__ int cluster_wait_slow(uint64_t *bar, uint32_t parity, Waits *w)
{
    if (!w->gone && bar != w->expire && mbar_wait_for(bar, parity, w->limit, kSpinLimit)) return 0;
    if (!w->gone) atomicExch(w->err, 1);
    w->gone = 1;
    return 1;
}

template <int J>
struct Job { static constexpr int value = J; };
template <int E, int D, int R, int VW>
struct Width { static constexpr int kE = E, kD = D, kR = R, kVW = VW; };

// Shared memory of a block, in floats from the start: what has a size known to the compiler first.  Rows of activations are padded
// by four floats: the rows that a warp reads side by side then lie in different banks.
template <int E, int R>
struct Lay {
    static constexpr int es = E + 4, qs = 3 * E + 4;                     // row strides
    static constexpr int seg = cluster_job_of(kJobQkv, E, 16).klp + 4;   // of a warp's own segment
    static constexpr ClusterJob f2 = cluster_job_of(kJobF2, E, 16);
    static constexpr int fs = f2.klen + 4;                               // of the block's segment of the feed-forward's inner row
    static constexpr int xb = 0, xa = xb + R * es, qkv = xa + R * es, ff = qkv + R * qs, f2s = ff + R * fs, aw = f2s + 16 * R * f2.nc, part = aw + kWarps * R * seg;
    static constexpr int part_stride = R * 16 * 64;
    static constexpr int unit = part + 2 * part_stride, amax = unit + 8 * 4 * 16 * 8, fixed = (amax + 32 * R * 2 + 3) & ~3;
    static constexpr int slot_bytes()
    {
        int most = 0;
        for (int i = 0; i < kJobs; ++i) { const int b = cluster_job_of(i, E, 64 * 64).chunk_bytes(); most = b > most ? b : most; }
        return (most + 127) & ~127;
    }
    static constexpr int kSlot = slot_bytes();
};
// ... then the attention records and the chunk table, then the ring.
struct Rest { int table, ring, slots, total; };
template <int E, int R>
Rest rest_of(int H, int D, int ns, int all_chunks)
{
    using L = Lay<E, R>;
    Rest r;
    r.table = L::fixed + ((R * H * ns * (D + 4) + 3) & ~3);
    r.ring = (r.table + 2 * all_chunks + 31) & ~31;
    r.slots = (kSmemMost - 4 * r.ring) / L::kSlot;
    if (r.slots > kMostSlots) r.slots = kMostSlots;
    if (r.slots < 0) r.slots = 0;
    r.total = 4 * r.ring + r.slots * L::kSlot;
    return r;
}

template <int E, int D, int R, int VW>
__global__ void __launch_bounds__(kThreads, 1)
cluster_steps_kernel(const __grid_constant__ ClusterPlan plan, const __grid_constant__ ClusterArgs a, const __grid_constant__ Rest lay)
{
    using C = Lay<E, R>;
    extern __shared__ __align__(128) float sm[];
    __shared__ uint64_t full[kMostSlots];
    __shared__ uint64_t hop[6];                      // qkv, attention records, xa, partial sums of the second feed-forward product, xb, first maxima
    __shared__ float2 stats[R];                      // (R > 1) a row's mean and 1 / sqrt(variance + eps)
    __shared__ int next_id[R];
    __shared__ Waits waits;
    enum { kQkv, kRec, kXa, kF2, kXb, kAm };
    static_assert(kRec == kHopRecords, "");

    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    int rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    const int row0 = (int)(blockIdx.x / kClusterBlocks) * R;
    const int rows = min(R, a.B - row0);             // sequences of this cluster
    constexpr int H = E / D, rstride = D + 4;
    const int V = a.V, ns = a.ns;

    float *xb = sm + C::xb, *xa = sm + C::xa, *qkv = sm + C::qkv, *rec = sm + C::fixed, *part = sm + C::part;
    float *aw = sm + C::aw + warp * (R * C::seg);    // this warp's own segment of the activations
    uint32_t *amax = reinterpret_cast<uint32_t *>(sm + C::amax);
    uint2 *table = reinterpret_cast<uint2 *>(sm + lay.table);
    uint8_t *ring = reinterpret_cast<uint8_t *>(sm + lay.ring);
    const int f2_own = cluster_f2_columns(E, rank);
    const bool f2_here = cluster_f2_columns(E, kClusterBlocks - 1) > 0 || f2_own > 0;
    auto tx = [&](int i) {
        return (uint32_t)(rows * (i == kQkv ? 12 * E : i == kRec ? H * ns * (D + 2) * 4 : i == kF2 ? 16 * 4 * f2_own : i == kAm ? 32 * 8 : 4 * E));
    };

    for (int i = tid; i < lay.table; i += kThreads) sm[i] = 0.0f;         // rows that the cluster does not have stay zero
    for (int i = tid; i < plan.all_chunks; i += kThreads) table[i] = a.table[i];
    if (tid == 0) {
        waits.gone = 0;
        waits.err = a.err;
        waits.limit = a.wait_cycles;
        waits.expire = blockIdx.x == 0 && a.expire_hop >= 0 ? &hop[a.expire_hop] : nullptr;
        for (int i = 0; i < lay.slots; ++i) mbar_init(&full[i], 1);
        for (int i = 0; i < 6; ++i) {
            mbar_init(&hop[i], 1);
            if (i != kF2 || f2_here) mbar_arrive_expect_tx(&hop[i], tx(i));
        }
    }
    __syncthreads();
    cluster_sync();

    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (!mbar_test(bar, parity)) cluster_wait_slow(bar, parity, &waits);
    };
    // what a hop delivers is complete; one thread opens the barrier's next phase
    uint32_t hop_phase = 0;                          // a bit per hop
    auto receive = [&](int i) {
        int gone = waits.gone;
        if (!mbar_test(&hop[i], (hop_phase >> i) & 1u)) gone = cluster_wait_slow(&hop[i], (hop_phase >> i) & 1u, &waits);
        hop_phase ^= 1u << i;
        if (tid == kThreads - 1 && !gone) mbar_arrive_expect_tx(&hop[i], tx(i));
    };
    // after a wait that has run out: through the barriers of this step and those to come with the others
    auto leave = [&](int step) {
        for (; step < a.nsteps; ++step) cluster_sync();
    };
    // an address of this block -> the same place in four of the blocks (those this thread stores into)
    const int dq = tid & 3;
    uint32_t peer[4];
#pragma unroll
    for (int d = 0; d < 4; ++d) peer[d] = peer_addr(smem_u32(sm), 4 * dq + d) - smem_u32(sm);

    // ---- the weights: the lanes of the last warp keep the ring full, in the order in which the steps consume it ----
    const uint8_t *share = a.stream + (size_t)rank * plan.block_bytes;
    int f_step = 0, f_pos = 0, f_slot = 0;           // the next chunk: its step, its place in the step, its slot
    auto step_chunks = [&](int step) { return a.p0 + step >= a.n_prompt - 1 ? plan.all_chunks : plan.layer_chunks; };     // an id is picked there
    auto fetch = [&](int n) {                        // the next n <= 16 chunks (as long as there are any), a lane each
        const int len = step_chunks(f_step);
        int pos = f_pos + lane, slot = f_slot + lane;
        const bool wraps = pos >= len;
        if (wraps) pos -= len;
        if (slot >= lay.slots) slot -= lay.slots;
        if (lane < n && f_step + (wraps ? 1 : 0) < a.nsteps && !waits.gone) {           // (no copy onto one that nobody saw land)
            const uint2 t = table[pos];
            mbar_arrive_expect_tx(&full[slot], t.y);
            bulk_load(ring + slot * C::kSlot, share + t.x, t.y, &full[slot]);
        }
        f_pos += n;
        if (f_pos >= len) { f_pos -= len; ++f_step; }
        f_slot += n;
        if (f_slot >= lay.slots) f_slot -= lay.slots;
    };
    if (warp == kWarps - 1)
#pragma unroll 1
        for (int i = 0; i < lay.slots; ++i) fetch(1);
    int slot0 = 0;                                   // slot of the next product's first chunk
    uint32_t slot_par = 0;                           // parity of the ring's round there
    int flip = 0;                                    // buffer of partial sums

    // a row's mean and 1 / sqrt(variance + eps): 32 lane-strided sums joined by a butterfly, nothing contracted.  With one row every warp forms them
    // for itself, without a barrier (B=5 E=192 L=4, 67 positions: 1825 -> 1790 us); with two, a warp a row: both rows in every warp cost more (9720 -> 10570).
    auto row_stats = [&](const float *row) {
        float v[E / 32];
        float s = 0.0f, q = 0.0f;
#pragma unroll
        for (int i = 0; i < E / 32; ++i) v[i] = row[lane + 32 * i];
#pragma unroll
        for (int i = 0; i < E / 32; ++i) s = __fadd_rn(s, v[i]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
        // a division by a power of two is a multiplication
        const float mean = (E & (E - 1)) == 0 ? __fmul_rn(s, 1.0f / E) : __fdiv_rn(s, (float)E);
#pragma unroll
        for (int i = 0; i < E / 32; ++i) {
            const float d = __fsub_rn(v[i], mean);
            q = __fadd_rn(q, __fmul_rn(d, d));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, o));
        const float var = (E & (E - 1)) == 0 ? __fmul_rn(q, 1.0f / E) : __fdiv_rn(q, (float)E);
        return make_float2(mean, __frcp_rn(__fsqrt_rn(__fadd_rn(var, 1e-5f))));
    };

    // One product's multiply-adds: this warp's segment of the inner dimension, all columns of the part.  The activations: rows at
    // `src` in shared memory, normalised first where the job says so; kJobO takes this warp's own segment.  Leaves the partial sums
    // in part + flip * part_stride and ends with a barrier of the block.  Lanes: up to 16 columns: (column, row of a pair); more:
    // columns lane, lane + 32, all rows.  Returns the part's bias for the column that this thread finishes.
    // `arrival` waits for the activations.  Before it the weights of this lane go to registers (where there are at most 64): they
    // have been in the ring for long, and reading them takes the shared memory's return path about as long as a hop takes.  (With two rows the
    // other warps wait with that until the sums before have been read: bar 9 in `finish`, 8874 -> 8779 us a request; with one row it costs as much.)
    auto product = [&](auto jn, const float *src, auto arrival) {
        constexpr int J = decltype(jn)::value;
        constexpr ClusterJob jb = cluster_job_of(J, E, 64 * 64);          // (the output projection's cut depends on V in its parts only)
        constexpr int pw = jb.width, klen = jb.klen, klp = jb.klp, sh = jb.seg_shift, nch = jb.chunks();
        constexpr int stride = C::es;
        int slot = slot0 + (warp >> sh);
        uint32_t par = slot_par;
        if (slot >= lay.slots) { slot -= lay.slots; par ^= 1u; }
        const float *chunk = reinterpret_cast<const float *>(ring + slot * C::kSlot);
        const int in_chunk = warp & ((1 << sh) - 1);
        const float4 *w4 = reinterpret_cast<const float4 *>(chunk + in_chunk * (klp * pw));
        const float *as = aw;
        constexpr bool kOwn = jb.ln || J == kJobO || (klen & 3) != 0;     // the activations are (copied) in this warp's own segment
        constexpr int astride = kOwn ? C::seg : stride;
        constexpr int NC = pw <= 16 ? 1 : (pw + 31) / 32;                // columns per lane
        constexpr bool kEarly = J != kJobVoc && NC * klp <= 64;
        const int wc0 = pw <= 16 ? (pw < 16 ? min(lane & 15, pw - 1) : lane & 15) : (pw < 32 ? min(lane, pw - 1) : lane);
        const float4 *wp = w4 + wc0, *wq = w4 + (pw < 64 ? min(lane + 32, pw - 1) : lane + 32);
        float4 held[kEarly ? NC * klp / 4 : 1];
        if constexpr (kEarly) {
            wait(&full[slot], par);
#pragma unroll
            for (int k = 0; k < klp / 4; ++k) {
                held[NC * k] = wp[k * pw];
                if constexpr (NC > 1) held[NC * k + 1] = wq[k * pw];
            }
        }
        arrival();
        float2 own = make_float2(0.f, 0.f);
        if constexpr (jb.ln != 0 && R == 1) own = row_stats(src);
        if constexpr (jb.ln != 0 && R > 1) {
            if (warp < rows) {
                const float2 st = row_stats(src + warp * stride);
                if (lane == 0) stats[warp] = st;
            }
            __syncthreads();
        }
        if constexpr (!kEarly) wait(&full[slot], par);
        if constexpr (jb.ln != 0) {
            const float *gm = chunk + jb.weight_floats() + in_chunk * klp, *bt = gm + (klp << sh);
#pragma unroll
            for (int t = 0; t < (R * klp + 31) / 32; ++t) {
                const int i = lane + 32 * t, r = i / klp, k = i % klp;
                if (i < R * klp) {
                    const float2 st = R == 1 ? own : stats[r];
                    aw[r * C::seg + k] = k < klen ? __fadd_rn(__fmul_rn(__fmul_rn(gm[k], __fsub_rn(src[r * stride + warp * klen + k], st.x)), st.y), bt[k]) : 0.0f;
                }
            }
            __syncwarp();
        } else if constexpr (kOwn && J != kJobO) {
#pragma unroll
            for (int t = 0; t < (R * klp + 31) / 32; ++t) {
                const int i = lane + 32 * t, r = i / klp, k = i % klp;
                if (i < R * klp) aw[r * C::seg + k] = k < klen ? src[r * stride + warp * klen + k] : 0.0f;
            }
            __syncwarp();
        } else if constexpr (!kOwn) {
            as = src + warp * klen;
        }
        float *dst = part + flip * C::part_stride + warp * pw;
        if constexpr (pw <= 16) {
            constexpr int RH = (R + 1) / 2;          // rows of a lane: r0, r0 + 2
            const int c = lane & 15, r0 = R > 1 ? lane >> 4 : 0;
            float acc[RH];
#pragma unroll
            for (int r = 0; r < RH; ++r) acc[r] = 0.0f;
#pragma unroll (kEarly ? klp / 4 : 8)
            for (int k = 0; k < klp / 4; ++k) {
                const float4 w = kEarly ? held[k] : wp[k * pw];
#pragma unroll
                for (int r = 0; r < RH; ++r) {
                    const float4 x = *reinterpret_cast<const float4 *>(as + (r0 + 2 * r) * astride + 4 * k);
                    acc[r] = fmaf(x.x, w.x, acc[r]);
                    acc[r] = fmaf(x.y, w.y, acc[r]);
                    acc[r] = fmaf(x.z, w.z, acc[r]);
                    acc[r] = fmaf(x.w, w.w, acc[r]);
                }
            }
            if (c < pw && (R > 1 || lane < 16))
#pragma unroll
                for (int r = 0; r < RH; ++r) dst[(r0 + 2 * r) * 16 * pw + c] = acc[r];
        } else {
            float acc[NC][R];
#pragma unroll
            for (int n = 0; n < NC; ++n)
#pragma unroll
                for (int r = 0; r < R; ++r) acc[n][r] = 0.0f;
#pragma unroll (kEarly ? klp / 4 : 4)
            for (int k = 0; k < klp / 4; ++k) {
                float4 w[NC];
                w[0] = kEarly ? held[NC * k] : wp[k * pw];
                if constexpr (NC > 1) w[1] = kEarly ? held[NC * k + 1] : wq[k * pw];
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 x = *reinterpret_cast<const float4 *>(as + r * astride + 4 * k);
#pragma unroll
                    for (int n = 0; n < NC; ++n) acc[n][r] = fmaf(x.x, w[n].x, acc[n][r]);
#pragma unroll
                    for (int n = 0; n < NC; ++n) acc[n][r] = fmaf(x.y, w[n].y, acc[n][r]);
#pragma unroll
                    for (int n = 0; n < NC; ++n) acc[n][r] = fmaf(x.z, w[n].z, acc[n][r]);
#pragma unroll
                    for (int n = 0; n < NC; ++n) acc[n][r] = fmaf(x.w, w[n].w, acc[n][r]);
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int n = 0; n < NC; ++n)
                    if (32 * (n + 1) <= pw || lane + 32 * n < pw) dst[r * 16 * pw + lane + 32 * n] = acc[n][r];
        }
        float bias = 0.0f;
        if constexpr (J != kJobVoc) {
            // the first chunk has landed: warp 0 waited for it; another warp may not have, and asks again
            if (tid < pw * R) {
                wait(&full[slot0], slot_par);
                bias = (reinterpret_cast<const float *>(ring + slot0 * C::kSlot) + jb.weight_floats() + jb.ln_floats())[R == 1 ? tid : tid % pw];
            }
        }
        __syncthreads();                             // the partial sums are there; the chunks may be overwritten
        if (warp == kWarps - 1) fetch(nch);
        slot0 += nch;
        if (slot0 >= lay.slots) { slot0 -= lay.slots; slot_par ^= 1u; }
        return bias;
    };
    // Four neighbouring threads' columns (where `mine`: of an existing row, within the block's share), stored by each into four of the sixteen blocks
    auto send_four = [&](float v, bool mine, int to_floats, int h) {
        const float4 four = make_float4(__shfl_sync(0xffffffffu, v, 0, 4), __shfl_sync(0xffffffffu, v, 1, 4), __shfl_sync(0xffffffffu, v, 2, 4), __shfl_sync(0xffffffffu, v, 3, 4));
        if (mine) {
            const uint32_t to = smem_u32(sm + (to_floats & ~3)), bar = smem_u32(&hop[h]);
#pragma unroll
            for (int d = 0; d < 4; ++d) send4(to + peer[d], bar + peer[d], four);
        }
        return four;
    };
    // Finishes part `pt` of a product: a thread adds up a column of a row (partial sums in ascending order; a warp reads whole lines: as four
    // columns per thread, with a thread per four receivers, each line was read four times, and that traffic stood in the chain) and hands it over with
    // its neighbours'.  The feed-forward's inner row stays in the block, which goes on with its segment of it.
    auto finish = [&](auto jn, int pt, float bias, int layer, int p) {
        constexpr int J = decltype(jn)::value;
        constexpr ClusterJob jb = cluster_job_of(J, E, 64 * 64);
        constexpr int pw = jb.width, stride = J == kJobQkv ? C::qs : C::es;
        constexpr int buf = J == kJobQkv ? C::qkv : C::xa;
        if (warp * 32 < pw * R) {                    // (whole warps)
            const int r = R == 1 ? 0 : tid / pw, c = tid - r * pw, n = rank * jb.nc + pt * pw + c;
            // the block's last columns may lie past its share (the last part) or past the matrix: four at a time
            const bool mine = tid < pw * R && r < rows && pt * pw + c < jb.nc && n < jb.n;
            float v = 0.0f;
            if (mine) {
                const float *ps = part + flip * C::part_stride + r * 16 * pw + c;
                v = ps[0];
#pragma unroll
                for (int s = 1; s < 16; ++s) v = __fadd_rn(v, ps[s * pw]);
                v = __fadd_rn(v, bias);
                if constexpr (J == kJobF1) sm[C::ff + r * C::fs + pt * pw + c] = fmaxf(0.0f, v);
                if constexpr (J == kJobO) v = __fadd_rn(sm[C::xb + r * stride + n], v);
            }
            if constexpr (J != kJobF1) {
                if constexpr (R > 1) asm volatile("bar.arrive 9, 512;" ::: "memory");
                const float4 four = send_four(v, mine, buf + r * stride + n, J == kJobQkv ? kQkv : kXa);
                if constexpr (J == kJobQkv) {
                    const int n0 = n & ~3;           // (shares and parts are whole fours)
                    if (mine && dq == (rank >> 2) && n0 >= E) {  // keys and values, for the later positions
                        float *cache = (n0 < 2 * E ? a.kc : a.vc) + (size_t)layer * a.layer_stride + ((size_t)(row0 + r) * a.S + p) * E;
                        *reinterpret_cast<float4 *>(cache + (n0 < 2 * E ? n0 - E : n0 - 2 * E)) = four;
                    }
                }
            }
        } else if constexpr (J != kJobF1 && R > 1) {
            asm volatile("bar.sync 9, 512;" ::: "memory");
        }
        flip ^= 1;
    };
    // The second product of the feed-forward: this block's columns of the first are a segment of its inner dimension, so they need no hop.  The last
    // warps take 32 columns each, all rows, and send the partial sums to the blocks that own the columns; these add them up in order (the same
    // order as everywhere) and hand the row out.  As a product like the others, the inner row by a hop (512 stores a block, 0.3 us to issue) and partial sums
    // through the block: 66 us a step instead of 64 at the default model, E=320 D=64 batch 4 10956 us a request instead of 8964, E=384 batch 8 10309 instead of 9027.
    auto second = [&]() {
        constexpr ClusterJob jb = C::f2;
        constexpr int G = jb.per * jb.width / 32, K4 = jb.klen / 4;      // warps at work
        constexpr int kHeld = K4 < 8 ? K4 : 8;                           // a column's first weights are in registers before the row is there (all: spills)
        float bias = 0.0f;
        const int own_r = R == 1 ? 0 : tid / jb.nc, own_c = tid - own_r * jb.nc, own_n = rank * jb.nc + own_c;
        const bool sums = f2_here && warp * 32 < jb.nc * R, mine = sums && tid < jb.nc * R && own_r < rows && own_n < E;
        if (sums) {
            wait(&full[slot0], slot_par);
            if (tid < jb.nc * R) bias = (reinterpret_cast<const float *>(ring + slot0 * C::kSlot) + jb.weight_floats())[own_c];
        }
#pragma unroll 1
        for (int pt = 0; pt < jb.parts; ++pt) {
            const int g = warp - (kWarps - G);
            if (g >= 0) {
                int slot = slot0 + g / (jb.width / 32);
                uint32_t par = slot_par;
                if (slot >= lay.slots) { slot -= lay.slots; par ^= 1u; }
                const float4 *wp = reinterpret_cast<const float4 *>(ring + slot * C::kSlot) + g % (jb.width / 32) * 32 + lane;
                wait(&full[slot], par);
                float4 w[kHeld];
#pragma unroll
                for (int k = 0; k < kHeld; ++k) w[k] = wp[k * jb.width];
                if (pt == 0) __syncthreads();        // the segment of the inner row is there
                float acc[R];
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = 0.0f;
                auto take = [&](int k, const float4 &wk) {
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 x = *reinterpret_cast<const float4 *>(sm + C::ff + r * C::fs + 4 * k);
                        acc[r] = fmaf(x.x, wk.x, acc[r]);
                        acc[r] = fmaf(x.y, wk.y, acc[r]);
                        acc[r] = fmaf(x.z, wk.z, acc[r]);
                        acc[r] = fmaf(x.w, wk.w, acc[r]);
                    }
                };
#pragma unroll
                for (int k = 0; k < kHeld; ++k) take(k, w[k]);
#pragma unroll 8
                for (int k = kHeld; k < K4; ++k) take(k, wp[k * jb.width]);
                // four columns of a row in one store, a lane of four per row
                const int n = (pt * G + g) * 32 + (lane & ~3), owner = n / jb.nc;
                const uint32_t to = smem_u32(sm + C::f2s + (rank * R + dq) * jb.nc + n - owner * jb.nc);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 four = make_float4(__shfl_sync(0xffffffffu, acc[r], 0, 4), __shfl_sync(0xffffffffu, acc[r], 1, 4), __shfl_sync(0xffffffffu, acc[r], 2, 4), __shfl_sync(0xffffffffu, acc[r], 3, 4));
                    if (dq == r && r < rows && n < E) send4(peer_addr(to, owner), peer_addr(smem_u32(&hop[kF2]), owner), four);
                }
                asm volatile("bar.sync 10, %0;" ::"n"(32 * G) : "memory");       // the chunks may be overwritten
                if (warp == kWarps - 1) fetch(jb.per);
            } else if (pt == 0) {
                __syncthreads();
            }
            slot0 += jb.per;
            if (slot0 >= lay.slots) { slot0 -= lay.slots; slot_par ^= 1u; }
        }
        // (the last warp opens the barrier's next phase, where there is one; the others have nothing to wait for)
        if (sums || (f2_here && warp == kWarps - 1)) receive(kF2);
        else hop_phase ^= 1u << kF2;
        if (sums) {
            float v = 0.0f;
            if (mine) {
                const float *ps = sm + C::f2s + own_r * jb.nc + own_c;
                v = ps[0];
#pragma unroll
                for (int s = 1; s < 16; ++s) v = __fadd_rn(v, ps[s * R * jb.nc]);
                v = __fadd_rn(sm[C::xa + own_r * C::es + own_n], __fadd_rn(v, bias));
            }
            send_four(v, mine, C::xb + own_r * C::es + own_n, kXb);
        }
    };

    // ---- the attention of one position: units of (row, head, split), dealt out over the blocks' warp groups.  attn_decode.cu gives a
    //      unit four warps; here a warp stands for VW of them, whose arithmetic it interleaves: two where the units of the cluster
    //      outnumber its groups of four warps (a second round costs more than the doubled work of a warp that is bound by latency).
    //      A key's head is read by LPK lanes (4 numbers each) ----
    constexpr int W4 = 4, GW = W4 / VW, GROUPS = kWarps / GW, AHEAD = kAhead / VW;
    constexpr int LPK = D / 4, KPW = 32 / LPK;
    const int group = warp / GW, wg = warp % GW, lik = lane % LPK, kg = lane / LPK;
    const float qscale = (1.0f / sqrtf((float)D)) * kLog2e;
    const int units = rows * H * ns;
    float *merge_s = sm + C::unit + group * (W4 * 16 * 8);
    struct Unit { int split, now, rec, mem; };       // its split; offsets of its head in qkv, of its record, of its row and head in a layer's cache
    auto make_unit = [&](int u) {
        const int split = u % ns, bh = u / ns, h = bh % H, r = bh / H;
        return Unit{split, r * C::qs + h * D, u * rstride, (row0 + r) * a.S * E + h * D};
    };
    const int u0 = rank + kClusterBlocks * group;
    const Unit first_unit = make_unit(min(u0, units - 1));
    int per = 0;                                     // positions of a split at this step
    float4 k4[VW][AHEAD], v4[VW][AHEAD];             // rows of a unit that earlier steps wrote
    auto ask = [&](const Unit &un, int layer, int p, int it0) {
        const int j0 = un.split * per + (it0 * W4 + wg * VW) * KPW + kg, k1 = min(p, un.split * per + per);
        const size_t at = (size_t)layer * a.layer_stride + (size_t)(un.mem + lik * 4) + (size_t)j0 * E;
        const float *kp = a.kc + at, *vp = a.vc + at;
#pragma unroll
        for (int w = 0; w < VW; ++w)
#pragma unroll
            for (int it = 0; it < AHEAD; ++it) {
                const int j = (it * W4 + w) * KPW;
                k4[w][it] = v4[w][it] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (j0 + j < k1) {
                    k4[w][it] = __ldcg(reinterpret_cast<const float4 *>(kp + j * E));
                    v4[w][it] = __ldcg(reinterpret_cast<const float4 *>(vp + j * E));
                }
            }
    };
    auto attend = [&](int layer, int p) {
#pragma unroll 1
        for (int u = u0; u < units; u += GROUPS * kClusterBlocks) {
            const Unit un = u == u0 ? first_unit : make_unit(u);
            const int k0 = un.split * per, k1 = min(p + 1, k0 + per);
            if (u != u0) ask(un, layer, p, 0);       // the first unit's rows were asked for ahead (the next one's too: spills, 105 us per step)
            const float *now = qkv + un.now + lik * 4;         // this position's query, key and value
            float4 q4 = *reinterpret_cast<const float4 *>(now);
            q4.x *= qscale; q4.y *= qscale; q4.z *= qscale; q4.w *= qscale;
            AttnPart acc[VW];
#pragma unroll
            for (int w = 0; w < VW; ++w) acc[w] = AttnPart{-1e30f, 0.0f, make_float4(0.f, 0.f, 0.f, 0.f)};
            constexpr int step = W4 * KPW;
#pragma unroll 1
            for (int it0 = 0; k0 + it0 * step < k1; it0 += AHEAD) {
                if (it0 > 0) ask(un, layer, p, it0);
                const int j0 = k0 + (it0 * W4 + wg * VW) * KPW + kg;
                const int own = p < k1 ? p - j0 : -1;               // where this position's own row is among them
                float s[VW][AHEAD];
#pragma unroll
                for (int w = 0; w < VW; ++w) {
#pragma unroll
                    for (int it = 0; it < AHEAD; ++it) {
                        if (own == it * step + w * KPW) {
                            k4[w][it] = *reinterpret_cast<const float4 *>(now + E);
                            v4[w][it] = *reinterpret_cast<const float4 *>(now + 2 * E);
                        }
                        float x = q4.x * k4[w][it].x;
                        x = fmaf(q4.y, k4[w][it].y, x);
                        x = fmaf(q4.z, k4[w][it].z, x);
                        s[w][it] = fmaf(q4.w, k4[w][it].w, x);
                    }
                }
#pragma unroll
                for (int o = 1; o < LPK; o <<= 1)
#pragma unroll
                    for (int i = 0; i < VW * AHEAD; ++i) s[i / AHEAD][i % AHEAD] += __shfl_xor_sync(0xffffffffu, s[i / AHEAD][i % AHEAD], o);
#pragma unroll
                for (int it = 0; it < AHEAD; ++it) {
                    if (k0 + (it0 + it) * step >= k1) break;               // no lane of the four warps has a row there
#pragma unroll
                    for (int w = 0; w < VW; ++w) {
                        AttnPart &t = acc[w];
                        const float x = j0 + it * step + w * KPW < k1 ? s[w][it] : -INFINITY;
                        const float mn = fmaxf(t.m, x);
                        const float alpha = ex2_approx(t.m - mn), pr = ex2_approx(x - mn);
                        t.l = fmaf(t.l, alpha, pr);
                        t.o.x = fmaf(pr, v4[w][it].x, t.o.x * alpha);
                        t.o.y = fmaf(pr, v4[w][it].y, t.o.y * alpha);
                        t.o.z = fmaf(pr, v4[w][it].z, t.o.z * alpha);
                        t.o.w = fmaf(pr, v4[w][it].w, t.o.w * alpha);
                        t.m = mn;
                    }
                }
            }
#pragma unroll
            for (int o = LPK; o < 32; o <<= 1) {
#pragma unroll
                for (int w = 0; w < VW; ++w) {
                    const float m2 = __shfl_xor_sync(0xffffffffu, acc[w].m, o);
                    const float l2 = __shfl_xor_sync(0xffffffffu, acc[w].l, o);
                    float4 o2;
                    o2.x = __shfl_xor_sync(0xffffffffu, acc[w].o.x, o);
                    o2.y = __shfl_xor_sync(0xffffffffu, acc[w].o.y, o);
                    o2.z = __shfl_xor_sync(0xffffffffu, acc[w].o.z, o);
                    o2.w = __shfl_xor_sync(0xffffffffu, acc[w].o.w, o);
                    merge_part(acc[w], m2, l2, o2);
                }
            }
            if (kg == 0) {
#pragma unroll
                for (int w = 0; w < VW; ++w) {
                    float *d = merge_s + ((wg * VW + w) * 16 + lik) * 8;
                    *reinterpret_cast<float4 *>(d) = acc[w].o;
                    *reinterpret_cast<float2 *>(d + 4) = make_float2(acc[w].m, acc[w].l);
                }
            }
            asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(32 * GW) : "memory");
            // each of the group's warps merges the columns of its lanes' `lik`; its key groups serve different receivers
            const float *m0 = merge_s + lik * 8;
            AttnPart t;
            t.o = *reinterpret_cast<const float4 *>(m0);
            t.m = m0[4]; t.l = m0[5];
#pragma unroll
            for (int w = 1; w < W4; ++w) {
                const float4 o2 = *reinterpret_cast<const float4 *>(m0 + w * 128);
                const float2 ml = *reinterpret_cast<const float2 *>(m0 + w * 128 + 4);
                merge_part(t, ml.x, ml.y, o2);
            }
            const uint32_t dst = smem_u32(rec + un.rec), bar = smem_u32(&hop[kRec]);
#pragma unroll 1
            for (int d = kg; d < 4 * VW; d += KPW) {
                const uint32_t pb = peer_addr(bar, 4 * VW * wg + d), pd = peer_addr(dst, 4 * VW * wg + d);
                send4(pd + lik * 16, pb, t.o);
                if (lik == 0) send2(pd + D * 4, pb, __float_as_uint(t.m), __float_as_uint(t.l));
            }
            if (u + GROUPS * kClusterBlocks < units) asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "n"(32 * GW) : "memory");
        }
    };
    // this warp's segment of the attention output from the records of all splits (attn_decode.cu's decode_combine_kernel)
    constexpr int o_klen = E / 16;
    auto combine = [&]() {
#pragma unroll
        for (int t = 0; t < (R * o_klen + 31) / 32; ++t) {
            const int i = lane + 32 * t, r = i / o_klen, e = warp * o_klen + i % o_klen;
            if (i < R * o_klen && r < rows) {
                const int h = e / D, d = e % D;
                const float *rc = rec + (r * H + h) * ns * rstride;
                float M = -1e30f, Lsum = 0.0f, acc = 0.0f;
                if (ns <= 8) {
                    // all loads in flight at once; a split that is not there counts as one without keys (which adds zeros), so nothing branches
                    float2 ml[8];
                    float os[8];
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        const float *at = rc + (s < ns ? s : 0) * rstride;
                        ml[s] = *reinterpret_cast<const float2 *>(at + D);
                        os[s] = at[d];
                        if (s >= ns) { ml[s] = make_float2(-INFINITY, 0.0f); os[s] = 0.0f; }
                    }
#pragma unroll
                    for (int s = 0; s < 8; ++s) M = fmaxf(M, ml[s].x);
#pragma unroll
                    for (int s = 0; s < 8; ++s) {
                        const float x = ex2_approx(ml[s].x - M);
                        Lsum += ml[s].y * x;
                        acc += os[s] * x;
                    }
                } else {
#pragma unroll 1
                    for (int s = 0; s < ns; ++s) M = fmaxf(M, rc[s * rstride + D]);
#pragma unroll 1
                    for (int s = 0; s < ns; ++s) {
                        const float x = ex2_approx(rc[s * rstride + D] - M);
                        Lsum += rc[s * rstride + D + 1] * x;
                        acc += rc[s * rstride + d] * x;
                    }
                }
                aw[r * C::seg + i % o_klen] = acc * (1.0f / fmaxf(Lsum, 1e-20f));
            }
        }
        if constexpr ((o_klen & 3) != 0) {           // the padding of the segment
            if (lane < R * 4 && (o_klen & ~3) + (lane & 3) >= o_klen) aw[(lane >> 2) * C::seg + (o_klen & ~3) + (lane & 3)] = 0.0f;
        }
        __syncwarp();
    };
    auto embed = [&](int p, int r, int id) {
        const bool ok = id >= 0 && id < V;
        if (tid < E) xb[r * C::es + tid] = ok ? __fadd_rn(a.tok[(size_t)id * E + tid], a.pos[(size_t)p * E + tid]) : 0.0f;
    };
    static_assert(E <= kThreads && E % 32 == 0, "");

#pragma unroll
    for (int r = 0; r < R; ++r)
        if (r < rows) embed(a.p0, r, a.p0 < a.n_prompt ? a.prompts[(size_t)(row0 + r) * a.n_prompt + a.p0] : a.ids[row0 + r]);
    __syncthreads();
#pragma unroll 1
    for (int step = 0; step < a.nsteps; ++step) {
        const int p = a.p0 + step;
        per = (p + ns) / ns;
#pragma unroll 1
        for (int l = 0; l < a.L; ++l) {
            if (l > 0 && l % kLayersChecked == 0 && __syncthreads_or(waits.gone)) {
                leave(step);
                step = a.nsteps;
                break;
            }
#pragma unroll 1
            for (int pt = 0; pt < cluster_job_of(kJobQkv, E, 0).parts; ++pt)
                finish(Job<kJobQkv>(), pt, product(Job<kJobQkv>(), xb, [&] { if (pt == 0 && l > 0) receive(kXb); }), l, p);
            ask(first_unit, l, p, 0);
            receive(kQkv);
            attend(l, p);
#pragma unroll 1
            for (int pt = 0; pt < cluster_job_of(kJobO, E, 0).parts; ++pt)
                finish(Job<kJobO>(), pt, product(Job<kJobO>(), nullptr, [&] { if (pt == 0) { receive(kRec); combine(); } }), 0, 0);
#pragma unroll 1
            for (int pt = 0; pt < cluster_job_of(kJobF1, E, 0).parts; ++pt)
                finish(Job<kJobF1>(), pt, product(Job<kJobF1>(), xa, [&] { if (pt == 0) receive(kXa); }), 0, 0);
            second();
        }
        if (step >= a.nsteps) break;
        receive(kXb);
        const bool head = p >= a.n_prompt - 1, last = step + 1 == a.nsteps;
        if (head) {
            // thread = (row, column of the part); columns ascend from part to part, so a thread keeps its first maximum
            float best = -INFINITY;
            int bi = 0x7fffffff;
            const int hr = tid >> 6, hc = tid & 63;
            constexpr int pw = cluster_job_of(kJobVoc, E, 64 * 64).width;
#pragma unroll 1
            for (int pt = 0; pt < plan.voc.parts; ++pt) {
                product(Job<kJobVoc>(), xb, [] {});
                const int n = rank * plan.voc.nc + pt * pw + hc;
                if (hr < rows && hc < pw && pt * pw + hc < plan.voc.nc && n < V) {
                    const float *pp = part + flip * C::part_stride + hr * 16 * pw + hc;
                    float v = pp[0];
#pragma unroll
                    for (int s = 1; s < 16; ++s) v = __fadd_rn(v, pp[s * pw]);
                    if (last) a.logits[(size_t)(row0 + hr) * V + n] = v;
                    if (v > best || bi == 0x7fffffff) { best = v; bi = n; }
                }
                flip ^= 1;
            }
            auto better = [&](float ov, int oi) {
                if (oi != 0x7fffffff && (bi == 0x7fffffff || ov > best || (ov == best && oi < bi))) { best = ov; bi = oi; }
            };
            auto butterfly = [&]() {
#pragma unroll 1
                for (int o = 16; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    better(ov, oi);
                }
            };
            if (hr < rows) {
                butterfly();
                if (lane < kClusterBlocks) {
                    const uint32_t dst = smem_u32(amax + (hr * 32 + rank * 2 + (warp & 1)) * 2);
                    send2(peer_addr(dst, lane), peer_addr(smem_u32(&hop[kAm]), lane), __float_as_uint(best), (uint32_t)bi);
                }
            }
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            receive(kAm);
            if (warp < rows) {
                best = __uint_as_float(amax[(warp * 32 + lane) * 2]);
                bi = (int)amax[(warp * 32 + lane) * 2 + 1];
                butterfly();
                if (lane == 0) {
                    next_id[warp] = bi;
                    if (rank == 0) {
                        a.ids[row0 + warp] = bi;
                        const int col = p - (a.n_prompt - 1);
                        if (col < a.n_new) a.out_ids[(size_t)(row0 + warp) * a.n_new + col] = bi;
                    }
                }
            }
            __syncthreads();
        } else {
            __syncthreads();                         // every warp is done with xb
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        }
        if (!last)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (r < rows) embed(p + 1, r, p + 1 < a.n_prompt ? a.prompts[(size_t)(row0 + r) * a.n_prompt + p + 1] : next_id[r]);
        // the keys and values of this position reach the other blocks before the next one is attended to; the barrier also keeps a
        // block from leaving while others still store into it
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        if (__syncthreads_or(waits.gone)) {
            leave(step + 1);
            break;
        }
    }
    if (waits.gone) linger();
}

// One chunk per block of this grid: (chunk, owner).  Columns and inner indices past the matrix (or the owner's share) are zeros.
__global__ void __launch_bounds__(256)
cluster_pack_kernel(const ClusterJob j, int pt, const float *__restrict__ w, const float *__restrict__ bias, const float *__restrict__ gamma,
                    const float *__restrict__ beta, uint8_t *dst, size_t block_bytes)
{
    const int pw = j.width, ch = blockIdx.x, owner = blockIdx.y;
    const int first = owner * j.nc + pt * pw, end = min(j.n, (owner + 1) * j.nc), segs = 1 << j.seg_shift;
    float *d = reinterpret_cast<float *>(dst + (size_t)owner * block_bytes + (size_t)ch * j.chunk_bytes());
    if (j.per) {
        for (int i = threadIdx.x; i < j.weight_floats(); i += blockDim.x) {
            const int u = i & 3, c = ((pt * j.per + ch) * pw) + (i >> 2) % pw, k = 4 * ((i >> 2) / pw) + u;
            d[i] = c < j.n ? w[(size_t)(owner * j.klen + k) * j.n + c] : 0.0f;
        }
        d += j.weight_floats();
        for (int i = threadIdx.x; i < j.nc; i += blockDim.x) d[i] = owner * j.nc + i < j.n ? bias[owner * j.nc + i] : 0.0f;
        return;
    }
    for (int i = threadIdx.x; i < j.weight_floats(); i += blockDim.x) {
        const int u = i & 3, c = (i >> 2) % pw, k4 = (i >> 2) / pw % (j.klp >> 2), s = (i >> 2) / pw / (j.klp >> 2);
        const int k = 4 * k4 + u;
        d[i] = (first + c < end && k < j.klen) ? w[(size_t)((ch * segs + s) * j.klen + k) * j.n + first + c] : 0.0f;
    }
    d += j.weight_floats();
    if (j.ln)
        for (int i = threadIdx.x; i < segs * j.klp; i += blockDim.x) {
            const int s = i / j.klp, k = i % j.klp, at = (ch * segs + s) * j.klen + k;
            d[i] = k < j.klen ? gamma[at] : 0.0f;
            d[segs * j.klp + i] = k < j.klen ? beta[at] : 0.0f;
        }
    d += j.ln_floats();
    for (int i = threadIdx.x; i < pw; i += blockDim.x) d[i] = (bias && first + i < end) ? bias[first + i] : 0.0f;
}

// A launch of `clusters` clusters of sixteen blocks
struct ClusterLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    ClusterLaunch(int clusters, size_t smem, cudaStream_t st)
    {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClusterBlocks;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.gridDim = dim3((unsigned)(clusters * kClusterBlocks));
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
};

template <int E, int D, int R, int VW>
cudaError_t prepare_kernel()
{
    auto kern = cluster_steps_kernel<E, D, R, VW>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMost);
}

// f(Width<E, D, R, VW>()) for the shape; -1 where there is no kernel for it
template <int R, int VW, typename F>
int with_width(int E, int D, F f)
{
    switch (E * 1000 + D) {
#define HIPGPT_CLUSTER(W, HD) case W * 1000 + HD: return f(Width<W, HD, R, VW>());
    HIPGPT_CLUSTER(128, 32) HIPGPT_CLUSTER(160, 32) HIPGPT_CLUSTER(192, 32) HIPGPT_CLUSTER(224, 32) HIPGPT_CLUSTER(256, 32) HIPGPT_CLUSTER(288, 32)
    HIPGPT_CLUSTER(320, 32) HIPGPT_CLUSTER(352, 32) HIPGPT_CLUSTER(384, 32)
    HIPGPT_CLUSTER(128, 64) HIPGPT_CLUSTER(192, 64) HIPGPT_CLUSTER(256, 64) HIPGPT_CLUSTER(320, 64) HIPGPT_CLUSTER(384, 64)
#undef HIPGPT_CLUSTER
    default: return -1;
    }
}
// `units`: (row, head, split) of a cluster.  Sixteen blocks have 64 groups of four warps.
template <typename F>
int with_kernel(int E, int D, int rows, int units, F f)
{
    if (rows == 1) return units <= 64 ? with_width<1, 1>(E, D, f) : with_width<1, 2>(E, D, f);
    return units <= 64 ? with_width<2, 1>(E, D, f) : with_width<2, 2>(E, D, f);
}

}  // namespace

ClusterPlan cluster_plan(int V, int S, int E, int L, int H, int F)
{
    ClusterPlan p = {};
    const int D = E / H;
    if ((D != 32 && D != 64) || F != 4 * E) return p;
    // the output projection's parts have the width the kernel is compiled for; the vocabulary decides how many there are
    p.voc = cluster_job_of(kJobVoc, E, 64 * 64);
    p.voc.n = V;
    p.voc.nc = 4 * ((V + 63) / 64);
    p.voc.parts = (p.voc.nc + p.voc.width - 1) / p.voc.width;
    for (int i = 0; i < kJobs; ++i) {
        const ClusterJob j = i == kJobVoc ? p.voc : cluster_job_of(i, E, V);
        const int times = i == kJobVoc ? 1 : L;
        p.block_bytes += (size_t)times * j.parts * j.chunks() * j.chunk_bytes();
        p.all_chunks += times * j.parts * j.chunks();
        if (i == kJobF2) p.layer_chunks = p.all_chunks;
    }
    if (p.all_chunks > 1024 || p.block_bytes > 0xffffffffu || (long long)S * E > 1 << 24) return p;
    // how many clusters of sixteen blocks, one block per SM, the GPU holds at the same time
    const int rc = with_kernel(E, D, 2, 1, [&](auto w) {
        using W = decltype(w);
        if (prepare_kernel<W::kE, W::kD, W::kR, W::kVW>() != cudaSuccess) return 1;
        ClusterLaunch l(1, kSmemMost, nullptr);
        return cudaOccupancyMaxActiveClusters(&p.clusters_most, cluster_steps_kernel<W::kE, W::kD, W::kR, W::kVW>, &l.cfg) == cudaSuccess ? 0 : 1;
    });
    if (rc > 0) cudaGetLastError();
    p.ok = rc == 0 && p.clusters_most > 0;
    return p;
}

void cluster_table(const ClusterPlan &p, int E, int L, uint2 *table)
{
    unsigned off = 0;
    auto job = [&](const ClusterJob &j) {
        for (int i = 0; i < j.parts * j.chunks(); ++i) {
            *table++ = make_uint2(off, (unsigned)j.chunk_bytes());
            off += (unsigned)j.chunk_bytes();
        }
    };
    for (int l = 0; l < L; ++l)
        for (int i = kJobQkv; i <= kJobF2; ++i) job(cluster_job_of(i, E, 0));
    job(p.voc);
}

int cluster_pack(const ClusterPlan &p, int E, const ClusterLayerWeights *layers, int L, const float *wout, uint8_t *dst, cudaStream_t st)
{
    size_t off = 0;
    auto job = [&](const ClusterJob &j, const float *w, const float *bias, const float *gamma, const float *beta) {
        for (int pt = 0; pt < j.parts; ++pt) {
            cluster_pack_kernel<<<dim3(j.chunks(), kClusterBlocks), 256, 0, st>>>(j, pt, w, bias, gamma, beta, dst + off, p.block_bytes);
            off += (size_t)j.chunks() * j.chunk_bytes();
        }
    };
    for (int l = 0; l < L; ++l) {
        const ClusterLayerWeights &w = layers[l];
        job(cluster_job_of(kJobQkv, E, 0), w.wqkv, w.bqkv, w.g1, w.be1);
        job(cluster_job_of(kJobO, E, 0), w.wo, w.bo, nullptr, nullptr);
        job(cluster_job_of(kJobF1, E, 0), w.w1, w.b1, w.g2, w.be2);
        job(cluster_job_of(kJobF2, E, 0), w.w2, w.b2, nullptr, nullptr);
    }
    job(p.voc, wout, nullptr, nullptr, nullptr);
    return check_launch("cluster_pack_kernel");
}

// One sequence per cluster while every cluster is resident, then two; larger batches take the launches, whose matmuls share a
// weight among eight rows.  The ring has to hold a part (sixteen chunks at most) and more.
// `positions` of the longest context: a cluster reads its sequences' keys and values with sixteen SMs, the launches theirs with all,
// so where few clusters have long contexts the launches are ahead.  us per position of a whole run by steps, cluster / launches (two layers): E = 256,
// 2 sequences: 37 / 67 at 8192, 71 / 80 at 16384, 143 / 104 at 32768; 4: 40 / 76, 70 / 101.  E = 128, 2: 39 / 69 at 16384, 71 / 80 at 32768; 8: 72 / 96,
// 128 / 130.  E = 384, 2: 75 / 96 at 8192.  The line, positions x E x (sequences per cluster) / clusters = 3 x 2^20 (24576 positions for the first), was
// found with a slower row kernel in the launches; by these figures both sides meet at 2 to 2.6 x 2^20, and at the line the launches are up to 15 % ahead.
// Where a prompt's positions are taken together (prompt_pass) the steps that remain are those of the longest contexts, and the sides meet earlier: E = 256,
// 8 sequences 129 / 133 us per step behind 8159 positions, 236 / 197 behind 16351; 14: 131 / 178, 243 / 287; E = 384, 8: 120 / 146 behind 4063, 205 / 188 behind 8159.
int cluster_rows(const ClusterPlan &p, int B, int E, int H, int ns, int positions)
{
    if (!p.ok) return 0;
    const int rows = B <= p.clusters_most ? 1 : (B + 1) / 2 <= p.clusters_most ? 2 : 0;
    if (rows == 0 || (long long)positions * E * rows > (3LL << 20) * ((B + rows - 1) / rows)) return 0;
    const int slots = with_kernel(E, E / H, rows, rows * H * ns, [&](auto w) { return rest_of<decltype(w)::kE, decltype(w)::kR>(H, E / H, ns, p.all_chunks).slots; });
    return slots >= 9 ? rows : 0;
}

int launch_cluster_steps(const ClusterPlan &p, const ClusterArgs &a, int E, int rows, cudaStream_t st)
{
    return with_kernel(E, E / a.H, rows, rows * a.H * a.ns, [&](auto w) {
        constexpr int kE = decltype(w)::kE, kD = decltype(w)::kD, kR = decltype(w)::kR, kVW = decltype(w)::kVW;
        const Rest lay = rest_of<kE, kR>(a.H, kE / a.H, a.ns, p.all_chunks);
        cudaError_t e = prepare_kernel<kE, kD, kR, kVW>();
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cluster_steps_kernel attributes: %s", cudaGetErrorString(e));
        ClusterLaunch l((a.B + rows - 1) / rows, (size_t)lay.total, st);
        e = cudaLaunchKernelEx(&l.cfg, cluster_steps_kernel<kE, kD, kR, kVW>, p, a, lay);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cluster_steps_kernel launch: %s", cudaGetErrorString(e));
        return HIPGPT_OK;
    });
}

}  // namespace hipgpt
