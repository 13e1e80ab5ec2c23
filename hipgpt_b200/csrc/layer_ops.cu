// The launchers that stand either side of attention in HipGPT's TransformerLayer::forward and
// GPTModel::forward (src/transformer_layer.cpp:214-253, src/gpt_model.cpp:97-118): projections,
// layer norm, dropout, residual add, ReLU, embedding lookup.  Plain sm_100a CUDA with the
// reference's arithmetic restated exactly, so that an unchanged HipGPT layer runs on this library.
//
//   matmul(+bias)   C[M][K] = A[M][N] B[N][K] (+ bias[K]): HipGPT's argument order, N is the inner
//                   dimension (src/hip_kernels.cpp:69-154).  One accumulator per output, terms added
//                   k ascending with fused multiply-add, the bias added once at the end: the
//                   summation order of the reference kernel, hence bit-identical to its arithmetic.
//                   Register-tiled, operands staged through shared memory.
//   layer norm      src/hip_kernels.cpp:757-848: mean, variance about the mean, 1/sqrt(var + 1e-5),
//                   gamma (x - mean) inv + beta.  One warp per row; the reference reduces in 64-lane
//                   waves, so sums agree to rounding (about 1e-7), not bitwise.
//   dropout         src/hip_kernels.cpp:944-970 with the generator at :24-42: the mask is a pure function
//                   of the element index; restated in integer arithmetic, bit-identical.
//   add, ReLU, embedding lookup   src/hip_kernels.cpp:721-730, :248-258, :537-599; bit-identical.
#include "tc_primitives.cuh"

#include <math.h>

#include <algorithm>
#include <initializer_list>

namespace hipgpt {
namespace {

// A tile is 8 TM x 16 TN outputs, 128 threads of TM x TN; TM and TN are chosen per call so that the tiles fill the SMs evenly
// (launch_matmul_tiles).
// Two bounds: the FFMA pipe, TM TN clocks per inner index and warp, and the return path of shared memory, which hands a warp 128
// bytes per clock whether lanes ask for the same words or not: 4 (TM + TN) clocks for the four warps of an SM's quarters.  8 x 8
// outputs per thread are bound by the second; 8 x 16 (and 7 x 16) leave it at three quarters of the first.  The rest is kept out
// of the issue slots: multiply-adds run on pairs of columns (fma.rn.f32x2, one instruction for two roundings), and both operands
// come by 16-byte asynchronous copies, three stages, A untransposed (a thread reads four inner indices of a row at once).
// Registers alone (the same multiply-adds without loads) reach 61 TFLOP/s; here 54 at 16384 x 512 x 1536 (one inner index after
// another in 128 x 128 tiles, operands through registers: 47.7).  With 8192 rows: 256 -> 768 columns 80 -> 63 us, 256 -> 256 35 -> 27,
// 256 -> 1024 105 -> 83, 1024 -> 256 125 -> 92.
// Small products (TN = 4) are bound by neither but by the distance from a load to its use and by what a stage costs besides: their fragments are read
// eight inner indices of B and four of A ahead, a stage has 32 inner indices, and where few tiles have to fill many SMs a block has TY = 4 rows of
// threads instead of 8: half as many warps at the return path.  (Not where each SM has many tiles and each few inner indices: three short stages then, which take little
// memory, so that many blocks share an SM.)  Rows x inner x columns: 100 x 1024 x 256 21.1 -> 12.4 us, 400 x 256 x 768 9.8 -> 7.5,
// 200 x 2048 x 512 41.3 -> 30.9, 2000 x 768 x 192 28.0 -> 19.5.  (Deeper stages for the tiles between, 5 x 8 and so on: 1407 x 512 x 2048 65 -> 66.)
template <int TM, int TN, int TY, bool DEEP>
struct TileCfg {
    static constexpr bool kSmall = DEEP;
    static constexpr int kBK = kSmall ? 32 : 16, kStages = kSmall ? 5 : 3;         // inner indices of a stage
    static constexpr int kThreads = 16 * TY, BM = TY * TM, BN = 16 * TN;
    static constexpr int kAheadB = kSmall ? 8 : 2, kAheadA = kSmall ? 2 : 1;      // fragments in registers: of an index of B, of four of A
    static constexpr int AStride = kBK + 4;                              // floats between rows of A in shared memory
    static constexpr int kStageFloats = BM * AStride + kBK * BN;
    static constexpr size_t kSmem = (size_t)kStages * kStageFloats * 4;
};
template <int TM, int TN, int TY, bool DEEP>
__global__ void __launch_bounds__(16 * TY, TM * TN > 64 ? 2 : 3)
matmul_tile_kernel(const float *A, const float *__restrict__ B, const float *__restrict__ bias, float *C,     // A and C may be one buffer
                   int M, int N, int K, int col_tiles)
{
    using T = TileCfg<TM, TN, TY, DEEP>;
    constexpr int BM = T::BM, BN = T::BN, kTileThreads = T::kThreads, kBK = T::kBK;
    extern __shared__ __align__(16) float tile_s[];                      // [stage][A: BM rows of kBK | B: kBK rows of BN]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    // column tile fastest: blocks that run side by side share rows of A
    const int row0 = (int)(blockIdx.x / col_tiles) * BM, col0 = (int)(blockIdx.x % col_tiles) * BN;

    dependency_wait();                                       // overlapped launch: nothing is read before the kernel before this one has completed
    dependents_may_start();
    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = make_float2(0.0f, 0.0f);

    const int ntiles = (N + kBK - 1) / kBK;
    auto copy = [&](int t) {
        if (t < ntiles) {
            float *as = tile_s + (t % T::kStages) * T::kStageFloats, *bs = as + BM * T::AStride;
            const int k0 = t * kBK;
#pragma unroll
            for (int i = 0; i < (BM * (kBK / 4) + kTileThreads - 1) / kTileThreads; ++i) {
                const int f = tid + i * kTileThreads, m = f / (kBK / 4), k = f % (kBK / 4) * 4;
                const bool in = row0 + m < M && k0 + k < N;
                if (BM * (kBK / 4) % kTileThreads == 0 || f < BM * (kBK / 4)) cp_async16(as + m * T::AStride + k, A + (in ? (size_t)(row0 + m) * N + k0 + k : 0), in);
            }
#pragma unroll
            for (int i = 0; i < kBK * BN / 4 / kTileThreads; ++i) {
                const int f = tid + i * kTileThreads, kr = f / (BN / 4), cc = (f % (BN / 4)) * 4;
                const bool in = k0 + kr < N && col0 + cc < K;
                cp_async16(bs + kr * BN + cc, B + (in ? (size_t)(k0 + kr) * K + col0 + cc : 0), in);
            }
        }
        cp_async_commit();
    };
#pragma unroll
    for (int t = 0; t + 1 < T::kStages; ++t) copy(t);
    for (int t = 0; t < ntiles; ++t) {
        cp_async_wait<T::kStages - 2>();                     // tile t is there (this thread's part)
        __syncthreads();                                     // everybody's part; and everybody is done with tile t - 1
        copy(t + T::kStages - 1);
        const float *as = tile_s + (t % T::kStages) * T::kStageFloats + ty * TM * T::AStride;
        const float *bs = tile_s + (t % T::kStages) * T::kStageFloats + BM * T::AStride + tx * 4;
        constexpr int PB = T::kAheadB, PA = T::kAheadA;
        float2 b[PB][TN / 2];
        auto load_b = [&](int k) {
#pragma unroll
            for (int j = 0; j < TN / 4; ++j) *reinterpret_cast<float4 *>(&b[k % PB][2 * j]) = *reinterpret_cast<const float4 *>(bs + k * BN + 64 * j);
        };
        float a[PA][TM][4];
        auto load_a = [&](int i, int k) { *reinterpret_cast<float4 *>(a[k / 4 % PA][i]) = *reinterpret_cast<const float4 *>(as + i * T::AStride + k); };
#pragma unroll
        for (int i = 0; i < TM; ++i) load_a(i, 0);
#pragma unroll
        for (int k = 0; k + 1 < PB; ++k) load_b(k);
#pragma unroll
        for (int k = 0; k < kBK; ++k) {
            if (k + PB - 1 < kBK) load_b(k + PB - 1);
            if (PA > 1 && (k & 3) == 0 && k + 4 < kBK)
#pragma unroll
                for (int i = 0; i < TM; ++i) load_a(i, k + 4);
            float2 aa[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) aa[i] = make_float2(a[k / 4 % PA][i][k & 3], a[k / 4 % PA][i][k & 3]);
            if (PA == 1 && (k & 3) == 3 && k + 1 < kBK)
#pragma unroll
                for (int i = 0; i < TM; ++i) load_a(i, k + 1);
#pragma unroll
            for (int j = 0; j < TN / 2; ++j)
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = ffma2(aa[i], b[k % PB][j], acc[i][j]);
        }
    }
    float4 bb[TN / 4];
#pragma unroll
    for (int j = 0; j < TN / 4; ++j) {
        const int c = col0 + tx * 4 + 64 * j;
        bb[j] = (bias && c < K) ? *reinterpret_cast<const float4 *>(bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = row0 + ty * TM + i;
        if (r >= M) continue;
#pragma unroll
        for (int j = 0; j < TN / 4; ++j) {
            const int c = col0 + tx * 4 + 64 * j;
            if (c >= K) continue;                            // K % 4 == 0 on this path: a group of four is in or out
            float4 v = make_float4(acc[i][2 * j].x, acc[i][2 * j].y, acc[i][2 * j + 1].x, acc[i][2 * j + 1].y);
            if (bias) { v.x += bb[j].x; v.y += bb[j].y; v.z += bb[j].z; v.w += bb[j].w; }
            *reinterpret_cast<float4 *>(C + (size_t)r * K + c) = v;
        }
    }
}

// Any sizes and alignments: one thread per output, the same order of additions.
__global__ void matmul_plain_kernel(const float *__restrict__ A, const float *__restrict__ B, const float *__restrict__ bias,
                                    float *__restrict__ C, int M, int N, int K)
{
    const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (long long)M * K) return;
    const int r = (int)(idx / K), c = (int)(idx % K);
    float s = 0.0f;
    for (int k = 0; k < N; ++k) s = fmaf(A[(size_t)r * N + k], B[(size_t)k * K + c], s);
    C[idx] = bias ? s + bias[c] : s;
}

// The kernels below are passes over memory of a few microseconds: 16-byte accesses where the pointers allow, and overlapped
// launches, so that a kernel's blocks are placed while the kernel before it drains (without: about a microsecond between two).

// One warp per row.  Sums: lane l adds elements l, l + 32, ... ascending, then a butterfly over the lanes.
// Separately rounded multiplies and adds (no contraction), IEEE division and square root: the CPU oracle
// built without contraction reproduces every bit.  NV > 0: the row (E <= 32 NV) stays in registers between the three sweeps.
template <int NV>
__global__ void layer_norm_rows_kernel(const float *x, float *y, const float *__restrict__ g,
                                       const float *__restrict__ b, int rows, int E)
{
    dependency_wait();
    dependents_may_start();
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= rows) return;
    const float *xr = x + (size_t)row * E;
    float *yr = y + (size_t)row * E;
    float v[NV > 0 ? NV : 1];
    float s = 0.0f, q = 0.0f;
    if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) v[i] = lane + 32 * i < E ? xr[lane + 32 * i] : 0.0f;
#pragma unroll
        for (int i = 0; i < NV; ++i) s = lane + 32 * i < E ? __fadd_rn(s, v[i]) : s;
    } else {
        for (int e = lane; e < E; e += 32) s = __fadd_rn(s, xr[e]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    const float mean = __fdiv_rn(s, (float)E);
    if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            v[i] = __fsub_rn(v[i], mean);
            q = lane + 32 * i < E ? __fadd_rn(q, __fmul_rn(v[i], v[i])) : q;
        }
    } else {
        for (int e = lane; e < E; e += 32) {
            const float d = __fsub_rn(xr[e], mean);
            q = __fadd_rn(q, __fmul_rn(d, d));
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q = __fadd_rn(q, __shfl_xor_sync(0xffffffffu, q, o));
    const float inv = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(q, (float)E), 1e-5f)));
    if constexpr (NV > 0) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int e = lane + 32 * i;
            if (e < E) yr[e] = __fadd_rn(__fmul_rn(__fmul_rn(__ldg(g + e), v[i]), inv), __ldg(b + e));
        }
    } else {
        for (int e = lane; e < E; e += 32)
            yr[e] = __fadd_rn(__fmul_rn(__fmul_rn(g[e], __fsub_rn(xr[e], mean)), inv), b[e]);
    }
}

// The reference seeds a xorwow state from the element index, its 256-thread block and its thread
// (a = idx + 1, b = block + 1, c = thread + 1, d = idx * block + 1) and draws once: only a and d reach
// that first draw.  u = (t + 1) / 2^32; the element is dropped when u < p, else divided by (1 - p).
__device__ __forceinline__ bool dropped(unsigned idx, float p)
{
    const unsigned s = idx + 1u;
    unsigned t = idx * (idx >> 8) + 1u;          // the reference's block of an element is idx / 256
    t ^= t >> 2;
    t ^= t << 1;
    t ^= s ^ (s << 4);
    return __fmul_rn((float)(t + 1u), 2.3283064365386963e-10f) < p;       // / 2^32: exact
}

// out = dropout(in), or out = residual + dropout(in): the sub-layer tail of the reference's block (dropout in place, then
// the residual add, src/transformer_layer.cpp:242-244 and :250-252) in one pass over memory instead of three, bit-identical to
// hipgpt_dropout followed by hipgpt_add_inplace.  Four consecutive elements per thread when the count and the pointers allow
// 16-byte accesses.
template <bool RESIDUAL>
__global__ void __launch_bounds__(256)
dropout_kernel(const float *in, const float *residual, float *out, float *__restrict__ mask, float p, unsigned n, int vec)   // out may be in or residual
{
    dependency_wait();
    dependents_may_start();
    const float keep = __fsub_rn(1.0f, p);
    if (vec) {
        const unsigned i4 = (blockIdx.x * 256u + threadIdx.x) * 4u;
        if (i4 >= n) return;
        const float4 x = *reinterpret_cast<const float4 *>(in + i4);
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (RESIDUAL) r = *reinterpret_cast<const float4 *>(residual + i4);
        const bool d0 = dropped(i4, p), d1 = dropped(i4 + 1u, p), d2 = dropped(i4 + 2u, p), d3 = dropped(i4 + 3u, p);
        float4 o;
        o.x = d0 ? 0.0f : __fdiv_rn(x.x, keep);
        o.y = d1 ? 0.0f : __fdiv_rn(x.y, keep);
        o.z = d2 ? 0.0f : __fdiv_rn(x.z, keep);
        o.w = d3 ? 0.0f : __fdiv_rn(x.w, keep);
        if (RESIDUAL) { o.x = __fadd_rn(r.x, o.x); o.y = __fadd_rn(r.y, o.y); o.z = __fadd_rn(r.z, o.z); o.w = __fadd_rn(r.w, o.w); }
        *reinterpret_cast<float4 *>(out + i4) = o;
        if (mask) *reinterpret_cast<float4 *>(mask + i4) = make_float4(d0 ? 0.f : 1.f, d1 ? 0.f : 1.f, d2 ? 0.f : 1.f, d3 ? 0.f : 1.f);
    } else {
        const unsigned idx = blockIdx.x * 256u + threadIdx.x;
        if (idx >= n) return;
        const bool d = dropped(idx, p);
        const float o = d ? 0.0f : __fdiv_rn(in[idx], keep);
        out[idx] = RESIDUAL ? __fadd_rn(residual[idx], o) : o;
        if (mask) mask[idx] = d ? 0.0f : 1.0f;
    }
}

// a = a + b, or a = max(0, a); `n4` groups of four elements, then the rest one by one.  A thread takes U groups (or rest elements), 256 apart
template <bool ADD, int U>
__global__ void __launch_bounds__(256)
pass_kernel(float *a, const float *__restrict__ b, long long n4, long long n)
{
    dependency_wait();
    dependents_may_start();
    const long long i0 = (long long)blockIdx.x * (256 * U) + threadIdx.x;
    float4 x[U], y[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = i0 + 256 * u;
        if (i < n4) {
            x[u] = reinterpret_cast<const float4 *>(a)[i];
            if (ADD) y[u] = __ldg(reinterpret_cast<const float4 *>(b) + i);
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const long long i = i0 + 256 * u;
        if (i < n4) {
            if (ADD) x[u] = make_float4(__fadd_rn(x[u].x, y[u].x), __fadd_rn(x[u].y, y[u].y), __fadd_rn(x[u].z, y[u].z), __fadd_rn(x[u].w, y[u].w));
            else x[u] = make_float4(fmaxf(0.0f, x[u].x), fmaxf(0.0f, x[u].y), fmaxf(0.0f, x[u].z), fmaxf(0.0f, x[u].w));
            reinterpret_cast<float4 *>(a)[i] = x[u];
        } else {
            const long long e = 4 * n4 + (i - n4);
            if (e < n) a[e] = ADD ? __fadd_rn(a[e], b[e]) : fmaxf(0.0f, a[e]);
        }
    }
}

// out[t][e] = tok[id_t][e] + pos[t mod S][e]; an id outside [0, V) gives a row of zeros.  VEC: four elements per thread.
template <bool VEC>
__global__ void __launch_bounds__(256)
embedding_kernel(const int *__restrict__ ids, const float *__restrict__ tok, const float *__restrict__ pos,
                 float *__restrict__ out, long long T, int S, int V, int E)
{
    dependency_wait();
    dependents_may_start();
    constexpr int W = VEC ? 4 : 1;
    const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * W;
    if (i >= T * E) return;
    const long long t = i / E;
    const int e = (int)(i % E), id = ids[t];
    const bool ok = id >= 0 && id < V;
    if constexpr (VEC) {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (ok) {
            const float4 x = __ldg(reinterpret_cast<const float4 *>(tok + (size_t)id * E + e)), y = __ldg(reinterpret_cast<const float4 *>(pos + (size_t)(t % S) * E + e));
            o = make_float4(__fadd_rn(x.x, y.x), __fadd_rn(x.y, y.y), __fadd_rn(x.z, y.z), __fadd_rn(x.w, y.w));
        }
        *reinterpret_cast<float4 *>(out + i) = o;
    } else {
        out[i] = ok ? __fadd_rn(tok[(size_t)id * E + e], pos[(size_t)(t % S) * E + e]) : 0.0f;
    }
}

bool aligned16(std::initializer_list<const void *> ps)
{
    uintptr_t all = 0;
    for (const void *p : ps) all |= reinterpret_cast<uintptr_t>(p);
    return (all & 15) == 0;
}

bool overlap(const void *a, size_t na, const void *b, size_t nb)
{
    const uintptr_t a0 = reinterpret_cast<uintptr_t>(a), b0 = reinterpret_cast<uintptr_t>(b);
    return a0 < b0 + nb && b0 < a0 + na;
}

}  // namespace

// The tile of a product.  In place (C over A) a block must own whole rows: it stores after its last read.  Cost: clocks of the SM with the most tiles: a tile's own
// bound (see above) times the inner indices, whole stages of them, and what a block costs besides; an SM with a single block of four warps hides less latency,
// about a fifth; of blocks of two warps with five stages only three to five fit an SM, a tenth where there are more; the wide tiles stay 30 % off
// their bound, the tiles of 64 columns within 10 %.  The larger tile among equals.
// Fitted to the times of all nineteen tiles at eighty shapes (30 - 120000 rows, 8 - 400 inner, 8 - 400 columns and a few beyond): 1.1 % above the best
// tile in the geometric mean, 14 % at most.  By the bound alone, and without the tiles of three short stages: 6.8 % and 62 %, worst where a short inner
// dimension meets many rows (rows x inner x columns 40114 x 48 x 8 16.1 us, now 10; 61815 x 36 x 12 23.9, now 18; 29618 x 104 x 52 19.4, now 15).
struct TileChoice {
    void (*kernel)(const float *, const float *, const float *, float *, int, int, int, int);
    int tm, tn, ty, bk;
    size_t smem;
};
template <int TM, int TN, int TY = 8, bool DEEP = TN == 4>
TileChoice tile_choice() { return {matmul_tile_kernel<TM, TN, TY, DEEP>, TM, TN, TY, TileCfg<TM, TN, TY, DEEP>::kBK, TileCfg<TM, TN, TY, DEEP>::kSmem}; }

static int launch_matmul_tiles(const float *A, const float *B, const float *bias, float *C, int M, int N, int K, bool whole_rows, cudaStream_t st)
{
    static const TileChoice choices[] = {tile_choice<8, 16>(), tile_choice<7, 16>(), tile_choice<6, 16>(), tile_choice<5, 16>(), tile_choice<8, 8>(), tile_choice<7, 8>(),
                                         tile_choice<6, 8>(), tile_choice<5, 8>(), tile_choice<4, 8>(), tile_choice<3, 8>(), tile_choice<4, 4>(),
                                         tile_choice<6, 4, 4>(), tile_choice<5, 4, 4>(), tile_choice<4, 4, 4>(), tile_choice<3, 4, 4>(), tile_choice<2, 4, 4>(), tile_choice<1, 4, 4>(), tile_choice<4, 4, 8, false>(), tile_choice<2, 4, 8, false>()};
    constexpr int kSms = 148, kSmSharedBytes = 228 * 1024;
    const TileChoice *best = nullptr;
    double best_cost = 0.0;
    long long best_tiles = 0;
    for (const TileChoice &c : choices) {
        if (whole_rows && K > 16 * c.tn) continue;
        const long long tiles = (long long)((M + c.ty * c.tm - 1) / (c.ty * c.tm)) * ((K + 16 * c.tn - 1) / (16 * c.tn));
        const long long per_sm = (tiles + kSms - 1) / kSms;
        const int fma = c.tm * c.tn, loads = c.ty / 2 * (c.tm + c.tn), clocks = fma > loads ? fma : loads;
        const double inner = (double)((N + c.bk - 1) & -c.bk), fixed = c.tn == 16 ? 1300.0 : c.tn == 8 ? 900.0 : c.ty == 4 ? 300.0 : 0.0, off = c.tn > 4 ? 1.3 : c.ty == 4 && per_sm >= 3 ? 1.1 : 1.0;
        const double cost = (double)per_sm * (clocks * inner * off + fixed) * (per_sm == 1 ? 1.2 : 1.0);
        if (!best || cost < best_cost) { best = &c; best_cost = cost; best_tiles = tiles; }
    }
    if (best_tiles > 2147483647LL) return fail(HIPGPT_ERR_BAD_ARG, "matmul: %lld tiles are too many", best_tiles);
    // Blocks of an overlapped launch come in beside the last blocks of the kernel before, as many on an SM as fit, and so unevenly: where every SM is to
    // have one, two or three, a further one that fits leaves another SM without.  So a block asks for so much shared memory that no more than that fit.
    // Behind itself: 8192 x 256 x 256 34.3 -> 24.3 us, 8192 x 1024 x 256 130.7 -> 90.2, 5000 x 512 x 320 66.9 -> 46.4.  A block of the model, where the products
    // follow other kernels: 8192 rows E=256 333.7 -> 322.4, sixteen others of 47 - 4807 rows 0.69 - 0.99 of their time, 0.82 in the mean (with the line at two:
    // up to 1.26, where the kernel before has fewer blocks than fit).  More tiles per SM even out by themselves.
    const long long per_sm = (best_tiles + kSms - 1) / kSms;
    size_t smem = best->smem;
    if (per_sm <= 3) smem = std::max(smem, (size_t)(((size_t)kSmSharedBytes / (size_t)(per_sm + 1) + 128) & ~(size_t)127));
    cudaError_t e = cudaFuncSetAttribute(best->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)std::max(best->smem, (size_t)kSmSharedBytes / 2 + 128));
    if (e == cudaSuccess)
        e = launch_overlapped(best->kernel, dim3((unsigned)best_tiles), dim3((unsigned)(16 * best->ty)), smem, st, A, B, bias, C, M, N, K, (K + 16 * best->tn - 1) / (16 * best->tn));
    if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "matmul_tile_kernel: %s", cudaGetErrorString(e));
    return HIPGPT_OK;
}

int launch_matmul_exact(const float *A, const float *B, const float *bias, float *C, int M, int N, int K, cudaStream_t st)
{
    if (M == 0 || K == 0) return HIPGPT_OK;
    const bool vec = (N % 4 == 0) && (K % 4 == 0) &&
                     ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C) |
                       reinterpret_cast<uintptr_t>(bias)) & 15) == 0;
    // HipGPT's layer projects in place (src/transformer_layer.cpp:220 passes the same buffer as A and C).  That is
    // safe when one block holds whole rows of C: it reads its rows of A completely before it stores.
    const bool alias = overlap(A, (size_t)M * N * 4, C, (size_t)M * K * 4);
    if (alias && (!vec || K > 256)) return fail(HIPGPT_ERR_UNSUPPORTED, "matmul in place needs an output of at most 256 columns, a multiple of 4 (K=%d)", K);
    if (vec) return launch_matmul_tiles(A, B, bias, C, M, N, K, alias, st);
    const long long n = (long long)M * K;
    matmul_plain_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(A, B, bias, C, M, N, K);
    return check_launch("matmul_plain_kernel");
}

namespace {
int launched(cudaError_t e, const char *what) { return e == cudaSuccess ? HIPGPT_OK : fail(HIPGPT_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e)); }
}  // namespace

int launch_layer_norm_rows(const float *x, float *y, const float *g, const float *b, int rows, int E, cudaStream_t st)
{
    if (rows == 0 || E == 0) return HIPGPT_OK;
    const auto kern = E <= 128 ? layer_norm_rows_kernel<4> : E <= 256 ? layer_norm_rows_kernel<8> : E <= 512 ? layer_norm_rows_kernel<16>
                      : E <= 1024 ? layer_norm_rows_kernel<32> : layer_norm_rows_kernel<0>;
    return launched(launch_overlapped(kern, dim3((unsigned)((rows + 7) / 8)), dim3(256), 0, st, x, y, g, b, rows, E), "layer_norm_rows_kernel");
}

int launch_dropout_index(const float *in, float *out, float *mask, float p, long long n, cudaStream_t st)
{
    if (n == 0) return HIPGPT_OK;
    if (n > 0xffffffffLL) return fail(HIPGPT_ERR_BAD_ARG, "dropout over %lld elements: the reference's index is 32 bits wide", n);
    const int vec = n % 4 == 0 && aligned16({in, out, mask});
    return launched(launch_overlapped(dropout_kernel<false>, dim3((unsigned)(((vec ? n / 4 : n) + 255) / 256)), dim3(256), 0, st, in, (const float *)nullptr, out, mask, p,
                                      (unsigned)n, vec), "dropout_kernel");
}

int launch_dropout_residual(const float *in, const float *residual, float *out, float *mask, float p, long long n, cudaStream_t st)
{
    if (n == 0) return HIPGPT_OK;
    if (n > 0xffffffffLL) return fail(HIPGPT_ERR_BAD_ARG, "dropout over %lld elements: the reference's index is 32 bits wide", n);
    const int vec = n % 4 == 0 && aligned16({in, residual, out, mask});
    return launched(launch_overlapped(dropout_kernel<true>, dim3((unsigned)(((vec ? n / 4 : n) + 255) / 256)), dim3(256), 0, st, in, residual, out, mask, p, (unsigned)n, vec),
                    "dropout_kernel");
}

template <bool ADD>
static int launch_pass(float *a, const float *b, long long n, cudaStream_t st, const char *what)
{
    if (n == 0) return HIPGPT_OK;
    const long long n4 = aligned16({a, b}) ? n / 4 : 0, threads = n4 + (n - 4 * n4);
    // One group per thread while all blocks are on the SMs at once (148 x 2048 threads), else two: a block of the default model 323.3 -> 321.9 us, 6660 rows
    // E=160 221.8 -> 220.5, with packed weights (1407 rows, E=512) 83.1 -> 82.7; four: 323.3, 220.8, 87.1.
    const bool one = threads <= 148 * 2048;
    const auto kern = one ? pass_kernel<ADD, 1> : pass_kernel<ADD, 2>;
    const long long per = one ? 256 : 512;
    return launched(launch_overlapped(kern, dim3((unsigned)((threads + per - 1) / per)), dim3(256), 0, st, a, b, n4, n), what);
}

int launch_add_inplace_n(float *a, const float *b, long long n, cudaStream_t st) { return launch_pass<true>(a, b, n, st, "add_inplace"); }

int launch_relu_n(float *a, long long n, cudaStream_t st) { return launch_pass<false>(a, nullptr, n, st, "relu"); }

int launch_embedding_rows(const int *ids, const float *tok, const float *pos, float *out, int B, int S, int V, int E, cudaStream_t st)
{
    const long long n = (long long)B * S * E;
    if (n == 0) return HIPGPT_OK;
    const bool vec = E % 4 == 0 && aligned16({tok, pos, out});
    const long long threads = vec ? n / 4 : n;
    return launched(launch_overlapped(vec ? embedding_kernel<true> : embedding_kernel<false>, dim3((unsigned)((threads + 255) / 256)), dim3(256), 0, st, ids, tok, pos, out,
                                      (long long)B * S, S, V, E), "embedding_kernel");
}

}  // namespace hipgpt

using namespace hipgpt;

extern "C" {

int hipgpt_matmul(const float *d_A, const float *d_B, const float *d_bias, float *d_C, int M, int N, int K, void *stream)
{
    if (M < 0 || N < 0 || K < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: M=%d N=%d K=%d", M, N, K);
    if (M == 0 || K == 0) return HIPGPT_OK;
    if (!d_C || (N > 0 && (!d_A || !d_B))) return fail(HIPGPT_ERR_NULL, "A, B and C must not be NULL");
    return launch_matmul_exact(d_A, d_B, d_bias, d_C, M, N, K, static_cast<cudaStream_t>(stream));
}

int hipgpt_matmul_tc(const float *d_A, const float *d_B, const float *d_bias, float *d_C, int M, int N, int K, void *stream)
{
    if (M < 0 || N < 0 || K < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: M=%d N=%d K=%d", M, N, K);
    if (M == 0 || K == 0) return HIPGPT_OK;
    if (!d_C || (N > 0 && (!d_A || !d_B))) return fail(HIPGPT_ERR_NULL, "A, B and C must not be NULL");
    if (N == 0) return launch_matmul_exact(d_A, d_B, d_bias, d_C, M, N, K, static_cast<cudaStream_t>(stream));   // bias (or zeros) only
    if (d_C == d_A || d_C == d_B) return fail(HIPGPT_ERR_UNSUPPORTED, "the tensor-core product does not work in place; hipgpt_matmul does (K <= 256)");
    return launch_matmul_tc(d_A, d_B, d_bias, d_C, M, N, K, static_cast<cudaStream_t>(stream));
}

int hipgpt_matmul_tc_prepare(const float *d_B, int N, int K, hipgpt_packed_matrix **out, void *stream)
{
    if (!out || !d_B) return fail(HIPGPT_ERR_NULL, "B and out must not be NULL");
    if (N <= 0 || K <= 0) return fail(HIPGPT_ERR_BAD_ARG, "bad size: N=%d K=%d", N, K);
    PackedB *p = nullptr;
    const int rc = matmul_tc_prepare(d_B, N, K, &p, static_cast<cudaStream_t>(stream));
    if (rc == HIPGPT_OK) *out = reinterpret_cast<hipgpt_packed_matrix *>(p);
    return rc;
}

int hipgpt_matmul_tc_prepared(const float *d_A, const hipgpt_packed_matrix *b, const float *d_bias, float *d_C, int M, void *stream)
{
    if (!b) return fail(HIPGPT_ERR_NULL, "the packed right-hand side must not be NULL");
    if (M < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: M=%d", M);
    if (M == 0) return HIPGPT_OK;
    if (!d_A || !d_C) return fail(HIPGPT_ERR_NULL, "A and C must not be NULL");
    if (d_A == d_C) return fail(HIPGPT_ERR_UNSUPPORTED, "the tensor-core product does not work in place");
    return launch_matmul_tc_prepared(d_A, reinterpret_cast<const PackedB *>(b), d_bias, d_C, M, static_cast<cudaStream_t>(stream));
}

void hipgpt_matmul_tc_release(hipgpt_packed_matrix *b) { matmul_tc_release(reinterpret_cast<PackedB *>(b)); }

int hipgpt_ln_matmul_tc(const float *d_A, const float *d_gamma, const float *d_beta, const float *d_B, const float *d_bias, float *d_C,
                        int M, int N, int K, void *stream)
{
    if (M < 0 || N <= 0 || K < 0) return fail(HIPGPT_ERR_BAD_ARG, "bad size: M=%d N=%d K=%d", M, N, K);
    if (M == 0 || K == 0) return HIPGPT_OK;
    if (!d_A || !d_B || !d_C || !d_gamma || !d_beta) return fail(HIPGPT_ERR_NULL, "A, gamma, beta, B and C must not be NULL");
    if (d_C == d_A || d_C == d_B) return fail(HIPGPT_ERR_UNSUPPORTED, "the tensor-core product does not work in place");
    return launch_matmul_tc(d_A, d_B, d_bias, d_C, M, N, K, static_cast<cudaStream_t>(stream), d_gamma, d_beta);
}

int hipgpt_ln_matmul_tc_prepared(const float *d_A, const float *d_gamma, const float *d_beta, const hipgpt_packed_matrix *b, const float *d_bias,
                                 float *d_C, int M, void *stream)
{
    if (!b) return fail(HIPGPT_ERR_NULL, "the packed right-hand side must not be NULL");
    if (M < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: M=%d", M);
    if (M == 0) return HIPGPT_OK;
    if (!d_A || !d_C || !d_gamma || !d_beta) return fail(HIPGPT_ERR_NULL, "A, gamma, beta and C must not be NULL");
    if (d_A == d_C) return fail(HIPGPT_ERR_UNSUPPORTED, "the tensor-core product does not work in place");
    return launch_matmul_tc_prepared(d_A, reinterpret_cast<const PackedB *>(b), d_bias, d_C, M, static_cast<cudaStream_t>(stream), d_gamma, d_beta);
}

int hipgpt_layer_norm(const float *d_in, float *d_out, const float *d_gamma, const float *d_beta, int rows, int E, void *stream)
{
    if (rows < 0 || E < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: rows=%d E=%d", rows, E);
    if (rows == 0 || E == 0) return HIPGPT_OK;
    if (!d_in || !d_out || !d_gamma || !d_beta) return fail(HIPGPT_ERR_NULL, "input, output, gamma and beta must not be NULL");
    return launch_layer_norm_rows(d_in, d_out, d_gamma, d_beta, rows, E, static_cast<cudaStream_t>(stream));
}

int hipgpt_dropout(const float *d_in, float *d_out, float *d_mask, float p, int rows, int E, void *stream)
{
    if (rows < 0 || E < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: rows=%d E=%d", rows, E);
    if (!(p >= 0.0f && p < 1.0f)) return fail(HIPGPT_ERR_BAD_ARG, "dropout probability %g outside [0, 1)", (double)p);
    if (rows == 0 || E == 0) return HIPGPT_OK;
    if (!d_in || !d_out) return fail(HIPGPT_ERR_NULL, "input and output must not be NULL");
    return launch_dropout_index(d_in, d_out, d_mask, p, (long long)rows * E, static_cast<cudaStream_t>(stream));
}

int hipgpt_dropout_residual(const float *d_in, const float *d_residual, float *d_out, float *d_mask, float p, int rows, int E, void *stream)
{
    if (rows < 0 || E < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: rows=%d E=%d", rows, E);
    if (!(p >= 0.0f && p < 1.0f)) return fail(HIPGPT_ERR_BAD_ARG, "dropout probability %g outside [0, 1)", (double)p);
    if (rows == 0 || E == 0) return HIPGPT_OK;
    if (!d_in || !d_residual || !d_out) return fail(HIPGPT_ERR_NULL, "input, residual and output must not be NULL");
    return launch_dropout_residual(d_in, d_residual, d_out, d_mask, p, (long long)rows * E, static_cast<cudaStream_t>(stream));
}

int hipgpt_add_inplace(float *d_a, const float *d_b, long long n, void *stream)
{
    if (n < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: n=%lld", n);
    if (n == 0) return HIPGPT_OK;
    if (!d_a || !d_b) return fail(HIPGPT_ERR_NULL, "a and b must not be NULL");
    return launch_add_inplace_n(d_a, d_b, n, static_cast<cudaStream_t>(stream));
}

int hipgpt_relu(float *d_a, long long n, void *stream)
{
    if (n < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: n=%lld", n);
    if (n == 0) return HIPGPT_OK;
    if (!d_a) return fail(HIPGPT_ERR_NULL, "a must not be NULL");
    return launch_relu_n(d_a, n, static_cast<cudaStream_t>(stream));
}

int hipgpt_embedding_lookup(const int *d_ids, const float *d_tok, const float *d_pos, float *d_out, int B, int S, int V, int E, void *stream)
{
    if (B < 0 || S < 0 || V < 0 || E < 0) return fail(HIPGPT_ERR_BAD_ARG, "negative size: B=%d S=%d V=%d E=%d", B, S, V, E);
    if (B == 0 || S == 0 || E == 0) return HIPGPT_OK;
    if (!d_ids || !d_tok || !d_pos || !d_out) return fail(HIPGPT_ERR_NULL, "ids, embeddings and output must not be NULL");
    return launch_embedding_rows(d_ids, d_tok, d_pos, d_out, B, S, V, E, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
