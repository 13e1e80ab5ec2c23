// Shared device helpers and the error channel of the attention library (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>

#include "hipgpt_attn.h"

namespace hipgpt {

// Records the calling thread's failure text and returns `code` (host side, capi.cu).
int fail(int code, const char *fmt, ...);
// hipgpt_debug_expire_wait: (block << 8 | site) for the calling thread's next launch of the kernels whose status codes start at `family`,
// 0 where nothing was asked for.  Asking clears it.
int take_expiry(int family);
// Checks the launch that was just enqueued; HIPGPT_OK or HIPGPT_ERR_CUDA.
int check_launch(const char *what);

// Launch with programmatic stream serialization: the kernel's blocks may become resident, and run their prologue
// (barriers, TMEM, roles), while the last blocks of the kernel before it on the stream are still running, once those
// have let their dependents go.  Such a kernel must execute dependency_wait() before its first access to global
// memory; the wait returns when the kernel before it has completed and its writes are visible.
// HIPGPT_NO_OVERLAPPED_LAUNCH=1 launches the plain way.
// `cluster` > 1: that many consecutive blocks form a cluster.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_overlapped_clusters(void (*kern)(KArgs...), int cluster, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args)
{
    static const bool plain = [] { const char *e = getenv("HIPGPT_NO_OVERLAPPED_LAUNCH"); return e && *e && *e != '0'; }();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (!plain) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_overlapped(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args)
{
    return launch_overlapped_clusters(kern, 1, grid, block, smem, st, args...);
}

// A kernel's limit of dynamic shared memory belongs to the kernel on one device: set() runs at the first call on each.
// `done`: a bit per device, one word per kernel (or set of kernels).
template <typename Set>
inline cudaError_t once_per_device(std::atomic<unsigned long long> &done, int dev, Set set)
{
    const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    const cudaError_t e = set();
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_release);
    return e;
}

#ifdef __CUDACC__
// The kernel before this one on the stream has completed and its writes are visible (returns at once for a plain launch).
__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The kernel after this one on the stream may start its blocks as soon as every block of this grid has said so or exited.
__device__ __forceinline__ void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// All threads of a cluster meet; what each has stored before, in shared memory of any of its blocks too, is visible behind it.
__device__ __forceinline__ void cluster_sync() { asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory"); }

// Part of an attention row: maximum (log2 domain), sum of exponentials and four columns of the output, both relative to the maximum.
// Shared by the decode kernel and the forms of generation, whose results are the same bits.
struct AttnPart {
    float m, l;
    float4 o;
};
__device__ __forceinline__ void merge_part(AttnPart &a, float m2, float l2, const float4 &o2)
{
    const float mn = fmaxf(a.m, m2);
    const float a1 = ex2_approx(a.m - mn), a2 = ex2_approx(m2 - mn);
    // (the contraction written out: the compiler may choose either product for the multiply-add)
    a.l = fmaf(a.l, a1, __fmul_rn(l2, a2));
    a.o.x = fmaf(a.o.x, a1, __fmul_rn(o2.x, a2));
    a.o.y = fmaf(a.o.y, a1, __fmul_rn(o2.y, a2));
    a.o.z = fmaf(a.o.z, a1, __fmul_rn(o2.z, a2));
    a.o.w = fmaf(a.o.w, a1, __fmul_rn(o2.w, a2));
    a.m = mn;
}

// 16-byte asynchronous global -> shared copy; `valid == false` writes zeros and reads nothing.
__device__ __forceinline__ void cp_async16(void *smem_dst, const void *gmem_src, bool valid)
{
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem_src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Kernel launch wrappers (one per .cu file), all returning an HIPGPT_* status.
int launch_mha_rows(const float *q, const float *k, const float *v, float *out, float *probs,
                    int B, int S, int E, int H, int causal, int warps, cudaStream_t st);
bool mha_rows_supports(int D);
int launch_mha_tc(const float *q, const float *k, const float *v, float *out,
                  int B, int S, int E, int H, int causal, cudaStream_t st);
bool mha_tc_supports(int D);
int tc_status_fetch(int *status);
int launch_mha_tc16(const float *q, const float *k, const float *v, float *out, float *probs,
                    int B, int S, int E, int H, int causal, cudaStream_t st);
bool mha_tc16_supports(int head_dim);
int tc16_status_fetch(int *status);
void tc16_release_scratch();
// Copies `bytes` from src to each of up to seven peer addresses with plain stores (shard_push.cu).
int launch_shard_push(const void *src, void *const *dst, int ndst, size_t bytes, cudaStream_t st);
int tc16_notice_fetch(int *notice);
// whole-head kernel (head_dim 32, S <= 256): TMA loads, 128-key products, all score tiles of a head in TMEM
int launch_mha_head(const float *q, const float *k, const float *v, float *out, float *probs, int B, int S, int E, int H, int causal, cudaStream_t st);
bool mha_head_supports(int head_dim, int S, int E, const void *q, const void *k, const void *v, const void *out);
int head_status_fetch(int *status);
int head_notice_fetch(int *notice);
int probe_status_fetch(int *status);
int launch_mha_bf16(const void *q, const void *k, const void *v, void *out, int B, int S, int E, int H, int causal, cudaStream_t st,
                    int variant = 0);
bool mha_bf16_supports(int D);
int bf16_status_fetch(int *status);
// attention backward (attn_bwd.cu): scratch = 2 B H S floats (row sums w_i, then log-sum-exp of the rows)
size_t mha_backward_scratch_bytes(int B, int H, int S);
int launch_mha_backward(const float *g, const float *q, const float *k, const float *v, const float *probs,
                        float *dq, float *dk, float *dv, float *scratch, int B, int S, int E, int H, int causal, bool tensor, cudaStream_t st);
// the same on the tensor pipe, head_dim 32 / 64 (attn_bwd_tc.cu)
bool mha_backward_tc_supports(const void *g, const void *q, const void *k, const void *v, const void *probs, const void *dq, const void *dk,
                              const void *dv, int B, int S, int E, int H);
int launch_mha_backward_tc(const float *g, const float *q, const float *k, const float *v, const float *probs, float *dq, float *dk, float *dv,
                           int B, int S, int E, int H, int causal, cudaStream_t st);
int mha_backward_tc_status_fetch(int *status);
// a head whose operands fit shared memory, in one launch (attn_bwd_head.cu; the tensor pipe's conditions hold)
bool mha_backward_head_supports(int D, int S);
int launch_mha_backward_head(const float *g, const float *q, const float *k, const float *v, const float *probs, float *dq, float *dk, float *dv,
                             int B, int S, int E, int H, int causal, cudaStream_t st);
int mha_backward_head_status_fetch(int *status);
void mha_backward_tc_release();
// the launchers either side of attention (layer_ops.cu)
int launch_matmul_exact(const float *A, const float *B, const float *bias, float *C, int M, int N, int K, cudaStream_t st);
// The same product on the tensor pipe with fp32-grade (not bit-identical) results (gemm_tc.cu); its status word and scratch.
int launch_matmul_tc(const float *A, const float *B, const float *bias, float *C, int M, int N, int K, cudaStream_t st, const float *ln_g = nullptr, const float *ln_b = nullptr);
struct PackedB;                                  // a right-hand side packed once for many products
int matmul_tc_prepare(const float *B, int N, int K, PackedB **out, cudaStream_t st);
int launch_matmul_tc_prepared(const float *A, const PackedB *b, const float *bias, float *C, int M, cudaStream_t st, const float *ln_g = nullptr, const float *ln_b = nullptr);
void matmul_tc_release(PackedB *p);
int gemm_tc_status_fetch(int *status);
void gemm_tc_release_scratch();
int launch_mha_generic(const float *q, const float *k, const float *v, float *out, float *probs,
                       int B, int S, int E, int H, int causal, cudaStream_t st);
int launch_sdp(const float *Q, const float *K, float *scores, int B, int S, int D, cudaStream_t st);
int launch_softmax_rows(const float *scores, float *out, int B, int S, cudaStream_t st);
int launch_weighted_sum(const float *P, const float *V, float *out, int B, int S, int D, cudaStream_t st);
// pos_ptr (optional): device int holding ctx - 1; when given it overrides ctx inside the kernels,
// so that one captured launch serves every step of a generation loop.
int launch_decode(const float *q, const float *kc, const float *vc, float *out, float *scratch,
                  int B, int H, int D, int ctx, int cap, int nsplit, cudaStream_t st, const int *pos_ptr = nullptr);
int decode_splits(int B, int H, int D, int ctx);
// `rows` query rows, per_seq consecutive positions of each sequence, the first of which sees ctx0 keys
bool decode_rows_supports(int D, int nsplit);
int launch_decode_rows(const float *q, const float *kc, const float *vc, float *out, int rows, int per_seq, int H, int D, int ctx0, int cap, int nsplit, cudaStream_t st);

}  // namespace hipgpt
