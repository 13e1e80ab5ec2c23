// Greedy generation by clusters of sixteen blocks (gpt_cluster.cu): what the driver in gpt_decode.cu hands over, and the cut of the
// matrices, which host and kernel share.
#pragma once

#include "attn_common.cuh"

namespace hipgpt {

constexpr int kClusterBlocks = 16;
constexpr long long kClusterWaitCycles = 1LL << 31;    // about a second
constexpr int kHopRecords = 1;                         // the attention records among the kernel's hops

// One matrix of the model, cut for the sixteen blocks: block c owns columns [c * nc, (c + 1) * nc) in parts of `width` columns, and
// reads a part in chunks of 2^seg_shift of the sixteen segments of the inner dimension.  A segment of a part lies as
// [klp / 4][width][4]: four consecutive inner indices of a column side by side (klp: klen rounded up to a multiple of 4; what is
// past the matrix is zero).  After the weights a chunk carries gamma and beta of its segments (where a layer norm precedes the
// product) and the part's bias.
// Where the block already has a segment of the inner dimension (`per` > 0: the second matrix of the feed-forward, whose segments are the
// blocks' columns of the first) it owns that segment for all columns: chunks of `width` columns, [klen / 4][width][4], `per` to a part, each
// with the bias of the nc columns whose partial sums this block adds up.
struct ClusterJob {
    int n, nc, width, parts, klen, klp, seg_shift, ln, per;
    __host__ __device__ constexpr int chunks() const { return per ? per : 16 >> seg_shift; }
    __host__ __device__ constexpr int weight_floats() const { return per ? klen * width : (klp * width) << seg_shift; }
    __host__ __device__ constexpr int ln_floats() const { return ln ? (2 * klp) << seg_shift : 0; }
    __host__ __device__ constexpr int chunk_bytes() const { return 4 * (weight_floats() + ln_floats() + (per ? nc : width)); }
};
enum { kJobQkv, kJobO, kJobF1, kJobF2, kJobVoc, kJobs };

// Columns n, inner dimension k.  A part is at most 64 columns and 72 KB of weights: two parts fit the ring.
__host__ __device__ constexpr ClusterJob cluster_job(int n, int k, int ln)
{
    ClusterJob j = {};
    j.n = n;
    j.nc = 4 * ((n + 63) / 64);
    j.klen = k / 16;
    j.klp = (j.klen + 3) & ~3;
    j.ln = ln;
    j.width = j.nc < 64 ? j.nc : 64;
    while (j.width > 4 && j.width * j.klp * 64 > 72 * 1024) j.width = j.width > 32 ? 32 : j.width > 16 ? 16 : j.width / 2 & ~3;
    if (j.width < 4) j.width = 4;
    j.parts = (j.nc + j.width - 1) / j.width;
    j.seg_shift = 4;
    while (j.seg_shift > 1 && j.chunk_bytes() > 18 * 1024) --j.seg_shift;
    return j;
}
// The same, a segment per block.  64 columns to a chunk where that is at most 16 KB; at most eight chunks to a part.
__host__ __device__ constexpr ClusterJob cluster_job_by_segment(int n, int k)
{
    ClusterJob j = {};
    j.n = n;
    j.nc = 4 * ((n + 63) / 64);
    j.klen = j.klp = k / 16;
    j.width = j.klen <= 64 ? 64 : 32;
    const int total = (n + j.width - 1) / j.width;
    j.parts = total > 8 ? 2 : 1;
    j.per = (total + j.parts - 1) / j.parts;
    return j;
}
__host__ __device__ constexpr ClusterJob cluster_job_of(int i, int E, int V)
{
    return i == kJobQkv ? cluster_job(3 * E, E, 1) : i == kJobO ? cluster_job(E, E, 0) : i == kJobF1 ? cluster_job(4 * E, E, 1) : i == kJobF2 ? cluster_job_by_segment(E, 4 * E)
                                                                                                                          : cluster_job(V, E, 0);
}
// Columns of the second feed-forward product whose partial sums come to block `rank`.  Shares are whole fours, so the last blocks may have none
// (E = 160, 224: two of them; 288, 352: one).  Such a block takes no part in that hop: a phase that expects no bytes is complete when it is
// opened, and who tests for it after the next one has been opened sees neither.
__host__ __device__ constexpr int cluster_f2_columns(int E, int rank)
{
    const int nc = cluster_job_of(kJobF2, E, 16).nc, left = E - rank * nc;
    return left < 0 ? 0 : left < nc ? left : nc;
}

struct ClusterPlan {
    ClusterJob voc;
    size_t block_bytes;          // a block's share of all weights, in the order in which a step reads it
    int layer_chunks, all_chunks;          // chunks of a step: its layers, and with the output projection
    int clusters_most;           // clusters that run at the same time
    bool ok;
};

struct ClusterArgs {
    const float *tok, *pos;
    const uint8_t *stream;       // [16][block_bytes]
    const uint2 *table;          // [all_chunks]: offset in the block's share and bytes of every chunk of a step
    float *kc, *vc;              // [L][max_batch][S][E]
    size_t layer_stride;
    float *logits;
    int *ids, *out_ids, *err;
    const int *prompts;
    int V, S, L, H, B, n_prompt, n_new, ns;
    int p0, nsteps;              // first position, number of positions
    long long wait_cycles;       // limit of a wait
    int expire_hop;              // test hook: the hop whose wait runs out at once in the first block, -1: none
};

struct ClusterLayerWeights { const float *wqkv, *wo, *w1, *w2, *bqkv, *bo, *b1, *b2, *g1, *be1, *g2, *be2; };

// The plan of a model; ok = false where the kernel does not take its shape.
ClusterPlan cluster_plan(int V, int S, int E, int L, int H, int F);
// Lays the weights (checkpoint order, device memory) out as the blocks' shares: dst [16][plan.block_bytes]; and the chunk table.
int cluster_pack(const ClusterPlan &p, int E, const ClusterLayerWeights *layers, int L, const float *wout, uint8_t *dst, cudaStream_t st);
void cluster_table(const ClusterPlan &p, int E, int L, uint2 *table);
// Sequences per cluster for a batch with contexts of up to `positions`, 0 where the launches are to run.
int cluster_rows(const ClusterPlan &p, int B, int E, int H, int ns, int positions);
int launch_cluster_steps(const ClusterPlan &p, const ClusterArgs &a, int E, int rows, cudaStream_t st);

}  // namespace hipgpt
