"""Greedy KV-cache generation: the CPU oracle against plain numpy on a tiny model (CPU), and the
GPU driver against the oracle: token ids must be identical, logits within 1e-4."""
import os
import subprocess

import numpy as np
import pytest

from hipgpt_b200 import synth
from oracle import bindings as ob


def _numpy_generate(w, V, S, E, L, H, F, prompts, n_new, margins=None):
    """Independent float64 restatement: full causal recompute per step, no cache."""
    D = E // H
    off = 0

    def take(*shape):
        nonlocal off
        n = int(np.prod(shape))
        a = w[off:off + n].astype(np.float64).reshape(shape)
        off += n
        return a
    tok, pos = take(V, E), take(S, E)
    layers = []
    for _ in range(L):
        layers.append(dict(wqkv=take(E, 3 * E), wo=take(E, E), w1=take(E, F), w2=take(F, E), bqkv=take(3 * E), bo=take(E),
                           b1=take(F), b2=take(E), g1=take(E), be1=take(E), g2=take(E), be2=take(E)))
    wout = take(E, V)

    def ln(x, g, b):
        m = x.mean(-1, keepdims=True)
        v = ((x - m) ** 2).mean(-1, keepdims=True)
        return g * (x - m) / np.sqrt(v + 1e-5) + b
    out = np.zeros((prompts.shape[0], n_new), dtype=np.int64)
    for bi, prm in enumerate(prompts):
        seq = list(prm)
        for i in range(n_new):
            T = len(seq)
            x = tok[seq] + pos[:T]
            for lw in layers:
                h = ln(x, lw["g1"], lw["be1"])
                qkv = h @ lw["wqkv"] + lw["bqkv"]
                q, k, v = (qkv[:, j * E:(j + 1) * E].reshape(T, H, D).transpose(1, 0, 2) for j in range(3))
                s = q @ k.transpose(0, 2, 1) / np.sqrt(D)
                s = np.where(np.tril(np.ones((T, T), bool)), s, -np.inf)
                p = np.exp(s - s.max(-1, keepdims=True))
                p /= p.sum(-1, keepdims=True)
                a = (p @ v).transpose(1, 0, 2).reshape(T, E)
                x = x + a @ lw["wo"] + lw["bo"]
                h = ln(x, lw["g2"], lw["be2"])
                x = x + np.maximum(h @ lw["w1"] + lw["b1"], 0) @ lw["w2"] + lw["b2"]
            logits = x[-1] @ wout
            nxt = int(np.argmax(logits))
            out[bi, i] = nxt
            if margins is not None:
                top2 = np.partition(logits, -2)[-2:]
                margins.append(float(top2[1] - top2[0]))
            seq.append(nxt)
    return out


def test_oracle_generation_matches_numpy_on_a_tiny_model():
    cfg = dict(V=50, S=24, E=32, L=2, H=4, F=64)
    w = synth.gpt_weights(9, **cfg, std=0.3)          # wide weights: logits well separated
    assert w.size == ob.gpt_weight_count(**cfg)
    prompts = synth.token_ids(9, (3, 5), cfg["V"])
    for fma in (False, True):
        ids, logits = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=12, fma=fma)
        assert np.array_equal(ids, _numpy_generate(w, **cfg, prompts=prompts, n_new=12))
        assert np.isfinite(logits).all()


def test_oracle_generation_matches_numpy_on_the_default_model():
    """The benchmark's whole generation case (E=256 L=8 H=8 F=1024 V=5000 S=256, weights N(0, 0.02) seed 3, 8 prompts
    of 16 ids, 128 new tokens): all 1024 ids of the fp32 oracle against float64 arithmetic that shares nothing with it,
    with the gap between the two largest logits of every step: the room an fp32 rounding difference (about 1e-6 here)
    has before it changes an id.  Measured: smallest gap 2.9e-5, 4 steps below 1e-4, median 2.4e-2."""
    cfg = dict(synth.GPT_DEFAULT)
    w = synth.gpt_weights(3, **cfg)
    prompts = synth.token_ids(3, (8, 16), cfg["V"])
    n_new = 128
    margins = []
    want = _numpy_generate(w, **cfg, prompts=prompts, n_new=n_new, margins=margins)
    ids, _ = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=n_new, fma=True)
    assert len(margins) == 1024 and min(margins) > 1e-5, f"a step of this seed is decided by {min(margins):.2e}: below fp32 noise"
    assert np.array_equal(ids, want)


def test_oracle_rejects_requests_past_the_position_table():
    cfg = dict(V=50, S=8, E=32, L=1, H=4, F=64)
    w = synth.gpt_weights(1, **cfg)
    with pytest.raises(ValueError):
        ob.gpt_generate(w, **cfg, prompts=np.zeros((1, 5), np.int32), n_new=5)     # 5 + 5 - 1 > 8


@pytest.mark.gpu
@pytest.mark.parametrize("mode", ["persistent", "graph"])
@pytest.mark.parametrize("shape", ["tiny", "default"])
def test_gpu_generation_ids_equal_the_oracle(shape, mode):
    pytest.importorskip("torch")
    from hipgpt_b200 import generation
    if shape == "tiny":
        cfg, B, n_prompt, n_new, seed = dict(V=50, S=24, E=32, L=2, H=4, F=64), 3, 5, 12, 9
    else:
        cfg, B, n_prompt, n_new, seed = dict(synth.GPT_DEFAULT), 8, 16, 128, 3      # the benchmark's whole-model case
    w = synth.gpt_weights(seed, **cfg)
    prompts = synth.token_ids(seed, (B, n_prompt), cfg["V"])
    ref_ids, ref_logits = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=n_new, fma=True)
    dec = generation.GptDecoder(w, **cfg, max_batch=B,
                                mode=generation.MODE_PERSISTENT if mode == "persistent" else generation.MODE_GRAPH)
    ids, logits, ms_prompt, ms_decode = dec.generate(prompts, n_new)
    dec.close()
    if not np.array_equal(ids, ref_ids):
        b, i = np.argwhere(ids != ref_ids)[0]
        pytest.fail(f"first differing id at prompt {b}, step {i}: gpu {ids[b, i]} oracle {ref_ids[b, i]}")
    assert float(np.abs(logits - ref_logits).max()) <= 1e-4
    assert ms_prompt > 0 and ms_decode > 0


@pytest.mark.gpu
def test_gpu_generation_forms_agree_and_a_handle_serves_many_requests():
    """The persistent kernel and the replayed graph run the same arithmetic; one handle answers
    requests of different batch sizes and lengths in either form, in any order (the grid barrier's
    generation word and the position word carry over from call to call)."""
    pytest.importorskip("torch")
    from hipgpt_b200 import generation
    cfg = dict(V=300, S=48, E=64, L=3, H=2, F=128)          # head_dim 32
    w = synth.gpt_weights(21, **cfg)
    dec = generation.GptDecoder(w, **cfg, max_batch=5)
    for B, n_prompt, n_new in [(5, 4, 20), (2, 7, 1), (1, 1, 48), (3, 10, 30)]:
        prompts = synth.token_ids(100 + B, (B, n_prompt), cfg["V"])
        ref_ids, ref_logits = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=n_new, fma=True)
        got = {}
        for mode in (generation.MODE_PERSISTENT, generation.MODE_GRAPH, generation.MODE_PERSISTENT):
            dec.set_mode(mode)
            ids, logits, _, _ = dec.generate(prompts, n_new)
            assert np.array_equal(ids, ref_ids)
            assert float(np.abs(logits - ref_logits).max()) <= 1e-4
            got[mode] = logits
        assert float(np.abs(got[generation.MODE_PERSISTENT] - got[generation.MODE_GRAPH]).max()) <= 1e-5
    dec.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cfg,B,n_prompt,n_new", [
    (dict(V=131, S=40, E=128, L=2, H=4, F=512), 1, 3, 20),          # one cluster, fewer columns than blocks times four
    (dict(V=777, S=64, E=160, L=2, H=5, F=640), 3, 1, 30),          # segments of 10 inner indices: padded
    (dict(V=1000, S=300, E=256, L=1, H=4, F=1024), 9, 5, 40),       # head_dim 64, two sequences per cluster, one left over
    (dict(V=1371, S=96, E=384, L=1, H=12, F=1536), 2, 4, 24),       # products in several parts
    (dict(V=150, S=40, E=224, L=2, H=7, F=896), 3, 2, 12),          # a chunk of the second feed-forward matrix half past its columns
    (dict(V=150, S=40, E=288, L=2, H=9, F=1152), 9, 2, 12),         # ... and one wholly, in the second of two parts; two sequences per cluster
    (dict(V=300, S=700, E=128, L=1, H=2, F=512), 2, 300, 60),       # contexts of more rows than a lane asks for ahead
    (dict(V=200, S=2100, E=128, L=1, H=4, F=512), 2, 2060, 40),     # a long context, several rounds of a unit
    (dict(V=200, S=40, E=128, L=1, H=4, F=512), 15, 2, 10),         # a batch for the replayed graph
    (dict(V=200, S=40, E=128, L=1, H=4, F=256), 2, 2, 10)])         # a feed-forward width for the replayed graph
def test_gpu_generation_by_clusters_at_its_edges(cfg, B, n_prompt, n_new):
    pytest.importorskip("torch")
    from hipgpt_b200 import generation
    w = synth.gpt_weights(31, **cfg, std=0.08)
    prompts = synth.token_ids(32, (B, n_prompt), cfg["V"])
    ref_ids, ref_logits = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=n_new, fma=True)
    dec = generation.GptDecoder(w, **cfg, max_batch=B)
    for _ in range(2):
        ids, logits, _, _ = dec.generate(prompts, n_new)
        assert np.array_equal(ids, ref_ids)
        assert float(np.abs(logits - ref_logits).max()) <= 1e-4
    dec.close()


_F2_HOP = r"""
#include "gpt_cluster.cuh"
#include <cstdio>
using namespace hipgpt;
// A barrier of one arrival: the phase it is in, complete once it has been opened and the bytes it expects have come.
struct Barrier {
    int phase = 0, bytes = 0;
    bool opened = false;
    void open(int expect) { opened = true; bytes += expect; settle(); }
    void come(int n) { bytes -= n; settle(); }
    void settle() { if (opened && bytes == 0) { ++phase; opened = false; } }
    bool test(int parity) const { return (phase & 1) != parity; }
};
int main()
{
    int bad = 0;
    for (int E = 128; E <= 384; E += 32)
        for (int rank = 0; rank < kClusterBlocks; ++rank) {
            const int own = cluster_f2_columns(E, rank);
            const bool waits = HIPGPT_TEST_WAITS;
            Barrier b;
            if (waits) b.open(64 * own);
            for (int layer = 0; layer < 6 && waits; ++layer) {
                b.come(64 * own);                    // the sixteen blocks' partial sums
                // the last warp comes first: it sees its phase and opens the next one
                bad += !b.test(layer & 1);
                b.open(64 * own);
                bad += !b.test(layer & 1);           // a warp that adds up, after it
            }
            if (!waits && own) ++bad;
        }
    std::printf("%d\n", bad);
}
"""


@pytest.mark.parametrize("waits,ok", [("own > 0", True), ("true", False)])
def test_generation_by_clusters_no_block_waits_for_sums_that_nobody_sends(tmp_path, waits, ok):
    """The second feed-forward product's hop with the last warp ahead of those that add up: blocks with columns see their phase whatever the order; a
    block without would look for one that has come and gone (which is why it stays out of the hop)."""
    from hipgpt_b200 import build
    src, exe = tmp_path / "hop.cu", tmp_path / "hop"
    src.write_text(_F2_HOP)
    subprocess.run([build.nvcc(), *build.ARCH, "-std=c++17", f"-DHIPGPT_TEST_WAITS=({waits})", "-I", build.CSRC, "-I", os.path.join(build.ROOT, "include"), str(src), "-o", str(exe)], check=True)
    assert (int(subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout) == 0) is ok


@pytest.mark.gpu
@pytest.mark.parametrize("E,B", [(160, 1), (160, 9), (224, 9), (288, 1), (352, 2), (352, 9)])
def test_gpu_generation_by_clusters_with_blocks_that_own_no_columns(E, B):
    """Widths whose last blocks have no column of the second feed-forward product, one sequence per cluster and two, many layers and positions."""
    pytest.importorskip("torch")
    from hipgpt_b200 import generation
    cfg = dict(V=200, S=72, E=E, L=5, H=E // 32, F=4 * E)
    w = synth.gpt_weights(41, **cfg, std=0.05)
    prompts = synth.token_ids(42, (B, 3), cfg["V"])
    ref_ids, ref_logits = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=64, fma=True)
    dec = generation.GptDecoder(w, **cfg, max_batch=B)
    for _ in range(4):
        ids, logits, _, _ = dec.generate(prompts, 64)
        assert np.array_equal(ids, ref_ids)
        assert float(np.abs(logits - ref_logits).max()) <= 1e-4
    dec.close()


@pytest.mark.gpu
def test_gpu_generation_by_clusters_ends_where_the_graph_is_ahead():
    """Few sequences with long contexts, and batches that do not fit, replay the graph."""
    pytest.importorskip("torch")
    from hipgpt_b200 import _capi, generation
    cfg = dict(V=64, S=32768, E=256, L=1, H=8, F=1024)
    dec = generation.GptDecoder(synth.gpt_weights(5, **cfg), **cfg, max_batch=64)
    rows = lambda B, positions: _capi.lib().hipgpt_gpt_debug_cluster_rows(dec._h, B, positions)      # noqa: E731
    assert [rows(2, n) for n in (1, 16384, 24576, 24577, 32768)] == [1, 1, 1, 0, 0]
    most = next(b for b in range(2, 65) if rows(b, 100) != 1) - 1
    assert rows(most, 32768) == 1 and rows(2 * most, 32768) == 2 and rows(2 * most + 1, 100) == 0
    assert rows(most + 1, 24576) == 2 and rows(most + 1, 32768) == (2 if (most + 2) // 2 * 3 >= 16 else 0)
    assert rows(0, 5) == _capi.ERR_BAD_ARG and rows(65, 5) == _capi.ERR_BAD_ARG and rows(1, 32769) == _capi.ERR_BAD_ARG
    dec.close()


@pytest.mark.gpu
def test_gpu_generation_lays_the_weights_out_again_only_for_batches_that_use_it():
    torch = pytest.importorskip("torch")
    from hipgpt_b200 import generation
    cfg = dict(V=5000, S=64, E=256, L=4, H=8, F=1024)
    w = synth.gpt_weights(6, **cfg)
    weights = 4 * (12 * cfg["L"] * cfg["E"] ** 2 + cfg["E"] * cfg["V"])
    prompts = {B: synth.token_ids(7, (B, 3), cfg["V"]) for B in (4, 40)}
    free = lambda: torch.cuda.mem_get_info()[0]              # noqa: E731

    def used(max_batch, *batches):
        """Device memory that each batch's first request takes, and the ids."""
        dec, out, ids = generation.GptDecoder(w, **cfg, max_batch=max_batch), [], []
        for B in batches:
            before = free()
            ids.append(dec.generate(prompts[B], 5)[0])
            out.append(before - free())
        dec.close()
        return out, ids
    used(64, 4, 40)                                          # the kernels are loaded
    (large, small), ids = used(64, 40, 4)
    assert large < weights // 2 and small >= weights
    (at_once,), again = used(4, 4)
    assert at_once < weights // 2 and np.array_equal(ids[1], again[0]) and np.array_equal(ids[1], ids[0][:4])


@pytest.mark.gpu
def test_gpu_generation_handles_of_different_widths_side_by_side():
    """A narrower model's handle does not take shared memory away from a wider one's kernels."""
    pytest.importorskip("torch")
    from hipgpt_b200 import generation
    wide, narrow = dict(V=90, S=24, E=64, L=1, H=2, F=4096), dict(V=90, S=24, E=64, L=1, H=2, F=1600)
    w = synth.gpt_weights(41, **wide)
    prompts = synth.token_ids(42, (2, 3), wide["V"])
    want, _ = ob.gpt_generate(w, **wide, prompts=prompts, n_new=6, fma=True)
    a = generation.GptDecoder(w, **wide, max_batch=2)
    b = generation.GptDecoder(synth.gpt_weights(43, **narrow), **narrow, max_batch=2)
    for mode in (generation.MODE_GRAPH, generation.MODE_PERSISTENT):
        a.set_mode(mode)
        assert np.array_equal(a.generate(prompts, 6)[0], want)
    a.close()
    b.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cfg,B,n_prompt,n_new", [
    (dict(V=90, S=24, E=64, L=2, H=4, F=128), 3, 5, 6),             # head_dim 16, one split
    (dict(V=90, S=24, E=128, L=2, H=4, F=512), 3, 5, 6),            # clusters: as few positions as are taken together there
    (dict(V=90, S=160, E=128, L=2, H=1, F=256), 2, 150, 4),         # head_dim 128, splits of more keys than a block's lanes hold
    (dict(V=300, S=300, E=320, L=2, H=5, F=1280), 7, 80, 5),        # clusters; more rows than fit at a time
    (dict(V=90, S=40, E=60 * 16, L=1, H=12, F=960), 1, 33, 3),      # head_dim 80
    (dict(V=90, S=40, E=60 * 16, L=2, H=12, F=960), 2, 2, 5)])      # the graph: a single position
def test_gpu_generation_takes_the_positions_of_a_prompt_together(cfg, B, n_prompt, n_new):
    pytest.importorskip("torch")
    from hipgpt_b200 import generation
    w = synth.gpt_weights(51, **cfg, std=0.08)
    prompts = synth.token_ids(52, (B, n_prompt), cfg["V"])
    ref_ids, ref_logits = ob.gpt_generate(w, **cfg, prompts=prompts, n_new=n_new, fma=True)
    dec = generation.GptDecoder(w, **cfg, max_batch=B)
    for n in (n_prompt, 4, n_prompt):                                # (the steps in between, on the same handle)
        ids, logits, _, _ = dec.generate(prompts[:, :n], n_new)
        if n == n_prompt:
            assert np.array_equal(ids, ref_ids)
            assert float(np.abs(logits - ref_logits).max()) <= 1e-4
    dec.close()
