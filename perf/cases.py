"""The work that a user of this library has it do, as cases that can be timed and compared.

Each case is one call (or, for a block of the model, one sequence of calls) through the public entry points, the
Python mirror of the launchers where it has one and the C ABI elsewhere.  Shapes are those of the benchmark's configurations
and of the tests, or lie between them.  Five kinds:

  attention   launch_multihead_attention on three stacked planes: fp32 with or without the mask and with or
              without the stored probabilities, and the bf16 form
  backward    gradients of the planes from the gradient of the output, with the stored probabilities or without
  decode      one query row per (batch, head) over a key / value cache
  block       one transformer block forward: in the reference's own sequence of launchers ("exact", the
              summation order of its matmul), or with the weights packed once and the fused forms ("packed")
  generate    greedy generation from prompts on the host to ids on the host
"""
from __future__ import annotations

import ctypes as C
import math

import torch

from hipgpt_b200 import _capi, launchers
from hipgpt_b200.generation import GptDecoder


def listed():
    return [
        # the smallest benchmark configuration: latency of one call
        dict(name="attn_small", kind="attention", B=2, H=8, S=64, D=32, causal=True, probs=False, dtype="fp32"),
        # the default model's training shape, as the benchmark times it
        dict(name="attn_train", kind="attention", B=32, H=8, S=256, D=32, causal=True, probs=False, dtype="fp32"),
        # the same shape as the reference's layer asks for it: no mask, probabilities stored for the backward
        dict(name="attn_train_probs", kind="attention", B=32, H=8, S=256, D=32, causal=False, probs=True, dtype="fp32"),
        # a longer context at head_dim 64
        dict(name="attn_long", kind="attention", B=16, H=8, S=1024, D=64, causal=True, probs=False, dtype="fp32"),
        # the scaling configuration's shape in 16-bit storage: the largest call
        dict(name="attn_bf16_large", kind="attention", B=64, H=16, S=2048, D=64, causal=True, probs=False, dtype="bf16"),
        # one layer of a training step at the default model: what the reference's layer backward calls
        dict(name="backward_train", kind="backward", B=32, H=8, S=256, D=32, causal=False, probs=True),
        # a ragged longer context whose forward stored nothing: probabilities formed again
        dict(name="backward_long", kind="backward", B=3, H=12, S=777, D=64, causal=True, probs=False),
        # a token of a small serving batch, early in its context
        dict(name="decode_small", kind="decode", B=8, H=8, D=32, ctx=77, cap=256),
        # a token of a large serving batch, late in its context
        dict(name="decode_large", kind="decode", B=64, H=16, D=64, ctx=2047, cap=2048),
        # one block of the default model at its training shape, the reference's launchers in its order
        dict(name="block_exact", kind="block", B=32, H=8, S=256, D=32, form="exact"),
        # a wider block on a ragged batch with the weights packed once
        dict(name="block_packed", kind="block", B=7, H=8, S=201, D=64, form="packed"),
        # the benchmark's generation: the default model, 8 prompts of 16 ids, 128 new tokens
        dict(name="generate", kind="generate", V=5000, S=256, E=256, L=8, H=8, B=8, n_prompt=16, n_new=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _batch_for(rng, per_batch, most, lo=1, hi=64):
    """A batch size over [lo, hi] whose whole call stays within `most` units of work."""
    return _log_int(rng, lo, max(lo, min(hi, int(most // max(per_batch, 1)))))


def draw(rng):
    kind = rng.choice(["attention", "attention", "attention", "backward", "backward", "decode", "decode", "block", "block", "generate"])
    D = rng.choice([32, 64])
    if kind == "attention":
        dtype = rng.choice(["fp32", "fp32", "fp32", "bf16"])
        D = 64 if dtype == "bf16" else D
        H, S = rng.randint(4, 16), _log_int(rng, 33, 2048)
        probs = dtype == "fp32" and rng.random() < 0.3
        # at most the largest listed call's products, and 2^27 stored probabilities
        B = _batch_for(rng, H * S * S * D, 2.7e11 if dtype == "bf16" else 7e10)
        if probs:
            B = min(B, max(1, (1 << 27) // (H * S * S)))
        return dict(kind=kind, B=B, H=H, S=S, D=D, causal=rng.random() < 0.6, probs=probs, dtype=dtype)
    if kind == "backward":
        H, S = rng.randint(4, 16), _log_int(rng, 33, 1024)
        probs = rng.random() < 0.5
        B = _batch_for(rng, H * S * S * D, 1.4e9, hi=32)
        return dict(kind=kind, B=B, H=H, S=S, D=D, causal=not probs and rng.random() < 0.7, probs=probs)
    if kind == "decode":
        H, ctx = rng.randint(4, 16), _log_int(rng, 17, 2048)
        return dict(kind=kind, B=_log_int(rng, 1, 64), H=H, D=D, ctx=ctx, cap=ctx + rng.randint(0, ctx // 4 + 1))
    if kind == "block":
        H, S = rng.randint(4, 512 // D), _log_int(rng, 33, 512)
        B = _batch_for(rng, S, 8192, hi=64)
        return dict(kind=kind, B=B, H=H, S=S, D=D, form=rng.choice(["exact", "packed"]))
    H = rng.randint(4, 384 // D)
    n_prompt = rng.randint(4, 32)
    return dict(kind=kind, V=_log_int(rng, 500, 5000), S=256, E=H * D, L=rng.randint(2, 6), H=H, B=rng.randint(1, 8), n_prompt=n_prompt,
                n_new=rng.randint(16, 128))


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, scale=1.0):
    return torch.randn(*shape, generator=g, device="cuda") * scale


def prepare(case, seed):
    g, st = _gen(seed), dict(case)
    kind = case["kind"]
    if kind == "attention":
        B, S, E = case["B"], case["S"], case["H"] * case["D"]
        st["qkv"] = _randn(g, 3, B * S, E)
        if case["dtype"] == "bf16":
            st["qkv"] = st["qkv"].bfloat16()
        st["out"] = torch.empty(B * S, E, device="cuda", dtype=st["qkv"].dtype)
        st["p"] = torch.empty(B, case["H"], S, S, device="cuda") if case["probs"] else None
    elif kind == "backward":
        B, S, H, E = case["B"], case["S"], case["H"], case["H"] * case["D"]
        st["qkv"], st["grad_out"] = _randn(g, 3, B * S, E), _randn(g, B * S, E)
        st["grad_qkv"] = torch.empty(3, B * S, E, device="cuda")
        st["p"] = None
        if case["probs"]:                                # as the forward left them
            st["p"] = torch.empty(B, H, S, S, device="cuda")
            launchers.launch_multihead_attention(st["qkv"], torch.empty(B * S, E, device="cuda"), st["p"], B, S, E, H, causal=case["causal"])
    elif kind == "decode":
        B, H, D = case["B"], case["H"], case["D"]
        st["q"], st["kc"], st["vc"] = _randn(g, B, H * D), _randn(g, B, case["cap"], H * D), _randn(g, B, case["cap"], H * D)
        st["out"] = torch.empty(B, H * D, device="cuda")
        nbytes = launchers.decode_scratch_bytes(B, H, D, case["ctx"])
        st["scratch"] = torch.empty(nbytes // 4, device="cuda") if nbytes else None
    elif kind == "block":
        _prepare_block(case, st, g)
    else:
        V, S, E, L, H = (case[k] for k in ("V", "S", "E", "L", "H"))
        F = 4 * E
        n = int(_capi.lib().hipgpt_gpt_weight_count(V, S, E, L, H, F))
        w = _randn(g, n, scale=0.02).cpu().numpy()
        st["prompts"] = torch.randint(0, V, (case["B"], case["n_prompt"]), generator=g, device="cuda", dtype=torch.int32).cpu().numpy()
        st["model"] = GptDecoder(w, V, S, E, L, H, F, max_batch=case["B"])
    return st


class _Packed:
    """A right-hand side packed once, kept for the life of the layer."""

    def __init__(self, w, N, K):
        self.h = C.c_void_p()
        _capi.check(_capi.lib().hipgpt_matmul_tc_prepare(w.data_ptr(), N, K, C.byref(self.h), torch.cuda.current_stream().cuda_stream))

    def __del__(self):
        _capi.lib().hipgpt_matmul_tc_release(self.h)


def _prepare_block(case, st, g):
    B, S, H, E = case["B"], case["S"], case["H"], case["H"] * case["D"]
    T, F = B * S, 4 * E
    st["x"] = _randn(g, T, E)
    for name, shape in (("wqkv", (E, 3 * E)), ("wo", (E, E)), ("w1", (E, F)), ("w2", (F, E))):
        st[name] = _randn(g, *shape, scale=1.0 / math.sqrt(shape[0]))
        st["b" + name[1:]] = _randn(g, shape[1], scale=0.02)
        if case["form"] == "packed":
            st["packed_" + name] = _Packed(st[name], *shape)
    for k in ("1", "2"):
        st["gamma" + k], st["beta" + k] = 1.0 + _randn(g, E, scale=0.1), _randn(g, E, scale=0.1)
    st["norm"], st["qkv"], st["att"] = torch.empty(T, E, device="cuda"), torch.empty(T, 3 * E, device="cuda"), torch.empty(T, E, device="cuda")
    st["proj"], st["mid"] = torch.empty(T, E, device="cuda"), torch.empty(T, E, device="cuda")
    st["ff"], st["y"] = torch.empty(T, F, device="cuda"), torch.empty(T, E, device="cuda")
    st["p"] = torch.empty(B, H, S, S, device="cuda") if case["form"] == "exact" else None


def run(state):
    c = state
    kind = c["kind"]
    if kind == "attention":
        B, S, H = c["B"], c["S"], c["H"]
        E = H * c["D"]
        if c["dtype"] == "bf16":
            launchers.mha_forward_bf16(c["qkv"], c["out"], B, S, E, H, causal=c["causal"])
        else:
            launchers.launch_multihead_attention(c["qkv"], c["out"], c["p"], B, S, E, H, causal=c["causal"])
        return [c["out"], c["p"]]
    if kind == "backward":
        E = c["H"] * c["D"]
        _capi.check(_capi.lib().hipgpt_mha_backward_planes(c["grad_out"].data_ptr(), c["qkv"].data_ptr(), c["p"].data_ptr() if c["p"] is not None else None,
                                                           c["grad_qkv"].data_ptr(), c["B"], c["S"], E, c["H"], int(c["causal"]),
                                                           torch.cuda.current_stream().cuda_stream))
        return [c["grad_qkv"]]
    if kind == "decode":
        launchers.mha_decode(c["q"], c["kc"], c["vc"], c["out"], c["scratch"], c["B"], c["H"], c["D"], c["ctx"], c["cap"])
        return [c["out"]]
    if kind == "block":
        return _run_block_exact(c) if c["form"] == "exact" else _run_block_packed(c)
    ids, logits, _, _ = c["model"].generate(c["prompts"], c["n_new"])
    return [ids, logits]


def _run_block_exact(c):
    """The reference's block: layer norm, projection (the output read as three stacked planes), attention, output projection,
    dropout, residual; layer norm, two matmuls with a ReLU between them, dropout, residual."""
    lib, chk, stream = _capi.lib(), _capi.check, torch.cuda.current_stream().cuda_stream
    B, S, H = c["B"], c["S"], c["H"]
    E = H * c["D"]
    T, F = B * S, 4 * E
    p = {k: v.data_ptr() for k, v in c.items() if isinstance(v, torch.Tensor)}
    chk(lib.hipgpt_layer_norm(p["x"], p["norm"], p["gamma1"], p["beta1"], T, E, stream))
    chk(lib.hipgpt_matmul(p["norm"], p["wqkv"], p["bqkv"], p["qkv"], T, E, 3 * E, stream))
    chk(lib.hipgpt_mha_forward_planes(p["qkv"], p["att"], p["p"], B, S, E, H, 0, stream))
    chk(lib.hipgpt_matmul(p["att"], p["wo"], p["bo"], p["mid"], T, E, E, stream))
    chk(lib.hipgpt_dropout(p["mid"], p["mid"], None, 0.1, T, E, stream))
    chk(lib.hipgpt_add_inplace(p["mid"], p["x"], T * E, stream))
    chk(lib.hipgpt_layer_norm(p["mid"], p["norm"], p["gamma2"], p["beta2"], T, E, stream))
    chk(lib.hipgpt_matmul(p["norm"], p["w1"], p["b1"], p["ff"], T, E, F, stream))
    chk(lib.hipgpt_relu(p["ff"], T * F, stream))
    chk(lib.hipgpt_matmul(p["ff"], p["w2"], p["b2"], p["y"], T, F, E, stream))
    chk(lib.hipgpt_dropout(p["y"], p["y"], None, 0.1, T, E, stream))
    chk(lib.hipgpt_add_inplace(p["y"], p["mid"], T * E, stream))
    return [c["y"], c["p"]]


def _run_block_packed(c):
    """The same block with the layer norms inside the projections, dropout and residual in one call and no stored probabilities."""
    lib, chk, stream = _capi.lib(), _capi.check, torch.cuda.current_stream().cuda_stream
    B, S, H = c["B"], c["S"], c["H"]
    E = H * c["D"]
    T, F = B * S, 4 * E
    p = {k: v.data_ptr() for k, v in c.items() if isinstance(v, torch.Tensor)}
    chk(lib.hipgpt_ln_matmul_tc_prepared(p["x"], p["gamma1"], p["beta1"], c["packed_wqkv"].h, p["bqkv"], p["qkv"], T, stream))
    chk(lib.hipgpt_mha_forward_planes(p["qkv"], p["att"], None, B, S, E, H, 0, stream))
    chk(lib.hipgpt_matmul_tc_prepared(p["att"], c["packed_wo"].h, p["bo"], p["proj"], T, stream))
    chk(lib.hipgpt_dropout_residual(p["proj"], p["x"], p["mid"], None, 0.1, T, E, stream))
    chk(lib.hipgpt_ln_matmul_tc_prepared(p["mid"], p["gamma2"], p["beta2"], c["packed_w1"].h, p["b1"], p["ff"], T, stream))
    chk(lib.hipgpt_relu(p["ff"], T * F, stream))
    chk(lib.hipgpt_matmul_tc_prepared(p["ff"], c["packed_w2"].h, p["b2"], p["proj"], T, stream))
    chk(lib.hipgpt_dropout_residual(p["proj"], p["mid"], p["y"], None, 0.1, T, E, stream))
    return [c["y"]]


def work(case):
    kind = case["kind"]
    if kind == "generate":
        E, L, V, B = case["E"], case["L"], case["V"], case["B"]
        steps = case["n_prompt"] + case["n_new"] - 1
        per_layer = 4 * E * E + 8 * E * E
        weights = L * per_layer + E * V
        ctx_sum = steps * (steps + 1) // 2
        # every step needs every weight once and the keys and values of its context
        return {"bytes": 4.0 * (steps * weights + 2 * L * B * E * ctx_sum),
                "flops": 2.0 * B * steps * weights + 4.0 * L * B * E * ctx_sum}
    B, H, D = case["B"], case["H"], case["D"]
    E = H * D
    if kind == "decode":
        return {"bytes": 4.0 * B * E * (2 * case["ctx"] + 2), "flops": 4.0 * B * E * case["ctx"]}
    S = case["S"]
    pairs = B * H * (S * (S + 1) // 2 if case.get("causal") else S * S)
    if kind == "attention":
        size = 2 if case["dtype"] == "bf16" else 4
        return {"bytes": float(size * 4 * B * S * E + (4 * B * H * S * S if case["probs"] else 0)), "flops": 4.0 * pairs * D}
    if kind == "backward":
        # g.V, dQ, dK, dV and, where the probabilities are formed again, Q.K
        return {"bytes": float(4 * 7 * B * S * E + (4 * B * H * S * S if case["probs"] else 0)),
                "flops": (8.0 if case["probs"] else 10.0) * pairs * D}
    # block: the input, the weights and the output once, and the probabilities where they are stored
    T, F = B * S, 4 * E
    weights = 4 * E * E + 2 * E * F
    return {"bytes": 4.0 * (2 * T * E + weights + (B * H * S * S if case["form"] == "exact" else 0)),
            "flops": 2.0 * T * weights + 4.0 * B * H * S * S * D}


def tolerance(case):
    if case.get("dtype") == "bf16":
        return {"rel": 1e-2}                             # outputs and probabilities are rounded to bf16
    if case["kind"] == "generate":
        return {"rel": 1e-5, "differ": 0.01}             # an id may turn where two logits are equal to rounding
    return {"rel": 1e-5}                                 # 32-bit sums
