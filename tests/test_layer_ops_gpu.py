"""GPU parity tests of the launchers either side of attention in HipGPT's layer and model forward
(projections, layer norm, dropout, residual add, ReLU, embedding lookup), of the attention backward, and of
HipGPT's own TransformerLayer / GPTModel classes running on this library (oracle/_ref/ref_model_run, built
where the HipGPT tree is mounted).  Integer and order-preserving arithmetic is held to bit equality with the
CPU oracle; the rest to the stated tolerances."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from hipgpt_b200 import _capi, checkpoint, synth
from oracle import bindings as ob

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from tests.gpu_util import dev  # noqa: E402

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
REF_RUN = os.path.join(ROOT, "oracle", "_ref", "ref_model_run")


def _st():
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("M,N,K,bias", [(300, 256, 768, True), (64, 1024, 256, True), (257, 256, 1024, False), (130, 64, 5000, False),
                                        (33, 100, 20, True), (5, 7, 3, False), (1, 256, 256, True)])
def test_matmul_is_bit_identical_to_the_reference_order(M, N, K, bias):
    lib = _capi.lib()
    A, W = synth.normal(1, (M, N)), synth.normal(2, (N, K), 0.1)
    b = synth.normal(3, (K,)) if bias else None
    want = ob.matmul(A, W, b, M, N, K, fma=True)
    dA, dW, dC = dev(A), dev(W), torch.full((M, K), float("nan"), device="cuda")
    db = dev(b) if bias else None
    _capi.check(lib.hipgpt_matmul(dA.data_ptr(), dW.data_ptr(), db.data_ptr() if bias else None, dC.data_ptr(), M, N, K, _st()))
    torch.cuda.synchronize()
    assert np.array_equal(dC.cpu().numpy(), want)


@pytest.mark.parametrize("M,K", [(8903, 388), (7123, 388), (6222, 388), (4747, 132), (4194, 132), (3556, 132), (5922, 68), (4739, 4), (1805, 132),
                                 (2374, 68), (2371, 4), (1, 20)])
def test_matmul_tiles_are_bit_identical_to_the_reference_order(M, K):
    """One shape for every tile the exact matmul chooses from, with rows and columns left over, an inner dimension that is no
    multiple of a tile's depth, and (for 256 columns at most) the same product in place."""
    lib = _capi.lib()
    N = 36
    A, W, b = synth.normal(4, (M, N)), synth.normal(5, (N, K), 0.1), synth.normal(6, (K,))
    want = ob.matmul(A, W, b, M, N, K, fma=True)
    dA, dW, db, dC = dev(A), dev(W), dev(b), torch.full((M, K), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_matmul(dA.data_ptr(), dW.data_ptr(), db.data_ptr(), dC.data_ptr(), M, N, K, _st()))
    torch.cuda.synchronize()
    assert np.array_equal(dC.cpu().numpy(), want)
    if K <= 256:                                        # square in place
        W2 = synth.normal(7, (K, K), 0.1)
        A2 = synth.normal(8, (M, K))
        want = ob.matmul(A2, W2, b, M, K, K, fma=True)
        dA2, dW2 = dev(A2), dev(W2)
        _capi.check(lib.hipgpt_matmul(dA2.data_ptr(), dW2.data_ptr(), db.data_ptr(), dA2.data_ptr(), M, K, K, _st()))
        torch.cuda.synchronize()
        assert np.array_equal(dA2.cpu().numpy(), want)


@pytest.mark.parametrize("M,K", [(1002, 388), (1249, 388), (664, 388), (495, 388), (157, 388), (79, 388), (2965, 132), (2393, 20), (1795, 20), (1210, 20), (612, 20), (14, 20)])
def test_matmul_small_tiles_are_bit_identical_to_the_reference_order(M, K):
    """One shape for each of the tiles of small products, with rows and columns left over and several stages of an inner dimension that is no multiple of
    one; and, where a block has whole rows, in place."""
    lib = _capi.lib()
    N = 300
    A, W, b = synth.normal(14, (M, N)), synth.normal(15, (N, K), 0.1), synth.normal(16, (K,))
    want = ob.matmul(A, W, b, M, N, K, fma=True)
    dA, dW, db, dC = dev(A), dev(W), dev(b), torch.full((M, K), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_matmul(dA.data_ptr(), dW.data_ptr(), db.data_ptr(), dC.data_ptr(), M, N, K, _st()))
    torch.cuda.synchronize()
    assert np.array_equal(dC.cpu().numpy(), want)
    if K <= 64:
        W2, A2 = synth.normal(17, (K, K), 0.1), synth.normal(18, (M, K))
        want = ob.matmul(A2, W2, b, M, K, K, fma=True)
        dA2, dW2 = dev(A2), dev(W2)
        _capi.check(lib.hipgpt_matmul(dA2.data_ptr(), dW2.data_ptr(), db.data_ptr(), dA2.data_ptr(), M, K, K, _st()))
        torch.cuda.synchronize()
        assert np.array_equal(dA2.cpu().numpy(), want)


@pytest.mark.parametrize("M,N,K", [(2400, 52, 132), (1800, 44, 20), (1249, 300, 388), (16353, 52, 28), (40114, 48, 8), (9000, 16, 16)])
def test_matmul_of_many_rows_and_few_inner_indices_is_bit_identical_to_the_reference_order(M, N, K):
    """The tiles of short stages, with inner dimensions of less than the stages hold and with rows and columns left over; the last in place too."""
    lib = _capi.lib()
    A, W, b = synth.normal(24, (M, N)), synth.normal(25, (N, K), 0.1), synth.normal(26, (K,))
    want = ob.matmul(A, W, b, M, N, K, fma=True)
    dA, dW, db, dC = dev(A), dev(W), dev(b), torch.full((M, K), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_matmul(dA.data_ptr(), dW.data_ptr(), db.data_ptr(), dC.data_ptr(), M, N, K, _st()))
    torch.cuda.synchronize()
    assert np.array_equal(dC.cpu().numpy(), want)
    if N == K:
        _capi.check(lib.hipgpt_matmul(dA.data_ptr(), dW.data_ptr(), db.data_ptr(), dA.data_ptr(), M, N, K, _st()))
        torch.cuda.synchronize()
        assert np.array_equal(dA.cpu().numpy(), want)


@pytest.mark.parametrize("M,N,K,bias", [(8192, 256, 768, True), (300, 256, 768, True), (64, 1024, 256, True), (257, 256, 1024, False), (130, 64, 5000, False),
                                        (33, 100, 20, True), (5, 7, 3, False), (1, 256, 256, True), (129, 65, 129, True),
                                        (1407, 512, 509, True), (1407, 2048, 512, False), (700, 330, 260, True),     # slices of a tile on 2, 3 and 3 blocks
                                        (1152, 512, 510, True), (1408, 520, 384, False),         # 36 and 33 tiles: as many clusters of four as fit, or fewer
                                        (4700, 520, 256, True), (4700, 260, 256, False), (4750, 520, 250, False)])    # 74 tiles: all the pairs there are, one block each; 76
def test_tensor_core_matmul_is_fp32_grade(M, N, K, bias):
    """hipgpt_matmul_tc: the projections on the tensor pipe.  Not the reference's summation order, so not its bits: the
    bar is 1e-5 relative to the largest output against a float64 product (the exact-order kernel's own distance from
    float64 on these shapes is ~1e-6), for unit-scale operands and for operands far outside fp16's range."""
    lib = _capi.lib()
    for sa, sw in ((1.0, 0.1), (1e6, 1e-9), (3e-7, 2e4)):
        A, W = synth.normal(1, (M, N)) * np.float32(sa), synth.normal(2, (N, K)) * np.float32(sw)
        b = (synth.normal(3, (K,)) * np.float32(sa * sw)) if bias else None
        want = A.astype(np.float64) @ W.astype(np.float64) + (b.astype(np.float64) if bias else 0.0)
        dA, dW, dC = dev(A), dev(W), torch.full((M, K), float("nan"), device="cuda")
        db = dev(b) if bias else None
        _capi.check(lib.hipgpt_matmul_tc(dA.data_ptr(), dW.data_ptr(), db.data_ptr() if bias else None, dC.data_ptr(), M, N, K, _st()))
        torch.cuda.synchronize()
        st = C.c_int(-1)
        _capi.check(lib.hipgpt_kernel_status(C.byref(st)))
        assert st.value == 0
        got = dC.cpu().numpy().astype(np.float64)
        assert np.isfinite(got).all()
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max(), (sa, sw)
    # in place is refused (the exact kernel supports it)
    sq = torch.zeros((64, 64), device="cuda")
    assert lib.hipgpt_matmul_tc(sq.data_ptr(), sq.data_ptr(), None, sq.data_ptr(), 64, 64, 64, _st()) == _capi.ERR_UNSUPPORTED


def test_tensor_core_matmul_with_weights_packed_once():
    """hipgpt_matmul_tc_prepare / _prepared: the right-hand side packed once gives the bits of the one-call form, for any
    number of left-hand sides, also after the original weights have been overwritten."""
    lib = _capi.lib()
    N, K = 256, 768
    W, b = synth.normal(12, (N, K), 0.05), synth.normal(13, (K,))
    dW, db = dev(W), dev(b)
    h = C.c_void_p()
    _capi.check(lib.hipgpt_matmul_tc_prepare(dW.data_ptr(), N, K, C.byref(h), _st()))
    torch.cuda.synchronize()
    dW2 = dW.clone()
    dW.fill_(float("nan"))                              # the packed form does not refer to the original
    for M in (1, 130, 1000):
        A = synth.normal(14 + M, (M, N))
        dA = dev(A)
        c1 = torch.full((M, K), float("nan"), device="cuda")
        c2 = torch.full((M, K), float("nan"), device="cuda")
        _capi.check(lib.hipgpt_matmul_tc_prepared(dA.data_ptr(), h, db.data_ptr(), c1.data_ptr(), M, _st()))
        _capi.check(lib.hipgpt_matmul_tc(dA.data_ptr(), dW2.data_ptr(), db.data_ptr(), c2.data_ptr(), M, N, K, _st()))
        torch.cuda.synchronize()
        assert torch.equal(c1, c2)
        want = A.astype(np.float64) @ W.astype(np.float64) + b.astype(np.float64)
        assert np.abs(c1.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
    lib.hipgpt_matmul_tc_release(h)


@pytest.mark.parametrize("M,N,K", [(8192, 256, 768), (130, 100, 136), (5, 64, 7)])
def test_layer_norm_fused_into_the_tensor_core_projection(M, N, K):
    """hipgpt_ln_matmul_tc(_prepared): LayerNorm(A) B + bias against a float64 restatement (mean, variance / N, eps 1e-5)."""
    lib = _capi.lib()
    A, W = synth.normal(30, (M, N)) * np.float32(3.0) + np.float32(0.5), synth.normal(31, (N, K), 0.1)
    g, be, b = synth.normal(32, (N,)) * np.float32(0.2) + np.float32(1.0), synth.normal(33, (N,), 0.1), synth.normal(34, (K,))
    a64 = A.astype(np.float64)
    mu, var = a64.mean(axis=1, keepdims=True), a64.var(axis=1, keepdims=True)
    ln = g.astype(np.float64) * (a64 - mu) / np.sqrt(var + 1e-5) + be.astype(np.float64)
    want = ln @ W.astype(np.float64) + b.astype(np.float64)
    dA, dW, dg, dbe, db = dev(A), dev(W), dev(g), dev(be), dev(b)
    c1 = torch.full((M, K), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_ln_matmul_tc(dA.data_ptr(), dg.data_ptr(), dbe.data_ptr(), dW.data_ptr(), db.data_ptr(), c1.data_ptr(), M, N, K, _st()))
    h = C.c_void_p()
    _capi.check(lib.hipgpt_matmul_tc_prepare(dW.data_ptr(), N, K, C.byref(h), _st()))
    c2 = torch.full((M, K), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_ln_matmul_tc_prepared(dA.data_ptr(), dg.data_ptr(), dbe.data_ptr(), h, db.data_ptr(), c2.data_ptr(), M, _st()))
    torch.cuda.synchronize()
    lib.hipgpt_matmul_tc_release(h)
    assert torch.equal(c1, c2)
    assert np.abs(c1.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()
    # and against the separate launchers of this library: hipgpt_layer_norm, then the product
    y = torch.empty_like(dA)
    _capi.check(lib.hipgpt_layer_norm(dA.data_ptr(), y.data_ptr(), dg.data_ptr(), dbe.data_ptr(), M, N, _st()))
    c3 = torch.full((M, K), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_matmul_tc(y.data_ptr(), dW.data_ptr(), db.data_ptr(), c3.data_ptr(), M, N, K, _st()))
    torch.cuda.synchronize()
    assert float((c1 - c3).abs().max()) <= 1e-5 * np.abs(want).max()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_kernels_with_large_shared_memory_on_a_second_device_of_the_process():
    """A kernel's limit of dynamic shared memory is set per device; calls on one after the other, each on its own data."""
    lib = _capi.lib()
    M, N, K = 300, 256, 768
    A, W = synth.normal(60, (M, N)), synth.normal(61, (N, K), 0.1)
    B, H, S, D = 2, 4, 200, 32
    qkv = synth.qkv_planes(62, B, S, H * D)
    want_c, want_o = A.astype(np.float64) @ W.astype(np.float64), ob.mha(qkv, B, S, H * D, H, causal=True)[0]
    for device in range(2):
        with torch.cuda.device(device):
            dA, dW, dq = dev(A), dev(W), dev(qkv)
            c, o = torch.full((M, K), float("nan"), device="cuda"), torch.full((B * S, H * D), float("nan"), device="cuda")
            _capi.check(lib.hipgpt_matmul_tc(dA.data_ptr(), dW.data_ptr(), None, c.data_ptr(), M, N, K, _st()))
            _capi.check(lib.hipgpt_mha_forward_planes(dq.data_ptr(), o.data_ptr(), None, B, S, H * D, H, 1, _st()))
            torch.cuda.synchronize()
            assert np.abs(c.cpu().numpy() - want_c).max() <= 1e-5 * np.abs(want_c).max()
            assert np.abs(o.cpu().numpy() - want_o).max() <= 1e-5


def test_matmul_in_place_like_the_layers_output_projection():
    """src/transformer_layer.cpp:220 passes d_attn_output_ as both A and C."""
    lib = _capi.lib()
    M, N = 500, 256
    A, W, b = synth.normal(4, (M, N)), synth.normal(5, (N, N), 0.1), synth.normal(6, (N,))
    want = ob.matmul(A, W, b, M, N, N, fma=True)
    dA, dW, db = dev(A), dev(W), dev(b)
    raw = C.CDLL(_capi.lib_path())
    fn = getattr(raw, _capi.CXX_LAUNCHERS["launch_matmul_add_bias"])
    fn.restype = None
    fn.argtypes = [C.c_void_p] * 4 + [C.c_int] * 3
    torch.cuda.synchronize()
    fn(dA.data_ptr(), dW.data_ptr(), db.data_ptr(), dA.data_ptr(), M, N, N)         # legacy default stream
    torch.cuda.synchronize()
    assert np.array_equal(dA.cpu().numpy(), want)
    # in place with an output too wide for one block per row band: refused, not raced
    wide = torch.zeros((64, 512), device="cuda")
    w2 = torch.zeros((512, 512), device="cuda")
    assert lib.hipgpt_matmul(wide.data_ptr(), w2.data_ptr(), None, wide.data_ptr(), 64, 512, 512, _st()) == _capi.ERR_UNSUPPORTED


@pytest.mark.parametrize("rows,E", [(300, 256), (7, 64), (5, 100), (3, 1000), (2, 2048), (9, 1)])
def test_layer_norm(rows, E):
    lib = _capi.lib()
    x = synth.normal(7 + E, (rows, E)) * np.float32(2.0) + np.float32(0.3)
    g, b = synth.normal(8, (E,)), synth.normal(9, (E,))
    dx, dg, db = dev(x), dev(g), dev(b)
    dy = torch.full((rows, E), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_layer_norm(dx.data_ptr(), dy.data_ptr(), dg.data_ptr(), db.data_ptr(), rows, E, _st()))
    torch.cuda.synchronize()
    got = dy.cpu().numpy()
    assert np.array_equal(got, ob.layer_norm(x, g, b, rows, E, ref_order=False))       # the kernel's own order of sums
    assert float(np.abs(got - ob.layer_norm(x, g, b, rows, E, ref_order=True)).max()) <= 2e-6   # the reference kernel's order


def test_dropout_mask_is_the_reference_index_hash():
    lib = _capi.lib()
    rows, E, p = 900, 256, 0.1                    # 230400 elements: past index 185384, where the generator first keeps one
    x = synth.normal(10, (rows, E))
    want = ob.dropout_oracle(x, p).reshape(rows, E)
    dx = dev(x)
    dy = torch.full((rows, E), float("nan"), device="cuda")
    dm = torch.full((rows, E), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_dropout(dx.data_ptr(), dy.data_ptr(), dm.data_ptr(), p, rows, E, _st()))
    _capi.check(lib.hipgpt_dropout(dx.data_ptr(), dx.data_ptr(), None, p, rows, E, _st()))      # in place, no mask
    torch.cuda.synchronize()
    assert np.array_equal(dy.cpu().numpy(), want)
    assert np.array_equal(dx.cpu().numpy(), want)
    mask = dm.cpu().numpy()
    assert set(np.unique(mask)) <= {0.0, 1.0}
    assert np.array_equal(mask == 0.0, (want == 0.0) & (x != 0.0))
    assert 0 < (mask[-100:] == 1.0).mean() <= 1.0
    assert lib.hipgpt_dropout(dx.data_ptr(), dx.data_ptr(), None, 1.0, rows, E, _st()) == _capi.ERR_BAD_ARG


@pytest.mark.parametrize("rows,E", [(8192, 256), (33, 100), (7, 3), (1, 1)])
def test_fused_dropout_residual_equals_the_two_launchers(rows, E):
    """hipgpt_dropout_residual = hipgpt_dropout followed by hipgpt_add_inplace, bit for bit, mask included; in place too."""
    lib = _capi.lib()
    x, r = synth.normal(70 + E, (rows, E)), synth.normal(71 + E, (rows, E))
    dx, dr = dev(x), dev(r)
    two, mask2 = torch.empty_like(dx), torch.empty_like(dx)
    _capi.check(lib.hipgpt_dropout(dx.data_ptr(), two.data_ptr(), mask2.data_ptr(), C.c_float(0.1), rows, E, _st()))
    res = dr.clone()
    _capi.check(lib.hipgpt_add_inplace(res.data_ptr(), two.data_ptr(), rows * E, _st()))
    one, mask1 = torch.full_like(dx, float("nan")), torch.full_like(dx, float("nan"))
    _capi.check(lib.hipgpt_dropout_residual(dx.data_ptr(), dr.data_ptr(), one.data_ptr(), mask1.data_ptr(), C.c_float(0.1), rows, E, _st()))
    torch.cuda.synchronize()
    assert torch.equal(one, res) and torch.equal(mask1, mask2)
    # in place on the residual, without a mask, from an address that is not 16-byte aligned
    buf = torch.zeros(rows * E + 1, device="cuda")
    buf[1:] = dr.view(-1)
    _capi.check(lib.hipgpt_dropout_residual(dx.data_ptr(), buf[1:].data_ptr(), buf[1:].data_ptr(), None, C.c_float(0.1), rows, E, _st()))
    torch.cuda.synchronize()
    assert torch.equal(buf[1:].view(rows, E), res)


def test_add_relu_embedding_are_exact():
    lib = _capi.lib()
    n = 100003
    a, b = synth.normal(11, (n,)), synth.normal(12, (n,))
    da, dbb = dev(a), dev(b)
    _capi.check(lib.hipgpt_add_inplace(da.data_ptr(), dbb.data_ptr(), n, _st()))
    _capi.check(lib.hipgpt_relu(dbb.data_ptr(), n, _st()))
    B, S, V, E = 3, 17, 50, 24
    ids = synth.token_ids(5, (B, S), V).copy()
    ids[0, 3], ids[2, 5] = -1, V
    tok, pos = synth.normal(13, (V, E)), synth.normal(14, (S, E))
    d_ids, d_tok, d_pos = torch.from_numpy(ids).cuda(), dev(tok), dev(pos)
    d_out = torch.full((B * S, E), float("nan"), device="cuda")
    _capi.check(lib.hipgpt_embedding_lookup(d_ids.data_ptr(), d_tok.data_ptr(), d_pos.data_ptr(), d_out.data_ptr(), B, S, V, E, _st()))
    torch.cuda.synchronize()
    assert np.array_equal(da.cpu().numpy(), a + b)
    assert np.array_equal(dbb.cpu().numpy(), np.maximum(b, 0.0))
    assert np.array_equal(d_out.cpu().numpy(), ob.embedding(ids, tok, pos, B, S, V, E))


def _run_backward(g, qkv, probs, B, S, E, H, causal, planes=False):
    lib = _capi.lib()
    dg, dq = dev(g), dev(qkv.reshape(3, B * S, E))
    dp = dev(probs) if probs is not None else None
    dout = torch.full((3, B * S, E), float("nan"), device="cuda")
    if planes:
        _capi.check(lib.hipgpt_mha_backward_planes(dg.data_ptr(), dq.data_ptr(), dp.data_ptr() if dp is not None else None,
                                                   dout.data_ptr(), B, S, E, H, int(causal), _st()))
    else:
        nbytes = int(lib.hipgpt_mha_backward_scratch_bytes(B, H, S))
        scratch = torch.full((nbytes // 4,), float("nan"), device="cuda")
        _capi.check(lib.hipgpt_mha_backward(dg.data_ptr(), dq[0].data_ptr(), dq[1].data_ptr(), dq[2].data_ptr(),
                                            dp.data_ptr() if dp is not None else None, dout[0].data_ptr(), dout[1].data_ptr(),
                                            dout[2].data_ptr(), scratch.data_ptr(), nbytes, B, S, E, H, int(causal), _st()))
    torch.cuda.synchronize()
    return dout.cpu().numpy().reshape(-1)


@pytest.mark.parametrize("shape", [(2, 2, 40, 32), (1, 3, 70, 64), (2, 1, 9, 16), (1, 2, 33, 128), (2, 8, 256, 32), (1, 2, 300, 64), (1, 1, 1, 32)])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("stored", [True, False])
def test_attention_backward_matches_oracle(shape, causal, stored):
    B, H, S, D = shape
    E = H * D
    qkv = synth.qkv_planes(800 + S + D, B, S, E)
    g = synth.normal(801 + S, (B * S, E))
    probs = ob.mha(qkv, B, S, E, H, causal=causal, want_probs=True)[1] if stored else None
    want = ob.mha_backward(g, qkv, probs, B, S, E, H, causal=causal, fma=True)
    got = _run_backward(g, qkv, probs, B, S, E, H, causal)
    assert np.isfinite(got).all()
    # sums of up to S terms of size ~|g||v|: rounding differences of a reordered fp32 sum
    assert float(np.abs(got - want).max()) <= 1e-5 * max(1.0, float(np.abs(want).max()))
    again = _run_backward(g, qkv, probs, B, S, E, H, causal, planes=True)
    assert np.array_equal(again, got)                      # no atomics: the same bits on every run and entry point


@pytest.mark.parametrize("shape", [(1, 2, 63, 32), (1, 2, 64, 64), (2, 1, 65, 64), (1, 3, 127, 32), (1, 1, 128, 64), (1, 2, 129, 64), (1, 1, 450, 32), (65, 8, 128, 64)])
@pytest.mark.parametrize("causal,stored", [(False, True), (True, False), (False, False)])
def test_attention_backward_tensor_kernels_at_tile_edges(shape, causal, stored):
    """head_dim 32 / 64: tiles of 64 keys or queries, blocks of 128 rows, sequence lengths at and beside both, odd lengths (the
    stored probabilities then have no 16-byte rows), one and several groups of batches (the last shape)."""
    B, H, S, D = shape
    E = H * D
    qkv = synth.qkv_planes(820 + S, B, S, E)
    g = synth.normal(821 + S, (B * S, E))
    probs = ob.mha(qkv, B, S, E, H, causal=causal, want_probs=True)[1] if stored else None
    want = ob.mha_backward(g, qkv, probs, B, S, E, H, causal=causal, fma=True)
    got = _run_backward(g, qkv, probs, B, S, E, H, causal)
    assert float(np.abs(got - want).max()) <= 4e-6 * max(1.0, float(np.abs(want).max()))
    st = C.c_int(-1)
    _capi.check(_capi.lib().hipgpt_kernel_status(C.byref(st)))
    assert st.value == 0


@pytest.mark.parametrize("shape", [(1, 1, 4, 32), (1, 2, 132, 32), (1, 1, 451, 32), (2, 1, 452, 32), (1, 2, 388, 64)])
@pytest.mark.parametrize("causal", [False, True])
def test_attention_backward_ring_of_stored_probabilities(shape, causal):
    """The stored probabilities through a ring of two or three tiles: fewer tiles than the ring and several rounds of it, rows
    and columns that end inside a box, and (an odd length) the path without it."""
    B, H, S, D = shape
    E = H * D
    qkv = synth.qkv_planes(840 + S, B, S, E)
    g = synth.normal(841 + S, (B * S, E))
    probs = ob.mha(qkv, B, S, E, H, causal=causal, want_probs=True)[1]
    want = ob.mha_backward(g, qkv, probs, B, S, E, H, causal=causal, fma=True)
    got = _run_backward(g, qkv, probs, B, S, E, H, causal)
    assert float(np.abs(got - want).max()) <= 4e-6 * max(1.0, float(np.abs(want).max()))


@pytest.mark.parametrize("B,H,S,D", [(1, 1, 1, 32), (2, 3, 3, 32), (1, 2, 66, 32), (3, 2, 191, 32), (1, 3, 192, 32), (2, 2, 255, 32), (40, 4, 256, 32), (1, 2, 1, 64), (2, 2, 68, 64), (160, 1, 127, 64)])
@pytest.mark.parametrize("causal,stored", [(False, True), (True, True), (True, False), (False, False)])
def test_attention_backward_of_a_whole_head(B, H, S, D, causal, stored):
    """One block or a cluster of two per head: tiles of 64 keys and blocks of 128 rows that end inside, probabilities with and without 16-byte rows, more
    blocks than SMs; planes on 16-byte boundaries that are not 32-byte ones give the same bits."""
    E = H * D
    qkv, g = synth.qkv_planes(870 + S + D, B, S, E), synth.normal(871 + S, (B * S, E))
    probs = ob.mha(qkv, B, S, E, H, causal=causal, want_probs=True)[1] if stored else None
    want = ob.mha_backward(g, qkv, probs, B, S, E, H, causal=causal, fma=True)
    got = _run_backward(g, qkv, probs, B, S, E, H, causal, planes=True)
    assert float(np.abs(got - want).max()) <= 4e-6 * max(1.0, float(np.abs(want).max()))
    buf = torch.empty(4 + 3 * B * S * E, device="cuda")
    shifted = buf[4:]
    shifted.copy_(torch.from_numpy(np.ascontiguousarray(qkv).reshape(-1)))
    dg, dp, dout = dev(g), dev(probs) if stored else None, torch.full((3 * B * S * E,), float("nan"), device="cuda")
    _capi.check(_capi.lib().hipgpt_mha_backward_planes(dg.data_ptr(), shifted.data_ptr(), dp.data_ptr() if stored else None, dout.data_ptr(), B, S, E, H, int(causal), _st()))
    torch.cuda.synchronize()
    assert np.array_equal(dout.cpu().numpy().reshape(-1), got.reshape(-1))
    st = C.c_int(-1)
    _capi.check(_capi.lib().hipgpt_kernel_status(C.byref(st)))
    assert st.value == 0


def test_attention_backward_ring_of_stored_probabilities_many_times():
    """head_dim 32: the workers may be three tiles of probabilities ahead of the warp that fetches them.  It once could miss that a
    tile had been read, now and then, and the block gave up after a second."""
    B, H, S, D = 4, 8, 388, 32
    E = H * D
    qkv, g = torch.randn(3, B * S, E, device="cuda"), torch.randn(B * S, E, device="cuda")
    p, out, grad = torch.empty(B, H, S, S, device="cuda"), torch.empty(B * S, E, device="cuda"), torch.empty(3, B * S, E, device="cuda")
    _capi.check(_capi.lib().hipgpt_mha_forward_planes(qkv.data_ptr(), out.data_ptr(), p.data_ptr(), B, S, E, H, 0, _st()))
    for _ in range(4000):
        _capi.check(_capi.lib().hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), p.data_ptr(), grad.data_ptr(), B, S, E, H, 0, _st()))
    st = C.c_int(-1)
    _capi.check(_capi.lib().hipgpt_kernel_status(C.byref(st)))
    assert st.value == 0


def test_attention_backward_of_any_magnitude_and_captured_into_a_graph():
    B, H, S, D = 2, 2, 96, 64
    E = H * D
    qkv = synth.qkv_planes(830, B, S, E).reshape(3, B * S, E)
    qkv[0] *= np.float32(1e-6); qkv[1] *= np.float32(1e6); qkv[2] *= np.float32(3e8)
    g = synth.normal(831, (B * S, E)) * np.float32(2e-9)
    want = ob.mha_backward(g, qkv, None, B, S, E, H, fma=True).reshape(3, -1)
    got = _run_backward(g, qkv, None, B, S, E, H, False).reshape(3, -1)
    for w, o in zip(want, got):
        assert float(np.abs(o - w).max()) <= 1e-5 * float(np.abs(w).max())
    dg, dq, dout = dev(g), dev(qkv), torch.full((3, B * S, E), float("nan"), device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _capi.check(_capi.lib().hipgpt_mha_backward_planes(dg.data_ptr(), dq.data_ptr(), None, dout.data_ptr(), B, S, E, H, 0, _st()))
    for _ in range(2):
        dout.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(dout.cpu().numpy().reshape(3, -1), got)


@pytest.mark.parametrize("D,S", [(32, 130), (64, 97)])
@pytest.mark.parametrize("stored", [False, True])
def test_attention_backward_tiles_of_their_own_scale(D, S, stored):
    """The operands are cut relative to the largest magnitude of a 64-row tile: tiles of zeros, tiles 2^40 apart, and an infinity, which stays
    in its own row of dQ and leaves the tile's other rows their bits."""
    B, H = 1, 2
    E = H * D
    qkv = synth.qkv_planes(850 + S, B, S, E).reshape(3, S, E)
    g = synth.normal(851 + S, (S, E))
    zero = np.zeros_like(qkv)
    p_of = lambda x, causal: ob.mha(x, B, S, E, H, causal=causal, want_probs=True)[1] if stored else None
    got = _run_backward(g, zero, p_of(zero, True), B, S, E, H, True)
    want = ob.mha_backward(g, zero, p_of(zero, True), B, S, E, H, causal=True, fma=True)
    assert float(np.abs(got - want).max()) <= 4e-6 * max(1.0, float(np.abs(want).max()))
    # the second tile's V and dO 2^-40 of the first's: dP's own factor per pair of tiles, and dQ, dK of each tile to its own scale
    qkv[2, 64:] *= np.float32(2.0 ** -40)
    g[64:] *= np.float32(2.0 ** -40)
    probs = p_of(qkv, True)
    got = _run_backward(g, qkv, probs, B, S, E, H, True).reshape(3, S, E)
    want = ob.mha_backward(g, qkv, probs, B, S, E, H, causal=True, fma=True).reshape(3, S, E)
    for part in (slice(0, 64), slice(64, S)):
        for plane in range(3):
            w = want[plane, part]
            assert float(np.abs(got[plane, part] - w).max()) <= 1e-5 * float(np.abs(w).max())
    bad = g.copy()
    bad[5, 3] = np.inf                                     # a row of the first tile, in head 0
    hit = _run_backward(bad, qkv, probs, B, S, E, H, True).reshape(3, S, E)
    same = np.ones(S, bool)
    same[5] = False
    assert not np.isfinite(hit[0, 5, :D]).any()
    assert np.array_equal(hit[0, same], got[0, same]) and np.array_equal(hit[:, :, D:], got[:, :, D:])


def _backward_in_64_bits(g, qkv, probs, B, S, E, H, causal):
    """The three gradients [plane][B*S][E] in float64, and for each element the sum of its terms' magnitudes."""
    D, c = E // H, 1.0 / (E // H) ** 0.5
    heads = lambda x: torch.as_tensor(x, device="cuda").double().reshape(B, S, H, D).transpose(1, 2)      # noqa: E731
    back = lambda x: x.transpose(1, 2).reshape(B * S, E)      # noqa: E731
    q, k, v, g = *(heads(x) for x in torch.as_tensor(qkv).reshape(3, B * S, E)), heads(g)
    most = 0.0
    if probs is not None:
        p = torch.as_tensor(probs, device="cuda").double().reshape(B, H, S, S)
    else:
        s = c * q @ k.transpose(-1, -2)
        most = float(s.abs().max())
        p = (s.masked_fill(torch.ones(S, S, dtype=torch.bool, device="cuda").triu(1), float("-inf")) if causal else s).softmax(-1)
    vd, a = g @ v.transpose(-1, -2), g.abs() @ v.abs().transpose(-1, -2)
    ds, da = p * (vd - (p * vd).sum(-1, keepdim=True)), p.abs() * (a + (p.abs() * a).sum(-1, keepdim=True))
    t = lambda x: x.transpose(-1, -2)      # noqa: E731
    want = torch.stack([back(x) for x in (c * ds @ k, c * t(ds) @ q, t(p) @ g)])
    terms = torch.stack([back(x) for x in (c * da @ k.abs(), c * t(da) @ q.abs(), t(p).abs() @ g.abs())])
    return want, terms, most


def _assert_rows_are_near(got, want, terms, most):
    """Row by row of a head: within 5e-6 of the row's largest sum of magnitudes.  (Three factors to 2^-22 each, up to thirty truncations and roundings of
    2^-24 on the way through the two products, the sums of a row and of the tiles: below 40 x 2^-23.)  Where probabilities are formed again, their
    exponent's rounding too: 2^-21 of the largest score."""
    got, D = torch.as_tensor(got).cuda().double().reshape(want.shape), 32
    err, bound = ((x.reshape(*x.shape[:2], -1, D).amax(-1)) for x in ((got - want).abs(), terms))
    tol = 5e-6 + 2.0 ** -21 * most
    worst = float((err / bound.clamp_min(1e-300)).max())
    assert bool(torch.isfinite(got).all()) and worst <= tol, (worst, tol)


@pytest.mark.parametrize("D,S", [(32, 130), (64, 97), (32, 300), (64, 200)])
@pytest.mark.parametrize("stored", [False, True])
@pytest.mark.parametrize("plane", ["dO", "V", "K"])
def test_attention_backward_rows_of_a_tile_far_apart(D, S, stored, plane):
    """Rows of one 64-row tile down to 2^-28 of its largest, in any order, each output row to its own scale: with the mask a key of the last rows is
    seen by few queries, and those may all be small."""
    B, H = 1, 2
    E = H * D
    rng = np.random.default_rng(S)
    scale = (2.0 ** -rng.integers(0, 29, (S, 1))).astype(np.float32)
    qkv, g = synth.qkv_planes(890 + S, B, S, E).reshape(3, S, E).copy(), synth.normal(891 + S, (S, E))
    if plane == "dO":
        g = g * scale
    else:
        qkv[2 if plane == "V" else 1] *= scale
    for causal in (True, False):
        probs = ob.mha(qkv, B, S, E, H, causal=causal, want_probs=True)[1] if stored else None
        got = _run_backward(g, qkv, probs, B, S, E, H, causal)
        _assert_rows_are_near(got, *_backward_in_64_bits(g, qkv, probs, B, S, E, H, causal))


@pytest.mark.parametrize("D,S", [(32, 130), (32, 256), (64, 128), (32, 300), (64, 200)])
@pytest.mark.parametrize("stored", [False, True])
def test_attention_backward_of_keys_that_get_little_probability(D, S, stored):
    """Keys whose probabilities go down to e^-18 for every query: their rows of dK and dV to their own scale."""
    B, H = 1, 2
    E = H * D
    rng = np.random.default_rng(S + 1)
    qkv, g = synth.qkv_planes(892 + S, B, S, E).reshape(3, S, H, D) * np.float32(0.25), synth.normal(893 + S, (S, E))
    qkv[0, :, :, 0] = D ** 0.5
    qkv[1, :, :, 0] = -18.0 * rng.random((S, 1))
    qkv[1, 7, :, 0] = 0.0
    qkv = np.ascontiguousarray(qkv, dtype=np.float32).reshape(3, S, E)
    probs = ob.mha(qkv, B, S, E, H, want_probs=True)[1] if stored else None
    got = _run_backward(g, qkv, probs, B, S, E, H, False)
    _assert_rows_are_near(got, *_backward_in_64_bits(g, qkv, probs, B, S, E, H, False))


@pytest.mark.parametrize("D,S,B,H", [(32, 300, 1, 2), (64, 200, 1, 2), (32, 2200, 1, 1), (64, 384, 24, 8)])
@pytest.mark.parametrize("causal,stored", [(False, True), (True, False)])
def test_attention_backward_long_contexts_each_tile_of_its_own_scale(D, S, B, H, causal, stored):
    """The kernels of the longer contexts: a power of two of its own for each 64-row tile of Q, K, V and dO, more tiles than factors are read at a time
    (2200 rows), and more than one group of batches (24 x 8 heads of 384 rows)."""
    E = H * D
    tile = np.arange(S) // 64
    power = lambda n, lo: (2.0 ** -((tile * n) % 7 * lo)).astype(np.float32)[None, :, None]      # noqa: E731
    gen = torch.Generator(device="cuda").manual_seed(S)
    qkv = torch.randn(3, B, S, E, generator=gen, device="cuda")
    g = torch.randn(B, S, E, generator=gen, device="cuda") * torch.from_numpy(power(3, 5)).cuda()
    for i, (n, lo) in enumerate(((1, 1), (2, 1), (4, 6))):
        qkv[i] *= torch.from_numpy(power(n, lo)).cuda()
    p = torch.empty(B, H, S, S, device="cuda") if stored else None
    out, grad = torch.empty(B * S, E, device="cuda"), torch.full((3, B * S, E), float("nan"), device="cuda")
    if stored:
        _capi.check(_capi.lib().hipgpt_mha_forward_planes(qkv.data_ptr(), out.data_ptr(), p.data_ptr(), B, S, E, H, int(causal), _st()))
    _capi.check(_capi.lib().hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), p.data_ptr() if stored else None, grad.data_ptr(), B, S, E, H, int(causal), _st()))
    torch.cuda.synchronize()
    for b in range(0, B, 8):                               # (the comparison in parts: float64 scores take room)
        rows, n = slice(b * S, (b + 8) * S), min(8, B - b)
        args = (g[b:b + 8], qkv[:, b:b + 8], p[b:b + 8] if stored else None)
        _assert_rows_are_near(grad[:, rows], *_backward_in_64_bits(*args, n, S, E, H, causal))


@pytest.mark.parametrize("D,S", [(32, 300), (64, 200)])
def test_attention_backward_long_contexts_an_infinity_stays_in_its_row(D, S):
    """An infinity of dO becomes NaN in its own row of dQ and leaves the other rows, and the other head, their bits."""
    B, H = 1, 2
    E = H * D
    qkv, g = synth.qkv_planes(894 + S, B, S, E).reshape(3, S, E), synth.normal(895 + S, (S, E))
    for stored in (False, True):
        probs = ob.mha(qkv, B, S, E, H, causal=True, want_probs=True)[1] if stored else None
        want = _run_backward(g, qkv, probs, B, S, E, H, True).reshape(3, S, E)
        bad = g.copy()
        bad[70, 3] = np.inf
        got = _run_backward(bad, qkv, probs, B, S, E, H, True).reshape(3, S, E)
        same = np.arange(S) != 70
        assert not np.isfinite(got[0, 70, :D]).any()
        assert np.array_equal(got[0, same], want[0, same]) and np.array_equal(got[:, :, D:], want[:, :, D:])


@pytest.mark.parametrize("D,S", [(32, 130), (64, 200)])
@pytest.mark.parametrize("stored", [False, True])
def test_attention_backward_with_the_full_range_asked_for(D, S, stored):
    """hipgpt_set_full_range: rows 2^-60 apart inside a tile, each to its own scale, through both entry points; and afterwards the tensor pipe's bits again."""
    B, H, lib = 1, 2, _capi.lib()
    E = H * D
    rng = np.random.default_rng(S + 2)
    qkv, g0 = synth.qkv_planes(896 + S, B, S, E).reshape(3, S, E), synth.normal(897 + S, (S, E))
    g = g0 * (2.0 ** -rng.integers(0, 61, (S, 1))).astype(np.float32)
    probs = ob.mha(qkv, B, S, E, H, causal=True, want_probs=True)[1] if stored else None
    before = _run_backward(g0, qkv, probs, B, S, E, H, True)
    _capi.check(lib.hipgpt_set_full_range(1))
    try:
        got = [_run_backward(g, qkv, probs, B, S, E, H, True, planes=planes) for planes in (False, True)]
    finally:
        _capi.check(lib.hipgpt_set_full_range(0))
    assert np.array_equal(got[0], got[1])
    _assert_rows_are_near(got[0], *_backward_in_64_bits(g, qkv, probs, B, S, E, H, True))
    assert np.array_equal(_run_backward(g0, qkv, probs, B, S, E, H, True), before)


@pytest.mark.parametrize("D,S", [(32, 5), (32, 128), (32, 201), (32, 256), (64, 66), (64, 128), (32, 388), (32, 301), (64, 200), (64, 387)])
def test_attention_backward_moves_rows_of_one_probability_unchanged(D, S):
    """Stored probabilities of one key each, a permutation: dV is dO's rows bit for bit, whatever their magnitudes (powers of two over 2^100)."""
    B, H = 2, 2
    E = H * D
    rng = np.random.default_rng(S)
    qkv, g = synth.qkv_planes(880 + S, B, S, E), synth.normal(881 + S, (B, S, H, D)) * (2.0 ** rng.integers(-50, 51, (B, S, H, 1))).astype(np.float32)
    keys = np.stack([rng.permutation(S) for _ in range(B * H)]).reshape(B, H, S)
    probs = np.zeros((B, H, S, S), np.float32)
    np.put_along_axis(probs, keys[..., None], 1.0, axis=-1)
    dv = _run_backward(g.reshape(B * S, E), qkv, probs, B, S, E, H, False, planes=True).reshape(3, B, S, H, D)[2]
    for b in range(B):
        for h in range(H):
            assert np.array_equal(dv[b, keys[b, h], h], g[b, :, h])


@pytest.mark.parametrize("shape", [(8, 8, 256, 32), (8, 8, 128, 64), (4, 8, 700, 32), (2, 12, 777, 64)])
@pytest.mark.parametrize("causal,stored", [(False, True), (False, False), (True, False)])
def test_attention_backward_is_not_smaller_or_larger_than_it_should_be_on_the_average(shape, causal, stored):
    """The tensor core truncates where it adds; what that takes on the average, on unit normals, is given back: what is left is below a unit in the last
    place (2^-23) of the gradients as a whole."""
    B, H, S, D = shape
    E = H * D
    gen = torch.Generator(device="cuda").manual_seed(S + D)
    qkv, g = torch.randn(3, B * S, E, generator=gen, device="cuda"), torch.randn(B * S, E, generator=gen, device="cuda")
    p = torch.empty(B, H, S, S, device="cuda") if stored else None
    out, grad = torch.empty(B * S, E, device="cuda"), torch.empty(3, B * S, E, device="cuda")
    if stored:
        _capi.check(_capi.lib().hipgpt_mha_forward_planes(qkv.data_ptr(), out.data_ptr(), p.data_ptr(), B, S, E, H, int(causal), _st()))
    _capi.check(_capi.lib().hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), p.data_ptr() if stored else None, grad.data_ptr(), B, S, E, H, int(causal), _st()))
    want = _backward_in_64_bits(g, qkv, p, B, S, E, H, causal)[0]
    for plane in range(3):
        off = float(((grad[plane].double() - want[plane]) * want[plane]).sum() / (want[plane] ** 2).sum())
        assert abs(off) <= 2.0 ** -23, (plane, off)


@pytest.mark.parametrize("D,S", [(32, 300), (64, 200)])
@pytest.mark.parametrize("stored", [False, True])
def test_attention_backward_long_contexts_of_any_magnitude_and_captured_into_a_graph(D, S, stored):
    B, H = 2, 2
    E = H * D
    qkv = synth.qkv_planes(832 + S, B, S, E).reshape(3, B * S, E)
    qkv[0] *= np.float32(1e-6); qkv[1] *= np.float32(1e6); qkv[2] *= np.float32(3e8)
    g = synth.normal(833 + S, (B * S, E)) * np.float32(2e-9)
    probs = ob.mha(qkv, B, S, E, H, want_probs=True)[1] if stored else None
    got = _run_backward(g, qkv, probs, B, S, E, H, False)
    _assert_rows_are_near(got, *_backward_in_64_bits(g, qkv, probs, B, S, E, H, False))
    dg, dq, dp, dout = dev(g), dev(qkv), dev(probs) if stored else None, torch.full((3, B * S, E), float("nan"), device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _capi.check(_capi.lib().hipgpt_mha_backward_planes(dg.data_ptr(), dq.data_ptr(), dp.data_ptr() if stored else None, dout.data_ptr(), B, S, E, H, 0, _st()))
    for _ in range(2):
        dout.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert np.array_equal(dout.cpu().numpy().reshape(-1), got)


def test_attention_backward_reference_named_launcher():
    raw = C.CDLL(_capi.lib_path())
    fn = getattr(raw, _capi.CXX_LAUNCHERS["launch_multihead_attention_backward"])
    fn.restype = None
    fn.argtypes = [C.c_void_p] * 4 + [C.c_int] * 4
    B, H, S, D = 2, 4, 64, 32
    E = H * D
    qkv = synth.qkv_planes(810, B, S, E)
    g = synth.normal(811, (B * S, E))
    _, probs = ob.mha(qkv, B, S, E, H, want_probs=True)
    want = ob.mha_backward(g, qkv, probs, B, S, E, H)
    dg, dq, dp = dev(g), dev(qkv), dev(probs)
    dout = torch.full((3 * B * S * E,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    fn(dg.data_ptr(), dq.data_ptr(), dp.data_ptr(), dout.data_ptr(), B, S, E, H)
    torch.cuda.synchronize()
    assert float(np.abs(dout.cpu().numpy() - want).max()) <= 1e-5


needs_ref_run = pytest.mark.skipif(not os.path.exists(REF_RUN), reason="oracle/_ref/ref_model_run was not built (HipGPT tree not mounted at build time)")


@needs_ref_run
@pytest.mark.parametrize("fast_matmul", [False, True])
@pytest.mark.parametrize("B,S,E,H,F", [(2, 64, 64, 2, 96), (32, 256, 256, 8, 1024)])
def test_reference_transformer_layer_runs_on_this_library(tmp_path, B, S, E, H, F, fast_matmul):
    """HipGPT's own TransformerLayer (src/transformer_layer.cpp compiled where it lies): load() the weights,
    forward() on the GPU with every launcher resolved by this library, against the CPU oracle of the block.
    The second shape is the training default (benchmark configuration 2)."""
    w = synth.layer_weights(50 + E, E, H, F)
    x = synth.normal(51 + E, (B * S, E))
    with open(os.path.join(tmp_path, "layer.bin"), "wb") as f:
        checkpoint.write_layer(f, w, E, H, F)
    x.tofile(os.path.join(tmp_path, "x.bin"))
    r = subprocess.run([REF_RUN, "layer", os.path.join(tmp_path, "layer.bin"), os.path.join(tmp_path, "x.bin"),
                        os.path.join(tmp_path, "y.bin")] + [str(v) for v in (B, S, E, H, F)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, HIPGPT_FAST_MATMUL="1" if fast_matmul else "0"))    # 1: the tensor-core projections
    assert r.returncode == 0, r.stderr
    got = np.fromfile(os.path.join(tmp_path, "y.bin"), dtype=np.float32).reshape(B * S, E)
    want = ob.layer_forward(x, w, B, S, E, H, F, dropout_p=0.1)
    assert np.isfinite(got).all()
    # projections, layer norms, dropout and residuals are bit-exact restatements; attention agrees to 1e-5 and the
    # output projection and FFN carry that on (gains of a few)
    assert float(np.abs(got - want).max()) <= 1e-4
    kept = want != x            # where dropout kept something the block's output differs from its input
    assert kept.mean() > 0.5 if B * S * E > 400000 else True


@needs_ref_run
@pytest.mark.parametrize("cfg,n_new", [(dict(V=64, S=32, E=32, L=2, H=2, F=64), 6), (dict(synth.GPT_DEFAULT), 8)])
def test_reference_generation_loop_runs_on_this_library(tmp_path, cfg, n_new):
    """HipGPT's own GPTModel::generate (left-padded window re-run per token, dropout on, host sampling with
    top_k = 1) on the GPU against this library, ids against the CPU oracle of that loop."""
    w = synth.gpt_weights(3, **cfg)
    path = os.path.join(tmp_path, "model.bin")
    checkpoint.write_checkpoint(path, w, **cfg)
    prompt = synth.token_ids(3, (1, 5), cfg["V"])
    r = subprocess.run([REF_RUN, "generate", path] + [str(cfg[k]) for k in ("V", "S", "E", "H", "F", "L")] + [str(n_new)] +
                       [str(int(t)) for t in prompt[0]], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr
    got = np.array([int(t) for t in r.stdout.split()], dtype=np.int32)
    want, _ = ob.gpt_generate_window(w, **cfg, prompts=prompt, n_new=n_new, dropout_p=0.1)
    assert np.array_equal(got, want[0])


def test_generation_driver_reads_a_checkpoint_file(tmp_path):
    from hipgpt_b200.generation import GptDecoder
    cfg = dict(V=97, S=48, E=64, L=2, H=2, F=128)
    w = synth.gpt_weights(9, **cfg)
    path = os.path.join(tmp_path, "run_step7.bin")
    checkpoint.write_checkpoint(path, w, **cfg)
    checkpoint.write_run_config(os.path.join(tmp_path, "latest_config.json"), cfg["V"], cfg["S"], cfg["E"], cfg["H"], cfg["F"], cfg["L"],
                                "run_step7.bin", step=7)
    prompts = synth.token_ids(10, (3, 4), cfg["V"])
    base = GptDecoder(w, **cfg, max_batch=3)
    ids0 = base.generate(prompts, 12)[0]
    base.close()
    for src in (path, os.path.join(tmp_path, "latest_config.json")):
        dec = GptDecoder.from_checkpoint(src, max_batch=3)
        assert dec.shape == tuple(cfg[k] for k in ("V", "S", "E", "L", "H", "F"))
        assert np.array_equal(dec.generate(prompts, 12)[0], ids0)
        dec.close()
