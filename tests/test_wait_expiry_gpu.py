"""The give-up paths of the bounded waits, exercised on a healthy GPU: a barrier at which nothing arrives with a
limit of a fraction of a millisecond.  Nothing here traps, faults or spins without a limit; the launches return
by themselves, the status word names the wait, nothing is stored, and the next normal launch is unaffected."""
import ctypes as C

import numpy as np
import pytest

from hipgpt_b200 import _capi, synth
from oracle import bindings as ob

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
from tests.gpu_util import gpu_mha  # noqa: E402


def _status():
    st = C.c_int(-1)
    _capi.check(_capi.lib().hipgpt_kernel_status(C.byref(st)))
    return st.value


def test_a_wait_that_runs_out_is_reported_and_stores_nothing():
    lib = _capi.lib()
    assert _status() == 0
    canary = torch.full((4096,), -7.0, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    _capi.check(lib.hipgpt_debug_wait_expiry(canary.data_ptr(), canary.numel(), 200000, st))     # ~0.1 ms at 1.9 GHz
    torch.cuda.synchronize()
    assert _status() == 907                      # 900 + the site of the wait that ran out; not the one that completed (1),
    assert _status() == 0                        # not the one cut short by the flag (8); read once, then cleared
    assert bool((canary == -7.0).all())          # the block skipped its stores
    # the next normal launch is unaffected
    B, H, S, D = 2, 4, 256, 32
    qkv = synth.qkv_planes(5, B, S, H * D)
    out, _ = gpu_mha(qkv, B, S, H * D, H, True, False)
    assert float(np.abs(out - ob.mha(qkv, B, S, H * D, H, causal=True)[0]).max()) <= 1e-5
    assert _status() == 0
    # limits outside the hook's range are refused
    assert lib.hipgpt_debug_wait_expiry(canary.data_ptr(), canary.numel(), 1 << 30, st) == _capi.ERR_BAD_ARG


def test_a_stalled_grid_barrier_ends_the_persistent_generation_call_with_an_error():
    from hipgpt_b200.generation import GptDecoder, MODE_PERSISTENT
    cfg = dict(V=97, S=48, E=64, L=2, H=2, F=128)
    w = synth.gpt_weights(9, **cfg)
    prompts = synth.token_ids(10, (3, 4), cfg["V"])
    dec = GptDecoder(w, **cfg, max_batch=3)
    want = dec.generate(prompts, 10)[0]                     # graph mode
    dec.set_mode(MODE_PERSISTENT)
    assert np.array_equal(dec.generate(prompts, 10)[0], want)
    _capi.check(_capi.lib().hipgpt_gpt_debug_stall_barrier(dec._h, 400000))      # ~0.2 ms
    with pytest.raises(_capi.HipGPTError, match="grid barrier"):
        dec.generate(prompts, 10)
    assert np.array_equal(dec.generate(prompts, 10)[0], want)                  # the handle stays usable
    dec.close()


def test_stalled_clusters_end_the_generation_call_with_an_error():
    """One block's wait runs out; it sends nothing after its layer, so the other blocks' waits run out too, and all leave."""
    from hipgpt_b200.generation import GptDecoder
    cfg = dict(V=131, S=64, E=128, L=3, H=4, F=512)
    w = synth.gpt_weights(9, **cfg)
    prompts = synth.token_ids(10, (9, 6), cfg["V"])
    dec = GptDecoder(w, **cfg, max_batch=9)
    assert _capi.lib().hipgpt_gpt_debug_cluster_rows(dec._h, 9, 20) > 0
    want = dec.generate(prompts, 15)
    for _ in range(2):
        _capi.check(_capi.lib().hipgpt_gpt_debug_stall_barrier(dec._h, 400000))      # ~0.2 ms
        with pytest.raises(_capi.HipGPTError, match="inside a cluster"):
            dec.generate(prompts, 15)
        again = dec.generate(prompts, 15)
        assert np.array_equal(again[0], want[0]) and np.array_equal(again[1], want[1])    # the handle stays usable
    dec.close()


def _expired(code, block, call, *outs):
    """The outputs of `call` with the wait of this code run out in one block, canaries where nothing was stored.  What is waited for
    may have come before, so that nothing has to wait: then once more."""
    for _ in range(20):
        for o in outs:
            o.fill_(-7.0)
        _capi.check(_capi.lib().hipgpt_debug_expire_wait(code, block))
        call()
        torch.cuda.synchronize()
        status = _status()
        if status:
            break
    assert status == code and _status() == 0
    return [o.clone() for o in outs]


@pytest.mark.parametrize("code,block", [(501, 0), (501, 147), (502, 3), (503, 5)])
def test_an_expired_wait_of_a_projection_stores_none_of_the_blocks_tiles(code, block):
    """20 x 20 tiles: a block has two or three, none of them may be stored; the others and the next call are as ever."""
    M, N, K = 2560, 320, 2560
    a, w = (torch.randn(*s, generator=torch.Generator(device="cuda").manual_seed(3), device="cuda") for s in ((M, N), (N, K)))
    out = torch.empty(M, K, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    run = lambda: _capi.check(_capi.lib().hipgpt_matmul_tc(a.data_ptr(), w.data_ptr(), None, out.data_ptr(), M, N, K, st))      # noqa: E731
    run()
    want = out.clone()
    got, = _expired(code, block, run, out)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for t in range(400):
        piece = (slice(t // 20 * 128, t // 20 * 128 + 128), slice(t % 20 * 128, t % 20 * 128 + 128))
        if t % sms == block:
            assert bool((got[piece] == -7.0).all()), t
        else:
            assert torch.equal(got[piece], want[piece]), t
    run()
    assert torch.equal(out, want) and _status() == 0
    assert _capi.lib().hipgpt_debug_expire_wait(401, 0) == _capi.ERR_BAD_ARG


BWD_SHAPE = B_, H_, S_ = 2, 2, 300


def _backward(D, stored):
    E = H_ * D
    gen = torch.Generator(device="cuda").manual_seed(4)
    qkv, g = torch.randn(3, B_ * S_, E, generator=gen, device="cuda"), torch.randn(B_ * S_, E, generator=gen, device="cuda")
    p, grad, st = None, torch.empty(3, B_ * S_, E, device="cuda"), torch.cuda.current_stream().cuda_stream
    if stored:
        p, out = torch.empty(B_, H_, S_, S_, device="cuda"), torch.empty(B_ * S_, E, device="cuda")
        _capi.check(_capi.lib().hipgpt_mha_forward_planes(qkv.data_ptr(), out.data_ptr(), p.data_ptr(), B_, S_, E, H_, 0, st))
    run = lambda: _capi.check(_capi.lib().hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), p.data_ptr() if stored else None,       # noqa: E731
                                                                     grad.data_ptr(), B_, S_, E, H_, 0, st))
    return run, grad, (qkv, g, p)


def _blocks(x, D):
    """Gradients [3][B S][E] as [3][B][block of 128 rows][H][row, D]."""
    x = x.view(3, B_, S_, H_, D)
    return [[x[i, :, j:j + 128].permute(0, 2, 1, 3) for j in range(0, S_, 128)] for i in range(3)]


@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("stored", [True, False])
@pytest.mark.parametrize("code", [601, 604, 605, 606, 611, 614, 615, 616])
def test_an_expired_wait_of_the_backward_stores_none_of_the_blocks_rows(D, stored, code):
    """Block 1: the second 128 queries (dQ) or keys (dK, dV) of the first head."""
    if stored:
        code = {601: 607, 614: 617}.get(code, code)          # the stored probabilities come later than the operands and the scores
    run, grad, keep = _backward(D, stored)
    run()
    want = grad.clone()
    got, = _expired(code, 1, run, grad)
    touched = (0,) if code < 610 else (1, 2)
    for i in range(3):
        for j, (g, w) in enumerate(zip(_blocks(got, D)[i], _blocks(want, D)[i])):
            if i in touched and j == 1:
                assert bool((g[0, 0] == -7.0).all())
                g[0, 0] = w[0, 0]
            if code in (601, 604, 605, 607) and (i == 1 or (i == 2 and not stored)):
                # formed from row sums (and log-sum-exps) that the block did not leave (605: unless it had, the wait that runs out is
                # the first that has to wait at all)
                lost = bool(torch.isnan(g[0, 0]).all())
                assert lost or code == 605
                if lost:
                    g[0, 0] = w[0, 0]
            assert torch.equal(g, w), (i, j)
    run()
    assert torch.equal(grad, want) and _status() == 0


@pytest.mark.parametrize("code,block", [(501, 1), (503, 6), (501, 79)])
def test_an_expired_wait_of_a_split_product_leaves_the_whole_tile_out(code, block):
    """Four blocks of a cluster share a tile's slices and store a quarter of its columns each: none may, with one's sum unfinished."""
    M, N, K = 1280, 1024, 256
    a, w = (torch.randn(*s, generator=torch.Generator(device="cuda").manual_seed(5), device="cuda") for s in ((M, N), (N, K)))
    out = torch.empty(M, K, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    run = lambda: _capi.check(_capi.lib().hipgpt_matmul_tc(a.data_ptr(), w.data_ptr(), None, out.data_ptr(), M, N, K, st))      # noqa: E731
    run()
    want = out.clone()
    got, = _expired(code, block, run, out)
    for t in range(20):
        piece = (slice(t // 2 * 128, t // 2 * 128 + 128), slice(t % 2 * 128, t % 2 * 128 + 128))
        if t == block // 4:
            assert bool((got[piece] == -7.0).all())
        else:
            assert torch.equal(got[piece], want[piece]), t
    run()
    assert torch.equal(out, want) and _status() == 0


@pytest.mark.parametrize("D,S", [(32, 200), (64, 100)])
@pytest.mark.parametrize("stored,code", [(s, c) for s in (True, False) for c in (621, 623, 624, 625, 626) if not s or c != 623])
def test_an_expired_wait_of_a_whole_head_stores_none_of_its_rows(D, S, stored, code):
    """The last block of the first head: nothing of its rows is stored, the other block of the head stores what does not depend on it or nothing, and the
    other heads are as ever.  (Stored probabilities, 622, and g V^T, 623 with them, are there before they are waited for.)"""
    B, H = 2, 2
    E, block = H * D, 1 if S > 128 else 0
    gen = torch.Generator(device="cuda").manual_seed(6)
    qkv, g = torch.randn(3, B * S, E, generator=gen, device="cuda"), torch.randn(B * S, E, generator=gen, device="cuda")
    p, grad, st = torch.empty(B, H, S, S, device="cuda"), torch.empty(3, B * S, E, device="cuda"), torch.cuda.current_stream().cuda_stream
    _capi.check(_capi.lib().hipgpt_mha_forward_planes(qkv.data_ptr(), grad.data_ptr(), p.data_ptr(), B, S, E, H, 0, st))
    run = lambda: _capi.check(_capi.lib().hipgpt_mha_backward_planes(g.data_ptr(), qkv.data_ptr(), p.data_ptr() if stored else None, grad.data_ptr(), B, S, E, H, 0, st))   # noqa: E731
    run()
    want = grad.clone()
    got, = _expired(code, block, run, grad)
    got, want4 = got.view(3, B, S, H, D), want.view(3, B, S, H, D)
    mine = slice(128 * block, S)
    assert bool((got[:, 0, mine, 0] == -7.0).all())
    if block:
        assert torch.equal(got[0, 0, :128, 0], want4[0, 0, :128, 0])         # dQ needs nothing of the other block
        for i in (1, 2):
            part = got[i, 0, :128, 0]
            assert torch.equal(part, want4[i, 0, :128, 0]) or bool((part == -7.0).all())
    assert torch.equal(got[:, :, :, 1], want4[:, :, :, 1]) and torch.equal(got[:, 1], want4[:, 1])
    run()
    assert torch.equal(grad, want) and _status() == 0
