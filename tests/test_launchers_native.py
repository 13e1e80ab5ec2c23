"""The Python mirror's calls that go through the extension: what they take, and what they refuse, is what attribute look-ups and ctypes took."""
from __future__ import annotations

import ctypes
import os
import subprocess
import sys
import threading
import time

import pytest

torch = pytest.importorskip("torch")

from hipgpt_b200 import _capi, build, launchers  # noqa: E402


class Subclass(torch.Tensor):
    pass


def test_what_is_not_a_cuda_tensor_is_refused():
    cpu = torch.zeros(96)
    with pytest.raises(ValueError, match="contiguous CUDA float32"):
        launchers.launch_multihead_attention(cpu, cpu, None, 1, 1, 32, 1)
    with pytest.raises(ValueError, match="contiguous CUDA float32"):
        launchers.mha_decode(cpu.as_subclass(Subclass), None, None, None, None, 1, 1, 32, 1, 1)
    with pytest.raises(ValueError, match="contiguous CUDA bfloat16"):
        launchers.mha_forward_bf16(cpu, cpu, 1, 1, 64, 1)
    with pytest.raises(AttributeError):
        launchers.mha_forward_bf16(None, None, 1, 1, 64, 1)
    with pytest.raises(AttributeError):
        launchers.launch_multihead_attention("planes", None, None, 1, 1, 32, 1)
    with pytest.raises(ValueError, match="Bad MHA config"):
        launchers.launch_multihead_attention(cpu, cpu, None, 1, 1, 33, 2)


@pytest.mark.gpu
def test_tensors_parameters_subclasses_and_addresses_are_taken():
    B, H, S, D = 2, 3, 40, 32
    E = H * D
    qkv, want, got = torch.randn(3, B * S, E, device="cuda"), torch.empty(B * S, E, device="cuda"), torch.empty(B * S, E, device="cuda")
    launchers.launch_multihead_attention(qkv, want, None, B, S, E, H, causal=True)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for x in (torch.nn.Parameter(qkv, requires_grad=False), qkv.as_subclass(Subclass), qkv.data_ptr()):
        with torch.cuda.stream(side):                      # torch's current stream, whatever it is
            got.fill_(float("nan"))
            launchers.launch_multihead_attention(x, got, None, B, S, E, H, causal=True)
        side.synchronize()
        assert torch.equal(got, want)
    q, kc, vc = torch.randn(B, E, device="cuda"), torch.randn(B, 300, E, device="cuda"), torch.randn(B, 300, E, device="cuda")
    n = launchers.decode_scratch_bytes(B, H, D, 290)
    scratch = torch.empty(n // 4, device="cuda")
    out, again = torch.empty(B, E, device="cuda"), torch.empty(B, E, device="cuda")
    launchers.mha_decode(q, kc, vc, out, scratch, B, H, D, 290, 300)
    launchers.mha_decode(q.as_subclass(Subclass), kc.data_ptr(), vc, again, scratch.as_subclass(Subclass), B, H, D, 290, 300)
    torch.cuda.synchronize()
    assert n > 0 and torch.equal(out, again)


@pytest.mark.gpu
def test_refusals_on_the_gpu():
    B, H, S, D = 1, 2, 40, 32
    E = H * D
    qkv, out = torch.randn(3, B * S, E, device="cuda"), torch.empty(B * S, E, device="cuda")
    for bad in (qkv.double(), qkv.transpose(1, 2), qkv.cpu()):
        with pytest.raises(ValueError):
            launchers.launch_multihead_attention(bad, out, None, B, S, E, H)
    with pytest.raises(TypeError):
        launchers.mha_decode(qkv, qkv, qkv, out, None, 1.5, H, D, 1, 1)
    with pytest.raises(_capi.HipGPTError):
        launchers.launch_multihead_attention(None, out, None, B, S, E, H)
    with pytest.raises(_capi.HipGPTError, match="scratch"):
        launchers.mha_decode(qkv, qkv, qkv, out, None, B, H, D, 100, 100)
    with pytest.raises(_capi.HipGPTError):
        launchers.mha_forward_bf16(qkv.bfloat16(), out.bfloat16(), B, S, E, H)          # head_dim 32


def test_the_library_needs_no_torch(tmp_path):
    """Its build neither imports torch nor makes the extension, and its being up to date does not hang on one."""
    code = """
import sys
sys.modules["torch"] = None                              # an import of it fails
from hipgpt_b200 import build
build.LIB, build.OBJDIR = sys.argv[1] + "/lib.so", sys.argv[1]
class Done: returncode, stdout, stderr = 0, "", ""
def run(cmd, **kw):
    open(cmd[cmd.index("-o") + 1], "w").close()
    return Done
build.subprocess.run = run
assert build.build() == build.LIB and build.up_to_date()
"""
    subprocess.run([sys.executable, "-c", code, str(tmp_path)], check=True, cwd=build.ROOT)


def test_importing_the_mirror_builds_and_loads_nothing():
    code = """
from hipgpt_b200 import _capi, build
def refuse(*a, **kw): raise AssertionError("built or loaded")
_capi.native = _capi.lib = build.build = build.build_extension = refuse
import hipgpt_b200.launchers
"""
    subprocess.run([sys.executable, "-c", code], check=True, cwd=build.ROOT)


def test_an_extension_belongs_to_one_torch_and_appears_when_it_is_whole(tmp_path, monkeypatch):
    mine = build.extension_path()
    monkeypatch.setattr(torch, "__version__", "9.9.9")
    assert build.extension_path() != mine
    monkeypatch.setattr(build, "LIBDIR", str(tmp_path))
    out = build.extension_path()

    class Done:
        returncode, stdout, stderr = 1, "", "no"

    def run(cmd, **kw):
        target = cmd[cmd.index("-o") + 1]
        assert target != out and not os.path.exists(out)
        with open(target, "w") as f:
            f.write("half")
        return Done
    monkeypatch.setattr(build.subprocess, "run", run)
    with pytest.raises(RuntimeError, match="launchers_py"):
        build.build_extension()
    assert os.listdir(tmp_path) == []
    Done.returncode = 0
    assert build.build_extension() == out and os.listdir(tmp_path) == [os.path.basename(out)]


def test_threads_that_call_first_together_load_one_extension(monkeypatch):
    loaded, real, start = [], _capi.native, threading.Barrier(8)

    def native():
        loaded.append(threading.get_ident())
        time.sleep(0.2)
        return real()
    monkeypatch.setattr(_capi, "native", native)
    monkeypatch.setattr(launchers, "_native", launchers._AtFirstCall())
    refused = []

    def call():
        start.wait()
        try:
            launchers.mha_decode(torch.zeros(4), None, None, None, None, 1, 1, 32, 1, 1)
        except ValueError:
            refused.append(1)
    threads = [threading.Thread(target=call) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(loaded) == 1 and len(refused) == 8


@pytest.fixture
def without_extension(monkeypatch):
    def refuse():
        raise RuntimeError("no g++")
    monkeypatch.setattr(_capi, "native", refuse)
    monkeypatch.setattr(launchers, "_native", launchers._AtFirstCall())


def test_without_the_extension_the_same_is_refused(without_extension):
    with pytest.warns(RuntimeWarning, match="no g"), pytest.raises(ValueError, match="contiguous CUDA float32"):
        launchers.launch_multihead_attention(torch.zeros(96), torch.zeros(96), None, 1, 1, 32, 1)
    test_what_is_not_a_cuda_tensor_is_refused()


@pytest.mark.filterwarnings("ignore:the extension of the hot calls")
@pytest.mark.parametrize("native", [True, False])
def test_sizes_are_what_ctypes_takes(native, request):
    """As through ctypes: an int or a c_int; what is neither is ctypes.ArgumentError, and a TypeError, before anything is called."""
    if not native:
        request.getfixturevalue("without_extension")
    for bad in (1.5, "4", None, ctypes.c_long(4)):
        with pytest.raises(ctypes.ArgumentError) as e:
            launchers.mha_decode(None, None, None, None, None, bad, 1, 32, 1, 1)
        assert isinstance(e.value, TypeError)
    assert launchers._int(ctypes.c_int(7)) == 7 and launchers._int(True) == 1


@pytest.mark.gpu
@pytest.mark.filterwarnings("ignore:the extension of the hot calls")
@pytest.mark.parametrize("native", [True, False])
def test_c_ints_are_taken(native, request):
    if not native:
        request.getfixturevalue("without_extension")
    B, H, D, cap = 2, 3, 32, 50
    E = H * D
    q, kc, vc = torch.randn(B, E, device="cuda"), torch.randn(B, cap, E, device="cuda"), torch.randn(B, cap, E, device="cuda")
    want, got = torch.empty(B, E, device="cuda"), torch.empty(B, E, device="cuda")
    launchers.mha_decode(q, kc, vc, want, None, B, H, D, 17, cap)
    launchers.mha_decode(q, kc, vc, got, None, *(ctypes.c_int(x) for x in (B, H, D, 17, cap)))
    assert torch.equal(want, got)
    S = 20
    qkv, a, b = torch.randn(3, B * S, E, device="cuda"), torch.empty(B * S, E, device="cuda"), torch.empty(B * S, E, device="cuda")
    launchers.launch_multihead_attention(qkv, a, None, B, S, E, H, causal=True)
    launchers.launch_multihead_attention(qkv, b, None, ctypes.c_int(B), ctypes.c_int(S), E, H, causal=True)
    assert torch.equal(a, b)
    E = 2 * 64
    qkv, a, b = (torch.randn(n, B * S, E, device="cuda").bfloat16() for n in (3, 1, 1))
    launchers.mha_forward_bf16(qkv, a, B, S, E, 2)
    launchers._ThroughCtypes.attention_bf16(qkv, b, B, S, E, 2, 0, 0)
    assert torch.equal(a, b)
