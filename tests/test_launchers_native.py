"""The Python mirror's calls that go through the extension: what they take, and what they refuse, is what attribute look-ups and ctypes took."""
from __future__ import annotations

import pytest

torch = pytest.importorskip("torch")

from hipgpt_b200 import _capi, launchers  # noqa: E402


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
