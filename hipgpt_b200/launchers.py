"""Host-side mirror of the attention group of HipGPT's kernel API (include/hip_kernels.h:38-46
in the HipGPT tree) on top of the C ABI.  Names, argument order and meaning are the
reference's; arguments are CUDA float32 torch tensors (or raw device addresses) and the
calls are asynchronous on torch's current stream.  torch is used for device memory and
streams only; every kernel is the library's own.
"""
from __future__ import annotations

import ctypes
import threading
import warnings

import torch

from . import _capi


_FLOAT32 = torch.float32


def _ptr(t):
    if t is None or isinstance(t, int):
        return t
    if not (t.is_cuda and t.dtype is _FLOAT32 and t.is_contiguous()):
        raise ValueError("expected a contiguous CUDA float32 tensor")
    return t.data_ptr()


def _ptr_bf16(t):
    if not (t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous()):
        raise ValueError("expected a contiguous CUDA bfloat16 tensor")
    return t.data_ptr()


# the current stream's handle without the Stream object around it (3.2 us of host time per call)
_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)
_current_device = torch.cuda.current_device


def _stream():
    if _raw_stream is None:
        return torch.cuda.current_stream().cuda_stream
    return _raw_stream(_current_device())


class ArgumentError(ctypes.ArgumentError, TypeError):
    """A size that is no integer."""


def _int(x):
    """What ctypes takes for an int: an int, a c_int, or what stands for one."""
    if isinstance(x, int):
        return x
    if isinstance(x, ctypes.c_int):
        return x.value
    if hasattr(x, "_as_parameter_"):
        return _int(x._as_parameter_)
    raise ArgumentError(f"int expected instead of {type(x).__name__} instance")


class _ThroughCtypes:
    """The extension's calls without it."""

    @staticmethod
    def attention(d_qkv, d_output, d_attn_probs, B, S, E, H, causal):
        return _capi.lib().hipgpt_mha_forward_planes(_ptr(d_qkv), _ptr(d_output), _ptr(d_attn_probs), _int(B), _int(S), _int(E), _int(H), causal, _stream())

    @staticmethod
    def attention_bf16(d_qkv, d_output, B, S, E, H, causal, variant):
        p, out = _ptr_bf16(d_qkv), _ptr_bf16(d_output)
        plane = B * S * E * 2                               # bytes
        return _capi.lib().hipgpt_mha_forward_bf16_ex(p, p + plane, p + 2 * plane, out, B, S, E, H, causal, variant, _stream())

    @staticmethod
    def decode(q, kcache, vcache, out, scratch, nbytes, B, H, D, ctx, cap):
        p = [_ptr(t) for t in (q, kcache, vcache, out, scratch)]
        if nbytes is None:
            nbytes = 0 if scratch is None else scratch.numel() * scratch.element_size()
        return _capi.lib().hipgpt_mha_decode(*p, nbytes, _int(B), _int(H), _int(D), _int(ctx), _int(cap), _stream())


class _AtFirstCall:
    """Stands for the extension until it is needed, by the first of however many threads: importing this module builds and loads nothing."""

    _lock = threading.Lock()

    def __getattr__(self, name):
        global _native
        with self._lock:
            if _native is self:
                try:
                    native = _capi.native()
                    native.bind(_ptr, _ptr_bf16, _int)
                except (RuntimeError, ImportError, OSError) as e:       # no g++, no headers: the same library through ctypes
                    warnings.warn(f"the extension of the hot calls cannot be built or loaded, they go through ctypes (a few microseconds more each): {e}", RuntimeWarning, stacklevel=3)
                    native = _ThroughCtypes
                _native = native
        return getattr(_native, name)


_native = _AtFirstCall()


def launch_multihead_attention(d_qkv, d_output, d_attn_probs, B: int, S: int, E: int, H: int, *, causal: bool = False):
    """softmax(Q K^T / sqrt(E/H)) V per (batch, head).  d_qkv: three stacked [B*S, E] planes;
    d_output [B*S, E]; d_attn_probs [B, H, S, S] or None.  Not causal unless asked: the
    reference never masks (src/hip_kernels.cpp:287-319)."""
    if H <= 0 or E % H != 0:
        raise ValueError(f"Bad MHA config: E={E} H={H}")   # the reference aborts here
    rc = _native.attention(d_qkv, d_output, d_attn_probs, B, S, E, H, int(causal))
    if rc:
        _capi.check(rc)


def mha_forward(q, k, v, out, probs, B: int, S: int, E: int, H: int, *, causal: bool = False,
                algo: int = _capi.ALGO_AUTO, warps: int = 0):
    """The same on separate Q, K, V planes, with the kernel selector exposed."""
    _capi.check(_capi.lib().hipgpt_mha_forward_ex(_ptr(q), _ptr(k), _ptr(v), _ptr(out), _ptr(probs),
                                                  B, S, E, H, int(causal), algo, warps, _stream()))


def mha_forward_bf16(d_qkv, d_output, B: int, S: int, E: int, H: int, *, causal: bool = False, variant: int = 0):
    """The launcher's contract with bf16 storage: d_qkv = three stacked [B*S, E] bf16 planes, d_output
    [B*S, E] bf16 (head_dim 64), fp32 accumulation."""
    rc = _native.attention_bf16(d_qkv, d_output, B, S, E, H, int(causal), int(variant))
    if rc:
        _capi.check(rc)


def launch_scaled_dot_product(Q, K, scores, B: int, S: int, D: int):
    _capi.check(_capi.lib().hipgpt_scaled_dot_product(_ptr(Q), _ptr(K), _ptr(scores), B, S, D, _stream()))


def launch_softmax(scores, softmax_out, B: int, S: int):
    _capi.check(_capi.lib().hipgpt_softmax(_ptr(scores), _ptr(softmax_out), B, S, _stream()))


def launch_attention_weighted_sum(softmax, V, output, B: int, S: int, D: int):
    _capi.check(_capi.lib().hipgpt_attention_weighted_sum(_ptr(softmax), _ptr(V), _ptr(output), B, S, D, _stream()))


def decode_scratch_bytes(B: int, H: int, D: int, ctx: int) -> int:
    return int(_capi.lib().hipgpt_mha_decode_scratch_bytes(B, H, D, ctx))


def mha_decode(q, kcache, vcache, out, scratch, B: int, H: int, D: int, ctx: int, cap: int):
    """One query row per (batch, head) over the first ctx rows of the caches."""
    nbytes = None if scratch is None or type(scratch) is torch.Tensor else scratch.numel() * scratch.element_size()
    rc = _native.decode(q, kcache, vcache, out, scratch, nbytes, B, H, D, ctx, cap)
    if rc:
        _capi.check(rc)


def mha_forward_host(h_qkv, h_out, h_probs, B: int, S: int, E: int, H: int, *, causal: bool = False):
    """Host buffers in, host buffers out (numpy float32 arrays or CPU torch tensors, ideally
    pinned): the copies and the kernel run inside the call, which returns when h_out is ready."""
    def hp(a):
        if a is None:
            return None
        if isinstance(a, torch.Tensor):
            assert not a.is_cuda and a.dtype == torch.float32 and a.is_contiguous()
            return a.data_ptr()
        assert a.dtype.name == "float32" and a.flags["C_CONTIGUOUS"]
        return a.ctypes.data
    _capi.check(_capi.lib().hipgpt_mha_forward_host(hp(h_qkv), hp(h_out), hp(h_probs), B, S, E, H, int(causal)))


def mha_forward_bf16_host(h_qkv, h_out, B: int, S: int, E: int, H: int, *, causal: bool = False):
    """The host-buffer call for bf16 planes: CPU torch.bfloat16 tensors (ideally pinned), h_qkv three
    stacked [B*S, E] planes, h_out [B*S, E]; head_dim 64."""
    for t in (h_qkv, h_out):
        if not (isinstance(t, torch.Tensor) and not t.is_cuda and t.dtype == torch.bfloat16 and t.is_contiguous()):
            raise ValueError("expected a contiguous CPU bfloat16 tensor")
    _capi.check(_capi.lib().hipgpt_mha_forward_bf16_host(h_qkv.data_ptr(), h_out.data_ptr(), B, S, E, H, int(causal)))
