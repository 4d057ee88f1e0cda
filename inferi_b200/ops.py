"""Host-side mirror of the reference's op objects for the token loop, over the C ABI.

Each class keeps the name, argument meaning and error behaviour of its counterpart in
crates/inferi/src/ops/ (`GemvQuant`, `RmsNorm`, `RoPE`, `Silu`, `FusedAttention`) and of the façade methods in
crates/inferi/src/context.rs:336-719; shape-contract violations raise `InferiError` where the reference panics.
Device buffers are torch CUDA tensors (torch is only the allocator and the stream provider here).
"""
from __future__ import annotations

import ctypes as C
import importlib
from dataclasses import dataclass

import numpy as np
import torch

from . import _lib
from ._lib import AttnParams, InferiError, KV_F16, KV_F32, ROPE_NEOX, ROPE_ORIGINAL, check  # noqa: F401
from .build import binding_stamp
from .quant import BLOCK_BYTES, BLOCK_ELEMS, F32, NAMES, Q4_K, Q5_K, Q6_K, Q8_0, row_bytes  # noqa: F401


_f16, _f32, _tensor = torch.float16, torch.float32, torch.Tensor
# (a torch without CUDA has neither: it can import this module, make quantized data and read files; no launch gets as far as these)
_current_device, _raw_stream = getattr(torch._C, "_cuda_getDevice", None), getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream_ptr() -> int:
    """The current device's current stream as an integer, without building a `torch.cuda.Stream` object per call (3.2 us against 0.15)."""
    if not torch.cuda.is_initialized():
        return torch.cuda.current_stream().cuda_stream
    return _raw_stream(_current_device())


def _f32_dev(t: torch.Tensor, name: str) -> int:
    if isinstance(t, _tensor) and t.dtype is _f32 and t.is_cuda and t.is_contiguous():
        return t.data_ptr()
    raise InferiError(1, f"{name}: expected a contiguous float32 CUDA tensor")


# A launch goes through the compiled binding (csrc/binding.cpp), which checks what the code behind it checks and answers with the library's status, or
# with -1 where it has not launched anything: for arguments that it does not know (tensor subclasses), and for those that are refused.  The Python
# way then does the call or raises the error, and does all of them where there is no binding, or one of another torch.
class _NoBinding:
    gemv = gemm = rms_norm = rope = silu = add = attention = argmax = sample = staticmethod(lambda *a: -1)
    bind = staticmethod(lambda *a: None)


def _load_binding():
    try:
        m = importlib.import_module("._binding", __package__)
    except ImportError:
        return _NoBinding
    return m if getattr(m, "stamp", None) == binding_stamp() else _NoBinding


_fast = _load_binding()
_BOUND = ("ib_gemv_quant", "ib_gemm_quant", "ib_rms_norm", "ib_rope", "ib_silu_mul", "ib_add_assign", "ib_attention", "ib_argmax", "ib_sample")


# The Python ways take their tensors' addresses first: with a CUDA tensor among them CUDA is initialised, and the stream can be
# read without asking.


class Backend:
    """≙ `GpuBackend` + `LlmOps::new` (crates/inferi/src/context.rs:58-85): one context per device."""

    def __init__(self, device: int = 0):
        self.lib = _lib.load()
        h = C.c_void_p()
        check(self.lib.ib_ctx_create(device, C.byref(h)))
        self.handle = h
        self._address = h.value
        self.device = device
        _fast.bind(*(C.cast(getattr(self.lib, name), C.c_void_p).value for name in _BOUND))

    def launch_count(self) -> int:
        n = C.c_uint64()
        check(self.lib.ib_ctx_launch_count(self.handle, C.byref(n)))
        return int(n.value)

    def reset_launch_count(self) -> None:
        check(self.lib.ib_ctx_reset_launch_count(self.handle))

    def set_wait_limit(self, nanoseconds: int) -> None:
        """How long a wait inside a kernel may last before the kernel gives up and the next synchronising call returns
        IB_ERR_TIMEOUT (default 2 s).  Applies to launches issued, and token graphs recorded, after the call."""
        check(self.lib.ib_ctx_set_wait_limit(self.handle, int(nanoseconds)))

    def close(self) -> None:
        if getattr(self, "handle", None):
            self.lib.ib_ctx_destroy(self.handle)
            self.handle = self._address = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


class GpuQuantTensor:
    """≙ `GpuQuantTensor` (crates/inferi/src/quantized_matrix.rs:11-54) built by `GgufTensor::to_gpu_quant`
    (crates/inferi/src/gguf.rs:141-197): a [rows, cols] matrix of GGUF blocks on the device."""

    def __init__(self, backend: Backend, qtype: int, rows: int, cols: int, blocks):
        self.backend = backend
        self.qtype, self.rows, self.cols = qtype, rows, cols
        h = C.c_void_p()
        if isinstance(blocks, torch.Tensor) and blocks.is_cuda:
            b = blocks.contiguous().view(torch.uint8)
            check(backend.lib.ib_qtensor_upload(backend.handle, qtype, rows, cols, b.data_ptr(), b.numel(), 1, C.byref(h)))
        else:
            if isinstance(blocks, torch.Tensor):
                blocks = blocks.contiguous().view(torch.uint8).numpy()
            b = np.ascontiguousarray(blocks).view(np.uint8).reshape(-1)
            check(backend.lib.ib_qtensor_upload(backend.handle, qtype, rows, cols, b.ctypes.data_as(C.c_void_p), b.size, 0, C.byref(h)))
        self.handle = h
        self._address = h.value

    @property
    def nbytes(self) -> int:
        return self.rows * row_bytes(self.qtype, self.cols)

    def close(self) -> None:
        if getattr(self, "handle", None):
            self.backend.lib.ib_qtensor_destroy(self.handle)
            self.handle = self._address = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


class GemvQuant:
    """≙ `GemvQuant` (crates/inferi/src/ops/gemv_quant.rs:105-341)."""

    def __init__(self, backend: Backend):
        self.backend = backend

    @classmethod
    def from_backend(cls, backend: Backend) -> "GemvQuant":
        return cls(backend)

    def launch(self, out: torch.Tensor, m: GpuQuantTensor, v: torch.Tensor) -> None:
        """out[rows] = m . v[cols] on the current stream (asynchronous, like recording into a pass)."""
        rc = _fast.gemv(self.backend and self.backend._address, out, m._address, m.rows, m.cols, v)
        if rc == 0:
            return
        if rc > 0:
            check(rc)
        if v.numel() != m.cols or out.numel() != m.rows:
            raise InferiError(1, f"gemv: matrix is {m.rows}x{m.cols} but v has {v.numel()} and out {out.numel()} elements")
        b, out_ptr, v_ptr = self.backend, _f32_dev(out, "out"), _f32_dev(v, "v")
        rc = b.lib.ib_gemv_quant(b.handle, _raw_stream(_current_device()), out_ptr, m.handle, v_ptr)
        if rc:
            check(rc)

    def launch_host(self, m: GpuQuantTensor, v: np.ndarray) -> np.ndarray:
        """The same op for host buffers: copy in, run, copy out, synchronise."""
        v = np.ascontiguousarray(v, dtype=np.float32)
        if v.size != m.cols:
            raise InferiError(1, f"gemv: matrix has {m.cols} columns but v has {v.size} elements")
        out = np.empty(m.rows, dtype=np.float32)
        check(self.backend.lib.ib_gemv_quant_host(self.backend.handle, out.ctypes.data_as(C.c_void_p), m.handle, v.ctypes.data_as(C.c_void_p)))
        return out


class GemmQuant:
    """n quantized GEMVs as one GEMM on the tensor cores (prompt prefill); no counterpart in the reference, which repeats
    `GemvQuant::launch` per token."""

    def __init__(self, backend: Backend):
        self.backend = backend

    def launch(self, out: torch.Tensor, m: GpuQuantTensor, x: torch.Tensor) -> None:
        """out[n, rows] = x[n, cols] . m^T on the current stream."""
        rc = _fast.gemm(self.backend and self.backend._address, out, m._address, m.rows, m.cols, x)
        if rc == 0:
            return
        if rc > 0:
            check(rc)
        n = x.shape[0]
        if x.dim() != 2 or x.shape[1] != m.cols or tuple(out.shape) != (n, m.rows) or not x.is_contiguous() or not out.is_contiguous():
            raise InferiError(1, f"gemm: matrix is {m.rows}x{m.cols}, x {tuple(x.shape)}, out {tuple(out.shape)}")
        check(self.backend.lib.ib_gemm_quant(self.backend.handle, _stream_ptr(), _f32_dev(out, "out"), m.handle, _f32_dev(x, "x"), n))


class FfnGateUp:
    """`rms_norm_assign` + `matmul_quant_assign` (gate) + `matmul_quant_assign` (up) + `silu` of
    crates/inferi/src/models/llama2/transformer.rs:454-464 as one launch."""

    def __init__(self, backend: Backend):
        self.backend = backend

    def launch(self, out: torch.Tensor, gate: GpuQuantTensor, up: GpuQuantTensor, x: torch.Tensor, norm_w: torch.Tensor | None = None, eps: float = 1e-5) -> None:
        if x.numel() != gate.cols or out.numel() != gate.rows:
            raise InferiError(1, f"ffn gate/up: matrices are {gate.rows}x{gate.cols} but x has {x.numel()} and out {out.numel()} elements")
        check(self.backend.lib.ib_ffn_gate_up(self.backend.handle, _stream_ptr(), _f32_dev(out, "out"), gate.handle, up.handle, _f32_dev(x, "x"),
                                              _f32_dev(norm_w, "norm_w") if norm_w is not None else None, float(eps)))


@dataclass
class RmsNormConfig:
    """≙ `RmsNormConfig` (crates/inferi-shaders/src/rms_norm.rs:24-26)."""
    nudge_factor: float


class RmsNorm:
    """≙ `RmsNorm` (crates/inferi/src/ops/rms_norm.rs:9-79)."""

    def __init__(self, backend: Backend):
        self.backend = backend

    from_backend = classmethod(lambda cls, backend: cls(backend))

    def launch(self, config: RmsNormConfig, result: torch.Tensor, value: torch.Tensor, weight: torch.Tensor) -> None:
        rc = _fast.rms_norm(self.backend and self.backend._address, result, value, weight, config.nudge_factor)
        if rc == 0:
            return
        if rc > 0:
            check(rc)
        n = value.numel()
        if result.numel() != n or weight.numel() != n:
            raise InferiError(1, "rms_norm: result, value and weight must have the same length")
        b, r, v, w = self.backend, _f32_dev(result, "result"), _f32_dev(value, "value"), _f32_dev(weight, "weight")
        rc = b.lib.ib_rms_norm(b.handle, _raw_stream(_current_device()), r, v, w, n, config.nudge_factor)
        if rc:
            check(rc)


@dataclass
class RoPEConfig:
    """≙ `RoPEConfig` (crates/inferi-shaders/src/rope.rs:21-26)."""
    head_size: int
    kv_dim: int
    pos: int
    base_freq: float


class RoPE:
    """≙ `RoPE` (crates/inferi/src/ops/rope.rs:12-135)."""

    def __init__(self, backend: Backend):
        self.backend = backend

    from_backend = classmethod(lambda cls, backend: cls(backend))

    def launch(self, variant: int, config: RoPEConfig, in_out_q: torch.Tensor, in_out_k: torch.Tensor) -> None:
        rc = _fast.rope(self.backend and self.backend._address, variant, in_out_q, in_out_k, config.kv_dim, config.head_size, config.pos, config.base_freq)
        if rc == 0:
            return
        if rc > 0:
            check(rc)
        if in_out_k.numel() < config.kv_dim:
            raise InferiError(1, "rope: k is shorter than kv_dim")
        b, q, k = self.backend, _f32_dev(in_out_q, "q"), _f32_dev(in_out_k, "k")
        rc = b.lib.ib_rope(b.handle, _raw_stream(_current_device()), variant, q, in_out_q.numel(), k, config.kv_dim, config.head_size, config.pos, config.base_freq)
        if rc:
            check(rc)


class Silu:
    """≙ `Silu` (crates/inferi/src/ops/silu.rs:9-63): h1 <- h2 * swish(h1)."""

    def __init__(self, backend: Backend):
        self.backend = backend

    from_backend = classmethod(lambda cls, backend: cls(backend))

    def launch(self, in_out_h1: torch.Tensor, in_h2: torch.Tensor) -> None:
        rc = _fast.silu(self.backend and self.backend._address, in_out_h1, in_h2)
        if rc == 0:
            return
        if rc > 0:
            check(rc)
        n = in_out_h1.numel()
        if n != in_h2.numel():
            raise InferiError(1, "silu: h1 and h2 must have the same length")
        b, h1, h2 = self.backend, _f32_dev(in_out_h1, "h1"), _f32_dev(in_h2, "h2")
        rc = b.lib.ib_silu_mul(b.handle, _raw_stream(_current_device()), h1, h2, n)
        if rc:
            check(rc)


class FusedAttention:
    """≙ `FusedAttention` (crates/inferi/src/ops/batched_multiquery_attention.rs:14-77)."""

    def __init__(self, backend: Backend):
        self.backend = backend

    from_backend = classmethod(lambda cls, backend: cls(backend))

    def launch(self, params: AttnParams, q: torch.Tensor, key_cache: torch.Tensor, value_cache: torch.Tensor, xb: torch.Tensor) -> None:
        """key_cache / value_cache: [seq_len, kv_dim] float32 or float16 CUDA tensors."""
        rc = _fast.attention(self.backend and self.backend._address, params, q, key_cache, value_cache, xb) if type(params) is AttnParams else -1
        if rc == 0:
            return
        if rc > 0:
            check(rc)
        dtype = key_cache.dtype
        if dtype is not value_cache.dtype or (dtype is not _f16 and dtype is not _f32):
            raise InferiError(1, "attention: the caches must both be float16 or both float32")
        need = params.seq_len * params.kv_dim
        for t, name in ((key_cache, "key_cache"), (value_cache, "value_cache")):
            if not (t.is_cuda and t.is_contiguous() and t.numel() >= need):
                raise InferiError(1, f"attention: {name} must be a contiguous CUDA tensor of at least seq_len*kv_dim elements")
        n = params.n_heads * params.head_size
        if q.numel() != n or xb.numel() != n:
            raise InferiError(1, "attention: q and xb must hold n_heads*head_size elements")
        b, q_ptr, xb_ptr = self.backend, _f32_dev(q, "q"), _f32_dev(xb, "xb")
        rc = b.lib.ib_attention(b.handle, _raw_stream(_current_device()), C.byref(params), q_ptr, key_cache.data_ptr(), value_cache.data_ptr(),
                                KV_F16 if dtype is _f16 else KV_F32, xb_ptr)
        if rc:
            check(rc)


def add_assign(backend: Backend, a: torch.Tensor, b: torch.Tensor) -> None:
    """≙ `LlmContext::add_assign` (crates/inferi/src/context.rs:516-530): a += b."""
    rc = _fast.add(backend and backend._address, a, b)
    if rc == 0:
        return
    if rc > 0:
        check(rc)
    n = a.numel()
    if n != b.numel():
        raise InferiError(1, "add_assign: length mismatch")
    a_ptr, b_ptr = _f32_dev(a, "a"), _f32_dev(b, "b")
    rc = backend.lib.ib_add_assign(backend.handle, _raw_stream(_current_device()), a_ptr, b_ptr, n)
    if rc:
        check(rc)


def argmax(backend: Backend, logits: torch.Tensor, out: torch.Tensor) -> None:
    """≙ greedy `Sampler::sample` (crates/inferi/src/models/sampler.rs:32-36, 54-56); out: int32/uint32[1] on the device."""
    rc = _fast.argmax(backend and backend._address, logits, out)
    if rc == 0:
        return
    if rc > 0:
        check(rc)
    if not (out.is_cuda and out.element_size() == 4):
        raise InferiError(1, "argmax: out must be a 4-byte CUDA tensor")
    check(backend.lib.ib_argmax(backend.handle, _stream_ptr(), _f32_dev(logits, "logits"), logits.numel(), out.data_ptr()))


class Sampler:
    """≙ `Sampler` (crates/inferi/src/models/sampler.rs:14-52) with the logits left on the device.  `coin` in [0, 1) is the
    caller's random number; temperature 0 is the greedy arg-max."""

    def __init__(self, backend: Backend, vocab_size: int, temperature: float, topp: float):
        self.backend, self.vocab_size, self.temperature, self.topp = backend, vocab_size, float(temperature), float(topp)

    def sample(self, logits: torch.Tensor, coin: float, out: torch.Tensor | None = None) -> torch.Tensor:
        if logits.numel() != self.vocab_size:
            raise ValueError(f"expected {self.vocab_size} logits, got {logits.numel()}")
        out = out if out is not None else torch.empty(1, dtype=torch.int32, device=logits.device)
        rc = _fast.sample(self.backend and self.backend._address, logits, self.vocab_size, self.temperature, self.topp, coin, out)
        if rc == 0:
            return out
        if rc > 0:
            check(rc)
        check(self.backend.lib.ib_sample(self.backend.handle, _stream_ptr(), _f32_dev(logits, "logits"), self.vocab_size, self.temperature, self.topp,
                                         float(coin), out.data_ptr()))
        return out

