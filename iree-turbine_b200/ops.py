"""The op library: ``torch.ops.b200k.*``.

Each op is a ``CustomOp`` registered the way the reference registers its op libraries
(iree/turbine/ops/__init__.py:7-11; e.g. iree/turbine/ops/conv_fwd.py:62-89 for a ``select``):
a schema string and a ``select`` that types every argument and declares the result meta tensors
(which also is the Meta implementation, so fake tensors and ``torch.compile`` tracing work).  The
CUDA implementations are native (``csrc/torch_ops.cpp``, built as ``_native.so``): they call the C
ABI on the current stream and cost a few microseconds of host time.  There is no CPU
implementation, so a CPU tensor fails in the dispatcher with torch's own "not implemented for CPU"
error; without the built ``_native.so`` a CUDA tensor fails there as well.
"""

from __future__ import annotations

import ctypes as C
import sys
import types
from typing import Optional

import torch
from torch import Tensor

from . import _launcher as L
from .op_reg import CustomOp, KernelSelection, def_library

__all__ = [
    "LIBRARY",
    "gemm_nt",
    "gemm_fp8_nt",
    "gemm",
    "bmm",
    "linear",
    "linear_act",
    "attention",
    "attention_lse",
    "attention_bwd",
    "sdpa",
    "decode_attention",
    "paged_decode_attention",
    "quantize_e4m3",
    "paged_gather",
    "kv_append",
    "paged_attention",
    "device_status",
    "reset_device_status",
]

LIBRARY = def_library("b200k")

try:
    from . import _native  # registers the CUDA implementations
except ImportError as _e:
    _native_error = _e

    class _native:  # every use says what is missing; the ops themselves have no CUDA implementation
        def __getattr__(self, name):
            raise RuntimeError(
                f"the operator implementations (_native.so) cannot be loaded: {_native_error}. Run "
                "`python csrc/build.py` in the package directory. There is no fallback.")

    _native = _native()

_HALF_TYPES = (torch.float16, torch.bfloat16)


def _status_word(device) -> Tensor:
    """The device's int32 status word: kernels OR a code into it if a bounded device-side wait gave up
    (see include/b200k.h).  Reading it synchronizes, so it is only read on request."""
    dev = torch.device("cuda") if device is None else torch.device(device)
    return _native.status_word(dev.index if dev.index is not None else torch.cuda.current_device())


def _status_ptr(device: torch.device) -> int:
    return _status_word(device).data_ptr()


def device_status(device=None) -> int:
    """Returns the device status word (0 = no kernel reported a timed-out wait).  Synchronizes."""
    return int(_status_word(device).item())


def reset_device_status(device=None) -> None:
    _status_word(device).zero_()


_raw_stream = getattr(torch._C, "_cuda_getCurrentRawStream", None)


def _stream(t: Tensor) -> C.c_void_p:
    """The current stream of the tensor's device as a raw cudaStream_t (the direct binding when torch
    has it: building a Stream object per launch costs several microseconds)."""
    if _raw_stream is not None and t.device.index is not None:
        return C.c_void_p(_raw_stream(t.device.index))
    return C.c_void_p(torch.cuda.current_stream(t.device).cuda_stream)


def _row_major_2d(t: Tensor) -> Tensor:
    """A 2-D view whose last dim is contiguous and whose row stride is a multiple of 16 bytes."""
    if t.stride(1) != 1 or (t.stride(0) * t.element_size()) % 16 != 0 or t.data_ptr() % 16 != 0:
        t = t.contiguous()
    return t


# ---------------------------------------------------------------------------------------------
# GEMM
# ---------------------------------------------------------------------------------------------
def _gemm_out_dtype(in_dtype: torch.dtype, out_dtype) -> torch.dtype:
    if in_dtype in _HALF_TYPES:
        od = torch.float32 if out_dtype is None else out_dtype
        torch._check(od in (torch.float32, in_dtype), lambda: f"gemm_nt: out_dtype must be float32 or {in_dtype}")
        return od
    od = torch.bfloat16 if out_dtype is None else out_dtype
    torch._check(od in (torch.bfloat16, torch.float32), lambda: "gemm_fp8_nt: out_dtype must be bfloat16 or float32")
    return od


def _launch_gemm(a: Tensor, b: Tensor, out: Tensor, scale_a, scale_b, tile_n: int = 0, tile_m: int = 0,
                 bias: Optional[Tensor] = None, activation: str = "none", a_km: bool = False,
                 b_kn: bool = False, split_k: int = 0) -> None:
    """a is stored [M, K] ([K, M] with a_km); b is stored [N, K] ([K, N] with b_kn).  split_k: 0 = the
    library decides, 1 = whole tiles only, 2 / 4 / 8 = CTAs per output tile."""
    a = _row_major_2d(a)
    b = _row_major_2d(b)
    args = L.GemmArgs()
    args.a, args.b, args.c = a.data_ptr(), b.data_ptr(), out.data_ptr()
    args.m, args.k = (a.size(1), a.size(0)) if a_km else (a.size(0), a.size(1))
    args.n = b.size(1) if b_kn else b.size(0)
    args.a_km, args.b_kn = int(a_km), int(b_kn)
    args.lda, args.ldb, args.ldc = a.stride(0), b.stride(0), out.stride(0)
    args.in_dtype = L.DTYPE_CODES[a.dtype]
    args.out_dtype = L.DTYPE_CODES[out.dtype]
    args.scale_a = scale_a.data_ptr() if scale_a is not None else None
    args.scale_b = scale_b.data_ptr() if scale_b is not None else None
    args.status = _status_ptr(a.device)
    args.tile_n = tile_n
    args.tile_m = tile_m
    args.split_k = split_k
    if activation not in L.ACTIVATION_CODES:
        raise ValueError(f"unknown activation {activation!r}; expected one of {sorted(L.ACTIVATION_CODES)}")
    args.activation = L.ACTIVATION_CODES[activation]
    if bias is not None:
        bias = bias.contiguous()
        args.bias = bias.data_ptr()
        args.bias_dtype = L.DTYPE_CODES[bias.dtype]
    L.check(L.lib().b200k_gemm_nt(C.byref(args), _stream(a)))


@CustomOp.register(library=LIBRARY, register_impl=False)
class gemm_nt(CustomOp):
    """C[M,N] = A[M,K] @ B[N,K]^T, f16 or bf16 operands, fp32 accumulation.

    Output dtype: float32 unless ``out_dtype`` names the operand dtype.
    """

    signature = "gemm_nt(Tensor a, Tensor b, ScalarType? out_dtype=None) -> Tensor"

    def select(self, sel: KernelSelection):
        a = sel.arg_tensor(0)
        b = sel.arg_tensor(1)
        od = sel.attr_optional(2)
        torch._check(a.t.dim() == 2 and b.t.dim() == 2, lambda: "gemm_nt: a and b must be 2-D")
        torch._check(a.t.dtype in _HALF_TYPES, lambda: f"gemm_nt: dtype must be float16 or bfloat16, got {a.t.dtype}")
        torch._check(a.t.dtype == b.t.dtype, lambda: "gemm_nt: a and b must have the same dtype")
        torch._check(a.t.size(1) == b.t.size(1), lambda: f"gemm_nt: K mismatch: a is {list(a.t.shape)}, b is {list(b.t.shape)}")
        torch._check(a.t.size(1) % 8 == 0, lambda: "gemm_nt: K must be a multiple of 8")
        a.specialize_dims(1)
        b.specialize_dims(1)
        sel.return_new_tensor([a.t.size(0), b.t.size(0)], _gemm_out_dtype(a.t.dtype, od.v))


@CustomOp.register(library=LIBRARY, register_impl=False)
class gemm(CustomOp):
    """C = op(a) @ op(b) with BLAS-style flags: ``a`` is [M, K] ([K, M] with ``trans_a``), ``b`` is
    [K, N] ([N, K] with ``trans_b``); f16 / bf16, fp32 accumulation.  No operand is repacked: the
    kernel reads either storage order.  ``gemm_nt(a, b)`` is ``gemm(a, b, trans_b=True)``."""

    signature = ("gemm(Tensor a, Tensor b, bool trans_a=False, bool trans_b=False, "
                 "ScalarType? out_dtype=None) -> Tensor")

    @staticmethod
    def _mnk(a, b, trans_a, trans_b):
        m, k = (a.size(1), a.size(0)) if trans_a else (a.size(0), a.size(1))
        kb, n = (b.size(1), b.size(0)) if trans_b else (b.size(0), b.size(1))
        return m, n, k, kb

    def select(self, sel: KernelSelection):
        a = sel.arg_tensor(0)
        b = sel.arg_tensor(1)
        ta = sel.attr_bool(2)
        tb_ = sel.attr_bool(3)
        od = sel.attr_optional(4)
        torch._check(a.t.dim() == 2 and b.t.dim() == 2, lambda: "gemm: a and b must be 2-D")
        torch._check(a.t.dtype in _HALF_TYPES and a.t.dtype == b.t.dtype,
                     lambda: f"gemm: a and b must both be float16 or bfloat16, got {a.t.dtype}, {b.t.dtype}")
        m, n, k, kb = self._mnk(a.t, b.t, bool(ta.v), bool(tb_.v))
        torch._check(k == kb, lambda: f"gemm: contraction sizes differ ({k} vs {kb})")
        torch._check(a.t.size(1) % 8 == 0 and b.t.size(1) % 8 == 0,
                     lambda: "gemm: the contiguous dimension of each operand must be a multiple of 8")
        sel.return_new_tensor([m, n], _gemm_out_dtype(a.t.dtype, od.v))


@CustomOp.register(library=LIBRARY, register_impl=False)
class bmm(CustomOp):
    """Batched product ``a[B, M, K] @ b[B, K, N]`` (aten::bmm; the reference's BOO layer registers it
    beside mm and addmm, kernel/boo/op_exports/registry.py:99-104), f16 / bf16, fp32 accumulation, every
    problem's tiles in one persistent launch.  Either operand may be a transposed view (e.g.
    ``k.transpose(1, 2)``): the kernel reads both storage orders."""

    signature = "bmm(Tensor a, Tensor b, ScalarType? out_dtype=None) -> Tensor"

    def select(self, sel: KernelSelection):
        a = sel.arg_tensor(0)
        b = sel.arg_tensor(1)
        od = sel.attr_optional(2)
        torch._check(a.t.dim() == 3 and b.t.dim() == 3, lambda: "bmm: a and b must be 3-D")
        torch._check(a.t.dtype in _HALF_TYPES and a.t.dtype == b.t.dtype,
                     lambda: f"bmm: a and b must both be float16 or bfloat16, got {a.t.dtype}, {b.t.dtype}")
        torch._check(a.t.size(0) == b.t.size(0) and a.t.size(2) == b.t.size(1),
                     lambda: f"bmm: shapes {list(a.t.shape)} and {list(b.t.shape)} do not multiply")
        torch._check(a.t.size(1) % 8 == 0 or a.t.size(2) % 8 == 0, lambda: "bmm: M or K must be a multiple of 8")
        sel.return_new_tensor([a.t.size(0), a.t.size(1), b.t.size(2)], _gemm_out_dtype(a.t.dtype, od.v))


@CustomOp.register(library=LIBRARY, register_impl=False)
class col_sum(CustomOp):
    """Column sums of a f16 / bf16 matrix, summed in fp32: the bias gradient of ``linear``."""

    signature = "col_sum(Tensor x) -> Tensor"

    def select(self, sel: KernelSelection):
        x = sel.arg_tensor(0)
        torch._check(x.t.dim() == 2 and x.t.dtype in _HALF_TYPES, lambda: "col_sum: x must be a float16 or bfloat16 matrix")
        sel.return_new_tensor([x.t.size(1)], x.t.dtype)


@CustomOp.register(library=LIBRARY, register_impl=False)
class linear_op(CustomOp):
    """``linear`` as an operator (its autograd formula is native, see ``linear`` below)."""

    signature = "linear(Tensor x, Tensor w, Tensor? bias=None) -> Tensor"

    def select(self, sel: KernelSelection):
        x = sel.arg_tensor(0)
        w = sel.arg_tensor(1)
        sel.arg_optional_tensor(2)
        torch._check(x.t.dim() == 2 and w.t.dim() == 2 and x.t.size(1) == w.t.size(1),
                     lambda: "linear: x must be [M, K] and w [N, K]")
        sel.return_new_tensor([x.t.size(0), w.t.size(0)], x.t.dtype)


def linear(x: Tensor, w: Tensor, bias: Optional[Tensor] = None) -> Tensor:
    """Differentiable ``x[M, K] @ w[N, K]^T + bias`` (f16 / bf16 CUDA tensors) on the b200k GEMM, with both
    backward products on the same kernel (the reference wraps its own op the same way,
    kernel/boo/ops/conv.py:313-372; the products are those of kernel/boo/op_exports/gemm.py:233-270):
    dx = dy @ w, dw = dy^T @ x, db = sum(dy)."""
    return torch.ops.b200k.linear(x, w, bias)


@CustomOp.register(library=LIBRARY, register_impl=False)
class linear_act(CustomOp):
    """act(A[M,K] @ W[N,K]^T + bias[N]) in one kernel: the GEMM with bias and activation applied in
    its epilogue (the shape of a linear layer with trailing optional bias).  ``activation`` is
    "none", "relu", "gelu" (erf form) or "silu"; output dtype as for ``gemm_nt``."""

    signature = ("linear_act(Tensor a, Tensor w, Tensor? bias=None, str activation=\"none\", "
                 "ScalarType? out_dtype=None) -> Tensor")

    def select(self, sel: KernelSelection):
        a = sel.arg_tensor(0)
        w = sel.arg_tensor(1)
        bias = sel.arg_optional_tensor(2)
        act = sel.attr_str(3)
        od = sel.attr_optional(4)
        torch._check(a.t.dim() == 2 and w.t.dim() == 2, lambda: "linear_act: a and w must be 2-D")
        torch._check(a.t.dtype in _HALF_TYPES and a.t.dtype == w.t.dtype,
                     lambda: f"linear_act: a and w must both be float16 or bfloat16, got {a.t.dtype}, {w.t.dtype}")
        torch._check(a.t.size(1) == w.t.size(1) and a.t.size(1) % 8 == 0,
                     lambda: "linear_act: K must match and be a multiple of 8")
        torch._check(act.v in L.ACTIVATION_CODES, lambda: f"linear_act: unknown activation {act.v!r}")
        bt = bias.t if bias is not None else None
        if bt is not None:
            torch._check(bt.dim() == 1 and bt.size(0) == w.t.size(0), lambda: "linear_act: bias must be [N]")
            torch._check(bt.dtype in (torch.float32,) + _HALF_TYPES, lambda: "linear_act: bias must be float32 / float16 / bfloat16")
        sel.return_new_tensor([a.t.size(0), w.t.size(0)], _gemm_out_dtype(a.t.dtype, od.v))


@CustomOp.register(library=LIBRARY, register_impl=False)
class gemm_fp8_nt(CustomOp):
    """C = (A8 @ B8^T) * scale_a * scale_b with float8_e4m3fn operands and per-tensor fp32 scales.

    ``scale_a`` / ``scale_b`` are one-element float32 device tensors.  Output bfloat16 (default)
    or float32.
    """

    signature = (
        "gemm_fp8_nt(Tensor a, Tensor b, Tensor scale_a, Tensor scale_b, ScalarType? out_dtype=None) -> Tensor"
    )

    def select(self, sel: KernelSelection):
        a = sel.arg_tensor(0)
        b = sel.arg_tensor(1)
        sa = sel.arg_tensor(2)
        sb = sel.arg_tensor(3)
        od = sel.attr_optional(4)
        torch._check(a.t.dim() == 2 and b.t.dim() == 2, lambda: "gemm_fp8_nt: a and b must be 2-D")
        torch._check(
            a.t.dtype == torch.float8_e4m3fn and b.t.dtype == torch.float8_e4m3fn,
            lambda: "gemm_fp8_nt: a and b must be float8_e4m3fn",
        )
        torch._check(a.t.size(1) == b.t.size(1), lambda: "gemm_fp8_nt: K mismatch")
        torch._check(a.t.size(1) % 16 == 0, lambda: "gemm_fp8_nt: K must be a multiple of 16")
        torch._check(
            sa.t.numel() == 1 and sb.t.numel() == 1 and sa.t.dtype == torch.float32 and sb.t.dtype == torch.float32,
            lambda: "gemm_fp8_nt: scales must be one-element float32 tensors",
        )
        sel.return_new_tensor([a.t.size(0), b.t.size(0)], _gemm_out_dtype(a.t.dtype, od.v))


@CustomOp.register(library=LIBRARY, register_impl=False)
class quantize_e4m3(CustomOp):
    """Per-tensor quantisation: returns (x / s cast to float8_e4m3fn, s) with s = max|x| / 448."""

    signature = "quantize_e4m3(Tensor x) -> (Tensor, Tensor)"

    def select(self, sel: KernelSelection):
        x = sel.arg_tensor(0)
        torch._check(x.t.dtype == torch.float32, lambda: "quantize_e4m3: x must be float32")
        sel.return_new_tensor(list(x.t.shape), torch.float8_e4m3fn)
        sel.return_new_tensor([1], torch.float32)


# ---------------------------------------------------------------------------------------------
# attention forward
# ---------------------------------------------------------------------------------------------
class _OpsModule(types.ModuleType):
    """This module with one checked attribute.  ``ATTENTION_KERNEL`` says which forward kernel
    ``attention`` / ``attention_lse`` / ``paged_attention`` ask for: 0 lets the library choose (one-tile or
    tile-pair kernel, see include/b200k.h), 1 / 2 force one of them (head dim 64 only exists in the pair
    kernel).  A tuning and testing knob, like the GEMM tile shape; the native implementations keep it."""

    @property
    def ATTENTION_KERNEL(self) -> int:
        return _native.attention_kernel()

    @ATTENTION_KERNEL.setter
    def ATTENTION_KERNEL(self, value: int) -> None:
        _native.set_attention_kernel(int(value))


sys.modules[__name__].__class__ = _OpsModule


def _fill_attention_args(q: Tensor, k: Tensor, v: Tensor, o: Tensor, scale: float, causal: bool) -> L.AttentionArgs:
    args = L.AttentionArgs()
    args.batch, args.q_heads, args.seq_q, args.head_dim = q.shape
    args.kernel = _native.attention_kernel() if args.head_dim == 128 else L.ATTN_AUTO
    args.q, args.k, args.v, args.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr()
    _, args.kv_heads, args.seq_kv, _ = k.shape
    args.q_stride_b, args.q_stride_h, args.q_stride_s, _ = q.stride()
    args.k_stride_b, args.k_stride_h, args.k_stride_s, _ = k.stride()
    args.v_stride_b, args.v_stride_h, args.v_stride_s, _ = v.stride()
    args.o_stride_b, args.o_stride_h, args.o_stride_s, _ = o.stride()
    args.dtype = L.DTYPE_CODES[q.dtype]
    args.causal = 1 if causal else 0
    args.scale = float(scale)
    return args


def _attention_out_like(q: Tensor, device) -> Tensor:
    """The output takes the memory layout of q when q's rows are contiguous (as
    aten.scaled_dot_product_attention does: a [B, H, S, D] view of [B, S, H, D] memory stays one),
    so graphs traced against the ATen op keep their views valid; otherwise it is contiguous.  The
    kernel writes any layout with contiguous rows."""
    if q.dim() == 4 and q.stride(-1) == 1:
        return torch.empty_like(q, device=device)
    return torch.empty(q.shape, dtype=q.dtype, device=device)


def _attention_select(sel: KernelSelection):
    q = sel.arg_tensor(0)
    k = sel.arg_tensor(1)
    v = sel.arg_tensor(2)
    sel.attr_float(3)
    sel.attr_bool(4)
    torch._check(q.t.dim() == 4 and k.t.dim() == 4 and v.t.dim() == 4, lambda: "attention: q, k, v must be 4-D [B,H,S,D]")
    torch._check(q.t.dtype in _HALF_TYPES, lambda: f"attention: dtype must be float16 or bfloat16, got {q.t.dtype}")
    torch._check(q.t.dtype == k.t.dtype == v.t.dtype, lambda: "attention: q, k, v must share a dtype")
    torch._check(q.t.size(3) in (64, 128) and k.t.size(3) == q.t.size(3) and v.t.size(3) == q.t.size(3),
                 lambda: "attention: head dim must be 128 or 64, the same for q, k and v")
    torch._check(k.t.shape == v.t.shape, lambda: "attention: k and v must have the same shape")
    torch._check(q.t.size(0) <= k.t.size(0), lambda: "attention: batch mismatch")
    torch._check(q.t.size(1) % k.t.size(1) == 0, lambda: "attention: query heads must be a multiple of kv heads")
    q.specialize_dims(3)
    sel.return_tensor(_attention_out_like(q.t, "meta"))
    return q


@CustomOp.register(library=LIBRARY, register_impl=False)
class attention(CustomOp):
    """O = softmax(scale * Q K^T [causal]) V.  q [B,Hq,Sq,D], k/v [B,Hkv,Skv,D] -> [B,Hq,Sq,D], D = 128 or 64."""

    signature = "attention(Tensor q, Tensor k, Tensor v, float scale, bool is_causal) -> Tensor"

    def select(self, sel: KernelSelection):
        _attention_select(sel)


@CustomOp.register(library=LIBRARY, register_impl=False)
class attention_lse(CustomOp):
    """``attention`` that also returns the row statistic the backward needs:
    lse[b, h, i] = ln sum_j exp(scale * q_i . k_j) over the visible keys (float32, -inf for a row
    that sees none)."""

    signature = "attention_lse(Tensor q, Tensor k, Tensor v, float scale, bool is_causal) -> (Tensor, Tensor)"

    def select(self, sel: KernelSelection):
        q = _attention_select(sel)
        sel.return_new_tensor(list(q.t.shape[:3]), torch.float32)


def _attention_bwd_checks(q: Tensor, k: Tensor, v: Tensor, o: Tensor, d_o: Tensor, lse: Optional[Tensor] = None) -> None:
    if lse is not None:
        torch._check(lse.dtype == torch.float32 and tuple(lse.shape) == tuple(q.shape[:3]),
                     lambda: "attention_bwd: lse must be float32 [B, Hq, Sq]")
    for t in (q, k, v, o, d_o):
        torch._check(t.dim() == 4 and t.size(3) in (64, 128) and t.size(3) == q.size(3),
                     lambda: "attention_bwd: tensors must be [B,H,S,D] with D = 128 or 64, the same for all")
        torch._check(t.dtype == q.dtype, lambda: "attention_bwd: all tensors must share a dtype")
    torch._check(q.dtype in _HALF_TYPES, lambda: f"attention_bwd: dtype must be float16 or bfloat16, got {q.dtype}")
    torch._check(k.shape == v.shape, lambda: "attention_bwd: k and v must have the same shape")
    torch._check(o.shape == q.shape and d_o.shape == q.shape, lambda: "attention_bwd: o and d_o must have q's shape")
    torch._check(q.size(0) == k.size(0), lambda: "attention_bwd: batch mismatch")
    torch._check(k.size(1) > 0 and q.size(1) % k.size(1) == 0,
                 lambda: "attention_bwd: query heads must be a multiple of kv heads")


@CustomOp.register(library=LIBRARY, register_impl=False)
class attention_bwd(CustomOp):
    """Gradients of ``attention``: (q, k, v, o, d_o) -> (d_q, d_k, d_v).  d_k / d_v are summed over
    the query heads of a group.  Only the forward OUTPUT is needed; row statistics are recomputed."""

    signature = ("attention_bwd(Tensor q, Tensor k, Tensor v, Tensor o, Tensor d_o, float scale, bool is_causal, "
                 "Tensor? lse=None) -> (Tensor, Tensor, Tensor)")

    def select(self, sel: KernelSelection):
        q, k, v, o, d_o = (sel.arg_tensor(i) for i in range(5))
        sel.attr_float(5)
        sel.attr_bool(6)
        lse = sel.arg_optional_tensor(7)
        _attention_bwd_checks(q.t, k.t, v.t, o.t, d_o.t, lse.t if lse is not None else None)
        sel.return_new_tensor(list(q.t.shape), q.t.dtype)
        sel.return_new_tensor(list(k.t.shape), q.t.dtype)
        sel.return_new_tensor(list(k.t.shape), q.t.dtype)


@CustomOp.register(library=LIBRARY, register_impl=False)
class sdpa_op(CustomOp):
    """``sdpa`` as an operator (its autograd formula is native: ``attention_lse`` forward, ``attention_bwd``
    backward)."""

    signature = "sdpa(Tensor q, Tensor k, Tensor v, float scale, bool is_causal) -> Tensor"

    def select(self, sel: KernelSelection):
        _attention_select(sel)


def sdpa(q: Tensor, k: Tensor, v: Tensor, scale: Optional[float] = None, is_causal: bool = False) -> Tensor:
    """Differentiable scaled-dot-product attention on the b200k kernels ([B, H, S, D] f16 / bf16
    CUDA tensors, D = 128 or 64; grouped-query heads; causal mask aligned to the bottom-right corner)."""
    if q.size(-1) not in (64, 128):
        raise ValueError("sdpa: head dim must be 128 or 64")
    if scale is None:
        scale = 1.0 / (q.size(-1) ** 0.5)
    return torch.ops.b200k.sdpa(q, k, v, float(scale), bool(is_causal))


# ---------------------------------------------------------------------------------------------
# decode / paged decode
# ---------------------------------------------------------------------------------------------
def _check_table(name: str, table: Tensor, sequences) -> None:
    """As the CUDA implementations check it: rows kept for more sequences than the call's are fine."""
    torch._check(table.dtype == torch.int32 and table.dim() == 2 and table.size(0) >= sequences,
                 lambda: f"{name}: block_table must be int32 [num_seqs, max_pages]")


def _check_per_sequence(name: str, what: str, t: Tensor, sequences) -> None:
    torch._check(t.dtype == torch.int32 and sum(n != 1 for n in t.shape) <= 1 and t.numel() >= sequences,
                 lambda: f"{name}: {what} must be int32 [num_seqs]")


def _decode_common_checks(name: str, q: Tensor, kc: Tensor, vc: Tensor, lens: Tensor):
    torch._check(q.dim() == 3, lambda: f"{name}: q must be [num_seqs, q_heads, head_dim]")
    torch._check(q.dtype in _HALF_TYPES, lambda: f"{name}: dtype must be float16 or bfloat16, got {q.dtype}")
    torch._check(q.dtype == kc.dtype == vc.dtype, lambda: f"{name}: q and the KV cache must share a dtype")
    torch._check(q.size(2) in (64, 128), lambda: f"{name}: head dim must be 128 or 64")
    torch._check(kc.dim() == 4 and kc.shape == vc.shape, lambda: f"{name}: k and v caches must be 4-D and equal in shape")
    torch._check(kc.size(3) == q.size(2), lambda: f"{name}: cache head dim must equal q's")
    _check_per_sequence(name, "seq_lens", lens, q.size(0))
    torch._check(q.size(1) % kc.size(1) == 0 and q.size(1) // kc.size(1) <= 16,
                 lambda: f"{name}: query heads must be a multiple (at most 16x) of kv heads")


@CustomOp.register(library=LIBRARY, register_impl=False)
class decode_attention(CustomOp):
    """One query token per sequence against a contiguous KV history.

    q [num_seqs, Hq, D]; k, v [num_seqs, Hkv, max_len, D]; seq_lens int32 [num_seqs]
    (tokens t >= seq_lens[s] are ignored; D = 128 or 64).  Returns [num_seqs, Hq, D].
    """

    signature = (
        "decode_attention(Tensor q, Tensor k, Tensor v, Tensor seq_lens, float scale, int chunk_tokens=0) -> Tensor"
    )

    def select(self, sel: KernelSelection):
        q = sel.arg_tensor(0)
        k = sel.arg_tensor(1)
        v = sel.arg_tensor(2)
        lens = sel.arg_tensor(3)
        sel.attr_float(4)
        sel.attr_int(5)
        _decode_common_checks("decode_attention", q.t, k.t, v.t, lens.t)
        torch._check(k.t.size(0) >= q.t.size(0), lambda: "decode_attention: k must have one history per sequence")
        sel.return_new_tensor(list(q.t.shape), q.t.dtype)


@CustomOp.register(library=LIBRARY, register_impl=False)
class paged_decode_attention(CustomOp):
    """One query token per sequence against a paged KV cache.

    q [num_seqs, Hq, D]; k_cache, v_cache [num_pages, Hkv, page_size, D], D = 128 or 64;
    block_table int32 [num_seqs, max_pages]: physical page of logical page p of sequence s;
    seq_lens int32 [num_seqs].  Returns [num_seqs, Hq, D].
    """

    signature = (
        "paged_decode_attention(Tensor q, Tensor k_cache, Tensor v_cache, Tensor block_table, Tensor seq_lens, "
        "float scale, int chunk_tokens=0) -> Tensor"
    )

    def select(self, sel: KernelSelection):
        q = sel.arg_tensor(0)
        kc = sel.arg_tensor(1)
        vc = sel.arg_tensor(2)
        bt = sel.arg_tensor(3)
        lens = sel.arg_tensor(4)
        sel.attr_float(5)
        sel.attr_int(6)
        _decode_common_checks("paged_decode_attention", q.t, kc.t, vc.t, lens.t)
        _check_table("paged_decode_attention", bt.t, q.t.size(0))
        torch._check(kc.t.size(2) % 16 == 0, lambda: "paged_decode_attention: page size must be a multiple of 16")
        sel.return_new_tensor(list(q.t.shape), q.t.dtype)


@CustomOp.register(library=LIBRARY, register_impl=False)
class paged_gather(CustomOp):
    """out[s, h, t, :] = cache[block_table[s, t // page], h, t % page, :] for t < seq_lens[s].

    Uses the paged decode kernel's address function; rows beyond seq_lens[s] are zero.
    """

    signature = "paged_gather(Tensor cache, Tensor block_table, Tensor seq_lens, int max_seq_len) -> Tensor"

    def select(self, sel: KernelSelection):
        c = sel.arg_tensor(0)
        bt = sel.arg_tensor(1)
        lens = sel.arg_tensor(2)
        n = sel.attr_int(3)
        torch._check(c.t.dim() == 4, lambda: "paged_gather: cache must be [num_pages, heads, page_size, head_dim]")
        _check_table("paged_gather", bt.t, 0)
        _check_per_sequence("paged_gather", "seq_lens", lens.t, bt.t.size(0))
        sel.return_new_tensor([bt.t.size(0), c.t.size(1), n.v, c.t.size(3)], c.t.dtype)


@CustomOp.register(library=LIBRARY, register_impl=False)
class kv_append(CustomOp):
    """Writes new K/V rows into the paged cache through the block table (in place).

    ``k_new`` / ``v_new``: [num_seqs, new_tokens, kv_heads, head_dim]; row ``t`` of sequence ``s``
    goes to token position ``positions[s] + t``, i.e. to
    ``cache[block_table[s, p // page], h, p % page, :]``.  The pages must already be in the table.
    Same address function as the paged decode kernel.
    """

    signature = ("kv_append(Tensor k_new, Tensor v_new, Tensor(a!) k_cache, Tensor(b!) v_cache, "
                 "Tensor block_table, Tensor positions) -> ()")

    def select(self, sel: KernelSelection):
        kn = sel.arg_tensor(0)
        vn = sel.arg_tensor(1)
        kc = sel.arg_tensor(2)
        vc = sel.arg_tensor(3)
        bt = sel.arg_tensor(4)
        pos = sel.arg_tensor(5)
        torch._check(kn.t.dim() == 4 and vn.t.shape == kn.t.shape,
                     lambda: "kv_append: k_new and v_new must be [num_seqs, new_tokens, kv_heads, head_dim]")
        torch._check(kc.t.dim() == 4 and vc.t.shape == kc.t.shape,
                     lambda: "kv_append: caches must be [num_pages, kv_heads, page_size, head_dim]")
        torch._check(kc.t.dtype == kn.t.dtype and vc.t.dtype == kn.t.dtype and vn.t.dtype == kn.t.dtype,
                     lambda: "kv_append: dtypes of new rows and caches must match")
        torch._check(kn.t.size(2) == kc.t.size(1) and kn.t.size(3) == kc.t.size(3),
                     lambda: "kv_append: heads / head_dim of new rows and caches must match")
        _check_table("kv_append", bt.t, kn.t.size(0))
        _check_per_sequence("kv_append", "positions", pos.t, kn.t.size(0))


@CustomOp.register(library=LIBRARY, register_impl=False)
class paged_attention(CustomOp):
    """Attention forward (prefill) over a paged K/V cache.

    q [B, Hq, Sq, 128]; caches [num_pages, Hkv, page_size, 128]; block_table int32 [B, max_pages];
    seq_lens int32 [B] = number of keys of each sequence.  The Sq queries of a sequence are its last
    Sq tokens (append their K/V first, see ``kv_append``); with ``is_causal`` query i sees keys
    j <= i + seq_lens[b] - Sq.  Rows of a sequence's last page past its length must be finite.
    """

    signature = ("paged_attention(Tensor q, Tensor k_cache, Tensor v_cache, Tensor block_table, Tensor seq_lens, "
                 "float scale, bool is_causal) -> Tensor")

    def select(self, sel: KernelSelection):
        q = sel.arg_tensor(0)
        kc = sel.arg_tensor(1)
        vc = sel.arg_tensor(2)
        bt = sel.arg_tensor(3)
        lens = sel.arg_tensor(4)
        sel.attr_float(5)
        sel.attr_bool(6)
        torch._check(q.t.dim() == 4 and q.t.size(3) in (64, 128), lambda: "paged_attention: q must be [B, Hq, Sq, 128 or 64]")
        torch._check(q.t.dtype in _HALF_TYPES, lambda: f"paged_attention: dtype must be float16 or bfloat16, got {q.t.dtype}")
        torch._check(kc.t.dim() == 4 and kc.t.shape == vc.t.shape and kc.t.size(3) == q.t.size(3),
                     lambda: "paged_attention: caches must be [num_pages, Hkv, page_size, head dim of q] and equal in shape")
        torch._check(kc.t.dtype == q.t.dtype and vc.t.dtype == q.t.dtype, lambda: "paged_attention: dtypes must match")
        torch._check(kc.t.size(2) in (16, 32, 64, 128), lambda: "paged_attention: page_size must be 16, 32, 64 or 128")
        torch._check(q.t.size(1) % kc.t.size(1) == 0, lambda: "paged_attention: query heads must be a multiple of kv heads")
        _check_table("paged_attention", bt.t, q.t.size(0))
        _check_per_sequence("paged_attention", "seq_lens", lens.t, q.t.size(0))
        sel.return_tensor(_attention_out_like(q.t, "meta"))

