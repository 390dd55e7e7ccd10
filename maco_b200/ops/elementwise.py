"""Element-wise and row-wise operators backed by this package's CUDA kernels (csrc/elementwise.cuh).

These are the stand-alone launches; the same device code runs as tasks inside the persistent
kernel. Reference counterparts: the device tasks of maco/csrc/maco_worker.cuh:66-177.
"""
from __future__ import annotations

import ctypes
from typing import Optional

import torch

from .. import _native as N

T_LAYERNORM, T_RMSNORM, T_GELU, T_SILU, T_SOFTMAX, T_SILU_GATE, T_ROPE = 103, 104, 105, 106, 107, 108, 109
T_SCALE, T_ADD, T_GELU_BWD, T_AXPBY, T_COPY = 112, 113, 114, 115, 300

_declared = False


def _fn():
    global _declared
    lib = N.lib()
    if not _declared:
        P, I, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
        lib.maco_elementwise.restype = I
        lib.maco_elementwise.argtypes = [I, P, P, P, P, I, I, I, I, I, F, F, I, I, P]
        _declared = True
    return lib.maco_elementwise


def _rows2d(t: torch.Tensor) -> torch.Tensor:
    if t.dim() == 0:
        t = t.reshape(1, 1)
    t2 = t.reshape(-1, t.shape[-1]) if t.is_contiguous() else t.contiguous().reshape(-1, t.shape[-1])
    return t2


def _launch(kind: int, x: torch.Tensor, in1=None, in2=None, out: Optional[torch.Tensor] = None, f0=0.0, f1=0.0,
            i0=0, i1=0, rows=None, cols=None, ld=None) -> torch.Tensor:
    if not x.is_cuda:
        raise ValueError("maco_b200 element-wise operators need CUDA tensors")
    if x.dtype not in N.DTYPE_CODE:
        raise ValueError(f"unsupported dtype {x.dtype}")
    xc = x if x.is_contiguous() else x.contiguous()
    if out is None:
        out = torch.empty_like(xc)
    if not out.is_contiguous():
        raise ValueError("out must be contiguous")
    if xc.numel() == 0:
        return out
    c = cols if cols is not None else xc.shape[-1]
    r = rows if rows is not None else xc.numel() // c
    a1 = in1.contiguous() if in1 is not None else None
    a2 = in2.contiguous() if in2 is not None else None
    ld = ld if ld is not None else c
    rc = _fn()(kind, xc.data_ptr(), N.ptr(a1), N.ptr(a2), out.data_ptr(), r, c, N.DTYPE_CODE[x.dtype], ld, ld,
               float(f0), float(f1), int(i0), int(i1), N.current_stream_ptr())
    N.check(rc, "maco_elementwise")
    return out


def _load_quick(kind, x, *rest):
    global _quick
    if not x.is_cuda:
        return None
    _quick = N.fastcall("elementwise")
    return _quick(kind, x, *rest)


# The ordinary call, plain contiguous tensors on the GPU, as one call into C; None: it is not one, and the general path decides.
# 4 x 512 bf16, host time of an RMSNorm: 8.3 us through Python and ctypes, 5.8 this way (2.6 the launch, 1.4 the result's allocation).
_quick = _load_quick


def _run(kind: int, x, in1, in2, out, f0, f1) -> torch.Tensor:
    res = _quick(kind, x, in1, in2, out, f0, f1)
    if res is None:
        return _launch(kind, x, in1=in1, in2=in2, out=out, f0=f0, f1=f1)
    if res.__class__ is int:
        N.check(res, "maco_elementwise")
    return res


def gelu(x, out=None): return _run(T_GELU, x, None, None, out, 0.0, 0.0)
def silu(x, out=None): return _run(T_SILU, x, None, None, out, 0.0, 0.0)
def softmax(x, out=None): return _run(T_SOFTMAX, x, None, None, out, 0.0, 0.0)
def scale(x, factor: float, out=None): return _run(T_SCALE, x, None, None, out, factor, 0.0)
def add(a, b, out=None): return _run(T_ADD, a, b, None, out, 0.0, 0.0)
def silu_gate(gate, up, out=None): return _run(T_SILU_GATE, gate, up, None, out, 0.0, 0.0)
def gelu_bwd(dy, pre, out=None): return _run(T_GELU_BWD, dy, pre, None, out, 0.0, 0.0)
def axpby(x, y, a: float, b: float, out=None): return _run(T_AXPBY, x, y, None, out, a, b)
def rmsnorm(x, weight, eps: float = 1e-6, out=None): return _run(T_RMSNORM, x, weight, None, out, eps, 0.0)
def layernorm(x, weight, bias, eps: float = 1e-5, out=None):
    return _run(T_LAYERNORM, x, weight, bias, out, eps, 0.0)


def rope(x: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor, out=None) -> torch.Tensor:
    """Half-rotation RoPE on [tokens, heads, head_dim]; cos/sin are [tokens, head_dim // 2]."""
    tokens, heads, hd = x.shape
    return _launch(T_ROPE, x, in1=cos.to(x.dtype), in2=sin.to(x.dtype), out=out, i0=heads, i1=0,
                   rows=tokens * heads, cols=hd, ld=heads * hd)


def qknorm_rope(x: torch.Tensor, weight: torch.Tensor, cos_sin: torch.Tensor, eps: float = 1e-6, out=None,
                token_offset: int = 0) -> torch.Tensor:
    """Per-head RMSNorm then RoPE on [tokens, heads, head_dim]; ``cos_sin`` is [tokens, head_dim]
    with cos in the first half of each row and sin in the second."""
    tokens, heads, hd = x.shape
    return _launch(T_ROPE, x, in1=weight, in2=cos_sin.to(x.dtype), out=out, f0=eps, f1=1.0, i0=heads,
                   i1=token_offset, rows=tokens * heads, cols=hd, ld=heads * hd)


def mse_gelu_bwd(a: torch.Tensor, target: torch.Tensor, z: torch.Tensor, out: torch.Tensor, factor: float,
                 stream: Optional[torch.cuda.Stream] = None) -> torch.Tensor:
    """``out = factor * (a - target) * gelu'(z)``: gradient of a mean-squared error through the last layer's GELU, in one pass.
    Contiguous 16-bit tensors of one shape and type."""
    for t in (target, z, out):
        if t.shape != a.shape or t.dtype != a.dtype or t.device != a.device:
            raise ValueError("mse_gelu_bwd: tensors of one shape, type and device")
    if not a.is_cuda or not all(t.is_contiguous() for t in (a, target, z, out)):
        raise ValueError("mse_gelu_bwd: contiguous CUDA tensors only")
    lib = N.lib()
    rc = lib.maco_mse_gelu_bwd(ctypes.c_void_p(a.data_ptr()), ctypes.c_void_p(target.data_ptr()), ctypes.c_void_p(z.data_ptr()),
                               ctypes.c_void_p(out.data_ptr()), ctypes.c_longlong(a.numel()), N.DTYPE_CODE[a.dtype], ctypes.c_float(factor),
                               ctypes.c_void_p(N.current_stream_ptr(stream)))
    N.check(rc, "maco_mse_gelu_bwd")
    return out
