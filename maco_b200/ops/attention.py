"""Split-KV decode attention for grouped-query attention (head_dim 128, up to 8 query heads per KV
head). The kernel streams each K and V row once; see csrc/attention_decode.cuh. The reference has
no attention kernel (its example materialises softmax(QK^T)V, examples/test_overlap_attention.py:111-113).
"""
from __future__ import annotations

import ctypes
from typing import Optional, Tuple

import torch

from .. import _native as N

_declared = False


def _lib():
    global _declared
    lib = N.lib()
    if not _declared:
        P, I, LL, F = ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong, ctypes.c_float
        lib.maco_attention_decode.restype = I
        lib.maco_attention_decode.argtypes = [P, P, P, P, P, I, I, I, I, I, I, I, LL, LL, F, P]
        lib.maco_attention_decode_stream.restype = I
        lib.maco_attention_decode_stream.argtypes = [P, P, P, P, P, I, I, I, I, I, LL, LL, F, P]
        lib.maco_attention_stream_scratch_bytes.restype = ctypes.c_ulonglong
        lib.maco_attention_stream_scratch_bytes.argtypes = [I]
        lib.maco_attention_decode_scratch_bytes.restype = ctypes.c_ulonglong
        lib.maco_attention_decode_scratch_bytes.argtypes = [I, I, I, I]
        _declared = True
    return lib


def default_splits(batch: int, kv_heads: int, seq: int) -> int:
    """Enough (batch, head, split) tasks to cover the SMs about twice, at least 256 keys per split."""
    sms = torch.cuda.get_device_properties(torch.cuda.current_device()).multi_processor_count
    want = max(1, (2 * sms + batch * kv_heads - 1) // (batch * kv_heads))
    return max(1, min(want, max(1, seq // 256), 32))


def _kv_strides(cache: torch.Tensor) -> Optional[Tuple[int, int]]:
    """(batch, head) strides of a cache [B, Hkv, S, D] with contiguous rows, None if its rows are not. A dimension of size 1 has
    no stride worth comparing or handing on: it counts as contiguous, whatever tensor it was cut from."""
    B, H, S, D = cache.shape
    sb, sh, sr, sd = cache.stride()
    if (D > 1 and sd != 1) or (S > 1 and sr != D):
        return None
    head = sh if H > 1 else S * D
    return (sb if B > 1 else H * head), head


def _stream_form(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: torch.Tensor, scale: float, kv_len: int) -> bool:
    """One launch of the streaming kernel (csrc/attention_api.cu) plus its merge; False when the caches cannot be addressed
    by a tensor map."""
    lib = _lib()
    B, Hq, D = q.shape
    Hkv = k.shape[1]
    scratch = torch.empty(lib.maco_attention_stream_scratch_bytes(Hq // Hkv) // 4, dtype=torch.float32, device=q.device)
    sb, sh = _kv_strides(k)
    rc = lib.maco_attention_decode_stream(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), scratch.data_ptr(), B, Hq, Hkv, kv_len,
                                          N.DTYPE_CODE[q.dtype], sb, sh, scale, N.current_stream_ptr())
    if rc == -2:
        return False
    N.check(rc, "maco_attention_decode_stream")
    return True


def attention_decode_tensor_core(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, out: torch.Tensor, *,
                                 scale: Optional[float] = None, kv_len: Optional[int] = None) -> torch.Tensor:
    """Decode attention on the tensor cores: contiguous 16-bit ``q`` [B, Hq, 128], ``k``/``v`` [B, Hkv, S, 128], ``out``
    [B, Hq, 128]; the first ``kv_len`` keys (default: all). The kernel addresses the caches by ``kv_len`` and by ``k``'s
    strides alone, so everything it takes for granted is checked here."""
    B, Hq, D = q.shape
    _, Hkv, S, _ = k.shape
    kv_len = S if kv_len is None else int(kv_len)
    if D != 128 or Hq % Hkv or Hq // Hkv > 8 or not 1 <= kv_len <= S:
        raise ValueError("attention_decode: head_dim 128, at most 8 query heads per kv head, 1 <= kv_len <= cache length")
    if tuple(k.shape) != (B, Hkv, S, D) or v.shape != k.shape or out.numel() != q.numel() or {k.dtype, v.dtype, out.dtype} != {q.dtype}:
        raise ValueError("attention_decode: q and out [B, Hq, 128], k and v [B, Hkv, S, 128], one data type")
    if not (q.is_contiguous() and k.is_contiguous() and v.is_contiguous() and out.is_contiguous()):
        raise ValueError("attention_decode: contiguous tensors only")
    if not _stream_form(q, k, v, out, float(scale if scale is not None else D ** -0.5), kv_len):
        N.check(-2, "maco_attention_decode_stream")
    return out


def _load_quick(q, *rest):
    global _quick
    if not q.is_cuda:
        return None
    _lib()
    _quick = N.fastcall("attention")
    return _quick(q, *rest)


_quick = _load_quick       # the ordinary call as one call into C (csrc/py/fastcall.c); None: not an ordinary one


def attention_decode(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, *, scale: Optional[float] = None,
                     splits: Optional[int] = None, out: Optional[torch.Tensor] = None,
                     scratch: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``q`` [B, Hq, 128], ``k``/``v`` [B, Hkv, S, 128] (last two dims contiguous) -> [B, Hq, 128].
    Without an explicit ``splits`` / ``scratch`` the call streams K and V through the tensor cores, one equal share per
    SM; with one of them it runs the CUDA-core kernel with that many splits (into that scratch). Scores, softmax and sums are
    fp32 in both, and so are the probabilities (on the tensor cores each is the sum of two values of the operand type)."""
    if splits is None and scratch is None:
        res = _quick(q, k, v, out, 128 ** -0.5 if scale is None else scale)
        if res.__class__ is int:
            N.check(res, "maco_attention_decode_stream")
        if res is not None:
            return res
    B, Hq, D = q.shape
    _, Hkv, S, _ = k.shape
    strides = _kv_strides(k)
    if k.shape != v.shape or k.shape[3] != D or k.shape[0] < B or strides is None or strides != _kv_strides(v):
        raise ValueError("k and v must share a [B, Hkv, S, 128] layout with contiguous rows")
    q = q.contiguous()
    sm_scale = float(scale if scale is not None else D ** -0.5)
    if splits is None and scratch is None and D == 128 and S > 0 and Hq % Hkv == 0 and Hq // Hkv <= 8 and (out is None or out.is_contiguous()):
        res = out if out is not None else torch.empty_like(q)
        if _stream_form(q, k, v, res, sm_scale, S):
            return res
    splits = splits or default_splits(B, Hkv, S)
    lib = _lib()
    need = lib.maco_attention_decode_scratch_bytes(B, Hq, Hkv, splits)
    if scratch is None:
        scratch = torch.empty(need // 4, dtype=torch.float32, device=q.device)
    elif scratch.numel() * scratch.element_size() < need:
        raise ValueError(f"scratch too small: need {need} bytes")
    if out is None:
        out = torch.empty_like(q)
    rc = lib.maco_attention_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), scratch.data_ptr(), B, Hq,
                                   Hkv, S, D, splits, N.DTYPE_CODE[q.dtype], strides[0], strides[1], sm_scale, N.current_stream_ptr())
    N.check(rc, "maco_attention_decode")
    return out
