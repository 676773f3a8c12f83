"""ctypes glue for the sm_100a attention backward (csrc/attention_sm100.cu).

The backward needs scratch memory beyond its inputs and outputs: ``delta = rowsum(dO * O)``,
one fp32 per query row and head, which both backward kernels read, and, when the dK/dV kernel
splits the query heads of a KV head over several CTAs (few KV heads per GPU), their fp32
partial sums.  The scratch is taken from a small per-device cache here so that the hot path
does not allocate.
"""
from __future__ import annotations

import ctypes
import math
from ctypes import c_float, c_int, c_int64, c_void_p

import torch

from .. import kernels as K

_scratch = {}


def _scratch_for(device, nbytes: int):
    key = (device.index, K.current_raw_stream(device))
    buf = _scratch.get(key)
    if buf is None or buf.numel() < nbytes:
        buf = torch.empty(nbytes, dtype=torch.uint8, device=device)
        _scratch[key] = buf
    return buf


def attn_bwd_native(dout, q, k, v, out, lse, dq, dk, dv, causal, scale, sm_budget=0, stream=None):
    Sq, B, Hq, d = q.shape
    Sk, Hk = k.shape[0], k.shape[2]
    for t in (dout, q, k, v, out, dq, dk, dv):
        assert t.stride(3) == 1 and t.dtype == torch.bfloat16
    nbytes_fn = K.proto("dh_attn_bwd_scratch_bytes", [c_int, c_int, c_int, c_int, c_int], c_int64)
    scratch = _scratch_for(q.device, nbytes_fn(B, Hq, Hk, Sq, Sk))
    strides = []
    for t in (dout, q, k, v, out, dq, dk, dv):
        strides += [t.stride(0), t.stride(1), t.stride(2)]
    arr = (c_int64 * 24)(*strides)
    fn = K.proto("dh_attn_bwd", [c_void_p] * 10 + [ctypes.POINTER(c_int64), c_int, c_int, c_int, c_int, c_int, c_int, c_int,
                                                   c_float, c_int, c_void_p])
    K.check(fn(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), dq.data_ptr(),
               dk.data_ptr(), dv.data_ptr(), scratch.data_ptr(), arr, B, Hq, Hk, Sq, Sk, d, 1 if causal else 0, scale,
               sm_budget, K.stream_ptr(stream)), "dh_attn_bwd")


def _packed_offsets(cu):
    return (c_int * len(cu))(*cu)


def _packed_strides(operands, d, device):
    """``(row, head)`` strides of ``(tensor, heads)`` pairs.  The kernels see addresses and strides only: that these are bf16 rows of
    ``[T, heads, d]`` on one device is made sure of here."""
    strides = []
    for t, heads in operands:
        _, h, c = t.shape
        row, head, column = t.stride()
        assert h == heads and c == d and column == 1 and t.dtype == torch.bfloat16 and t.get_device() == device
        strides.append((row, head))
    return strides


def attn_fwd_packed(q, k, v, cq, ck, max_q, causal, scale, sm_budget=0, stream=None):
    """Packed batch in one launch: ``q [Tq, Hq, d]``, ``k, v [Tk, Hk, d]``, offsets as Python lists that ascend (checked by
    the caller); rows past the last sequence are not looked at.  Returns ``(out like q, lse [b, Hq, max_q])``; statistics past a
    sequence's end are ``-inf``."""
    Tq, Hq, d = q.shape
    Tk, Hk = min(k.shape[0], v.shape[0]), k.shape[1]
    out = torch.empty_like(q)
    strides = _packed_strides(((q, Hq), (k, Hk), (v, Hk), (out, Hq)), d, q.get_device())
    assert cq[-1] <= Tq and ck[-1] <= Tk
    scale = scale if scale is not None else 1.0 / math.sqrt(d)
    b = len(cq) - 1
    whole = all(cq[i + 1] - cq[i] == max_q for i in range(b))
    shape = (b, Hq, max_q)
    lse = torch.empty(shape, dtype=torch.float32, device=q.device) if whole else \
        torch.full(shape, float("-inf"), dtype=torch.float32, device=q.device)
    if Tk == 0:                                  # no key anywhere, nothing to launch
        return out.zero_(), lse.fill_(float("-inf"))
    fn = K.proto("dh_attn_fwd_packed", [c_void_p] * 5 + [ctypes.POINTER(c_int64), c_int, ctypes.POINTER(c_int), ctypes.POINTER(c_int),
                                                         c_int, c_int, c_int, c_int, c_int, c_int, c_int, c_float, c_int, c_void_p])
    K.check(fn(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), (c_int64 * 8)(*(s for p in strides for s in p)), b,
               _packed_offsets(cq), _packed_offsets(ck), Tq, Tk, max_q, Hq, Hk, d, 1 if causal else 0, scale, sm_budget,
               K.stream_ptr(stream)), "dh_attn_fwd_packed")
    return out, lse


def attn_bwd_packed(dout, q, k, v, out, lse, dq, dk, dv, cq, ck, causal, scale, sm_budget=0, stream=None):
    """Backward of ``attn_fwd_packed`` into ``dq, dk, dv``."""
    Hq, d, Hk, device = q.shape[1], q.shape[2], k.shape[1], q.get_device()
    strides = []
    for row, head in _packed_strides(((dout, Hq), (q, Hq), (k, Hk), (v, Hk), (out, Hq), (dq, Hq), (dk, Hk), (dv, Hk)), d, device):
        strides += (row, row, head)
    Tq, Tk = min(t.shape[0] for t in (q, dout, out, dq)), min(t.shape[0] for t in (k, v, dk, dv))
    assert cq[-1] <= Tq and ck[-1] <= Tk and lse.dtype == torch.float32 and lse.get_device() == device
    if Tq == 0 or Tk == 0:
        for t in (dq, dk, dv):
            t.zero_()
        return
    scale = scale if scale is not None else 1.0 / math.sqrt(d)
    lse = lse.contiguous()
    b = len(cq) - 1
    cu_q, cu_k = _packed_offsets(cq), _packed_offsets(ck)
    p_int = ctypes.POINTER(c_int)
    nbytes = K.proto("dh_attn_bwd_packed_scratch_bytes", [c_int, p_int, c_int, c_int, c_int, c_int], c_int64)
    scratch = _scratch_for(q.device, nbytes(b, cu_k, Hq, Hk, Tq, Tk))
    fn = K.proto("dh_attn_bwd_packed", [c_void_p] * 10 + [ctypes.POINTER(c_int64), c_int, p_int, p_int, c_int, c_int, c_int, c_int, c_int,
                                                          c_int, c_int, c_float, c_int, c_void_p])
    K.check(fn(dout.data_ptr(), q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), lse.data_ptr(), dq.data_ptr(),
               dk.data_ptr(), dv.data_ptr(), scratch.data_ptr(), (c_int64 * 24)(*strides), b, cu_q, cu_k, Tq, Tk, lse.shape[2], Hq,
               Hk, d, 1 if causal else 0, scale, sm_budget, K.stream_ptr(stream)), "dh_attn_bwd_packed")
