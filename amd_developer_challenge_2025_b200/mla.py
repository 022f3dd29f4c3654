"""Host side of the two custom kernels around the KV down-projection of the reference's MLA-decode
submission, plus that projection itself as an FP8 block-scaled GEMM.

`mla_decode` and `div_softmax` keep the names, argument order and meaning of the reference's pybind module
(3-amd-mla-decode/amd-mla-submission.py:7-11, 110-125, 221-225); the work is done by sm_100a CUDA kernels in
lib/libb200fp8mm.so reached through the C ABI of include/b200_mla_consumers.h. There is no CPU path."""
from __future__ import annotations

import torch

from . import _lib
from .fp8_mm import Fp8MmError, _check, fp8_mm


def _check_range(name, t, off, d0, d1, d2, s1, s2):
    """Every element off + i0*s1 + i1*s2 + j (strides of either sign) lies inside the bf16 tensor's storage."""
    first = last = off + t.storage_offset()
    for span in ((d0 - 1) * s1, (d1 - 1) * s2):
        if span < 0:
            first += span
        else:
            last += span
    _check(off >= 0 and first >= 0 and last + d2 <= t.untyped_storage().nbytes() // 2, f"{name}: range outside the tensor")


def mla_decode(x, y, pos: int, xoff: int, yoff: int, d0: int, d1: int, d2: int, xs1: int, xs2: int, ys1: int,
               ys2: int):
    """Rotary position embedding, the reference's `module.mla_decode`: reads the bf16 elements
    x.data_ptr() + xoff + i0*xs1 + i1*xs2 + j and writes the rotated values to y at yoff + i0*ys1 + i1*ys2 + j
    (i0 < d0, i1 < d1, j < d2; row i1 has position pos + i1). y may be x. Runs on the current stream."""
    if _lib.host_calls().mla_decode(x, y, pos, xoff, yoff, d0, d1, d2, xs1, xs2, ys1, ys2):
        return y
    # Not the plain case, or a call that will be refused: the same checks here, with their errors.
    _check(x.is_cuda and y.is_cuda and x.device == y.device, "x and y must be CUDA tensors on one device")
    _check(x.dtype == torch.bfloat16 and y.dtype == torch.bfloat16, "x and y must be bfloat16")
    _check(d0 > 0 and d1 > 0 and d2 > 0 and d2 % 2 == 0, "d0, d1, d2 must be positive and d2 even")
    _check_range("x", x, xoff, d0, d1, d2, xs1, xs2)
    _check_range("y", y, yoff, d0, d1, d2, ys1, ys2)
    with torch.cuda.device(x.device):
        rc = _lib.load().b200_mla_rope(x.data_ptr() + 2 * xoff, y.data_ptr() + 2 * yoff, pos, d0, d1, d2, xs1, xs2, ys1,
                                       ys2, torch.cuda.current_stream(x.device).cuda_stream)
    if rc != 0:
        raise Fp8MmError(rc, "mla_decode (rope)")
    return y


def div_softmax(qk, bs: int, nh: int, sl: int, dnope: int, drope: int):
    """In-place softmax(qk / sqrt(dnope + drope)) over the last dimension of the contiguous bf16 tensor
    qk [bs, nh, sl], the reference's `module.div_softmax`. Runs on the current stream."""
    if _lib.host_calls().div_softmax(qk, bs, nh, sl, dnope, drope):
        return qk
    _check(qk.is_cuda and qk.dtype == torch.bfloat16 and qk.is_contiguous(), "qk must be a contiguous bfloat16 CUDA tensor")
    _check(qk.numel() == bs * nh * sl and bs > 0 and nh > 0 and sl > 0, "qk must hold bs * nh * sl elements")
    with torch.cuda.device(qk.device):
        rc = _lib.load().b200_mla_div_softmax(qk.data_ptr(), bs, nh, sl, dnope, drope,
                                              torch.cuda.current_stream(qk.device).cuda_stream)
    if rc != 0:
        raise Fp8MmError(rc, "div_softmax")
    return qk


def kv_down_projection_fp8(x, x_scale, w_dkv, w_scale, out=None):
    """The KV down-projection `x @ wDKV.T` (3-amd-mla-decode/amd-mla-submission.py:269; [bs, d] x [dkv + drope, d],
    i.e. N = 576, K = 7168 for the reference's model) as the FP8 block-scaled GEMM of this package: x and w_dkv
    in e4m3fn with fp32 scales per (row, 128 of K) and per (128 rows of w, 128 of K). Returns bf16 [bs, dkv + drope]
    (the row the reference writes into its KV cache)."""
    if out is None:
        out = torch.empty(x.shape[0], w_dkv.shape[0], dtype=torch.bfloat16, device=x.device)
    return fp8_mm(x, w_dkv, x_scale, w_scale, out)
