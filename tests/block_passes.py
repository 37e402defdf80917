"""The row and column passes of a transformer block (include/na1d_b200.h) on torch tensors, one call each: what the autograd node
chains, for tests of the single passes."""
import ctypes

import torch

from pcf_nat_b200 import _lib
from pcf_nat_b200._lib import check
from pcf_nat_b200.block import _CODE, _L, _stream


def layer_norm(x, dx, w, b, eps, stats):
    """(y, s, mean, rstd): y = LN(s) with s = x, or x + dx rounded to x's dtype; mean and rstd are None without ``stats``."""
    rows, D = x.numel() // x.shape[-1], x.shape[-1]
    y = torch.empty_like(x)
    s = x if dx is None else torch.empty_like(x)
    mean = rstd = None
    if stats:
        mean, rstd = torch.empty((2, (rows + 3) // 4 * 4), dtype=torch.float32, device=x.device)
    check(_L.na1d_layer_norm_forward(y.data_ptr(), None if dx is None else s.data_ptr(), mean.data_ptr() if stats else None,
                                     rstd.data_ptr() if stats else None, x.data_ptr(), None if dx is None else dx.data_ptr(),
                                     w.data_ptr(), b.data_ptr(), rows, D, eps, _CODE[x.dtype], _stream(x)), "na1d_layer_norm_forward")
    return y, s, mean, rstd


def scratch_for(rows, D, F, device):
    return torch.empty(_L.na1d_block_scratch_floats(rows, D, F), dtype=torch.float32, device=device)


def layer_norm_backward(dy, s, mean, rstd, w, res, scratch):
    """(ds, sums): ds = LN'(dy) + res, sums (3, D) = gradients of w and b, column sums of ds."""
    rows, D = s.numel() // s.shape[-1], s.shape[-1]
    ds = torch.empty_like(s)
    sums = torch.empty((3, D), dtype=torch.float32, device=s.device)
    check(_L.na1d_layer_norm_backward(ds.data_ptr(), sums.data_ptr(), scratch.data_ptr(), dy.data_ptr(), s.data_ptr(), mean.data_ptr(),
                                      rstd.data_ptr(), w.data_ptr(), None if res is None else res.data_ptr(), rows, D, _CODE[s.dtype],
                                      _stream(s)), "na1d_layer_norm_backward")
    return ds, sums


def gelu(x):
    y = torch.empty_like(x)
    check(_L.na1d_gelu_forward(y.data_ptr(), x.data_ptr(), x.numel(), _CODE[x.dtype], _stream(x)), "na1d_gelu_forward")
    return y


def gelu_backward(dy, x, scratch):
    """(dx, column sums of dx)."""
    F = x.shape[-1]
    dx = torch.empty_like(x)
    sums = torch.empty(F, dtype=torch.float32, device=x.device)
    check(_L.na1d_gelu_backward(dx.data_ptr(), sums.data_ptr(), scratch.data_ptr(), dy.data_ptr(), x.data_ptr(), x.numel() // F, F,
                                _CODE[x.dtype], _stream(x)), "na1d_gelu_backward")
    return dx, sums


def column_sums(x, scratch):
    F = x.shape[-1]
    sums = torch.empty(F, dtype=torch.float32, device=x.device)
    check(_L.na1d_column_sums(sums.data_ptr(), scratch.data_ptr(), x.data_ptr(), x.numel() // F, F, _CODE[x.dtype], _stream(x)),
          "na1d_column_sums")
    return sums


def cast_parameters(params, dtype):
    """The fp32 tensors rounded to ``dtype``: views of one buffer, written by one launch (at most 16 tensors)."""
    n = len(params)
    sizes = [p.numel() for p in params]
    offs, total = [], 0
    for k in sizes:
        offs.append(total)
        total += (k + 63) // 64 * 64      # 128-byte slots
    buf = torch.empty(total, dtype=dtype, device=params[0].device)
    check(_L.na1d_cast_parameters(buf.data_ptr(), (ctypes.c_void_p * n)(*(p.data_ptr() for p in params)), (ctypes.c_int64 * n)(*offs),
                                  (ctypes.c_int64 * n)(*sizes), n, _CODE[dtype], _stream(buf)), "na1d_cast_parameters")
    return buf, offs
