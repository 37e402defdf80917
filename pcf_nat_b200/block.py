"""The transformer block and the statistics pooling of the extractor as single autograd nodes on the library's kernels.

Between the four projections of a block (models/PCF_NATransformer.py:228-303: x + NA(LN(x)); x + MLP(LN(x))) PyTorch's autocast
runs a kernel per LayerNorm, addition, GELU, cast of a parameter and bias gradient. Here each of them is part of a
pass that has to touch the tensor anyway: the residual addition happens inside the LayerNorm that follows it or at the end of the MLP,
which is one kernel forward and one backward where its sizes allow (256 channels), a block's eight projection parameters are rounded to
16 bits by one launch, the weight and bias gradients of a branch come from one. The remaining products are library GEMMs, the attention
is the fused operator on the packed projection output.

Rounding points are those of the autocast network: 16-bit activations and projection weights, fp32 statistics and sums; the
LayerNorm parameters and the weight gradients are not rounded to 16 bits on the way, nor is the gradient of GELU's values in the MLP's
backward kernel.
"""
import torch
import torch.nn as nn

from . import _lib, ops
from ._lib import check
from .nattention import NAttention, _plain_linear, global_hooks, hooked

_L = _lib.lib()
_CODE = {torch.bfloat16: _lib.NA1D_BF16, torch.float16: _lib.NA1D_FP16}


def _stream(t):
    return torch.cuda.current_stream(t.device).cuda_stream


# ------------------------------------------------------------------ the features of all stages side by side
def add_to_rows(out, x, dx=None):
    """out = x (+ dx), x dense (batch, T, D), out a slice of D columns of wider rows."""
    D = x.shape[-1]
    with ops._on_device(x.device):
        check(_L.na1d_add_to_rows(out.data_ptr(), out.stride(1), x.data_ptr(), None if dx is None else dx.data_ptr(), x.numel() // D, D,
                                  _CODE[x.dtype], _stream(x)), "na1d_add_to_rows")
    return out


def feature_rows(x, parts):
    """Room for ``parts`` tensors like the 16-bit CUDA tensor x (batch, T, D) side by side, or None where the stages cannot write
    into slices of it (gradients are wanted, another kind of tensor)."""
    if (type(x) is not torch.Tensor or not x.is_cuda or x.dtype not in _CODE or x.dim() != 3 or x.shape[-1] % 8 or torch.is_grad_enabled() or
            x.numel() == 0 or torch.compiler.is_compiling() or not ops.native.eager_mode() or global_hooks()):
        return None
    return torch.empty(x.shape[0], x.shape[1], parts * x.shape[2], dtype=x.dtype, device=x.device)


# ------------------------------------------------------------------ the block (its autograd node is in csrc/torch_nodes.cpp)
def _block_parameters(blk, x):
    """The parameters of a block in the order of the node's arguments, or None where the block is anything but the plain one
    on fp32 parameters (a replaced or hooked submodule, another dtype, an odd size): it then runs module by module."""
    from .model import NABlock       # (model.py imports this module)
    if type(blk) is not NABlock:     # a subclass or a wrapper has a forward of its own
        return None
    a, n1, n2, f1, f2 = blk.attn, blk.norm1, blk.norm2, blk.fc1, blk.fc2
    if type(a) is not NAttention or type(n1) is not nn.LayerNorm or type(n2) is not nn.LayerNorm or a._na1d_layout != "channels_last":
        return None
    if "forward" in a.__dict__ or any(type(m) is not nn.Linear for m in (a.qkv, a.proj, f1, f2)):
        return None
    mods = (blk, a, n1, n2, f1, f2, a.qkv, a.proj, a.attn_drop, a.proj_drop)
    if any(hooked(m) for m in mods) or any("forward" in m.__dict__ for m in mods):
        return None
    if type(a.attn_drop) is not nn.Dropout or type(a.proj_drop) is not nn.Dropout or a.dilation != 1:
        return None
    if a.training and a.attn_drop.p or a.proj_drop.training and a.proj_drop.p:     # (each by the flag that its dropout follows)
        return None
    ps = (a.qkv.weight, a.qkv.bias, a.proj.weight, a.proj.bias, f1.weight, f1.bias, f2.weight, f2.bias, n1.weight, n1.bias, n2.weight,
          n2.bias, a.relative_position_bias)
    dev, D = x.device, x.shape[-1]
    for p in ps:
        if p is None or type(p) not in (nn.Parameter, torch.Tensor) or p.dtype != torch.float32 or p.device != dev or not p.is_contiguous() or p.data_ptr() % 16:
            return None
    Fh, H = f1.weight.shape[0], a.num_heads
    if (D % 8 or D > 1024 or Fh % 8 or Fh > 1 << 20 or Fh * D > (2 ** 31 - 1) // 16 or D % H or n1.normalized_shape != (D,) or n2.normalized_shape != (D,) or ps[0].shape != (3 * D, D) or
            ps[2].shape != (D, D) or ps[4].shape != (Fh, D) or ps[6].shape != (D, Fh) or ps[12].numel() != H * a.win_size):
        return None
    return ps


def run_blocks(blocks, x, valid, out=None, training=None):
    """The blocks applied to the residual stream x (batch, T, D), or None where they have to run module by module.
    ``valid``: valid tokens per utterance (an integer tensor on any device) or None. ``out``: a slice of wider rows, (batch, T, D), that
    takes the result (no gradients). ``training``: the state every layer has to be in, where ``valid`` depends on it."""
    if (type(x) is not torch.Tensor or not x.is_cuda or x.dim() != 3 or x.numel() == 0 or torch.compiler.is_compiling() or
            not torch.is_autocast_enabled() or not ops.native.eager_mode() or torch.autograd.forward_ad._current_level >= 0):
        return None
    dt = torch.get_autocast_dtype("cuda")
    if x.dtype != dt or dt not in _CODE or global_hooks() or x.shape[0] * x.shape[1] * x.shape[2] >= 2 ** 31:
        return None
    B, T, D = x.shape
    plan = []
    for blk in blocks:
        ps = _block_parameters(blk, x)
        if ps is None or training is not None and blk.attn.training != training or B * T * ps[4].shape[0] > 2 ** 40:
            return None
        a = blk.attn
        C = D // a.num_heads
        # (the kernels that take dense rows of heads stand in where those on the packed projection do not take the shape; larger ones are left
        # to the modules, which refuse what no kernel takes)
        if not ops.packed_supported(a.num_heads, T, C, a.win_size, a.left, 1, dt) and (
                C not in (8, 16, 24, 32, 48, 64, 96, 128) or a.win_size > 128 or a.num_heads * a.win_size > 4096 or B > 65535 or
                B * a.num_heads * T * a.win_size >= 2 ** 31):
            return None
        plan.append((ps, (a.num_heads, a.win_size, a.left, float(a.scale)), (blk.norm1.eps, blk.norm2.eps)))
    x, dx = x.contiguous(), None
    if x.data_ptr() % 16:
        return None
    if valid is not None:
        valid = valid.to(device=x.device, dtype=torch.int32)      # (one copy for all blocks)
    for i, (ps, cfg, eps) in enumerate(plan):
        y = ops.native.block(x, dx, valid, *cfg, *eps, ps, out if i + 1 == len(plan) else None)
        if y is None:                                             # (the first block, or none: they are given the same lengths)
            return None
        x, dx = y
    if out is not None:
        return x if x is out or x.data_ptr() == out.data_ptr() else add_to_rows(out, x, dx)
    return x if dx is None else x + dx


# ------------------------------------------------------------------ a projection of the features so far
def fuse(linear, feats):
    """``linear(torch.cat(feats, -1))`` as one node, for a backward pass: the result and the features as what comes next has to read
    them, so that their gradients are summed inside its products; None where it has to run in PyTorch's operations."""
    x = feats[0]
    if (not torch.is_grad_enabled() or type(x) is not torch.Tensor or not x.is_cuda or x.dim() != 3 or x.numel() == 0 or torch.compiler.is_compiling() or
            not torch.is_autocast_enabled() or not ops.native.eager_mode() or torch.autograd.forward_ad._current_level >= 0 or global_hooks()):
        return None
    dt = torch.get_autocast_dtype("cuda")
    if x.dtype != dt or dt not in _CODE or not _plain_linear(linear):
        return None
    w, b = linear.weight, linear.bias
    for p in (w, b):
        if (p is None or type(p) not in (nn.Parameter, torch.Tensor) or p.dtype != torch.float32 or p.device != x.device or not p.is_contiguous() or
                p.data_ptr() % 16):
            return None
    for f in feats:
        if type(f) is not torch.Tensor or f.shape != x.shape or f.dtype != dt or f.device != x.device or not f.is_contiguous() or f.data_ptr() % 16:
            return None
    D, K = x.shape[-1], x.shape[-1] * len(feats)
    if (D % 8 or w.shape[0] % 8 or w.shape[1] != K or b.shape != w.shape[:1] or K > 1 << 20 or w.shape[0] > 1 << 20 or w.numel() > (2 ** 31 - 1) // 16 or
            x.shape[0] * x.shape[1] * max(K, w.shape[0]) >= 2 ** 31):
        return None
    y, *rest = ops.native.fuse(w, b, list(feats))
    return y, rest


# ------------------------------------------------------------------ statistics pooling
def weighted_stats(logits, x, floor):
    """The pooling in PyTorch's operations."""
    w = torch.softmax(logits.float(), dim=1)
    xf = x.float()
    mu = (w * xf).sum(1)
    var = (w * xf * xf).sum(1) - mu * mu
    return torch.cat([mu, var.clamp_min(floor).sqrt()], dim=1)


def _pool_gradients(logits, x, d_out, floor):
    """The backward pass in PyTorch's operations, for a backward that is differentiated again (create_graph)."""
    w = torch.softmax(logits.float(), dim=1)
    xf = x.float()
    mu, e2 = (w * xf).sum(1, keepdim=True), (w * xf * xf).sum(1, keepdim=True)
    var = e2 - mu * mu
    d_mu, d_std = d_out.unsqueeze(1).chunk(2, dim=-1)
    d_var = torch.where(var < floor, 0.0, 0.5 * d_std / var.clamp_min(floor).sqrt())
    d_mu = d_mu - 2 * mu * d_var
    q = xf * (d_mu + xf * d_var)
    d_logits = w * (q - (mu * d_mu + e2 * d_var))
    return d_logits.to(logits.dtype), (w * (d_mu + 2 * xf * d_var)).to(x.dtype)


class _StatsPoolFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, x, floor):
        N, T, C = x.shape
        out = torch.empty((N, 2 * C), dtype=torch.float32, device=x.device)
        stats = torch.empty((3, N, C), dtype=torch.float32, device=x.device)
        with ops._on_device(x.device):
            check(_L.na1d_stats_pool_forward(out.data_ptr(), stats.data_ptr(), logits.data_ptr(), x.data_ptr(), C, N, T, C, floor,
                                             _CODE[x.dtype], _stream(x)), "na1d_stats_pool_forward")
        ctx.save_for_backward(logits, x, out, stats)
        ctx.floor = floor
        return out

    @staticmethod
    def backward(ctx, d_out):
        logits, x, out, stats = ctx.saved_tensors
        if torch.is_grad_enabled():
            return _pool_gradients(logits, x, d_out, ctx.floor) + (None,)
        N, T, C = x.shape
        d_out = d_out.contiguous()
        if d_out.data_ptr() % 16:
            d_out = d_out.clone()
        d_logits, dx = torch.empty_like(logits), torch.empty_like(x)
        with ops._on_device(x.device):
            check(_L.na1d_stats_pool_backward(d_logits.data_ptr(), dx.data_ptr(), d_out.data_ptr(), out.data_ptr(), stats.data_ptr(),
                                              logits.data_ptr(), x.data_ptr(), N, T, C, ctx.floor, _CODE[x.dtype],
                                              _stream(x)), "na1d_stats_pool_backward")
        return d_logits, dx, None


def stats_pool(logits, x, floor):
    """(N, 2C) fp32: mean and standard deviation of x (N, T, C) over T under softmax-over-T weights, or None where the inputs
    are not a pair of dense 16-bit CUDA tensors that the kernel takes."""
    if (type(x) is not torch.Tensor or type(logits) is not torch.Tensor or not x.is_cuda or x.dtype not in _CODE or logits.dtype != x.dtype or
            logits.shape != x.shape or logits.device != x.device or x.dim() != 3 or torch.compiler.is_compiling() or not ops.native.eager_mode() or
            torch.autograd.forward_ad._current_level >= 0):
        return None
    N, T, C = x.shape
    if not 0 < N <= 65535 or not 0 < T <= 1 << 20 or C == 0 or C % 8 or C > 1 << 20:
        return None
    logits = logits.contiguous()
    if not torch.is_grad_enabled() and x.stride(2) == 1 and x.stride(0) == T * x.stride(1) and x.stride(1) % 8 == 0 and C <= x.stride(1) <= 1 << 20:
        ld = x.stride(1)                     # a slice of wider rows is read in place
    else:
        x, ld = x.contiguous(), C
    if logits.data_ptr() % 16 or x.data_ptr() % 16:
        return None
    if not torch.is_grad_enabled():
        out = torch.empty((N, 2 * C), dtype=torch.float32, device=x.device)
        with ops._on_device(x.device):
            check(_L.na1d_stats_pool_forward(out.data_ptr(), None, logits.data_ptr(), x.data_ptr(), ld, N, T, C, floor, _CODE[x.dtype], _stream(x)),
                  "na1d_stats_pool_forward")
        return out
    return _StatsPoolFunction.apply(logits, x, floor)
