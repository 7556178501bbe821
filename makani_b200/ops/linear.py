"""Linear layers on the last dimension ("traditional" token layout [..., C]) as tcgen05 GEMMs.

`Y[t, o] = act(sum_c X[t, c] W[o, c] + b[o])`: both operands are K-major, the bias is per output column and the
result is written row-major.  Used by the AFNO / ViT token MLPs.
"""

from __future__ import annotations

import torch

from . import _ext
from .conv import records_grad
from .gemm import ACT_NONE


def fast_path_ok(x: torch.Tensor) -> bool:
    return _ext.native() and x.is_cuda and x.dtype == torch.bfloat16 and x.is_contiguous() and x.shape[-1] % 8 == 0


class _MLP2Last(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, train):
        shp = x.shape
        x2 = x.reshape(-1, shp[-1])
        # second output of the first layer: GELU'(pre-activation), where a backward pass will want it
        y, w1q, w2q, dact, h = _ext.require().mlp_forward(x2, w1, b1, w2, b2, None, -1, train)
        ctx.save_for_backward(x2, w1q, w2q, dact, h)
        ctx.flags = (b1 is not None, b2 is not None)
        ctx.shp = shp
        return y.reshape(*shp[:-1], w2.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, w1q, w2q, dact, h = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1]).contiguous()
        dx, dw1, db1, dw2, db2 = _ext.require().mlp_backward(dy2, x2, w1q, w2q, dact, h, x2.shape[1], ctx.needs_input_grad[0], *ctx.flags)
        return (None if dx is None else dx.reshape(ctx.shp)), dw1, db1, dw2, db2, None


class _LinearLast(torch.autograd.Function):
    """y = x W^T + b on the last dimension: one GEMM forward, data- and weight-gradient GEMMs backward."""

    @staticmethod
    def forward(ctx, x, w, b):
        shp = x.shape
        x2 = x.reshape(-1, shp[-1])
        y, wq, _ = _ext.require().conv_forward(x2, w, b, None, ACT_NONE, -1, False)
        ctx.save_for_backward(x2, wq)
        ctx.has_bias, ctx.shp = b is not None, shp
        return y.reshape(*shp[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        x2, wq = ctx.saved_tensors
        dy2 = dy.reshape(-1, dy.shape[-1]).contiguous()
        dx, dw, db = _ext.require().conv_backward(dy2, x2, wq, x2.shape[1], ctx.needs_input_grad[0], ctx.needs_input_grad[1], ctx.has_bias)
        return (None if dx is None else dx.reshape(ctx.shp)), dw, db


def linear_lastdim(x, w, b=None):
    """`torch.nn.functional.linear` for bf16 CUDA tokens whose feature counts are multiples of 8; anything else falls
    back to the torch op."""
    if fast_path_ok(x) and w.shape[0] % 8 == 0:
        _ext.require()
        return _LinearLast.apply(x, w, b)
    return torch.nn.functional.linear(x, w.to(x.dtype), None if b is None else b.to(x.dtype))


def mlp2_lastdim(x, w1, b1, w2, b2):
    _ext.require()
    return _MLP2Last.apply(x, w1, b1, w2, b2, records_grad(x, w1, b1, w2, b2))
