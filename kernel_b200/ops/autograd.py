"""Differentiable front-ends of the two fused GEMM+collective ops.

The two ops are each other's transpose, which makes training a sequence-parallel
tensor-parallel block need nothing new on the device:

* ``y = AG(x_local) @ W^T``  (column-parallel; ``AGGemm``)
  has ``dx_local = RS(dy @ W)``, a GEMM fused with reduce-scatter;
* ``y_local = RS(x @ W^T)``  (row-parallel; ``GemmRS``)
  has ``dx = AG(dy_local) @ W``, an all-gather fused with a GEMM.

The weight gradients contract over the token dimension and need the gathered
operand (``x`` resp. ``dy``); it is gathered with one library collective and the
product is the local tcgen05 GEMM, which reads operands that are contiguous along
either dimension.  The gather runs on the same stream as the fused
kernel, before it: the fused kernels are persistent, fill every SM and wait (with a
limit) for their peers, so a collective kernel of another stream that is scheduled
behind them on one rank and ahead of them on another could make the ranks wait on
each other until the limit expires.  CPU tensors take the torch paths of the ops, so the wiring
is testable on gloo ranks.

The reference has forward-only kernels (``gemm_rs/submission.py:5-29``); nothing
there corresponds to this file.
"""
from __future__ import annotations

from typing import Optional

import torch
import torch.distributed as dist

from ..parallel.symm import _dist_info
from .gemm import AGGemm, GemmRS
from .local import col_sum, product


def _gather_rows(t_local: torch.Tensor, world: int, group) -> torch.Tensor:
    if world == 1:
        return t_local
    full = torch.empty((t_local.shape[0] * world, t_local.shape[1]), dtype=t_local.dtype, device=t_local.device)
    dist.all_gather_into_tensor(full, t_local.contiguous(), group=group)
    return full


def _wgrad(dy_full: torch.Tensor, x_full: torch.Tensor) -> torch.Tensor:
    """``dW[N, K] = dy_full[M, N]^T @ x_full[M, K]``, both operands read as they lie."""
    return product(dy_full.contiguous(), x_full.contiguous(), a_t=True, b_t=True)


def _one_gpu(layer, t: torch.Tensor) -> bool:
    return t.is_cuda and layer.world == 1


def _input_grad(layer, dy: torch.Tensor, w: torch.Tensor) -> torch.Tensor:
    """``dy @ w`` through the layer's backward context.  On one GPU there is nothing to
    exchange: the product reads the weights as they lie, instead of a transposed copy for
    the fused kernel's operand layout, and reports a failed wait in the same status words."""
    if _one_gpu(layer, dy):
        return product(dy, w.contiguous(), b_t=True, status=layer.bwd.status)
    return layer.bwd(dy, w.t().contiguous())


class _ColumnParallelFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x_local, w, bias, layer):
        ctx.layer = layer
        ctx.save_for_backward(x_local, w)
        ctx.has_bias = bias is not None
        return layer.fwd(x_local.contiguous(), w.contiguous(), bias)

    @staticmethod
    def backward(ctx, dy):
        layer = ctx.layer
        x_local, w = ctx.saved_tensors
        dy = dy.contiguous()
        dx = dw = db = None
        need_dw = ctx.needs_input_grad[1]
        if need_dw:
            x_full = _gather_rows(x_local, layer.world, layer.group)
        if ctx.needs_input_grad[0]:
            # dx_local[M/world, K] = RS(dy[M, Nl] @ W[Nl, K]): contraction over the sharded Nl
            dx = _input_grad(layer, dy, w)
        if need_dw:
            dw = _wgrad(dy, x_full)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            db = col_sum(dy)
        return dx, dw, db, None


class _RowParallelFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, bias, layer):
        ctx.layer = layer
        ctx.save_for_backward(x, w)
        ctx.has_bias = bias is not None
        return layer.fwd(x.contiguous(), w.contiguous(), bias)

    @staticmethod
    def backward(ctx, dy_local):
        layer = ctx.layer
        x, w = ctx.saved_tensors
        dy_local = dy_local.contiguous()
        dx = dw = db = None
        need_dw = ctx.needs_input_grad[1]
        if need_dw:
            dy_full = _gather_rows(dy_local, layer.world, layer.group)
        if ctx.needs_input_grad[0]:
            # dx[M, Kl] = AG(dy_local)[M, N] @ W[N, Kl]
            dx = _input_grad(layer, dy_local, w)
        if need_dw:
            dw = _wgrad(dy_full, x)
        if ctx.has_bias and ctx.needs_input_grad[2]:
            # the bias is added once to every output row; this is the sum over this
            # rank's rows, to be summed over ranks with the other replicated parameters
            db = col_sum(dy_local)
        return dx, dw, db, None


class LocalMLPFn(torch.autograd.Function):
    """``act(x @ w1^T + b1) @ w2^T + b2`` on one GPU: two products forward, four backward,
    the activation in the first one's epilogue (which keeps the value before it), its
    slope in the epilogue of the hidden gradient's product.  No transposed copy and no
    elementwise pass: both were 40 % of a step at 8192 x 8192 x 29568.  ``up`` is the
    ``AGGemm`` context whose shape ``x`` and ``w1`` have to fit; operands of other strides
    are made contiguous first, as the two linear layers do."""

    @staticmethod
    def forward(ctx, x, w1, b1, w2, b2, act, up):
        x, w1, w2 = x.contiguous(), w1.contiguous(), w2.contiguous()
        up.check(x, w1)
        status = getattr(up, "status", None)  # CPU contexts have none
        pre = torch.empty((x.shape[0], w1.shape[0]), dtype=x.dtype, device=x.device)
        h = product(x, w1, b1, act=act, pre_out=pre, status=status)
        ctx.act, ctx.status = act, status
        ctx.save_for_backward(x, w1, w2, pre, h)
        return product(h, w2, b2, status=status, early=True)

    @staticmethod
    def backward(ctx, dy):
        x, w1, w2, pre, h = ctx.saved_tensors
        status = ctx.status
        need_x, need_w1, need_b1, need_w2, need_b2 = ctx.needs_input_grad[:5]
        dy = dy.contiguous()
        dx = dw1 = db1 = dw2 = db2 = None
        if need_w2:
            dw2 = product(dy, h, a_t=True, b_t=True, status=status)
        if need_b2:
            db2 = col_sum(dy)
        if need_x or need_w1 or need_b1:
            dpre = product(dy, w2, b_t=True, act=ctx.act, pre_in=pre, status=status, early=need_w2)  # else its weights may just have been copied
            if need_w1:
                dw1 = product(dpre, x, a_t=True, b_t=True, status=status)
            if need_b1:
                db1 = col_sum(dpre)
            if need_x:
                dx = product(dpre, w1, b_t=True, status=status, early=True)
        return dx, dw1, db1, dw2, db2, None, None


class ColumnParallelLinear(torch.nn.Module):
    """``y[M, out/world] = all_gather(x_local)[M, in] @ W_shard^T + b_shard`` with
    the all-gather fused into the GEMM forward and the reduce-scatter fused into
    the input-gradient GEMM backward.  ``tokens`` is the global row count M."""

    def __init__(self, tokens: int, in_features: int, out_features_local: int, bias: bool = True, group=None,
                 device: Optional[torch.device] = None, dtype: torch.dtype = torch.bfloat16):
        super().__init__()
        dev = torch.device(device) if device is not None else torch.device("cpu")
        self.group = group
        self.rank, self.world = _dist_info(group)
        self.weight = torch.nn.Parameter(torch.empty(out_features_local, in_features, dtype=dtype, device=dev))
        self.bias = torch.nn.Parameter(torch.zeros(out_features_local, dtype=dtype, device=dev)) if bias else None
        torch.nn.init.normal_(self.weight, std=in_features ** -0.5)
        self.fwd = AGGemm(tokens, in_features, group=group, device=dev)
        self.bwd = GemmRS(tokens, in_features, group=group, device=dev)

    def forward(self, x_local: torch.Tensor) -> torch.Tensor:
        return _ColumnParallelFn.apply(x_local, self.weight, self.bias, self)

    def close(self) -> None:
        for c in (self.fwd, self.bwd):
            if c.heap is not None:
                c.heap.close()


class RowParallelLinear(torch.nn.Module):
    """``y_local[M/world, out] = reduce_scatter(x[M, in/world] @ W_shard^T) + b`` with
    the reduce-scatter fused into the GEMM forward and the all-gather fused into
    the input-gradient GEMM backward.  The bias is replicated: its gradient here is
    the sum over this rank's rows."""

    def __init__(self, tokens: int, in_features_local: int, out_features: int, bias: bool = True, group=None,
                 device: Optional[torch.device] = None, dtype: torch.dtype = torch.bfloat16):
        super().__init__()
        dev = torch.device(device) if device is not None else torch.device("cpu")
        self.group = group
        self.rank, self.world = _dist_info(group)
        self.weight = torch.nn.Parameter(torch.empty(out_features, in_features_local, dtype=dtype, device=dev))
        self.bias = torch.nn.Parameter(torch.zeros(out_features, dtype=dtype, device=dev)) if bias else None
        torch.nn.init.normal_(self.weight, std=(in_features_local * self.world) ** -0.5)
        self.fwd = GemmRS(tokens, out_features, group=group, device=dev)
        self.bwd = AGGemm(tokens, out_features, group=group, device=dev)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return _RowParallelFn.apply(x, self.weight, self.bias, self)

    def close(self) -> None:
        for c in (self.fwd, self.bwd):
            if c.heap is not None:
                c.heap.close()
