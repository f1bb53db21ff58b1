"""Sequence-parallel tensor-parallel MLP: the region that the reference's two
collectives bracket (``gemm_rs/task.yml:16-22`` describes the exit GEMM).

Activations enter and leave sharded along the token dimension.  The up
projection is column-parallel and needs every token: all-gather fused with the
GEMM.  The down projection is row-parallel (its K dimension is the sharded
hidden dimension of the MLP) and produces partial sums for every token: GEMM
fused with the reduce-scatter.  ``SequenceParallelMLP`` is the forward-only block over
given weights; ``TrainableSequenceParallelMLP`` owns parameters and has a backward pass.
"""
from __future__ import annotations

from typing import Optional

import torch
from torch.nn.modules.module import _has_any_global_hook

from .._native import ACTS
from ..ops.autograd import ColumnParallelLinear, LocalMLPFn, RowParallelLinear
from ..ops.gemm import AGGemm, GemmRS
from ..ops.local import product
from ..parallel.symm import _dist_info


class SequenceParallelMLP:
    """``y_local = RS( act( AG(x_local) @ W1_shard^T + b1_shard ) @ W2_shard^T ) + b2``.

    ``w1`` is this rank's ``[ffn/world, hidden]`` shard, ``w2`` its ``[hidden,
    ffn/world]`` shard; ``tokens`` is the global token count (a multiple of the
    world size).
    """

    def __init__(self, tokens: int, hidden: int, w1: torch.Tensor, w2: torch.Tensor, b1: Optional[torch.Tensor] = None,
                 b2: Optional[torch.Tensor] = None, activation: str = "gelu", group=None):
        self.rank, self.world = _dist_info(group)
        if w1.shape[1] != hidden or w2.shape[0] != hidden or w2.shape[1] != w1.shape[0]:
            raise ValueError("w1 must be [ffn/world, hidden] and w2 [hidden, ffn/world]")
        self.w1, self.w2, self.b1, self.b2 = w1.contiguous(), w2.contiguous(), b1, b2
        self.activation = activation
        dev = w1.device
        self.up = AGGemm(tokens, hidden, group=group, device=dev)
        self.down = GemmRS(tokens, hidden, group=group, device=dev)

    def _act(self, h: torch.Tensor) -> torch.Tensor:
        if self.activation == "gelu":
            return torch.nn.functional.gelu(h, approximate="tanh")
        if self.activation == "relu":
            return torch.relu(h)
        if self.activation == "silu":
            return torch.nn.functional.silu(h)
        raise ValueError(f"unknown activation {self.activation!r}")

    def _plain(self) -> bool:
        """One rank, and the up-projection and the activation are the block's own (a context put in
        the projection's place may span several ranks)."""
        return (self.world == 1 and self.activation in ACTS and type(self.up) is AGGemm and self.up.world == 1
                and getattr(self._act, "__func__", None) is SequenceParallelMLP._act)

    def __call__(self, x_local: torch.Tensor) -> torch.Tensor:
        if x_local.is_cuda and self._plain():
            self.up.check(x_local, self.w1)
            h = product(x_local, self.w1, self.b1, act=self.activation, status=self.up.status)   # the activation in the product's epilogue
            if type(self.down) is GemmRS and self.down.world == 1 and h.shape[0] == self.down.M and self.w2.shape[0] == self.down.N:
                return product(h, self.w2, self.b2, status=self.down.status, early=True)
            return self.down(h, self.w2, self.b2)
        h = self.up(x_local, self.w1, self.b1)           # [tokens, ffn/world]
        h = self._act(h)
        return self.down(h, self.w2, self.b2)            # [tokens/world, hidden]

    def reference(self, x_full: torch.Tensor, w1_full: torch.Tensor, w2_full: torch.Tensor, b1_full=None, b2=None) -> torch.Tensor:
        """Unsharded fp32 result for all tokens (tests)."""
        h = x_full.float() @ w1_full.float().t()
        if b1_full is not None:
            h = h + b1_full.float()
        h = self._act(h.to(torch.bfloat16)).float()
        y = h @ w2_full.float().t()
        if b2 is not None:
            y = y + b2.float()
        return y

    def close(self) -> None:
        for ctx in (self.up, self.down):
            if ctx.heap is not None:
                ctx.heap.close()


def _plain(layer: torch.nn.Module, kind: type) -> bool:
    """One rank, and nothing (a replacement, a ``forward`` set on the instance, hooks of the
    layer or of all modules) asks for the layer to be called by itself."""
    return type(layer) is kind and layer.world == 1 and "forward" not in vars(layer) and not (
        layer._forward_hooks or layer._forward_pre_hooks or layer._backward_hooks or layer._backward_pre_hooks or _has_any_global_hook())


class TrainableSequenceParallelMLP(torch.nn.Module):
    """The same block as ``SequenceParallelMLP`` with parameters and a backward
    pass: ``ColumnParallelLinear`` (all-gather fused forward, reduce-scatter fused
    input gradient) -> activation -> ``RowParallelLinear`` (the mirror image).
    ``ffn_local`` is this rank's share of the MLP's hidden dimension."""

    def __init__(self, tokens: int, hidden: int, ffn_local: int, bias: bool = True, activation: str = "gelu", group=None,
                 device: Optional[torch.device] = None):
        super().__init__()
        self.up = ColumnParallelLinear(tokens, hidden, ffn_local, bias=bias, group=group, device=device)
        self.down = RowParallelLinear(tokens, ffn_local, hidden, bias=bias, group=group, device=device)
        self.activation = activation

    def forward(self, x_local: torch.Tensor) -> torch.Tensor:
        up, down = self.up, self.down
        if (x_local.is_cuda and self.activation in ACTS and _plain(up, ColumnParallelLinear) and _plain(down, RowParallelLinear)
                and down.weight.dtype == torch.bfloat16 and down.weight.shape == (down.fwd.N, up.weight.shape[0])):
            return LocalMLPFn.apply(x_local, up.weight, up.bias, down.weight, down.bias, self.activation, up.fwd)
        h = self.up(x_local)
        if self.activation == "gelu":
            h = torch.nn.functional.gelu(h, approximate="tanh")
        elif self.activation == "relu":
            h = torch.relu(h)
        elif self.activation == "silu":
            h = torch.nn.functional.silu(h)
        else:
            raise ValueError(f"unknown activation {self.activation!r}")
        return self.down(h)

    def close(self) -> None:
        self.up.close()
        self.down.close()
