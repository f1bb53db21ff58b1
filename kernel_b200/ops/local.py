"""Products whose operands are all on this GPU, and the row movement of a MoE layer
whose experts are all on this GPU: front-ends of ``csrc/kernels/gemm_local.cu`` and
``csrc/kernels/moe_rows.cu``.

``product`` is the dense one; an operand may be given transposed (``a_t``, ``b_t``),
which the kernel reads as it lies in memory.  ``rows_product`` multiplies groups of
rows by their group's own matrix, ``contract_product`` contracts over the rows of each
group (weight gradients); both take the group table from device memory.  CPU tensors
take a plain fp32 torch formulation with the same rounding points, so that the layers
built on them are testable without a GPU.
"""
from __future__ import annotations

import ctypes as C
from typing import Optional

import torch

from .. import _native as N
from . import gemm as G

ROW_ALIGN = 64  # rows of a group in a table made for contract_product start at multiples of the kernel's k block

_ACTS = {
    "gelu": lambda x: torch.nn.functional.gelu(x, approximate="tanh"),
    "relu": torch.relu,
    "silu": torch.nn.functional.silu,
}


def _slope(act: str, pre: torch.Tensor) -> torch.Tensor:
    with torch.enable_grad():
        x = pre.float().detach().requires_grad_(True)
        return torch.autograd.grad(_ACTS[act](x).sum(), x)[0]


def _finish(res: torch.Tensor, act, pre_out, pre_in, out) -> torch.Tensor:
    """The kernel's epilogue on an fp32 product."""
    if pre_in is not None:
        res = (res * _slope(act, pre_in)).to(torch.bfloat16)
    else:
        res = res.to(torch.bfloat16)
        if pre_out is not None:
            pre_out.copy_(res)
        if act is not None:
            res = _ACTS[act](res.float()).to(torch.bfloat16)
    if out is None:
        return res
    out.copy_(res)
    return out


def _ptr(t: Optional[torch.Tensor]):
    return t.data_ptr() if t is not None else None


def _stream(device: torch.device) -> int:
    return torch._C._cuda_getCurrentRawStream(device.index if device.index is not None else torch.cuda.current_device())


def _check_operand(t: torch.Tensor, name: str, dims: int, device: torch.device) -> None:
    if t.dtype != torch.bfloat16 or t.dim() != dims or not t.is_contiguous() or t.device != device:
        raise ValueError(f"{name} must be a contiguous {dims}-D bf16 tensor on {device}")


def _check_results(shape, device: torch.device, *results: Optional[torch.Tensor]) -> None:
    """Matrices that are read or written by their address, row for row like the product."""
    for t in results:
        if t is not None and (t.shape != shape or t.dtype != torch.bfloat16 or not t.is_contiguous() or t.device != device):
            raise ValueError(f"results and saved values must be contiguous bf16 matrices of shape {tuple(shape)} on {device}")


def _check_choices(t: torch.Tensor, name: str, dtype: torch.dtype, shape, device: torch.device) -> None:
    if t.dtype != dtype or t.shape != shape or not t.is_contiguous() or t.device != device:
        raise ValueError(f"{name} must be contiguous {dtype} of shape {tuple(shape)} on {device}")


def _check_table(start: torch.Tensor, count: torch.Tensor, groups: int, device: torch.device) -> None:
    for t in (start, count):
        if t.dtype != torch.int32 or t.shape != (groups,) or not t.is_contiguous() or t.device != device:
            raise ValueError(f"group tables must be contiguous int32 [{groups}] on {device}")


def _expert_matrices(b: torch.Tensor) -> torch.Tensor:
    """``b[E, ...]`` as one block.  Matrices that are contiguous one by one (every second
    expert of a larger tensor, one matrix expanded over the experts) are gathered; a
    transposed matrix is not an operand layout, ``b_t`` says which one is meant."""
    if b.dim() == 3 and not b.is_contiguous() and b[:1].is_contiguous():
        return b.contiguous()
    return b


def _args(kind: int, M: int, Nn: int, K: int, status: Optional[torch.Tensor]) -> N.LocalGemmArgs:
    args = N.LocalGemmArgs()
    args.kind, args.M, args.N, args.K, args.pair = kind, M, Nn, K, -1
    args.status, args.wait_limit_ns = _ptr(status), G._WAIT_LIMIT_NS
    return args


def _launch(args: N.LocalGemmArgs, device: torch.device) -> None:
    code = N.lib().kb_gemm_local(C.byref(args), _stream(device))
    if code:
        N.check(code)
    G.launch_count += 1


def product(a: torch.Tensor, b: torch.Tensor, bias: Optional[torch.Tensor] = None, *, a_t: bool = False, b_t: bool = False,
            act: Optional[str] = None, pre_out: Optional[torch.Tensor] = None, pre_in: Optional[torch.Tensor] = None,
            out: Optional[torch.Tensor] = None, status: Optional[torch.Tensor] = None, early: bool = False) -> torch.Tensor:
    """``A @ B^T (+ bias)`` in bf16 with fp32 accumulation, ``A`` being ``a[M, K]`` (``a_t``: ``a[K, M]``)
    and ``B`` being ``b[N, K]`` (``b_t``: ``b[K, N]``); ``a_t`` needs ``b_t``.

    ``act``: the activation of the rounded product, which ``pre_out`` also receives;
    with ``pre_in`` the product is multiplied by the activation's slope there.
    ``early``: the stream's previous launch is one of this module's kernels and did not write ``b``, so the product may
    fetch it before that one has ended."""
    _check_operand(a, "a", 2, a.device)
    _check_operand(b, "b", 2, a.device)
    K, M = a.shape if a_t else a.shape[::-1]
    Kb, Nn = b.shape if b_t else b.shape[::-1]
    if Kb != K:
        raise ValueError("inner dimensions differ")
    _check_results((M, Nn), a.device, out, pre_out, pre_in)
    if not a.is_cuda:
        A, B = a.float(), b.float()
        res = (A.t() if a_t else A) @ (B if b_t else B.t())
        return _finish(res if bias is None else res + bias.float(), act, pre_out, pre_in, out)
    if out is None:
        out = torch.empty((M, Nn), dtype=torch.bfloat16, device=a.device)
    args = _args(N.LOCAL_DENSE, M, Nn, K, status)
    args.a_mn, args.b_mn, args.early = a_t, b_t, early
    args.bias, args.bias_scale = _ptr(bias), 1.0
    args.A, args.B, args.out = a.data_ptr(), b.data_ptr(), out.data_ptr()
    args.act, args.pre_out, args.pre_in = N.ACTS.get(act, 0), _ptr(pre_out), _ptr(pre_in)
    _launch(args, a.device)
    return out


def col_sum(x: torch.Tensor) -> torch.Tensor:
    """``x[R, C].sum(0)`` accumulated in fp32, in bf16 (bias gradients)."""
    R, Cn = x.shape
    if not x.is_cuda or x.dtype != torch.bfloat16 or R == 0 or Cn % 8 or x.data_ptr() % 16:
        return x.float().sum(0).to(x.dtype)
    lib = N.lib()
    parts = lib.kb_col_sum_parts(R, Cn)
    partial = torch.empty((parts, Cn), dtype=torch.float32, device=x.device) if parts > 1 else None
    out = torch.empty(Cn, dtype=torch.bfloat16, device=x.device)
    N.check(lib.kb_col_sum(x.data_ptr(), R, Cn, _ptr(partial), out.data_ptr(), _stream(x.device)))
    return out


def rows_product(a: torch.Tensor, b: torch.Tensor, start: torch.Tensor, count: torch.Tensor, *, b_t: bool = False,
                 act: Optional[str] = None, pre_out: Optional[torch.Tensor] = None, pre_in: Optional[torch.Tensor] = None,
                 out: Optional[torch.Tensor] = None, status: Optional[torch.Tensor] = None, early: bool = False,
                 expect: int = 0) -> torch.Tensor:
    """Rows ``start[e] .. start[e] + count[e]`` of ``a[R, K]`` times ``b[e]`` transposed
    (``b[E, N, K]``, ``b_t``: ``b[E, K, N]``).  Rows outside every group are left alone.  ``early``: the stream's previous
    launch is a kernel of this module and wrote neither ``b`` nor the table.  ``expect``: rows expected in all groups, where
    ``R`` is a capacity (the choice of tiles depends on it, nothing else)."""
    given = b
    b = _expert_matrices(b)
    early = early and b is given  # else that launch is the copy
    _check_operand(a, "a", 2, a.device)
    _check_operand(b, "b", 3, a.device)
    R, K = a.shape
    E = b.shape[0]
    Kb, Nn = b.shape[1:] if b_t else (b.shape[2], b.shape[1])
    if Kb != K:
        raise ValueError("inner dimensions differ")
    _check_table(start, count, E, a.device)
    _check_results((R, Nn), a.device, out, pre_out, pre_in)
    if out is None:
        out = torch.empty((R, Nn), dtype=torch.bfloat16, device=a.device)
    if R == 0:
        return out
    if not a.is_cuda:
        for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
            if n:
                B = b[e].float()
                sl = slice(s, s + n)
                _finish(a[sl].float() @ (B if b_t else B.t()), act, None if pre_out is None else pre_out[sl],
                        None if pre_in is None else pre_in[sl], out[sl])
        return out
    args = _args(N.LOCAL_ROWS, R, Nn, K, status)
    args.b_mn, args.groups, args.expect, args.early = b_t, E, expect, early
    args.row_start, args.row_count = start.data_ptr(), count.data_ptr()
    args.A, args.B, args.out = a.data_ptr(), b.data_ptr(), out.data_ptr()
    args.act, args.pre_out, args.pre_in = N.ACTS.get(act, 0), _ptr(pre_out), _ptr(pre_in)
    _launch(args, a.device)
    return out


def contract_product(a: torch.Tensor, b: torch.Tensor, start: torch.Tensor, count: torch.Tensor,
                     status: Optional[torch.Tensor] = None, expect: int = 0) -> torch.Tensor:
    """``out[e] = a[rows of e]^T @ b[rows of e]`` for ``a[R, M]``, ``b[R, N]``.  Groups start at
    multiples of ``ROW_ALIGN``; rows between a group's last and the next multiple are
    zero in one operand and finite in the other."""
    _check_operand(a, "a", 2, a.device)
    _check_operand(b, "b", 2, a.device)
    (R, M), Nn, E = a.shape, b.shape[1], start.shape[0]
    if b.shape[0] != R:
        raise ValueError("a and b have different numbers of rows")
    _check_table(start, count, E, a.device)
    if not a.is_cuda or R == 0:
        out = torch.zeros((E, M, Nn), dtype=torch.bfloat16, device=a.device)
        for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
            out[e] = (a[s:s + n].float().t() @ b[s:s + n].float()).to(torch.bfloat16)
        return out
    out = torch.empty((E, M, Nn), dtype=torch.bfloat16, device=a.device)
    args = _args(N.LOCAL_CONTRACT, M, Nn, R, status)
    args.groups, args.expect = E, expect
    args.row_start, args.row_count = start.data_ptr(), count.data_ptr()
    args.A, args.B, args.out = a.data_ptr(), b.data_ptr(), out.data_ptr()
    _launch(args, a.device)
    return out


class ExpertRows:
    """Expert-major copies of a batch's token rows on one GPU, one row per (token, choice).

    ``rows[R, H]``; group table ``start``, ``count`` (``padded``: count rounded up to
    ``pad`` rows, zero rows in between); ``slots[T, k]`` maps a choice to its row.
    No count travels to the host, so ``R`` is a capacity: ``T * k`` rows and ``pad - 1`` for
    every expert that can have one.  The price of staying off the host is memory: with
    ``pad`` = 64 the activations of 64 tokens, top-8 of 1024 experts, take 32768 rows for 512
    real ones (rows behind the last padded expert are neither written nor read)."""

    @staticmethod
    def capacity(T: int, k: int, experts: int, pad: int) -> int:
        return T * k + min(experts, T * k) * (pad - 1)

    def __init__(self, x: torch.Tensor, indices: torch.Tensor, experts: int, pad: int = 1, status: Optional[torch.Tensor] = None):
        _check_operand(x, "x", 2, x.device)
        (T, H), k, dev = x.shape, indices.shape[1], x.device
        _check_choices(indices, "indices", torch.int32, (T, k), dev)
        rows = torch.empty((self.capacity(T, k, experts, pad), H), dtype=torch.bfloat16, device=dev)
        self._set(rows, torch.empty(3 * experts + T * k, dtype=torch.int32, device=dev), T, k, experts)
        N.check(N.lib().kb_moe_permute(x.data_ptr(), indices.data_ptr(), T, k, experts, H, pad, self.rows.data_ptr(),
                                       self.slots.data_ptr(), self.start.data_ptr(), self.count.data_ptr(), self.padded.data_ptr(),
                                       _ptr(status), _stream(dev)))

    def _set(self, rows: torch.Tensor, table: torch.Tensor, T: int, k: int, experts: int) -> None:
        self.T, self.k, self.E, self.H = T, k, experts, rows.shape[1]
        self.rows, self.table = rows, table
        self.start, self.count, self.padded = table[:experts], table[experts:2 * experts], table[2 * experts:3 * experts]
        self.slots = table[3 * experts:].view(T, k)

    @classmethod
    def saved(cls, rows: torch.Tensor, table: torch.Tensor, T: int, k: int, experts: int) -> "ExpertRows":
        """The rows and tables an earlier instance made (``rows``, ``table``), for a backward pass."""
        er = cls.__new__(cls)
        er._set(rows, table, T, k, experts)
        return er

    def _check(self, y: torch.Tensor, weights: Optional[torch.Tensor]) -> None:
        _check_results(self.rows.shape, self.rows.device, y)
        if weights is not None:
            _check_choices(weights, "weights", torch.float32, (self.T, self.k), self.rows.device)

    def combine(self, y: torch.Tensor, weights: Optional[torch.Tensor]) -> torch.Tensor:
        """``out[t] = sum_j weights[t, j] * y[slots[t, j]]`` (``None``: unit weights)."""
        self._check(y, weights)
        out = torch.empty((self.T, self.H), dtype=torch.bfloat16, device=y.device)
        N.check(N.lib().kb_moe_combine(y.data_ptr(), self.slots.data_ptr(), _ptr(weights), self.T, self.k, self.H, out.data_ptr(),
                                       _stream(y.device)))
        return out

    def grad_rows(self, dy: torch.Tensor, y: torch.Tensor, weights: torch.Tensor):
        """Backward of ``combine``: ``(dY rows, d weights)``."""
        self._check(y, weights)
        _check_results((self.T, self.H), self.rows.device, dy)
        dyr = torch.empty_like(y)
        dw = torch.empty((self.T, self.k), dtype=torch.float32, device=dy.device)
        N.check(N.lib().kb_moe_grad_rows(dy.data_ptr(), y.data_ptr(), self.slots.data_ptr(), weights.data_ptr(), self.T, self.k, self.E,
                                         self.H, dyr.data_ptr(), dw.data_ptr(), self.start.data_ptr(), self.count.data_ptr(),
                                         self.padded.data_ptr(), _stream(dy.device)))
        return dyr, dw
