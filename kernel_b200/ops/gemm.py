"""Front-ends of the tcgen05 GEMM family: plain GEMM, GEMM + reduce-scatter and
all-gather + GEMM.

On CUDA tensors these always launch hand-written sm_100a kernels: the fused ones
(``csrc/kernels/gemm_sm100.cu``) with several ranks, the product family of one GPU
(``csrc/kernels/gemm_local.cu``) otherwise; there is no library fallback on a GPU.  CPU
tensors take a torch reference path (``torch.matmul`` plus gloo collectives) so
that host-side logic can be tested without a GPU; with more than one CPU rank the
fused ops run the kernels' protocol over a host-backed symmetric heap.

Counterparts in the reference: ``gemm_rs/submission.py:5-29`` (matmul, bias add,
``reduce_scatter_tensor``).  The all-gather variant has no counterpart there.
"""
from __future__ import annotations

import ctypes as C
import os
from typing import Optional

import torch
import torch.distributed as dist

from .. import _native as N
from ..parallel.symm import SymmHeap, _dist_info

_WAIT_LIMIT_NS = int(float(os.environ.get("KB200_WAIT_LIMIT_MS", "2000")) * 1e6)

launch_count = 0  # kernels launched by this module (bench accounting)


def _check_bf16_2d(t: torch.Tensor, name: str) -> None:
    if t.dtype != torch.bfloat16 or t.dim() != 2 or not t.is_contiguous():
        raise ValueError(f"{name} must be a contiguous 2-D bf16 tensor")


def _launch(args: N.GemmArgs, device: torch.device) -> None:
    global launch_count
    stream = torch.cuda.current_stream(device).cuda_stream
    code = N.lib().kb_gemm(C.byref(args), stream)
    if code:
        N.check(code)
    launch_count += 1


def _check_out(out: torch.Tensor, rows: int, cols: int, device: torch.device) -> None:
    """The kernel writes ``rows x cols`` values from ``out``'s address on, whatever its shape
    (a flat or a larger buffer is filled from its start)."""
    if out.dtype != torch.bfloat16 or not out.is_contiguous() or out.device != device or out.numel() < rows * cols:
        raise ValueError(f"out must be a contiguous bf16 tensor of at least {rows} x {cols} elements on {device}")


def _local_args(status: Optional[torch.Tensor]) -> N.LocalGemmArgs:
    """Argument block of a product whose operands are all on this GPU."""
    args = N.LocalGemmArgs()
    args.kind, args.pair, args.bias_scale = N.LOCAL_DENSE, -1, 1.0
    args.status = status.data_ptr() if status is not None else None
    args.wait_limit_ns = _WAIT_LIMIT_NS
    return args


def _launch_local(args: N.LocalGemmArgs, device: torch.device) -> None:
    global launch_count
    index = device.index
    code = N.lib().kb_gemm_local(C.byref(args), torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if index is None else index))
    if code:
        N.check(code)
    launch_count += 1


def _run_local(ctx, a: torch.Tensor, w: torch.Tensor, bias, bias_scale: float, out: torch.Tensor) -> torch.Tensor:
    """The fused ops on one rank: nothing to exchange, a dense product.  The argument
    block is kept with the context; a call refreshes what changes."""
    args = ctx._hot
    if args is None:
        args = ctx._hot = _local_args(ctx.status)
    _check_out(out, a.shape[0], w.shape[0], a.device)
    (args.M, args.K), args.N = a.shape, w.shape[0]
    args.A, args.B, args.out = a.data_ptr(), w.data_ptr(), out.data_ptr()
    args.bias = bias.data_ptr() if bias is not None else None
    args.bias_scale = bias_scale
    _launch_local(args, a.device)
    return out


def _cpu_heap_path() -> bool:
    """CPU ranks run the kernels' protocol over a memfd-backed symmetric heap
    (``csrc/symm/gemm_host.cpp``) unless ``KB200_GEMM_CPU_PATH=collectives`` selects
    torch matmul + gloo collectives."""
    return os.environ.get("KB200_GEMM_CPU_PATH", "heap") == "heap"


def _new_heap(nbytes: int, group, device, native: bool) -> SymmHeap:
    if native:
        return SymmHeap(nbytes, group=group, device=device)  # with an NVLS multicast mapping when KB200_NVLS=1
    return SymmHeap(nbytes, group=group, backend="host", timeout_s=_WAIT_LIMIT_NS / 1e9 + 5)


def _mc_base(heap: Optional[SymmHeap]):
    """Multicast mapping of the heap for the kernels, or None (peer loads and stores)."""
    return heap.mc_ptr if heap is not None and getattr(heap, "mc_ptr", None) else None


def _host_args(ctx, mode: int, M: int, Nn: int, K: int, a, w, bias, bias_scale: float, out) -> N.GemmArgs:
    args = N.GemmArgs()
    args.mode = mode
    args.M, args.N, args.K = M, Nn, K
    args.A, args.B, args.out = a.data_ptr(), w.data_ptr(), out.data_ptr()
    args.bias = bias.data_ptr() if bias is not None else None
    args.bias_scale = bias_scale
    args.rank, args.world, args.epoch = ctx.rank, ctx.world, ctx.epoch
    args.peer_base = ctx.heap.peer_array()
    args.data_off, args.flag_off = ctx.data_off, ctx.flag_off
    args.wait_limit_ns = _WAIT_LIMIT_NS
    return args


def _rows_bad(rpo: int) -> bool:
    """The tile schedule needs the rows per rank to divide, or be a multiple of, the 128-row block."""
    return rpo <= 0 or (rpo % 128 != 0 and 128 % rpo != 0)


class _HostPipeline:
    """Streams, events and device buffers of a ``run_from_host`` call: chunk i+1 is
    copied in on one stream while chunk i runs on the caller's stream and chunk
    i-1's result is copied out on a third.  Two input and two output buffers.  For
    CPU ranks the three steps simply run one after the other."""

    def __init__(self, device: torch.device, in_shape, out_shape):
        self.cuda = device.type == "cuda"
        self.device = device
        if self.cuda:
            self.h2d, self.d2h = torch.cuda.Stream(device), torch.cuda.Stream(device)
        self.inp = [torch.empty(in_shape, dtype=torch.bfloat16, device=device) for _ in range(2)]
        self.out = [torch.empty(out_shape, dtype=torch.bfloat16, device=device) for _ in range(2)]

    def begin(self, chunks: int) -> None:
        if self.cuda:
            self.cur = torch.cuda.current_stream(self.device)
            self.in_ready, self.computed, self.out_done = ([torch.cuda.Event() for _ in range(chunks)] for _ in range(3))
            self.h2d.wait_stream(self.cur)

    def copy_in(self, i: int, fn) -> None:
        if not self.cuda:
            return fn()
        with torch.cuda.stream(self.h2d):
            if i >= 2:
                self.h2d.wait_event(self.computed[i - 2])  # the kernel that read this buffer has finished
            fn()
            self.in_ready[i].record(self.h2d)

    def compute(self, i: int, fn) -> None:
        if not self.cuda:
            return fn()
        self.cur.wait_event(self.in_ready[i])
        if i >= 2:
            self.cur.wait_event(self.out_done[i - 2])  # its previous result has left the output buffer
        fn()
        self.computed[i].record(self.cur)

    def copy_out(self, i: int, fn) -> None:
        if not self.cuda:
            return fn()
        with torch.cuda.stream(self.d2h):
            self.d2h.wait_event(self.computed[i])
            fn()
            self.out_done[i].record(self.d2h)

    def end(self) -> None:
        if self.cuda:
            self.cur.wait_stream(self.d2h)


def _pieces(M: int, Nn: int, K: int, most: int) -> list:
    """Rows of the pieces of a product on one GPU whose rows come from the host: the fewest microseconds by a model of the three
    stages (53 GB/s each way and 10 for every copy; a product reads its weights at 5.5 TB/s or makes 1200 TFLOP/s) and of
    the host, which takes 30 for a call and 11 for a piece.  Beside a direction that is by far the longer one sizes fall (way in)
    or rise (way out) by a constant ratio, so that little of the other one is exposed: 8192 x 8192 x 1024 2565 us in
    four equal pieces, 2511 in these; 4096 x 1024 x 8192 1312 and 1270.  Where both directions are busy most of the time they slow
    each other down and unequal pieces gain nothing (2048 x 4096 x 7168: 692 and 719; two, eight and sixteen equal ones 756, 735
    and 862).  Whole tiles of 64 rows."""
    best, rows = None, [M]
    blocks = -(-M // 64)
    ratios = (1.0,) if 5 * K < 12 * Nn and 5 * Nn < 12 * K else (1.0, 0.8, 0.65, 0.5, 0.4, 0.3) if K > Nn else (1.0, 1.25, 1.5, 2.0, 2.5, 3.3)
    for n in range(1, min(most, blocks) + 1):
        for ratio in ratios if n > 1 else (1.0,):
            share = [ratio ** i for i in range(n)]
            cut = [round(blocks * sum(share[:i]) / sum(share)) * 64 for i in range(n)] + [M]
            r = [b - a for a, b in zip(cut, cut[1:])]
            if min(r) <= 0:
                continue
            there = made = back = 0.0
            for m in r:
                there += 2 * m * K / 53e3 + 10
                made = max(made, there) + max(2 * m * Nn * K / 1.2e9, 2 * Nn * K / 5.5e6) + 4
                back = max(back, made) + 2 * m * Nn / 53e3 + 10
            t = max(back, 30 + 11 * n)
            if best is None or t < best:
                best, rows = t, r
    return rows


# Rows and result of a `run_from_host` that one GPU holds whole.  Above it the buffers of two chunks of the general path: such a call
# takes 80 ms on the link, beside which the 0.2 ms that the native calls save are nothing, and rows need not fit the GPU's memory.
_WHOLE_ROWS_BYTES = 4 << 30
# Up to here they are held without a look at the memory that is left.
_SMALL_ROWS_BYTES = 64 << 20


def _room(device: torch.device) -> int:
    """Bytes that a tensor can still get on the GPU."""
    return torch.cuda.mem_get_info(device)[0] + torch.cuda.memory_reserved(device) - torch.cuda.memory_allocated(device)


class _OneGpuStream:
    """Device buffers, side streams and events of a context's ``run_from_host`` calls on one GPU (``csrc/kernels/gemm_stream.cu``):
    one pair of buffers for all of them, as large as the largest so far."""

    def __init__(self, device: torch.device, status: torch.Tensor):
        self.device = device
        self.inward, self.outward = torch.cuda.Stream(device), torch.cuda.Stream(device)
        self.inp = self.out = None
        self.kept = []   # pairs that a graph may hold
        self.plans = {}  # (chunks, N, K) -> rows of the pieces, the same for C
        args = self.args = N.GemmStreamArgs()
        args.product = _local_args(status)
        args.inward, args.outward = self.inward.cuda_stream, self.outward.cuda_stream
        self.count, self.events = 0, (C.c_void_p * N.lib().kb_gemm_stream_events(64))()
        self.destroy = N.lib().kb_events_destroy  # at hand when the interpreter has let go of the module
        args.events = C.addressof(self.events)

    def _allocate(self, count: int) -> torch.Tensor:
        return torch.empty(count, dtype=torch.bfloat16, device=self.device)

    def hold(self, a: int, o: int) -> bool:
        """Buffers of at least ``a`` and ``o`` elements; False where they would take more than a quarter of the memory that is left."""
        capturing = torch.cuda.is_current_stream_capturing()
        if self.inp is None or self.inp.numel() < a or self.out.numel() < o:
            had = (self.inp.numel(), self.out.numel()) if self.inp is not None else (0, 0)
            self.inp = self.out = None  # frees the old pair, or leaves it to the graph that has it
            sizes = max(a, had[0]), max(o, had[1])
            if 2 * sum(sizes) > _WHOLE_ROWS_BYTES:
                sizes = a, o
            if not capturing and 2 * sum(sizes) > _SMALL_ROWS_BYTES and 8 * sum(sizes) > _room(self.device):
                return False
            try:
                self.inp, self.out = self._allocate(sizes[0]), self._allocate(sizes[1])
            except torch.OutOfMemoryError:
                self.inp = self.out = None
                return False
            self.inp.record_stream(self.inward)
            self.out.record_stream(self.outward)
            self.home = torch._C._cuda_getCurrentRawStream(self.device.index)
            self.args.product.A, self.args.product.out = self.inp.data_ptr(), self.out.data_ptr()
        if capturing and all(pair[0] is not self.inp for pair in self.kept):
            self.kept.append((self.inp, self.out))
        return True

    def _plan(self, M: int, Nn: int, K: int, chunks: int):
        plan = self.plans.get((chunks, Nn, K))
        if plan is None:
            rows = _pieces(M, Nn, K, max(1, min(chunks, 64)))
            events = N.lib().kb_gemm_stream_events(len(rows))
            if events > self.count:
                more = (C.c_void_p * (events - self.count)).from_buffer(self.events, self.count * C.sizeof(C.c_void_p))
                N.check(N.lib().kb_events_create(events - self.count, more))
                self.count = events
            plan = self.plans[chunks, Nn, K] = (rows, (C.c_int32 * len(rows))(*rows))
        return plan

    def run(self, a_host: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor], bias_scale: float, out_host: torch.Tensor, chunks: int) -> bool:
        global launch_count
        (M, K), Nn = a_host.shape, w.shape[0]
        if not self.hold(M * K, M * Nn):
            return False
        lib, args, index = N.lib(), self.args, self.device.index
        rows, table = self._plan(M, Nn, K, chunks)
        args.product.M, args.product.N, args.product.K = M, Nn, K
        args.product.B, args.product.bias, args.product.bias_scale = w.data_ptr(), bias.data_ptr() if bias is not None else None, bias_scale
        args.a_host, args.out_host = a_host.data_ptr(), out_host.data_ptr()
        args.pieces, args.rows = len(rows), C.addressof(table)
        stream = args.stream = torch._C._cuda_getCurrentRawStream(index)
        if stream != self.home:  # its products may still run when the buffers are freed
            other = torch.cuda.current_stream(w.device)
            self.inp.record_stream(other)
            self.out.record_stream(other)
        first, last = rows[0], M - rows[-1]
        N.check(lib.kb_gemm_stream_begin(C.byref(args)))
        # torch's copies make its allocator of pinned memory wait for the side streams before it hands out a buffer again
        self._copy(self.inward, index, self.inp[:first * K], a_host[:first].view(-1))
        N.check(lib.kb_gemm_stream_run(C.byref(args)))
        self._copy(self.outward, index, out_host[last:].view(-1), self.out[last * Nn:M * Nn])
        N.check(lib.kb_gemm_stream_end(C.byref(args)))
        launch_count += args.pieces
        return True

    @staticmethod
    def _copy(stream: torch.cuda.Stream, index: int, dst: torch.Tensor, src: torch.Tensor) -> None:
        """On ``stream``: what ``with torch.cuda.stream(stream)`` does on the current device, in a tenth of its time."""
        current = torch._C._cuda_getCurrentStream(index)
        torch._C._cuda_setStream(stream_id=stream.stream_id, device_index=stream.device_index, device_type=stream.device_type)
        try:
            dst.copy_(src, non_blocking=True)
        finally:
            torch._C._cuda_setStream(stream_id=current[0], device_index=current[1], device_type=current[2])

    def __del__(self):
        events, destroy = getattr(self, "events", None), getattr(self, "destroy", None)
        if events is not None and destroy is not None:
            destroy(len(events), events)


def _from_host_on_one_gpu(ctx, a_host: torch.Tensor, w: torch.Tensor, bias, bias_scale: float, out_host: torch.Tensor, chunks: int) -> bool:
    """``run_from_host`` where nothing is exchanged and the weights are on the current device; False elsewhere."""
    if ctx.world != 1 or chunks < 1 or not ctx.native or not w.is_cuda or w.device.index != torch._C._cuda_getDevice():
        return False
    (M, K), Nn = a_host.shape, w.shape[0]
    if 2 * M * (Nn + K) > _WHOLE_ROWS_BYTES:
        return False
    states = ctx.__dict__.setdefault("_one_gpu_streams", {})
    st = states.get(w.device.index)
    if st is None:
        st = states[w.device.index] = _OneGpuStream(w.device, ctx.status)
    if not st.run(a_host, w, bias, bias_scale, out_host, chunks):
        return False
    ctx.epoch += 1
    return True


def _host_buffer(shape) -> torch.Tensor:
    t = torch.empty(shape, dtype=torch.bfloat16)
    return t.pin_memory() if torch.cuda.is_available() else t


def _check_pinned(t: torch.Tensor, name: str, shape) -> None:
    if t.is_cuda or t.dtype != torch.bfloat16 or tuple(t.shape) != tuple(shape) or not t.is_contiguous():
        raise ValueError(f"{name} must be a contiguous bf16 host tensor of shape {tuple(shape)}")
    if not os.environ.get("KB200_ALLOW_PAGEABLE") and torch.cuda.is_available() and not t.is_pinned():
        raise ValueError(f"{name} must be in pinned host memory (tensor.pin_memory()), or the copies cannot overlap the kernel")


def gemm(a: torch.Tensor, b: torch.Tensor, bias: Optional[torch.Tensor] = None, out: Optional[torch.Tensor] = None,
         bias_scale: float = 1.0, status: Optional[torch.Tensor] = None, num_ctas: int = 0,
         pair: Optional[bool] = None) -> torch.Tensor:
    """``out[M,N] = a[M,K] @ b[N,K]^T (+ bias_scale * bias)`` in bf16 with fp32 accumulation.

    ``pair=True`` uses clusters of two CTAs sharing 256x256 tiles (``cta_group::2``,
    more than 128 rows), ``pair=False`` tiles of one CTA, both with the rows on the tensor cores' M side;
    ``None`` lets the launcher pick the side and the tile from the sizes (``choose`` in ``csrc/kernels/gemm_local.cu``)."""
    _check_bf16_2d(a, "a")
    _check_bf16_2d(b, "b")
    M, K = a.shape
    Nn = b.shape[0]
    if b.shape[1] != K:
        raise ValueError("inner dimensions differ")
    if not a.is_cuda:
        res = a.float() @ b.float().t()
        if bias is not None:
            res = res + bias_scale * bias.float()
        res = res.to(torch.bfloat16)
        if out is not None:
            out.copy_(res)
            return out
        return res
    if out is None:
        out = torch.empty((M, Nn), dtype=torch.bfloat16, device=a.device)
    _check_out(out, M, Nn, a.device)
    args = _local_args(status)
    args.M, args.N, args.K = M, Nn, K
    args.A, args.B, args.out = a.data_ptr(), b.data_ptr(), out.data_ptr()
    args.bias = bias.data_ptr() if bias is not None else None
    args.bias_scale = bias_scale
    args.num_ctas = num_ctas
    args.pair = -1 if pair is None else int(pair)
    _launch_local(args, a.device)
    return out


class GemmRS:
    """GEMM fused with reduce-scatter for one problem shape.

    Each rank holds ``a[M, K_local]`` and ``w[N, K_local]``; the result
    ``sum_r a_r @ w_r^T (+ bias_scale * bias)`` is row-scattered so that this
    rank returns rows ``[rank*M/world, (rank+1)*M/world)``.  Construction is
    collective (it allocates symmetric staging memory); calls are collective in
    the sense that every rank must make the same sequence of calls.
    """

    def __init__(self, M: int, Nn: int, group=None, device: Optional[torch.device] = None, heap: Optional[SymmHeap] = None):
        self.M, self.N = M, Nn
        self.group = group
        self.rank, self.world = _dist_info(group)
        if M % self.world:
            raise ValueError("M must be divisible by the world size")
        self.native = torch.cuda.is_available() and (device is None or torch.device(device).type == "cuda")
        self.epoch = 0
        self.heap = None
        self._hot = None
        self.host_heap = not self.native and self.world > 1 and _cpu_heap_path() and not _rows_bad(M // self.world)
        if (self.native and self.world > 1) or self.host_heap:
            lib = N.lib()
            data = int(lib.kb_gemm_rs_data_bytes(M, Nn, self.world))
            flags = int(lib.kb_gemm_rs_flag_bytes(M, Nn, self.world))
            self.heap = heap or _new_heap(data + flags + 1024, group, device, self.native)
            self.data_off = self.heap.alloc(data)
            self.flag_off = self.heap.alloc(flags)
            self.status = self.heap.status
        elif self.native:
            self.status = torch.zeros(8, dtype=torch.int32, device=device or torch.device("cuda", torch.cuda.current_device()))

    def __call__(self, a: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None, bias_scale: float = 1.0,
                 out: Optional[torch.Tensor] = None) -> torch.Tensor:
        _check_bf16_2d(a, "a")
        _check_bf16_2d(w, "w")
        M, K = a.shape
        if M != self.M or w.shape[0] != self.N or w.shape[1] != K:
            raise ValueError("shape does not match this GemmRS context")
        rows = M // self.world
        if not a.is_cuda and self.host_heap:
            if out is None:
                out = torch.empty((rows, self.N), dtype=torch.bfloat16)
            self.epoch += 1
            args = _host_args(self, N.GEMM_RS, M, self.N, K, a, w, bias, bias_scale, out)
            N.check(N.lib().kb_gemm_host(C.byref(args), max(1, _WAIT_LIMIT_NS // 1_000_000)))
            return out
        if not a.is_cuda:
            full = a.float() @ w.float().t()
            full = full.to(torch.bfloat16)
            res = torch.empty((rows, self.N), dtype=torch.bfloat16)
            if self.world > 1:
                dist.reduce_scatter_tensor(res, full, group=self.group)
            else:
                res.copy_(full)
            if bias is not None:
                res = (res.float() + bias_scale * bias.float()).to(torch.bfloat16)
            if out is not None:
                out.copy_(res)
                return out
            return res
        if out is None:
            out = torch.empty((rows, self.N), dtype=torch.bfloat16, device=a.device)
        self.epoch += 1
        if self.world == 1:
            return _run_local(self, a, w, bias, bias_scale, out)
        args = self._hot
        if args is None:  # built once; calls only refresh pointers, K and the epoch
            args = self._hot = N.GemmArgs()
            args.mode = N.GEMM_RS
            args.M, args.N = M, self.N
            args.rank, args.world = self.rank, self.world
            if self.heap is not None:
                args.peer_base = self.heap.peer_array()
                args.data_off, args.flag_off = self.data_off, self.flag_off
                args.mc_base = _mc_base(self.heap)
            args.status = self.status.data_ptr()
            args.wait_limit_ns = _WAIT_LIMIT_NS
        args.K = K
        args.A, args.B, args.out = a.data_ptr(), w.data_ptr(), out.data_ptr()
        args.bias = bias.data_ptr() if bias is not None else None
        args.bias_scale = bias_scale
        args.epoch = self.epoch
        _launch(args, a.device)
        return out

    def recover(self) -> None:
        """Collective.  After ``heap.check_status()`` reported a failed wait: waits
        for this rank's kernels, clears the status words and moves every rank to the
        same call number, past every flag value already written."""
        if self.heap is None:
            return
        if self.native:
            torch.cuda.synchronize(self.heap.device)
        self.heap.status.zero_()
        self.epoch = self.heap.agree_epoch(self.epoch) + 1
        self.heap._control_barrier()

    def run_from_host(self, a_host: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None,
                      bias_scale: float = 1.0, out_host: Optional[torch.Tensor] = None, chunks: int = 4) -> torch.Tensor:
        """The op with its activations in pinned host memory and its result wanted
        there: ``a_host [M, K_local]`` -> ``out_host [M/world, N]`` (``w``, ``bias`` on
        the device).  The rows every rank owns are cut into ``chunks`` pieces; piece i
        of all owners forms a problem of ``M/chunks`` rows that runs through the
        same fused kernel, while piece i+1 is on its way in and the result of
        piece i-1 on its way out (one ``cudaMemcpyAsync`` per contiguous block), so
        the PCIe transfers overlap the kernel instead of bracketing it.  On one GPU, where
        any rows can form a piece, there are at most ``chunks``, of the sizes that pay (``_pieces``).  Returns
        ``out_host``; the caller's stream is done when everything has arrived.
        Calls of one context share device buffers; on one GPU a call waits for the one before it, also on another stream, but
        replays of a graph that holds a call are for the program to order against other calls.
        Collective like ``__call__``.  The reference has no counterpart (its
        evaluator clones the inputs on the device inside its timed region,
        ``eval.py:358``)."""
        world, M, Nn = self.world, self.M, self.N
        rows_rank, asked = M // world, chunks
        while chunks > 1 and (rows_rank % chunks or _rows_bad(rows_rank // chunks)):
            chunks -= 1
        rows = rows_rank // chunks
        K = a_host.shape[1]
        _check_pinned(a_host, "a_host", (M, K))
        if out_host is None:
            out_host = _host_buffer((rows_rank, Nn))
        _check_pinned(out_host, "out_host", (rows_rank, Nn))
        dev = w.device
        if world == 1 and dev.type == "cuda":
            _check_bf16_2d(w, "w")
            if w.shape[0] != Nn or w.shape[1] != K:
                raise ValueError("shape does not match this GemmRS context")
            if _from_host_on_one_gpu(self, a_host, w, bias, bias_scale, out_host, asked):
                return out_host
        key = (chunks, K)
        st = self._stream_state.get(key) if hasattr(self, "_stream_state") else None
        if st is None:
            if not hasattr(self, "_stream_state"):
                self._stream_state = {}
            sub = self if chunks == 1 else GemmRS(M // chunks, Nn, group=self.group, device=dev)
            st = self._stream_state[key] = (sub, _HostPipeline(dev, (world, rows, K), (rows, Nn)))
        sub, pipe = st
        src = a_host.view(world, chunks, rows, K)
        dst = out_host.view(chunks, rows, Nn)
        pipe.begin(chunks)
        for i in range(chunks):
            buf, res = pipe.inp[i % 2], pipe.out[i % 2]

            def copy_in():
                for r in range(world):
                    buf[r].copy_(src[r, i], non_blocking=True)

            pipe.copy_in(i, copy_in)
            pipe.compute(i, lambda: sub(buf.view(world * rows, K), w, bias, bias_scale=bias_scale, out=res))
            pipe.copy_out(i, lambda: dst[i].copy_(res, non_blocking=True))
        pipe.end()
        return out_host

    def close(self) -> None:
        """Frees this context's workspaces (collective)."""
        for sub, _ in getattr(self, "_stream_state", {}).values():
            if sub is not self and sub.heap is not None:
                sub.heap.close()
        self._stream_state = {}
        self.__dict__.pop("_one_gpu_streams", None)
        if self.heap is not None:
            self.heap.close()


class AGGemm:
    """All-gather fused with GEMM for one problem shape.

    Each rank holds ``a_local[M/world, K]`` and a column shard ``w[N_local, K]``;
    returns ``all_gather(a_local) @ w^T (+ bias)`` of shape ``[M, N_local]``.
    """

    def __init__(self, M: int, K: int, group=None, device: Optional[torch.device] = None, heap: Optional[SymmHeap] = None):
        self.M, self.K = M, K
        self.group = group
        self.rank, self.world = _dist_info(group)
        if M % self.world:
            raise ValueError("M must be divisible by the world size")
        self.native = torch.cuda.is_available() and (device is None or torch.device(device).type == "cuda")
        self.epoch = 0
        self.heap = None
        self._hot = None
        self.host_heap = not self.native and self.world > 1 and _cpu_heap_path() and not _rows_bad(M // self.world)
        if (self.native and self.world > 1) or self.host_heap:
            lib = N.lib()
            data = int(lib.kb_gemm_ag_data_bytes(M, K))
            flags = int(lib.kb_gemm_ag_flag_bytes(M, self.world))
            ctr = int(lib.kb_gemm_ag_counter_bytes(M, self.world))
            self.heap = heap or _new_heap(data + flags + ctr + 2048, group, device, self.native)
            self.data_off = self.heap.alloc(data)
            self.flag_off = self.heap.alloc(flags)
            self.counter_off = self.heap.alloc(ctr)
            self.status = self.heap.status
        elif self.native:
            self.status = torch.zeros(8, dtype=torch.int32, device=device or torch.device("cuda", torch.cuda.current_device()))

    def check(self, a_local: torch.Tensor, w: torch.Tensor) -> None:
        """Raises unless the operands fit this context."""
        _check_bf16_2d(a_local, "a_local")
        _check_bf16_2d(w, "w")
        rows, K = a_local.shape
        if rows * self.world != self.M or K != self.K or w.shape[1] != K:
            raise ValueError("shape does not match this AGGemm context")

    def __call__(self, a_local: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None,
                 out: Optional[torch.Tensor] = None) -> torch.Tensor:
        self.check(a_local, w)
        Nl, K = w.shape
        if not a_local.is_cuda and self.host_heap:
            if out is None:
                out = torch.empty((self.M, Nl), dtype=torch.bfloat16)
            self.epoch += 1
            args = _host_args(self, N.GEMM_AG, self.M, Nl, K, a_local, w, bias, 1.0, out)
            N.check(N.lib().kb_gemm_host(C.byref(args), max(1, _WAIT_LIMIT_NS // 1_000_000)))
            return out
        if not a_local.is_cuda:
            full = torch.empty((self.M, K), dtype=a_local.dtype)
            if self.world > 1:
                dist.all_gather_into_tensor(full, a_local, group=self.group)
            else:
                full.copy_(a_local)
            res = full.float() @ w.float().t()
            if bias is not None:
                res = res + bias.float()
            res = res.to(torch.bfloat16)
            if out is not None:
                out.copy_(res)
                return out
            return res
        if out is None:
            out = torch.empty((self.M, Nl), dtype=torch.bfloat16, device=a_local.device)
        self.epoch += 1
        if self.world == 1:
            return _run_local(self, a_local, w, bias, 1.0, out)
        args = self._hot
        if args is None:
            args = self._hot = N.GemmArgs()
            args.mode = N.GEMM_AG
            args.M, args.K = self.M, K
            args.bias_scale = 1.0
            args.rank, args.world = self.rank, self.world
            if self.heap is not None:
                args.peer_base = self.heap.peer_array()
                args.data_off, args.flag_off, args.counter_off = self.data_off, self.flag_off, self.counter_off
                args.mc_base = _mc_base(self.heap)
            args.status = self.status.data_ptr()
            args.wait_limit_ns = _WAIT_LIMIT_NS
        args.N = Nl
        args.A, args.B, args.out = a_local.data_ptr(), w.data_ptr(), out.data_ptr()
        args.bias = bias.data_ptr() if bias is not None else None
        args.epoch = self.epoch
        _launch(args, a_local.device)
        return out

    def recover(self) -> None:
        """Collective.  After ``heap.check_status()`` reported a failed wait: waits
        for this rank's kernels, clears the status words, zeroes the push counters
        and moves every rank to the same call number, past every flag value already
        written."""
        if self.heap is None:
            return
        if self.native:
            torch.cuda.synchronize(self.heap.device)
        self.heap.status.zero_()
        self.heap.tensor(self.counter_off, (256,), torch.int32).zero_()
        self.epoch = self.heap.agree_epoch(self.epoch) + 1
        if self.native:
            torch.cuda.synchronize(self.heap.device)
        self.heap._control_barrier()

    def run_from_host(self, a_host: torch.Tensor, w: torch.Tensor, bias: Optional[torch.Tensor] = None,
                      out_host: Optional[torch.Tensor] = None, chunks: int = 4) -> torch.Tensor:
        """The op with its activations in pinned host memory and its result wanted
        there: ``a_host [M/world, K]`` -> ``out_host [M, N_local]``.  This rank's rows
        are cut into ``chunks`` pieces; piece i of every rank forms a gathered problem
        of ``M/chunks`` rows for the same fused kernel, overlapped with the copy of
        piece i+1 coming in and of piece i-1's result going out (see
        ``GemmRS.run_from_host``).  Collective like ``__call__``."""
        world, M, K = self.world, self.M, self.K
        rows_rank, asked = M // world, chunks
        while chunks > 1 and (rows_rank % chunks or _rows_bad(rows_rank // chunks)):
            chunks -= 1
        rows = rows_rank // chunks
        Nl = w.shape[0]
        _check_pinned(a_host, "a_host", (rows_rank, K))
        if out_host is None:
            out_host = _host_buffer((M, Nl))
        _check_pinned(out_host, "out_host", (M, Nl))
        dev = w.device
        if world == 1 and dev.type == "cuda":
            _check_bf16_2d(w, "w")
            if w.shape[1] != K:
                raise ValueError("shape does not match this AGGemm context")
            if _from_host_on_one_gpu(self, a_host, w, bias, 1.0, out_host, asked):
                return out_host
        key = (chunks, Nl)
        st = self._stream_state.get(key) if hasattr(self, "_stream_state") else None
        if st is None:
            if not hasattr(self, "_stream_state"):
                self._stream_state = {}
            sub = self if chunks == 1 else AGGemm(M // chunks, K, group=self.group, device=dev)
            st = self._stream_state[key] = (sub, _HostPipeline(dev, (rows, K), (world, rows, Nl)))
        sub, pipe = st
        src = a_host.view(chunks, rows, K)
        dst = out_host.view(world, chunks, rows, Nl)
        pipe.begin(chunks)
        for i in range(chunks):
            buf, res = pipe.inp[i % 2], pipe.out[i % 2]

            def copy_out():
                for r in range(world):
                    dst[r, i].copy_(res[r], non_blocking=True)

            pipe.copy_in(i, lambda: buf.copy_(src[i], non_blocking=True))
            pipe.compute(i, lambda: sub(buf, w, bias, out=res.view(world * rows, Nl)))
            pipe.copy_out(i, copy_out)
        pipe.end()
        return out_host

    def close(self) -> None:
        """Frees this context's workspaces (collective)."""
        for sub, _ in getattr(self, "_stream_state", {}).values():
            if sub is not self and sub.heap is not None:
                sub.heap.close()
        self._stream_state = {}
        self.__dict__.pop("_one_gpu_streams", None)
        if self.heap is not None:
            self.heap.close()
