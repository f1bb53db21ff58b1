"""Small single-GPU cases of each hand-written kernel, for profilers.

    python -m kernel_b200.utils.profile_cases gemm   [--m 8192 --n 8192 --k 2048] [--iters 3]
    python -m kernel_b200.utils.profile_cases a2a    [--tokens 256] [--iters 3]
    python -m kernel_b200.utils.profile_cases a2a3   (the three-launch variant)
    python -m kernel_b200.utils.profile_cases local  (one launch of each kernel of the one-GPU path per iteration)

Each case holds a few hundred MB on the device (more than the L2, far less than
a full-size workload), runs a handful of launches and exits, so that a capture
ends by itself.  On one GPU the reduce-scatter and all-gather variants of the
GEMM reduce to a plain product and the round trip to one pass over the rows; their communication paths need several ranks
and are measured with CUDA events instead (``kernel_b200.utils.sweep``).
"""
from __future__ import annotations

import argparse
import os

import torch


def run_gemm(m: int, n: int, k: int, iters: int, pair=None) -> None:
    from ..ops.gemm import gemm

    dev = torch.device("cuda", 0)
    torch.manual_seed(0)
    a = torch.randn(m, k, device=dev).to(torch.bfloat16)
    b = (torch.randn(n, k, device=dev) / k ** 0.5).to(torch.bfloat16)
    bias = (torch.randn(n, device=dev) * 0.02).to(torch.bfloat16)
    out = torch.empty(m, n, device=dev, dtype=torch.bfloat16)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    for i in range(iters):
        if i == iters - 1:
            ev[0].record()
        gemm(a, b, bias, out=out, pair=pair)
    ev[1].record()
    torch.cuda.synchronize()
    us = ev[0].elapsed_time(ev[1]) * 1e3
    ref = a[:256].float() @ b.float().t() + bias.float()
    err = (out[:256].float() - ref).abs().max().item()
    print(f"gemm {m}x{n}x{k}: {us:.1f} us, {2 * m * n * k / us / 1e6:.1f} TFLOP/s, max err {err:.4f}")


def run_a2a(tokens: int, iters: int, fused: bool) -> None:
    os.environ["KB200_A2A_FUSED"] = "1" if fused else "0"
    from ..ops.dispatch_combine import SCALE_EXPERT, MoEAllToAll

    dev = torch.device("cuda", 0)
    torch.manual_seed(0)
    E, k, H = 256, 8, 7168
    ctx = MoEAllToAll(E, k, H, tokens, dtype=torch.bfloat16, device=dev)
    x = torch.randn(tokens, H, device=dev).to(torch.bfloat16)
    idx = torch.rand(tokens, E, device=dev).argsort(1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn(tokens, k, device=dev), -1)
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    for i in range(iters):
        if i == iters - 1:
            ev[0].record()
        out = ctx.dispatch_scale_combine(x, idx, w, SCALE_EXPERT)
    ev[1].record()
    torch.cuda.synchronize()
    ctx.heap.check_status()
    print(f"a2a T={tokens} fused={fused}: {ev[0].elapsed_time(ev[1]) * 1e3:.1f} us, out mean {out.float().abs().mean().item():.4f}")


def run_local(iters: int) -> None:
    from ..ops import local as L
    from ..ops.dispatch_combine import SCALE_EXPERT, MoEAllToAll

    dev = torch.device("cuda", 0)
    torch.manual_seed(0)

    def normal(*shape):
        return torch.randn(*shape, device=dev).to(torch.bfloat16)

    def routing(tokens, experts, k):
        return torch.rand(tokens, experts, device=dev).argsort(1)[:, :k].to(torch.int32).contiguous(), torch.rand(tokens, k, device=dev)

    E, H, F = 64, 2048, 1024

    def rows(n):
        return torch.arange(E, dtype=torch.int32, device=dev) * n, torch.full((E,), n, dtype=torch.int32, device=dev)

    dense = [(normal(m, k), normal(n, k)) for m, n, k in ((8192, 8192, 2048), (64, 7168, 18432), (256, 14336, 4096), (256, 4096, 14336))]
    w_up, w_down, few, many = normal(E, F, H), normal(E, H, F), normal(E * 4, H), normal(E * 128, H)
    pre, tokens, (idx, weights) = normal(E * 128, F), normal(1024, H), routing(1024, E, 8)
    ctx = MoEAllToAll(256, 8, 7168, 2048, dtype=torch.bfloat16, device=dev)
    x, (a2a_idx, a2a_weights), wide = normal(2048, 7168), routing(2048, 256, 8), normal(8192, 29568)
    er = L.ExpertRows(tokens, idx, E, pad=64)
    y = er.combine(er.rows, weights)
    launches = [
        *((f"dense {a.shape[0]} x {b.shape[0]} x {a.shape[1]}", lambda a=a, b=b: L.product(a, b)) for a, b in dense),
        ("rows, 64 groups of 4, 1024 x 2048, SiLU", lambda: L.rows_product(few, w_up, *rows_few, act="silu")),
        ("rows, 64 groups of 128, 1024 x 2048, SiLU kept", lambda: L.rows_product(many, w_up, *rows_many, act="silu", pre_out=pre)),
        ("rows, 64 groups of 128, 1024 x 2048 from [2048, 1024], slope",
         lambda: L.rows_product(many, w_down, *rows_many, b_t=True, act="silu", pre_in=pre)),
        ("contract, 64 groups of 128, 2048 x 1024", lambda: L.contract_product(many, pre, *rows_many)),
        ("permute 1024 x 2048, top-8 of 64", lambda: L.ExpertRows(tokens, idx, E, pad=64)),
        ("combine 1024 x 2048, top-8", lambda: er.combine(er.rows, weights)),
        ("grad_rows 1024 x 2048, top-8", lambda: er.grad_rows(y, er.rows, weights)),
        ("round trip 2048 x 7168, top-8 of 256", lambda: ctx.dispatch_scale_combine(x, a2a_idx, a2a_weights, SCALE_EXPERT)),
        ("column sums 8192 x 29568 (two launches)", lambda: L.col_sum(wide)),
    ]
    rows_few, rows_many = rows(4), rows(128)
    for i in range(iters):
        for name, launch in launches:
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            torch.cuda._sleep(400000)  # the launch is queued before the first event is reached
            ev[0].record()
            launch()
            ev[1].record()
            ev[1].synchronize()
            if i == iters - 1:
                print(f"{name}: {ev[0].elapsed_time(ev[1]) * 1e3:.1f} us")
    ctx.heap.check_status()


def main() -> None:
    ap = argparse.ArgumentParser()
    ap.add_argument("case", choices=["gemm", "a2a", "a2a3", "local"])
    ap.add_argument("--m", type=int, default=8192)
    ap.add_argument("--n", type=int, default=8192)
    ap.add_argument("--k", type=int, default=2048)
    ap.add_argument("--tokens", type=int, default=256)
    ap.add_argument("--iters", type=int, default=3)
    ap.add_argument("--pair", type=int, default=None, help="gemm: 1 = CTA-pair kernel, 0 = single-CTA kernel, default: the faster of the two")
    ns = ap.parse_args()
    if ns.case == "gemm":
        run_gemm(ns.m, ns.n, ns.k, ns.iters, None if ns.pair is None else bool(ns.pair))
    elif ns.case == "local":
        run_local(ns.iters)
    else:
        run_a2a(ns.tokens, ns.iters, fused=ns.case == "a2a")


if __name__ == "__main__":
    main()
