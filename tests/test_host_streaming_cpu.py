"""``run_from_host`` of the two fused GEMM front-ends on CPU ranks: the chunked
row bookkeeping (which rows of the host tensors form which sub-problem) against
the un-chunked call.  The overlap of copies and kernels needs a GPU and is
covered by the GPU tests; the arithmetic of the split does not."""
import pytest
import torch

from _mp import run_ranks


def _rs(rank, world, M, Nn, Kl, chunks):
    from kernel_b200.ops.gemm import GemmRS

    ctx = GemmRS(M, Nn, device="cpu")
    g = torch.Generator().manual_seed(5 + rank)
    a = torch.randn(M, Kl, generator=g).to(torch.bfloat16)
    w = (torch.randn(Nn, Kl, generator=g) / Kl ** 0.5).to(torch.bfloat16)
    bias = (torch.randn(Nn, generator=torch.Generator().manual_seed(1)) * 0.1).to(torch.bfloat16)
    whole = ctx(a, w, bias, bias_scale=2.0)
    streamed = ctx.run_from_host(a, w, bias, bias_scale=2.0, chunks=chunks)
    again = ctx.run_from_host(a, w, bias, bias_scale=2.0, out_host=torch.empty_like(streamed), chunks=chunks)
    ctx.close()
    return bool(torch.equal(whole, streamed)), bool(torch.equal(streamed, again)), tuple(streamed.shape)


def _ag(rank, world, M, Nl, K, chunks):
    from kernel_b200.ops.gemm import AGGemm

    ctx = AGGemm(M, K, device="cpu")
    g = torch.Generator().manual_seed(9 + rank)
    a = torch.randn(M // world, K, generator=g).to(torch.bfloat16)
    w = (torch.randn(Nl, K, generator=g) / K ** 0.5).to(torch.bfloat16)
    bias = (torch.randn(Nl, generator=g) * 0.1).to(torch.bfloat16)
    whole = ctx(a, w, bias)
    streamed = ctx.run_from_host(a, w, bias, chunks=chunks)
    ctx.close()
    return bool(torch.equal(whole, streamed)), True, tuple(streamed.shape)


@pytest.mark.parametrize("world,M,chunks", [(1, 512, 4), (2, 1024, 4), (2, 512, 3), (4, 1024, 2)])
def test_gemm_rs_streamed_equals_whole(world, M, chunks):
    for same, repeat, shape in run_ranks(_rs, world, M, 264, 40, chunks):
        assert same and repeat and shape == (M // world, 264)


@pytest.mark.parametrize("world,M,chunks", [(1, 512, 4), (2, 1024, 4), (4, 1024, 2)])
def test_ag_gemm_streamed_equals_whole(world, M, chunks):
    for same, _, shape in run_ranks(_ag, world, M, 136, 72, chunks):
        assert same and shape == (M, 136)


def test_pieces_are_the_rows():
    from kernel_b200.ops.gemm import _pieces

    for M, N, K in [(1, 8, 8), (63, 8, 8192), (64, 4096, 4096), (65, 8192, 1024), (2047, 1024, 8192), (8192, 8192, 8192), (16384, 1024, 1024)]:
        for most in (1, 2, 4, 7, 64):
            rows = _pieces(M, N, K, most)
            assert sum(rows) == M and min(rows) > 0 and len(rows) <= most
            assert all(r % 64 == 0 for r in rows[:-1])
    assert len(_pieces(256, 1024, 1024, 4)) == 1 and _pieces(2048, 4096, 7168, 4) == [512] * 4
    assert _pieces(8192, 8192, 1024, 4) == sorted(_pieces(8192, 8192, 1024, 4)) and _pieces(4096, 1024, 8192, 4)[0] > 2048


def test_stream_arguments_are_checked():
    """Before anything is asked of the device."""
    import ctypes as C

    from kernel_b200 import _native as N

    def code(rows, M=128, **kw):
        table = (C.c_int32 * max(1, len(rows)))(*rows)
        events = (C.c_void_p * 64)()
        a = N.GemmStreamArgs()
        a.product.M, a.product.N, a.product.K = M, 8, 8
        a.pieces, a.rows, a.events, a.a_host, a.out_host = len(rows), C.addressof(table), C.addressof(events), 16, 16
        for k, v in kw.items():
            setattr(a, k, v)
        return N.lib().kb_gemm_stream_run(C.byref(a))

    for bad in (dict(rows=[]), dict(rows=[64, 63]), dict(rows=[128, 0]), dict(rows=[192, -64]), dict(rows=[2] * 65, M=130), dict(rows=[128], a_host=None),
                dict(rows=[128], out_host=None), dict(rows=[128], events=None)):
        assert code(**bad) == N.KB_ERR_ARG, bad
