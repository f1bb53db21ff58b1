"""Refusals of the one-GPU front-ends (``ops/local.py``): operands whose addresses the kernels
take are checked on the host, before any launch, so the refusals show on CPU tensors too."""
import pytest
import torch

from kernel_b200.ops import local as L

E, R, Nn, K = 2, 8, 24, 16


def _z(*shape, dtype=torch.bfloat16):
    return torch.zeros(*shape, dtype=dtype)


def _table(n=E, dtype=torch.int32):
    return torch.tensor([0, 4][:n], dtype=dtype), torch.tensor([4, 4][:n], dtype=dtype)


# expert weights that do not fit the rows: a dtype the kernel would misread, a transposed matrix, extents that
# would make it read past the tensor
BAD_WEIGHTS = [_z(E, Nn, K, dtype=torch.float32), _z(E, Nn, K, dtype=torch.float16), _z(E, K, Nn).transpose(1, 2),
               _z(E, Nn, K - 8), _z(E, Nn, K + 8), _z(Nn, K)]


@pytest.mark.parametrize("b", BAD_WEIGHTS)
def test_rows_product_refuses_weights(b):
    with pytest.raises(ValueError):
        L.rows_product(_z(R, K), b, *_table())
    if b.is_contiguous():
        with pytest.raises(ValueError):
            L.rows_product(_z(R, K), b.transpose(-1, -2).contiguous(), *_table(), b_t=True)


@pytest.mark.parametrize("kw", [dict(out=_z(R, Nn + 8)), dict(out=_z(R - 1, Nn)), dict(out=_z(R, Nn, dtype=torch.float32)),
                                dict(out=_z(Nn, R).t()), dict(pre_out=_z(R, 8), act="silu"), dict(pre_in=_z(R + 1, Nn), act="silu")])
def test_products_refuse_results_of_another_form(kw):
    with pytest.raises(ValueError):
        L.rows_product(_z(R, K), _z(E, Nn, K), *_table(), **kw)
    with pytest.raises(ValueError):
        L.product(_z(R, K), _z(Nn, K), **kw)


def test_grouped_products_refuse_tables():
    a, b = _z(R, K), _z(E, Nn, K)
    start, count = _table()
    for s, c in [(start.long(), count), (start, count.float()), (start[:1], count), (start, count[:1]), (start.repeat(2)[::2], count)]:
        with pytest.raises(ValueError):
            L.rows_product(a, b, s, c)
    with pytest.raises(ValueError):
        L.rows_product(a, b, *_table(1))
    with pytest.raises(ValueError):
        L.contract_product(a, _z(R, Nn), start, count.long())


@pytest.mark.parametrize("a,b", [(_z(R, K), _z(R - 1, Nn)), (_z(R, K, dtype=torch.float32), _z(R, Nn)), (_z(R, K), _z(R, Nn, dtype=torch.float16)),
                                 (_z(K, R).t(), _z(R, Nn)), (_z(R, K), _z(Nn, R).t())])
def test_contract_product_refuses_operands(a, b):
    with pytest.raises(ValueError):
        L.contract_product(a, b, *_table())


@pytest.mark.parametrize("a_t,b_t", [(False, False), (False, True), (True, True)])
def test_product_refuses_operands(a_t, b_t):
    a, b = _z(*((K, R) if a_t else (R, K))), _z(*((K, Nn) if b_t else (Nn, K)))
    assert L.product(a, b, a_t=a_t, b_t=b_t).shape == (R, Nn)
    short = _z(*((K - 8, Nn) if b_t else (Nn, K - 8)))
    for x, y in [(a.float(), b), (a, b.half()), (a.t().contiguous().t(), b), (a, b.t().contiguous().t()), (a, short), (a, b[None])]:
        with pytest.raises(ValueError):
            L.product(x, y, a_t=a_t, b_t=b_t)


def test_expert_matrices_that_are_contiguous_one_by_one_are_taken():
    g = torch.Generator().manual_seed(0)
    a = torch.randn(R, K, generator=g).to(torch.bfloat16)
    big = torch.randn(2 * E, Nn, K, generator=g).to(torch.bfloat16)
    for b in (big[::2], big[:1].expand(E, Nn, K)):
        assert not b.is_contiguous()
        assert torch.equal(L.rows_product(a, b, *_table()), L.rows_product(a, b.contiguous(), *_table()))


H, F = 64, 128
LAYER_WEIGHTS = {"fp32": (_z(E, F, H, dtype=torch.float32), _z(E, H, F, dtype=torch.float32)),
                 "fp16": (_z(E, F, H, dtype=torch.float16), _z(E, H, F, dtype=torch.float16)),
                 "up_short": (_z(E, F, H - 8), _z(E, H, F)), "down_short": (_z(E, F, H), _z(E, H, F - 8))}


@pytest.mark.parametrize("which", list(LAYER_WEIGHTS) + ["transposed"])
def test_moe_layers_refuse_weights(which):
    from kernel_b200.models import MoELayer, TrainableMoELayer

    x, idx, w = _z(3, H), torch.tensor([[0, 1]] * 3, dtype=torch.int32), torch.ones(3, 2)
    layer = TrainableMoELayer(E, 2, H, F, 4)
    layer.w_up.data, layer.w_down.data = LAYER_WEIGHTS.get(which, (_z(E, H, F).transpose(1, 2), _z(E, H, F)))
    with pytest.raises(ValueError):
        layer(x, idx, w)
    layer.close()
    if which in LAYER_WEIGHTS:  # MoELayer makes its weights contiguous
        layer = MoELayer(E, 2, H, 4, *LAYER_WEIGHTS[which])
        with pytest.raises(ValueError):
            layer(x, idx, w)
        layer.close()


def test_expert_rows_refuse_what_they_would_misread():
    er = L.ExpertRows.saved(_z(R, K), torch.zeros(3 * E + R, dtype=torch.int32), R // 2, 2, E)
    w = torch.ones(R // 2, 2)
    for y, weights in [(_z(R, K - 8), w), (_z(R - 1, K), w), (_z(R, K, dtype=torch.float32), w), (_z(R, K), w.double()), (_z(R, K), torch.ones(R, 1))]:
        with pytest.raises(ValueError):
            er.combine(y, weights)
    with pytest.raises(ValueError):
        er.grad_rows(_z(R, K), _z(R, K), w)
    for x, idx in [(_z(R, K, dtype=torch.float32), torch.zeros(R, 2, dtype=torch.int32)), (_z(R, K), torch.zeros(R, 2)),
                   (_z(R, K), torch.zeros(R - 1, 2, dtype=torch.int32)), (_z(K, R).t(), torch.zeros(R, 2, dtype=torch.int32))]:
        with pytest.raises(ValueError):
            L.ExpertRows(x, idx, E)


@pytest.mark.parametrize("shape", [(8, 24), (8 * 24,), (24, 8), (8, 64), (2, 8, 24)])
def test_one_rank_product_takes_its_columns_from_the_weights(shape, monkeypatch):
    """``out`` is an address: a flat or a larger buffer receives the same matrix."""
    from types import SimpleNamespace

    from kernel_b200.ops import gemm as G

    seen = []
    monkeypatch.setattr(G, "_launch_local", lambda args, device: seen.append((args.M, args.N, args.K)))
    G._run_local(SimpleNamespace(_hot=None, status=None), _z(R, K), _z(Nn, K), None, 1.0, _z(*shape))
    assert seen == [(R, Nn, K)]


@pytest.mark.parametrize("out", [_z(R, Nn - 8), _z(R * Nn, dtype=torch.float16), _z(R, 2 * Nn)[:, :Nn], _z(1).expand(R, Nn)])
def test_one_rank_product_refuses_out(out, monkeypatch):
    from types import SimpleNamespace

    from kernel_b200.ops import gemm as G

    monkeypatch.setattr(G, "_launch_local", lambda args, device: None)
    with pytest.raises(ValueError):
        G._run_local(SimpleNamespace(_hot=None, status=None), _z(R, K), _z(Nn, K), None, 1.0, out)


@pytest.mark.parametrize("which", ["x", "up", "down"])
def test_fused_mlp_takes_operands_of_any_strides(which):
    """The block of one GPU accepts what the two linear layers accept: a transposed view in
    place of the input or of either weight, forward and backward."""
    from kernel_b200.ops.autograd import LocalMLPFn
    from kernel_b200.ops.gemm import AGGemm

    g = torch.Generator().manual_seed(1)
    make = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)
    x, w1, b1, w2, b2, dy = make(R, K), make(Nn, K), make(Nn), make(K, Nn), make(K), make(R, K)
    grads = []
    for strided in (False, True):
        args = {"x": x, "up": w1, "down": w2}
        if strided:
            args[which] = args[which].t().contiguous().t()
            assert not args[which].is_contiguous()
        leaves = [args["x"], args["up"], b1, args["down"], b2]
        leaves = [t.detach().requires_grad_(True) for t in leaves]
        y = LocalMLPFn.apply(*leaves, "silu", AGGemm(R, K))
        grads.append([y.detach(), *torch.autograd.grad(y, leaves, dy)])
    assert all(torch.equal(p, q) for p, q in zip(*grads))


@pytest.mark.parametrize("kind", ["ColumnParallelLinear", "RowParallelLinear"])
def test_one_gpu_input_gradient_reports_to_the_layers_status(kind, monkeypatch):
    from kernel_b200.ops import autograd as A

    layer = getattr(A, kind)(R, K, Nn)
    layer.bwd.status = torch.zeros(8, dtype=torch.int32)
    seen = []
    monkeypatch.setattr(A, "_one_gpu", lambda layer, t: True)
    real = A.product
    monkeypatch.setattr(A, "product", lambda *a, **kw: seen.append(kw) or real(*a, **kw))
    x = _z(R, K).requires_grad_(True)
    layer(x).sum().backward()
    assert [kw["status"] for kw in seen if not kw.get("a_t")] == [layer.bwd.status]


def test_round_trip_takes_token_rows_with_trailing_unit_dimensions():
    from kernel_b200.ops.dispatch_combine import MoEAllToAll

    ctx = MoEAllToAll(4, 2, 64, 4, dtype=torch.bfloat16, device=torch.device("cpu"))
    x = torch.randn(3, 64, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16)
    idx, w = torch.tensor([[0, 1], [2, 3], [1, 3]], dtype=torch.int32), torch.ones(3, 2)
    want = ctx.dispatch_scale_combine(x, idx, w, 2)
    assert torch.equal(ctx.dispatch_scale_combine(x[..., None], idx, w, 2), want[..., None])
    ctx.heap.close()


def test_row_capacity_holds_every_routing_and_is_reached():
    """The padded rows of any routing fit; the routing that spreads one row to as many experts as
    it can and the rest so that each fills one more row than a multiple needs all of it."""
    import itertools

    for T, k, experts, pad in [(0, 2, 4, 64), (1, 2, 4, 64), (2, 1, 3, 4), (3, 2, 3, 2), (2, 2, 5, 3), (4, 1, 2, 3)]:
        most = 0
        for pick in itertools.product(range(experts), repeat=T * k):
            n = torch.bincount(torch.tensor(pick, dtype=torch.long), minlength=experts)
            most = max(most, int(((n + pad - 1) // pad * pad).sum()))
        capacity = L.ExpertRows.capacity(T, k, experts, pad)
        assert most <= capacity <= T * k + experts * (pad - 1)
        if T * k <= experts:
            assert most == capacity
