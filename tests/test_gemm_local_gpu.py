"""Products of one GPU (``ops/local.py``) at the edges of their tiles, against plain fp32 torch.

Operands are small integers: every product and sum is exact in fp32 in any order, so a
result differs from the reference only if a value is wrong, and the comparison is
exact.  Activations are compared within two bf16 roundings (2 ** -8 each)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda"


def _ints(*shape, seed=0):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randint(-2, 3, shape, device=DEV, generator=g).to(torch.bfloat16)


def _clean(status):
    torch.cuda.synchronize()
    assert status.cpu().tolist()[0] == 0, status.cpu().tolist()


def _status():
    return torch.zeros(8, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (7, 72, 72), (127, 256, 64), (128, 264, 136), (129, 512, 200), (257, 1000, 584),
                                   (513, 320, 1032), (64, 2048, 4104), (300, 136, 8200), (1025, 2056, 264)])
@pytest.mark.parametrize("layout", ["tn", "nn", "nt"])
def test_dense_product(M, N, K, layout):
    from kernel_b200.ops.local import product

    a_t, b_t = layout == "nt", layout != "tn"
    if a_t:
        M, K = (M + 7) // 8 * 8, K + 3  # contiguous along M: whole 16-byte units there, any K
    a, b, bias = _ints(M, K, seed=1), _ints(N, K, seed=2), _ints(N, seed=3)
    st = _status()
    out = product(a.t().contiguous() if a_t else a, b.t().contiguous() if b_t else b, bias, a_t=a_t, b_t=b_t, status=st)
    _clean(st)
    assert torch.equal(out, (a.float() @ b.float().t() + bias.float()).to(torch.bfloat16))


@pytest.mark.parametrize("pair,bn,split", [(0, 32, 1), (0, 96, 8), (0, 256, 5), (1, 64, 4), (1, 160, 3), (1, 256, 2), (2, 256, 1)])
def test_dense_configurations(pair, bn, split):
    """Every tile shape the launcher can pick gives the same numbers, also where the last tile is mostly padding."""
    from kernel_b200 import _native as N
    from kernel_b200.ops import local as L

    M, Nn, K = 264, 296, 2120  # k blocks for eight members of a split
    a, b = _ints(M, K, seed=4), _ints(Nn, K, seed=5)
    out = torch.full((M, Nn), 7.0, dtype=torch.bfloat16, device=DEV)
    st = _status()
    args = L._args(N.LOCAL_DENSE, M, Nn, K, st)
    args.bias_scale, args.A, args.B, args.out = 1.0, a.data_ptr(), b.data_ptr(), out.data_ptr()
    args.pair, args.bn, args.split = pair, bn, split
    L._launch(args, a.device)
    _clean(st)
    assert torch.equal(out, (a.float() @ b.float().t()).to(torch.bfloat16))


@pytest.mark.parametrize("act", ["gelu", "relu", "silu"])
@pytest.mark.parametrize("M,N,K", [(5, 72, 64), (200, 264, 328), (600, 520, 128)])
def test_activation_and_slope_in_the_epilogue(act, M, N, K):
    from kernel_b200.ops.local import _ACTS, _slope, product

    a, b = _ints(M, K, seed=6), (_ints(N, K, seed=7).float() / K ** 0.5).to(torch.bfloat16)
    st = _status()
    pre = torch.empty((M, N), dtype=torch.bfloat16, device=DEV)
    out = product(a, b, act=act, pre_out=pre, status=st)
    g = product(a, b.t().contiguous(), b_t=True, act=act, pre_in=pre, status=st)
    _clean(st)
    full = a.float() @ b.float().t()
    assert (pre.float() - full).abs().max() <= 2 ** -8 * full.abs().max()
    want = _ACTS[act](pre.float())
    assert ((out.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()
    want = full * _slope(act, pre)
    assert ((g.float() - want).abs() <= 2 ** -7 * want.abs() + 1e-4 * full.abs()).all()


@pytest.mark.parametrize("act", ["gelu", "silu"])
def test_activation_and_slope_of_every_bf16_value(act):
    """Against 64-bit arithmetic: one bf16 rounding (2 ** -9 relative, below the normal range half of the
    spacing 2 ** -133) plus 110 ulp of the fast exponential (2 ** -16); the bound is twice that."""
    from kernel_b200.ops.local import product

    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    x = x[x.float().abs() < 1e12]   # the slope of gelu holds x ** 3
    first = torch.zeros((x.numel(), 8), dtype=torch.bfloat16)
    first[:, 0] = 1.0
    ones = torch.zeros((8, 8), dtype=torch.bfloat16, device=DEV)
    ones[:, 0] = 1.0
    val = product((first * x[:, None]).to(DEV), ones, act=act)[:, 0].double().cpu()
    slope = product(first.to(DEV), ones.t().contiguous(), b_t=True, act=act, pre_in=x[:, None].repeat(1, 8).to(DEV))[:, 0].double().cpu()
    leaf = x.double().requires_grad_(True)
    arg = leaf if act == "silu" else 2 * (2 / torch.pi) ** 0.5 * (leaf + 0.044715 * leaf ** 3)
    want = leaf * torch.sigmoid(arg)
    want_slope, = torch.autograd.grad(want.sum(), leaf)
    for got, ref in ((val, want.detach()), (slope, want_slope)):
        bad = (got - ref).abs() > 2 ** -8 * ref.abs() + 2 ** -133
        assert not bad.any(), (x[bad], got[bad], ref[bad])


def test_relu_slope_selects():
    """Where ReLU is off an infinite gradient is zero; a NaN input passes the gradient on (as torch does)."""
    from kernel_b200.ops.local import product

    a = torch.zeros((8, 8), dtype=torch.bfloat16, device=DEV)
    a[:, 0] = float("inf")
    b = torch.zeros((8, 8), dtype=torch.bfloat16, device=DEV)
    b[0] = 1.0
    pre = torch.tensor([-1.0, 0.0, 1.0, float("nan")] * 2, device=DEV).to(torch.bfloat16).repeat(8, 1).contiguous()
    out = product(a, b, b_t=True, act="relu", pre_in=pre).float()
    assert out.cpu().tolist()[0] == [0.0, 0.0, float("inf"), float("inf")] * 2


COUNTS = [[0, 1, 33, 0, 128, 300, 64], [0, 0, 0], [5], [257, 0, 255, 256], [1] * 40]


def _table(counts, pad):
    n = torch.tensor(counts)
    padded = (n + pad - 1) // pad * pad
    start = padded.cumsum(0) - padded
    return start.int().to(DEV), n.int().to(DEV), max(1, int(padded.sum()))


def _force(monkeypatch, pair, bn=0, split=0, tok=0):
    """Tile shape of the products made through ``ops.local``."""
    from kernel_b200.ops import local as L

    made = L._args

    def forced(*a):
        args = made(*a)
        args.pair, args.bn, args.split, args.tok = pair, bn, split, tok
        return args

    monkeypatch.setattr(L, "_args", forced)
    return L


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("b_t", [False, True])
@pytest.mark.parametrize("N,K", [(264, 72), (64, 520)])
@pytest.mark.parametrize("pair", [-1, 0, 1])
def test_rows_product(counts, b_t, N, K, pair, monkeypatch):
    L = _force(monkeypatch, pair)
    start, count, R = _table(counts, 1)
    a, b = _ints(R, K, seed=8), _ints(len(counts), N, K, seed=9)
    st = _status()
    out = torch.full((R, N), 7.0, dtype=torch.bfloat16, device=DEV)
    L.rows_product(a, b.transpose(1, 2).contiguous() if b_t else b, start, count, b_t=b_t, out=out, status=st)
    _clean(st)
    want = torch.full((R, N), 7.0, dtype=torch.bfloat16, device=DEV)
    for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
        want[s:s + n] = (a[s:s + n].float() @ b[e].float().t()).to(torch.bfloat16)
    assert torch.equal(out, want)


def _check_epilogues(act, full, pre, out, grad):
    """``full`` is exact in fp32 (small integers times a power of two), so ``pre`` is its rounding;
    value and slope: one bf16 rounding (2 ** -9) and some ulp of the fast exponential, of the factors where
    the slope cancels.  The bounds are twice that."""
    leaf = pre.double().requires_grad_(True)
    arg = 2 * (2 / torch.pi) ** 0.5 * (leaf + 0.044715 * leaf ** 3)
    want = torch.relu(leaf) if act == "relu" else leaf * torch.sigmoid(leaf if act == "silu" else arg)
    slope, = torch.autograd.grad(want.sum(), leaf)
    assert torch.equal(pre, full.to(torch.bfloat16))
    assert ((out.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -133).all()
    want = full.double() * slope
    assert ((grad.double() - want).abs() <= 2 ** -8 * want.abs() + 2 ** -16 * full.double().abs()).all()


@pytest.mark.parametrize("act", ["gelu", "relu", "silu"])
@pytest.mark.parametrize("pair,bn,split,M,N,K", [
    *((*shape, 520, 296, 2120) for shape in [(0, 64, 1), (0, 192, 1), (0, 128, 5), (0, 256, 8), (1, 128, 1), (1, 256, 1), (1, 128, 3),
                                             (1, 256, 4), (2, 256, 1)]),
    *((*shape, 40, 72, 1096) for shape in [(0, 64, 1), (0, 192, 1), (0, 128, 5), (0, 256, 8)])])
def test_epilogues_of_every_tile_shape(act, pair, bn, split, M, N, K, monkeypatch):
    """One CTA, pairs, 512-row tiles and the exchange of a split, with full and ragged tiles and (one CTA)
    a matrix smaller than the tile."""
    L = _force(monkeypatch, pair, bn, split)
    a, b = _ints(M, K, seed=30), _ints(N, K, seed=31) * 2 ** -5
    st = _status()
    pre = torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    out = L.product(a, b, act=act, pre_out=pre, status=st)
    grad = L.product(a, b.t().contiguous(), b_t=True, act=act, pre_in=pre, status=st)
    _clean(st)
    _check_epilogues(act, a.float() @ b.float().t(), pre, out, grad)


@pytest.mark.parametrize("act", ["gelu", "relu", "silu"])
@pytest.mark.parametrize("pair,bn,split", [(3, 64, 1), (3, 128, 1), (3, 64, 3), (3, 128, 8), (4, 128, 1), (4, 256, 1), (4, 128, 4), (4, 256, 2)])
@pytest.mark.parametrize("M,N,K", [(1, 264, 2120), (64, 296, 1096), (165, 72, 520), (520, 264, 1096)])
def test_epilogues_with_exchanged_operands(act, pair, bn, split, M, N, K, monkeypatch):
    """Token rows on the MMA's N side: one token, whole and ragged blocks, several of them, columns that end inside a tile."""
    L = _force(monkeypatch, pair, bn, split)
    a, b = _ints(M, K, seed=34), _ints(N, K, seed=35) * 2 ** -5
    bt, bias = b.t().contiguous(), _ints(N, seed=36)
    st = _status()
    pre, plain = (torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    out, grad = torch.empty_like(pre), torch.empty_like(pre)
    torch.cuda.synchronize()
    L.product(a, b, act=act, pre_out=pre, out=out, status=st)
    L.product(a, bt, b_t=True, act=act, pre_in=pre, out=grad, status=st, early=True)   # behind a product that wrote neither weights
    L.product(a, b, bias, out=plain, status=st, early=True)
    _clean(st)
    full = a.float() @ b.float().t()
    _check_epilogues(act, full, pre, out, grad)
    assert torch.equal(plain, (full + bias.float()).to(torch.bfloat16))


@pytest.mark.parametrize("pair,bn,split", [(3, 32, 1), (3, 56, 2), (3, 80, 7), (3, 112, 5), (4, 80, 1), (4, 176, 2), (4, 208, 1), (4, 240, 3)])
@pytest.mark.parametrize("M,N,K,tok", [(1, 264, 2120, 0), (64, 480, 1096, 32), (165, 72, 520, 0), (520, 264, 1096, 96), (300, 1664, 520, 256)])
def test_exchanged_tiles_that_end_inside_a_warp(pair, bn, split, M, N, K, tok, monkeypatch):
    """Weights along K come in tiles of any multiple of 8 columns per CTA: whole tiles and cut ones, splits that do not divide the
    k blocks, token blocks of a chosen height."""
    L = _force(monkeypatch, pair, bn, split, tok)
    a, b, bias = _ints(M, K, seed=46), _ints(N, K, seed=47), _ints(N, seed=48)
    st = _status()
    pre, out, plain = (torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3))
    torch.cuda.synchronize()
    L.product(a, b, act="relu", pre_out=pre, out=out, status=st)
    L.product(a, b, bias, out=plain, status=st, early=True)
    _clean(st)
    full = a.float() @ b.float().t()
    assert torch.equal(pre, full.to(torch.bfloat16)) and torch.equal(out, torch.relu(full).to(torch.bfloat16))
    assert torch.equal(plain, (full + bias.float()).to(torch.bfloat16))


@pytest.mark.parametrize("pair,bn,tok", [(3, 64, 0), (3, 128, 0), (4, 128, 0), (4, 256, 0), (3, 128, 16), (3, 64, 48), (3, 128, 256), (4, 256, 32), (4, 128, 96),
                                         (4, 256, 256)])
@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("N", [264, 320])  # 320: a multiple of 64, weights along N come in whole boxes, the last tile ends inside
def test_grouped_rows_with_exchanged_operands(N, pair, bn, tok, counts, monkeypatch):
    """``tok``: most rows of a block; groups of several uneven blocks."""
    L = _force(monkeypatch, pair, bn, tok=tok)
    K = 520
    start, count, R = _table(counts, 1)
    a, b = _ints(R, K, seed=37), _ints(len(counts), N, K, seed=38) * 2 ** -4
    st = _status()
    pre, out, grad, plain = (torch.full((R, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(4))
    L.rows_product(a, b, start, count, act="silu", pre_out=pre, out=out, status=st)
    L.rows_product(a, b.transpose(1, 2).contiguous(), start, count, b_t=True, act="silu", pre_in=pre, out=grad, status=st)
    L.rows_product(a, b, start, count, out=plain, status=st, early=True, expect=len(counts))
    _clean(st)
    inside = torch.zeros(R, dtype=torch.bool, device=DEV)
    for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
        inside[s:s + n] = True
        sl = slice(s, s + n)
        full = a[sl].float() @ b[e].float().t()
        _check_epilogues("silu", full, pre[sl], out[sl], grad[sl])
        assert torch.equal(plain[sl], full.to(torch.bfloat16))
    assert all((t[~inside] == 7.0).all() for t in (pre, out, grad, plain))


def test_weights_fetched_early_are_those_of_the_call():
    """The second product's weights change right before the block runs, call after call."""
    from kernel_b200.models import SequenceParallelMLP

    T, H, F = 24, 1032, 2056
    w1, w2 = _ints(F, H, seed=39) * 2 ** -6, _ints(H, F, seed=40) * 2 ** -6
    mlp = SequenceParallelMLP(T, H, w1, w2, activation="relu")
    x = _ints(T, H, seed=41)
    want = mlp(x)
    for i in range(40):
        mlp.w2.neg_()
        want = -want
        assert torch.equal(mlp(x), want), i
    mlp.up.status.cpu()
    _clean(mlp.up.status)
    _clean(mlp.down.status)


@pytest.mark.parametrize("pair", [3, 4])
def test_moe_weights_fetched_early_are_those_of_the_call(pair, monkeypatch):
    """Rewritten directly before the inference block, and between a forward pass and its backward pass (the block reads the
    parameters themselves): the output is odd in the second matrix, the token gradient in each of them."""
    from kernel_b200.models import MoELayer, TrainableMoELayer

    _force(monkeypatch, pair)
    torch.manual_seed(6)
    E, k, H, F, T = 16, 2, 1024, 1032, 96
    layer = TrainableMoELayer(E, k, H, F, T, device=torch.device(DEV))
    fixed = MoELayer(E, k, H, T, layer.w_up.data.clone(), layer.w_down.data.clone())
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_(True)
    idx = torch.rand(T, E, device=DEV).argsort(1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn(T, k, device=DEV), -1)
    dy = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    want = fixed(x.detach(), idx, w)
    grad, = torch.autograd.grad(layer(x, idx, w), x, dy)
    for i in range(10):
        fixed.w_down.neg_()
        want = -want
        assert torch.equal(fixed(x.detach(), idx, w), want), i
        y = layer(x, idx, w)
        for weights in ((layer.w_down,), (layer.w_up,), (layer.w_up, layer.w_down)):
            for p in weights:
                p.data.neg_()
            got, = torch.autograd.grad(y, x, dy, retain_graph=True)
            assert torch.equal(got, grad if len(weights) == 2 else -grad), i
            for p in weights:
                p.data.neg_()
    layer.a2a.heap.check_status()
    fixed.a2a.heap.close()
    layer.close()


@pytest.mark.parametrize("pair", [3, 4])
def test_mlp_gradients_fetch_the_weights_of_the_call(pair, monkeypatch):
    """As above: the token gradient is odd in each weight matrix."""
    from kernel_b200.models import TrainableSequenceParallelMLP
    from kernel_b200.ops import local as L

    launch = L._launch

    def exchanged(args, device):
        if not args.a_mn:
            args.pair = pair
        launch(args, device)

    monkeypatch.setattr(L, "_launch", exchanged)
    torch.manual_seed(7)
    mlp = TrainableSequenceParallelMLP(48, 1032, 4104, activation="relu", device=torch.device(DEV))
    x = torch.randn(48, 1032, device=DEV).to(torch.bfloat16).requires_grad_(True)
    dy = torch.randn(48, 1032, device=DEV).to(torch.bfloat16)
    leaves = (x, mlp.down.weight)          # with the second one the hidden gradient follows a product of this module
    grad, dw2 = torch.autograd.grad(mlp(x), leaves, dy)
    for i in range(10):
        y = mlp(x)
        for weights in ((mlp.down.weight,), (mlp.up.weight,)):
            for p in weights:
                p.data.neg_()
            got = torch.autograd.grad(y, leaves, dy, retain_graph=True)
            assert torch.equal(got[0], -grad) and torch.equal(got[1], dw2), i
            for p in weights:
                p.data.neg_()
    mlp.close()


@pytest.mark.parametrize("act", ["gelu", "relu", "silu"])
@pytest.mark.parametrize("pair,bn", [(0, 64), (0, 256), (1, 128), (1, 256)])
@pytest.mark.parametrize("counts", COUNTS)
def test_epilogues_of_grouped_rows(act, pair, bn, counts, monkeypatch):
    L = _force(monkeypatch, pair, bn)
    N, K = 264, 520
    start, count, R = _table(counts, 1)
    a, b = _ints(R, K, seed=32), _ints(len(counts), N, K, seed=33) * 2 ** -4
    st = _status()
    pre, out, grad = (torch.full((R, N), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(3))
    L.rows_product(a, b, start, count, act=act, pre_out=pre, out=out, status=st)
    L.rows_product(a, b.transpose(1, 2).contiguous(), start, count, b_t=True, act=act, pre_in=pre, out=grad, status=st)
    _clean(st)
    inside = torch.zeros(R, dtype=torch.bool, device=DEV)
    for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
        inside[s:s + n] = True
        sl = slice(s, s + n)
        _check_epilogues(act, a[sl].float() @ b[e].float().t(), pre[sl], out[sl], grad[sl])
    assert all((t[~inside] == 7.0).all() for t in (pre, out, grad))


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("M,N", [(136, 72), (64, 264), (520, 128)])
@pytest.mark.parametrize("pair", [-1, 0, 1])
def test_contract_product(counts, M, N, pair, monkeypatch):
    L = _force(monkeypatch, pair)
    start, count, R = _table(counts, L.ROW_ALIGN)
    a, b = torch.zeros((R, M), dtype=torch.bfloat16, device=DEV), torch.zeros((R, N), dtype=torch.bfloat16, device=DEV)
    for s, n in zip(start.tolist(), count.tolist()):
        a[s:s + n], b[s:s + n] = _ints(n, M, seed=10 + s), _ints(n, N, seed=11 + s)
    st = _status()
    out = L.contract_product(a, b, start, count, status=st)
    _clean(st)
    for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
        assert torch.equal(out[e], (a[s:s + n].float().t() @ b[s:s + n].float()).to(torch.bfloat16)), e


@pytest.mark.parametrize("counts", COUNTS)
@pytest.mark.parametrize("M,N", [(192, 320), (64, 576), (320, 72), (136, 192)])
@pytest.mark.parametrize("pair,bn", [(0, 64), (0, 256), (1, 128), (1, 256)])
def test_contractions_whose_columns_come_in_one_box(counts, M, N, pair, bn, monkeypatch):
    """Extents that are multiples of 64 (one box per operand and stage) and end inside a tile, both, one or the other operand."""
    L = _force(monkeypatch, pair, bn)
    start, count, R = _table(counts, L.ROW_ALIGN)
    a, b = torch.zeros((R, M), dtype=torch.bfloat16, device=DEV), torch.zeros((R, N), dtype=torch.bfloat16, device=DEV)
    for s, n in zip(start.tolist(), count.tolist()):
        a[s:s + n], b[s:s + n] = _ints(n, M, seed=50 + s), _ints(n, N, seed=51 + s)
    st = _status()
    out = L.contract_product(a, b, start, count, status=st)
    dense = L.product(a, b, a_t=True, b_t=True, status=st)
    _clean(st)
    for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
        assert torch.equal(out[e], (a[s:s + n].float().t() @ b[s:s + n].float()).to(torch.bfloat16)), e
    assert torch.equal(dense, (a.float().t() @ b.float()).to(torch.bfloat16))


@pytest.mark.parametrize("M,N", [(1000, 1416), (1104, 1344), (600, 2416)])
def test_contractions_over_one_k_block_with_two_stages(M, N):
    """Outputs of more than 180 MB, whose operand ring has two stages: empty groups, whole blocks and a group of several."""
    from kernel_b200.ops import local as L

    counts = ([0, 1, 17, 64, 5, 33, 0, 40] * 8)[:63] + [200]
    start, count, R = _table(counts, L.ROW_ALIGN)
    a, b = torch.zeros((R, M), dtype=torch.bfloat16, device=DEV), torch.zeros((R, N), dtype=torch.bfloat16, device=DEV)
    for s, n in zip(start.tolist(), count.tolist()):
        a[s:s + n], b[s:s + n] = _ints(n, M, seed=80 + s), _ints(n, N, seed=81 + s)
    st = _status()
    out = L.contract_product(a, b, start, count, status=st, expect=sum(counts))
    _clean(st)
    for e, (s, n) in enumerate(zip(start.tolist(), count.tolist())):
        assert torch.equal(out[e], (a[s:s + n].float().t() @ b[s:s + n].float()).to(torch.bfloat16)), e


@pytest.mark.parametrize("R,Cn", [(1, 8), (63, 264), (65, 2048), (1000, 520), (8192, 72)])
def test_col_sum(R, Cn):
    from kernel_b200.ops.local import col_sum

    x = _ints(R, Cn, seed=12)
    assert torch.equal(col_sum(x), x.float().sum(0).to(torch.bfloat16))


def test_col_sum_of_a_misaligned_matrix():
    from kernel_b200.ops.local import col_sum

    x = _ints(17 * 64 + 1, seed=13)[1:].view(17, 64)
    assert torch.equal(col_sum(x), x.float().sum(0).to(torch.bfloat16))


@pytest.mark.parametrize("T,k,E,H,pad", [(0, 2, 8, 64, 1), (1, 1, 1, 8, 64), (3, 8, 256, 1032, 1), (130, 6, 64, 256, 64),
                                         (777, 4, 1024, 72, 64), (40, 64, 100, 520, 1)])
def test_expert_rows(T, k, E, H, pad):
    """Row movement of a single-rank MoE layer: permutation, combine and its backward."""
    from kernel_b200.ops.local import ExpertRows

    g = torch.Generator(device=DEV).manual_seed(T)
    idx = torch.rand((T, E), device=DEV, generator=g).argsort(1)[:, :k].to(torch.int32).contiguous()
    x, w = _ints(T, H, seed=14), torch.randint(-3, 4, (T, k), device=DEV, generator=g).float()
    st = _status()
    er = ExpertRows(x, idx, E, pad=pad, status=st)
    _clean(st)
    count = torch.bincount(idx.reshape(-1).long(), minlength=E)
    padded = (count + pad - 1) // pad * pad
    assert torch.equal(er.count.long(), count) and torch.equal(er.padded.long(), padded)
    assert torch.equal(er.start.long(), padded.cumsum(0) - padded)
    slots = er.slots.long()
    assert torch.equal(er.rows[slots], x.unsqueeze(1).expand(T, k, H))
    real = torch.zeros(er.rows.shape[0], dtype=torch.bool, device=DEV)
    real[slots.reshape(-1)] = True
    used = int(padded.sum())
    assert int(real.sum()) == T * k and not real[used:].any() and not er.rows[:used][~real[:used]].any()
    y = _ints(er.rows.shape[0], H, seed=15)
    assert torch.equal(er.combine(y, w), (y[slots].float() * w.unsqueeze(-1)).sum(1).to(torch.bfloat16))
    assert torch.equal(er.combine(y, None), y[slots].float().sum(1).to(torch.bfloat16))
    dy = _ints(T, H, seed=16)
    dyr, dw = er.grad_rows(dy, y, w)
    assert torch.equal(dyr[slots], (dy.unsqueeze(1).float() * w.unsqueeze(-1)).to(torch.bfloat16))
    assert not dyr[:used][~real[:used]].any()
    assert torch.equal(dw, (dy.unsqueeze(1).float() * y[slots].float()).sum(-1))


@pytest.mark.parametrize("T,k,E", [(0, 2, 8), (1, 1, 256), (5, 2, 300), (150, 2, 4)])
def test_moe_training_step_with_more_experts_than_rows(T, k, E):
    """Gradients of every input where most experts have no row, and with no token at all."""
    from kernel_b200.models import TrainableMoELayer

    torch.manual_seed(T)
    H, F = 64, 72
    layer = TrainableMoELayer(E, k, H, F, max(T, 1), device=torch.device(DEV))
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_(True)
    w = torch.rand(T, k, device=DEV).requires_grad_(True)
    idx = torch.rand(T, E, device=DEV).argsort(1)[:, :k].to(torch.int32).contiguous()
    dy = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    y = layer(x, idx, w)
    got = [y, *torch.autograd.grad(y, (x, w, layer.w_up, layer.w_down), dy)]
    leaves = [t.detach().double().requires_grad_(True) for t in (x, w, layer.w_up, layer.w_down)]
    h = torch.nn.functional.silu(torch.einsum("th,tkfh->tkf", leaves[0], leaves[2][idx.long()]))
    rows = torch.einsum("tkf,tkhf->tkh", h, leaves[3][idx.long()])
    ref = (rows * leaves[1].unsqueeze(-1)).sum(1)
    want = [ref, *torch.autograd.grad(ref, leaves, dy.double())]
    for i, (p, q) in enumerate(zip(got, want)):
        assert p.shape == q.shape
        # at most four bf16 roundings (2 ** -9 each) between the inputs and a result; the error of a routing weight's
        # gradient <dy, row> is relative to the lengths of both vectors (their product may cancel)
        scale = (dy.double().norm(dim=1, keepdim=True) * rows.norm(dim=2)).norm() if i == 2 else q.norm()
        assert (p.double() - q).norm() <= 4 * 2 ** -9 * scale
    layer.a2a.heap.check_status()
    layer.close()


def test_expert_rows_out_of_range_id_is_reported_and_skipped():
    from kernel_b200.ops.local import ExpertRows

    x, idx = _ints(4, 64, seed=17), torch.tensor([[0, 5], [1, -1], [2, 3], [3, 0]], dtype=torch.int32, device=DEV)
    st = _status()
    er = ExpertRows(x, idx, 4, status=st)
    torch.cuda.synchronize()
    assert st.cpu().tolist()[0] != 0
    assert er.slots.cpu().tolist() == [[0, -1], [2, -1], [3, 4], [5, 1]]
    assert torch.equal(er.combine(er.rows, None), torch.stack([x[0], x[1], 2 * x[2], 2 * x[3]]))


@pytest.mark.parametrize("E,k,H,T", [(8, 2, 8, 1), (64, 6, 1032, 33), (256, 8, 7168, 300), (128, 4, 2880, 2048), (64, 33, 520, 70)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("mode", [0, 1, 2])
def test_single_rank_round_trip_equals_the_general_kernels(E, k, H, T, dtype, mode):
    """Bit for bit; a traced call runs the general kernels."""
    from kernel_b200.ops.dispatch_combine import MoEAllToAll

    g = torch.Generator(device=DEV).manual_seed(H)
    ctx = MoEAllToAll(E, k, H, T, dtype=dtype, device=torch.device(DEV))
    x = torch.randn((T, H), device=DEV, generator=g).to(dtype)
    idx = torch.rand((T, E), device=DEV, generator=g).argsort(1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn((T, k), device=DEV, generator=g), -1)
    out = ctx.dispatch_scale_combine(x, idx, w, mode)
    ctx.enable_trace()
    general = ctx.dispatch_scale_combine(x, idx, w, mode)
    torch.cuda.synchronize()
    ctx.heap.check_status()
    assert torch.equal(out, general)
    ctx.heap.close()


@pytest.mark.parametrize("M,N,K,chunks", [(2, 8, 8, 4), (64, 72, 136, 4), (300, 264, 1032, 1), (515, 128, 2048, 7), (1024, 2048, 136, 4), (4096, 72, 2048, 4)])
def test_rows_from_the_host_in_pieces(M, N, K, chunks):
    """Sizes for which the pieces are one, equal, falling and rising, call after call with other rows, and on another stream."""
    from kernel_b200.ops.gemm import AGGemm, GemmRS

    w, bias = _ints(N, K, seed=60), _ints(N, seed=61)
    rs, ag = GemmRS(M, N, device=torch.device(DEV)), AGGemm(M, K, device=torch.device(DEV))
    side = torch.cuda.Stream()
    for i in range(4):
        a = _ints(M, K, seed=62 + i)
        want = a.float() @ w.float().t() + bias.float()
        host, out = a.cpu().pin_memory(), torch.zeros((M, N), dtype=torch.bfloat16).pin_memory()
        with torch.cuda.stream(side if i % 2 else torch.cuda.current_stream()):
            rs.run_from_host(host, w, bias, out_host=out, chunks=chunks)
            got = ag.run_from_host(host, w, bias, chunks=chunks)
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), want.to(torch.bfloat16)) and torch.equal(got.to(DEV), want.to(torch.bfloat16))
    _clean(rs.status)
    rs.close()
    ag.close()


@pytest.mark.parametrize("M,N,K,chunks,rows", [
    (2, 8, 8, 4, [2]), (64, 72, 136, 4, [64]), (300, 264, 1032, 1, [300]), (4096, 72, 2048, 4, [4096]),
    (515, 4096, 4096, 4, [192, 192, 131]), (2048, 2048, 2048, 4, [512] * 4), (1111, 1024, 8192, 4, [896, 215]), (1111, 8192, 1024, 4, [256, 855]),
    (2000, 4096, 4096, 7, [320, 256, 320, 256, 320, 256, 272])])
def test_rows_from_the_host_in_several_pieces_queued_on_two_streams(M, N, K, chunks, rows):
    """One piece, equal, falling and rising ones: calls of one context queued behind each other on two streams, other rows in each."""
    from kernel_b200.ops.gemm import AGGemm, GemmRS, _pieces

    assert _pieces(M, N, K, chunks) == rows
    w, bias = _ints(N, K, seed=60), _ints(N, seed=61)
    rs, ag = GemmRS(M, N, device=torch.device(DEV)), AGGemm(M, K, device=torch.device(DEV))
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    host = [_ints(M, K, seed=62 + i).cpu().pin_memory() for i in range(6)]
    out = [[torch.zeros((M, N), dtype=torch.bfloat16).pin_memory() for _ in host] for _ in (rs, ag)]
    torch.cuda.synchronize()
    for i in range(len(host)):
        with torch.cuda.stream(streams[i % 2]):
            rs.run_from_host(host[i], w, bias, out_host=out[0][i], chunks=chunks)
            ag.run_from_host(host[i], w, bias, out_host=out[1][i], chunks=chunks)
    torch.cuda.synchronize()
    for i, a in enumerate(host):
        want = (a.to(DEV).float() @ w.float().t() + bias.float()).to(torch.bfloat16)
        assert torch.equal(out[0][i].to(DEV), want) and torch.equal(out[1][i].to(DEV), want), i
    with torch.cuda.stream(streams[0]):   # all that a caller waits for is its own stream
        got = rs.run_from_host(host[0], w, bias, out_host=torch.zeros((M, N), dtype=torch.bfloat16).pin_memory(), chunks=chunks)
    streams[0].synchronize()
    assert torch.equal(got, out[0][0])
    _clean(rs.status)
    rs.close()
    ag.close()


@pytest.mark.parametrize("above", [0, 1])  # the last size that is held whole and the first that is not
def test_rows_from_the_host_that_are_too_many_to_hold(above, monkeypatch):
    from kernel_b200.ops import gemm

    M, N, K = 512, 264, 520
    monkeypatch.setattr(gemm, "_WHOLE_ROWS_BYTES", 2 * M * (N + K) - above)
    w, a = _ints(N, K, seed=68), _ints(M, K, seed=69)
    want = (a.float() @ w.float().t()).to(torch.bfloat16)
    for ctx in (gemm.GemmRS(M, N, device=torch.device(DEV)), gemm.AGGemm(M, K, device=torch.device(DEV))):
        out = ctx.run_from_host(a.cpu().pin_memory(), w)
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), want) and ("_one_gpu_streams" in ctx.__dict__) == (not above)
        ctx.close()


def test_rows_from_the_host_in_a_graph():
    from kernel_b200.ops.gemm import GemmRS

    M, N, K = 512, 264, 520
    w, a = _ints(N, K, seed=66), _ints(M, K, seed=67)
    ctx = GemmRS(M, N, device=torch.device(DEV))
    host, out = a.cpu().pin_memory(), torch.zeros((M, N), dtype=torch.bfloat16).pin_memory()
    want = (a.float() @ w.float().t()).to(torch.bfloat16)
    ctx.run_from_host(host, w, out_host=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.run_from_host(host, w, out_host=out)
    for sign in (-1, 1):
        host.neg_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), sign * want)
        ctx.run_from_host(host.neg_(), w, out_host=out)   # between two replays, outside of the graph
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), -sign * want)
        host.neg_()
    ctx.close()


@pytest.mark.parametrize("M,N,K,pieces", [(512, 264, 520, 1), (515, 4096, 4096, 3)])
def test_several_pieces_in_a_graph(M, N, K, pieces):
    from kernel_b200.ops.gemm import GemmRS, _pieces

    assert len(_pieces(M, N, K, 4)) == pieces
    w, a = _ints(N, K, seed=66), _ints(M, K, seed=67)
    ctx = GemmRS(M, N, device=torch.device(DEV))
    host, out = a.cpu().pin_memory(), torch.zeros((M, N), dtype=torch.bfloat16).pin_memory()
    want = (a.float() @ w.float().t()).to(torch.bfloat16)
    ctx.run_from_host(host, w, out_host=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        ctx.run_from_host(host, w, out_host=out)
    for sign in (-1, 1):
        host.neg_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), sign * want)
        ctx.run_from_host(host.neg_(), w, out_host=out)   # between two replays, outside of the graph
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), -sign * want)
        host.neg_()
    ctx.close()


def test_rows_from_the_host_after_a_capture_wait_for_the_call_before_it():
    """On a third stream, the first call still under way; the capture's own call comes out right as well."""
    from kernel_b200.ops.gemm import GemmRS

    M, N, K = 2048, 2048, 2048   # 160 us on the link each way
    w, ctx = _ints(N, K, seed=70), GemmRS(M, N, device=torch.device(DEV))
    hosts = [_ints(M, K, seed=71 + i).cpu().pin_memory() for i in range(3)]
    outs = [torch.zeros((M, N), dtype=torch.bfloat16).pin_memory() for _ in hosts]
    streams = [torch.cuda.Stream() for _ in hosts]
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    for i, (host, out, stream) in enumerate(zip(hosts, outs, streams)):
        with torch.cuda.stream(stream):
            if i == 1:
                graph.capture_begin(capture_error_mode="thread_local")
            ctx.run_from_host(host, w, out_host=out)
            if i == 1:
                graph.capture_end()
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    for host, out in zip(hosts, outs):
        assert torch.equal(out.to(DEV), (host.to(DEV).float() @ w.float().t()).to(torch.bfloat16))
    ctx.close()


def test_rows_from_the_host_of_several_widths_share_their_buffers():
    """Nothing is held beside the largest rows and the largest result; a graph keeps those that it was captured with."""
    from kernel_b200.ops.gemm import AGGemm

    M, K = 1536, 1024
    a = _ints(M, K, seed=74)
    host, ctx = a.cpu().pin_memory(), AGGemm(M, K, device=torch.device(DEV))
    ws = {N: _ints(N, K, seed=75) for N in (1024, 4096, 520, 4096, 8192)}
    outs = {N: torch.zeros((M, N), dtype=torch.bfloat16).pin_memory() for N in ws}
    want = {N: (a.float() @ w.float().t()).to(torch.bfloat16) for N, w in ws.items()}
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    before, most = torch.cuda.memory_allocated(), 0
    for N, chunks in ((1024, 4), (4096, 4), (520, 1), (4096, 7), (1024, 2)):
        most = max(most, N)
        ctx.run_from_host(host, ws[N], out_host=outs[N], chunks=chunks)
        torch.cuda.synchronize()
        assert torch.equal(outs[N].to(DEV), want[N])
        # torch's allocator splits a cached block only if more than 1 MB of it is left over
        assert torch.cuda.memory_allocated() - before <= 2 * M * (K + most) + (2 << 20)
    with torch.cuda.graph(graph):
        ctx.run_from_host(host, ws[4096], out_host=outs[4096])
    ctx.run_from_host(host, ws[8192], out_host=outs[8192])   # the others are too small for it
    torch.cuda.synchronize()
    taken = [torch.full((M * N,), -1.0, dtype=torch.bfloat16, device=DEV) for N in (K, 4096)]
    outs[4096].zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(outs[4096].to(DEV), want[4096]) and torch.equal(outs[8192].to(DEV), want[8192])
    assert all(bool((t == -1).all()) for t in taken)
    ctx.close()


@pytest.mark.parametrize("fault", ["room", "allocation"])
def test_rows_from_the_host_that_cannot_be_held_go_in_chunks(fault, monkeypatch):
    from kernel_b200.ops import gemm

    M, N, K = 512, 264, 520
    w, a = _ints(N, K, seed=76), _ints(M, K, seed=77)
    want, host = (a.float() @ w.float().t()).to(torch.bfloat16), a.cpu().pin_memory()
    for ctx in (gemm.GemmRS(M, N, device=torch.device(DEV)), gemm.AGGemm(M, K, device=torch.device(DEV))):
        with monkeypatch.context() as patch:
            if fault == "room":
                patch.setattr(gemm, "_SMALL_ROWS_BYTES", 0)
                patch.setattr(gemm, "_room", lambda device: 8 * M * (N + K) - 1)   # four times the buffers' bytes, but for one
            else:
                def full(self, count):
                    raise torch.OutOfMemoryError("planted")
                patch.setattr(gemm._OneGpuStream, "_allocate", full)
            out = ctx.run_from_host(host, w)
            torch.cuda.synchronize()
            assert torch.equal(out.to(DEV), want) and hasattr(ctx, "_stream_state") and ctx._stream_state
        ctx._stream_state.clear()
        if fault == "room":
            monkeypatch.setattr(gemm, "_room", lambda device: 8 * M * (N + K))
            monkeypatch.setattr(gemm, "_SMALL_ROWS_BYTES", 0)
        out = ctx.run_from_host(host, w)   # as soon as there is room
        torch.cuda.synchronize()
        assert torch.equal(out.to(DEV), want) and not ctx._stream_state
        ctx.close()


@pytest.mark.parametrize("E", [256, 512, 100, 1024])  # bf16: exact scales, scales of more digits, no power of two; fp16: exact up to 1024
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("H,T,k", [(1032, 9, 1), (7168, 150, 8), (2056, 700, 3)])
def test_round_trip_of_special_values_equals_the_general_kernels(E, dtype, H, T, k):
    """Subnormal, infinite and undefined values, signed zeros, tokens whose scales are all 1: each kind of scale has a kernel of its own."""
    from kernel_b200.ops.dispatch_combine import MoEAllToAll

    g = torch.Generator(device=DEV).manual_seed(E + H)
    ctx = MoEAllToAll(E, k, H, T, dtype=dtype, device=torch.device(DEV))
    x = torch.randn((T, H), device=DEV, generator=g)
    tiny, huge = torch.finfo(dtype).tiny, torch.finfo(dtype).max
    special = torch.tensor([0.0, -0.0, tiny, -tiny, tiny / 2, tiny / 100, huge, -huge, float("inf"), float("-inf"), float("nan")], device=DEV)
    x[:, ::7] = special[torch.randint(0, len(special), x[:, ::7].shape, device=DEV, generator=g)]
    x = x.to(dtype)
    idx = torch.rand((T, E), device=DEV, generator=g).argsort(1)[:, :k].to(torch.int32).contiguous()
    idx[::3, 0] = E - 1   # scale 1 (and, for k = 1, nothing else)
    w = torch.softmax(torch.randn((T, k), device=DEV, generator=g), -1)
    for mode in (0, 2):
        ctx.enable_trace(False)
        out = ctx.dispatch_scale_combine(x, idx, w, mode)
        ctx.enable_trace()
        general = ctx.dispatch_scale_combine(x, idx, w, mode)
        torch.cuda.synchronize()
        ctx.heap.check_status()
        assert torch.equal(out.isnan(), general.isnan()) and torch.equal(out.nan_to_num(), general.nan_to_num())
    ctx.heap.close()


@pytest.mark.parametrize("E", [256, 512, 100, 1024])  # bf16: exact scales, scales of more digits, no power of two; fp16: exact up to 1024
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("H,T,k", [(1032, 9, 1), (7168, 150, 8), (2056, 700, 3)])
def test_round_trip_of_special_values_equals_the_general_kernels_bit_by_bit(E, dtype, H, T, k):
    """Subnormal, infinite and undefined values, signed zeros, tokens whose scales are all 1: each kind of scale has a kernel of its own."""
    from kernel_b200.ops.dispatch_combine import MoEAllToAll

    g = torch.Generator(device=DEV).manual_seed(E + H)
    ctx = MoEAllToAll(E, k, H, T, dtype=dtype, device=torch.device(DEV))
    x = torch.randn((T, H), device=DEV, generator=g)
    tiny, huge = torch.finfo(dtype).tiny, torch.finfo(dtype).max
    special = torch.tensor([0.0, -0.0, tiny, -tiny, tiny / 2, tiny / 100, huge, -huge, float("inf"), float("-inf"), float("nan")], device=DEV)
    x[:, ::7] = special[torch.randint(0, len(special), x[:, ::7].shape, device=DEV, generator=g)]
    x = x.to(dtype)
    idx = torch.rand((T, E), device=DEV, generator=g).argsort(1)[:, :k].to(torch.int32).contiguous()
    idx[::3, 0] = E - 1   # scale 1 (and, for k = 1, nothing else)
    w = torch.softmax(torch.randn((T, k), device=DEV, generator=g), -1)
    for mode in (0, 2):
        ctx.enable_trace(False)
        out = ctx.dispatch_scale_combine(x, idx, w, mode)
        ctx.enable_trace()
        general = ctx.dispatch_scale_combine(x, idx, w, mode)
        torch.cuda.synchronize()
        ctx.heap.check_status()
        nan, bits = general.isnan(), torch.int32 if dtype == torch.float32 else torch.int16
        assert torch.equal(out.isnan(), nan) and torch.equal(out.view(bits)[~nan], general.view(bits)[~nan])
        assert (general == 0).any() and general.isinf().any() and nan.any() and not nan.all()
    ctx.heap.close()


def test_a_product_is_the_first_cuda_call_of_its_thread():
    """As in an autograd worker whose memory comes from the allocator's cache: no runtime call has bound a context."""
    import threading

    from kernel_b200.ops.local import product

    a, b, failed = _ints(136, 264, seed=18), _ints(72, 264, seed=19), []
    outs = [torch.zeros(136, 72, dtype=torch.bfloat16, device=DEV) for _ in range(3)]
    product(a, b, out=outs[0])
    torch.cuda.synchronize()

    def work(i, *args, **kw):
        try:
            product(*args, out=outs[i], **kw)
        except Exception as e:  # reported in the test's thread
            failed.append(e)

    for i, args, kw in ((1, (a, b), {}), (2, (a, b.t().contiguous()), dict(b_t=True))):
        torch.cuda.synchronize()
        t = threading.Thread(target=work, args=(i, *args), kwargs=kw)
        t.start()
        t.join()
    torch.cuda.synchronize()
    assert not failed, failed
    assert torch.equal(outs[1], outs[0]) and torch.equal(outs[2], outs[0])


def test_overlapped_launches_keep_their_order_eagerly_and_in_a_graph():
    """A chain in which every kernel reads what the one before wrote, also across a fork and a
    join of streams, with torch kernels and copies in between."""
    from kernel_b200.ops.local import product

    a, eye = _ints(256, 512, seed=20), torch.eye(512, dtype=torch.bfloat16, device=DEV)
    side = torch.cuda.Stream()
    w = torch.zeros(512, 512, dtype=torch.bfloat16, device=DEV)
    res = torch.zeros(256, 512, dtype=torch.bfloat16, device=DEV)
    other = torch.zeros(256, 512, dtype=torch.bfloat16, device=DEV)

    def chain():
        cur = torch.cuda.current_stream()
        w.zero_()
        w.copy_(eye)                     # read by the next product
        y = a
        for _ in range(6):
            y = product(y, w)            # each reads the one before
        w.mul_(2.0)                      # after the last read, before the next
        side.wait_stream(cur)
        with torch.cuda.stream(side):
            other.copy_(product(a, w))
        y = product(y, w)
        cur.wait_stream(side)
        res.copy_(product(other, eye))   # first kernel behind the join
        res.add_(y)

    chain()
    torch.cuda.synchronize()
    assert torch.equal(res, 4 * a)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for _ in range(3):
        res.zero_()
        other.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(res, 4 * a)


def test_overlapped_row_kernels_keep_their_order_eagerly_and_in_a_graph():
    """Permutation, grouped products, combine and its backward, each reading what the launch before
    wrote, with the routing table, the weights and the tokens rewritten directly before they are read."""
    from kernel_b200.ops.local import ExpertRows, contract_product, rows_product

    T, k, E, H = 96, 2, 8, 128
    g = torch.Generator(device=DEV).manual_seed(3)
    tables = [torch.rand((T, E), device=DEV, generator=g).argsort(1)[:, :k].to(torch.int32).contiguous() for _ in range(2)]
    tokens = [_ints(T, H, seed=40 + i) for i in range(2)]
    eye = torch.eye(H, dtype=torch.bfloat16, device=DEV).repeat(E, 1, 1)
    which = torch.zeros((), dtype=torch.int64, device=DEV)
    x, idx, b, w = torch.zeros_like(tokens[0]), torch.zeros_like(tables[0]), torch.zeros_like(eye), torch.zeros((T, k), device=DEV)
    both_tables, both_tokens, res = torch.stack(tables), torch.stack(tokens), {}

    def chain():
        b.copy_(eye * (1 + which))
        w.copy_((2 + which).float().expand(T, k))
        idx.copy_(both_tables.index_select(0, which.view(1))[0])
        x.copy_(both_tokens.index_select(0, which.view(1))[0])
        er = ExpertRows(x, idx, E, pad=64)                             # reads x and idx as just written
        y = rows_product(er.rows, b, er.start, er.padded)              # reads b, the table and the rows
        y = rows_product(y, b, er.start, er.padded, b_t=True)
        res["out"] = er.combine(y, w)
        dyr, res["dw"] = er.grad_rows(res["out"], y, w)                # reads what combine wrote
        res["c"] = contract_product(dyr, er.rows, er.start, er.count)  # reads what grad_rows wrote
        w.zero_()                                                      # after its last reader

    def check(i):
        s = (1 + i) ** 2
        xi, wi = tokens[i].float(), float(2 + i)
        out = (k * wi * s * xi).to(torch.bfloat16)
        assert torch.equal(res["out"], out)
        assert torch.equal(res["dw"], (out.float() * s * xi).sum(1, keepdim=True).expand(T, k))
        for e in range(E):
            rows = (tables[i] == e).any(1)
            assert torch.equal(res["c"][e], ((wi * out[rows].float()).to(torch.bfloat16).float().t() @ xi[rows]).to(torch.bfloat16))

    for i in (0, 1, 0):
        which.fill_(i)
        chain()
        torch.cuda.synchronize()
        check(i)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        chain()
    for i in (1, 0, 1):
        which.fill_(i)
        graph.replay()
        torch.cuda.synchronize()
        check(i)


@pytest.mark.parametrize("hot", [1.0, 0.5])
@pytest.mark.parametrize("T,k,E", [(300, 2, 64), (33, 4, 256)])
def test_moe_layers_with_skewed_routing(hot, T, k, E):
    """One expert receives every token, or every second one: the tile rule works from the average group."""
    from kernel_b200.models import MoELayer, TrainableMoELayer

    torch.manual_seed(4)
    H, F = 128, 136
    layer = TrainableMoELayer(E, k, H, F, T, device=torch.device(DEV))
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_(True)
    score = torch.rand(T, E, device=DEV)
    score[torch.rand(T, device=DEV) < hot, E // 2] = -1.0
    idx = score.argsort(1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn(T, k, device=DEV), -1).requires_grad_(True)
    dy = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    y = layer(x, idx, w)
    got = [y, *torch.autograd.grad(y, (x, layer.w_up, layer.w_down), dy)]
    fixed = MoELayer(E, k, H, T, layer.w_up.data, layer.w_down.data)
    assert torch.equal(fixed(x.detach(), idx, w.detach()), y)
    leaves = [t.detach().double().requires_grad_(True) for t in (x, layer.w_up, layer.w_down)]
    h = torch.nn.functional.silu(torch.einsum("th,tkfh->tkf", leaves[0], leaves[1][idx.long()]))
    ref = (torch.einsum("tkf,tkhf->tkh", h, leaves[2][idx.long()]) * w.detach().double().unsqueeze(-1)).sum(1)
    for p, q in zip(got, [ref, *torch.autograd.grad(ref, leaves, dy.double())]):
        assert (p.double() - q).norm() <= 4 * 2 ** -9 * q.norm()   # at most four bf16 roundings on the way
    layer.a2a.heap.check_status()
    fixed.a2a.heap.close()
    layer.close()


@pytest.mark.parametrize("activation", ["gelu", "silu", "relu"])
def test_mlp_with_hooks_equals_the_fused_block(activation):
    """Hooks on the two linear layers run: the block then takes the general path."""
    from kernel_b200.models import TrainableSequenceParallelMLP

    torch.manual_seed(0)
    mlp = TrainableSequenceParallelMLP(72, 136, 264, activation=activation, device=torch.device(DEV))
    x = torch.randn(72, 136, device=DEV).to(torch.bfloat16)
    fused = mlp(x)
    seen = []
    handle = mlp.up.register_forward_hook(lambda mod, inp, out: seen.append(out.shape))
    plain = mlp(x)
    handle.remove()
    assert seen == [(72, 264)]
    # the fused block's gelu and silu differ from torch's by at most one bf16 rounding of the hidden value
    assert (fused.float() - plain.float()).norm() <= 2 ** -8 * plain.float().norm()
    mlp.close()


def test_mlp_with_strided_parameters():
    """Transposed views as weights and input: the fused block gives what it gives for their copies."""
    from kernel_b200.models import TrainableSequenceParallelMLP

    torch.manual_seed(1)
    mlp = TrainableSequenceParallelMLP(72, 136, 264, device=torch.device(DEV))
    x = torch.randn(72, 136, device=DEV).to(torch.bfloat16)
    want = mlp(x)
    for t in (mlp.up.weight, mlp.down.weight):
        t.data = t.data.t().contiguous().t()
    assert torch.equal(mlp(x.t().contiguous().t()), want)
    mlp.close()


def test_stamped_time_leaves_out_the_previous_kernel():
    """``KB200_GEMM_TIMING`` (read once per process) stamps a product's own time, although the
    product is set up while the one before it, on 64 of the SMs, still runs."""
    import os
    import subprocess
    import sys
    from pathlib import Path

    code = """
import torch
from kernel_b200.ops.gemm import gemm
a, b = (torch.zeros(8192, 8192, dtype=torch.bfloat16, device="cuda") for _ in range(2))
st = [torch.zeros(8, dtype=torch.int32, device="cuda") for _ in range(2)]
small = torch.zeros(128, 128, dtype=torch.bfloat16, device="cuda")
for _ in range(3):
    for s in st: s.zero_()
    gemm(a, b, status=st[0], num_ctas=64)
    gemm(small, small, status=st[1])
torch.cuda.synchronize()
print(int(st[0][7]), int(st[1][7]))
"""
    out = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, KB200_GEMM_TIMING="1"), cwd=Path(__file__).parents[1], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stderr
    large, small = map(int, out.stdout.split())
    assert large > 200 and small < large / 4, (large, small)


def test_moe_layers_take_token_rows_with_trailing_unit_dimensions():
    from kernel_b200.models import MoELayer, TrainableMoELayer

    torch.manual_seed(2)
    E, k, H, F, T = 4, 2, 64, 128, 5
    layer = TrainableMoELayer(E, k, H, F, 8, device=torch.device(DEV))
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    idx = torch.rand(T, E, device=DEV).argsort(1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn(T, k, device=DEV), -1)
    res = []
    for shape in ((T, H), (T, H, 1)):
        leaf = x.view(shape).requires_grad_(True)
        y = layer(leaf, idx, w)
        fixed = MoELayer(E, k, H, 8, layer.w_up.data, layer.w_down.data)
        res.append([y.detach(), fixed(x.view(shape), idx, w), *torch.autograd.grad(y, leaf, torch.ones_like(y))])
        assert all(t.shape == shape for t in res[-1])
        fixed.a2a.heap.close()
    assert all(torch.equal(p.view(T, H), q.view(T, H)) for p, q in zip(*res))
    layer.close()
