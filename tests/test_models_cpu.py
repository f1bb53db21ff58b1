"""Model blocks on the CPU paths of the ops (single process)."""
import torch


def test_sequence_parallel_mlp_cpu_single_rank():
    from kernel_b200.models import SequenceParallelMLP

    torch.manual_seed(0)
    tokens, hidden, ffn = 32, 64, 128
    x = torch.randn(tokens, hidden).to(torch.bfloat16)
    w1 = (torch.randn(ffn, hidden) / hidden ** 0.5).to(torch.bfloat16)
    w2 = (torch.randn(hidden, ffn) / ffn ** 0.5).to(torch.bfloat16)
    b1 = (torch.randn(ffn) * 0.02).to(torch.bfloat16)
    mlp = SequenceParallelMLP(tokens, hidden, w1, w2, b1, None, activation="silu")
    y = mlp(x)
    ref = mlp.reference(x, w1, w2, b1, None)
    assert y.shape == (tokens, hidden) and torch.allclose(y.float(), ref, rtol=2e-2, atol=2e-2)


def test_moe_layer_dense_formulation_matches_manual():
    from kernel_b200.models import MoELayer

    torch.manual_seed(1)
    E, k, H, F, T = 4, 2, 32, 64, 6
    w_up = (torch.randn(E, F, H) / H ** 0.5).to(torch.bfloat16)
    w_down = (torch.randn(E, H, F) / F ** 0.5).to(torch.bfloat16)
    layer = MoELayer(E, k, H, T, w_up, w_down)
    x = torch.randn(T, H).to(torch.bfloat16)
    idx = torch.rand(T, E).argsort(1)[:, :k].to(torch.int32)
    w = torch.softmax(torch.randn(T, k), -1)
    y = layer(x, idx, w)
    manual = torch.zeros(T, H)
    for t in range(T):
        for j in range(k):
            e = int(idx[t, j])
            h = torch.nn.functional.silu(x[t].float() @ w_up[e].float().t())
            manual[t] += w[t, j] * (h @ w_down[e].float().t())
    assert torch.allclose(y.float(), manual, rtol=5e-2, atol=5e-2)


def _moe_layer_ranks(rank, world):
    """Forward of the expert-parallel layer on CPU ranks (host-heap dispatch and
    combine around real expert MLPs) against the single-process formulation with all experts."""
    from kernel_b200.models import MoELayer

    E, k, H, F, T = 3 * world, 2, 32, 64, 5 + rank
    El = E // world
    full = torch.Generator().manual_seed(9)
    w_up = (torch.randn(E, F, H, generator=full) / H ** 0.5).to(torch.bfloat16)
    w_down = (torch.randn(E, H, F, generator=full) / F ** 0.5).to(torch.bfloat16)
    layer = MoELayer(E, k, H, 8, w_up[rank * El:(rank + 1) * El], w_down[rank * El:(rank + 1) * El])
    g = torch.Generator().manual_seed(20 + rank)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16)
    idx = torch.rand(T, E, generator=g).argsort(1)[:, :k].to(torch.int32).contiguous()
    w = torch.softmax(torch.randn(T, k, generator=g), -1)
    y1 = layer(x, idx, w)
    y2 = layer(x, idx, w)
    manual = torch.zeros(T, H)
    for t in range(T):
        for j in range(k):
            e = int(idx[t, j])
            h = torch.nn.functional.silu(x[t].float() @ w_up[e].float().t())
            manual[t] += w[t, j] * (h @ w_down[e].float().t())
    ok = torch.allclose(y1.float(), manual, rtol=5e-2, atol=5e-2) and torch.equal(y1, y2)
    layer.close()
    return bool(ok)


def test_moe_layer_on_cpu_ranks_world3():
    from _mp import run_ranks

    assert all(run_ranks(_moe_layer_ranks, 3))


def test_layers_that_are_asked_for_by_themselves_are_not_fused():
    """The one-GPU block passes its linear layers by only when nothing could notice: no hook of a
    layer or of all modules, no replaced layer, no ``forward`` set on the instance."""
    from torch.nn.modules import module as M

    from kernel_b200.models.tp_mlp import TrainableSequenceParallelMLP, _plain
    from kernel_b200.ops.autograd import ColumnParallelLinear

    up = TrainableSequenceParallelMLP(8, 16, 24).up
    assert _plain(up, ColumnParallelLinear)
    hook = lambda *a: None
    for register in (up.register_forward_hook, up.register_forward_pre_hook, up.register_full_backward_hook, up.register_full_backward_pre_hook,
                     M.register_module_forward_hook, M.register_module_forward_pre_hook, M.register_module_full_backward_hook,
                     M.register_module_full_backward_pre_hook):
        handle = register(hook)
        assert not _plain(up, ColumnParallelLinear), register
        handle.remove()
        assert _plain(up, ColumnParallelLinear)
    up.forward = lambda x: x
    assert not _plain(up, ColumnParallelLinear)


def test_inference_block_calls_what_was_put_in_place_of_its_parts():
    from kernel_b200.models import SequenceParallelMLP

    w1, w2 = torch.zeros(24, 16, dtype=torch.bfloat16), torch.zeros(16, 24, dtype=torch.bfloat16)
    assert SequenceParallelMLP(8, 16, w1, w2)._plain()

    class Clipped(SequenceParallelMLP):
        def _act(self, h):
            return super()._act(h).clamp(max=1.0)

    assert not Clipped(8, 16, w1, w2)._plain()
    mlp = SequenceParallelMLP(8, 16, w1, w2)
    mlp.up = lambda x, w, b: x
    assert not mlp._plain()
    mlp = SequenceParallelMLP(8, 16, w1, w2)
    mlp._act = torch.relu
    assert not mlp._plain()


def test_inference_block_leaves_the_exchange_to_parts_that_span_several_ranks(monkeypatch):
    """A block of one rank whose down (or up) projection was replaced by a context over two ranks calls it: the
    one-GPU product would return the unreduced sum (or a part of the rows)."""
    from kernel_b200.models import SequenceParallelMLP, tp_mlp
    from kernel_b200.ops.gemm import AGGemm, GemmRS

    class OnGpu(torch.Tensor):
        is_cuda = property(lambda self: True)

    products, exchanged = [], []
    monkeypatch.setattr(tp_mlp, "product", lambda a, b, *args, **kw: products.append(kw) or torch.zeros(a.shape[0], b.shape[0], dtype=a.dtype))
    for kind in (AGGemm, GemmRS):
        monkeypatch.setattr(kind, "__call__", lambda self, a, w, *args: exchanged.append(self) or torch.zeros(self.M, w.shape[0], dtype=a.dtype))
    w1, w2 = torch.zeros(24, 16, dtype=torch.bfloat16), torch.zeros(16, 24, dtype=torch.bfloat16)

    def block():
        mlp = SequenceParallelMLP(8, 16, w1, w2)
        mlp.up.status = mlp.down.status = None
        return mlp

    def call(mlp, rows=8):
        products.clear()
        exchanged.clear()
        mlp(torch.zeros(rows, 16, dtype=torch.bfloat16).as_subclass(OnGpu))
        return len(products), exchanged

    assert call(block()) == (2, [])
    mlp = block()
    mlp.down.world = 2
    assert call(mlp) == (1, [mlp.down])
    mlp = block()
    mlp.up.world = 2
    assert call(mlp, rows=4) == (0, [mlp.up, mlp.down])


def test_expected_rows_of_padded_experts():
    """What the tile rules are told of a table that stays on the device.  An expert with any row has a whole alignment of them;
    the rules take a tile that holds the average and two standard deviations: neither half an alignment nor two."""
    from kernel_b200.models.moe import _expected_rows
    from kernel_b200.ops.local import ROW_ALIGN, ExpertRows

    er = ExpertRows.__new__(ExpertRows)
    for er.E in (8, 64, 256):
        for er.k in (1, 8):
            for er.T in range(1, 2000, 7):
                real, padded = _expected_rows(er)
                assert real == er.T * er.k and real < padded <= ExpertRows.capacity(er.T, er.k, er.E, ROW_ALIGN)
                n = padded / er.E
                if er.E // 2 <= real < 16 * er.E:
                    assert ROW_ALIGN // 2 < n + 2 * n ** 0.5 <= ROW_ALIGN, (er.E, er.k, er.T)
