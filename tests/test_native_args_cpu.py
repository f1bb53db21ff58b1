"""Argument checks of the device entry points that run before any CUDA call: a bad
problem is refused with a message, on a machine without a GPU too."""
import ctypes as C

import pytest

from kernel_b200 import _native as N


def _args(**kw):
    a = N.GemmArgs()
    buf = C.create_string_buffer(4096 + 16)
    base = (C.addressof(buf) + 15) & ~15
    a.mode, a.M, a.N, a.K = N.GEMM_PLAIN, 128, 256, 64
    a.A = a.B = a.out = base
    a.rank, a.world, a.epoch = 0, 1, 1
    for k, v in kw.items():
        setattr(a, k, v)
    a._keepalive = buf
    return a, base


@pytest.mark.parametrize("kw,needle", [
    (dict(M=0), "need M,N,K > 0"),
    (dict(K=60), "multiples of 8"),
    (dict(N=100), "multiples of 8"),
    (dict(world=0), "bad rank/world"),
    (dict(world=2, rank=2), "bad rank/world"),
    (dict(world=N.KB_MAX_WORLD + 1), "bad rank/world"),
])
def test_gemm_refuses_bad_problem(kw, needle):
    a, _ = _args(**kw)
    assert N.lib().kb_gemm(C.byref(a), None) == N.KB_ERR_ARG
    assert needle in N.last_error()


def test_gemm_refuses_misaligned_operands():
    a, base = _args()
    a.B = base + 8
    assert N.lib().kb_gemm(C.byref(a), None) == N.KB_ERR_ARG
    assert "16-byte aligned" in N.last_error()
    a, base = _args()
    a.bias = base + 2
    assert N.lib().kb_gemm(C.byref(a), None) == N.KB_ERR_ARG


@pytest.mark.parametrize("mode", [N.GEMM_RS, N.GEMM_AG])
def test_fused_gemm_refuses_bad_sharding(mode):
    lib = N.lib()
    a, _ = _args(mode=mode, world=3, rank=0, M=128)
    assert lib.kb_gemm(C.byref(a), None) == N.KB_ERR_ARG and "divisible by world" in N.last_error()
    a, _ = _args(mode=mode, world=2, rank=0, M=192)      # 96 rows per rank
    assert lib.kb_gemm(C.byref(a), None) == N.KB_ERR_ARG and "rows per rank" in N.last_error()
    a, _ = _args(mode=mode, world=2, rank=1, M=256)      # no peer segments given
    assert lib.kb_gemm(C.byref(a), None) == N.KB_ERR_ARG and "peer_base[0] is null" in N.last_error()


def test_null_argument_block():
    assert N.lib().kb_gemm(None, None) == N.KB_ERR_ARG
    assert N.lib().kb_gemm_host(None, 1) == N.KB_ERR_ARG
    assert N.lib().kb_a2a_round_trip_host(None, 1) == N.KB_ERR_ARG
    assert N.lib().kb_a2a_dispatch_host(None, 1) == N.KB_ERR_ARG
    assert N.lib().kb_a2a_combine_host(None, 1) == N.KB_ERR_ARG


def test_schedule_refuses_bad_problem():
    lib = N.lib()
    blk, nb = C.c_int(), C.c_int()
    assert lib.kb_gemm_schedule(N.GEMM_RS, 100, 256, 0, 3, 0, 0, C.byref(blk), C.byref(nb)) == -1    # M % world
    assert lib.kb_gemm_schedule(N.GEMM_RS, 256, 256, 2, 2, 0, 0, C.byref(blk), C.byref(nb)) == -1    # rank out of range
    assert lib.kb_gemm_schedule(N.GEMM_AG, 256, 256, 0, 2, 1, 0, C.byref(blk), C.byref(nb)) == -1    # pairs need 256-row shards


def _local(**kw):
    a = N.LocalGemmArgs()
    buf = C.create_string_buffer(4096 + 16)
    base = (C.addressof(buf) + 15) & ~15
    a.kind, a.M, a.N, a.K, a.pair = N.LOCAL_DENSE, 128, 256, 64, -1
    a.A = a.B = a.out = base
    for k, v in kw.items():
        setattr(a, k, base + v if k in ("A", "bias", "pre_out", "pre_in") else v)
    a._keepalive = buf
    return a


@pytest.mark.parametrize("kw,needle", [
    (dict(M=0), "M,N,K > 0"),
    (dict(K=60), "multiples of 8"),
    (dict(N=100), "multiples of 8"),
    (dict(a_mn=1, b_mn=1, M=100), "multiples of 8"),
    (dict(a_mn=1), "only with B contiguous along N"),
    (dict(kind=3), "unknown kind"),
    (dict(act=4), "unknown kind"),
    (dict(pre_in=0), "belong to an activation"),
    (dict(kind=N.LOCAL_ROWS, groups=4), "bad groups"),
    (dict(A=8), "16-byte aligned"),
    (dict(bias=2), "16-byte aligned"),
])
def test_local_gemm_refuses_bad_problem(kw, needle):
    a = _local(**kw)
    assert N.lib().kb_gemm_local(C.byref(a), None) in (N.KB_ERR_ARG, N.KB_ERR_UNSUPPORTED)
    assert needle in N.last_error()


def test_moe_rows_refuse_misaligned_rows():
    lib = N.lib()
    buf = C.create_string_buffer(4096 + 16)
    p = (C.addressof(buf) + 15) & ~15
    assert lib.kb_moe_permute(p + 2, p, 1, 1, 4, 8, 1, p, p, p, p, p, p, None) == N.KB_ERR_ARG and "16-byte aligned" in N.last_error()
    assert lib.kb_moe_permute(p, p + 2, 1, 1, 4, 8, 1, p, p, p, p, p, p, None) == N.KB_ERR_ARG and "4-byte aligned" in N.last_error()
    assert lib.kb_moe_grad_rows(p + 2, p, p, p, 1, 1, 4, 8, p, p, p, p, p, None) == N.KB_ERR_ARG


def test_local_gemm_tile_rule_gives_launchable_configurations():
    """Whatever the sizes, the picked tile has a legal width for its layout, a pair has rows
    for both CTAs and a split has k blocks for every member."""
    import random

    rng = random.Random(0)
    lib = N.lib()
    pair, bn, split = C.c_int(), C.c_int(), C.c_int()
    for _ in range(3000):
        M, Nn, K = (8 * int(2 ** rng.uniform(0, 12)) for _ in range(3))
        a_mn, b_mn = rng.choice([(0, 0), (0, 1), (1, 1)])
        sms = rng.choice([148, 132, 16, 2])
        assert lib.kb_gemm_local_config(M, Nn, K, a_mn, b_mn, sms, C.byref(pair), C.byref(bn), C.byref(split)) == N.KB_OK
        per_cta = bn.value // 2 if pair.value else bn.value
        assert 64 <= bn.value <= 256 and (per_cta % 64 == 0 if b_mn else bn.value % 32 == 0)
        assert pair.value == 0 or M > 128
        assert 1 <= split.value <= (8, 4, 1)[pair.value] and split.value <= (K + 63) // 64


def _pick(sms, **kw):
    """What ``kb_gemm_local`` launches: (exchanged operands, pair, columns, rows of a tile, split)."""
    a, p = _local(**kw), N.LocalPick()
    assert N.lib().kb_gemm_local_pick(C.byref(a), sms, C.byref(p)) == N.KB_OK, (kw, N.last_error())
    return p.exchanged, p.pair, p.bn, p.rows, p.split


def _exchanged_tile_runs(pair, bn, tok, split, K, w_mn, groups, rows):
    """The limits of the exchanged-operand kernel, restated: 128 columns per CTA, blocks of at most 256 tokens, two stages and
    the partial tiles of a split in 232448 bytes of shared memory."""
    ctas, step = (2, 32) if pair else (1, 16)
    w_cols, tok_cta = bn // ctas, tok // ctas
    assert bn % ctas == 0 and 8 <= w_cols <= 128 and w_cols % (64 if w_mn else 8) == 0
    assert step <= tok <= 256 and tok % step == 0
    assert 1 <= split <= (4 if pair else 8) and split <= (K + 63) // 64 and (split == 1 or not groups)
    box = tok_cta
    if groups:  # boxes of half the block that most groups fit
        most = rows / groups + 2 * (rows / groups) ** 0.5
        block = (int(most) // step + 1) * step // ctas if most < tok else tok_cta
        box = min(max((block + 15) // 16 * 8, 16), tok_cta)
    stage = w_cols * 128 + -(-tok_cta // box) * box * 128
    stages = min(16, (232448 - 1024 - 512 - 4 * (3 * groups + 1)) // stage)
    assert box % 8 == 0 and stages >= 2
    assert w_cols * 128 + stages * (stage - w_cols * 128) >= 128 * 128  # the MMA reads 128 rows from the last weight slot on
    if split > 1:
        chunks = -(-(tok // 8) // split)  # of the member that owns most
        assert chunks * (split - 1) * 128 * 8 * 4 <= stages * stage


def test_picked_tiles_are_launchable():
    """Dense products with either operand layout and grouped rows, with few and many rows on few and many SMs: the tile
    that is launched, whichever kind it is."""
    import random

    rng = random.Random(1)
    seen = set()
    for i in range(6000):
        M, Nn, K = int(2 ** rng.uniform(0, 13)), 8 * int(2 ** rng.uniform(0, 12)), 8 * int(2 ** rng.uniform(0, 12))
        sms = rng.choice([148, 148, 132, 16, 2, 1])
        b_mn = rng.choice([0, 1])
        kw = dict(M=M, N=Nn, K=K, b_mn=b_mn)
        if i % 2:
            groups = int(2 ** rng.uniform(0, 10))
            kw.update(kind=N.LOCAL_ROWS, groups=groups, expect=rng.choice([0, 1 + M // 2]))
            kw.update(row_start=16, row_count=16)  # not read
        swap, pair, bn, rows, split = _pick(sms, **kw)
        seen.add((i % 2, b_mn, swap, pair))
        assert sms > 1 or not pair
        if swap:
            _exchanged_tile_runs(pair, bn, rows, split, K, b_mn, kw.get("groups", 0), kw.get("expect") or M)
        else:
            assert 32 <= bn <= 256 and ((bn // 2 if pair else bn) % 64 == 0 if b_mn else bn % 32 == 0)
            assert 1 <= split <= (8, 4, 1)[pair] and split <= (K + 63) // 64 and (split == 1 or not i % 2)
    # every kind of tile was picked for every kind of product
    assert seen >= {(g, b, s, p) for g in (0, 1) for b in (0, 1) for s in (0, 1) for p in (0, 1)}, seen


def test_tiles_that_no_kernel_runs_are_refused():
    p = N.LocalPick()
    for kw in (dict(pair=3, bn=136), dict(pair=4, bn=64, b_mn=1), dict(pair=3, bn=64, tok=24), dict(pair=3, bn=64, tok=272),
               dict(pair=3, split=2), dict(pair=0, bn=40), dict(pair=1, bn=64, b_mn=1, M=256), dict(pair=0, bn=64, split=9)):
        a = _local(**kw)
        assert N.lib().kb_gemm_local_pick(C.byref(a), 148, C.byref(p)) == N.KB_ERR_UNSUPPORTED, kw


def test_a_tile_that_is_asked_for_is_of_the_kind_with_rows_on_the_m_side():
    """Columns (or a split) without a kind mean the M side, in grouped products as in dense ones."""
    free = dict(kind=N.LOCAL_ROWS, M=192, N=1024, K=2048, groups=64, row_start=16, row_count=16)
    assert _pick(148, **free)[0] == 1
    for bn in (64, 128, 256):
        assert _pick(148, **free, bn=bn)[:3:2] == (0, bn)
    assert _pick(148, M=64, N=1104, K=20000)[0] == 1
    assert _pick(148, M=64, N=1104, K=20000, bn=96)[:3:2] == (0, 96)
    assert _pick(148, **free, pair=3, bn=64)[:3:2] == (1, 64)


def test_which_launches_of_split_products_are_overlapped():
    """All but clusters of an odd size that fill the chip and long reads of weights by clusters of two on less than 9/10 of
    the SMs."""
    def overlapped(pair, clusters, split, K):
        a, p = _local(M=64, N=128 * clusters, K=K, pair=pair, bn=128, split=split), N.LocalPick()
        assert N.lib().kb_gemm_local_pick(C.byref(a), 148, C.byref(p)) == N.KB_OK and (p.bn, p.split) == (128, split)
        return p.overlapped

    for pair in (0, 3):
        assert [overlapped(pair, n, 3, 4096) for n in (43, 44, 45)] == [1, 0, 0]
        assert [overlapped(pair, n, 5, 4096) for n in (20, 25, 26)] == [1, 1, 0]
        assert [overlapped(pair, n, 7, 4096) for n in (10, 15)] == [1, 1]
        for split in (4, 6, 8):
            assert all(overlapped(pair, n, split, 20000) for n in range(8, 148 // split + 1))
        assert [overlapped(pair, n, 2, 20000) for n in (40, 64, 66, 67, 74)] == [0, 0, 0, 1, 1]
        assert [overlapped(pair, 64, 2, K) for K in (9600, 9768)] == [1, 0]   # 157, 160 MB


def test_kind_of_dense_products_whose_difference_was_measured():
    """Products at least 10 % apart on a B200: the faster kind (us, rows on the M side / exchanged)."""
    for M, Nn, K, b_mn in ((267, 4120, 1344, 0),     # 12.3 16.5
                           (443, 3624, 2352, 0),     # 13.7 15.9
                           (164, 3072, 1728, 0),     # 10.5 16.5
                           (301, 1136, 1600, 0),     # 9.2 14.2
                           (182, 7496, 1488, 1),     # 11.7 13.6
                           (256, 4096, 14336, 0)):   # 36.5 46.0
        assert _pick(148, M=M, N=Nn, K=K, b_mn=b_mn)[0] == 0, (M, Nn, K)
    for M, Nn, K, b_mn in ((400, 25000, 1504, 0),    # 35.1 31.2
                           (142, 1184, 23256, 0),    # 31.9 24.0
                           (309, 8208, 23040, 0),    # 126 100
                           (4, 1632, 6040, 1),       # 13.4 10.4
                           (285, 4640, 5696, 0)):    # 24.2 19.3
        assert _pick(148, M=M, N=Nn, K=K, b_mn=b_mn)[0] == 1, (M, Nn, K)
    for M, Nn, K in ((285, 17576, 1712), (190, 12288, 3216), (1051, 4920, 4448)):   # with a slope: 51.4 30.9, 38.7 27.6, 89.9 65.6
        assert _pick(148, M=M, N=Nn, K=K, b_mn=1, act=N.ACTS["silu"], pre_in=0)[0] == 1, (M, Nn, K)


def test_tiles_of_few_rows_whose_difference_was_measured():
    """At least 7 % apart on a B200, repeated (us, this tile / the one a shorter time per box of a pair gives)."""
    slope = dict(b_mn=1, act=N.ACTS["gelu"], pre_in=16)
    for (M, Nn, K), kw, want in (((1, 23464, 1504), {}, (1, 0, 80, 16, 1)),              # 14.7 16.4
                                 ((1, 21248, 3704), {}, (1, 0, 72, 16, 1)),              # 30.6 32.9
                                 ((7, 9592, 7560), {}, (1, 0, 72, 16, 1)),               # 31.0 34.3
                                 ((23, 25792, 7536), dict(b_mn=1), (1, 1, 256, 32, 1)),  # 67.8 77.9
                                 ((56, 24048, 14832), dict(b_mn=1), (1, 1, 256, 64, 1)), # 144 158
                                 ((37, 27056, 3488), slope, (1, 1, 256, 64, 1)),         # 40.7 47.0
                                 ((29, 22272, 12976), slope, (1, 1, 256, 32, 1))):       # 109 125
        assert _pick(148, M=M, N=Nn, K=K, **kw)[:5] == want, (M, Nn, K)


def test_512_rows_with_an_activation():
    """On a B200, repeated, at least 5 % apart (us, 512-row tiles / pairs): rows of odd multiples of 16 bytes want them, others do not."""
    gelu = N.ACTS["gelu"]
    for M, Nn, K, keep, want in ((8009, 13128, 8424, 0, 2),    # 1503 1852
                                 (3032, 2496, 8504, 0, 2),     # 121 146
                                 (7121, 25744, 8408, 1, 2),    # 2589 3322
                                 (1570, 9032, 14968, 1, 2),    # 427 519
                                 (7416, 17744, 5200, 0, 1),    # 1179 1016
                                 (5626, 16064, 4192, 0, 1),    # 633 591
                                 (8192, 14336, 4096, 1, 1),    # 850 731
                                 (8083, 12864, 4528, 1, 1)):   # 839 794
        assert _pick(148, M=M, N=Nn, K=K, act=gelu, **(dict(pre_out=16) if keep else {}))[:2] == (0, want), (M, Nn, K)
    for M, Nn, K, want in ((7974, 21272, 6984, 2),    # 2423 2875 (exchanged pairs)
                           (4799, 12416, 17208, 2),   # 1744 2070
                           (4728, 4904, 4544, 1),     # 256 205
                           (8192, 14336, 4096, 1)):   # 855 762
        assert _pick(148, M=M, N=Nn, K=K, b_mn=1, act=gelu, pre_in=16)[1] == want, (M, Nn, K)


def test_a_product_that_may_fetch_its_weights_early_is_exchanged_sooner():
    """Near ties: the exchanged kernel alone fetches them under the previous launch."""
    for M, Nn, K in ((128, 4096, 4096), (330, 6296, 1304), (672, 10008, 2040)):
        assert [_pick(148, M=M, N=Nn, K=K, early=early)[0] for early in (0, 1)] == [0, 1], (M, Nn, K)
    assert _pick(148, M=256, N=4096, K=14336, early=1)[0] == 0   # 36.5 us, exchanged 46.0


def test_kind_of_grouped_products_whose_difference_was_measured():
    """At least 8 % apart on a B200 with uniformly routed rows (us, rows on the M side / exchanged)."""
    def kind(groups, rows, Nn, K, **kw):
        return _pick(148, kind=N.LOCAL_ROWS, M=rows, N=Nn, K=K, groups=groups, row_start=16, row_count=16, **kw)[0]

    assert kind(8, 968, 640, 2960) == 0      # 15.9 20.7
    assert kind(8, 446, 712, 1280) == 0      # 8.2 10.4
    assert kind(16, 3400, 560, 864) == 0     # 12.0 11.1, but 8.0 with groups of one size
    assert kind(64, 192, 760, 2728) == 1     # 99.5 89.4
    assert kind(64, 8192, 1024, 2048) == 1   # 75.3 67.7
    slope = dict(b_mn=1, act=N.ACTS["silu"], pre_in=0)
    assert kind(64, 10240, 1024, 2048, **slope) == 1   # 90.8 75.4
    assert kind(64, 4096, 2872, 552, **slope) == 1     # 50.0 35.3, 64 rows of padding and tokens in every group
    assert kind(8, 4000, 4096, 4096, **slope) == 1     # 116 94.4


def test_tiles_of_grouped_products_of_few_rows_whose_difference_was_measured():
    """At least 8 % apart on a B200 (us, rows on the M side / exchanged, one CTA / exchanged pair)."""
    def tile(groups, rows, Nn, K, **kw):
        return _pick(148, kind=N.LOCAL_ROWS, M=rows, N=Nn, K=K, groups=groups, row_start=16, row_count=16, **kw)[:2]

    silu = dict(act=N.ACTS["silu"])
    assert tile(16, 4, 832, 3600, **silu) == (1, 0)          # 16.4 in pairs, 14.3 before them
    assert tile(8, 2, 3816, 3632, **silu) == (1, 0)          # 18.3 15.6 17.1
    assert tile(64, 12, 520, 3504, early=1) == (1, 0)        # 15.5 13.5 14.8
    assert tile(32, 850, 672, 2016) == (0, 0)                # 18.8 24.1 23.5
    assert tile(8, 168, 2456, 2144, b_mn=1) == (0, 0)        # 19.9 24.0 24.5
    assert tile(8, 156, 2696, 2688, b_mn=1) == (0, 0)        # 25.8 30.1 30.9
    assert tile(64, 192, 1024, 2048, **silu) == (1, 0)       # 47.6 45.5


def test_tiles_of_contractions_whose_difference_was_measured():
    """At least 5 % apart on a B200 (us, one CTA / pair)."""
    def pair(groups, rows, M, Nn):
        return _pick(148, kind=N.LOCAL_CONTRACT, M=M, N=Nn, K=groups * (rows + 63), groups=groups, expect=groups * rows, row_start=16, row_count=16)[1]

    for product in ((8, 171, 832, 1088),      # 7.1 9.0
                    (8, 77, 616, 2384),       # 9.8 11.6
                    (8, 69, 640, 1024),       # 6.1 7.1
                    (16, 94, 608, 560),       # 6.8 7.7
                    (16, 74, 896, 1408),      # 12.4 13.5
                    (64, 32, 2048, 1024)):    # 57 58: one k block
        assert pair(*product) == 0, product
    for product in ((64, 128, 2048, 1024),    # 77.5 71.7
                    (8, 180, 976, 1704),      # 14.0 12.9
                    (16, 157, 1720, 584),     # 19.1 17.4
                    (32, 97, 696, 1560),      # 28.8 26.5
                    (128, 79, 704, 1480),     # 92.8 83.3
                    (32, 242, 1160, 568)):    # 31.1 26.7
        assert pair(*product) == 1, product


def test_weights_that_are_asked_for_ahead():
    """Only where that gains more for weights in memory than it costs for weights in the L2 (us without / with, from the L2; from memory)."""
    def ahead(M, Nn, K, **kw):
        a, p = _local(M=M, N=Nn, K=K, **kw), N.LocalPick()
        assert N.lib().kb_gemm_local_pick(C.byref(a), 148, C.byref(p)) == N.KB_OK
        return p.ahead

    for product in ((16, 2336, 5544), (38, 1712, 7840), (73, 9200, 1632)):   # 7.9 8.5, 9.5 9.2; 8.8 9.4, 10.4 10.1; 8.5 9.1, 10.6 10.1
        assert ahead(*product) == 0, product
    for product in ((8, 4096, 4096), (16, 4608, 4608), (32, 7168, 4096)):    # 7.4 7.8, 10.1 9.6; 8.4 8.8, 11.6 10.3; 10.0 10.4, 14.2 12.8
        assert ahead(*product) == 1, product
    for kw in (dict(b_mn=1), dict(early=1)):
        assert ahead(32, 7168, 4096, **kw) == 0, kw
    assert ahead(129, 7168, 4096) == 0


def test_ring_of_contractions_over_one_k_block():
    """At least 5 % apart on a B200 (us, three stages / two)."""
    def stages(groups, rows, M, Nn):
        a, p = _local(kind=N.LOCAL_CONTRACT, M=M, N=Nn, K=groups * (rows + 63), groups=groups, expect=groups * rows, row_start=16, row_count=16), N.LocalPick()
        assert N.lib().kb_gemm_local_pick(C.byref(a), 148, C.byref(p)) == N.KB_OK and p.pair == 0
        return p.stages

    for product in ((64, 22, 3448, 960),      # 92.2 81.4
                    (64, 19, 3656, 648),      # 95.9 77.6
                    (64, 5, 2320, 1752),      # 165 134
                    (32, 22, 2064, 2888),     # 110 93.4
                    (64, 16, 2048, 1024),     # 56.1 51.5
                    (128, 6, 656, 2160)):     # 85.3 80.2
        assert stages(*product) == 2, product
    for product in ((32, 24, 3792, 1424),     # 63.9 72.1
                    (64, 45, 3112, 1248),     # 88.9 96.9
                    (128, 10, 1848, 624),     # 58.3 65.8
                    (32, 24, 1128, 2416),     # 35.0 38.7
                    (32, 30, 2816, 2848),     # 94.2 103
                    (16, 29, 3744, 2960),     # 65.8 72.1
                    (64, 64, 2048, 1024)):    # more than one k block
        assert stages(*product) == 3, product


def test_vectors_per_lane_of_the_round_trip():
    """Where a form was at least 5 % faster than the others on a B200 (us with 1 / 2 / 4 vectors per lane)."""
    vecs = lambda tokens, hidden, elem=2: N.lib().kb_a2a_local_vecs(tokens, hidden, elem, 148)
    for tokens, hidden in ((2048, 7168), (2048, 4096), (300, 7168)):
        assert vecs(tokens, hidden) == vecs(tokens, hidden, 4) == 4        # 28.6 25.4 21.5 for the first
    for tokens, hidden in ((1, 7168), (60, 7168), (101, 2880), (130, 1024)):
        assert vecs(tokens, hidden) == 1
    for tokens, hidden in ((700, 1048), (700, 1280)):
        assert vecs(tokens, hidden) == 1, (tokens, hidden)                 # 3.7 4.0 4.6 for the first
    for tokens, hidden in ((2048, 2056), (2048, 2560), (300, 4104), (700, 1536)):
        assert vecs(tokens, hidden) == 2, (tokens, hidden)                 # 10.6 9.6 11.7 for the first
    assert vecs(2048, 2560, 4) == 4                                        # fp32: 14.4 14.4 11.8 for 2880 values
