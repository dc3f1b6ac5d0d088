"""The tensor-core triple-dot-product backward where its tiles, ranges and scales end."""
import pytest
import torch

from _parity import assert_close
from oracle import trittention_oracle as orc
from flash_trittention import _native

DEV = "cuda:0"
NAMES = ("dq", "dk1", "dk2", "dv1", "dv2")


def _backward(t, do, alpha, causal, windows=(None,) * 4):
    B, N, T, _ = t[0].shape
    o, lse = torch.empty_like(t[0]), torch.empty(B, N, T, device=DEV)
    _native.tdp_fwd(*t, o, lse, alpha, causal, *windows)
    g = [torch.empty_like(t[0]) for _ in range(5)]
    _native.tdp_bwd(*t, o, do, lse, *g, alpha, causal, *windows)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0, "a bounded barrier wait ran out"
    return g


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("T,D,dtype", [(260, 64, torch.float16), (260, 128, torch.bfloat16), (1100, 64, torch.bfloat16)])
def test_a_query_that_is_not_finite_stays_in_its_tile(T, D, dtype, value):
    """An infinite or NaN upstream row of query 0, which attends key 0 alone.  The products of its tile of 128 queries
    and of 128 keys see it (0 * inf); the rows past the sequence and the rows that the tensor-core kernel leaves to the
    exact first queries must not, so that every key past the first 128 and every other dQ row is what a zero row gives."""
    t = [x.to(DEV) for x in orc.make_inputs(1, 2, T, D, scale=0.5, seed=T + D, dtype=dtype)]
    do = t.pop()
    bad, zero = do.clone(), do.clone()
    bad[:, :, 0], zero[:, :, 0] = value, 0
    got, want = _backward(t, bad, 1.0 / D, True), _backward(t, zero, 1.0 / D, True)
    for name, a, b in zip(NAMES, got, want):
        a, b = (x[:, :, 1 if name == "dq" else 128:].float() for x in (a, b))
        assert torch.isfinite(a).all(), f"{name}: {int((~torch.isfinite(a)).sum())} of {a.numel()} values are not finite"
        # (two runs of the same sums: the order of the fp32 reduce-adds, and where it meets the final rounding)
        assert float((a - b).norm()) <= 1e-3 * float(b.norm()), name


def test_backward_refuses_a_register_count_that_its_split_was_not_written_for():
    """The warpgroups' shares add up to exactly the registers of the launch: with fewer, setmaxnreg.inc would wait for
    ever (88 and below), with another count one of its directions would be wrong."""
    check = _native.lib().tritt_selftest_bwd_registers
    assert check(96) == 0
    for launched in (64, 80, 88, 104, 128):
        assert check(launched) == -30
        assert b"registers per thread" in _native.lib().tritt_last_error()


@pytest.mark.parametrize("dtype", [_native.BF16, _native.F16])
@pytest.mark.parametrize("T", [200, 1024, 2051])
@pytest.mark.parametrize("q_mod", [1, 2, 3, 8, 64])
def test_exact_first_queries_are_the_first_queries_of_the_sequence(T, q_mod, dtype):
    """... and not the first 32 rows of a shard, whose queries lie q_mod apart."""
    for q_rem in {0, 1 % q_mod, q_mod // 2, q_mod - 1}:
        first, cells, by_queries = _native.tdp_bwd_plan(T, 64, dtype, True, None, None, None, None, q_mod, q_rem)
        assert first == (0 if by_queries else len(range(q_rem, 32 if T >= 1024 else 16, q_mod)))
        assert cells > 0
        assert _native.tdp_bwd_plan(T, 64, dtype, False, None, None, None, None, q_mod, q_rem)[0] == 0
    assert _native.tdp_bwd_plan(14, 64, dtype, True, None, None, None, None) == (14, 0, 0)


@pytest.mark.parametrize("T,windows,first", [
    (1500, (None,) * 4, 32), (1000, (None,) * 4, 16), (479, (9, 5, 3, 2), 16), (480, (9, 5, 3, 2), 0), (1024, (127, 0, 1, 1), 0),
    (1023, (127, 0, 1, 1), 16), (4096, (None, 0, 9, 9), 32), (40, (0, 4, 4, 4), 0), (39, (0, 4, 4, 4), 16), (12, (None,) * 4, 12)])
@pytest.mark.parametrize("dtype", [_native.BF16, _native.F16])
def test_narrow_windows_have_no_first_queries(T, windows, first, dtype):
    """Where no query has more than T / 8 pairs the first ones are no larger than the others."""
    assert _native.tdp_bwd_plan(T, 64, dtype, True, *windows, 1, 0)[0] == first


@pytest.mark.gpu
@pytest.mark.parametrize("T,q_mod", [(1030, 8), (1024, 64)])
def test_shards_with_exact_first_queries_sum_to_the_whole(T, q_mod):
    """Shards that hold some of the first 32 queries, and shards that hold none."""
    B, N, D, alpha = 1, 1, 64, 1 / 64
    t = [x.to(DEV) for x in orc.make_inputs(B, N, T, D, scale=0.5, seed=T + q_mod, dtype=torch.bfloat16)]
    do = t.pop()
    full = _backward(t, do, alpha, True)
    o, lse = torch.empty_like(do), torch.empty(B, N, T, device=DEV)
    _native.tdp_fwd(*t, o, lse, alpha, True, None, None, None, None)
    dq, n = torch.zeros_like(do), do.numel()
    acc = torch.zeros(4 * n, device=DEV)
    for rem in range(q_mod):
        ws = _native.tdp_bwd(*t, o, do, lse, dq, None, None, None, None, alpha, True, None, None, None, None,
                             q_mod=q_mod, q_rem=rem, flags=_native.FLAG_BWD_PARTIAL)
        acc += ws[: 16 * n].view(torch.float32)
    ws[: 16 * n].view(torch.float32).copy_(acc)
    got = [dq] + [torch.empty_like(do) for _ in range(4)]
    _native.tdp_bwd_finalize(t[3], *got[1:], ws)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    for name, a, b in zip(NAMES, got, full):
        assert_close(name, a, b, torch.bfloat16)


FULL = (None,) * 4


@pytest.mark.parametrize("T,D,windows", [(333, 128, FULL), (1024, 64, FULL), (2048, 128, FULL), (4096, 64, FULL),
                                         (2048, 64, (128, 128, 32, 32)), (1500, 64, (10, 700, 3, 5)), (1500, 128, (300, 20, 50, 9))])
@pytest.mark.parametrize("q_mod", [2, 3, 4, 8, 64])
def test_a_shard_executes_its_share_of_the_cells(T, D, windows, q_mod):
    """Either kernel costs at most what the one that steps over queries costs, whose cells are the queries' own and whose
    shards add up to the whole; the shares of the ranks are alike."""
    causal, cost = True, []
    whole = sum((q // 128 + 1) ** 2 * 128 * 128 for q in range(T))   # cells of the queries' tiles, without windows
    for q_rem in range(q_mod):
        first, cells, by_queries = _native.tdp_bwd_plan(T, D, _native.BF16, causal, *windows, q_mod, q_rem)
        cost.append(cells if by_queries else 0.8 * cells)
        if windows == FULL:
            own = sum((q // 128 + 1) ** 2 * 128 * 128 for q in range(q_rem, T, q_mod))
            assert cells == own if by_queries else 0.8 * cells <= own
    if windows == FULL:
        assert sum(cost) <= whole
    assert max(cost) <= 1.25 * min(cost) + 64 * 128 * 128
    assert _native.tdp_bwd_plan(T, D, _native.BF16, causal, *windows, 1, 0)[2] == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,D,q_mod,windows", [(130, 64, 2, FULL), (257, 128, 4, FULL), (300, 64, 8, (40, 100, 20, 9)),
                                               (300, 128, 3, (100, 40, 10, 30)), (600, 64, 2, FULL)])
def test_shards_sum_to_the_whole(T, D, q_mod, windows, dtype):
    """Both kernels: the dQ rows of the shards and the sum of their key-side sums are those of the whole call."""
    B, N, alpha = 1, 2, 1.0 / D
    t = [x.to(DEV) for x in orc.make_inputs(B, N, T, D, scale=0.5, seed=T + q_mod, dtype=dtype)]
    do = t.pop()
    full = _backward(t, do, alpha, True, windows)
    o, lse = torch.empty_like(do), torch.empty(B, N, T, device=DEV)
    _native.tdp_fwd(*t, o, lse, alpha, True, *windows)
    dq, n = torch.full_like(do, float("nan")), do.numel()
    acc = torch.zeros(4 * n, device=DEV)
    for rem in range(q_mod):
        ws = _native.tdp_bwd(*t, o, do, lse, dq, None, None, None, None, alpha, True, *windows, q_mod=q_mod, q_rem=rem,
                             flags=_native.FLAG_BWD_PARTIAL)
        acc += ws[: 16 * n].view(torch.float32)
    ws[: 16 * n].view(torch.float32).copy_(acc)
    got = [dq] + [torch.empty_like(do) for _ in range(4)]
    _native.tdp_bwd_finalize(t[3], *got[1:], ws)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    for name, a, b in zip(NAMES, got, full):
        assert_close(name, a, b, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("T,D,dtype", [(100, 64, torch.float16), (14, 128, torch.bfloat16), (700, 128, torch.bfloat16)])
def test_captured_backward_replays(T, D, dtype):
    """The exact first queries run beside the tensor-core kernel: the same under capture, for new inputs in the same buffers,
    and for a replay right behind another that uses the same workspace."""
    t = [x.to(DEV) for x in orc.make_inputs(1, 2, T, D, scale=0.5, seed=T, dtype=dtype)]
    do = t.pop()
    o, lse = torch.empty_like(do), torch.empty(1, 2, T, device=DEV)
    g = [torch.empty_like(do) for _ in range(5)]
    ws = _native.workspace(_native.OP_TDP_BWD, 1, 2, T, D, _native.dtype_code(dtype), do.device)
    call = lambda: _native.tdp_bwd(*t, o, do, lse, *g, 1.0 / D, True, *FULL, ws=ws)
    _native.tdp_fwd(*t, o, lse, 1.0 / D, True, *FULL)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for x, y in zip(t + [do], orc.make_inputs(1, 2, T, D, scale=0.5, seed=T + 1, dtype=dtype)):
        x.copy_(y)
    _native.tdp_fwd(*t, o, lse, 1.0 / D, True, *FULL)
    for x in g:
        x.fill_(float("nan"))
    for _ in range(20):
        graph.replay()
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    got = [x.clone() for x in g]
    want = _backward(t, do, 1.0 / D, True)
    for name, a, b in zip(NAMES, got, want):
        assert float((a.float() - b.float()).norm()) <= 2e-3 * float(b.float().norm()), name


@pytest.mark.gpu
@pytest.mark.parametrize("T,D,dtype", [(150, 64, torch.float16), (1100, 64, torch.bfloat16), (333, 128, torch.bfloat16)])
def test_calls_in_turn_on_the_same_buffers(T, D, dtype):
    """Two sets of inputs that take turns in the same tensors and workspace, back to back: every call sees its own inputs
    and its own preparation, although its kernels overlap (small scores, then large ones: the other operand as well)."""
    sets = [[x.to(DEV) for x in orc.make_inputs(1, 4, T, D, scale=sc, seed=T + i, dtype=dtype)] for i, sc in ((0, 0.5), (1, 1.0))]
    want, saved = [], []
    for x in sets:
        o, lse = torch.empty_like(x[0]), torch.empty(1, 4, T, device=DEV)
        _native.tdp_fwd(*x[:5], o, lse, 1 / 8, True, *FULL)
        saved.append((o, lse))
        want.append(_backward(x[:5], x[5], 1 / 8, True))
    t = [torch.empty_like(x) for x in sets[0]]
    o, lse = torch.empty_like(t[0]), torch.empty(1, 4, T, device=DEV)
    ws = _native.workspace(_native.OP_TDP_BWD, 1, 4, T, D, _native.dtype_code(dtype), o.device)
    results = []
    for i in range(40):
        for dst, src in zip(t + [o, lse], sets[i & 1] + list(saved[i & 1])):
            dst.copy_(src)
        g = [torch.empty_like(o) for _ in range(5)]
        _native.tdp_bwd(*t[:5], o, t[5], lse, *g, 1 / 8, True, *FULL, ws=ws)
        results.append(g)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    for i, g in enumerate(results):
        for name, a, b in zip(NAMES, g, want[i & 1]):
            assert float((a.float() - b.float()).norm()) <= 2e-3 * float(b.float().norm()), (i, name)


@pytest.mark.gpu
@pytest.mark.parametrize("D,dtype,scale", [(64, torch.bfloat16, 16.0), (128, torch.bfloat16, 24.0), (128, torch.float16, 24.0),
                                           (64, torch.float32, 24.0)])
@pytest.mark.parametrize("T", [8, 300])
def test_scores_past_the_exponents_range_stay_finite(T, D, dtype, scale):
    """Scores of order 1e5 to 1e6, which rounding moves by hundreds: the exponential of an exact score less the
    log-sum-exp of rounded ones overflows.  All gradients are finite, and dV2 is what probabilities can give."""
    g = torch.Generator().manual_seed(T + D)
    t = [torch.randn(1, 8, T, D, generator=g) for _ in range(6)]
    t = [(x * scale if i < 3 else x).to(dtype).to(DEV) for i, x in enumerate(t)]
    do = t.pop()
    got = _backward(t, do, 1.0, True)
    for name, x in zip(NAMES, got):
        assert torch.isfinite(x).all(), f"{name}: {int((~torch.isfinite(x)).sum())} of {x.numel()} values are not finite"
    # every P is at most 1 but for the fp32 rounding of a score in its exponent (1e6 * 2^-24 * a few: less than 1 in log2)
    silu = torch.nn.functional.silu(t[3].float()).abs().amax()
    bound = 2 * silu * do.float().abs().sum(2, keepdim=True)
    assert (got[4].float().abs() <= bound).all()


@pytest.mark.gpu
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (128, torch.float16)])
@pytest.mark.parametrize("T", [17, 18, 19, 20, 21, 131])
def test_rows_of_a_short_last_batch(T, D, dtype):
    """An item's K2 / V2 rows come in batches of four; the last batch copies what is left of the item, and the sequence's
    last row is the tensor's end."""
    t = orc.make_inputs(1, 2, T, D, scale=0.5, seed=T, dtype=dtype)
    got = _backward([x.to(DEV) for x in t[:5]], t[5].to(DEV), 1.0 / D, True)
    ref = orc.tdp_backward(*[x.float() for x in t], 1.0 / D, True)
    for name, a, b in zip(NAMES, got, ref):
        assert_close(name, a, b, dtype)


# j-tiles of 128 (head dimension 64) or 64 rows that overlap: the widest stride (no band at all), strides that leave a short last
# tile, a band to one side, the narrowest stride taken and the first one that is not, windows narrower than the band and than a tile.
BANDS = [(64, (70, 70, 0, 0)), (64, (200, 150, 32, 32)), (64, (40, 300, 1, 100)), (64, (300, 30, 90, 30)), (64, (120, 90, 60, 61)),
         (64, (3, 9, 2, 5)), (128, (70, 70, 0, 0)), (128, (150, 130, 16, 16)), (128, (40, 300, 0, 40)), (128, (90, 300, 28, 28))]


def _cells_side_by_side(T, D, windows):
    """Cells of the tiles that do not overlap."""
    k1w, k2w, kkl, kkr = windows
    JT, n = 128 if D == 64 else 64, 0
    for qa in range(0, T, 128):
        qb = min(qa + 127, T - 1)
        for ja in range(max(0, qa - k1w) // JT * JT, qb + 1, JT):
            n += max(0, min(qb, ja + JT - 1 + kkl) - max(0, qa - k2w, ja - kkr) + 1)
    return n * 128 * JT


def test_overlapping_tiles_are_taken_where_they_execute_less():
    for D, windows in BANDS:
        cells, stride = _native.tdp_bwd_plan(2000, D, _native.BF16, True, *windows)[1], (128 if D == 64 else 64) - sum(windows[2:])
        side_by_side = _cells_side_by_side(2000, D, windows)
        assert (cells < side_by_side) if sum(windows[2:]) and stride >= 8 else (cells == side_by_side), (D, windows)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,scale", [(torch.float16, 0.5), (torch.bfloat16, 1.0)])
@pytest.mark.parametrize("T", [127, 258, 391])
@pytest.mark.parametrize("D,windows", BANDS)
def test_overlapping_tiles(D, windows, T, dtype, scale):
    t = orc.make_inputs(1, 2, T, D, scale=scale, seed=T + D, dtype=dtype)
    alpha = 1.0 / D if scale < 1 else 1 / 8
    got = _backward([x.to(DEV) for x in t[:5]], t[5].to(DEV), alpha, True, windows)
    ref = orc.tdp_backward(*[x.float() for x in t], alpha, True, *windows, device=DEV)
    for name, a, b in zip(NAMES, got, ref):
        assert_close(name, a, b, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("D,windows", [(64, (128, 128, 30, 30)), (64, (60, 300, 0, 9)), (128, (128, 128, 16, 8)), (128, (30, 70, 0, 20))])
@pytest.mark.parametrize("which", ["do", "q", "k1", "v1"])
def test_a_row_that_is_not_finite_stays_in_its_tile_of_overlapping_ones(which, D, windows):
    """The products of a tile of 128 queries see an infinite row (0 * inf) where tiles side by side would: query 100 keys below 128
    alone, key 140 queries from 128 on alone, which the j-tiles overlap to both sides."""
    T, dtype = 391, torch.bfloat16
    t = [x.to(DEV) for x in orc.make_inputs(1, 2, T, D, scale=1.0, seed=D, dtype=dtype)]   # (scores too large for steps over diagonals)
    bad = [x.clone() for x in t]
    row = 100 if which in ("do", "q") else 140
    bad[{"q": 0, "k1": 1, "v1": 3, "do": 5}[which]][:, :, row] = float("inf")
    o, lse = torch.empty_like(t[0]), torch.empty(1, 2, T, device=DEV)
    _native.tdp_fwd(*t[:5], o, lse, 1 / 8, True, *windows)
    got, want = [torch.empty_like(o) for _ in range(5)], [torch.empty_like(o) for _ in range(5)]
    for x, g in ((bad, got), (t, want)):
        _native.tdp_bwd(*x[:5], o, x[5], lse, *g, 1 / 8, True, *windows)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    for name, a, b in zip(NAMES, got, want):
        if row == 100:
            a, b = (x[:, :, 128:].float() for x in (a, b))
        elif name == "dq":
            a, b = (x[:, :, :128].float() for x in (a, b))
        else:
            continue   # (the keys' sums meet the row's own queries)
        assert torch.isfinite(a).all(), f"{name}: {int((~torch.isfinite(a)).sum())} of {a.numel()} values are not finite"
        # (two runs of the same sums: their order, and bf16's rounding)
        assert float((a - b).norm()) <= 8e-3 * float(b.norm()), name
