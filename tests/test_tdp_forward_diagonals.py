"""The forward of narrow bands by the kernel that steps over the band's diagonals: tile edges, cut query tiles, and whom it serves."""
import pytest
import torch

from _parity import assert_close
from oracle import trittention_oracle as orc
from flash_trittention import _native

DEV = "cuda:0"


def _forward(t, alpha, windows, ws=None):
    B, N, T, _ = t[0].shape
    o, lse = torch.full_like(t[0], float("nan")), torch.full((B, N, T), float("nan"), device=DEV)
    before = _native.lib().tritt_kernel_launches()
    _native.tdp_fwd(*t, o, lse, alpha, True, *windows, ws=ws)
    _forward.launched = _native.lib().tritt_kernel_launches() - before   # 3 (preparation, this kernel, the band kernel) where it is asked
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0, "a bounded barrier wait ran out"
    return o, lse


def _workspace_without_it(t):
    """Room for SiLU(V1) and three statistics a head: the call runs on the kernel of four queries by 32 rows."""
    B, N, T, D = t[0].shape
    return torch.empty((B * N * T * D * 2 + 255) // 256 * 256 + 3 * B * N * 4, dtype=torch.uint8, device=DEV)


def _inputs(heads, T, scale, dtype, seed):
    return [x.to(DEV) for x in orc.make_inputs(1, heads, T, 64, scale=scale, seed=seed, dtype=dtype)[:5]]


# The widest band and windows, the narrowest, bands to one side, and either window as the one that bounds the reach to 128; heads: enough
# for the call to be asked of this kernel (a narrow window needs more), which also cuts query tiles between CTAs.
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [129, 255, 256, 257, 400])
@pytest.mark.parametrize("windows,heads", [((128, 128, 48, 48), 60), ((128, 128, 96, 0), 60), ((128, 400, 0, 96), 60), ((300, 100, 28, 9), 60),
                                           ((1, 1, 1, 1), 120), ((0, 9, 2, 5), 120)])
def test_against_the_oracle(windows, heads, T, dtype):
    t = _inputs(heads, T, 0.5, dtype, T + heads)
    o, lse = _forward(t, 1 / 64, windows)
    assert _forward.launched == (2 if T == 129 and sum(windows[2:]) == 96 else 3)   # (97 diagonals of a tile of one query cost more)
    ref_o, ref_lse = orc.tdp_forward(*[x.float() for x in t], 1 / 64, True, *windows, device=DEV)
    assert_close("o", o, ref_o, dtype)
    # scores of order 0.1, operands of 8 or 11 bits: the log of a sum of exponentials moves by less than 2^-9 of the largest score
    assert float((lse - ref_lse).abs().max()) <= 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("windows,heads,T", [((128, 128, 32, 32), 16, 1024), ((128, 128, 32, 32), 17, 1000), ((20, 20, 4, 4), 600, 140),
                                             ((128, 128, 48, 48), 6, 2600)])
def test_long_calls_add_up_their_pieces_in_the_kernel(windows, heads, T, dtype):
    """From 128 tiles of the band kernel on (a CTA) the warp that brings the last piece of a tile adds them up, in the pieces' order:
    the same bits each time, beside calls of other inputs in the same workspace."""
    t, u = _inputs(heads, T, 0.5, dtype, T), _inputs(heads, T, 0.4, dtype, T + 1)
    o, lse = _forward(t, 1 / 64, windows)
    assert _forward.launched == 3
    ref_o, ref_lse = orc.tdp_forward(*[x.float() for x in t], 1 / 64, True, *windows, device=DEV)
    assert_close("o", o, ref_o, dtype)
    assert float((lse - ref_lse).abs().max()) <= 2e-3   # (as above)
    ws = _native.workspace(_native.OP_TDP_FWD, 1, heads, T, 64, _native.dtype_code(dtype), o.device)
    for _ in range(5):
        _forward(u, 1 / 64, windows, ws)
        again = _forward(t, 1 / 64, windows, ws)
        assert torch.equal(again[0], o) and torch.equal(again[1], lse)
    t[0][0, heads - 1] *= 400   # large scores: the band kernel, bit for bit
    a, b = _forward(t, 1 / 64, windows, ws), _forward(t, 1 / 64, windows, _workspace_without_it(t))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


@pytest.mark.gpu
@pytest.mark.parametrize("windows,heads,T,asked", [((128, 128, 32, 32), 8, 1000, True), ((27, 22, 11, 38), 32, 768, False), ((1, 2, 47, 10), 8, 2052, False),
                                                   ((4, 27, 35, 4), 32, 1265, True), ((60, 60, 30, 30), 4, 1000, False),
                                                   ((20, 20, 40, 40), 16, 1000, False), ((128, 128, 48, 48), 22, 129, False), ((1, 1, 0, 0), 32, 300, False), ((99, 18, 24, 19), 64, 747, True)])
def test_asked_where_its_steps_cost_less_than_the_other_kernels_tiles(windows, heads, T, asked):
    """Narrow windows leave the band kernel one tile for four queries, and a wide band this one many diagonals (89 us for 59), a second tile of
    one query doubles them (57 for 36), and a single diagonal is an item of one step (42 for 38)."""
    _forward(_inputs(heads, T, 0.5, torch.float16, 1), 1 / 64, windows)
    assert _forward.launched == (3 if asked else 2)


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [1, -1])
def test_fp16_scores_near_their_bound(sign):
    """Queries, K1 and K2 rows that are all alike: every score is within a binade of the bound (8 to 13 in log2 units) or of its
    negative, where P is 2^-12 at the reference that the bound gives."""
    windows, heads, T = (128, 128, 32, 32), 16, 300
    t = _inputs(heads, T, 0.1, torch.float16, 7)
    for x in t[:3]:
        x += 1
    t[0] *= sign
    alpha = 8.5 / 64 / 1.4427
    a, b = _forward(t, alpha, windows), _forward(t, alpha, windows, _workspace_without_it(t))
    assert not torch.equal(a[0], b[0])
    ref_o, ref_lse = orc.tdp_forward(*[x.float() for x in t], alpha, True, *windows, device=DEV)
    assert_close("o", a[0], ref_o, torch.float16)
    # operands of 11 bits: a score of 13 (9 in natural units) moves by 9 * 2^-11 at most
    assert float((a[1] - ref_lse).abs().max()) <= 5e-3


def _bound(t):
    """|Q row| |K1 row| max|K2|, the factor of alpha in the bound on a head's scores, of the head that has the largest."""
    q, k1, k2 = (x[0].float() for x in t[:3])
    return float((q.norm(dim=-1).amax(-1) * k1.norm(dim=-1).amax(-1) * k2.abs().amax((1, 2))).max())


@pytest.mark.gpu
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("dtype,limit", [(torch.bfloat16, 16), (torch.float16, 13.5)])
def test_scores_just_within_the_bound_and_just_beyond(dtype, limit, sign):
    """Rows that are all alike, and an alpha that puts the bound one part in a thousand below the limit, or above it."""
    windows, heads, T = (128, 128, 32, 32), 16, 300
    t = _inputs(heads, T, 0.1, dtype, 8)
    for x in t[:3]:
        x += 1
    t[0] *= sign
    for factor in (0.999, 1.001):
        alpha = factor * limit / _bound(t) / 1.4426950408889634
        a, b = _forward(t, alpha, windows), _forward(t, alpha, windows, _workspace_without_it(t))
        assert torch.equal(a[0], b[0]) == (factor > 1)
        ref_o, ref_lse = orc.tdp_forward(*[x.float() for x in t], alpha, True, *windows, device=DEV)
        assert_close("o", a[0], ref_o, dtype)
        # a score of 11 (9 in fp16) in natural units moves by its operands' rounding, 2^-9 (2^-12) of it, twice
        assert float((a[1] - ref_lse).abs().max()) <= (0.045 if dtype == torch.bfloat16 else 5e-3)


@pytest.mark.gpu
@pytest.mark.parametrize("T", [300, 1024])
def test_fp32_tensors(T):
    """Through their fp16 copies: the conversions to and from, the preparation and the two kernels."""
    windows, heads = (128, 128, 32, 32), 16
    t = _inputs(heads, T, 0.5, torch.float32, T)
    o, lse = _forward(t, 1 / 64, windows)
    assert _forward.launched == 5
    ref_o, ref_lse = orc.tdp_forward(*t, 1 / 64, True, *windows, device=DEV)
    assert_close("o", o, ref_o, torch.float16)   # (the operands' and the output's type)
    assert float((lse - ref_lse).abs().max()) <= 2e-3


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_large_scores_of_one_head_are_left_to_the_other_kernel(dtype):
    """Small scores: this kernel, whose roundings are others.  One head with large ones, or not finite: the whole call is the
    other kernel's, bit for bit."""
    windows, heads, T = (100, 128, 20, 30), 16, 300
    t = _inputs(heads, T, 0.5, dtype, 1)
    a, b = _forward(t, 1 / 64, windows), _forward(t, 1 / 64, windows, _workspace_without_it(t))
    assert not torch.equal(a[0], b[0])
    assert float((a[0].float() - b[0].float()).norm()) <= (2e-3 if dtype == torch.float16 else 1e-2) * float(b[0].float().norm())
    for value in (60.0, float("inf")):
        t[0][0, heads - 1, T - 1, 5] = value
        t[1][0, heads - 1, 7, 5] = 50.0
        a, b = _forward(t, 1 / 8, windows), _forward(t, 1 / 8, windows, _workspace_without_it(t))
        assert torch.equal(a[0].nan_to_num(1e4), b[0].nan_to_num(1e4)) and torch.equal(a[1].nan_to_num(1e4), b[1].nan_to_num(1e4))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_values_that_are_not_finite_reach_no_more_queries(value, dtype):
    """Small scores but for one element, of any of the five tensors: the whole call is the other kernel's, bit for bit, and with it the
    queries that 0 * inf reaches: tiles of four queries by 32 rows, where the products of this one would reach 256 queries."""
    windows, heads, T = (100, 128, 20, 30), 16, 300
    for which in range(5):
        t = _inputs(heads, T, 0.5, dtype, 1)
        t[which][0, heads - 1, 200, 63] = value
        a, b = _forward(t, 1 / 64, windows), _forward(t, 1 / 64, windows, _workspace_without_it(t))
        for x, y in zip(a, b):
            assert torch.equal(x.isnan(), y.isnan()) and torch.equal(x.nan_to_num(1e4), y.nan_to_num(1e4)), which
        assert a[0][0, :-1].isfinite().all() and a[0][0, -1, :64].isfinite().all(), which


@pytest.mark.gpu
def test_captured_call_replays_for_new_inputs():
    windows, heads, T = (128, 128, 32, 32), 16, 700
    t = _inputs(heads, T, 0.5, torch.float16, 2)
    o, lse = torch.empty_like(t[0]), torch.empty(1, heads, T, device=DEV)
    ws = _native.workspace(_native.OP_TDP_FWD, 1, heads, T, 64, _native.F16, t[0].device)
    call = lambda: _native.tdp_fwd(*t, o, lse, 1 / 64, True, *windows, ws=ws)
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for scale, alpha_seed in ((0.5, 3), (0.4, 4)):
        for x, y in zip(t, _inputs(heads, T, scale, torch.float16, alpha_seed)):
            x.copy_(y)
        for _ in range(3):
            graph.replay()
        torch.cuda.synchronize()
        want = _forward(t, 1 / 64, windows)
        assert torch.equal(o, want[0]) and torch.equal(lse, want[1])
