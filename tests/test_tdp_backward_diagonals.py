"""The backward of narrow bands by the kernel that steps over the band's diagonals: tile edges, cut items, and whom it serves."""
import pytest
import torch

from _parity import assert_close
from oracle import trittention_oracle as orc
from flash_trittention import _native

DEV = "cuda:0"
NAMES = ("dq", "dk1", "dk2", "dv1", "dv2")


def _backward(t, do, alpha, windows):
    """The gradients, and the kernels that a backward launched."""
    B, N, T, _ = t[0].shape
    o, lse = torch.empty_like(t[0]), torch.empty(B, N, T, device=DEV)
    _native.tdp_fwd(*t, o, lse, alpha, True, *windows)
    g = [torch.full_like(t[0], float("nan")) for _ in range(5)]
    before = _native.lib().tritt_kernel_launches()
    _native.tdp_bwd(*t, o, do, lse, *g, alpha, True, *windows)
    launched = _native.lib().tritt_kernel_launches() - before
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0, "a bounded barrier wait ran out"
    return g, launched


def _inputs(heads, T, dtype, seed, scale=0.5):
    t = [x.to(DEV) for x in orc.make_inputs(1, heads, T, 64, scale=scale, seed=seed, dtype=dtype)]
    return t[:5], t[5]


# The widest bands (to both sides, to one) and none, windows below, at and beyond a tile, either window as the one that bounds the
# reach, no windows.  Heads: enough for the kernel to be asked, which also cuts items between CTAs.  The last one launches a
# kernel less (its windows leave the first queries no path of their own).
CASES = [((128, 128, 36, 36), 100, 0), ((None, None, 72, 0), 100, 0), ((128, 400, 0, 72), 100, 0), ((300, 40, 28, 9), 60, 0),
         ((None, None, 0, 0), 40, 0), ((257, 257, 5, 60), 60, 0), ((9, 3, 2, 5), 120, 1)]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T", [200, 256, 257, 391])
@pytest.mark.parametrize("windows,heads,fewer", CASES)
def test_against_the_oracle(windows, heads, fewer, T, dtype):
    t, do = _inputs(heads, T, dtype, T + heads)
    got, launched = _backward(t, do, 1 / 64, windows)
    first = 0 if fewer and 8 * 10 * 4 <= T else 1
    assert launched == 4 + first   # preparation, first queries, this kernel, the other one, the outputs
    ref = orc.tdp_backward(*[x.float() for x in t], do.float(), 1 / 64, True, *windows, device=DEV)
    for name, a, b in zip(NAMES, got, ref):
        assert_close(name, a, b, dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_large_scores_of_one_head_are_left_to_the_other_kernel(dtype):
    windows, heads, T = (100, 128, 20, 30), 40, 300
    t, do = _inputs(heads, T, dtype, 1)
    # (scores of order 1, the bound on them 9 times the others': 50.  Far larger ones test the operands: R of 11 bits moves a score of
    # 50 by up to 50 * 2^-12 = 0.012, and P with it.)
    t[0][0, heads - 1] *= 3
    t[1][0, heads - 1] *= 3
    got, launched = _backward(t, do, 1 / 8, windows)
    assert launched == 5
    ref = orc.tdp_backward(*[x.float() for x in t], do.float(), 1 / 8, True, *windows, device=DEV)
    for name, a, b in zip(NAMES, got, ref):
        assert_close(name, a[:, :-1], b[:, :-1], dtype)
        assert_close(name, a[:, -1:], b[:, -1:], dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("heads,T", [(40, 300), (200, 140), (5, 1500)])
def test_heads_of_both_kinds(heads, T, dtype):
    """Each head is the one kernel's or the other's: CTAs whose part has heads of one kind or of both, one or many of them."""
    windows = (100, 128, 20, 30)
    t, do = _inputs(heads, T, dtype, 6)
    large, bad = [h for h in range(heads) if h % 7 in (1, 2) or h > heads - 3], heads // 2
    for h in large:
        t[0][0, h] *= 3
        t[1][0, h] *= 3
    t[4][0, bad, T - 1, 3] = float("inf")   # (which reaches the last queries; all other heads are the oracle's)
    got, launched = _backward(t, do, 1 / 8, windows)
    assert launched == 5
    ref = orc.tdp_backward(*[x.float() for x in t], do.float(), 1 / 8, True, *windows, device=DEV)
    for name, a, b in zip(NAMES, got, ref):
        for h in [h for h in range(heads) if h != bad]:
            assert_close(f"{name} of head {h}", a[:, h], b[:, h], dtype)


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_a_query_that_is_not_finite_stays_in_its_tile(value):
    """An infinite or NaN upstream row of query 0: the products of its tile of 128 queries and keys see it (0 * inf), no other row."""
    windows = (128, 128, 30, 30)
    t, do = _inputs(40, 391, torch.float16, 3)
    bad, zero = do.clone(), do.clone()
    bad[:, :, 0], zero[:, :, 0] = value, 0
    (got, launched), (want, _) = _backward(t, bad, 1 / 64, windows), _backward(t, zero, 1 / 64, windows)
    assert launched == 5
    for name, a, b in zip(NAMES, got, want):
        a, b = (x[:, :, 1 if name == "dq" else 128:].float() for x in (a, b))
        assert torch.isfinite(a).all(), name
        # (two runs of the same sums: the order of the fp32 reduce-adds, and where it meets the final rounding)
        assert float((a - b).norm()) <= 1e-3 * float(b.norm()), name


@pytest.mark.gpu
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("which", ["k1", "k2", "v1", "v2"])
def test_a_key_that_is_not_finite_reaches_no_query_of_the_tile_before(which, value):
    """Key 130, which diagonals would pair with rows j of the tile of queries below 128.  (The forward's results are those of finite keys:
    what the backward adds is looked at.)"""
    windows = (128, 128, 30, 30)
    t, do = _inputs(40, 391, torch.float16, 4)
    B, N, T, _ = t[0].shape
    o, lse = torch.empty_like(t[0]), torch.empty(B, N, T, device=DEV)
    _native.tdp_fwd(*t, o, lse, 1 / 64, True, *windows)
    bad = [x.clone() for x in t]
    bad[{"k1": 1, "k2": 2, "v1": 3, "v2": 4}[which]][:, :, 130] = value
    got, want = [torch.empty_like(o) for _ in range(5)], [torch.empty_like(o) for _ in range(5)]
    for x, g in ((bad, got), (t, want)):
        _native.tdp_bwd(*x, o, do, lse, *g, 1 / 64, True, *windows)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    a, b = got[0][:, :, :128].float(), want[0][:, :, :128].float()
    assert torch.isfinite(a).all(), f"{int((~torch.isfinite(a)).sum())} of {a.numel()} values of dQ are not finite"
    # (other kernels, whose errors against the oracle are up to 5e-3 each)
    assert float((a - b).norm()) <= 1e-2 * float(b.norm())


@pytest.mark.gpu
def test_fp32_tensors():
    """Through their fp16 copies: dO's largest element, the copies, and what a 16-bit call launches."""
    windows = (128, 128, 36, 36)
    t, do = _inputs(60, 391, torch.float32, 7)
    got, launched = _backward(t, do, 1 / 64, windows)
    assert launched == 7
    ref = orc.tdp_backward(*t, do, 1 / 64, True, *windows, device=DEV)
    for name, a, b in zip(NAMES, got, ref):
        assert_close(name, a, b, torch.float16)


@pytest.mark.gpu
def test_capture():
    windows = (128, 128, 36, 36)
    t, do = _inputs(60, 391, torch.bfloat16, 5)
    want, _ = _backward(t, do, 1 / 64, windows)
    B, N, T, _ = t[0].shape
    o, lse, g = torch.empty_like(t[0]), torch.empty(B, N, T, device=DEV), [torch.empty_like(t[0]) for _ in range(5)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        _native.tdp_fwd(*t, o, lse, 1 / 64, True, *windows)
        _native.tdp_bwd(*t, o, do, lse, *g, 1 / 64, True, *windows)
    for _ in range(2):
        graph.replay()
    torch.cuda.synchronize()
    for a, b in zip(g, want):
        assert float((a.float() - b.float()).norm()) <= 8e-3 * float(b.float().norm())   # (sums in another order, then bf16's rounding)
