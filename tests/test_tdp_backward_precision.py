"""How exact the tensor-core triple-dot-product backward is against fp64.

The yardstick is what the kernel's precision class gives: 16-bit operands, fp32 sums, with the row products formed per
query as the forward forms them (Q K2 and dO V2 for dQ, dK2, dV2; Q K1 and dO SiLU(V1) for dK1, dV1), P and dS rounded to
16 bits.  It is computed here beside the fp64 result; the kernel may not be further from fp64 than it, up to the spread
between the roundings of two formations of one sum (the error of a norm over n rounded values spreads by about 1 / sqrt(n)
and is small here, but the first queries carry most of a causal gradient: 8 % covers the seeds tried)."""
import math

import pytest
import torch

from oracle import trittention_oracle as orc
from flash_trittention import _native

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NAMES = ("dq", "dk1", "dk2", "dv1", "dv2")
LOG2E = 1.4426950408889634
SPREAD = 1.08


def _mask(T, causal, windows):
    q, j, k = (torch.arange(T, device=DEV).view(s) for s in ((-1, 1, 1), (1, 1, -1), (1, -1, 1)))   # [q, k, j]
    if not causal:
        return torch.ones(T, T, T, dtype=torch.bool, device=DEV)
    w1, w2, kl, kr = (T if w is None else w for w in windows)
    return (j <= q) & (q - j <= w1) & (k <= q) & (q - k <= w2) & (k - j <= kl) & (j - k <= kr)


def _exact(x, do, alpha, ok):
    """Dense fp64, one head: the five gradients."""
    q, k1, k2, v1, v2 = (t.double() for t in x)
    do, sig = do.double(), torch.sigmoid(v1)
    s1 = v1 * sig
    A = alpha * q[:, None] * k2
    P = torch.where(ok, A @ k1.T, -torch.inf).flatten(1).softmax(1).view(ok.shape)
    U = P @ s1
    O = (U * v2).sum(1)
    A2 = do[:, None] * v2
    dS = P * (A2 @ s1.T - (do * O).sum(1)[:, None, None])
    G = alpha * dS @ k1
    return [(G * k2).sum(1), torch.einsum("qkj,qkh->jh", dS, A), (G * q[:, None]).sum(0),
            torch.einsum("qkj,qkh->jh", P, A2) * (sig + s1 * (1 - sig)), (U * do[:, None]).sum(0)]


def _rounded(x, do, o, lse, alpha, ok):
    """The same with the precision class's roundings, from the forward's output and log-sum-exp.  fp32 tensors run on fp16
    copies, dO times the power of two that brings its largest value to (0.5, 1]."""
    out_t, dt = x[0].dtype, torch.float16 if x[0].dtype == torch.float32 else x[0].dtype
    scale = 2.0 ** -math.frexp(float(do.abs().max()))[1] if out_t == torch.float32 else 1.0
    do, o = (do.float() * scale).to(dt), o.to(dt)
    rd = lambda t: t.to(dt).float()
    q, k1, k2, v1, v2 = (rd(t) for t in x)
    do = do.float()
    sig = torch.sigmoid(v1)
    s1 = rd(v1 * sig)
    Dq = (do * o.float()).sum(1)[:, None, None]
    single = ok.flatten(1).sum(1).view(-1, 1, 1) == 1
    # (P and dS take a power of two in fp16: probabilities below its normal range keep their bits)
    sh = torch.exp2(ok.flatten(1).sum(1).float().log2().floor().clamp(max=10)).view(-1, 1, 1) if dt == torch.float16 else 1.0
    out = {}
    for row, col, yr, yc, m in ((k2, k1, v2, s1, ok), (k1, k2, s1, v2, ok.transpose(1, 2))):
        S = rd(q[:, None] * (alpha * LOG2E) * row) @ col.T
        P = torch.where(m, torch.exp2(S - lse[:, None, None] * LOG2E), 0.0) * sh
        P = rd(P)
        dS = torch.where(single, 0.0, rd(P * (rd(do[:, None] * yr) @ yc.T - Dq))) / sh
        G, U = alpha * (dS @ col), (P / sh) @ yc
        out[row is k1] = [(G * row).sum(1), (G * q[:, None]).sum(0), (U * do[:, None]).sum(0)]
    return [(t / scale).to(out_t) for t in (out[0][0], out[1][1], out[0][1], out[1][2] * (sig + v1 * sig * (1 - sig)), out[0][2])]


def _errors(T, D, dtype, unit, causal, windows, names=NAMES, seeds=(0, 1), std=(1, 1, 1, 1), columns=None, heads=3,
            head_scale=None):
    """Relative rms errors against fp64, kernel over yardstick, over a few heads and seeds.  std: Q, the keys, the values
    and dO times this.  columns [D], head_scale [heads]: Q and K1 times this."""
    alpha = 1 / 8 if unit else 1.0 / D
    got, bound = torch.zeros(5), torch.zeros(5)
    ok = _mask(T, causal, windows)
    for seed in seeds:
        x = [t.to(DEV) for t in orc.make_inputs(1, heads, T, D, scale=1.0 if unit else 0.5, seed=100 * seed + T + D)]
        for t in x[:2]:
            t *= 1 if columns is None else columns.to(DEV)
            t *= 1 if head_scale is None else head_scale.view(1, -1, 1, 1).to(DEV)
        x = [(t * std[i]).to(dtype) for t, i in zip(x, (0, 1, 1, 2, 2, 3))]
        do = x.pop()
        o, lse = torch.empty_like(do), torch.empty(1, heads, T, device=DEV)
        _native.tdp_fwd(*x, o, lse, alpha, causal, *windows)
        g = [torch.empty_like(do) for _ in range(5)]
        _native.tdp_bwd(*x, o, do, lse, *g, alpha, causal, *windows)
        torch.cuda.synchronize()
        assert _native.read_status(torch.device(DEV)) == 0
        for h in range(heads):
            xh = [t[0, h] for t in x]
            e = _exact(xh, do[0, h], alpha, ok)
            r = _rounded(xh, do[0, h], o[0, h], lse[0, h], alpha, ok)
            for i in range(5):
                got[i] += float((g[i][0, h].double() - e[i]).norm() / e[i].norm())
                bound[i] += float((r[i].double() - e[i]).norm() / e[i].norm())
    return [(n, float(a / b)) for n, a, b in zip(NAMES, got, bound) if n in names]


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,D", [(60, 64), (192, 64), (130, 128)])
def test_probabilities_of_the_first_queries_sum_to_one(T, D, dtype):
    """dV1 and dV2 are sums of P alone: where the recomputed P of a query with few pairs does not match the forward's
    log-sum-exp, they are off by the difference."""
    for name, ratio in _errors(T, D, dtype, True, True, (None,) * 4, names=("dv1", "dv2"), seeds=(0, 1, 2)):
        assert ratio <= SPREAD, f"{name}: error {ratio:.2f} times that of the precision class"


@pytest.mark.parametrize("T,windows", [(128, (None,) * 4), (300, (None,) * 4), (300, (100, 60, 50, 40))])
def test_small_score_gradients_keep_their_bits(T, windows):
    """fp32 tensors (fp16 operands, no final rounding), values of 0.01: dP is about 1e-3, times a probability of 1 / 16000
    at T = 128, against fp16's smallest normal value of 6e-5."""
    for name, ratio in _errors(T, 64, torch.float32, False, True, windows, names=("dk1", "dk2"), std=(1, 1, 0.02, 1)):
        assert ratio <= SPREAD, f"{name}: error {ratio:.2f} times that of the precision class"


@pytest.mark.parametrize("dtype,T,D", [(torch.float16, 192, 64), (torch.float16, 130, 128), (torch.float32, 192, 64)])
@pytest.mark.parametrize("keys,dout", [(0.02, 2048), (0.01, 2048), (200, 1 / 1024)])
def test_products_of_small_and_large_keys(dtype, T, D, keys, dout):
    """Keys of 0.01 and 0.005 under a loss scale of 1024: K1 K2 is far below fp16's smallest normal value.  Keys of 100 (Q of
    0.001, as such keys want it): K1 K2 reaches fp16's largest value."""
    ratios = _errors(T, D, dtype, False, True, (None,) * 4, std=(1 if keys < 1 else 2e-3, keys, 1, dout))
    assert all(r <= SPREAD for _, r in ratios), f"errors over those of the precision class: {ratios}"


@pytest.mark.parametrize("T,D", [(192, 64), (130, 128)])
@pytest.mark.parametrize("q,keys", [(30, 3e-4), (1, 1e-4), (30, 1e-4), (1e-3, 100)])
def test_products_of_keys_beside_queries_of_another_size(T, D, q, keys):
    """fp32 tensors (fp16 operands, no final rounding).  The range of K1 K2, which dQ is formed from, is that of the keys alone,
    whatever the queries are."""
    ratios = _errors(T, D, torch.float32, False, True, (None,) * 4, std=(2 * q, 2 * keys, 1, 1))
    assert all(r <= SPREAD for _, r in ratios), f"errors over those of the precision class: {ratios}"


@pytest.mark.parametrize("D,q,keys", [(64, 1, 1), (64, 1e-3, 400), (128, 1e-3, 600)])
def test_a_workspace_without_the_statistics_is_accepted(D, q, keys):
    """... and is as good for inputs of ordinary size, and for keys of 200 and 300, whose products are beyond fp16's range but
    not those with alpha."""
    T = 200
    x = orc.make_inputs(1, 2, T, D, scale=0.5, seed=5)
    x = [(t * s).to(DEV, torch.float16) for t, s in zip(x, (q, keys, keys, 1, 1, 1))]
    do = x.pop()
    o, lse = torch.empty_like(do), torch.empty(1, 2, T, device=DEV)
    _native.tdp_fwd(*x, o, lse, 1 / D, True, None, None, None, None)
    n, full = do.numel(), _native.workspace(_native.OP_TDP_BWD, 1, 2, T, D, _native.F16, DEV)
    out = []
    for ws in (full, full[: 22 * n + 4 * 2 * T]):
        out.append([torch.empty_like(do) for _ in range(5)])
        _native.tdp_bwd(*x, o, do, lse, *out[-1], 1 / D, True, None, None, None, None, ws=ws)
    with pytest.raises(ValueError, match="workspace"):
        _native.tdp_bwd(*x, o, do, lse, *out[-1], 1 / D, True, None, None, None, None, ws=full[: 22 * n])
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    for name, a, b in zip(NAMES, *out):
        assert float((a.float() - b.float()).norm()) <= 2e-3 * float(b.float().norm()), name


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("unit", [True, False])
@pytest.mark.parametrize("T,D,causal,windows", [
    (192, 64, True, (None,) * 4), (330, 128, True, (None,) * 4), (300, 64, False, (None,) * 4), (200, 128, False, (None,) * 4),
    (400, 64, True, (128, 128, 32, 32)), (350, 128, True, (40, 100, 20, 9)), (350, 64, True, (9, 5, 3, 2)),
    (480, 64, True, (9, 5, 3, 2)), (150, 128, True, (3, 2, 1, 2)), (200, 64, True, (0, 24, 24, 24))])
def test_errors_are_those_of_the_precision_class(T, D, causal, windows, dtype, unit):
    """All five gradients, scores of order 1 to 10 and of order 0.01."""
    ratios = _errors(T, D, dtype, unit, causal, windows)
    print(T, D, causal, windows, dtype, unit, " ".join(f"{n} {r:.2f}" for n, r in ratios))
    assert all(r <= SPREAD for _, r in ratios), f"errors over those of the precision class: {ratios}"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("half", [0, 1])
def test_scores_that_few_pairs_carry(half, D, dtype):
    """Scores of order 3, from one half of the columns: P has to match the forward's log-sum-exp."""
    columns = torch.full((D,), 0.05)
    columns[half * D // 2:(half + 1) * D // 2] = 1.6
    ratios = _errors(200, D, dtype, True, False, (None,) * 4, columns=columns)
    print(half, D, dtype, " ".join(f"{n} {r:.2f}" for n, r in ratios))
    assert all(r <= SPREAD for _, r in ratios), f"errors over those of the precision class: {ratios}"


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("T", [33, 70, 150])
def test_heads_with_small_and_large_scores_in_one_cta(T, D):
    """More heads than SMs, so that a CTA's part holds heads of both kinds; short, ragged lengths."""
    heads = 160
    ratios = _errors(T, D, torch.bfloat16, True, True, (None,) * 4, heads=heads, seeds=(0,),
                     head_scale=torch.tensor([0.1, 1.2, 1.2, 0.2] * (heads // 4)))
    print(T, D, " ".join(f"{n} {r:.2f}" for n, r in ratios))
    assert all(r <= SPREAD for _, r in ratios), f"errors over those of the precision class: {ratios}"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("T,D,windows", [(50, 64, (None,) * 4), (120, 128, (None,) * 4), (120, 128, (9, 5, 3, 2))])
def test_first_queries_with_large_scores(T, D, windows, dtype):
    """Scores of order 4 to 6: single pairs carry the first queries, in whichever kernel forms them."""
    ratios = _errors(T, D, dtype, True, True, windows, seeds=(0, 1, 2), std=(3, 1, 1, 1))
    print(T, D, dtype, windows, " ".join(f"{n} {r:.2f}" for n, r in ratios))
    assert all(r <= SPREAD for _, r in ratios), f"errors over those of the precision class: {ratios}"


@pytest.mark.parametrize("T", [2, 5, 12])
@pytest.mark.parametrize("D,dtype", [(64, torch.bfloat16), (128, torch.bfloat16), (64, torch.float16), (128, torch.float16)])
def test_few_queries_of_large_scores_are_exact(T, D, dtype):
    """Sequences that the exact first queries take alone, with scores of order 3 to 10, so that in most rows one pair has
    nearly all the mass and dP - Dq cancels.  Everything is formed in fp32, so the gradients of 16 heads together are as far
    from fp64 as rounding them to the 16-bit type may put them (u at most, 0.42 u in the mean; the fp32 sums need the rest)."""
    x = [t.to(DEV) for t in orc.make_inputs(1, 16, T, D, scale=1.5, seed=T + D, dtype=dtype)]
    do = x.pop()
    o, lse = torch.empty_like(do), torch.empty(1, 16, T, device=DEV)
    _native.tdp_fwd(*x, o, lse, 0.125, True, None, None, None, None)
    g = [torch.empty_like(do) for _ in range(5)]
    _native.tdp_bwd(*x, o, do, lse, *g, 0.125, True, None, None, None, None)
    ok = _mask(T, True, (None,) * 4)
    want = [torch.stack(t) for t in zip(*(_exact([t[0, h] for t in x], do[0, h], 0.125, ok) for h in range(16)))]
    u = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    for name, a, b in zip(NAMES, g, want):
        err = float((a[0].double() - b).norm() / b.norm())
        assert err <= u, f"{name}: {err:.2e} of the norm, more than {u:.1e}"
