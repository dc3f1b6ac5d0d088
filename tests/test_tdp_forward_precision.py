"""How exact the tensor-core triple-dot-product forward's output is against fp64.

The yardstick is what the kernel's precision class gives: the row products s Q K2 and SiLU(V1) rounded to 16 bits, P = exp2(S - m)
rounded to 16 bits with a reference m of each row's own (its score bound, or its maximum where that is large), fp32 sums, the
output rounded.  Where a few pairs carry the first queries, which are most of the output's norm, the reference decides on which part
of the 16-bit grid P lies: the yardstick's rows are spread over it.  The kernel may not be further from fp64 than it, up to the
spread of the two: the errors are those of about 1000 independent roundings (two queries of 512 heads), whose squares' sum has a
relative deviation of 0.9 / sqrt(1000) = 3 %, its root half of that, the ratio of two 2 %; SPREAD is twice that."""
import pytest
import torch

from flash_trittention import _native
from oracle import trittention_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
LOG2E = 1.4426950408889634
SPREAD = 1.04


def _forward(x, alpha, causal=True):
    o, lse = torch.empty_like(x[0]), torch.empty(x[0].shape[:3], device=DEV)
    _native.tdp_fwd(*x, o, lse, alpha, causal, None, None, None, None)
    torch.cuda.synchronize()
    assert _native.read_status(torch.device(DEV)) == 0
    return o[0]


def _references(x, alpha, causal):
    """fp64 and the yardstick, [heads, T, D], from [1, heads, T, D]; a few heads at a time."""
    exact, rounded = [], []
    dt, (heads, T) = x[0].dtype, x[0].shape[1:3]
    t = torch.arange(T, device=DEV)
    ok = ((t[None, :, None] <= t[:, None, None]) & (t[None, None, :] <= t[:, None, None])) if causal else torch.ones(T, T, T, device=DEV, dtype=torch.bool)
    limit = 40 if dt == torch.bfloat16 else 6
    for h in range(0, heads, 8):
        q, k1, k2, v1, v2 = (y[0, h:h + 8].double() for y in x)
        s1 = v1 * torch.sigmoid(v1)
        A = alpha * LOG2E * q[:, :, None] * k2[:, None]                           # [heads, q, k, h]
        S = torch.einsum("nqkh,njh->nqkj", A, k1).masked_fill(~ok, -torch.inf)
        P = torch.exp2(S - S.amax((2, 3), keepdim=True))
        exact.append(torch.einsum("nqkj,njh,nkh->nqh", P, s1, v2) / P.sum((2, 3))[..., None])
        rd = lambda y: y.to(dt).float()
        Af = rd(A.float())
        S = (Af @ k1.float().transpose(1, 2)[:, None]).masked_fill(~ok, -torch.inf)
        m = Af.norm(dim=3) * k1.float().norm(dim=2).amax(1)[:, None, None]
        m = torch.where(m <= limit, m, S.amax(3))[..., None]
        m = torch.where(m > -torch.inf, m, 0.0)
        w = torch.exp2(m - m.amax((2, 3), keepdim=True))
        P = torch.exp2(S - m)
        O = ((rd(P) @ rd(s1.float())[:, None]) * w * v2.float()[:, None]).sum(2) / (P * w).sum((2, 3))[..., None]
        rounded.append(rd(O).double())
    return torch.cat(exact), torch.cat(rounded)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T,D,scale,causal,kinds", [
    (24, 64, 0.5, True, (1.0,)), (24, 128, 0.5, True, (1.0,)), (33, 128, 0.5, False, (1.0,)), (24, 64, 0.02, True, (1.0,)),
    (24, 64, 0.5, True, (2.5,)), (24, 128, 0.5, True, (2.0,)),
    (40, 64, 0.5, True, (1.0, 4.0)), (40, 128, 0.5, True, (1.0, 1.0, 4.0))])
def test_the_output_is_as_exact_as_the_precision_class(T, D, scale, causal, kinds, dtype):
    """Small scores (of 0.01 to 0.3, in log2 units); heads with small and large scores (Q and the keys times 4: bounds of 80 and more) in one CTA."""
    heads = 512
    x = [t.to(DEV) for t in orc.make_inputs(1, heads, T, D, scale=scale, seed=T + D)[:5]]
    kind = torch.tensor([kinds[h % len(kinds)] for h in range(heads)], device=DEV)
    x = [(t * kind.view(1, -1, 1, 1) if i < 3 else t).to(dtype) for i, t in enumerate(x)]
    got = _forward(x, 1 / D, causal).double()
    exact, rounded = _references(x, 1 / D, causal)
    for s in set(kinds):
        e = exact[kind == s]
        ratio = float((got[kind == s] - e).norm() / (rounded[kind == s] - e).norm())
        print(T, D, dtype, scale, s, f"{float((got[kind == s] - e).norm() / e.norm()):.2e} {ratio:.3f}")
        assert ratio <= SPREAD, f"error {ratio:.3f} times that of the precision class (Q and keys times {s})"


@pytest.mark.parametrize("D", [64, 128])
def test_small_values_are_not_lost(D):
    """bf16 values of 1e-13: P SiLU(V1) V2 is 1e-26, which times a P of 2^-40 would be below fp32's smallest normal number."""
    x = [t.to(DEV) for t in orc.make_inputs(1, 4, 150, D, scale=0.5, seed=D)[:5]]
    x = [(t * (1e-13 if i >= 3 else 1)).to(torch.bfloat16) for i, t in enumerate(x)]
    got = _forward(x, 1 / D)
    for h in range(4):
        exact = _references([t[:, h:h + 1] for t in x], 1 / D, True)[0][0]
        assert float((got[h].double() - exact).norm()) <= 2.0 ** -7 * float(exact.norm())
