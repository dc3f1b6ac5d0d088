"""The calls that stand for the use of this package: what is timed, on which inputs, and how exact the results must be.

Two operators, each through its public entry point and autograd:

* ``tdp``: ``flash_trittention`` (triple-dot-product), forward alone (inference) or forward and backward (a training
  step returns the output and the five gradients);
* ``dps``: the ``TrittentionTriton`` module (dot-product-sum), which returns the output and the log-sum-exp.

A case is a dict of plain values: ``op``, ``mode`` ("fwd" or "train"), the sizes ``B N T D``, ``dtype``, ``causal``, the
windows ``k1w k2w kkl kkr`` (0 = the whole sequence; ``k_diff`` for dps), and ``dist``, the inputs' distribution:
"half" is N(0,1)/2 with alpha = 1/D (the benchmark's own setting), "unit" is N(0,1) with alpha = 1/8 (the entry
points' default scale and the tests' setting; its logits are of order 1-10).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.getcwd(), "flash-3-way-attention_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from flash_trittention.dot_product_sum.trittention_triton import TrittentionTriton  # noqa: E402
from flash_trittention.triple_dot_product.flash_trittention import flash_trittention  # noqa: E402

_DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}


def _case(name, op, mode, B, N, T, D, dtype, causal=True, windows=(0, 0, 0, 0), k_diff=0, dist="half"):
    k1w, k2w, kkl, kkr = windows
    case = dict(op=op, mode=mode, B=B, N=N, T=T, D=D, dtype=dtype, causal=causal, dist=dist)
    case.update(dict(k_diff=k_diff) if op == "dps" else dict(k1w=k1w, k2w=k2w, kkl=kkl, kkr=kkr))
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the headline benchmark: a training step of one long sequence, sixteen heads, whole causal triangle
        _case("tdp_train_16x2048x128_bf16", "tdp", "train", 1, 16, 2048, 128, "bf16"),
        # the longest sequence of the benchmark, few heads (the largest call)
        _case("tdp_train_4x4096x64_bf16", "tdp", "train", 1, 4, 4096, 64, "bf16"),
        # inference on a batch of medium sequences
        _case("tdp_fwd_32x512x64_bf16", "tdp", "fwd", 4, 8, 512, 64, "bf16"),
        # training on medium sequences at the default scale, logits of order 1-10
        _case("tdp_train_16x512x64_fp16_unit", "tdp", "train", 2, 8, 512, 64, "fp16", dist="unit"),
        # local attention: a training step under the banded benchmark's windows
        _case("tdp_train_16x2048x64_fp16_band", "tdp", "train", 2, 8, 2048, 64, "fp16", windows=(128, 128, 32, 32)),
        # local attention over a long context, inference
        _case("tdp_fwd_16x8192x64_fp16_band", "tdp", "fwd", 2, 8, 8192, 64, "fp16", windows=(128, 128, 32, 32)),
        # a ragged length and few heads, as a variable-length training batch has them
        _case("tdp_train_4x333x128_bf16", "tdp", "train", 1, 4, 333, 128, "bf16"),
        # bidirectional (encoder) training
        _case("tdp_train_16x512x64_fp16_noncausal", "tdp", "train", 2, 8, 512, 64, "fp16", causal=False),
        # training with fp32 tensors
        _case("tdp_train_32x512x64_fp32", "tdp", "train", 4, 8, 512, 64, "fp32"),
        # a small head dimension in fp32: the size of the parity configuration
        _case("tdp_train_2x64x32_fp32", "tdp", "train", 1, 2, 64, 32, "fp32"),
        # dot-product-sum training
        _case("dps_train_16x1024x64_fp16", "dps", "train", 2, 8, 1024, 64, "fp16"),
        # one short prompt: the latency of a call
        _case("tdp_fwd_8x64x64_bf16", "tdp", "fwd", 1, 8, 64, 64, "bf16"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: the kinds of the listed ones with sizes spread over their ranges (lengths of any residue)."""
    cap = 0.4 * work(listed()[1])["flops"]
    while True:
        kind = rng.choice(["full", "full", "full", "full", "band", "band", "noncausal", "fp32", "small", "dps", "dps"])
        mode = rng.choice(["fwd", "train", "train"])
        dist = rng.choice(["half", "unit"])
        dtype = rng.choice(["bf16", "fp16"])
        D = rng.choice([64, 128])
        B, N = rng.choice([1, 2, 4]), rng.choice([1, 2, 4, 8, 16])
        if kind == "band":
            w = [_log_int(rng, 1, 256) for _ in range(2)] + [_log_int(rng, 1, 64) for _ in range(2)]
            c = _case(None, "tdp", mode, B, N, _log_int(rng, 128, 8192), D, dtype, windows=w, dist=dist)
        elif kind == "noncausal":
            c = _case(None, "tdp", mode, B, N, _log_int(rng, 33, 1024), D, dtype, causal=False, dist=dist)
        elif kind == "fp32":
            c = _case(None, "tdp", mode, B, N, _log_int(rng, 33, 1024), D, "fp32", dist=dist)
        elif kind == "small":
            c = _case(None, "tdp", mode, 1, rng.choice([1, 2, 4]), _log_int(rng, 33, 128), rng.choice([16, 32]), "fp32",
                      causal=rng.choice([True, False]), dist=dist)
        elif kind == "dps":
            T = _log_int(rng, 33, 2048)
            c = _case(None, "dps", mode, B, N, T, D, dtype, causal=rng.choice([True, True, False]),
                      k_diff=rng.choice([0, 0, _log_int(rng, 2, T)]), dist=dist)
        else:
            c = _case(None, "tdp", mode, B, N, _log_int(rng, 33, 4096), D, dtype, dist=dist)
        if work(c)["flops"] <= cap:
            return c


def prepare(case, seed):
    """Inputs and upstream gradient on the GPU, and, for dps, the module a program keeps."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (case["B"], case["N"], case["T"], case["D"])
    scale = 0.5 if case["dist"] == "half" else 1.0
    dtype = _DTYPES[case["dtype"]]
    train = case["mode"] == "train"
    ins = [(torch.randn(shape, generator=g, device="cuda") * scale).to(dtype).requires_grad_(train) for _ in range(5)]
    dz = (torch.randn(shape, generator=g, device="cuda") * scale).to(dtype)
    alpha = 1.0 / case["D"] if case["dist"] == "half" else 1.0 / 8.0
    state = dict(ins=ins, dz=dz, train=train)
    if case["op"] == "dps":
        state["module"] = TrittentionTriton(causal=case["causal"], softmax_scale=alpha, k_diff=case["k_diff"] or case["T"])
    else:
        state["kw"] = dict(softmax_scale=alpha, causal=case["causal"], k1_window=case["k1w"] or None,
                           k2_window=case["k2w"] or None, kk_left=case["kkl"] or None, kk_right=case["kkr"] or None)
    return state


def run(state):
    ins = state["ins"]
    if "module" in state:
        out = state["module"](*ins)
        o, rest = out[0], [out[1]]
    else:
        o, rest = flash_trittention(*ins, **state["kw"]), []
    if not state["train"]:
        return [o, *rest]
    grads = torch.autograd.grad(o, ins, state["dz"])
    return [o.detach(), *rest, *grads]


def _exact_tdp(case, ins, dz, alpha):
    """Dense fp64 triple-dot-product, in chunks of queries: the output and, for a training step, the five gradients."""
    T, causal = case["T"], case["causal"]
    w1, w2, kl, kr = (min(case[k] or T, T) for k in ("k1w", "k2w", "kkl", "kkr"))
    Q, K1, K2, V1, V2 = ins
    sig = torch.sigmoid(V1)
    S1 = V1 * sig
    O = torch.zeros_like(Q)
    dQ, dK1, dK2, dS1, dV2 = (torch.zeros_like(Q) for _ in range(5))
    n = max(1, min(64, int(6e7 / min(T, max(w1, w2) + 64) ** 2)))
    for h in range(Q.shape[0]):
        for a in range(0, T, n):
            b = min(T, a + n)
            j0, k0, end = (max(0, a - w1), max(0, a - w2), b) if causal else (0, 0, T)
            k1, s1, k2, v2 = K1[h, j0:end], S1[h, j0:end], K2[h, k0:end], V2[h, k0:end]
            A = alpha * Q[h, a:b, None] * k2                                     # [q, k, h]
            P = A @ k1.T                                                         # [q, k, j]
            if causal:
                q = torch.arange(a, b, device=Q.device)[:, None]
                j, k = (torch.arange(x, end, device=Q.device) for x in (j0, k0))
                ok = ((k <= q) & (q - k <= w2))[:, :, None] & ((j <= q) & (q - j <= w1))[:, None, :]
                ok &= ((j >= k[:, None] - kl) & (j <= k[:, None] + kr))
                P.masked_fill_(~ok, -math.inf)
            P.sub_(P.amax((1, 2), keepdim=True)).exp_()
            P.div_(P.sum((1, 2), keepdim=True))
            U = P @ s1
            O[h, a:b] = (U * v2).sum(1)
            if case["mode"] == "fwd":
                continue
            do = dz[h, a:b, None]
            A2 = do * v2
            dV2[h, k0:end] += (U * do).sum(0)
            dS1[h, j0:end] += P.flatten(0, 1).T @ A2.flatten(0, 1)
            dP = A2 @ s1.T
            dP.sub_((do[:, 0] * O[h, a:b]).sum(-1)[:, None, None]).mul_(P)       # the scores' gradient
            G = alpha * (dP @ k1)
            dQ[h, a:b] = (G * k2).sum(1)
            dK2[h, k0:end] += (G * Q[h, a:b, None]).sum(0)
            dK1[h, j0:end] += dP.flatten(0, 1).T @ A.flatten(0, 1)
    if case["mode"] == "fwd":
        return [O]
    return [O, dQ, dK1, dK2, dS1 * (sig + S1 * (1 - sig)), dV2]


def _exact_dps(case, ins, dz, alpha):
    """Dense fp64 dot-product-sum: the soft-max over (s, t) as two chained ones, autograd for the gradients."""
    T = case["T"]
    ins = [x.requires_grad_(True) for x in ins]
    Q, K1, K2, V1, V2 = ins
    t = torch.arange(T, device=Q.device)
    E, F = alpha * (K2 @ K1.transpose(1, 2)), alpha * (Q @ K2.transpose(1, 2))   # [t, s], [q, t]
    if case["causal"]:
        kd = case["k_diff"] or T
        E = E.masked_fill(~((t <= t[:, None]) & (t[:, None] - t <= kd)), -math.inf)
        F = F.masked_fill(t > t[:, None], -math.inf)
    F = F + torch.logsumexp(E, -1)[:, None]
    o = torch.softmax(F, -1) @ (torch.softmax(E, -1) @ torch.nn.functional.silu(V1) * V2)
    out = [o, torch.logsumexp(F, -1)]
    if case["mode"] == "train":
        out += torch.autograd.grad(o, ins, dz)
    return [x.detach() for x in out]


def exact(case, seed):
    """The outputs of ``run`` for the same inputs by plain fp64 tensor algebra."""
    state = prepare(case, seed)
    alpha = 1.0 / case["D"] if case["dist"] == "half" else 1.0 / 8.0
    shape = state["dz"].shape
    ins = [x.detach().double().flatten(0, 1) for x in state["ins"]]
    dz = state["dz"].double().flatten(0, 1)
    out = (_exact_dps if case["op"] == "dps" else _exact_tdp)(case, ins, dz, alpha)
    return [x.unflatten(0, shape[:2]) for x in out]


def _attended(case):
    """Attended (q, j, k) triples of one head (tdp), or pairs of the two chained attentions (dps)."""
    T = case["T"]
    if case["op"] == "dps":
        if not case["causal"]:
            return 2 * T * T
        kd = min(case["k_diff"] or T, T)
        t = np.arange(T, dtype=np.int64)
        return int(np.sum(np.minimum(t, kd) + 1)) + T * (T + 1) // 2
    if not case["causal"]:
        return T ** 3
    w1, w2, kl, kr = (min(case[k] or T, T) for k in ("k1w", "k2w", "kkl", "kkr"))
    if min(w1, w2, kl, kr) >= T:
        return T * (T + 1) * (2 * T + 1) // 6

    def at(q):
        k = np.arange(max(0, q - w2), q + 1, dtype=np.int64)
        lo = np.maximum(np.maximum(0, q - w1), k - kl)
        return int(np.sum(np.maximum(0, np.minimum(q, k + kr) - lo + 1)))

    edge = min(T, max(w1, w2) + 1)   # from there on every query attends the same number
    return sum(at(q) for q in range(edge)) + (T - edge) * (at(edge) if edge < T else 0)


def work(case):
    bn, n = case["B"] * case["N"], case["B"] * case["N"] * case["T"] * case["D"]
    # forward: two products per attended triple (pair); backward: six per triple of tdp, five per pair of dps
    products = 2 if case["mode"] == "fwd" else (8 if case["op"] == "tdp" else 7)
    size = 4 if case["dtype"] == "fp32" else 2
    tensors = 6 if case["mode"] == "fwd" else 12
    lse = 4 * bn * case["T"] if case["op"] == "dps" else 0
    return {"bytes": tensors * n * size + lse, "flops": 2.0 * products * case["D"] * bn * _attended(case)}


def tolerance(case):
    """About four times the largest relative error against dense fp64 results (measured over lengths 33-1500, all masks
    and both distributions)."""
    if case["dtype"] == "fp32" and case["D"] < 64:
        return {"rel": 5e-6}     # exact fp32 arithmetic: up to 7e-7
    if case["dtype"] == "bf16":
        return {"rel": 2e-2}     # 16-bit operands: 3e-3 to 7e-3
    # fp16, and fp32 tensors, whose products take operands of 11 significant bits: 3e-4 to 1.6e-3.  Without the causal
    # mask dQ and dK1 are small differences of large sums (4e-3 to 6e-3).
    return {"rel": 6e-3 if case["causal"] else 2e-2}
