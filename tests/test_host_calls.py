"""Calls made by the native host extension against the same calls made by the Python code, and whom it leaves to that code."""
import importlib.util
import os

import pytest
import torch

from flash_trittention import TrittentionTriton, _native, flash_trittention

DEV = "cuda:0"
SCALARS = (0.125, True, 0)


def _loaded():
    _native.lib()
    return _native._host


def test_what_the_extension_does_not_take():
    host = _loaded()
    assert host is not None, "the host extension is not built"
    x = torch.zeros(1, 1, 8, 16)
    assert host.forward() is None and host.forward(0, 1, 2) is None and host.backward(1, x) is None
    assert host.forward(_native.OP_TDP_FWD, *[x] * 5, *SCALARS, 1, 1, 1, 1) is None          # not on a GPU
    assert host.forward(_native.OP_TDP_FWD, *["q"] * 5, *SCALARS, 1, 1, 1, 1) is None
    assert host.backward(_native.OP_DPS_BWD, *[x] * 8, *SCALARS, 4, None) is None


def test_an_extension_for_another_pytorch_is_not_used(monkeypatch):
    L = _native.lib()
    for name in ("_host", "host_forward", "host_backward"):
        monkeypatch.setattr(_native, name, None)
    monkeypatch.setattr(torch, "__version__", "0.1")
    with pytest.warns(UserWarning, match="built for PyTorch .* not 0.1"):
        _native._load_host(L)
    assert _native._host is None and _native.host_forward is None


def test_the_extension_is_rebuilt_for_what_it_depends_on(monkeypatch, tmp_path):
    path = os.path.join(os.path.dirname(os.path.dirname(_native.LIB_PATH)), "build.py")
    spec = importlib.util.spec_from_file_location("tritt_build", path)
    build = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(build)
    files = {name: str(tmp_path / name) for name in ("HOST", "HOST_STAMP", "HOST_SRC", "ABI_HEADER")}
    for i, (name, f) in enumerate(files.items()):
        monkeypatch.setattr(build, name, f)
        open(f, "w").close()
        os.utime(f, (1000, 1000))
    recipe = build._host_recipe()
    os.utime(files["HOST"], (2000, 2000))
    assert not build.host_is_current(recipe)   # an extension of which nothing is known
    with open(files["HOST_STAMP"], "w") as f:
        f.write("\n".join(recipe))
    assert build.host_is_current(recipe)
    for name in ("HOST_SRC", "ABI_HEADER"):
        os.utime(files[name], (3000, 3000))
        assert not build.host_is_current(recipe), name
        os.utime(files[name], (1000, 1000))
    monkeypatch.setattr(torch, "__version__", "0.1")
    assert not build.host_is_current(build._host_recipe())
    # without a compiler the library is built alone
    monkeypatch.setattr(build.shutil, "which", lambda name: None)
    with pytest.warns(UserWarning, match="host extension was not built.*g.. not found"):
        build.build_host_if_possible()


class Counted:
    """host_forward / host_backward that count the calls they took, or take none."""

    def __init__(self, monkeypatch, take):
        self.taken = 0
        for name in ("host_forward", "host_backward"):
            f = getattr(_native._host, name[5:])
            monkeypatch.setattr(_native, name, (lambda *a, f=f: self._count(f(*a))) if take else (lambda *a: None))

    def _count(self, out):
        self.taken += out is not None
        return out


def _step(op, ins, kw, dz):
    if op == "dps":
        o, m = TrittentionTriton(**kw)(*ins)
    else:
        o, m = flash_trittention(*ins, **kw), torch.zeros(1, device=DEV)
    return [o.detach(), m.detach(), *torch.autograd.grad(o, ins, dz)]


def _tensors(shape, dtype, seed=0, grad=True):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return [(torch.randn(shape, generator=g, device=DEV) * 0.5).to(dtype).requires_grad_(grad) for _ in range(5)]


WINDOWS = dict(k1_window=20, k2_window=None, kk_left=3, kk_right=None)
CALLS = [("tdp", dict(softmax_scale=0.125, causal=True, **WINDOWS)), ("tdp", dict(softmax_scale=0.02, causal=False, **WINDOWS)),
         ("tdp", dict(causal=True, convert_to_float32=True, **WINDOWS)), ("tdp", dict(input_precision="ieee", **WINDOWS)),
         ("dps", dict(softmax_scale=0.125, causal=True, k_diff=30)), ("dps", dict(causal=False, k_diff=100, convert_to_float32=True))]


@pytest.mark.gpu
@pytest.mark.parametrize("op,kw", CALLS)
@pytest.mark.parametrize("dtype", [torch.float32, torch.float16, torch.bfloat16])
def test_against_the_python_code(op, kw, dtype, monkeypatch):
    ins = _tensors((2, 1, 100, 64), dtype)
    dz = torch.randn_like(ins[0])
    _loaded()
    _native.status_word(DEV)
    Counted(monkeypatch, False)
    before = _native.launches
    ref = _step(op, ins, kw, dz)
    assert _native.launches == before + 2
    host = Counted(monkeypatch, True)
    out = _step(op, ins, kw, dz)
    assert host.taken == 2 and _native.launches == before + 4
    # the tensor cores' forward is the same twice; all else may add fp32 numbers in another order, then rounds once to the type
    exact = 2 if "input_precision" not in kw and not kw.get("convert_to_float32") and dtype != torch.float32 else 0
    for i, (a, b) in enumerate(zip(out, ref)):
        assert i >= exact or torch.equal(a, b)
        eps = {torch.float32: 1e-5, torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]
        assert a.shape == b.shape and a.stride() == b.stride() and float((a - b).norm()) <= eps * float(b.norm())
    assert _native.read_status(DEV) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("take", [False, True])
@pytest.mark.parametrize("windows,most", [((None,) * 4, 12e6), ((128, 128, 32, 32), 40e6)])
def test_a_forward_allocates_what_its_windows_need(windows, most, take, monkeypatch):
    ins = _tensors((4, 8, 600, 64), torch.float16, grad=False)
    kw = dict(softmax_scale=1 / 64, k1_window=windows[0], k2_window=windows[1], kk_left=windows[2], kk_right=windows[3])
    _loaded()
    _native.status_word(DEV)
    Counted(monkeypatch, take)
    flash_trittention(*ins, **kw)
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    flash_trittention(*ins, **kw)
    used = torch.cuda.max_memory_allocated() - before
    assert used <= most and (windows[0] is None or used > 16e6)   # (tensors of 2.5 MB; the areas of a narrow band 20 MB)


class Labelled(torch.Tensor):
    pass


@pytest.mark.gpu
@pytest.mark.parametrize("op,kw", [CALLS[0], CALLS[4]])
def test_calls_left_to_the_python_code(op, kw, monkeypatch):
    _loaded()
    _native.status_word(DEV)
    host = Counted(monkeypatch, True)
    ins = _tensors((1, 2, 65, 64), torch.float16)
    dz = torch.randn_like(ins[0])
    ref = _step(op, ins, kw, dz)
    assert host.taken == 2
    # one operand off a 16-byte boundary, one transposed: copied in Python, in the forward alone
    off = torch.empty(ins[1].numel() + 1, device=DEV, dtype=torch.float16)[1:].view_as(ins[1]).copy_(ins[1].detach())
    turned = ins[2].detach().transpose(1, 2).contiguous().transpose(1, 2)
    again = [ins[0], off.requires_grad_(), turned.requires_grad_(), *ins[3:]]
    out = _step(op, again, kw, dz)
    assert host.taken == 3 and torch.equal(out[0], ref[0]) and torch.equal(out[1], ref[1])
    # an upstream gradient that is one number, expanded
    o = TrittentionTriton(**kw)(*ins)[0] if op == "dps" else flash_trittention(*ins, **kw)
    o.sum().backward()
    assert host.taken == 4 and all(bool(t.grad.isfinite().all()) for t in ins)
    # subclasses give subclasses
    sub = [t.detach().as_subclass(Labelled) for t in ins]
    o = TrittentionTriton(**kw)(*sub)[0] if op == "dps" else flash_trittention(*sub, **kw)
    assert type(o) is Labelled and host.taken == 4 and torch.equal(o.as_subclass(torch.Tensor), ref[0])
    # saved tensors that come back from the host's memory
    with torch.autograd.graph.save_on_cpu():
        out = _step(op, ins, kw, dz)
    assert torch.equal(out[0], ref[0])
    # errors
    with pytest.raises(ValueError):
        _step(op, [ins[0], ins[1][:, :, :64], *ins[2:]], kw, dz)
    with pytest.raises(ValueError):
        _step(op, [ins[0], ins[1].float(), *ins[2:]], kw, dz)
    with pytest.raises(ValueError):
        _step(op, [t[..., :48].contiguous() for t in ins], kw, dz[..., :48])
    # a kernel of an earlier call that gave up
    _native.status_word(DEV)[0] = 2
    with pytest.raises(_native.TrittError):
        _step(op, ins, kw, dz)
    assert _native.read_status(DEV) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("op,kw", [CALLS[0], CALLS[4]])
def test_capture_and_other_streams(op, kw):
    ins = _tensors((1, 2, 130, 64), torch.float16)
    dz = torch.randn_like(ins[0])
    _step(op, ins, kw, dz)
    ref = _step(op, ins, kw, dz)
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        out = _step(op, ins, kw, dz)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        captured = _step(op, ins, kw, dz)
    g.replay()
    torch.cuda.synchronize()
    for got in (out, captured):
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
        for a, b in zip(got[2:], ref[2:]):
            assert float((a - b).norm()) <= 2e-3 * float(b.norm())
