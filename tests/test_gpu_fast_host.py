"""GPU: the compiled autograd functions (csrc/fast.cpp) against the Python Functions they stand in for: the same bits and the
same gradients for plain calls, and the Python Function for every call that is not plain."""
import importlib

import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu
DEV = "cuda"


class Spy:
    """The module, noting of each call whether it took it (True) or left it to the Python Function (False)."""

    def __init__(self, module):
        self.taken = []
        for name in ("layer", "experts", "conv_router"):
            setattr(self, name, self._noting(getattr(module, name)))

    def _noting(self, fn):
        def call(*a):
            self.taken.append(True)       # so is one that raises: a native error, a checkpoint's end of its second forward
            res = fn(*a)
            self.taken[-1] = res is not None
            return res
        return call


@pytest.fixture()
def spy(pkg, monkeypatch):
    """The compiled functions under a Spy; `spy.off` takes them away."""
    L = importlib.import_module(pkg.__name__ + "._lib")
    real = L.fast
    s = Spy(real())
    s.off = False
    monkeypatch.setattr(L, "fast", lambda: None if s.off or real() is None else s)
    return s


def _rand(*s, seed=0):
    return (torch.randn(*s, generator=torch.Generator().manual_seed(seed + sum(s))) * 0.1).to(torch.bfloat16).to(DEV)


def _call(pkg, kind, x_grad=True):
    """(outputs, leaves) of one forward; fresh leaves every time."""
    g = torch.Generator().manual_seed(5)
    if kind == "conv":
        x, w = _rand(3, 40, 64).requires_grad_(x_grad), _rand(16, 64, 4).requires_grad_()
        idx, wt, counts = pkg.fused_router(x, w, torch.linspace(-1, 1, 16, device=DEV), 3, 16, return_counts=True)
        return (wt, idx, counts), [x, w]
    T, H, I, E, k = 70, 64, 72, 8, 3
    if kind in ("layer", "codes"):
        torch.manual_seed(1)
        layer = pkg.MoELayer(H, I, E, top_k=k, act_codes=[0, 1, 5, 0, 1, 5, 0, 0] if kind == "codes" else None).to(DEV).to(torch.bfloat16)
        x = _rand(2, T // 2, H).requires_grad_(x_grad)
        out = layer(x)
        return (out, layer.last_counts, layer.load), [x, layer.gate.weight, layer.gate_up_proj, layer.down_proj]
    special = 2 if kind == "poly" else 0
    x, gu, dn = _rand(T, H).requires_grad_(x_grad), _rand(E, 2 * I, H).requires_grad_(), _rand(E, H, I).requires_grad_()
    idx = torch.stack([torch.randperm(E + special, generator=g)[:k] for _ in range(T)]).to(DEV)
    w = torch.rand(T, k, generator=g).to(DEV).requires_grad_()
    codes = torch.tensor([0, 1, 2, 5, 6, 7, 0, 5, 3, 4][:E + special] if special else [0] * E, dtype=torch.int32, device=DEV)
    act = torch.linspace(0.8, 1.2, 2 * (E + 2), device=DEV).view(E + 2, 2).requires_grad_() if special else None
    out = pkg.moe(x, idx, w, gu, dn, codes, act)
    return (out,), [x, w, gu, dn] + ([act] if special else [])


@pytest.mark.parametrize("kind", ["layer", "codes", "moe", "poly", "conv"])
@pytest.mark.parametrize("x_grad", [True, False])
def test_compiled_equals_python(pkg, spy, kind, x_grad):
    res = []
    for spy.off in (True, False):
        outs, leaves = _call(pkg, kind, x_grad)
        outs[0].backward(torch.ones_like(outs[0]) * 0.25)
        with torch.no_grad():
            quiet, _ = _call(pkg, kind, x_grad)
        some, leaves2 = _call(pkg, kind, x_grad)      # a gradient of one input only
        one = torch.autograd.grad(some[0].sum(), leaves2[1])[0]
        assert not quiet[0].requires_grad and outs[0].requires_grad
        res.append([t for t in (*outs, *[p.grad for p in leaves], quiet[0], one)])
        assert spy.taken == ([] if spy.off else [True] * 3)
    pkg.check_status()
    for a, b in zip(*res):
        assert (a is None and b is None) or (a.shape == b.shape and a.dtype == b.dtype and torch.equal(a, b))


@pytest.mark.parametrize("kind", ["layer", "poly", "conv"])
def test_saved_tensors_pass_through_hooks(pkg, spy, kind):
    outs, leaves = _call(pkg, kind)
    outs[0].sum().backward()
    want = [p.grad.clone() for p in leaves]
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t.cpu(), lambda t: t.to(DEV)):
        outs, leaves = _call(pkg, kind)
    outs[0].sum().backward()
    assert spy.taken == [True, True]
    assert len(packed) >= 4 and all(torch.equal(a, p.grad) for a, p in zip(want, leaves))
    pkg.check_status()


class Passing(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_calls_that_are_not_plain_take_the_python_function(pkg, spy):
    def declined(f):
        """f's result; every compiled function that it called left the call to Python."""
        n = len(spy.taken)
        try:
            return f()
        finally:
            assert spy.taken[n:] and not any(spy.taken[n:])

    layer = pkg.MoELayer(64, 72, 8, top_k=2).to(DEV).to(torch.bfloat16)
    wide = _rand(40, 128)
    x = wide[:, :64]                                   # rows 128 apart: made contiguous by the Python Function
    with torch.no_grad():
        want = layer(x.contiguous())
        assert spy.taken == [True]
        assert torch.equal(declined(lambda: layer(x)), want)
        with Passing():                                # a mode that has to see the allocations
            assert torch.equal(declined(lambda: layer(x.contiguous())), want)
        f32 = layer.float()                            # cast under autocast
        with torch.autocast("cuda", dtype=torch.bfloat16):
            cast = declined(lambda: f32(x.float()))
        assert torch.equal(cast, layer.to(torch.bfloat16)(x.contiguous()))
    with pytest.raises(ValueError):
        declined(lambda: layer(x.float()))             # no autocast: refused
    with pytest.raises(ValueError):
        declined(lambda: layer(torch.zeros(4, 56, dtype=torch.bfloat16, device=DEV)))
    with pytest.raises(ValueError):                    # native errors keep their Python types
        pkg.fused_router(_rand(1, 8, 64), _rand(16, 64, 4), None, 17, 16)
    xs = x.contiguous()
    for transform in (lambda: torch.func.vmap(lambda a: layer(a))(xs.view(2, 20, 64)),
                      lambda: torch.func.grad(lambda a: layer(a).float().sum())(xs),
                      lambda: torch.func.jvp(lambda a: layer(a), (xs,), (xs,))):
        errors = []
        for spy.off in (True, False):
            with pytest.raises(Exception) as e:
                transform() if spy.off else declined(transform)
            errors.append(type(e.value))
        assert errors[0] is errors[1]
    n = len(spy.taken)
    y = torch.utils.checkpoint.checkpoint(layer, xs.clone().requires_grad_(), use_reentrant=False)
    y.sum().backward()
    assert spy.taken[n:] == [True, True]
    pkg.check_status()
