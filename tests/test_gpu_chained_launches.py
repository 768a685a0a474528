"""GPU: launches whose set-up overlaps the kernel before them.  Passes in flight one after the other, weights and inputs
rewritten between them on the stream, must give what the same passes give with the device idle before each, what they give
beside passes on another stream, and what plain launches give."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
KINDS = ["one token", "few rows", "mxfp8", "train", "mxfp8 train", "conv"]
SPLIT_SUM = {"train": 2, "mxfp8 train": 2, "conv": 3}     # the router weight's gradient: summed in as many parts as there are free SMs


def _program(pkg, kind):
    """A function of the pass number that rewrites the input and the weights and queues a pass; its outputs."""
    torch.manual_seed(3)
    T, H, E, I, k = {"one token": (1, 256, 16, 136, 4), "few rows": (300, 264, 32, 264, 4), "mxfp8": (40, 256, 8, 256, 2),
                     "train": (700, 264, 16, 200, 3), "mxfp8 train": (700, 256, 8, 256, 2), "conv": (0, 256, 32, 0, 4)}[kind]
    if kind == "conv":
        w = (torch.randn(E, H, 4, device=DEV) * 0.02).to(torch.bfloat16).requires_grad_()
        x = torch.randn(3, 200, H, device=DEV).to(torch.bfloat16).requires_grad_()
        params = [w]
    else:
        with torch.device(DEV):
            layer = pkg.MoELayer(H, I, E, top_k=k, precision="mxfp8" if "mxfp8" in kind else "bf16")
        layer = layer.to(DEV).to(torch.bfloat16)
        x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_("train" in kind)
        params = [layer.gate.weight, layer.gate_up_proj, layer.down_proj]

    def run(i, between=lambda: None):
        between()
        with torch.no_grad():
            x.mul_(-0.75).add_(0.125)
            for p in params:
                p.mul_(-1.0 if i % 2 else 1.25)
        between()
        if kind == "conv":
            x.grad = w.grad = None
            idx, wt = pkg.fused_router(x, w, None, k, E)
            wt.backward(torch.ones_like(wt) * torch.arange(k, device=DEV))
            return [idx, wt.detach(), x.grad, w.grad]
        if "train" in kind:
            layer.zero_grad(set_to_none=True)
            x.grad = None
            out = layer(x)
            out.backward(out.detach())
            return [out.detach(), x.grad] + [p.grad for p in params]
        with torch.no_grad():
            return [layer(x)]
    return run


def _passes(pkg, kind, n=12, between=lambda: None):
    run = _program(pkg, kind)
    res = [run(i, between) for i in range(n)]
    torch.cuda.synchronize()
    return res


def _equal(a, b):
    return all(torch.equal(s, t) for p, q in zip(a, b) for s, t in zip(p, q))


@pytest.mark.parametrize("kind", KINDS)
def test_passes_in_flight_equal_passes_alone(pkg, kind):
    alone = _passes(pkg, kind, between=torch.cuda.synchronize)
    assert _equal(alone, _passes(pkg, kind))
    # two programs on two streams, a pass of each in turn, no synchronisation until both are done
    side = torch.cuda.Stream()
    here = _program(pkg, kind)
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        there = _program(pkg, kind)
    a, b = [], []
    for i in range(12):
        a.append(here(i))
        with torch.cuda.stream(side):
            b.append(there(i))
    torch.cuda.synchronize()
    assert _equal(alone, a) and _equal(alone, b)
    pkg.check_status()


@pytest.mark.parametrize("kind", KINDS)
def test_chained_launches_equal_plain_launches(pkg, kind):
    """With SMs kept free for an exchange every launch is a plain one.  Fewer SMs deal the tiles out differently, which changes no
    sum but those split over the SMs: in another order they differ by far less than a bf16 step (2^-8 of a value), so that the
    rounded results differ by one step at most; a sum that nearly cancels by fp32's share (1e-5) of the others."""
    chained = _passes(pkg, kind, 6)
    pkg.lib().b200moe_set_reserved_sms(2)
    try:
        plain = _passes(pkg, kind, 6)
    finally:
        pkg.lib().b200moe_set_reserved_sms(0)
    for p, q in zip(chained, plain):
        for j, (s, t) in enumerate(zip(p, q)):
            if j == SPLIT_SUM.get(kind):
                assert ((s.float() - t.float()).abs() <= t.float().abs() * 2.0 ** -7 + 1e-5 * t.float().abs().max()).all(), kind
            else:
                assert torch.equal(s, t), (kind, j)
    pkg.check_status()
