"""GPU: launches whose set-up overlaps the kernel before them.  Passes in flight one after the other, weights and inputs
rewritten between them on the stream, must give what the same passes give with the device idle before each."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _passes(pkg, kind, n, sync):
    """Outputs of n passes; the input and the weights change on the stream before each."""
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
    res = []
    for i in range(n):
        if sync:
            torch.cuda.synchronize()
        with torch.no_grad():
            x.mul_(-0.75).add_(0.125)
            for p in params:
                p.mul_(-1.0 if i % 2 else 1.25)
        if sync:
            torch.cuda.synchronize()
        if kind == "conv":
            x.grad = w.grad = None
            idx, wt = pkg.fused_router(x, w, None, k, E)
            wt.backward(torch.ones_like(wt) * torch.arange(k, device=DEV))
            res += [idx, wt.detach(), x.grad, w.grad]
        elif "train" in kind:
            layer.zero_grad(set_to_none=True)
            x.grad = None
            out = layer(x)
            out.backward(out.detach())
            res += [out.detach(), x.grad] + [p.grad for p in params]
        else:
            with torch.no_grad():
                res.append(layer(x))
    torch.cuda.synchronize()
    return res


@pytest.mark.parametrize("kind", ["one token", "few rows", "mxfp8", "train", "mxfp8 train", "conv"])
def test_passes_in_flight_equal_passes_alone(pkg, kind):
    alone = _passes(pkg, kind, 12, True)
    assert all(torch.equal(a, b) for a, b in zip(alone, _passes(pkg, kind, 12, False)))
    # on two streams, other layers beside them: the results stay those of each layer alone
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        other = _passes(pkg, kind, 12, False)
    assert all(torch.equal(a, b) for a, b in zip(alone, other))
    # plain launches, as with SMs kept free for an exchange (fewer SMs: other splits of sums, none in these products)
    pkg.lib().b200moe_set_reserved_sms(8)
    try:
        plain = _passes(pkg, "one token" if kind == "one token" else "few rows", 4, False)
    finally:
        pkg.lib().b200moe_set_reserved_sms(0)
    chained = _passes(pkg, "one token" if kind == "one token" else "few rows", 4, True)
    assert all(torch.equal(a, b) for a, b in zip(plain, chained))
    pkg.check_status()
