"""GPU: the layer's single host call each way against the router and the experts called one after the other."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _layer(pkg, H, I, E, k, codes=None, **kw):
    layer = pkg.MoELayer(H, I, E, top_k=k, act_codes=codes, **kw).to(DEV).to(torch.bfloat16)
    layer.bias.copy_(torch.randn(E, device=DEV) * 0.01)
    return layer


def _composed(pkg, layer, x):
    idx, w, counts = pkg.fused_mlp_router(x, layer.gate.weight, layer.bias, layer.top_k, layer.num_experts, layer.norm_topk_prob,
                                          layer.routed_scaling_factor, return_counts=True)
    return pkg.moe(x, idx, w, layer.gate_up_proj, layer.down_proj, layer.act_codes), counts


# both sides of the small router's token limit, one pick, mixed codes, one pick without renormalisation
@pytest.mark.parametrize("T,H,I,E,k,codes,kw", [(1, 64, 64, 8, 2, None, {}), (2368, 264, 136, 16, 3, None, {}),
                                                (2369, 264, 136, 16, 1, [0, 1, 5, 0] * 4, {}),
                                                (2000, 512, 264, 40, 6, None, dict(norm_topk_prob=False, routed_scaling_factor=2.5))])
def test_layer_equals_router_then_experts(pkg, T, H, I, E, k, codes, kw):
    torch.manual_seed(T)
    layer = _layer(pkg, H, I, E, k, codes, **kw)
    x = torch.randn(T, H, device=DEV).to(torch.bfloat16).requires_grad_()
    gy = torch.randn(T, H, device=DEV).to(torch.bfloat16)
    leaves = [x, layer.gate.weight, layer.gate_up_proj, layer.down_proj]
    out = layer(x)
    got = torch.autograd.grad(out, leaves, gy)
    counts, load = layer.last_counts.clone(), layer.load.clone()
    ref, ref_counts = _composed(pkg, layer, x)
    want = torch.autograd.grad(ref, leaves, gy)
    pkg.check_status()
    assert torch.equal(out, ref) and torch.equal(counts, ref_counts) and torch.equal(load, ref_counts.long())
    for a, b in zip(got[1:], want[1:]):
        assert torch.equal(a, b)
    # grad_x is rounded once here, the two shares and their sum there: at most three roundings of 2^-8 apart
    assert O.rel_l2(got[0].float(), want[0].float()) < 3 * 2 ** -8
    with torch.no_grad():      # the counts are added by every training forward, whatever the grad mode
        layer(x)
        layer.eval()
        layer(x)
    assert torch.equal(layer.load, 2 * ref_counts.long())


def test_layer_gradients_of_a_subset_and_of_saved_tensors_moved_away(pkg):
    torch.manual_seed(0)
    layer = _layer(pkg, 128, 64, 8, 2)
    x = torch.randn(300, 128, device=DEV).to(torch.bfloat16).requires_grad_()
    gy = torch.randn(300, 128, device=DEV).to(torch.bfloat16)
    leaves = [x, layer.gate.weight, layer.gate_up_proj, layer.down_proj]
    full = torch.autograd.grad(layer(x), leaves, gy)
    for i, leaf in enumerate(leaves):
        for t in leaves:
            t.requires_grad_(t is leaf)
        assert torch.equal(torch.autograd.grad(layer(x), [leaf], gy)[0], full[i])
    for t in leaves:
        t.requires_grad_()
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.to(DEV)):
        out = layer(x)
    torch.empty(64 << 20, dtype=torch.uint8, device=DEV).fill_(255)     # what the forward left on the device is gone
    for a, b in zip(torch.autograd.grad(out, leaves, gy), full):
        assert torch.equal(a, b)
    pkg.check_status()


def test_layer_on_a_side_stream(pkg):
    torch.manual_seed(1)
    layer = _layer(pkg, 256, 128, 8, 2)
    x = torch.randn(700, 256, device=DEV).to(torch.bfloat16)
    ref = layer(x).detach()
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        outs = [layer(x).detach() for _ in range(8)]
    torch.cuda.current_stream().wait_stream(s)
    assert all(torch.equal(o, ref) for o in outs)
    pkg.check_status()


def test_observer_sees_the_operations_of_the_native_sequences(pkg):
    layer = _layer(pkg, 256, 128, 8, 2)
    x = torch.randn(2400, 256, device=DEV).to(torch.bfloat16).requires_grad_()
    seen = []
    pkg.ops.set_hook(lambda name, launches, a, b: seen.append((name, launches, a, b)))
    try:
        layer(x).sum().backward()
    finally:
        pkg.ops.set_hook(None)
    torch.cuda.synchronize()
    assert [n for n, *_ in seen] == ["gemm_nt", "router_topk_fwd", "permute_build", "gather_rows", "expert_gate_up_swiglu",
                                     "expert_down", "combine", "combine_bwd", "expert_down_dgrad_glu", "expert_wgrad",
                                     "expert_wgrad", "expert_gate_up_dgrad", "router_topk_bwd", "gemm_nn", "gemm_tn", "combine"]
    assert all(a.elapsed_time(b) > 0 for _, _, a, b in seen)
    n = len(seen)
    layer(x)
    assert len(seen) == n


# SMs reserved for an exchange: the split products of the routers' weight gradients take fewer slices out of the same workspace
@pytest.mark.parametrize("reserved", [1, 40, 146])
def test_router_gradients_with_reserved_sms(pkg, reserved):
    g = torch.Generator().manual_seed(reserved)
    lib = pkg.lib()
    x = torch.randn(3000, 264, generator=g).to(torch.bfloat16).to(DEV)
    rand = lambda *s: (torch.randn(*s, generator=g) * 0.1).to(torch.bfloat16).to(DEV).requires_grad_()     # noqa: E731
    linear, wide, conv, wconv = rand(64, 264), rand(256, 264), rand(8, 264, 4), rand(128, 264, 3)
    G = torch.randn(3000, 4, generator=g).to(DEV)

    def grads():
        out = [torch.autograd.grad(pkg.fused_mlp_router(x, w, None, 4, w.shape[0])[1], w, G)[0] for w in (linear, wide)]
        return out + [torch.autograd.grad(pkg.fused_router(x.view(4, 750, 264), w, None, 4, w.shape[0])[1], w, G.view(4, 750, 4))[0]
                      for w in (conv, wconv)]

    want = grads()
    assert lib.b200moe_set_reserved_sms(reserved) == 0
    try:
        got = grads()
    finally:
        lib.b200moe_set_reserved_sms(0)
    pkg.check_status()
    for a, b in zip(got, want):      # fp32 sums in another order: single bf16 results round the other way
        assert torch.isfinite(a).all() and O.rel_l2(a.float(), b.float()) < 2e-3
