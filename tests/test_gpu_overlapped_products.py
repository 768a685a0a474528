"""GPU: a backward in chained launches, whose kernels are set up beside the end of the one before them (csrc/common.cuh), against plain launches."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# single-CTA tiles, pair tiles of few and of several waves, row kernels with special experts; passes of other routings one after the other in the same
# memory, so that a table or an operand read too early would be the one of the pass before; every subset of gradients that changes which kernels follow each other
@pytest.mark.parametrize("T,H,I,E,k,codes", [(512, 256, 512, 8, 2, (0,)), (3001, 1032, 680, 16, 4, (0, 1, 5)), (1200, 520, 264, 9, 2, (2, 0, 7)),
                                             (20, 72, 40, 3, 1, (0,)), (8200, 1032, 200, 6, 4, (0,))])
def test_overlapped_products_equal_plain_launches(pkg, T, H, I, E, k, codes):
    g = torch.Generator(device=DEV).manual_seed(T)
    rand = lambda *s: (torch.randn(*s, generator=g, device=DEV) * 0.1).bfloat16()     # noqa: E731
    special = [3, 4] if codes[0] == 2 else []
    n = E - len(special)
    cd = torch.tensor([codes[e % len(codes)] for e in range(n)] + special, dtype=torch.int32, device=DEV)
    gu, dn = rand(n, 2 * I, H), rand(n, H, I)
    passes = []
    for p in range(4):       # from one expert to all of them: other counts, offsets and tiles each time
        score = torch.rand(T, E, generator=g, device=DEV) + (torch.arange(E, device=DEV) < k) * (p % 2) * 2
        passes.append((rand(T, H), score.topk(k, 1).indices, torch.rand(T, k, generator=g, device=DEV), rand(T, H)))

    def run(want):
        out = []
        for x, idx, w, go in passes:
            leaves = [t.detach().requires_grad_(i in want) for i, t in enumerate((x, w, gu, dn))]
            y = pkg.moe(leaves[0], idx, leaves[1], leaves[2], leaves[3], cd)
            out.append([y.detach()] + list(torch.autograd.grad(y, [leaves[i] for i in want], go)))
        return out

    lib = pkg.lib()
    for want in ((0, 1, 2, 3), (3,), (0,), (0, 3), (2, 3), (1, 3)):
        got = run(want)
        assert lib.b200moe_set_reserved_sms(2) == 0      # launches are plain ones
        try:
            ref = run(want)
        finally:
            lib.b200moe_set_reserved_sms(0)
        pkg.check_status()
        for p, (a, b) in enumerate(zip(got, ref)):
            assert all(torch.equal(s, t) for s, t in zip(a, b)), (want, p)


# the router's backward behind the experts': its top-k kernel, dX and the weight gradient
@pytest.mark.parametrize("T,H,E,k", [(512, 256, 8, 2), (3001, 1032, 32, 4), (2500, 264, 128, 8)])
def test_overlapped_router_backward_equals_plain_launches(pkg, T, H, E, k):
    torch.manual_seed(T)
    layer = pkg.MoELayer(H, 136, E, top_k=k).to(DEV).bfloat16()
    xs = [torch.randn(T, H, device=DEV).bfloat16().requires_grad_() for _ in range(3)]
    gys = [torch.randn(T, H, device=DEV).bfloat16() for _ in range(3)]
    params = [layer.gate.weight, layer.gate_up_proj, layer.down_proj]

    def run():
        return [torch.autograd.grad(layer(x), [x] + params, gy) for x, gy in zip(xs, gys)]

    lib = pkg.lib()
    got = run()
    assert lib.b200moe_set_reserved_sms(2) == 0
    try:
        ref = run()
    finally:
        lib.b200moe_set_reserved_sms(0)
    pkg.check_status()
    for a, b in zip(got, ref):
        assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2]) and torch.equal(a[3], b[3])
        # fewer SMs, fewer slices: fp32 sums in another order, single bf16 results round the other way
        assert (a[1].float() - b[1].float()).norm() < 2e-3 * b[1].float().norm()
