"""GPU: a block pads the rows of its own buffers to whole lines (csrc/common.cuh, row_pitch); the steps called one by one over dense rows give
the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# remainders of the 32 elements that decide, on both sides: none, 8, 16, 24; single-CTA and pair tiles; a row of one vector and of no whole
# number of warps; fused activations and row kernels
@pytest.mark.parametrize("T,H,I,E,k", [(700, 72, 40, 5, 2), (700, 80, 136, 5, 2), (700, 96, 104, 5, 2), (300, 8, 8, 3, 1), (700, 264, 680, 5, 2),
                                       (3001, 1032, 680, 16, 4), (3001, 1048, 712, 16, 4), (3001, 1064, 696, 16, 4), (500, 2056, 8200, 2, 1)])
@pytest.mark.parametrize("codes", [(0,), (0, 1, 5), (2, 7, 0, 6)])
def test_block_equals_its_steps_over_dense_rows(pkg, T, H, I, E, k, codes):
    ops = pkg.ops
    g = torch.Generator(device=DEV).manual_seed(H + I)
    rand = lambda *s: (torch.randn(*s, generator=g, device=DEV) * 0.1).bfloat16()     # noqa: E731
    x, go, gu, dn = rand(T, H), rand(T, H), rand(E, 2 * I, H), rand(E, H, I)
    idx = torch.rand(T, E, generator=g, device=DEV).topk(k, 1).indices
    w = torch.rand(T, k, generator=g, device=DEV)
    cd = torch.tensor([codes[e % len(codes)] for e in range(E)], dtype=torch.int32, device=DEV)
    leaves = [t.clone().requires_grad_() for t in (x, w, gu, dn)]
    torch.full((256 << 20,), float("nan"), device=DEV)           # what the padding holds must not matter
    out = pkg.moe(leaves[0], idx, leaves[1], leaves[2], leaves[3], cd)
    got = [out.detach()] + list(torch.autograd.grad(out, leaves, go))
    with torch.no_grad():
        quiet = pkg.moe(x, idx, w, gu, dn, cd)
    perm = ops.permute_build(idx, E)
    x_s = ops.gather_rows(x, perm)
    rows = max(codes) in (2, 6, 7)
    if rows:
        gate_up = ops.expert_linear(x_s, gu, perm)
        inter = ops.glu_fwd_rows(gate_up, cd, None, perm)
    else:
        gate_up, inter = ops.expert_gate_up_swiglu(x_s, gu, perm, cd if any(codes) else None)
    eo = ops.expert_down(inter, dn, perm)
    want = [ops.combine(eo, w, perm)]
    geo, gw = ops.combine_bwd(go, eo, w, perm)
    if rows:
        ggu = ops.glu_bwd_rows(ops.expert_linear_t(geo, dn, perm), gate_up, cd, None, perm)
        ggu = ggu[0] if isinstance(ggu, tuple) else ggu
    else:
        ggu = ops.expert_down_dgrad_glu(geo, dn, gate_up, perm, cd if any(codes) else None)
    want += [ops.combine_raw(ops.expert_gate_up_dgrad(ggu, gu, perm), None, perm.slot_row, T, k), gw, ops.expert_wgrad(ggu, x_s, perm),
             ops.expert_wgrad(geo, inter, perm)]
    pkg.check_status()
    for name, a, b in zip(("out", "grad_x", "grad_w", "grad_gate_up", "grad_down"), got, want):
        assert torch.equal(a, b), name
    assert torch.equal(quiet, got[0])


# x_s padded and the results dense, both dense, inter padded or dense, all padded; with Identity and Zero experts, whose rows go from one to the other
@pytest.mark.parametrize("H,I", [(264, 520), (360, 256), (456, 200), (136, 72), (256, 456), (520, 264), (1288, 648)])
@pytest.mark.parametrize("codes", [(0,), (0, 1, 5), (2, 7, 0, 3, 4)])
def test_forward_without_backward_equals_the_one_with(pkg, H, I, codes):
    T, k = 3000, 3
    g = torch.Generator(device=DEV).manual_seed(H + I)
    rand = lambda *s: (torch.randn(*s, generator=g, device=DEV) * 0.1).bfloat16()     # noqa: E731
    E = 5 if 3 in codes else 8
    n = E - 2 if 3 in codes else E
    x, gu, dn = rand(T, H), rand(n, 2 * I, H), rand(n, H, I)
    idx = torch.rand(T, E, generator=g, device=DEV).topk(k, 1).indices
    w = torch.rand(T, k, generator=g, device=DEV)
    cd = torch.tensor([codes[e % len(codes)] for e in range(E)], dtype=torch.int32, device=DEV)
    kept = pkg.moe(x, idx, w, gu.clone().requires_grad_(), dn, cd).detach()
    torch.full((256 << 20,), float("nan"), device=DEV)           # what the padding holds must not matter
    with torch.no_grad():
        assert torch.equal(pkg.moe(x, idx, w, gu, dn, cd), kept)
    pkg.check_status()
