"""GPU: the activation row kernels and the router's top-k kernels at the edges of their row widths and expert counts."""
import types

import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
# outputs are fp32 values rounded once to bf16 (8 significant bits: at most 2^-8 = 3.9e-3 of each value), on fp32 arithmetic
# that adds well under a hundredth of that
TOL = 3.95e-3


def _act64(code, gate, alpha, gamma):
    g = gate
    if code in (2, 6, 7):
        g = gate / (gate.square().mean(1, keepdim=True) + 1e-6).sqrt()
    sig = torch.sigmoid(g)
    if code in (1, 6):
        return torch.relu(g).square()
    if code == 5:
        return gamma * torch.tanh(alpha * g) * sig
    return torch.tanh(g) * sig if code == 7 else g * sig


# row widths: one vector, both sides of every thread-group limit, no multiple of 8, beyond the register kernels
@pytest.mark.parametrize("I", [8, 504, 512, 520, 1024, 1032, 2048, 2056, 4096, 4104, 8192, 8200, 12])
def test_glu_rows_against_float64(pkg, I):
    codes = [0, 1, 2, 5, 6, 7, 5]
    E, rows = len(codes), 256 * len(codes)
    g = torch.Generator().manual_seed(I)
    gate_up = torch.randn(rows, 2 * I, generator=g).to(torch.bfloat16)
    go = torch.randn(rows, I, generator=g).to(torch.bfloat16)
    params = torch.rand(E, 2, generator=g) + 0.5
    perm = types.SimpleNamespace(cap=rows, E=E, tile_expert=torch.arange(E, dtype=torch.int32, device=DEV),
                                 poffs=torch.arange(E + 1, dtype=torch.int32, device=DEV) * 256,
                                 total_rows=torch.tensor([rows], dtype=torch.int32, device=DEV))
    cd, pd = torch.tensor(codes, dtype=torch.int32, device=DEV), params.to(DEV)
    inter = pkg.ops.glu_fwd_rows(gate_up.to(DEV), cd, pd, perm)
    ggu, da, dg = pkg.ops.glu_bwd_rows(go.to(DEV), gate_up.to(DEV), cd, pd, perm, True)
    sums = pkg.ops.expert_row_sums(da, dg, perm, torch.zeros(E, 2, device=DEV))
    for e, code in enumerate(codes):
        sl = slice(256 * e, 256 * (e + 1))
        gt, up = gate_up[sl, :I].double().requires_grad_(), gate_up[sl, I:].double().requires_grad_()
        al, ga = (params[e, i].double().expand(256, 1).clone().requires_grad_() for i in (0, 1))
        out = _act64(code, gt, al, ga) * up
        out.backward(go[sl].double())
        assert O.rel_l2(inter[sl].cpu().double(), out.detach()) < TOL, code
        assert O.rel_l2(ggu[sl, :I].cpu().double(), gt.grad) < TOL, code
        assert O.rel_l2(ggu[sl, I:].cpu().double(), up.grad) < TOL, code
        if code == 5:     # I signed fp32 terms: the rounding of the terms and of their sum stays under 1e-5 of the norm
            assert O.rel_l2(da[sl].cpu().double(), al.grad[:, 0]) < 1e-5
            assert O.rel_l2(dg[sl].cpu().double(), ga.grad[:, 0]) < 1e-5
            ref = torch.stack([al.grad.sum(), ga.grad.sum()])
            bound = 1e-5 * torch.stack([al.grad.abs().sum(), ga.grad.abs().sum()])
            assert ((sums[e].cpu().double() - ref).abs() <= bound).all()
        else:
            assert not da[sl].any() and not dg[sl].any()


# both sides of the limits between two and three vectors a thread
@pytest.mark.parametrize("I", [768, 776, 1536, 1544, 3072, 3080, 6144, 6152])
def test_glu_rows_of_three_vectors_a_thread(pkg, I):
    test_glu_rows_against_float64(pkg, I)


def test_glu_rows_of_special_values(pkg):
    """Infinite, NaN and huge gates give what the formulas give in fp32, and nothing beside them."""
    codes = [0, 1, 5]                                         # (a Norm code spreads such a gate over its row)
    vals = torch.tensor([0.0, 1e-30, 30.0, 87.0, 88.5, 104.0, 1e4, 1e30, float("inf"), float("nan")]).to(torch.bfloat16)
    vals = torch.cat([vals, -vals])
    rows = 256 * len(codes)
    gate_up = torch.ones(rows, 16, dtype=torch.bfloat16)
    gate_up[:, 3] = vals[torch.arange(rows) % len(vals)]
    perm = types.SimpleNamespace(cap=rows, E=3, tile_expert=torch.arange(3, dtype=torch.int32, device=DEV),
                                 poffs=torch.arange(4, dtype=torch.int32, device=DEV) * 256,
                                 total_rows=torch.tensor([rows], dtype=torch.int32, device=DEV))
    cd, pd = torch.tensor(codes, dtype=torch.int32, device=DEV), torch.ones(3, 2, device=DEV)
    inter = pkg.ops.glu_fwd_rows(gate_up.to(DEV), cd, pd, perm).cpu().float()
    ggu, _, _ = pkg.ops.glu_bwd_rows(torch.ones(rows, 8, dtype=torch.bfloat16, device=DEV), gate_up.to(DEV), cd, pd, perm, True)
    for e, code in enumerate(codes):
        sl = slice(256 * e, 256 * (e + 1))
        g = gate_up[sl, 3].float()
        s = 1 / (1 + torch.exp(-g))
        want = {0: g * s, 1: torch.fmax(g, torch.zeros(())).square(), 5: (2 / (1 + torch.exp(-2 * g)) - 1) * s}[code]
        for got in (inter[sl, 3], ggu.cpu().float()[sl, 8 + 3]):      # grad_up is the activation too
            assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.to(torch.bfloat16).isinf())
            ok = want.to(torch.bfloat16).isfinite()
            assert ((got - want)[ok].abs() <= 2 ** -8 * want[ok].abs() + 1e-35).all()      # one rounding; results of 2^-126 and less may be 0
    assert torch.isfinite(inter[:, torch.arange(8) != 3]).all()


@pytest.mark.parametrize("E,k", [(1, 1), (31, 8), (32, 32), (33, 5), (64, 8), (65, 8), (128, 8), (129, 32), (256, 32)])
def test_router_kernels_at_the_widths_of_a_lane(pkg, E, k):
    N = 1000
    g = torch.Generator().manual_seed(E)
    s = torch.sigmoid(torch.randn(N, E, generator=g)).to(torch.bfloat16).float()     # many exact ties
    bias = torch.randn(E, generator=g) * 0.1
    bias[0] = -float("inf")                                     # below the value that a picked expert falls to
    idx_o, w_o, c_o = O.topk_from_scores(s, bias, k, True, 1.0)
    idx, w, c = pkg.ops.router_topk_fwd(s.to(DEV), bias.to(DEV), k, True, 1.0, scores=True)
    assert torch.equal(idx.cpu(), idx_o) and torch.equal(c.cpu(), c_o) and torch.equal(w.cpu(), w_o)
    logits = torch.randn(N, E, generator=g).to(torch.bfloat16)
    G = torch.randn(N, k, generator=g)
    idx_o, _, _ = O.router_epilogue_fwd(logits, None, k, True, 1.5)
    gl = pkg.ops.router_topk_bwd(logits.to(DEV), idx_o.to(DEV), G.to(DEV), True, 1.5)
    x = logits.double().requires_grad_()
    p = torch.sigmoid(x).gather(1, idx_o)
    (1.5 * p / p.sum(1, keepdim=True) if k > 1 else 1.5 * p).backward(G.double())
    # bf16 results; the renormalised gradient is a difference of terms of the size of its largest one, kept in fp32
    assert O.rel_l2(gl.cpu().double(), x.grad) < TOL or (E == 1 and x.grad.norm() == 0)


# both sides of every limit of the split (1024, 2^17, 2^18, 2^20 slots), a remainder of one slot, experts without rows
@pytest.mark.parametrize("T,E,k", [(1, 1, 1), (128, 256, 8), (1025, 33, 1), (512, 256, 8), (16384, 256, 8), (131073, 256, 1),
                                   (32768, 128, 8), (262145, 256, 1), (131072, 64, 8), (131073, 256, 8), (299999, 7, 8)])
def test_permutation_at_the_edges_of_its_launches(pkg, T, E, k):
    idx = torch.randint(0, max(E - 1, 1), (T, k), generator=torch.Generator().manual_seed(T))
    tb = O.permutation_tables(idx, E)
    perm = pkg.ops.permute_build(idx.to(DEV), E, want_order=True)
    pkg.check_status()
    total = int(tb["poffs"][-1])
    for name in ("counts", "offs", "poffs", "slot_row"):
        assert torch.equal(getattr(perm, name).cpu(), tb[name]), name
    assert torch.equal(perm.order.cpu().long(), tb["order"])
    assert torch.equal(perm.slot_pos.cpu().long()[tb["order"]], torch.arange(T * k))
    assert torch.equal(perm.row_slot.cpu()[:total], tb["row_slot"])
    assert torch.equal(perm.tile_expert.cpu()[: total // 256], tb["tile_expert"])


# a token remainder and exactly 16, every lane width, one k-block and more than the ring holds, widths that fill no k-block
@pytest.mark.parametrize("T,H,E,k", [(1, 8, 8, 2), (148, 264, 24, 3), (16, 1032, 64, 6), (591, 512, 8, 8), (3, 4096, 128, 4),
                                     (151, 2048, 40, 1), (70, 64, 120, 32), (2368, 768, 128, 8)])
def test_small_router_against_gemm_and_top_k(pkg, T, H, E, k):
    g = torch.Generator().manual_seed(T + H)
    x = torch.randn(T, H, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, H, generator=g) * H ** -0.5).to(torch.bfloat16).to(DEV)
    bias = (torch.randn(E, generator=g) * 0.05).to(DEV)
    got = pkg.ops.router_small_fwd(x, w, bias, k, True, 1.5)
    logits = pkg.ops.gemm_nt(x, w)
    pkg.check_status()
    for a, b in zip(got, (logits, *pkg.ops.router_topk_fwd(logits, bias, k, True, 1.5))):
        assert torch.equal(a, b)
    assert O.rel_l2(logits.cpu().double(), x.cpu().double() @ w.cpu().double().T) < TOL


# row widths on both sides of every thread-group limit (32, 64, 128, 256 vectors), one vector, more than a CTA; one pick to 32
@pytest.mark.parametrize("H,k", [(8, 1), (248, 5), (256, 8), (264, 3), (512, 2), (520, 4), (1024, 6), (1032, 32), (2048, 6), (2056, 7)])
def test_copying_kernels_at_the_widths_of_a_row(pkg, H, k):
    T, E = 301, 40
    g = torch.Generator().manual_seed(H + k)
    idx = torch.stack([torch.randperm(E, generator=g)[:k] for _ in range(T)])
    x, go, add = (torch.randn(T, H, generator=g).to(torch.bfloat16) for _ in range(3))
    w = torch.rand(T, k, generator=g)
    ops = pkg.ops
    perm = ops.permute_build(idx.to(DEV), E)
    total = int(perm.poffs[-1])
    xs = ops.gather_rows(x.to(DEV), perm)
    rs = perm.row_slot[:total].cpu().long()
    live = rs >= 0
    assert torch.equal(xs[:total].cpu()[live], x[rs[live] // k]) and not xs[:total].cpu()[~live].any()
    eo = torch.randn(perm.cap, H, generator=g).to(torch.bfloat16)
    picked = eo[perm.slot_row.cpu().long()].double().view(T, k, H)
    out = ops.combine(eo.to(DEV), w.to(DEV), perm)
    assert O.rel_l2(out.cpu().double(), (picked * w.double().unsqueeze(2)).sum(1)) < TOL
    both = torch.empty(T, H, dtype=torch.bfloat16, device=DEV)
    rows, ad = eo.to(DEV), add.to(DEV)
    assert pkg.lib().b200moe_combine_add(rows.data_ptr(), None, perm.slot_row.data_ptr(), ad.data_ptr(), T, k, H, both.data_ptr(),
                                         torch.cuda.current_stream().cuda_stream) == 0
    assert O.rel_l2(both.cpu().double(), picked.sum(1) + add.double()) < TOL
    geo, gw = ops.combine_bwd(go.to(DEV), rows, w.to(DEV), perm)
    want = go[rs[live] // k].float() * w.flatten()[rs[live]].unsqueeze(1)
    assert torch.equal(geo[:total].cpu()[live], want.to(torch.bfloat16)) and not geo[:total].cpu()[~live].any()
    # H signed fp32 terms: within 1e-5 of the sum of their sizes
    terms = go.double().unsqueeze(1) * picked
    assert ((gw.cpu().double() - terms.sum(2)).abs() <= 1e-5 * terms.abs().sum(2)).all()
