"""GPU: the conv router over any sequence length and width, against float64 on the device's own picks."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one position, fewer positions than taps, one tap, tiles with a row and a column remainder, a width that is no multiple of 16,
# enough rows for pair tiles and several split-K slices, many taps
@pytest.mark.parametrize("B,S,H,E,K,k", [(1, 1, 8, 8, 1, 1), (2, 3, 64, 8, 4, 2), (3, 129, 72, 24, 3, 4), (2, 65, 272, 136, 4, 8),
                                         (7, 600, 256, 64, 4, 6), (2, 2048, 528, 256, 2, 8), (1, 200, 64, 16, 64, 2)])
def test_conv_router_against_float64(pkg, B, S, H, E, K, k):
    g = torch.Generator().manual_seed(S + H)
    x = torch.randn(B, S, H, generator=g).to(torch.bfloat16)
    w = (torch.randn(E, H, K, generator=g) * (H * K) ** -0.5).to(torch.bfloat16)
    bias = torch.randn(E, generator=g) * 0.05
    G = torch.randn(B, S, k, generator=g)
    xd, wd = x.to(DEV).requires_grad_(), w.to(DEV).requires_grad_()
    idx, wt, counts = pkg.fused_router(xd, wd, bias.to(DEV), k, E, return_counts=True)
    wt.backward(G.to(DEV))
    pkg.check_status()
    assert torch.equal(counts.cpu().long(), torch.bincount(idx.flatten().cpu(), minlength=E))
    x64, w64 = x.double().requires_grad_(), w.double().requires_grad_()
    xp = torch.nn.functional.pad(x64, (0, 0, K - 1, 0))
    logits = sum(xp[:, j:j + S] @ w64[:, :, j].T for j in range(K))
    picks = idx.cpu()
    sel = torch.sigmoid(logits.detach()) + bias.double()
    # every pick is the best of those left, up to the bf16 rounding of two logits (2^-8 of each; the sigmoid's slope <= 1/4)
    slack = 2 ** -8 * logits.detach().abs().amax() / 4 * 2
    left = sel.clone()
    for j in range(k):
        got = left.gather(-1, picks[..., j:j + 1])[..., 0]
        assert (got >= left.amax(-1) - slack).all()
        left.scatter_(-1, picks[..., j:j + 1], -1e30)
    p = torch.sigmoid(logits).gather(-1, picks)
    p = p / p.sum(-1, keepdim=True) if k > 1 else p
    p.backward(G.double())
    # weights: sigmoids of logits rounded to bf16; gradients: the logits' gradients rounded to bf16, fp32 sums, one rounding
    assert O.rel_l2(wt.detach().cpu().double(), p.detach()) < 4e-3
    assert O.rel_l2(xd.grad.cpu().double(), x64.grad) < 1e-2
    assert O.rel_l2(wd.grad.cpu().double(), w64.grad) < 1e-2


# weight gradient of up to 128 rows (taps * experts) on single-CTA tiles, of more on pair tiles: both sides of the line, a width
# that is a multiple of 256 and one that is not
@pytest.mark.parametrize("rows", [8, 128, 136])
@pytest.mark.parametrize("H", [64, 512, 1048])
def test_split_product_of_few_rows(pkg, rows, H):
    g = torch.Generator().manual_seed(rows + H)
    T = 1500
    u, x = (torch.randn(T, n, generator=g).to(torch.bfloat16).to(DEV) for n in (rows, H))
    got = pkg.ops.gemm_tn(u, x)
    pkg.check_status()
    assert O.rel_l2(got.double().cpu(), (u.double().T @ x.double()).cpu()) < 3.95e-3      # one bf16 rounding: 2^-8


# the in-place product at ragged lengths and widths gives the logits of the unfolded product to the bit (the same k order)
@pytest.mark.parametrize("B,S,H,E,K", [(3, 129, 80, 24, 3), (2, 300, 512, 64, 4), (4, 64, 1040, 128, 2), (2, 257, 96, 256, 4)])
def test_conv_logits_equal_the_unfolded_product(pkg, B, S, H, E, K):
    g = torch.Generator().manual_seed(S)
    x = torch.randn(B, S, H, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, H, K, generator=g) * 0.05).to(torch.bfloat16).to(DEV)
    lib = pkg.lib()
    wt = torch.empty(K * E, H, dtype=torch.bfloat16, device=DEV)
    logits = torch.full((B * S, E), float("nan"), dtype=torch.bfloat16, device=DEV)
    st, status = torch.cuda.current_stream().cuda_stream, torch.zeros(1, dtype=torch.int32, device=DEV)
    assert lib.b200moe_conv_weight_rows(w.data_ptr(), E, H, K, 0, wt.data_ptr(), st) == 0
    assert torch.equal(wt, w.permute(2, 0, 1).reshape(K * E, H))
    assert lib.b200moe_conv_gemm_logits(x.data_ptr(), wt.data_ptr(), logits.data_ptr(), B, S, H, E, K, status.data_ptr(), st) == 0
    wf = w.permute(0, 2, 1).reshape(E, K * H).contiguous()
    assert torch.equal(logits, pkg.ops.gemm_nt(pkg.ops.conv_unfold(x, K), wf))
    assert int(status.item()) == 0


# many short sequences, whose product runs over the unfolded copy, give what a few of them give, whose product runs in place
@pytest.mark.parametrize("B,S,H,E,K,k", [(4096, 1, 64, 8, 4, 2), (2048, 5, 272, 16, 3, 4), (1500, 16, 80, 136, 2, 8)])
def test_short_sequences_equal_a_part_of_them(pkg, B, S, H, E, K, k):
    g = torch.Generator().manual_seed(B)
    x = torch.randn(B, S, H, generator=g).to(torch.bfloat16).to(DEV).requires_grad_()
    w = (torch.randn(E, H, K, generator=g) * (H * K) ** -0.5).to(torch.bfloat16).to(DEV).requires_grad_()
    bias, G = torch.randn(E, generator=g).to(DEV) * 0.05, torch.randn(B, S, k, generator=g).to(DEV)
    n = 40
    ws = pkg.lib().b200moe_conv_router_fwd_ws_bytes
    assert ws(B, S, H, E, K) > 0 and ws(n, S, H, E, K) == 0
    idx, wt = pkg.fused_router(x, w, bias, k, E)
    gx, gw = torch.autograd.grad(wt, (x, w), G)
    for lo in (0, B - n):
        part = x.detach()[lo:lo + n].requires_grad_()
        i, p = pkg.fused_router(part, w, bias, k, E)
        assert torch.equal(i, idx[lo:lo + n]) and torch.equal(p, wt[lo:lo + n])
        assert torch.equal(torch.autograd.grad(p, part, G[lo:lo + n])[0], gx[lo:lo + n])
    pkg.check_status()


def test_observer_names_the_products_that_run(pkg):
    x = torch.randn(2, 300, 128, device=DEV).to(torch.bfloat16).requires_grad_()
    w = torch.randn(8, 128, 4, device=DEV).to(torch.bfloat16).requires_grad_()
    seen = []
    pkg.ops.set_hook(lambda name, launches, a, b: seen.append(name))
    try:
        pkg.fused_router(x, w, None, 2, 8)[1].sum().backward()
    finally:
        pkg.ops.set_hook(None)
    assert seen == ["conv_weight_rows", "conv_gemm_logits", "router_topk_fwd", "conv_topk_bwd", "gemm_nn", "gemm_tn_splitk",
                    "conv_weight_grad"]
