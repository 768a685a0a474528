"""GPU: the grouped products for few rows per expert against the row-tile kernels and an fp32 reference."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
# one bf16 rounding of the result (8 significant bits: at most 2^-8 = 3.9e-3 of each value) on fp32 sums
TOL = 3.95e-3


# rows an expert gets: none, one, both sides of the 16-row step and of the 64 / 128 / 192-row tiles, several tiles;
# widths that fill no tile, one k-block and a remainder, the smallest
@pytest.mark.parametrize("counts,H,I", [([1], 8, 8), ([0, 1, 0, 15, 16, 17, 0], 72, 136), ([63, 64, 65, 0], 256, 128),
                                        ([129, 100, 0, 128], 1032, 680), ([193, 150, 192, 0, 385], 264, 200),
                                        ([700, 0, 0, 0, 0, 0, 0, 0], 512, 264), ([2] * 256, 64, 128)])
@pytest.mark.parametrize("codes", [False, True])
def test_few_rows_products(pkg, counts, H, I, codes):
    E, M = len(counts), sum(counts)
    g = torch.Generator().manual_seed(M + H)
    idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(M, generator=g)].view(M, 1).to(DEV)
    x = torch.randn(M, H, generator=g).to(torch.bfloat16).to(DEV)
    gu = (torch.randn(E, 2 * I, H, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    dn = (torch.randn(E, H, I, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    act = torch.tensor([(0, 1, 5)[e % 3] for e in range(E)], dtype=torch.int32, device=DEV) if codes else None
    ops = pkg.ops
    perm = ops.permute_build(idx, E, want_order=True)
    inter = ops.expert_gate_up_few(ops.gather_compact(x, perm), gu, perm, act)
    out = ops.expert_linear_few(inter, dn, perm)
    pkg.check_status()
    # the same rounding points and k order as the row-tile kernels: bit-identical
    _, ref_inter = ops.expert_gate_up_swiglu(ops.gather_rows(x, perm), gu, perm, act)
    ref_out = ops.expert_down(ref_inter, dn, perm)
    r, c = perm.slot_row.long(), perm.slot_pos.long()
    assert torch.equal(inter[c], ref_inter[r]) and torch.equal(out[c], ref_out[r])
    e = idx[:, 0].cpu()
    ref = torch.einsum("mi,mhi->mh", inter[c].cpu().float(), dn.cpu().float()[e])
    assert O.rel_l2(out[c].cpu().float(), ref) < TOL


# wide enough that the tile follows the mean: 64, 128 and 192 rows, with experts on both sides of one and of several tiles; and one
# wave of 64-row chunks at a mean past each of the other limits
@pytest.mark.parametrize("counts,H,I", [([0, 63, 64, 65, 1, 0, 17, 40], 72, 1800), ([129, 100, 0, 128], 136, 2184),
                                        ([256, 30, 0, 127, 1, 200], 264, 1224), ([193, 150, 192, 0, 385], 136, 1032),
                                        ([576, 0, 191, 1], 1224, 136), ([193, 150, 192, 0, 385], 72, 136)])
def test_few_rows_products_of_wide_experts(pkg, counts, H, I):
    test_few_rows_products(pkg, counts, H, I, False)


@pytest.mark.parametrize("T,E,k", [(1, 8, 2), (40, 16, 4), (1279, 16, 2), (1281, 16, 2)])   # both sides of the limit
def test_forward_without_gradient_equals_the_training_forward(pkg, T, E, k):
    torch.manual_seed(T)
    layer = pkg.MoELayer(264, 136, E, top_k=k).to(DEV).to(torch.bfloat16)
    x = torch.randn(T, 264, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        quiet = layer(x)
    assert torch.equal(quiet, layer(x))
    pkg.check_status()


def test_bad_expert_index_without_gradient(pkg):
    """A slot whose expert index is out of range adds nothing and raises the status word."""
    x = torch.randn(3, 64, device=DEV).to(torch.bfloat16)
    gu, dn = (torch.randn(4, *s, device=DEV).to(torch.bfloat16) for s in ((128, 64), (64, 64)))
    idx = torch.tensor([[0, 9], [1, 2], [-1, 3]], device=DEV)
    w = torch.rand(3, 2, device=DEV)
    out = pkg.moe(x, idx, w, gu, dn, torch.zeros(4, dtype=torch.int32, device=DEV))
    with pytest.raises(RuntimeError, match="expert index"):
        pkg.check_status()
    ok = pkg.moe(x, idx.clamp(0, 3), w * torch.tensor([[1, 0], [1, 1], [0, 1]], device=DEV), gu, dn,
                 torch.zeros(4, dtype=torch.int32, device=DEV))
    pkg.check_status()
    assert torch.equal(out, ok)


# serving under skewed routing: frequencies ~ rank^-1.1, and every token's first pick on one expert; compact rows with 64-, 128- and
# 192-row tiles, and row tiles
@pytest.mark.parametrize("T,E,k,H,I", [(60, 32, 4, 264, 136), (900, 64, 6, 136, 520), (1500, 64, 6, 264, 520), (700, 8, 2, 1032, 1032)])
@pytest.mark.parametrize("hot", [False, True])
def test_skewed_forward_without_gradient_equals_the_training_forward(pkg, T, E, k, H, I, hot):
    g = torch.Generator().manual_seed(T)
    freq = torch.arange(1, E + 1).float().pow(-1.1).expand(T, E).clone()
    freq[:, 0] *= 1e6 if hot else 1
    idx = torch.multinomial(freq, k, generator=g).to(DEV)
    rand = lambda *s: (torch.randn(*s, generator=g) * 0.1).to(torch.bfloat16).to(DEV)     # noqa: E731
    x, gu, dn, w = rand(T, H), rand(E, 2 * I, H), rand(E, H, I).requires_grad_(), torch.rand(T, k, generator=g).to(DEV)
    codes = torch.zeros(E, dtype=torch.int32, device=DEV)
    with torch.no_grad():
        quiet = pkg.moe(x, idx, w, gu, dn, codes)
    assert torch.equal(quiet, pkg.moe(x, idx, w, gu, dn, codes).detach())
    pkg.check_status()


def test_few_rows_products_into_unaligned_memory(pkg):
    """Results that are not 16-byte aligned are written value by value, and nothing beside them."""
    L, ops = pkg.lib(), pkg.ops
    for counts, H, I in (([5, 0, 40], 72, 136), ([180, 150, 170, 192] * 8, 136, 1032)):     # 64- and 192-row tiles
        E, M = len(counts), sum(counts)
        g = torch.Generator().manual_seed(M)
        idx = torch.repeat_interleave(torch.arange(E), torch.tensor(counts))[torch.randperm(M, generator=g)].view(M, 1).to(DEV)
        x = torch.randn(M, H, generator=g).to(torch.bfloat16).to(DEV)
        gu = (torch.randn(E, 2 * I, H, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
        dn = (torch.randn(E, H, I, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
        perm = ops.permute_build(idx, E, want_order=True)
        xs = ops.gather_compact(x, perm)
        inter = ops.expert_gate_up_few(xs, gu, perm, None)
        out = ops.expert_linear_few(inter, dn, perm)
        st, stream = torch.zeros(1, dtype=torch.int32, device=DEV), torch.cuda.current_stream().cuda_stream
        for shift in (1, 4):
            a, b = (torch.full((M * w + 16,), 7.0, dtype=torch.bfloat16, device=DEV) for w in (I, H))
            assert L.b200moe_expert_gate_up_few(xs.data_ptr(), gu.data_ptr(), None, perm.counts.data_ptr(), perm.offs.data_ptr(), M, E,
                                                H, I, a.data_ptr() + 2 * shift, st.data_ptr(), stream) == 0
            assert L.b200moe_expert_linear_few(inter.data_ptr(), dn.data_ptr(), perm.counts.data_ptr(), perm.offs.data_ptr(), M, E, H,
                                               I, b.data_ptr() + 2 * shift, st.data_ptr(), stream) == 0
            for got, want in ((a, inter), (b, out)):
                n = want.numel()
                assert torch.equal(got[shift:shift + n], want.flatten())
                assert (got[:shift] == 7).all() and (got[shift + n:] == 7).all()
        assert int(st) == 0


# k-blocks of 64 channels in pairs: one, an odd number, a remainder of 8; experts up to one and several per lane
@pytest.mark.parametrize("H,E,k", [(8, 8, 1), (64, 32, 4), (72, 40, 8), (192, 64, 6), (200, 128, 8), (1032, 128, 2)])
def test_small_router_equals_the_large_batch(pkg, H, E, k):
    g = torch.Generator().manual_seed(H)
    T = 16 * torch.cuda.get_device_properties(0).multi_processor_count      # the most tokens of one launch
    x = torch.randn(T + 1, H, generator=g).to(torch.bfloat16).to(DEV)
    w = (torch.randn(E, H, generator=g) * 0.1).to(torch.bfloat16).to(DEV)
    bias = (torch.randn(E, generator=g) * 0.1).to(DEV)
    big = pkg.fused_mlp_router(x, w, bias, k, E, return_counts=True)
    for n in (1, 17, T):
        idx, wt, counts = pkg.fused_mlp_router(x[:n], w, bias, k, E, return_counts=True)
        assert torch.equal(idx, big[0][:n]) and torch.equal(wt, big[1][:n])
        assert torch.equal(counts.cpu(), torch.bincount(idx.flatten().cpu(), minlength=E).int())
    pkg.check_status()
