"""GPU: grouped products at ragged widths: the narrow last pair tile and both sides of the choice between pair and
single-CTA tiles, against fp32."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
TOL = 3.95e-3      # one bf16 rounding of fp32 sums: at most 2^-8 of each value (GLU values: of rounded gate and up, below)


# N tails of 8, 16, 24, 72, 136, 248 columns past a multiple of 256 and exactly 128 / 256; few rows take single-CTA tiles,
# many rows pair tiles
@pytest.mark.parametrize("N", [72, 128, 136, 256, 264, 280, 328, 392, 504, 1032])
@pytest.mark.parametrize("rows", [40, 1500])
def test_grouped_products_at_ragged_widths(pkg, N, rows):
    E, K = 12, 200
    g = torch.Generator().manual_seed(N + rows)
    ops, bf = pkg.ops, torch.bfloat16
    idx = torch.randint(0, E - 1, (rows * E, 1), generator=g).to(DEV)      # the last expert stays empty
    perm = ops.permute_build(idx, E)
    r, e = perm.slot_row.long(), idx[:, 0].long()
    M = rows * E
    rand = lambda *s: (torch.randn(*s, generator=g) * 0.2).to(bf).to(DEV)      # noqa: E731
    x, wide = rand(M, K), rand(M, N)
    xs, ws = ops.gather_rows(x, perm), ops.gather_rows(wide, perm)
    w_nk, w_kn, gu = rand(E, N, K), rand(E, K, N), rand(E, 2 * N, K)

    def per_expert(f, n):
        out = torch.empty(M, n, device=DEV)
        for i in range(E - 1):
            out[e == i] = f(i, e == i)
        return out

    assert O.rel_l2(ops.expert_linear(xs, w_nk, perm)[r].float(), per_expert(lambda i, m: x[m].float() @ w_nk[i].float().T, N)) < TOL
    assert O.rel_l2(ops.expert_linear_t(xs, w_kn, perm)[r].float(), per_expert(lambda i, m: x[m].float() @ w_kn[i].float(), N)) < TOL
    gate_up, inter = ops.expert_gate_up_swiglu(xs, gu, perm)
    ref = per_expert(lambda i, m: x[m].float() @ gu[i].float().T, 2 * N)
    assert O.rel_l2(gate_up[r].float(), ref) < TOL
    rg, ru = gate_up[r].float().split(N, dim=1)
    assert O.rel_l2(inter[r].float(), torch.nn.functional.silu(rg) * ru) < TOL
    # GLU backward: grad_inter (K = K here) is rounded to bf16 before it meets gate and up: two roundings
    ggu = ops.expert_down_dgrad_glu(xs, w_kn, gate_up, perm)
    gi = per_expert(lambda i, m: x[m].float() @ w_kn[i].float(), N)
    s = torch.sigmoid(rg)
    want = torch.cat([gi * ru * s * (1 + rg * (1 - s)), gi * rg * s], 1)
    assert O.rel_l2(ggu[r].float(), want) < 2 * TOL
    # weight gradients: N as the column and as the row extent, an expert without rows
    for a, b, sa, sb in ((xs, ws, x, wide), (ws, xs, wide, x)):
        got = ops.expert_wgrad(a, b, perm)
        ref = torch.stack([sa[e == i].float().T @ sb[e == i].float() for i in range(E)])
        assert O.rel_l2(got.float(), ref) < TOL and not got[E - 1].any()
    pkg.check_status()


# matrices whose smaller side leaves a padded remainder of 8, 56, 64, 120, 248 rows, or none; wide and tall; one iteration and several
@pytest.mark.parametrize("E,r,c", [(3, 248, 400), (2, 264, 520), (2, 320, 264), (1, 456, 640), (4, 8, 72), (2, 512, 512)])
def test_optimizer_iteration_over_the_live_part_equals_the_padded_products(pkg, E, r, c):
    import ctypes
    from importlib import import_module
    muon, ops, lib = import_module(pkg.__name__ + ".muon"), pkg.ops, pkg.lib()
    small, wide = min(r, c), max(r, c)
    Rp = -(-small // 256) * 256
    coeffs = [(3.4445, -4.7750, 2.0315), (2.0, -1.5, 0.5), (2.0, -1.5, 0.5)]
    X = torch.zeros(E, Rp, wide, dtype=torch.bfloat16, device=DEV)
    X[:, :small] = (torch.randn(E, small, wide, generator=torch.Generator().manual_seed(r)) / (small * wide) ** 0.5).to(torch.bfloat16)
    seg = muon._uniform_segments(E, Rp, X.device)
    full = lambda *s: torch.full(s, float("nan"), dtype=torch.bfloat16, device=DEV)      # noqa: E731
    for n in (1, 3):
        ref = X
        for a, b, cc in coeffs[:n]:
            A, A2, nxt = full(E * Rp, Rp), full(E * Rp, Rp), full(E * Rp, wide)
            ops.expert_gram(ref.view(E * Rp, wide), seg, out=A)
            ops.expert_linear_axpby(A, A.view(E, Rp, Rp), A, cc, b, a, seg, out=A2, symmetric=2)
            ref = ops.expert_linear_t(A2, ref.view(E, Rp, wide), seg, out=nxt).view(E, Rp, wide)
        bufs = [X.clone(), full(E, Rp, wide)]
        A, A2 = full(E * Rp, Rp), full(E * Rp, Rp)
        flat = [v for abc in coeffs[:n] for v in abc]
        status = torch.zeros(1, dtype=torch.int32, device=DEV)
        rc = lib.b200moe_newton_schulz(bufs[0].data_ptr(), bufs[1].data_ptr(), A.data_ptr(), A2.data_ptr(), seg.tile_expert.data_ptr(),
                                       seg.poffs.data_ptr(), E, Rp, small, wide, (ctypes.c_float * len(flat))(*flat), n,
                                       status.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0 and int(status.item()) == 0
        assert torch.equal(bufs[n % 2][:, :small], ref[:, :small])
