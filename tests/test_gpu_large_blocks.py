"""GPU: a token's results do not depend on how many others its block holds, and large blocks are as exact as small ones."""
import pytest
import torch

from oracle import moe_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROUND = 2 ** -9      # a bf16 rounding moves a value by at most 2^-9 of its binade; n of them, independent: sqrt(n) of it


def _run(pkg, x, idx, w, gu, dn, codes, go):
    leaves = [t.clone().requires_grad_() for t in (x, w, gu, dn)]
    out = pkg.moe(leaves[0], idx, leaves[1], leaves[2], leaves[3], codes)
    return [out.detach()] + list(torch.autograd.grad(out, leaves, go))


def _exact(x, idx, w, gu, dn, codes, go):
    leaves = [t.detach().double().requires_grad_() for t in (x, w, gu, dn)]
    X, W, GU, DN = leaves
    out = torch.zeros_like(X)
    for e in range(GU.shape[0]):
        t, j = (idx == e).nonzero(as_tuple=True)
        g, u = (X[t] @ GU[e].t()).chunk(2, dim=1)
        a = {0: lambda v: v * torch.sigmoid(v), 1: lambda v: torch.relu(v) ** 2, 5: lambda v: torch.tanh(v) * torch.sigmoid(v)}[int(codes[e])](g)
        out = out.index_add(0, t, ((a * u) @ DN[e].t()) * W[t, j, None])
    return [out.detach()] + list(torch.autograd.grad(out, leaves, go.double()))


# 64 MiB of routed rows and more, the halves less: single-CTA and pair tiles, columns that fill no tile of 128 or 256; one expert without rows, weights of
# zero and below
@pytest.mark.parametrize("T,H,I,E,k,mixed", [(8200, 1032, 200, 6, 4, False), (4100, 2048, 328, 9, 4, True), (32776, 520, 72, 5, 2, False),
                                             (8200, 1032, 680, 16, 4, True)])
def test_block_equals_its_halves(pkg, T, H, I, E, k, mixed):
    assert T * k * H * 2 >= 64 << 20 > T // 2 * k * H * 2
    g = torch.Generator(device=DEV).manual_seed(I)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)     # noqa: E731
    x, go = rand(T, H).bfloat16(), rand(T, H).bfloat16()
    gu, dn = (rand(E, 2 * I, H) * H ** -0.5).bfloat16(), (rand(E, H, I) * I ** -0.5).bfloat16()
    idx = torch.rand(T, E - 1, generator=g, device=DEV).topk(k, 1).indices          # nothing for the last expert
    w = torch.rand(T, k, generator=g, device=DEV) - 0.1
    w[::7, 0] = 0.0
    codes = torch.tensor([(0, 1, 5)[e % 3] if mixed else 0 for e in range(E)], dtype=torch.int32, device=DEV)
    got = _run(pkg, x, idx, w, gu, dn, codes, go)
    h = T // 2
    halves = [_run(pkg, x[s], idx[s], w[s], gu, dn, codes, go[s]) for s in (slice(0, h), slice(h, T))]
    pkg.check_status()
    for name, a, b, c in zip(("out", "grad_x", "grad_w"), got, *halves):
        assert torch.equal(a, torch.cat([b, c])), name
    ref = _exact(x, idx, w, gu, dn, codes, go)
    # roundings on the way: out gate, up, inter, row, out; grad_x w go, gate, up, grad_inter, grad_gate, grad_up, row, grad_x; grad_w gate, up, inter, row;
    # grad_gate_up w go, gate, up, grad_inter, grad_gate / up, result; grad_down w go, gate, up, inter, result.  Twice that for their uneven weights.
    for name, a, r, n in zip(("out", "grad_x", "grad_w", "grad_gate_up", "grad_down"), got, ref, (5, 8, 4, 6, 5)):
        err = O.rel_l2(a.double(), r)
        assert torch.isfinite(a).all() and err < 2 * n ** 0.5 * ROUND, (name, err)
    assert (got[3][-1] == 0).all() and (got[4][-1] == 0).all()


def test_gradients_of_a_subset_of_a_large_block(pkg):
    """Products that only unwanted gradients need are left out; the others stay what they were, to the bit."""
    g = torch.Generator(device=DEV).manual_seed(0)
    T, H, I, E, k = 8200, 1032, 136, 4, 4
    rand = lambda *s: (torch.randn(*s, generator=g, device=DEV) * 0.05).bfloat16()     # noqa: E731
    x, go, gu, dn = rand(T, H), rand(T, H), rand(E, 2 * I, H), rand(E, H, I)
    idx = torch.rand(T, E, generator=g, device=DEV).topk(k, 1).indices
    w, codes = torch.rand(T, k, generator=g, device=DEV), torch.zeros(E, dtype=torch.int32, device=DEV)
    full = _run(pkg, x, idx, w, gu, dn, codes, go)
    for i in range(4):
        leaves = [t.clone().requires_grad_(i == j) for j, t in enumerate((x, w, gu, dn))]
        out = pkg.moe(leaves[0], idx, leaves[1], leaves[2], leaves[3], codes)
        assert torch.equal(torch.autograd.grad(out, [leaves[i]], go)[0], full[i + 1]), i
    pkg.check_status()
