"""GPU: the activation row kernels where gates saturate: what is left of 1 - sigmoid and 1 - tanh^2 is as exact there as anywhere."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
BINS = [(-104, -88.75), (-88.7, -87.35), (-87, -40), (-40, -15), (-15, -12), (-12, -10), (-10, -8), (-8, -3), (3, 8), (8, 10), (10, 12), (12, 15), (15, 40), (40, 88)]


def _rows(rows, code, alpha=1.0, gamma=1.0):
    perm = types.SimpleNamespace(cap=rows, E=1, tile_expert=torch.zeros(rows // 256, dtype=torch.int32, device=DEV),
                                 poffs=torch.tensor([0, rows], dtype=torch.int32, device=DEV),
                                 total_rows=torch.tensor([rows], dtype=torch.int32, device=DEV))
    return perm, torch.tensor([code], dtype=torch.int32, device=DEV), torch.tensor([[alpha, gamma]], device=DEV)


# 1024 values a row: no lane idle; 776: some are (both of three vectors a thread or less)
@pytest.mark.parametrize("I", [776, 1024])
@pytest.mark.parametrize("code", [0, 5])
def test_saturated_gates_against_float64(pkg, code, I):
    R = 256
    alpha, gamma = (0.9, 1.1) if code == 5 else (1.0, 1.0)
    perm, cd, pr = _rows(R, code, alpha, gamma)
    alpha, gamma = (float(v) for v in pr[0].double())                                      # as rounded to fp32
    g = torch.Generator(device=DEV).manual_seed(code)
    for lo, hi in BINS:
        gate = (torch.rand(R, I, generator=g, device=DEV) * (hi - lo) + lo).bfloat16()
        one = torch.ones(R, I, dtype=torch.bfloat16, device=DEV)
        gate_up = torch.cat([gate, one], 1)
        inter = pkg.ops.glu_fwd_rows(gate_up, cd, pr, perm)
        ggu, da, dg = pkg.ops.glu_bwd_rows(one, gate_up, cd, pr, perm, True)
        G = gate.double()
        s, rest = torch.sigmoid(G), torch.sigmoid(-G)
        b = torch.exp(-2 * (alpha * G).abs())
        t, dt = torch.sign(G) * (1 - b) / (1 + b), 4 * b / (1 + b) ** 2
        act, d = (G * s, s * (1 + G * rest)) if code == 0 else (gamma * t * s, gamma * (alpha * dt * s + t * s * rest))
        # One rounding to bf16, 2^-8, or half the step of its subnormal numbers, 2^-134; before it an exponential of up to 2 * 104 (its argument is off by 2^-24 of
        # itself, 2^-16 of the result) and ten roundings.  Below 2^-126 an exponential is subnormal: off by up to two of their steps, 2^-148, times the gate.
        for name, got, want in (("act", inter, act), ("grad_up", ggu[:, I:], act), ("grad_gate", ggu[:, :I], d)):
            bound = (2.0 ** -8 + 2.0 ** -15) * want.abs() + 2.0 ** -134 + 2.0 ** -141
            assert ((got.double() - want).abs() <= bound).all(), (name, lo, hi)
        if code == 5 and max(-lo, hi) <= 40:          # sums of numbers of one sign: 2^-16 each, and those of the additions
            want = (gamma * G * dt * s).sum(1), (t * s).sum(1)
            for name, got, w in zip(("alpha", "gamma"), (da, dg), want):
                assert ((got.double() - w).abs() <= 2.0 ** -15 * w.abs()).all(), (name, lo, hi)


def test_saturated_gates_of_a_norm_code(pkg):
    """Code 7: a row of small gates and four large ones, which are sixteen times its root mean square."""
    R, I = 256, 1024
    perm, cd, pr = _rows(R, 7)
    g = torch.Generator(device=DEV).manual_seed(0)
    gate = torch.randn(R, I, generator=g, device=DEV) * 0.01
    gate[:, ::256] = (torch.rand(R, 4, generator=g, device=DEV) + 1) * torch.tensor([1.0, -1.0, 1.0, -1.0], device=DEV)
    gate_up = torch.cat([gate, torch.randn(R, I, generator=g, device=DEV)], 1).bfloat16()
    go = torch.randn(R, I, generator=g, device=DEV).bfloat16()
    inter = pkg.ops.glu_fwd_rows(gate_up, cd, pr, perm)
    ggu = pkg.ops.glu_bwd_rows(go, gate_up, cd, pr, perm)
    ggu = ggu[0] if isinstance(ggu, tuple) else ggu
    G, U = gate_up[:, :I].double().requires_grad_(), gate_up[:, I:].double().requires_grad_()
    n = G * torch.rsqrt(G.pow(2).mean(1, keepdim=True) + 1e-6)
    assert n.abs().max() > 10
    out = torch.tanh(n) * torch.sigmoid(n) * U
    out.backward(go.double())
    for name, got, want in (("inter", inter, out.detach()), ("grad_gate", ggu[:, :I], G.grad), ("grad_up", ggu[:, I:], U.grad)):
        err = (got.double() - want).norm() / want.norm()
        assert err < 2.0 ** -9, (name, float(err))            # a rounding to bf16: at most that


# 1024 values fill the lanes of a row, 776 and 72 do not, which must change nothing
@pytest.mark.parametrize("I", [72, 776, 1024])
@pytest.mark.parametrize("alpha,gamma", [(float("inf"), 1.5), (0.75, float("inf")), (float("-inf"), 1.0)])
def test_infinite_parameters_reach_the_sums_through_values_only(pkg, I, alpha, gamma):
    """An infinite alpha saturates tanh: its own gradient is 0 and that of gamma stays a number; an infinite gamma leaves its own gradient a number."""
    R = 256
    perm, cd, pr = _rows(R, 5, alpha, gamma)
    g = torch.Generator(device=DEV).manual_seed(I)
    gate = ((torch.rand(R, I, generator=g, device=DEV) + 0.5) * (1 - 2 * (torch.rand(R, I, generator=g, device=DEV) < 0.5).float())).bfloat16()
    up, go = (torch.randn(R, I, generator=g, device=DEV).bfloat16() for _ in range(2))
    _, da, dg = pkg.ops.glu_bwd_rows(go, torch.cat([gate, up], 1), cd, pr, perm, True)
    G, w = gate.double(), go.double() * up.double()
    want = w * torch.tanh(alpha * G) * torch.sigmoid(G)
    # sums of I fp32 values, each off by a few roundings, in any order
    assert ((dg.double() - want.sum(1)).abs() <= I * 2.0 ** -23 * want.abs().sum(1)).all()
    if gamma != float("inf"):
        assert (da == 0).all()
