"""CPU: host-side logic of the package that needs no kernel launch."""
import importlib
import os
import re

import torch

PKG = "triton-kernel-fused_b200"


def test_empty_batch_never_reaches_the_library():
    """T = 0: the public callables return empty results that still carry zero gradients, before any pointer is
    handed to the C ABI (so this runs without a GPU)."""
    pkg = importlib.import_module(PKG)
    H, I, E, k = 64, 32, 4, 2
    gu = torch.randn(E, 2 * I, H, requires_grad=True)
    dn = torch.randn(E, H, I, requires_grad=True)
    x = torch.zeros(0, H, requires_grad=True)
    w = torch.zeros(0, k, requires_grad=True)
    codes = torch.zeros(E, dtype=torch.int32)
    for fn in (pkg.moe, pkg.moe_grouped, pkg.moe_mxfp8):
        out = fn(x, torch.zeros(0, k, dtype=torch.int64), w, gu, dn, codes)
        assert out.shape == (0, H)
        gu.grad = dn.grad = None
        out.sum().backward()
        assert gu.grad.shape == gu.shape and float(gu.grad.abs().sum()) == 0.0
        assert dn.grad.shape == dn.shape and float(dn.grad.abs().sum()) == 0.0
    gate = torch.randn(E, H, requires_grad=True)
    idx, wts, counts = pkg.fused_mlp_router(torch.zeros(3, 0, H, requires_grad=True), gate, None, k, E,
                                            return_counts=True)
    assert idx.shape == (3, 0, k) and idx.dtype == torch.int64
    assert wts.shape == (3, 0, k) and wts.dtype == torch.float32
    assert counts.tolist() == [0] * E and counts.dtype == torch.int32
    wts.sum().backward()
    assert float(gate.grad.abs().sum()) == 0.0


def test_unknown_activation_codes_raise_value_error():
    pkg = importlib.import_module(PKG)
    H, I, E, k = 64, 32, 2, 1
    args = (torch.zeros(4, H), torch.zeros(4, k, dtype=torch.int64), torch.ones(4, k), torch.zeros(E, 2 * I, H),
            torch.zeros(E, H, I))
    try:
        pkg.moe(*args, torch.tensor([0, 9], dtype=torch.int32))
    except ValueError:
        return
    raise AssertionError("act code 9 must be rejected")


def test_muon_rejects_what_is_not_built_and_cpu_tensors():
    """Constructor checks of the optimizer and the device check of newton_schulz run before any launch."""
    import pytest
    pkg = importlib.import_module(PKG)
    p = torch.nn.Parameter(torch.zeros(2, 64, 64))
    for kw in (dict(scale_mode="no_such_mode"), dict(aurora_k=0), dict(ns_dtype=torch.float32),
               dict(xorth_post=0.1), dict(spectral_wd=0.1)):
        with pytest.raises(ValueError):
            pkg.FusedMuon([p], **kw)
    for mode in ("polar", "aurora", "normuon", "aurora_ema", "aurora_ema_v2"):     # every mode of the reference
        assert pkg.FusedMuon([p], scale_mode=mode, aurora_k=2, use_graph=True).scale_mode == mode
    opt = pkg.FusedMuon([p], lr=0.1, scale_mode="polar")
    opt.step()                                   # no gradient: nothing is stepped, nothing is launched
    assert float(p.detach().abs().sum()) == 0.0 and not opt.state[p]
    p.grad = torch.ones_like(p)
    with pytest.raises(ValueError):              # a CPU parameter never reaches the library
        opt.step()
    with pytest.raises(ValueError):
        pkg.newton_schulz(torch.zeros(8, 8))


def test_muon_uniform_segment_tables():
    """The row tables that stand in for a routing decision when the grouped GEMMs run over a stack."""
    pkg = importlib.import_module(PKG)
    seg = pkg.muon._uniform_segments(3, 512, "cpu")
    assert seg.cap == 1536 and seg.E == 3
    assert seg.poffs.tolist() == [0, 512, 1024, 1536]
    assert seg.tile_expert.tolist() == [0, 0, 1, 1, 2, 2]
    assert seg.tile_expert.dtype == torch.int32 and seg.poffs.dtype == torch.int32


def test_muon_accepts_the_reference_argument_list():
    """Every keyword of the reference's FusedMuon constructor is accepted; the ones that act only together with
    rejected options are ignored, a group that switches whitening on is rejected at step time."""
    import pytest
    pkg = importlib.import_module(PKG)
    p = torch.nn.Parameter(torch.zeros(2, 64, 64))
    opt = pkg.FusedMuon([{"params": [p], "xorth_post": 0.01}], lr=3e-4, momentum=0.95, nesterov=True, weight_decay=0.0,
                        ns_dtype=None, scale_mode="aurora", ns_batch_elems=4 * 1024 * 1024, use_graph=False,
                        graph_warmup=3, aurora_k=None, spectral_wd=0.0, swd_beta=0.99, xorth_post=0.0,
                        xorth_backend="ns", xorth_ns_iters=18, xorth_ema=0.95, xorth_gate_ref=0.3,
                        xorth_warmup_steps=0, xorth_where="post")
    p.grad = torch.zeros_like(p)
    with pytest.raises(ValueError):
        opt.step()


def test_muon_momentum_buffer_is_checked_before_the_kernel_sees_it():
    """A momentum buffer that `load_state_dict` cast to fp32 comes back as bf16 with the same values; a buffer of
    another size is refused (the kernel would otherwise read and write out of bounds)."""
    import pytest
    pkg = importlib.import_module(PKG)
    check = pkg.muon._checked_momentum
    cpu = torch.device("cpu")
    m = (torch.randn(2, 8, 16) * 0.1).to(torch.bfloat16)
    assert check(m, 2, 8, 16, cpu) is m                       # already right: passed through untouched
    back = check(m.float(), 2, 8, 16, cpu)
    assert back.dtype == torch.bfloat16 and torch.equal(back, m)
    flat = check(m.float().view(-1), 2, 8, 16, cpu)
    assert flat.shape == (2, 8, 16) and torch.equal(flat, m)
    for bad in (torch.zeros(1, 8, 16), torch.zeros(2, 8, 8), None):
        with pytest.raises(ValueError):
            check(bad, 2, 8, 16, cpu)


def test_status_codes_become_runtime_errors():
    """What a kernel leaves in the status word reaches the caller as a RuntimeError naming the cause; 7 is the
    cross-rank barrier that gave up waiting for a peer."""
    import pytest
    L = importlib.import_module(PKG + "._lib")
    L.raise_for_status(0)
    with pytest.raises(RuntimeError, match="peer rank did not arrive"):
        L.raise_for_status(7)
    with pytest.raises(RuntimeError, match="expert index"):
        L.raise_for_status(5)
    # argument errors of the barrier never reach the GPU
    lib = L.lib()
    assert lib.b200moe_ep_barrier(None, 2, 0, 1, 10**6, None, None) < 0
    assert b"status" in lib.b200moe_last_error_string()


def test_bf16_copies_of_frozen_stacks_are_reused_until_the_stack_changes():
    """fp32 / fp16 callers: the bf16 copy of an expert stack that needs no gradient is made once and reused until the
    stack is updated in place or freed; stacks that need a gradient are cast afresh (autograd needs the cast)."""
    moe_mod = importlib.import_module(PKG + ".moe")
    w = torch.randn(2, 8, 4)
    a = moe_mod._bf16_copy(w)
    assert a.dtype == torch.bfloat16 and moe_mod._bf16_copy(w) is a
    w.mul_(2.0)                                           # an optimizer step moves the version counter
    b = moe_mod._bf16_copy(w)
    assert b is not a and torch.equal(b, w.to(torch.bfloat16))
    p = torch.nn.Parameter(torch.randn(2, 8, 4))
    c = moe_mod._bf16_copy(p)
    assert c.requires_grad and moe_mod._bf16_copy(p) is not c
    with torch.no_grad():
        assert moe_mod._bf16_copy(p) is moe_mod._bf16_copy(p)
    n = len(moe_mod._BF16_COPIES)
    del w, a, b
    import gc
    gc.collect()
    assert len(moe_mod._BF16_COPIES) == n - 1             # freed with its tensor


def test_expert_groups_split_local_experts_by_rows():
    """The expert-parallel pipeline's grouping: consecutive experts, about equal padded rows, empty groups dropped,
    every row in exactly one group."""
    ep = importlib.import_module("triton-kernel-fused_b200.ep_p2p")
    ends = [256, 512, 768, 1024, 1280, 1536, 1792, 2048]
    assert ep.expert_groups(ends, 2) == [(0, 4, 0, 1024), (4, 8, 1024, 2048)]
    assert ep.expert_groups(ends, 4) == [(0, 2, 0, 512), (2, 4, 512, 1024), (4, 6, 1024, 1536), (6, 8, 1536, 2048)]
    assert ep.expert_groups(ends, 1) == [(0, 8, 0, 2048)]
    # one expert holds nearly everything: the cut falls behind it, nothing is lost, nothing is empty
    skew = [256, 256, 5120, 5376]
    for n in (2, 3, 4, 7):
        g = ep.expert_groups(skew, n)
        assert g[0][0] == 0 and g[-1][1] == 4 and g[0][2] == 0 and g[-1][3] == 5376
        assert all(a[1] == b[0] and a[3] == b[2] for a, b in zip(g, g[1:]))
        assert all(r_hi > r_lo for _, _, r_lo, r_hi in g)
    # experts without rows (ends repeat) and a rank without any row
    assert ep.expert_groups([0, 0, 256, 256], 2) == [(0, 3, 0, 256)] or ep.expert_groups([0, 0, 256, 256], 2) == [(0, 4, 0, 256)]
    assert ep.expert_groups([0, 0, 0, 0], 2) == []
    assert ep.expert_groups([], 2) == []


def test_load_telemetry_figures():
    """`load_stats` of the layers' load-balance mixin: the figures follow from the accumulated counts."""
    layer_mod = importlib.import_module("triton-kernel-fused_b200.layer")

    class Loop(layer_mod.LoadBalanceMixin, torch.nn.Module):
        def __init__(self):
            super().__init__()
            self._init_load(4)

    loop = Loop()
    assert loop.load_stats() == {"load": [0, 0, 0, 0], "tokens_routed": 0, "max_over_mean": 0.0, "min_over_mean": 0.0,
                                 "cv": 0.0, "idle_experts": 4}
    loop._record_counts(torch.tensor([6, 2, 0, 0], dtype=torch.int32))
    loop._record_counts(torch.tensor([2, 2, 4, 0], dtype=torch.int32))
    st = loop.load_stats()
    assert st["load"] == [8, 4, 4, 0] and st["tokens_routed"] == 16 and st["idle_experts"] == 1
    assert st["max_over_mean"] == 2.0 and st["min_over_mean"] == 0.0
    assert abs(st["cv"] - (8.0 ** 0.5) / 4.0) < 1e-12          # std of (8,4,4,0) = sqrt(8), mean 4


def test_fixed_capacity_rows():
    """Sizing of the expert-parallel layer's fixed-capacity buffers: factor x own routed rows, rounded up, clamped to
    the rows that exist; nonsense factors are refused before anything is allocated."""
    import pytest
    ep = importlib.import_module("triton-kernel-fused_b200.ep_p2p")
    assert ep.fixed_capacity_rows(8, 16384, 6, 1.5) == 147456
    assert ep.fixed_capacity_rows(8, 1000, 3, 1.0001) == 3001          # rounded up
    assert ep.fixed_capacity_rows(2, 1024, 4, 5.0) == 2 * 4096          # never more rows than exist
    assert ep.fixed_capacity_rows(4, 10, 2, 0.25) == 5
    for bad in (0, -1.0, float("nan")):
        with pytest.raises(ValueError):
            ep.fixed_capacity_rows(2, 8, 2, bad)


def test_workspaces_are_sized_for_every_sm_budget():
    """The split products take fewer slices while SMs are reserved; a workspace sized before or after holds them."""
    lib = importlib.import_module(PKG).lib()
    sizes = lambda: [f(*a) for f, cases in (     # noqa: E731
        (lib.b200moe_router_bwd_ws_bytes, [(16384, 2048, 64), (100, 256, 256)]),
        (lib.b200moe_conv_router_bwd_ws_bytes, [(16, 1024, 2048, 64, 4), (2, 100, 256, 8, 2)]),
        (lib.b200moe_conv_router_fwd_ws_bytes, [(341, 48, 2048, 64, 4), (300, 32, 2048, 64, 4)]),
        (lib.b200moe_layer_bwd_ws_bytes, [(16384, 2048, 1408, 64, 6)])) for a in cases]
    full = sizes()
    try:
        for n in (2, 60, 146):
            assert lib.b200moe_set_reserved_sms(n) == 0
            assert sizes() == full
    finally:
        lib.b200moe_set_reserved_sms(0)


def test_workspace_of_nothing_is_no_bytes():
    """Every workspace size takes an empty batch, width or stack: no bytes (the launches refuse such calls), never a signal."""
    lib = importlib.import_module(PKG).lib()
    full = {"moe_fwd": (4, 256, 512, 8, 8, 2, 1, 0), "moe_bwd": (4, 256, 512, 8, 8, 2, 0), "layer_fwd": (4, 256, 512, 8, 2, 1),
            "layer_bwd": (4, 256, 512, 8, 2), "router_bwd": (4, 256, 8), "conv_router_bwd": (2, 4, 256, 8, 3),
            "conv_router_fwd": (2, 4, 264, 8, 3)}
    extents = {"moe_fwd": (0, 1, 2, 3, 5), "moe_bwd": (0, 1, 2, 3, 5)}
    for name, args in full.items():
        size = getattr(lib, f"b200moe_{name}_ws_bytes")
        assert size(*args) > 0
        for i in extents.get(name, range(min(5, len(args)))):
            for v in (0, -3):
                assert size(*args[:i], v, *args[i + 1:]) == 0, (name, i, v)
    assert lib.b200moe_router_backward(16, 16, 16, 16, 16, 0, 256, 8, 2, 1, 1.0, 16, 16, 16, 16, None) != 0


def test_backward_of_given_picks_needs_all_of_its_buffers():
    """A moe backward without a place for the weights' gradient (or for any operand) is refused before anything is launched; the other gradients
    may be left out."""
    lib = importlib.import_module(PKG).lib()
    args = [16, 16, 16, 16, None, None, 4, 256, 512, 8, 8, 2, 0, 16, 16, None, 16, None, None, None, 16, None]
    null = lib.b200moe_layer_forward(None, 16, None, 16, 16, None, 4, 256, 512, 8, 2, 1, 1.0, 1, 16, 16, None, 16, 16, None)
    assert null != 0
    for i in (0, 1, 2, 3, 13, 14, 16):
        bad = list(args)
        bad[i] = None
        assert lib.b200moe_moe_backward(*bad) == null, i


def test_route_of_a_forward_without_backward():
    """Compact rows or row tiles: the workspace of the latter is that of a forward with a backward (it holds gate_up and the
    padded rows).  (experts, d_model, d_ff, picks, tokens, compact?): decoding; both sides of the limits on the mean rows of
    many and of few experts; a small stack inside and past one wave of 64-row chunks; a stack of half the SMs and one of more."""
    size = importlib.import_module(PKG).lib().b200moe_moe_fwd_ws_bytes
    for E, H, I, k, T, compact in ((64, 2048, 1408, 6, 1, True), (64, 2048, 1408, 6, 1706, True), (64, 2048, 1408, 6, 1707, False),
                                   (8, 4096, 14336, 2, 440, True), (8, 4096, 14336, 2, 441, False), (16, 2048, 1408, 4, 640, True),
                                   (16, 2048, 1408, 4, 641, False), (8, 512, 256, 2, 640, True), (8, 512, 256, 2, 641, False),
                                   (8, 1024, 1024, 2, 351, True), (8, 1024, 1024, 2, 352, False), (8, 1024, 1280, 2, 352, True)):
        kept, quiet = (size(T, H, I, E, E, k, keep, 0) for keep in (1, 0))
        assert (quiet < kept) == compact, (E, H, I, k, T)


def test_rows_of_a_forward_without_backward_are_padded_where_products_read_them():
    """With a backward to follow, every buffer's rows lie at whole lines; without, those of x_s and inter where their product has more than 512 columns
    or they are 448 wide, those of the others where they are 1280 wide.  Told from the workspaces' sizes (rows are multiples of 256, so each difference is exact)."""
    lib = importlib.import_module(PKG).lib()
    pitch = lambda n: n if n % 32 == 0 else (n + 63) // 64 * 64     # noqa: E731
    read = lambda n, cols: pitch(n) if cols > 512 or n >= 448 else n     # noqa: E731
    written = lambda n: pitch(n) if n >= 1280 else n     # noqa: E731
    T, E, k = 9000, 16, 4
    rows = lib.b200moe_padded_rows_cap(T * k, E)
    for row_kernels in (0, 1):
        for H, I in ((360, 256), (136, 72), (264, 520), (520, 264), (512, 200), (520, 200), (440, 256), (456, 256), (440, 264), (256, 440), (256, 456), (256, 256), (1288, 648), (1272, 632)):
            kept, quiet = (lib.b200moe_moe_fwd_ws_bytes(T, H, I, E, E, k, keep, row_kernels) for keep in (1, 0))
            less = 2 * pitch(H) + pitch(2 * I) + pitch(I) - (read(H, 2 * I) + written(H) + written(2 * I) + read(I, H))
            assert kept - quiet == 2 * rows * less, (H, I, row_kernels)


def test_chained_kernels_promise_no_constant_data():
    """A chained kernel (one with a grid_dep_wait) starts while the kernel before it still writes what it reads: none of its
    pointers may be __restrict__, nothing in its file read through the non-coherent path, and it waits."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), PKG, "csrc")
    seen = 0
    sources = {f: re.sub(r"//[^\n]*", "", open(os.path.join(csrc, f)).read()) for f in os.listdir(csrc) if f.endswith((".cu", ".cuh"))}
    for name, text in sources.items():
        for kernel in re.split(r"(?=\b__global__\b)", text)[1:]:
            head, body = kernel.split("{", 1)
            if not re.search(r"\bgrid_dep_(wait|begin|launch)\(", body):
                continue
            seen += 1
            assert "__restrict__" not in head, (name, head)
            assert re.search(r"\bgrid_dep_(wait|begin)\(", body), (name, head)
            assert not re.search(r"__ldg\(|ld\.global\.nc", text), name
    assert seen >= 25
    for shared in ("common.cuh", "ptx.cuh", "gemm_common.cuh", "few_tiles.cuh", "topk.cuh", "mxfp8_quant.cuh"):
        assert not re.search(r"__ldg\(|ld\.global\.nc", sources[shared]), shared


def test_chained_kernels_wait_before_they_read():
    """Every chained kernel waits for the one before it, in all of its threads, before it lets the next one begin and before it names what its
    pointers point to.  The few-rows kernel's loads of weights ahead of its wait are the only exception."""
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), PKG, "csrc")
    sources = {f: re.sub(r"//[^\n]*", "", open(os.path.join(csrc, f)).read()) for f in os.listdir(csrc) if f.endswith((".cu", ".cuh"))}
    exceptions = []
    for name, text in sources.items():
        for kernel in re.split(r"(?=\b__global__\b)", text)[1:]:
            head, body = kernel.split("{", 1)
            calls = list(re.finditer(r"\bgrid_dep_(\w+)\(", body))
            if not calls:
                continue
            title = re.search(r"(\w+)\s*\(", re.sub(r"__launch_bounds__\(.*?\)\)?", "", head, flags=re.S)).group(1)
            assert {c.group(1) for c in calls} <= {"wait", "begin", "launch"}, (name, title)
            before = body[:calls[0].start()]
            if re.search(r"(\)|\belse|[?:&|])\s*$", before):                        # the wait hangs on a condition
                exceptions.append(title)
                continue
            assert before.count("{") == before.count("}") and calls[0].group(1) in ("wait", "begin"), (name, title)
            for pointer in re.findall(r"\*\s*(?:const\s+)?(\w+)\s*[,)]", head):
                assert not re.search(r"\b%s\b" % pointer, before), (name, title, pointer)
    assert exceptions == ["few_rows_kernel"]


def test_kept_copies_of_stacks_are_safe_on_other_streams(monkeypatch):
    """Quantised and bf16 copies that one stream made: a call on another stream waits for it before it reads them, until they are
    known to be complete, and records itself as a user of their memory; the stream that made them does neither (the default stream records its event when one is asked for)."""
    moe_mod, mx, L = (importlib.import_module(PKG + n) for n in (".moe", ".mxfp8", "._lib"))
    log = []

    class Event:
        done = False

        def query(self):
            return self.done

    class Stream:
        def __init__(self, name):
            self.name, self.cuda_stream = name, 0 if name == "default" else hash(name)

        def record_event(self):
            log.append(("record", self.name))
            return Event()

        def wait_event(self, e):
            log.append(("wait", self.name))

    class Copy:
        is_cuda, device = True, torch.device("cuda", 0)

        def record_stream(self, s):
            log.append(("used by", s.name))

        def to(self, _):
            return self

        detach = lambda self: self     # noqa: E731
        data_ptr = lambda self: 16     # noqa: E731

    now = [Stream("a")]
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d=None: now[0])
    monkeypatch.setattr(torch.cuda, "default_stream", lambda d=None: Stream("default"))
    monkeypatch.setattr(L, "capturing", lambda t: False)
    monkeypatch.setattr(L, "stream_of", lambda t: now[0].cuda_stream)

    class Master(Copy):
        requires_grad, _version = False, 0

    for maker in ("a", "default"):
        stack, master, q = torch.zeros(2), Master(), (Copy(), Copy())
        for get in (lambda: mx._quantised_weights(stack, lambda: q, None, False), lambda: moe_mod._bf16_copy(master)):
            now[0], Event.done = Stream(maker), False
            log.clear()
            res = get()
            users = [("used by", "b")] * (len(res) if isinstance(res, tuple) else 1)
            get()
            made = [] if maker == "default" else [("record", "a")]
            assert log == made
            now[0] = Stream("b")
            assert get() == res
            assert log == [("record", maker), ("wait", "b")] + users
            Event.done = True
            log.clear()
            get()
            get()
            assert log == 2 * users
        del mx._QUANTISED[id(stack)], moe_mod._BF16_COPIES[id(master)]


def test_copies_made_under_capture_are_not_kept(monkeypatch):
    """A copy queued into a graph is filled by replays only and lies in the graph's memory: no later call may get it.  A captured
    forward reads kept copies; a captured pass with a backward makes its own, because its weights change between replays."""
    moe_mod, mx, L = (importlib.import_module(PKG + n) for n in (".moe", ".mxfp8", "._lib"))
    capturing = [True]
    monkeypatch.setattr(L, "capturing", lambda t: capturing[0])
    stack, made = torch.zeros(2, 4, 8), []
    get = lambda **kw: mx._quantised_weights(stack, lambda: made.append(0) or (torch.zeros(1), torch.zeros(1)), None, False, **kw)     # noqa: E731
    get()
    assert id(stack) not in mx._QUANTISED
    capturing[0] = False
    kept = get()
    assert len(made) == 2 and get()[0] is kept[0]
    capturing[0] = True
    assert get()[0] is kept[0] and get(keep=True)[0] is not kept[0] and len(made) == 3
    capturing[0] = False
    assert get(keep=True)[0] is kept[0]
    w = torch.randn(2, 8, 4)
    capturing[0] = True
    a = moe_mod._bf16_copy(w)
    assert id(w) not in moe_mod._BF16_COPIES
    capturing[0] = False
    b = moe_mod._bf16_copy(w)
    assert b is not a
    capturing[0] = True
    assert moe_mod._bf16_copy(w) is b


def test_bf16_copies_follow_assigned_data():
    """Assigning `.data` (what module.to() and weight swaps do) moves no version counter: the copy is made anew all the same."""
    moe_mod = importlib.import_module(PKG + ".moe")
    w = torch.randn(2, 8, 4)
    a = moe_mod._bf16_copy(w)
    w.data = torch.randn(2, 8, 4)
    b = moe_mod._bf16_copy(w)
    assert b is not a and torch.equal(b, w.to(torch.bfloat16)) and moe_mod._bf16_copy(w) is b
