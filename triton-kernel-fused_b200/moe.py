"""Expert pipeline of the MoE block behind the reference's callables.

Mirrors kernels/sm75/moe.py: `moe` (:838), `moe_grouped` (:621), `moe_per_expert` (:829) keep their
signatures and return the (N,H) combined output; all three run the one sm_100a path
(device-side counting sort -> gather -> grouped tcgen05 GEMMs with fused SwiGLU -> weighted
gather-combine), with a hand-written backward (dgrad + wgrad grouped GEMMs, fused GLU backward).
"""
from __future__ import annotations

import torch

from . import _lib as L

__all__ = ["moe", "moe_grouped", "moe_per_expert", "GROUPED_MIN_TOKENS"]

GROUPED_MIN_TOKENS = 4096   # kept for API compatibility (kernels/sm75/moe.py:78); one path here


def _amp_cast(*ts):
    """Under CUDA autocast cast float tensors to the autocast dtype (kernels/sm75/moe.py:97-104)."""
    if torch.is_autocast_enabled("cuda"):
        dt = torch.get_autocast_dtype("cuda")
        return tuple(t.to(dt) if t.is_floating_point() else t for t in ts)
    return ts


def _float32(t):
    return t if t.dtype == torch.float32 and t.is_contiguous() else t.float().contiguous()


def _codes_on(act_codes, device):
    c = act_codes
    if c.device != device or c.dtype != torch.int32 or not c.is_contiguous():
        c = c.to(device=device, dtype=torch.int32).contiguous()
    return c


def _check_experts(hidden, idx, wt, gate_up_proj, down_proj):
    for name, t in (("hidden", hidden), ("gate_up_proj", gate_up_proj), ("down_proj", down_proj)):
        L.require_cuda_bf16(name, t)
    L.require(hidden.dim() == 2 and gate_up_proj.dim() == 3, "hidden must be (N,H), gate_up_proj (E,2I,H)")
    (N, H), (E, twoI, H2) = hidden.shape, gate_up_proj.shape
    L.require(H2 == H and twoI % 2 == 0 and tuple(down_proj.shape) == (E, H, twoI // 2),
              f"weight shapes must be (E,2I,H) and (E,H,I); got {tuple(gate_up_proj.shape)}, {tuple(down_proj.shape)}")
    L.require(idx.is_cuda and idx.dtype == torch.int64 and idx.dim() == 2, "top_k_indices must be a CUDA int64 (N,k) tensor")
    L.require(idx.shape == wt.shape and idx.shape[0] == N, "indices/weights must be (N,k)")
    L.require(hidden.device == idx.device == gate_up_proj.device == down_proj.device, "all tensors must be on one device")


def _experts_forward(ctx, hidden, idx, wt, gate_up_proj, down_proj, codes_dev, params, E, row_kernels, keep):
    """One native call (csrc/block.cu); a forward that is followed by a backward keeps its workspace, in which the
    backward finds x_s, gate_up, inter, eo and the permutation tables."""
    hidden, gate_up_proj, down_proj = hidden.contiguous(), gate_up_proj.contiguous(), down_proj.contiguous()
    idx, w32, dev = idx.contiguous(), _float32(wt.detach()), hidden.device
    L.require(w32.device == dev, "top_k_weights must be on hidden's device")
    (N, H), n_glu, I, k = hidden.shape, gate_up_proj.shape[0], down_proj.shape[2], idx.shape[1]
    lib = L.lib()
    ws = L.workspace(lib.b200moe_moe_fwd_ws_bytes(N, H, I, E, n_glu, k, keep, row_kernels), dev)
    out = torch.empty(N, H, dtype=torch.bfloat16, device=dev)
    L.check(lib.b200moe_moe_forward(hidden.data_ptr(), idx.data_ptr(), w32.data_ptr(), gate_up_proj.data_ptr(),
                                    down_proj.data_ptr(), L.ptr(codes_dev), L.ptr(params), N, H, I, E, n_glu, k, keep,
                                    row_kernels, ws.data_ptr(), out.data_ptr(), L.status_word(dev).data_ptr(),
                                    L.stream_of(hidden)))
    if keep:
        ctx.dims = (N, H, I, E, n_glu, k, row_kernels)
        ctx.wt_dtype = wt.dtype
        ctx.save_for_backward(ws, w32, gate_up_proj, down_proj, codes_dev, params)
    return out


def _experts_backward(ctx, grad_out, need, want_params):
    """(grad_hidden, grad_wt, grad_gate_up_proj, grad_down_proj, grad_params), None where not needed."""
    ws, w32, gate_up_proj, down_proj, codes_dev, params = ctx.saved_tensors
    N, H, I, E, n_glu, k, row_kernels = ctx.dims
    need_x, _, need_w, need_gu, need_dn = need
    dev = ws.device
    grad_out = grad_out.to(torch.bfloat16).contiguous()
    lib, bf16 = L.lib(), dict(dtype=torch.bfloat16, device=dev)
    grad_w = torch.empty(N, k, dtype=torch.float32, device=dev)
    grad_x = torch.empty(N, H, **bf16) if need_x else None
    grad_gu = torch.empty(n_glu, 2 * I, H, **bf16) if need_gu else None
    grad_dn = torch.empty(n_glu, H, I, **bf16) if need_dn else None
    grad_ap = torch.empty(E, 2, dtype=torch.float32, device=dev) if want_params and params is not None else None
    tmp = L.workspace(lib.b200moe_moe_bwd_ws_bytes(N, H, I, E, n_glu, k, row_kernels), dev)
    L.check(lib.b200moe_moe_backward(grad_out.data_ptr(), w32.data_ptr(), gate_up_proj.data_ptr(), down_proj.data_ptr(),
                                     L.ptr(codes_dev), L.ptr(params), N, H, I, E, n_glu, k, row_kernels, ws.data_ptr(),
                                     tmp.data_ptr(), L.ptr(grad_x), grad_w.data_ptr(), L.ptr(grad_gu), L.ptr(grad_dn),
                                     L.ptr(grad_ap), L.status_word(dev).data_ptr(), L.stream_of(ws)))
    return grad_x, (grad_w.to(ctx.wt_dtype) if need_w else None), grad_gu, grad_dn, grad_ap


class _GroupedMoE(torch.autograd.Function):
    """Activation in the GEMM epilogues.  The forward keeps x_s, gate_up, inter, eo and the permutation tables, as the
    reference's grouped Function does (kernels/sm75/moe.py:576-599); backward follows :602-618."""

    @staticmethod
    def forward(ctx, hidden, idx, wt, gate_up_proj, down_proj, act_codes, keep=True):
        """keep=False: no backward will follow (the caller knows the grad mode, which is off in here)."""
        hidden, gate_up_proj, down_proj = _amp_cast(hidden, gate_up_proj, down_proj)
        _check_experts(hidden, idx, wt, gate_up_proj, down_proj)
        E = gate_up_proj.shape[0]
        L.require(act_codes.numel() == E, "act_codes must have one code per expert")
        # a stack that mixes the parameter-free codes 0 / 1 / 5 keeps the fused epilogues: the code of a tile's
        # expert picks the activation there; an all-SiLU stack runs the SiLU-only instantiations
        codes_dev = _codes_on(act_codes, hidden.device) if any(_code_info(act_codes)[0]) else None
        return _experts_forward(ctx, hidden, idx, wt, gate_up_proj, down_proj, codes_dev, None, E, 0, int(keep))

    @staticmethod
    def backward(ctx, grad_out):
        gx, gw, ggu, gdn, _ = _experts_backward(ctx, grad_out, ctx.needs_input_grad[:5], False)
        return (gx, None, gw, ggu, gdn, None, None)[:len(ctx.needs_input_grad)]


GLU_CODES = (0, 1, 2, 5, 6, 7)     # weight-carrying experts (kernels/sm75/moe.py:1-31)
FUSED_CODES = (0, 1, 5)            # applied inside the GEMM epilogues (no row reduction, no parameters)
SPECIAL_CODES = (3, 4)             # Identity, Zero: expert kinds without weights, listed after the GLU experts


def _code_info(act_codes: torch.Tensor):
    """(codes tuple, number of GLU experts), read from the device once per tensor lifetime: act_codes
    is static model config (the reference reads it with .tolist() on every call, moe.py:741)."""
    info = getattr(act_codes, "_code_info_cache", None)
    if info is None:
        codes = tuple(int(c) for c in act_codes.tolist())
        for c in codes:
            if c not in GLU_CODES + SPECIAL_CODES:
                raise ValueError(f"unknown act code {c}; supported: 0 SiLU, 1 ReLU^2, 2 NormSiLU, 3 Identity, "
                                 "4 Zero, 5 SiTU, 6 NormReLU^2, 7 NormSiTU")
        n_glu = sum(1 for c in codes if c in GLU_CODES)
        if any(c in SPECIAL_CODES for c in codes[:n_glu]):
            raise ValueError("GLU act codes must precede the Identity/Zero experts in act_codes")
        info = (codes, n_glu)
        try:
            act_codes._code_info_cache = info
        except Exception:
            pass
    return info


class _PolyGLUMoE(torch.autograd.Function):
    """Generic path for stacks that are not pure SiLU-GLU: the same sort / GEMMs / combine, with the
    activation as row kernels between the GEMMs (Norm codes need a row reduction over d_ff) and the
    Identity / Zero experts handled on their rows.  Mirrors _PerExpertMoE (kernels/sm75/moe.py:724-826)."""

    @staticmethod
    def forward(ctx, hidden, idx, wt, gate_up_proj, down_proj, act_codes, act_params):
        hidden, gate_up_proj, down_proj = _amp_cast(hidden, gate_up_proj, down_proj)
        _check_experts(hidden, idx, wt, gate_up_proj, down_proj)
        codes, n_glu = _code_info(act_codes)
        E_total, E = len(codes), gate_up_proj.shape[0]
        L.require(E == n_glu, f"gate_up_proj holds {E} experts but act_codes lists {n_glu} GLU experts")
        ap32 = None
        if act_params is not None:
            L.require(tuple(act_params.shape) == (E_total, 2), "act_params must be (E,2) [alpha, gamma]")
            ap32 = _float32(act_params.detach())
            L.require(ap32.device == hidden.device, "act_params must be on hidden's device")
        return _experts_forward(ctx, hidden, idx, wt, gate_up_proj, down_proj, _codes_on(act_codes, hidden.device), ap32,
                                E_total, 1, 1)

    @staticmethod
    def backward(ctx, grad_out):
        need = ctx.needs_input_grad
        gx, gw, ggu, gdn, gap = _experts_backward(ctx, grad_out, need[:5], need[6])
        return gx, None, gw, ggu, gdn, None, gap


def _empty_result(hidden, top_k_weights, *params):
    """No tokens: an empty (0,H) result that still hangs on every differentiable input, so that a backward pass
    gives zero gradients of the right shapes (what the reference's eager loop does with zero rows)."""
    out = _amp_cast(hidden)[0]
    out = out + top_k_weights.to(out.dtype).sum(dim=-1, keepdim=True)
    for p in params:
        if p is not None:
            out = out + 0.0 * p.sum().to(out.dtype)
    return out


class StackCopies:
    """Copies of a weight stack that outlive the call that made them.  The stream that wrote them need not be the one that reads
    them next: until they are known to be complete a reader on another stream waits for the writer's event, and their memory is
    not handed out again before that stream is done with it.  (While a graph is being captured neither is possible, nor needed:
    torch.cuda.graph waits for the device before it begins.)"""
    __slots__ = ("tensors", "stream", "event")

    def __init__(self, tensors):
        self.tensors = tensors
        self.stream = self.event = None
        if tensors[0].is_cuda:
            self.stream = L.stream_of(tensors[0])
            # on the default stream, which is there for good, only when one is asked for: an event of a stack's first pass costs it 15 us
            self.event = True if self.stream == 0 else torch.cuda.current_stream(tensors[0].device).record_event()

    def here(self):
        """The tensors, for the current stream."""
        if self.stream is not None and L.stream_of(self.tensors[0]) != self.stream:
            self._elsewhere(self.tensors[0])
        return self.tensors

    def _elsewhere(self, t):
        if L.capturing(t):
            return
        now = torch.cuda.current_stream(t.device)
        if self.event is True:
            self.event = torch.cuda.default_stream(t.device).record_event()
        if self.event is not None and self.event.query():
            self.event = None
        if self.event is not None:
            now.wait_event(self.event)
        for t in self.tensors:
            t.record_stream(now)


_BF16_COPIES = {}     # id(parameter) -> (weak reference, version, data pointer, StackCopies of the bf16 copy)


def _bf16_copy(t):
    """bf16 copy of an fp16 / fp32 expert stack, kept until the tensor changes (its autograd version counter moves
    on every in-place update, e.g. an optimizer step; its address when `.data` is assigned) or is freed.  Callers with
    fp32 master weights would otherwise pay a full copy of both stacks on every call.  Tensors that need a gradient are
    cast afresh, so that autograd carries the gradient back through the cast.  Under graph capture nothing is kept."""
    if t.requires_grad and torch.is_grad_enabled():
        return t.to(torch.bfloat16)
    import weakref
    key = id(t)
    hit = _BF16_COPIES.get(key)
    if hit is not None and hit[0]() is t and hit[1] == t._version and hit[2] == t.data_ptr():
        return hit[3].here()[0]
    c = t.detach().to(torch.bfloat16)
    if L.capturing(c):     # the graph's memory, which only a replay fills
        return c
    _BF16_COPIES[key] = (weakref.ref(t, lambda _r, k=key: _BF16_COPIES.pop(k, None)), t._version, t.data_ptr(), StackCopies((c,)))
    return c


def moe(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes, act_params=None):
    """hidden (N,H) bf16 (fp16 / fp32: computed in bf16), indices (N,k) int64, weights (N,k) float, gate_up_proj (E_glu,2I,H),
    down_proj (E_glu,H,I), act_codes (E,) int32, act_params (E,2) fp32 [alpha,gamma] for code 5 or None
    -> (N,H).  Same contract as the reference's `moe` (kernels/sm75/moe.py:838-855); differentiable
    w.r.t. hidden, weights, both projections and act_params.  A stack of SiLU / ReLU^2 / parameter-free SiTU experts
    (codes 0, 1, 5, no act_params, no Identity / Zero experts) runs with the activation fused into the GEMM epilogues;
    any other stack (Norm codes, learnable SiTU, special experts) runs the PolyGLU row kernels."""
    codes, n_glu = _code_info(act_codes)
    if hidden.shape[0] == 0:
        return _empty_result(hidden, top_k_weights, gate_up_proj, down_proj, act_params)
    if hidden.dtype in (torch.float16, torch.float32) and not torch.is_autocast_enabled("cuda"):
        # The reference computes in hidden's dtype.  The kernels here are bf16 (fp32 accumulation): fp16 / fp32 callers
        # get the bf16 computation, the result in their dtype and, through the casts, gradients in the dtypes of
        # their tensors.  Accuracy is that of the bf16 path (2e-2 relative L2 against fp32).
        bf = torch.bfloat16
        out = moe(hidden.to(bf), top_k_indices, top_k_weights, _bf16_copy(gate_up_proj), _bf16_copy(down_proj),
                  act_codes, act_params)
        return out.to(hidden.dtype)
    fused = act_params is None and n_glu == len(codes) and all(c in FUSED_CODES for c in codes)
    fast = L.fast() if hidden.is_cuda else None
    if fast is not None:
        codes_dev = None if fused and not any(codes) else _codes_on(act_codes, hidden.device)
        out = fast.experts(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, codes_dev, act_params,
                           L.status_word(hidden.device), len(codes), n_glu, int(not fused))
        if out is not None:
            return out
    if fused:
        keep = torch.is_grad_enabled() and any(t.requires_grad for t in (hidden, top_k_weights, gate_up_proj, down_proj))
        return _GroupedMoE.apply(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes, keep)
    return _PolyGLUMoE.apply(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes, act_params)


def moe_grouped(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes):
    """Same signature as kernels/sm75/moe.py:621 (which has no act_params: code 5 runs parameter-free)."""
    return moe(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes)


def moe_per_expert(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes, act_params=None):
    """Same signature as kernels/sm75/moe.py:829; runs the one grouped path."""
    return moe(hidden, top_k_indices, top_k_weights, gate_up_proj, down_proj, act_codes, act_params)
