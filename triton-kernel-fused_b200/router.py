"""Sigmoid-gate linear router behind the reference's callables (kernels/sm75/router.py).

`fused_mlp_router` (:277-289), `FusedMLPRouter` (:221-260) and `router_bias_update` (:292-301) keep
their signatures.  Logits are a tcgen05 GEMM (fp32 accumulate, stored in x's dtype as the reference
does), followed by the warp-level top-k epilogue kernel (a small batch: both in one launch); backward is the epilogue Jacobian kernel
plus two tcgen05 GEMMs (dX, and dW as a split-K reduction over the tokens).
"""
from __future__ import annotations

import torch

from . import _lib as L
from . import ops

__all__ = ["fused_mlp_router", "FusedMLPRouter", "fused_router", "FusedConvRouter", "router_bias_update"]


class FusedMLPRouter(torch.autograd.Function):
    """Returns (idx (N,k) int64, weights (N,k) fp32 final, counts (E,) int32); only `weights` is
    differentiable (kernels/sm75/router.py:229-242)."""

    @staticmethod
    def forward(ctx, x, weight, bias, top_k, num_experts, norm_topk=True, scale=1.0):
        if torch.is_autocast_enabled("cuda"):
            dt = torch.get_autocast_dtype("cuda")
            x, weight = x.to(dt), weight.to(dt)
        L.require_cuda_bf16("x", x)
        L.require_cuda_bf16("gate_weight", weight)
        L.require(weight.dim() == 2 and weight.shape[1] == x.shape[-1], "gate_weight must be (E,H)")
        L.require(num_experts is None or int(num_experts) == weight.shape[0], "num_experts must equal gate_weight.shape[0]")
        xf = x.reshape(-1, x.shape[-1]).contiguous()
        weight = weight.contiguous()
        bias32 = None
        if bias is not None:
            bias32 = bias.detach().float().contiguous()
        (T, H), E, dev, k = xf.shape, weight.shape[0], xf.device, int(top_k)
        if bias32 is not None:
            L.require(bias32.is_cuda and bias32.numel() == E, "bias must be a contiguous float32 CUDA tensor of E elements")
        L.require(weight.device == dev, "gate_weight must be on x's device")
        ctx.norm, ctx.scale = int(bool(norm_topk and top_k > 1)), float(scale)
        logits = torch.empty(T, E, dtype=torch.bfloat16, device=dev)
        idx = torch.empty(T, k, dtype=torch.int64, device=dev)
        w = torch.empty(T, k, dtype=torch.float32, device=dev)
        counts = torch.empty(E, dtype=torch.int32, device=dev)
        L.check(L.lib().b200moe_router_forward(xf.data_ptr(), weight.data_ptr(), L.ptr(bias32), T, H, E, k, ctx.norm,
                                               ctx.scale, logits.data_ptr(), idx.data_ptr(), w.data_ptr(), counts.data_ptr(),
                                               L.status_word(dev).data_ptr(), L.stream_of(xf)))
        ctx.xshape = x.shape
        ctx.save_for_backward(xf, weight, logits, idx)
        ctx.mark_non_differentiable(idx, counts)
        ctx.set_materialize_grads(False)      # no zero-filled gradients for idx and counts: two launches a pass
        return idx, w, counts

    @staticmethod
    def backward(ctx, grad_idx, grad_weights, grad_counts):
        if grad_weights is None:
            return (None,) * 7
        xf, weight, logits, idx = ctx.saved_tensors
        (T, H), E, dev = xf.shape, weight.shape[0], xf.device
        gw = grad_weights.contiguous().float()
        grad_x = torch.empty(ctx.xshape, dtype=torch.bfloat16, device=dev) if ctx.needs_input_grad[0] else None
        grad_w = torch.empty(E, H, dtype=torch.bfloat16, device=dev) if ctx.needs_input_grad[1] else None
        lib = L.lib()
        ws = L.workspace(lib.b200moe_router_bwd_ws_bytes(T, H, E), dev)
        L.check(lib.b200moe_router_backward(xf.data_ptr(), weight.data_ptr(), logits.data_ptr(), idx.data_ptr(), gw.data_ptr(),
                                            T, H, E, idx.shape[1], ctx.norm, ctx.scale, ws.data_ptr(), L.ptr(grad_x),
                                            L.ptr(grad_w), L.status_word(dev).data_ptr(), L.stream_of(xf)))
        return grad_x, grad_w, None, None, None, None, None


def _empty_routing(x, weight, top_k):
    """No tokens: empty picks and weights (the weights still hang on x and the gate weight), zero counts."""
    n = x.numel() // max(x.shape[-1], 1)
    idx = torch.zeros(n, top_k, dtype=torch.int64, device=x.device)
    w = (x.reshape(n, x.shape[-1])[:, :1].float() + 0.0 * weight.float().sum()).expand(n, top_k)
    counts = torch.zeros(weight.shape[0], dtype=torch.int32, device=x.device)
    return idx, w, counts


def fused_mlp_router(x, gate_weight, bias, top_k, num_experts, norm_topk_prob=True,
                     routed_scaling_factor=1.0, return_counts=False):
    """x (B,S,H) or (N,H), gate_weight (E,H), bias (E,) fp32 or None -> (idx, weights[, counts]);
    (B,S,k) shapes for 3-D x (kernels/sm75/router.py:277-289)."""
    if x.numel() == 0:
        idx, w, counts = _empty_routing(x, gate_weight, top_k)
    else:
        idx, w, counts = FusedMLPRouter.apply(x, gate_weight, bias, top_k, num_experts, norm_topk_prob,
                                              routed_scaling_factor)
    if x.ndim == 3:
        B, S, _ = x.shape
        idx = idx.view(B, S, top_k)
        w = w.view(B, S, top_k)
    return (idx, w, counts) if return_counts else (idx, w)


class FusedConvRouter(torch.autograd.Function):
    """Causal-conv router (kernels/sm75/router.py:172-218, FusedConvRouterCuDNN): logits[b,s,e] =
    sum_{j,h} x[b, s-(K-1)+j, h] * W[e,h,j], then the same sigmoid / bias / top-k epilogue.  One tcgen05 GEMM
    whose TMA producer reads x in place, tap by tap, through an (H, S, B) tensor map (kernels/sm120/router.py:34-85 is one
    launch too), or over an unfolded copy of x (H no multiple of 16, many short sequences); the backward's top-k kernel lays the gradients
    out tap by tap, and dX and dW are plain products with that.  One native call each way (csrc/block.cu); plain calls
    take the compiled form of this Function (csrc/fast.cpp)."""

    @staticmethod
    def forward(ctx, x, weight, bias, top_k, num_experts, norm_topk=True, scale=1.0):
        if torch.is_autocast_enabled("cuda"):
            dt = torch.get_autocast_dtype("cuda")
            x, weight = x.to(dt), weight.to(dt)
        L.require_cuda_bf16("x", x)
        L.require_cuda_bf16("conv_weight", weight)
        L.require(x.dim() == 3 and weight.dim() == 3 and weight.shape[1] == x.shape[2], "need x (B,S,H) and conv_weight (E,H,K)")
        (B, S, H), (E, _, K), dev, k = x.shape, weight.shape, x.device, int(top_k)
        L.require(num_experts is None or int(num_experts) == E, "num_experts must equal conv_weight.shape[0]")
        x, weight = x.contiguous(), weight.contiguous()
        bias32 = bias.detach().float().contiguous() if bias is not None else None
        if bias32 is not None:
            L.require(bias32.is_cuda and bias32.numel() == E, "bias must be a contiguous float32 CUDA tensor of E elements")
        L.require(weight.device == dev, "conv_weight must be on x's device")
        ctx.norm, ctx.scale = int(bool(norm_topk and top_k > 1)), float(scale)
        wt = torch.empty(K * E, H, dtype=torch.bfloat16, device=dev)
        logits = torch.empty(B * S, E, dtype=torch.bfloat16, device=dev)
        idx = torch.empty(B * S, k, dtype=torch.int64, device=dev)
        w = torch.empty(B * S, k, dtype=torch.float32, device=dev)
        counts = torch.empty(E, dtype=torch.int32, device=dev)
        lib = L.lib()
        ws = L.workspace(lib.b200moe_conv_router_fwd_ws_bytes(B, S, H, E, K), dev)
        L.check(lib.b200moe_conv_router_forward(x.data_ptr(), weight.data_ptr(), L.ptr(bias32), B, S, H, E, K, k, ctx.norm,
                                                ctx.scale, ws.data_ptr(), wt.data_ptr(), logits.data_ptr(), idx.data_ptr(),
                                                w.data_ptr(), counts.data_ptr(), L.status_word(dev).data_ptr(), L.stream_of(x)))
        ctx.shape = (B, S, H, E, K, k)
        ctx.save_for_backward(x, wt, logits, idx)
        ctx.mark_non_differentiable(idx, counts)
        ctx.set_materialize_grads(False)      # no zero-filled gradients for idx and counts: two launches a pass
        return idx, w, counts

    @staticmethod
    def backward(ctx, grad_idx, grad_weights, grad_counts):
        if grad_weights is None:
            return (None,) * 7
        x, wt, logits, idx = ctx.saved_tensors
        B, S, H, E, K, k = ctx.shape
        dev = x.device
        gw = grad_weights.contiguous().float()
        grad_x = torch.empty(B, S, H, dtype=torch.bfloat16, device=dev) if ctx.needs_input_grad[0] else None
        grad_w = torch.empty(E, H, K, dtype=torch.bfloat16, device=dev) if ctx.needs_input_grad[1] else None
        lib = L.lib()
        ws = L.workspace(lib.b200moe_conv_router_bwd_ws_bytes(B, S, H, E, K), dev)
        L.check(lib.b200moe_conv_router_backward(x.data_ptr(), wt.data_ptr(), logits.data_ptr(), idx.data_ptr(), gw.data_ptr(),
                                                 B, S, H, E, K, k, ctx.norm, ctx.scale, ws.data_ptr(), L.ptr(grad_x),
                                                 L.ptr(grad_w), L.status_word(dev).data_ptr(), L.stream_of(x)))
        return grad_x, grad_w, None, None, None, None, None


def fused_router(x, conv_weight, bias, top_k, num_experts, norm_topk_prob=True, routed_scaling_factor=1.0,
                 return_counts=False):
    """Whole conv router: x (B,S,H), conv_weight (E,H,K) from nn.Conv1d(H,E,K), bias (E,) fp32 or None ->
    (idx (B,S,k) int64, weights (B,S,k) fp32[, counts (E,) int32]); kernels/sm75/router.py:263-274."""
    B, S, _ = x.shape
    if x.numel() == 0:
        idx, w, counts = _empty_routing(x, conv_weight, top_k)
    else:
        fast = L.fast() if x.is_cuda else None
        res = None
        if fast is not None:
            res = fast.conv_router(x, conv_weight, bias, L.status_word(x.device), int(top_k),
                                   conv_weight.shape[0] if num_experts is None else int(num_experts),
                                   int(bool(norm_topk_prob and top_k > 1)), float(routed_scaling_factor))
        if res is not None:
            return res if return_counts else res[:2]
        idx, w, counts = FusedConvRouter.apply(x, conv_weight, bias, top_k, num_experts, norm_topk_prob,
                                               routed_scaling_factor)
    idx = idx.view(B, S, top_k)
    w = w.view(B, S, top_k)
    return (idx, w, counts) if return_counts else (idx, w)


@torch.no_grad()
def router_bias_update(bias, counts, u):
    """b += u*sign(mean_load - load), in place; `counts` must already be the global load (the caller
    all-reduces it across ranks first); no-op when u <= 0 (kernels/sm75/router.py:292-301)."""
    if u <= 0:
        return
    ops.router_bias_update(bias, counts.to(torch.int32).contiguous(), u)
