"""A Megatron-style MoE layer: router -> dispatch -> grouped experts -> combine.

The reference's "model" is exactly this loop with a random router stand-in
(`DeepEP_Megatron/test_deepep_moe_dispatch_combine.py:731-742,766-815`); here it is an
`nn.Module` with a learnable router so that forward AND backward run (dispatch and combine
are each other's backward, expert GEMMs have dgrad/wgrad).
"""
from __future__ import annotations

from typing import Optional, Tuple

import torch
from torch.autograd.forward_ad import unpack_dual

from .. import _ext
from .experts import build_experts
from .experts_tcgen05 import Tcgen05GroupedExperts
from .token_dispatcher import B200TokenDispatcher


def topk_softmax_router(logits: torch.Tensor, topk: int) -> Tuple[torch.Tensor, torch.Tensor]:
    """(indices int64 [T,K], probabilities f32 [T,K] renormalised over the chosen experts)."""
    probs = torch.softmax(logits.float(), dim=-1)
    w, idx = torch.topk(probs, topk, dim=-1)
    return idx, w / w.sum(-1, keepdim=True)


class _TopkSoftmax(torch.autograd.Function):
    """`topk_softmax_router` on this library's kernels, one launch forward and one backward (f32 like the torch form)."""

    @staticmethod
    def forward(ctx, logits, topk):
        idx, w = _ext.load().topk_softmax(logits, topk)
        ctx.num_experts = logits.shape[1]
        ctx.save_for_backward(idx, w)
        ctx.mark_non_differentiable(idx)
        return idx, w

    @staticmethod
    def backward(ctx, _grad_idx, grad_w):
        idx, w = ctx.saved_tensors
        if torch.is_grad_enabled() or _carries_more(grad_w):          # a graph, a tangent or a batch of gradients is asked for
            d = w * (grad_w - (w * grad_w).sum(-1, keepdim=True))
            return torch.zeros((w.shape[0], ctx.num_experts), dtype=w.dtype, device=w.device).scatter(1, idx, d), None
        return _ext.load().topk_softmax_bwd(idx, w, grad_w.float().contiguous(), ctx.num_experts), None


_LINEAR_FORWARD = torch.nn.Linear.forward
# a program that puts a router of its own in its place has it called
_OWN_ROUTER = topk_softmax_router


def _plain_linear(m: torch.nn.Module) -> bool:
    """Calling `m` does nothing but x @ weight.T in f32: the fused router may stand in for it. (Libraries that wrap
    modules put a `forward` of their own on the instance or the class.)"""
    return (type(m) is torch.nn.Linear and m.bias is None and type(m.weight) is torch.nn.Parameter
            and "forward" not in vars(m) and torch.nn.Linear.forward is _LINEAR_FORWARD
            and m.weight.dtype == torch.float32 and m.weight.is_contiguous() and m.weight.data_ptr() % 16 == 0
            and not (m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks)
            and not (torch.nn.modules.module._global_forward_hooks or torch.nn.modules.module._global_forward_pre_hooks)
            and not torch.is_autocast_enabled("cuda"))


# What `MoELayer`'s inference path stands in for or hands views and device-side counts to. Where a program subclasses,
# wraps or replaces one of these, its own version is called as the general path calls it.
_OWN_DISPATCHER = {n: vars(B200TokenDispatcher)[n] for n in ("dispatch", "dispatch_fp8", "dispatch_in_place")}
_OWN_EXPERTS = {n: vars(Tcgen05GroupedExperts)[n] for n in ("forward_fused_combine", "forward_fp8")}


def _unchanged(obj, methods) -> bool:
    return all(n not in getattr(obj, "__dict__", ()) and getattr(type(obj), n, None) is f for n, f in methods.items())


def _carries_more(t: Optional[torch.Tensor]) -> bool:
    """A tensor with a forward-mode tangent or inside a function transform (a batch of gradients is one, in a form of its
    own): kernels, which know nothing of either, would drop what it carries without a word or fail on it; the autograd
    functions of the general path refuse it."""
    F = torch._C._functorch
    return t is not None and (F.is_functorch_wrapped_tensor(t) or F.is_legacy_batchedtensor(t) or unpack_dual(t).tangent is not None)


class MoELayer(torch.nn.Module):
    def __init__(self, hidden_size: int, ffn_hidden_size: int, num_experts: int, topk: int, group=None, *,
                 ep_size: int = 1, ep_rank: int = 0, dtype=torch.bfloat16, activation: str = "swiglu",
                 expert_backend: str = "auto", dispatcher_mode: str = "fused", world=None, device="cuda",
                 fuse_combine: bool = True, use_fp8: bool = False):
        super().__init__()
        if num_experts % ep_size:
            raise ValueError("num_experts must be divisible by the EP size")
        self.hidden_size, self.num_experts, self.topk = hidden_size, num_experts, topk
        self.fuse_combine = fuse_combine
        self.num_local_experts = num_experts // ep_size
        self.router = torch.nn.Linear(hidden_size, num_experts, bias=False, dtype=torch.float32, device=device)
        torch.nn.init.normal_(self.router.weight, std=0.02)
        self.experts, self.expert_backend = build_experts(expert_backend, self.num_local_experts, hidden_size,
                                                          ffn_hidden_size, dtype, activation, device, use_fp8=use_fp8)
        # fp8 inference path: e4m3 rows with 1x128 scales leave the dispatch kernel and feed the
        # block-scaled fp8 fc1 directly (no dequantisation pass); training stays bf16
        self.use_fp8 = bool(use_fp8) and getattr(self.experts, "use_fp8", False)
        self.dispatcher = B200TokenDispatcher(group, self.num_local_experts, num_experts,
                                              ep_rank * self.num_local_experts, mode=dispatcher_mode, world=world)

    def _route(self, hidden_states: torch.Tensor, router_logits: Optional[torch.Tensor], inference: bool):
        """(expert ids, weights). For inference the router runs on this library's kernels (f32 like the
        module's own product); for training the logits are the module's own, softmax and choice this library's."""
        E, K = self.num_experts, self.topk
        C = _ext.load() if hidden_states.is_cuda and inference else None
        if C is None or E > C.ROUTER_MAX_EXPERTS or K > 32 or torch.compiler.is_compiling() or torch.jit.is_tracing():
            if router_logits is None:
                router_logits = self.router(hidden_states.float())
            l = router_logits
            if (not inference and topk_softmax_router is _OWN_ROUTER and type(l) is torch.Tensor and l.is_cuda and l.dim() == 2 and 1 <= K <= min(32, l.shape[1])
                    and l.get_device() == torch.cuda.current_device() and l.shape[1] <= _ext.load().ROUTER_MAX_EXPERTS and not _carries_more(l)
                    and not torch.compiler.is_compiling() and not torch.jit.is_tracing()):
                return _TopkSoftmax.apply(l.float().contiguous(), K)
            return topk_softmax_router(l, K)
        if router_logits is None:
            x = hidden_states
            if (type(x) is torch.Tensor and x.dtype == torch.bfloat16 and x.dim() == 2 and x.is_contiguous()
                    and x.data_ptr() % 16 == 0 and x.shape[1] % 8 == 0 and x.device == self.router.weight.device
                    and _plain_linear(self.router) and self.router.weight.shape == (E, x.shape[1])):
                return C.route(x, self.router.weight, K)
            router_logits = self.router(x.float())
        if type(router_logits) is not torch.Tensor or router_logits.dim() != 2 or router_logits.shape[1] > C.ROUTER_MAX_EXPERTS:
            return topk_softmax_router(router_logits, K)
        return C.topk_softmax(router_logits.float().contiguous(), K)

    def forward(self, hidden_states: torch.Tensor, router_logits: Optional[torch.Tensor] = None) -> torch.Tensor:
        """hidden_states [T,H]; router_logits [T,E] override the learnable router when given."""
        inference = not (torch.is_grad_enabled() or topk_softmax_router is not _OWN_ROUTER or _carries_more(hidden_states)
                         or _carries_more(router_logits) or _carries_more(getattr(self.router, "weight", None)))
        idx, probs = self._route(hidden_states, router_logits, inference)
        if (inference and self.dispatcher.mode == "fused" and hidden_states.dtype == torch.bfloat16
                and (self.use_fp8 or self.fuse_combine)
                and _unchanged(self.dispatcher, _OWN_DISPATCHER) and _unchanged(self.experts, _OWN_EXPERTS)):
            # Inference: the rows are consumed where they arrive, before the next dispatch can be issued on this
            # stream, so they need no copy of their own, and the GEMMs take their tile lists from the device.
            rows, row_probs, handle = self.dispatcher.dispatch_in_place(hidden_states, idx, probs, use_fp8=self.use_fp8)
            if self.use_fp8:
                El = self.num_local_experts
                off = handle.meta[2 + El: 2 + El + El + 1]
                return self.dispatcher.combine(self.experts.forward_fp8(rows, (), row_probs, expert_off=off))
            from . import fused_a2a as A
            buf = A.get_buffer(self.dispatcher.group, A.get_hidden_bytes(hidden_states), self.dispatcher.world)
            self.dispatcher.handle = None
            return self.experts.forward_fused_combine(rows, row_probs, buf, handle)
        if self.use_fp8 and not torch.is_grad_enabled() and self.dispatcher.mode == "fused":
            rows, tokens_per_expert, row_probs = self.dispatcher.dispatch_fp8(hidden_states, idx, probs)
            El = self.num_local_experts
            off = self.dispatcher.handle.meta[2 + El: 2 + El + El + 1]
            return self.dispatcher.combine(self.experts.forward_fp8(rows, tokens_per_expert, row_probs, expert_off=off))
        rows, tokens_per_expert, row_probs = self.dispatcher.dispatch(hidden_states, idx, probs)
        if (self.fuse_combine and self.dispatcher.mode == "fused" and hasattr(self.experts, "forward_fused_combine")
                and (not torch.is_grad_enabled() or self.experts.activation == "swiglu")):
            # the fc2 epilogue stores straight into the source ranks' slots (no combine-send kernel)
            from . import fused_a2a as A
            buf = A.get_buffer(self.dispatcher.group, A.get_hidden_bytes(hidden_states), self.dispatcher.world)
            handle = self.dispatcher.handle
            self.dispatcher.handle = None
            if torch.is_grad_enabled():
                return self.experts.forward_fused_combine_train(rows, tokens_per_expert, row_probs, buf, handle)
            return self.experts.forward_fused_combine(rows, row_probs, buf, handle)
        out_rows = self.experts(rows, tokens_per_expert, row_probs)
        return self.dispatcher.combine(out_rows)
