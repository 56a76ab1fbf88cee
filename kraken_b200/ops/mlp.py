"""MLP head on the tcgen05 Linear kernels (csrc/cuda/mlp_gemm.cu).

``fused_mlp(x, weights, biases)`` runs Linear+ReLU layers on bf16 activations
with fp32 parameters and fp32 accumulation; the last layer has no activation
and, when it has a single output, runs as a row-dot kernel that keeps the
logit in fp32.  The backward pass is hand-scheduled: per layer one split-K
weight-gradient GEMM that red-adds straight into the parameter's gradient
buffer and sums the bias gradient on the way, and one input-gradient GEMM with
the ReLU mask of the previous layer fused into its epilogue.
"""
from __future__ import annotations

from typing import List, Optional, Sequence

import torch

from .._native import C
from ..utils.profiler import engine_region
from . import counters

_status = {}
_side_streams = {}
_deferred_join = False
_pending_join = set()


_grad_ready = None


def set_grad_ready_callback(fn) -> None:
    """``fn(parameter, stream)`` is called by the backward pass once every kernel that writes a parameter's
    gradient this step has been enqueued on ``stream`` (the engine uses it to launch the fused dense step of a
    bucket while the backward pass is still running)."""
    global _grad_ready
    _grad_ready = fn


def _notify(params, stream) -> None:
    for p in params:
        _grad_ready(p, stream)


def set_deferred_join(on: bool) -> None:
    """With deferred join the backward pass leaves its side stream (weight and bias gradients)
    un-joined, and whoever consumes those gradients next - the engine's fused dense step - runs on
    that stream and joins it afterwards.  The sparse backward and push that follow the MLP in a
    recommender's backward pass then run beside the last weight gradients and the dense step
    instead of behind them.  Only safe when nothing reads ``param.grad`` of the MLP on the main
    stream before the dense step, which is why the engine option that turns it on is off by default."""
    global _deferred_join
    _deferred_join = bool(on)
    if not on:
        _pending_join.clear()


def take_pending_side_stream(device: torch.device) -> Optional[torch.cuda.Stream]:
    """The side stream with un-joined gradient work on ``device`` (and marks it as taken), or None."""
    key = (device.type, device.index)
    if key in _pending_join:
        _pending_join.discard(key)
        return _side_streams.get(key)
    return None


def _side_stream(device: torch.device) -> torch.cuda.Stream:
    """Second stream on which weight and bias gradients run beside the input-gradient chain."""
    key = (device.type, device.index)
    if key not in _side_streams:
        _side_streams[key] = torch.cuda.Stream(device=device)
    return _side_streams[key]



def _ids(stream: torch.cuda.Stream):
    """A stream as the native side takes it."""
    return stream.stream_id, stream.device_index, stream.device_type


class PreparedWeights:
    """bf16 copies of the hidden layers' weights, cast on the side stream: as they are and, for a forward pass that a
    backward pass will follow, transposed (``wt16s`` is empty otherwise)."""

    def __init__(self, w16s, wt16s, event):
        self.w16s, self.wt16s, self.event = w16s, wt16s, event


def _cast(weights: Sequence[torch.Tensor], transpose: bool):
    counters.add()
    return C.cast_weights(weights, transpose)


def prepare_weights(weights: Sequence[torch.Tensor]) -> PreparedWeights:
    """Starts the fp32 -> bf16 casts of the hidden layers' weights on the side stream and returns
    at once.  A model calls this before work that does not depend on the weights (the sparse
    pull of a recommender), hands the result to ``fused_mlp(prepared=...)``, and the casts run
    beside that work instead of in front of the first GEMM."""
    counters.add()
    return PreparedWeights(*C.prepare_weights(weights[:-1], torch.is_grad_enabled(), *_ids(_side_stream(weights[0].device))))


def gemm_status(device: torch.device) -> torch.Tensor:
    """Device word in which the GEMM kernels record a pipeline wait that gave up."""
    key = (device.type, device.index)
    if key not in _status:
        _status[key] = torch.zeros(1, dtype=torch.int32, device=device)
    return _status[key]


def check_gemm_status(device: torch.device) -> None:
    st = gemm_status(device)
    code = int(st.item())
    if code != 0:
        st.zero_()
        raise C.KrakenError(f"tcgen05 GEMM: {C.error_message(code)} (code {code})")


def supported(in_features: int, sizes: Sequence[int]) -> bool:
    """Whether the hidden layers meet the TMA pitch rule (widths in multiples of 8 elements).
    The last layer may have any width: 1 runs as a row-dot kernel, a multiple of 8 on the
    tensor cores, another one up to 16 (a 10-class head, say) in fp32 kernels of its own,
    anything else as a small fp32 matmul of the library."""
    dims = [in_features] + list(sizes)
    return len(sizes) >= 1 and all(d % 8 == 0 for d in dims[:-1])


def _grad_target(p: torch.Tensor) -> torch.Tensor:
    """The buffer a parameter's gradient is accumulated into (created zeroed if absent)."""
    if p.grad is None:
        p.grad = torch.zeros_like(p)
    return p.grad


class _FusedMLP(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, addend, n_layers, input_grad_cols, prepared, with_grad, *params):
        ws, bs = params[:n_layers], params[n_layers:]
        dev = x.device
        if prepared is not None and (prepared.wt16s or not with_grad):
            prepared.event.wait()
            w16s, wts = prepared.w16s, prepared.wt16s
        else:
            w16s, wts, _ = _cast(ws[:-1], with_grad)
        st = gemm_status(dev)
        h = x if x.dtype == torch.bfloat16 else x.to(torch.bfloat16)
        M = h.shape[0]
        # masks[i] is one bit per element of acts[i + 1] (> 0): the next layer's input gradient masks with it instead of
        # re-reading the activations
        counters.add(n_layers - 1)
        acts, masks = C.mlp_hidden_forward(h, w16s, bs[:-1], st, with_grad)
        h = acts[-1]
        wl, bl = ws[-1].detach(), bs[-1].detach()
        if wl.shape[0] == 1:
            out = torch.empty(M, dtype=torch.float32, device=dev)
            counters.add()
            C.rowdot_forward(h, wl.reshape(-1).contiguous(), bl, out,
                             addend.detach().float().contiguous() if addend is not None else None)
            out = out.view(M, 1)
            addend = None
        elif wl.shape[0] % 8 == 0:
            y = torch.empty((M, wl.shape[0]), dtype=torch.bfloat16, device=dev)
            counters.add()
            C.linear_forward(h, wl.to(torch.bfloat16), bl, False, y, st)
            out = y.float()
        elif C.head_supported(h, wl) and bl.is_contiguous():
            out = torch.empty((M, wl.shape[0]), dtype=torch.float32, device=dev)
            counters.add()
            C.head_forward(h, wl, bl, out)
        else:
            out = torch.addmm(bl, h.float(), wl.t())  # wider odd-width head: library fp32 matmul
        if addend is not None:
            out = out + addend.reshape(M, 1).to(out.dtype)
        ctx.acts, ctx.ws, ctx.bs, ctx.n_layers, ctx.wts, ctx.masks = acts, ws, bs, n_layers, wts, masks
        ctx.x_needs_grad = x.requires_grad
        ctx.input_grad_cols = input_grad_cols
        ctx.x_dtype = x.dtype
        return out

    @staticmethod
    def backward(ctx, gout):
        with engine_region("mlp_bwd"):
            return _FusedMLP._backward(ctx, gout)

    @staticmethod
    def _backward(ctx, gout):
        acts, ws, bs, L = ctx.acts, ctx.ws, ctx.bs, ctx.n_layers
        dev = gout.device
        st = gemm_status(dev)
        M = acts[0].shape[0]
        wl = ws[-1]
        h_last = acts[-1]
        need_dx_last = L > 1 or ctx.x_needs_grad
        if wl.shape[0] == 1:
            dy = gout.reshape(-1).float().contiguous()
            dh = torch.empty_like(h_last) if need_dx_last else None
            counters.add()
            C.rowdot_backward(h_last, wl.detach().reshape(-1).contiguous(), dy, L > 1, dh,
                              _grad_target(wl).view(-1), _grad_target(bs[-1]))
        elif (wl.shape[0] % 8 != 0 and C.head_supported(h_last, wl.detach(), _grad_target(wl))
              and _grad_target(bs[-1]).is_contiguous()):
            dh = torch.empty_like(h_last) if need_dx_last else None
            counters.add()
            C.head_backward(h_last, wl.detach(), gout.float().contiguous(), L > 1, dh, _grad_target(wl), _grad_target(bs[-1]))
        elif wl.shape[0] % 8 != 0:
            g32 = gout.float()
            h32 = h_last.float()
            _grad_target(wl).addmm_(g32.t(), h32)
            _grad_target(bs[-1]).add_(g32.sum(0))
            dh = None
            if need_dx_last:
                d = g32 @ wl.detach()
                if L > 1:
                    d = d * (h32 > 0)
                dh = d.to(torch.bfloat16)
        else:
            dy16 = gout.to(torch.bfloat16).contiguous()
            counters.add()
            C.linear_wgrad(dy16, h_last, _grad_target(wl), st, _grad_target(bs[-1]))
            dh = None
            if need_dx_last:
                dh = torch.empty_like(h_last)
                counters.add()
                C.linear_dgrad(dy16, wl.detach().t().contiguous().to(torch.bfloat16), None, dh, st,
                               ctx.masks[-1] if L > 1 else None)
        if _grad_ready is not None:
            _notify((wl, bs[-1]), torch.cuda.current_stream(dev))
        side = _side_stream(dev)
        if L > 1:
            counters.add(2 * (L - 1) - (0 if ctx.x_needs_grad else 1))
            ready = None
            if _grad_ready is not None:
                def ready(i):
                    _notify((ws[i], bs[i]), side)
            dh = C.mlp_hidden_backward(dh, acts, ctx.masks, ctx.wts, [_grad_target(w) for w in ws[:-1]],
                                       [_grad_target(b) for b in bs[:-1]], st, ctx.x_needs_grad,
                                       ctx.input_grad_cols or 0, *_ids(side), _deferred_join, ready)
        if _deferred_join:
            _pending_join.add((dev.type, dev.index))
        dx = None
        if ctx.x_needs_grad and dh is not None:
            dx = dh if ctx.x_dtype == torch.bfloat16 else dh.to(ctx.x_dtype)
        # parameter gradients were accumulated in place
        return (dx, gout.reshape(-1) if ctx.needs_input_grad[1] else None, None, None, None, None) + (None,) * (2 * L)


def fused_mlp(x: torch.Tensor, weights: List[torch.Tensor], biases: List[torch.Tensor],
              input_grad_cols: int = 0, addend: Optional[torch.Tensor] = None,
              prepared: Optional[PreparedWeights] = None) -> torch.Tensor:
    """x [M, K] (bf16 or fp32, CUDA) -> [M, out_features] fp32.  Parameter gradients are
    accumulated into ``param.grad`` in place by the backward kernels.  ``input_grad_cols``
    (a multiple of 8, 0 = all) limits the input gradient to the leading columns of x.
    ``addend`` [M] (single-output heads) is added to the output inside the head kernel.
    ``prepared`` is the result of an earlier ``prepare_weights`` call on the same weights."""
    with engine_region("mlp_fwd"):
        if addend is not None and weights[-1].shape[0] != 1:
            raise ValueError("addend needs a single-output head")
        return _FusedMLP.apply(x, addend, len(weights), int(input_grad_cols), prepared, torch.is_grad_enabled(), *weights,
                               *biases)
