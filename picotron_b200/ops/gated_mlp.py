"""Gated MLP ``down(silu(gate(x)) * up(x))`` with the activation inside the GEMMs.

Forward: the gate/up product computes the activation in its epilogue (``pico_gemm_swiglu``), then the down projection.
Backward: the input gradient of the down projection becomes the gradients of gate and up in its epilogue
(``pico_gemm_swiglu_bwd``), so the gradient of the activation is never stored. Few rows take the plain products and a
pass of its own for the activation (``pico_gemm_swiglu_pays``). Needs gate and up stored back to back
(``param_store``); otherwise, and off the kernels' types, the separate ops of ``swiglu`` and ``gemm`` serve.

Reference: picotron/model.py:258 (``down(silu(gate(x)) * up(x))``).
"""
from __future__ import annotations

import torch

from . import count_launch, ext, gemm, untracked, use_kernels


def fits(x: torch.Tensor, ws: "gemm.WeightSet", w_down: torch.Tensor) -> bool:
    """Whether the fused kernels take these operands: one [2*I, K] block of gate rows and up rows, a down projection of
    the same type, and rows of whole 16-byte units."""
    w = ws.fused_weight
    if w is None or len(ws.splits) != 2 or ws.splits[0] != ws.splits[1] or not use_kernels(x, w):
        return False
    inter = ws.splits[0]
    return (w_down.dtype == x.dtype and w.dtype == x.dtype and w_down.dim() == 2 and w_down.shape[1] == inter
            and w_down.is_contiguous() and x.shape[-1] == w.shape[1]
            and gemm._gemm_ok(x.shape[-1], inter, w_down.shape[0]) and x.numel() > 0)


def _forward(x, ws, w_down, keep: bool):
    x2 = gemm._as_2d(x)
    gate_up, act, n = ext().gemm_swiglu(x2, ws.fused_weight, keep)
    count_launch(n)
    y = gemm.gemm_nt(act, w_down)
    return y.view(*x.shape[:-1], w_down.shape[0]), x2, gate_up, act


class _GatedMLPFn(torch.autograd.Function):
    """The parameters behind ``ws`` are passed so that autograd runs the backward (and with it the ``main_grad``
    accumulation) even when x needs no gradient."""

    @staticmethod
    def forward(ctx, x, ws, w_down, *params):
        y, x2, gate_up, act = _forward(x, ws, w_down, True)
        ctx.ws, ctx.x_shape = ws, x.shape
        ctx.save_for_backward(x2, gate_up, act, w_down)
        return y

    @staticmethod
    def backward(ctx, dy):
        x2, gate_up, act, w_down = ctx.saved_tensors
        dy2 = gemm._as_2d(dy)
        # frozen gate and up of an input without gradient are not part of the graph of the separate operators
        gate_up_learns = ctx.needs_input_grad[0] or any(ctx.needs_input_grad[3:])
        if gate_up_learns:
            d_gate_up, n = ext().gemm_swiglu_bwd(dy2, w_down, gate_up)
            count_launch(n)
        dw = gemm.wgrad_into(w_down, dy2, act) if ctx.needs_input_grad[2] else None
        if not gate_up_learns:
            return (None, None, dw) + (None,) * (len(ctx.needs_input_grad) - 3)
        dx, grads = gemm.backward_all(d_gate_up, x2, ctx.ws, need_dx=ctx.needs_input_grad[0])
        return (dx.view(ctx.x_shape) if dx is not None else None, None, dw, *grads)


def gated_mlp(x: torch.Tensor, ws: "gemm.WeightSet", w_down: torch.Tensor) -> torch.Tensor:
    """``fits(x, ws, w_down)`` holds."""
    if untracked():
        return _forward(x, ws, w_down, False)[0]
    return _GatedMLPFn.apply(x, ws, w_down, *ws.params)
