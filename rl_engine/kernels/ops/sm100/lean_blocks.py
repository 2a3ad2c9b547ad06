"""Linear layers fused (at the autograd level) with the cheap op in front of them, so that the cheap op's output is
not kept for the backward pass but recomputed there.

``norm_linear(x, norm_weight, w)`` = ``rms_norm(x) @ w.T`` keeps ``x`` and the per-row ``rstd`` (``x`` is the residual
stream and alive anyway), not the normalised activations.  ``swiglu_linear(gate_up, w)`` = ``(silu(gate) * up) @ w.T``
keeps the packed ``[gate | up]`` GEMM output, not the activation.  For a Llama-3-8B layer that is 2 x 4096 + 14336
fewer elements per token out of 69632, paid for with three memory-bound kernels in the backward pass; the results are
the same bits as the unfused composition (same kernels, same order).

``sink`` / ``sinks``: gradient buffers of the parameters to add to in place of returning gradients (see ``weight_grad``);
only a caller that runs the backward pass itself and wants ``param.grad`` accumulated passes them.

More layers keep their activations in the same memory (``rl_engine.models.activation_plan``), which saves whole layer
recomputations.  The reference has no counterpart (its models are Hugging Face modules).
"""

from __future__ import annotations

import torch

from rl_engine.kernels.ops.base import require_ext
from rl_engine.kernels.ops.sm100.gemm import _as_2d, gemm


def _supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    return (x.is_cuda and x.dtype == torch.bfloat16 and w.dtype == torch.bfloat16 and x.shape[-1] % 8 == 0
            and x.numel() > 0)


def weight_grad(dy2, x2, sink):
    """``dy.T @ x``; with a ``sink`` (the parameter's gradient buffer) it is added there by the GEMM's epilogue (the bits of
    a separate addition) and ``None`` is returned: no gradient tensor of its own and no pass that adds it."""
    if sink is None:
        return gemm(dy2, x2, a_mn=True, b_mn=True)
    require_ext().gemm(dy2, x2, True, True, sink, False, False, 1.0, -1, sink)
    return None


class _NormLinear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, norm_weight, w, eps, sinks):
        ext = require_ext()
        x2 = _as_2d(x)
        nw = norm_weight.contiguous()
        w2 = _as_2d(w)
        h, rstd = ext.rmsnorm_fwd(x2, nw, eps, False, True)
        ctx.save_for_backward(x2, nw, rstd, w2)
        ctx.eps, ctx.x_shape, ctx.sinks = eps, x.shape, sinks
        return gemm(h, w2).reshape(*x.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        ext = require_ext()
        x2, nw, rstd, w2 = ctx.saved_tensors
        norm_sink, w_sink = ctx.sinks
        dy2 = _as_2d(dy)
        h, _ = ext.rmsnorm_fwd(x2, nw, ctx.eps, False, False)
        dw = weight_grad(dy2, h, w_sink) if ctx.needs_input_grad[2] else None
        del h
        dx, dnw = ext.rmsnorm_bwd(x2, nw, gemm(dy2, w2, b_mn=True), rstd, norm_sink)
        return dx.reshape(ctx.x_shape), (dnw if norm_sink is None else None), dw, None, None


def _residual(residual, shape):
    """``residual`` as the addend of the GEMM's epilogue, or ``None`` where it is not fit: another shape than the product's (left
    to the addition to broadcast or refuse), another type, rows that do not start on 16 bytes."""
    if residual is None or residual.dtype != torch.bfloat16 or shape[-1] % 8 or residual.shape != shape or not residual.is_cuda:
        return None
    rows = _as_2d(residual)
    return None if rows.data_ptr() % 16 or rows.stride(0) % 8 else rows


def _product_shape(x: torch.Tensor, w: torch.Tensor) -> torch.Size:
    return x.shape[:-1] + w.shape[:1]


class _SwiGLULinear(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gate_up, w, residual, sink):
        gu2 = _as_2d(gate_up)
        w2 = _as_2d(w)
        ctx.save_for_backward(gu2, w2)
        ctx.gu_shape, ctx.sink = gate_up.shape, sink
        y = _gemm_onto(require_ext().swiglu_packed_fwd(gu2), w2, _residual(residual, _product_shape(gate_up, w)))
        return y.reshape(*gate_up.shape[:-1], w.shape[0])

    @staticmethod
    def backward(ctx, dy):
        ext = require_ext()
        gu2, w2 = ctx.saved_tensors
        dy2 = _as_2d(dy)
        dw = None
        if ctx.needs_input_grad[1]:
            act = ext.swiglu_packed_fwd(gu2)
            dw = weight_grad(dy2, act, ctx.sink)
            del act
        dgu = ext.swiglu_packed_bwd(gu2, gemm(dy2, w2, b_mn=True))
        return dgu.reshape(ctx.gu_shape), dw, (dy if ctx.needs_input_grad[2] else None), None


class _ResidualLinear(torch.autograd.Function):
    """``residual + x @ w.T`` in one kernel."""

    @staticmethod
    def forward(ctx, residual, x, w, sink):
        x2, w2 = _as_2d(x), _as_2d(w)
        ctx.save_for_backward(x2, w2)
        ctx.x_shape, ctx.sink = x.shape, sink
        return _gemm_onto(x2, w2, _residual(residual, residual.shape)).reshape(residual.shape)

    @staticmethod
    def backward(ctx, dy):
        x2, w2 = ctx.saved_tensors
        dy2 = _as_2d(dy)
        dx = gemm(dy2, w2, b_mn=True).reshape(ctx.x_shape) if ctx.needs_input_grad[1] else None
        dw = weight_grad(dy2, x2, ctx.sink) if ctx.needs_input_grad[2] else None
        return (dy if ctx.needs_input_grad[0] else None), dx, dw, None


def _gemm_onto(x2, w2, residual):
    if residual is None:
        return gemm(x2, w2)
    return require_ext().gemm(x2, w2, False, False, None, False, False, 1.0, -1, residual)


def residual_linear(residual: torch.Tensor, x: torch.Tensor, w: torch.Tensor, sink=None) -> torch.Tensor:
    """``residual + x @ w.T``: the sum is taken in the GEMM's epilogue."""
    if _supported(x, w) and _residual(residual, _product_shape(x, w)) is not None:
        return _ResidualLinear.apply(residual, x, w, sink)
    from rl_engine.kernels.ops.sm100.gemm import matmul_nt

    return residual + (matmul_nt(x, w) if _supported(x, w) else x @ w.t())


def norm_linear(x: torch.Tensor, norm_weight: torch.Tensor, w: torch.Tensor, eps: float, sinks=(None, None)) -> torch.Tensor:
    """``rms_norm(x, norm_weight) @ w.T``; the normalised activations are recomputed in the backward pass."""
    if _supported(x, w) and norm_weight.dtype == torch.bfloat16:
        return _NormLinear.apply(x, norm_weight, w, float(eps), sinks)
    from rl_engine.kernels.registry import kernel_registry

    return kernel_registry.get_op("rms_norm")(x, norm_weight, eps=eps) @ w.t()


def swiglu_linear(gate_up: torch.Tensor, w: torch.Tensor, residual=None, sink=None) -> torch.Tensor:
    """``(silu(gate) * up) @ w.T (+ residual)`` for packed ``[rows, 2F] = [gate | up]``; the activation is recomputed in
    backward."""
    f = gate_up.shape[-1] // 2
    if _supported(gate_up, w) and f % 8 == 0:
        if residual is None or _residual(residual, _product_shape(gate_up, w)) is not None:
            return _SwiGLULinear.apply(gate_up, w, residual, sink)
        return residual + _SwiGLULinear.apply(gate_up, w, None, sink)
    from rl_engine.kernels.registry import kernel_registry

    y = kernel_registry.get_op("swiglu")(gate_up[..., :f], gate_up[..., f:]) @ w.t()
    return y if residual is None else residual + y
