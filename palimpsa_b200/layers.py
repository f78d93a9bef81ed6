"""Fused element-wise sides of the Palimpsa layer (one CUDA pass each, forward and backward).

The reference layer prepares the operator's inputs and post-processes its output with separate PyTorch
element-wise passes (palimpsa/layers/palimpsa.py:266-281 and :337-343).  :func:`layer_prologue` and
:func:`layer_epilogue` compute the same quantities, so the layer's ``forward`` can read::

    q, k, v, b, dt = layer_prologue(q, k, x, b_raw, self.dt_proj(h), self.bs_proj(h), self.dt_bias, self.b_scale)
    o = chunk_palimpsa(q, k, v, b, dt, A, Ip, ...)
    o = layer_epilogue(o, x, self.D, self.o_norm.weight, gate, eps=self.o_norm.eps)

Both are differentiable (autograd nodes of the native front end over the C ABI) and run on CUDA only.
"""
from __future__ import annotations

from typing import Optional

from torch import Tensor

from .ops.palimpsa import _core


def layer_prologue(q_raw: Tensor, k_raw: Tensor, x: Tensor, b_raw: Tensor, dt_raw: Tensor, bs_raw: Tensor,
                   dt_bias: Tensor, b_scale: Tensor):
    """Inputs of the operator from the layer's projections (palimpsa/layers/palimpsa.py:266-281).

    ``q_raw, k_raw [..., Hq, K]`` (after the short convolution / SiLU), ``x, b_raw [..., H, V]``,
    ``dt_raw, bs_raw [..., H]`` (outputs of ``dt_proj`` / ``bs_proj``), ``dt_bias, b_scale [H]``.
    Returns ``q, k [..., H, K]`` (L2-normalised, repeated over ``H // Hq`` value heads), ``v = x*bs``,
    ``b = sigmoid(b_raw) * softplus(b_scale) * bs`` in ``x.dtype`` and ``dt = softplus(dt_raw + dt_bias)`` in
    float32, where ``bs = sigmoid(bs_raw)`` rounded to ``x.dtype`` as in the layer."""
    return tuple((_core._native or _core.native()).layer_prologue(q_raw, k_raw, x, b_raw, dt_raw, bs_raw, dt_bias, b_scale))


def layer_epilogue(o: Tensor, x: Optional[Tensor], D: Optional[Tensor], weight: Tensor,
                   gate: Optional[Tensor] = None, eps: float = 1e-5) -> Tensor:
    """Output side of the layer (palimpsa/layers/palimpsa.py:337-343): ``z = o + x * D[h]`` (skipped when
    ``x`` / ``D`` are ``None``: ``use_residual=False``), then the RMS norm over the last axis with
    ``weight [V]``, multiplied by ``gate * sigmoid(gate)`` when ``gate [..., H, V]`` is given (the gated
    norm of flash-linear-attention's ``FusedRMSNormGated``, activation "swish").  float32 arithmetic, result
    in ``o.dtype``."""
    return (_core._native or _core.native()).layer_epilogue(o, x, D, weight, gate, float(eps))
