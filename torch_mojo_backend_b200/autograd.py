"""``AutogradPrivateUse1`` router for ``aten::scaled_dot_product_attention``.

Same design as the reference (torch_mojo_backend/mojo_device/mojo_device_autograd.py:565-643):
eligible calls are re-dispatched to ``aten::_scaled_dot_product_flash_attention`` so PyTorch's
generated autograd node (``ScaledDotProductFlashAttentionBackward0``) owns the saved tensors,
the version checks and the backward call.  Unlike the reference there is no math
decomposition behind it: an ineligible call raises ``NotImplementedError`` from the forward.

A call that nothing differentiates and nothing watches has no use for the operator's nine results:
it goes to the forward directly (B4 Hq32 Hkv8 Sk1000, one query row, whole call on a B200's host: 93 -> 47 us).
"""

from __future__ import annotations

import torch

from . import flash_ops
from .tensor import TorchMojoTensor

_registered = False


def _seen_by_nobody(query, key, value) -> bool:
    """No gradient or tangent will be asked of the call, and no dispatch mode, function transform, tensor subclass or
    profiler is there to see the operator it stands for."""
    if not (type(query) is type(key) is type(value) is TorchMojoTensor):
        return False
    if torch.is_grad_enabled() and (query.requires_grad or key.requires_grad or value.requires_grad):
        return False
    return (torch._C._len_torch_dispatch_stack() == 0 and torch._C._functorch.peek_interpreter_stack() is None
            and torch.autograd.forward_ad._current_level < 0 and not torch._C._autograd._profiler_enabled())


def scaled_dot_product_attention_autograd(query, key, value, attn_mask=None, dropout_p=0.0, is_causal=False, *,
                                          scale=None, enable_gqa=False):
    inputs = flash_ops.flash_inputs(query, key, value, attn_mask, dropout_p, is_causal, scale, enable_gqa)
    if inputs is None:
        raise NotImplementedError(
            "scaled_dot_product_attention on the mojo device serves only the flash path: fp32/bf16/fp16 "
            "(B,H,S,D) tensors, head_dim 64 or 128, no attn_mask, 0 <= dropout_p < 1, positive scale, "
            "and enable_gqa=True when the key/value head count differs (no fallback exists)"
        )
    if _seen_by_nobody(query, key, value):
        return flash_ops.forward_with_its_own_mask(*inputs, dropout_p, is_causal, scale)[0]
    return torch.ops.aten._scaled_dot_product_flash_attention.default(
        query, key, value, dropout_p, is_causal, False, scale=scale
    )[0]


def register_autograd_ops() -> None:
    global _registered
    if _registered:
        return
    torch.library.impl("aten::scaled_dot_product_attention", "AutogradPrivateUse1")(
        scaled_dot_product_attention_autograd
    )
    _registered = True
