"""Drop-in for the reference's ``LLMLayer`` (model.py:278-321): the decoder layer the
Mixture-of-Experts block sits in. Same constructor, attribute and parameter names and
``state_dict`` layout (``norm1``, ``mqa``, ``norm2``, ``moe`` or ``ffn``), same ``forward``
signature and return value (tensor, load-balancing loss).

What the layer adds over assigning ``layer.moe`` / ``layer.mqa`` in the reference's own layer:
in inference the second LayerNorm (model.py:298,312) is folded into the block's router and
dispatch kernels and the second skip connection (model.py:319) into its combine kernel, so
neither is a pass over the activations of its own; the first LayerNorm runs the library's row
kernel (``moe_b200_layernorm``); QKV and head gate are one launch, the attention core the next, output Linear and first
skip connection the last, and for a few short sequences the first LayerNorm is part of the first one
(``csrc/linear_rows.cu``).
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import _cabi, _host
from ._cabi import check, lib
from .attention import Attention
from .moe import MOE, FeedForward, _stream


_module = nn.modules.module


def _watched(m: nn.Module) -> bool:
    """Hooks that a call of the module would run."""
    return bool(m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks
                or _module._global_forward_hooks or _module._global_forward_pre_hooks or _module._global_backward_hooks
                or _module._global_backward_pre_hooks)


def _layernorm(norm: nn.LayerNorm, x: torch.Tensor) -> torch.Tensor:
    """norm(x) by the library's row kernel (moe_b200_layernorm) for bf16/fp32 CUDA
    tensors outside autograd; torch's own LayerNorm otherwise (training). What the native call
    declines (autocast, under which torch's LayerNorm would hand on fp32, torch function modes,
    tracing, other classes of tensors) takes the same kernel from here."""
    if not x.is_cuda or norm.weight is None or norm.bias is None:
        return norm(x)
    out = _host.layernorm(x.contiguous(), norm.weight, norm.bias, float(norm.eps))
    if out is not None:
        return out
    xc, d, params = x.contiguous(), x.shape[-1], (norm.weight, norm.bias)
    if (x.dtype not in (torch.bfloat16, torch.float32) or d % 8 != 0 or xc.data_ptr() % 16 != 0
            or any(p.dtype != x.dtype or p.device != x.device or p.numel() != d or not p.is_contiguous()
                   or p.data_ptr() % 16 != 0 for p in params)
            or (torch.is_grad_enabled() and any(t.requires_grad for t in (x, *params)))):
        return norm(x)
    out = torch.empty_like(xc)
    code = _cabi.BF16 if x.dtype == torch.bfloat16 else _cabi.F32
    with torch.cuda.device(x.device):
        check(lib.moe_b200_layernorm(xc.data_ptr(), norm.weight.data_ptr(), norm.bias.data_ptr(),
                                     float(norm.eps), xc.numel() // d, d, code, out.data_ptr(),
                                     _stream(x.device)), "layernorm")
    return out


class LLMLayer(nn.Module):
    def __init__(self, hidden_dim: int, head_dim: int, q_head: int, kv_head: int, embedding: nn.Module,
                 expansion_factor: int = 4, dropout_ratio: float = 0.1, use_moe: bool = False,
                 num_experts: int = 8, lora_rank: int = 16, lora_alpha: int = 32, device: str = "mps"):
        super().__init__()
        self.use_moe = use_moe
        self.norm1 = nn.LayerNorm(hidden_dim)
        self.mqa = Attention(hidden_dim, head_dim, q_head, kv_head, embedding, lora_rank=lora_rank,
                             lora_alpha=lora_alpha)
        self.norm2 = nn.LayerNorm(hidden_dim)
        if self.use_moe:
            self.moe = MOE(hidden_dim, num_experts=num_experts, expansion_factor=expansion_factor,
                           dropout_ratio=dropout_ratio, lora_rank=lora_rank, device=device)
        else:
            self.ffn = FeedForward(hidden_dim, expansion_factor=expansion_factor, dropout_ratio=dropout_ratio,
                                   lora_rank=lora_rank, lora_alpha=lora_alpha)
        self.device = device

    def device_status(self) -> int:
        """Status word of the layer's own kernels (0 = ok): the attention's, or else the block's; synchronises. Both are
        asked for and start clean again."""
        parts = [self.mqa, self.moe] if self.use_moe else [self.mqa]
        codes = [m.device_status() for m in parts if hasattr(m, "device_status")]
        return next((c for c in codes if c != 0), 0)

    def _attend(self, tensor, attention_mask, fine_tuning):
        """First LayerNorm, attention and first skip connection (model.py:297-308): in one native call, or step by step,
        whose results are the same to the bit."""
        mqa, norm = self.mqa, self.norm1
        if (type(mqa) is Attention and "forward" not in mqa.__dict__ and not _watched(mqa) and tensor.is_cuda
                and tensor.dtype == torch.bfloat16 and tensor.dim() == 3 and norm.weight is not None and norm.bias is not None
                and not (torch.is_grad_enabled() and (tensor.requires_grad or mqa.qkv.weight.requires_grad))):
            done = _host.attention(*mqa._arguments(tensor, attention_mask, fine_tuning), norm.weight, norm.bias,
                                   float(norm.eps))
            if done is not None:
                return done
        out = mqa(_layernorm(norm, tensor), attention_mask=attention_mask, fine_tuning=fine_tuning)
        return out + tensor                                    # model.py:308

    def forward(self, tensor: torch.Tensor, attention_mask: torch.Tensor = None, fine_tuning: bool = False):
        tensor = self._attend(tensor, attention_mask, fine_tuning)
        if self.use_moe:
            if self.moe.training:
                # training mode has no backward pass for the folded LayerNorm
                return self.moe(self.norm2(tensor), fine_tuning=fine_tuning, residual=tensor)
            # model.py:311-319 in the block's own kernels
            return self.moe(tensor, fine_tuning=fine_tuning, residual=tensor, norm=self.norm2)
        out = self.ffn(self.norm2(tensor), fine_tuning=fine_tuning) + tensor
        return out, torch.zeros((), dtype=out.dtype, device=out.device)   # no load-balancing loss (model.py:317)
