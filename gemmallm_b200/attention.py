"""Drop-in for the reference's ``Attention`` (model.py:59-152): same constructor, attribute
and parameter names, ``state_dict`` layout and ``forward`` signature. The fused QKV Linear and the
head gate are one launch (``moe_b200_linear_rows``), the output Linear another (torch's Linears where those are the
faster ones, ``moe_b200_attention_linears``, where sizes or places are not those it takes — a number of heads that is no
multiple of 8, from 129 rows on — and where their derivatives are asked for or their weights are of a class of their own);
everything between
them — head split, shared KV heads, RoPE from the model's own table, scores, mask, softmax,
the product with V and the sigmoid head gate — is one kernel of libmoe_b200
(``moe_b200_attention``), so the [B, H, S, S] score tensor is never materialised.

bf16 on CUDA, head_dim 64, contexts up to 128 tokens, mask None or one additive [S, S] mask
shared by the batch (the causal mask of model.py:585-591); other inputs raise.
"""
from __future__ import annotations

import math

import torch
import torch.nn as nn
import torch.nn.functional as F
from torch.autograd import forward_ad

from . import _cabi, _host
from ._cabi import lib, check
from .moe import _stream


class _MergedLinear:
    """W + s * B A and b + s * (B a + b_lora) of one Linear with its LoRA pair (model.py:98-102,
    144-149), refreshed when one of the six tensors changes."""

    def __init__(self):
        self.key, self.w, self.b = None, None, None

    def get(self, lin, a, b, scale):
        params = (lin.weight, lin.bias, a.weight, a.bias, b.weight, b.bias)
        key = tuple((p.data_ptr(), p._version) for p in params)
        if key != self.key:
            if self.w is None or self.w.shape != lin.weight.shape or self.w.device != lin.weight.device:
                self.w, self.b = torch.empty_like(lin.weight), torch.empty_like(lin.bias)
            dev = lin.weight.device
            with torch.cuda.device(dev):
                check(lib.moe_b200_lora_merge(
                    lin.weight.data_ptr(), lin.bias.data_ptr(), a.weight.data_ptr(), a.bias.data_ptr(),
                    b.weight.data_ptr(), b.bias.data_ptr(), float(scale), lin.out_features, lin.in_features,
                    a.out_features, _cabi.BF16, self.w.data_ptr(), self.b.data_ptr(), _stream(dev)),
                    "lora_merge")
            self.key = key
        return self.w, self.b


class Attention(nn.Module):
    _status = None          # (also of a module that was saved without it)

    def __init__(self, hidden_dim: int, head_dim: int, q_head: int, kv_head: int, embedding: nn.Module,
                 lora_rank: int = 16, lora_alpha: int = 32):
        super().__init__()
        self.head_dim = head_dim
        self.q_head = q_head
        self.kv_head = kv_head
        self.embedding = embedding          # the model's RoPE table: rows [cos | signed sin], model.py:14-36
        self.qkv = nn.Linear(hidden_dim, (q_head + kv_head * 2) * head_dim)
        self.o = nn.Linear(q_head * head_dim, hidden_dim)
        self.scaler = 1 / math.sqrt(head_dim)
        self.lora_scale = lora_alpha / lora_rank
        self.lora_qkv_a = nn.Linear(hidden_dim, lora_rank)
        self.lora_qkv_b = nn.Linear(lora_rank, (q_head + kv_head * 2) * head_dim)
        self.lora_o_a = nn.Linear(q_head * head_dim, lora_rank)
        self.lora_o_b = nn.Linear(lora_rank, hidden_dim)
        if q_head != kv_head:
            assert q_head % kv_head == 0
            self.multi_query_attention = True
            self.q_kv_scale = q_head // kv_head
        else:
            self.multi_query_attention = False
        self.gate = nn.Linear(hidden_dim, q_head)
        self._merged_qkv, self._merged_o = _MergedLinear(), _MergedLinear()
        self._table = None

    def _status_words(self, device):
        if self._status is None or self._status.device != device:
            self._status = torch.zeros(16, dtype=torch.int32, device=device)
        return self._status

    def device_status(self) -> int:
        """Status word of the calls since it was last asked for (0 = ok; see moe_b200.h); synchronises. A non-zero status
        is returned once, so that later calls start clean."""
        if self._status is None:
            return 0
        code = int(self._status[0])
        if code != 0:
            self._status.zero_()
        return code

    def _pos_table(self, device):
        pe = self.embedding.pos_emb
        key = (pe.data_ptr(), pe._version, str(device))
        if self._table is None or self._table[0] != key:
            self._table = (key, pe.detach().to(device=device, dtype=torch.float32).contiguous())
        return self._table[1]

    def _arguments(self, tensor, attention_mask, fine_tuning):
        """What the native call takes: input, weights (merged ones when fine-tuning), table and mask."""
        S, dev = tensor.shape[1], tensor.device
        if fine_tuning:
            wq, bq = self._merged_qkv.get(self.qkv, self.lora_qkv_a, self.lora_qkv_b, self.lora_scale)
            wo, bo = self._merged_o.get(self.o, self.lora_o_a, self.lora_o_b, self.lora_scale)
        else:
            wq, bq, wo, bo = self.qkv.weight, self.qkv.bias, self.o.weight, self.o.bias
        mask = attention_mask
        if mask is not None:
            if mask.numel() != S * S:
                raise NotImplementedError("one additive [S, S] mask for the whole batch is supported")
            if mask.dtype != torch.float32 or mask.device != dev or not mask.is_contiguous():
                mask = mask.reshape(S, S).to(device=dev, dtype=torch.float32).contiguous()
        return (tensor.contiguous(), wq, bq, self.gate.weight, self.gate.bias, wo, bo, self._pos_table(dev), mask, self.q_head,
                self.kv_head, self.head_dim, self.scaler, self._status_words(dev))

    def forward(self, tensor: torch.Tensor, attention_mask: torch.Tensor = None,
                fine_tuning: bool = False) -> torch.Tensor:
        if not tensor.is_cuda or tensor.dtype != torch.bfloat16:
            raise NotImplementedError("the attention kernel runs on CUDA tensors in bfloat16")
        if torch.is_grad_enabled() and (tensor.requires_grad or self.qkv.weight.requires_grad):
            raise NotImplementedError("the attention kernel has no backward pass; use torch.no_grad()")
        B, S, hid = tensor.shape
        dev = tensor.device
        args = self._arguments(tensor, attention_mask, fine_tuning)
        done = _host.attention(*args)
        if done is not None:
            return done
        x, wq, bq, wg, bg, wo, bo, table, mask = args[:9]
        inner = self.q_head * self.head_dim
        own = self._own_linears(args, B * S, hid, inner)
        if own:
            qkv, gate = _linear_rows(args[13], x, wq, bq, wg, bg)
        else:
            qkv = F.linear(x, wq, bq)
            gate = F.linear(x, wg, bg)                                # [B,S,q_head] logits (model.py:139)
        mask_ptr = None if mask is None else mask.data_ptr()
        if table.shape[0] < S or table.shape[1] != 2 * self.head_dim:
            raise ValueError("the RoPE table is shorter than the sequence or has another head_dim")
        out = torch.empty(B, S, inner, dtype=tensor.dtype, device=dev)
        with torch.cuda.device(dev):
            check(lib.moe_b200_attention(qkv.data_ptr(), gate.data_ptr(), table.data_ptr(), mask_ptr, B, S,
                                         self.q_head, self.kv_head, self.head_dim, float(self.scaler),
                                         out.data_ptr(), _stream(dev)), "attention")
        return _linear_rows(args[13], out, wo, bo)[0] if own else F.linear(out, wo, bo)

    def _own_linears(self, args, N, hid, inner):
        """Whether the Linears go through moe_b200_linear_rows: the same answer as the native call's. Not where derivatives are
        asked for: torch's Linears give those of the output projection; and not for weights of a class of their own (quantised
        ones, say), whose data may lie anywhere: they say themselves what a Linear is."""
        x, wq, bq, wg, bg, wo, bo = args[:7]
        if any(type(p) not in (torch.Tensor, nn.Parameter, type(None)) for p in args[1:7]) or any(_derived(p) for p in args[:7]):
            return False
        rows, many = (self.q_head + 2 * self.kv_head) * self.head_dim, N > lib.moe_b200_linear_rows_max()
        return (1 <= N <= 1 << 28 and lib.moe_b200_attention_linears(N, hid, self.q_head, self.kv_head, self.head_dim) != 0
                and hid % 8 == 0 and self.head_dim == 64 and self.q_head % self.kv_head == 0
                and x.shape[1] <= 128 and x.data_ptr() % 16 == 0 and not (many and self.q_head % 8 != 0)
                and all(w.shape == (r, c) and w.is_contiguous() and w.data_ptr() % 16 == 0 and b is not None and b.numel() == r
                        and b.is_contiguous() and not (many and b.data_ptr() % 16 != 0)
                        and all(p.dtype == torch.bfloat16 and p.device == x.device for p in (w, b))
                        for w, b, r, c in ((wq, bq, rows, hid), (wg, bg, self.q_head, hid), (wo, bo, hid, inner))))


def _derived(p):
    return p is not None and ((torch.is_grad_enabled() and p.requires_grad) or forward_ad.unpack_dual(p).tangent is not None)


def _linear_rows(status, x, w, b, w2=None, b2=None):
    """x W^T + b, and with the second Linear its output too, by the library's kernels."""
    N, K, dev = x.numel() // x.shape[-1], x.shape[-1], x.device
    out = torch.empty(*x.shape[:-1], w.shape[0], dtype=x.dtype, device=dev)
    out2 = None if w2 is None else torch.empty(*x.shape[:-1], w2.shape[0], dtype=x.dtype, device=dev)
    ptr = lambda t: None if t is None else t.data_ptr()
    with torch.cuda.device(dev):
        check(lib.moe_b200_linear_rows(x.data_ptr(), w.data_ptr(), b.data_ptr(), w.shape[0], ptr(w2), ptr(b2),
                                       0 if w2 is None else w2.shape[0], N, K, out.data_ptr(), ptr(out2), status.data_ptr(),
                                       _stream(dev)),
              "linear_rows")
    return out, out2
