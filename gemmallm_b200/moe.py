"""Drop-in modules for GemmaLLM's Mixture-of-Experts block.

``MOE`` and ``FeedForward`` keep the constructor, attribute names, parameter
names/shapes and ``state_dict`` layout of the reference classes
(model.py:192-198 and model.py:154-171), so
``new.load_state_dict(ref.state_dict(), strict=True)`` works in both
directions. ``forward`` runs the hand-written sm_100a kernels of
libmoe_b200.so through its C ABI: this module only hands over device pointers,
sizes and the current CUDA stream. There is no CPU or eager-PyTorch path.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import _cabi
from ._cabi import lib, check
from . import _host

_DTYPES = {torch.float32: _cabi.F32, torch.bfloat16: _cabi.BF16}


def _dtype_code(t: torch.Tensor) -> int:
    try:
        return _DTYPES[t.dtype]
    except KeyError:
        raise TypeError(f"libmoe_b200 computes in float32 or bfloat16, got {t.dtype}") from None


def _stream(device: torch.device) -> int:
    return torch.cuda.current_stream(device).cuda_stream


_LORA_NAMES = ("gate_and_up", "down", "lora_gate_and_up_a", "lora_gate_and_up_b", "lora_down_a",
               "lora_down_b")


def _expert_watch(ex, fine_tuning: bool) -> list:
    """(dictionary, key) of everything in an expert's module tree that a prepared call uses: the
    Linears, then weight and bias of each in the order of _LORA_NAMES."""
    names = _LORA_NAMES if fine_tuning else _LORA_NAMES[:2]
    watch = [(ex._modules, n) for n in names]
    for n in names:
        watch += [(getattr(ex, n)._parameters, "weight"), (getattr(ex, n)._parameters, "bias")]
    return watch


class _MergedExpert:
    """An expert's two Linears with the LoRA branch folded in (moe_b200_lora_merge):
    W' = W + s * B A and b' = b + s * (B a + b_lora), which makes
    x W'^T + b' = x W^T + b + s * (B (A x + a) + b_lora), the fine_tuning=True
    expression of model.py:175-179 and 185-189. Has the attribute shape _Plan expects
    (gate_and_up/down with .weight/.bias); the buffers are written in place on every
    refresh, so a plan built on them stays valid."""

    class _Lin:
        def __init__(self, w, b):
            self.weight, self.bias = w, b

    def __init__(self, ex):
        self.gate_and_up = self._Lin(torch.empty_like(ex.gate_and_up.weight), torch.empty_like(ex.gate_and_up.bias))
        self.down = self._Lin(torch.empty_like(ex.down.weight), torch.empty_like(ex.down.bias))


class _MergedLora:
    """Merged copies of a list of experts, refreshed only when one of their twelve tensors
    was replaced or written since the last call (data pointer and torch's version counter),
    so that a fine_tuning=True forward on unchanged parameters launches no merge kernel and
    rebuilds no plan. What the copies hold is recorded in ``native``, with the copies, for every
    call that reads them (csrc/host/host.cpp). A copy of this object starts empty."""

    def __init__(self):
        self.shapes = None
        self.merged = None
        self.native = None

    def __reduce__(self):
        return (_MergedLora, ())

    def get(self, experts, dtype: int, device: torch.device):
        params = [p for ex in experts for n in _LORA_NAMES
                  for p in (getattr(ex, n).weight, getattr(ex, n).bias)]
        for p in params:
            if p.device != device or _dtype_code(p) != dtype or not p.is_contiguous():
                raise ValueError("expert and LoRA parameters must be contiguous and share the "
                                 "input's device and dtype")
        shapes = (dtype, str(device), tuple(tuple(p.shape) for p in params))
        if shapes != self.shapes:
            self.merged = [_MergedExpert(ex) for ex in experts]
            self.native = _host.Merged([
                (lin.out_features, lin.in_features, a.out_features, out.weight, out.bias)
                for ex, mg in zip(experts, self.merged)
                for lin, a, out in ((ex.gate_and_up, ex.lora_gate_and_up_a, mg.gate_and_up),
                                    (ex.down, ex.lora_down_a, mg.down))])
            self.shapes = shapes
        self.native.refresh(params, [float(ex.lora_scale) for ex in experts], dtype, device.index)
        return self.merged


def _lora_table(experts, dev) -> torch.Tensor:
    """Device table of the LoRA tensors' addresses, [2 Linears][experts][A, a, B], for their gradients."""
    rows = [[p.data_ptr() for p in (a.weight, a.bias, b.weight)]
            for pair in (("lora_gate_and_up_a", "lora_gate_and_up_b"), ("lora_down_a", "lora_down_b"))
            for a, b in ((getattr(ex, pair[0]), getattr(ex, pair[1])) for ex in experts)]
    return torch.tensor(rows, dtype=torch.int64).to(dev)


def _lora_ranks(experts) -> list:
    return [a.out_features for ex in experts for a in (ex.lora_gate_and_up_a, ex.lora_down_a)]


def _expert_params(ex, fine_tuning: bool) -> list:
    """The tensors an expert's gradients belong to, in the order of _LORA_NAMES."""
    return [p for n in (_LORA_NAMES if fine_tuning else _LORA_NAMES[:2])
            for p in (getattr(ex, n).weight, getattr(ex, n).bias)]


class _Plan:
    """Device copy of the experts' parameter pointers and TMA tensor maps.

    Rebuilt whenever a parameter's storage, dtype or device changes (``.to()``,
    ``load_state_dict`` keep storage; ``.to(dtype)`` replaces it)."""

    def __init__(self):
        self.key = None
        self.buf = None

    def get(self, experts, d: int, f: int, dtype: int, device: torch.device) -> int:
        params = []
        for ex in experts:
            params += [ex.gate_and_up.weight, ex.gate_and_up.bias, ex.down.weight, ex.down.bias]
        key = (dtype, str(device), tuple(p.data_ptr() for p in params))
        if key != self.key:
            for p in params:
                if p.device != device or _dtype_code(p) != dtype or not p.is_contiguous():
                    raise ValueError("expert parameters must be contiguous and share the input's "
                                     "device and dtype")
            E = len(experts)
            nbytes = lib.moe_b200_plan_bytes(E)
            buf = torch.empty(nbytes + 128, dtype=torch.uint8, device=device)
            base = (buf.data_ptr() + 127) & ~127
            w1 = _cabi.ptr_array([ex.gate_and_up.weight.data_ptr() for ex in experts])
            b1 = _cabi.ptr_array([ex.gate_and_up.bias.data_ptr() for ex in experts])
            w2 = _cabi.ptr_array([ex.down.weight.data_ptr() for ex in experts])
            b2 = _cabi.ptr_array([ex.down.bias.data_ptr() for ex in experts])
            check(lib.moe_b200_plan_build(w1, b1, w2, b2, E, d, f, dtype, base, nbytes,
                                          _stream(device)), "plan_build")
            self.key, self.buf, self.base = key, buf, base
        return self.base


class _TracedFfn(torch.autograd.Function):
    """FeedForward's training forward as torch.jit.trace can record it, a Python operator: the native call's own graph
    stays inside, and every run of the traced function draws a mask."""

    @staticmethod
    def forward(ctx, module, tensor, fine_tuning, *params):
        with torch.enable_grad():
            x = tensor.detach().requires_grad_(tensor.requires_grad)
            y, _ = module._prepare_train(x, fine_tuning, module._native_train_ft if fine_tuning else module._native_train)
        ctx.graph = y, [t for t in (x, *params) if t.requires_grad], [t.requires_grad for t in (x, *params)]
        return y.detach()

    @staticmethod
    def backward(ctx, grad):
        y, inputs, wanted = ctx.graph
        grads = iter(torch.autograd.grad(y, inputs, grad, retain_graph=True))
        gx, *gp = [next(grads) if w else None for w in wanted]
        return (None, gx, None, *gp)


class _Asked:
    """How often the last call, plain and with LoRA branches, has had to be prepared. Binding a call to the native path
    costs about as much as it saves one call, so it is done the second, fourth, eighth ... time: not for a size seen once
    (generation without a cache has another length with every token), and seldom for calls that find the
    binding unusable. Other weights, slots or scales are another call and count anew."""

    def __init__(self):
        self.last = {}

    def bind_now(self, fine_tuning: bool, key) -> bool:
        was, count = self.last.get(fine_tuning, (None, 0))
        count = count + 1 if was == key else 1
        self.last[fine_tuning] = (key, count)
        return count > 1 and count & (count - 1) == 0


class _Calls(nn.Module):
    """A module with state that belongs to its calls (plans, workspaces, bound calls: addresses of this object's own
    tensors). A copy of the module, by copy, pickle or replication, starts without any."""

    @staticmethod
    def _fresh_calls() -> dict:
        raise NotImplementedError

    def _reset_calls(self) -> None:
        # one update: an nn.Module takes about 2 us to set an attribute, and a block has a hundred of these
        self.__dict__.update(self._fresh_calls())

    def __getstate__(self):
        drop = self._fresh_calls()
        return {n: v for n, v in self.__dict__.items() if n not in drop}

    def __setstate__(self, state):
        super().__setstate__(state)
        self._reset_calls()

    def _replicate_for_data_parallel(self):
        replica = super()._replicate_for_data_parallel()
        replica._reset_calls()
        return replica


class FeedForward(_Calls):
    """GeGLU feed-forward expert; mirrors reference model.py:154-190.

    ``gate_and_up`` maps d -> 2f (rows [0,f) gate, rows [f,2f) up), ``down`` maps
    f -> d, plus the four LoRA Linears of the reference (rank ``lora_rank``,
    scale ``lora_alpha / lora_rank``), used when ``fine_tuning=True``.

    ``d_ff`` (keyword-only) sets f directly for widths that are not an integer
    multiple of ``hidden_size``."""

    def __init__(self, hidden_size: int, expansion_factor: int = 4, dropout_ratio: float = 0.1,
                 lora_rank: int = 16, lora_alpha: int = 32, *, d_ff: int | None = None):
        super().__init__()
        f = hidden_size * expansion_factor if d_ff is None else d_ff
        self.hidden_size, self.d_ff = hidden_size, f
        self.gate_and_up = nn.Linear(hidden_size, f * 2)
        self.down = nn.Linear(f, hidden_size)
        self.dropout = nn.Dropout(p=dropout_ratio)
        self.lora_scale = lora_alpha / lora_rank
        self.lora_gate_and_up_a = nn.Linear(hidden_size, lora_rank)
        self.lora_gate_and_up_b = nn.Linear(lora_rank, f * 2)
        self.lora_down_a = nn.Linear(f, lora_rank)
        self.lora_down_b = nn.Linear(lora_rank, hidden_size)
        self.last_seed = None
        self._reset_calls()

    @staticmethod
    def _fresh_calls() -> dict:
        return dict(
            _calls=_Asked(), _plan=_Plan(), _plan_ft=_Plan(), _lora=_MergedLora(),
            # native calls prepared for the last number of rows: plain, and with the LoRA branches merged
            _native=_host.Ffn(), _native_ft=_host.Ffn(), _native_train=_host.Ffn(), _native_train_ft=_host.Ffn(),
            _offsets=None,      # ((rows, device), int32 [0, rows]) of the last call
            _tws=None, _tws_key=None,
            _generation=None)   # counts the forwards on _tws

    def _rows(self, tensor):
        x = tensor.reshape(-1, tensor.shape[-1]).contiguous()
        M, dev = x.shape[0], x.device
        if self._offsets is None or self._offsets[0] != (M, str(dev)):
            self._offsets = ((M, str(dev)), torch.tensor([0, M], dtype=torch.int32, device=dev))
        return x, M, dev, self._offsets[1]

    def _plan_of(self, fine_tuning: bool) -> _Plan:
        return self._plan_ft if fine_tuning else self._plan

    def _bound(self, fine_tuning: bool):
        """Merged weights and scales of a call that is bound."""
        return (self._lora.native, [float(self.lora_scale)]) if fine_tuning else (None, [])

    # -- training mode (bf16): dropout on h and a backward pass -----------------
    def _train_ws(self, M: int, device: torch.device):
        key = (M, str(device))
        if key != self._tws_key:
            d, f = self.hidden_size, self.d_ff
            nbytes = lib.moe_b200_train_workspace_bytes(M, d, f, 1, 1, _cabi.BF16)
            if nbytes == 0:
                raise _cabi.MoeB200Error(lib.moe_b200_last_error_string().decode())
            buf = torch.empty(nbytes + 1024, dtype=torch.uint8, device=device)
            base = (buf.data_ptr() + 1023) & ~1023
            check(lib.moe_b200_train_setup(M, d, f, 1, 1, _cabi.BF16, base, nbytes, _stream(device)), "train_setup")
            self._tws = (buf, base, nbytes)
            self._generation = _host.Generation()
            self._tws_key = key
            self._native_train.unbind()
            self._native_train_ft.unbind()
        return self._tws

    def _prepare_train(self, tensor, fine_tuning: bool, native):
        """Training forward of a call that differs from the one ``native`` was bound for: prepares plan,
        workspace and merged weights, binds them and runs."""
        d, f = self.hidden_size, self.d_ff
        if tensor.shape[-1] != d:
            raise ValueError(f"last dimension {tensor.shape[-1]} != hidden_size {d}")
        x, M, dev, offsets = self._rows(tensor)
        if not tensor.is_contiguous():
            done = native.train(x, self.dropout.p, None, self.lora_scale)
            if done is not None:
                return done[0].reshape(tensor.shape), done[1]
        with torch.cuda.device(dev):
            if fine_tuning:
                plan = self._plan_ft.get(self._lora.get([self], _cabi.BF16, dev), d, f, _cabi.BF16, dev)
            else:
                plan = self._plan.get([self], d, f, _cabi.BF16, dev)
            buf, tbase, tbytes = self._train_ws(M, dev)
            status = torch.zeros(16, dtype=torch.int32, device=dev)
            watch = _expert_watch(self, fine_tuning)
            usual = all(name in table for table, name in watch)
            native.unbind()
            native.bind(watch if usual else [], *self._bound(fine_tuning), plan, [self._plan_of(fine_tuning).buf],
                        offsets, status, M, d, f, _cabi.BF16, dev.index)
            table = _lora_table([self], dev) if fine_tuning else None
            native.bind_train(buf, tbase, tbytes, table, _lora_ranks([self]) if fine_tuning else [], self._generation)
            # the tensors themselves, wherever the module tree keeps them
            y, seed = native.train(x, float(self.dropout.p), _expert_params(self, fine_tuning), self.lora_scale)
        return y.reshape(tensor.shape), seed

    def forward(self, tensor: torch.Tensor, fine_tuning: bool = False) -> torch.Tensor:
        """y = down(gelu_tanh(gate) * up) for every row, through the grouped
        expert kernels with a single group. ``fine_tuning=True`` adds the LoRA
        branch (model.py:175-179,185-189) folded into merged copies of the two weight
        matrices (refreshed when a parameter changes); under ``.train()`` the LoRA tensors
        receive gradients too."""
        if not tensor.is_cuda:
            raise RuntimeError("libmoe_b200 runs on CUDA tensors only; there is no CPU path")
        if self.training and (torch.is_grad_enabled() or self.dropout.p > 0):
            if tensor.dtype != torch.bfloat16:
                raise NotImplementedError("training mode computes in bfloat16")
            native = self._native_train_ft if fine_tuning else self._native_train
            done = native.train(tensor, self.dropout.p, None, self.lora_scale)
            if done is None and torch.jit.is_tracing():
                return _TracedFfn.apply(self, tensor, bool(fine_tuning), *_expert_params(self, fine_tuning))
            if done is None:
                done = self._prepare_train(tensor, bool(fine_tuning), native)
            y, self.last_seed = done
            return y
        native = self._native_ft if fine_tuning else self._native
        y = native.forward(tensor, self.lora_scale)
        return self._forward_prepared(tensor, bool(fine_tuning), native) if y is None else y

    def _forward_prepared(self, tensor, fine_tuning: bool, native):
        """The forward of a call that differs from the one ``native`` was bound for: prepares plan,
        offsets and merged weights, runs, and binds the result."""
        dtype = _dtype_code(tensor)
        shape = tensor.shape
        d, f = self.hidden_size, self.d_ff
        if shape[-1] != d:
            raise ValueError(f"last dimension {shape[-1]} != hidden_size {d}")
        x, M, dev, offsets = self._rows(tensor)
        if not tensor.is_contiguous():
            y = native.forward(x, self.lora_scale)          # bound for these rows, contiguous
            if y is not None:
                return y.reshape(shape)
        with torch.cuda.device(dev):
            plan = (self._plan_ft if fine_tuning else self._plan).get(
                self._lora.get([self], dtype, dev) if fine_tuning else [self], d, f, dtype, dev)
            status = torch.zeros(16, dtype=torch.int32, device=dev)
            h = torch.empty(M, f, dtype=x.dtype, device=dev)
            y = torch.empty(M, d, dtype=x.dtype, device=dev)
            check(lib.moe_b200_experts(x.data_ptr(), offsets.data_ptr(), plan, M, d, f, 1, dtype, 0,
                                       h.data_ptr(), y.data_ptr(), status.data_ptr(), _stream(dev)),
                  "experts")
        if not self._calls.bind_now(fine_tuning, (M, dtype, str(dev), plan, self.lora_scale)):
            return y.reshape(shape)
        native.unbind()
        watch = _expert_watch(self, fine_tuning)
        if all(name in table for table, name in watch):
            native.bind(watch, *self._bound(fine_tuning), plan, [self._plan_of(fine_tuning).buf], offsets, status, M, d, f,
                        dtype, dev.index)
        return y.reshape(shape)


class MOE(_Calls):
    """Mixture-of-experts feed-forward block; mirrors reference model.py:192-276.

    Same positional/keyword arguments as the reference constructor
    (model.py:193); ``device`` is accepted and stored but not used, the kernels
    run where the input lives. Keyword-only extensions: ``top_k`` (the reference
    fixes 2, model.py:210) and ``d_ff`` (free per-branch width)."""

    def __init__(self, hidden_size: int, num_experts: int = 8, expansion_factor: int = 4,
                 dropout_ratio: float = 0.1, lora_rank: int = 16, lora_alpha: int = 32,
                 device: str = "mps", *, top_k: int = 2, d_ff: int | None = None):
        super().__init__()
        self.gate = nn.Linear(hidden_size, num_experts)
        self.num_experts = num_experts
        self.experts = nn.ModuleList([
            FeedForward(hidden_size, expansion_factor=expansion_factor, dropout_ratio=dropout_ratio,
                        lora_rank=lora_rank, lora_alpha=lora_alpha, d_ff=d_ff)
            for _ in range(num_experts)])
        self.device = device
        self.hidden_size = hidden_size
        self.d_ff = self.experts[0].d_ff
        self.top_k = top_k
        self._reset_calls()

    @staticmethod
    def _fresh_calls() -> dict:
        return dict(
            _calls=_Asked(), _plan=_Plan(), _plan_ft=_Plan(), _lora=_MergedLora(), _ws=None, _ws_key=None, _tws=None,
            _tws_key=None, _generation=None,      # counts the forwards on _tws
            _last_seed=None,
            # native calls prepared for the last input size: plain, and with the LoRA branches merged
            _native=_host.Block(), _native_ft=_host.Block(), _native_train=_host.Block(), _native_train_ft=_host.Block())

    @property
    def last(self) -> dict | None:
        """Views into the workspace of the most recent call (None before the first): logits, idx,
        w, cnt_slot, offsets, psum, row_of, status; after a training forward also its seed."""
        if self._ws is None or self._last_seed is False:
            return None
        N, _, _, E, k = self._ws_key
        views = {
            "logits": self._view("logits", torch.float32, (N, E)),
            "idx": self._view("idx", torch.int32, (N, k)),
            "w": self._view("w", torch.float32, (N, k)),
            "cnt_slot": self._view("cnt_slot", torch.int32, (k, E)),
            "offsets": self._view("offsets", torch.int32, (E + 1,)),
            "psum": self._view("psum", torch.float32, (E,)),
            "row_of": self._view("row_of", torch.int32, (N, k)),
            "status": self._view("status", torch.int32, (16,)),
        }
        if self._last_seed is not None:
            views["seed"] = self._last_seed
        return views

    @last.setter
    def last(self, value) -> None:
        if value is not None:
            raise ValueError("last can be cleared, not set")
        self._last_seed = False       # until the next call

    # -- workspace ---------------------------------------------------------
    def _workspace(self, N: int, dtype: int, device: torch.device):
        d, f, E, k = self.hidden_size, self.d_ff, self.num_experts, self.top_k
        key = (N, dtype, str(device), E, k)
        if key != self._ws_key:
            nbytes = _cabi.workspace_bytes(N, d, f, E, k, dtype)
            buf = torch.empty(nbytes + 1024, dtype=torch.uint8, device=device)
            base = (buf.data_ptr() + 1023) & ~1023
            self._ws = (buf, base, nbytes, _cabi.workspace_layout(N, d, f, E, k, dtype))
            self._ws_key = key
            for native in (self._native, self._native_ft, self._native_train, self._native_train_ft):
                native.unbind()
            # the small-N kernels keep their counters in the status region and leave them zero
            # after every call (FLAG_WS_CLEAN below); everything else is written before it is
            # read, except for what a call without tokens leaves as it is
            if N == 0:
                buf.zero_()
            self._view("status", torch.int32, (_cabi.READY_OFFSET + _cabi.READY_INTS,)).zero_()
        return self._ws

    def _view(self, name: str, dtype: torch.dtype, shape) -> torch.Tensor:
        buf, base, _, layout = self._ws
        start = base - buf.data_ptr() + layout[name]
        n = 1
        for s in shape:
            n *= s
        nbytes = n * torch.empty(0, dtype=dtype).element_size()
        return buf[start:start + nbytes].view(dtype).view(*shape)

    def forward(self, tensor: torch.Tensor, fine_tuning: bool = False, *,
                residual: torch.Tensor | None = None,
                norm: nn.LayerNorm | None = None) -> tuple[torch.Tensor, torch.Tensor]:
        """``tensor`` [B,S,d] -> ([B,S,d] in the input dtype, load-balancing loss).

        With ``residual`` (same shape and dtype) the caller's skip connection
        (model.py:319) is added inside the combine kernel. With ``norm`` (the caller's
        ``norm2``, model.py:298,312) ``tensor`` is the tensor BEFORE that LayerNorm: the
        block normalises it on the fly in its router and dispatch kernels, so
        ``moe(x, residual=x, norm=layer.norm2)`` replaces model.py:311-319. ``fine_tuning=True``
        runs the experts with their LoRA branches (model.py:175-179,185-189)
        folded into merged copies of their weights (refreshed when a parameter
        changes); under ``.train()`` the LoRA tensors receive gradients too."""
        if not tensor.is_cuda:
            raise RuntimeError("libmoe_b200 runs on CUDA tensors only; there is no CPU path")
        if self.training and (torch.is_grad_enabled() or self.experts[0].dropout.p > 0):
            # training mode: dropout on h (model.py:183) and a backward pass
            if norm is not None:
                raise NotImplementedError("training mode has no backward pass for the folded LayerNorm: "
                                          "apply the LayerNorm in front of the block")
            if tensor.dtype != torch.bfloat16:
                raise NotImplementedError("training mode computes in bfloat16")
            native = self._native_train_ft if fine_tuning else self._native_train
            done = native.train(tensor, residual, self.experts[0].dropout.p, None, self.top_k)
            if done is None and torch.jit.is_tracing():
                raise RuntimeError("the block's training forward cannot be traced")
            if done is None:
                done = self._prepare_train(tensor, residual, bool(fine_tuning), native)
            out, aux, self._last_seed = done
            return out, aux
        native = self._native_ft if fine_tuning else self._native
        self._last_seed = None
        done = native.forward(tensor, residual, norm, self.top_k)
        if done is None:
            done = self._forward_prepared(tensor, bool(fine_tuning), residual, norm, native)
        return done

    def _forward_prepared(self, tensor, fine_tuning: bool, residual, norm, native):
        """The forward of a call that differs from the one ``native`` was bound for: checks the
        arguments, prepares plan, workspace and merged weights, runs, and binds the result."""
        dtype = _dtype_code(tensor)
        shape = tensor.shape
        d, f, E, k = self.hidden_size, self.d_ff, self.num_experts, self.top_k
        if shape[-1] != d:
            raise ValueError(f"last dimension {shape[-1]} != hidden_size {d}")
        x = tensor.reshape(-1, d).contiguous()
        N = x.shape[0]
        dev = x.device
        res_ptr = None
        as_it_lies = tensor.is_contiguous() and (residual is None or residual.is_contiguous())
        if residual is not None:
            if residual.shape != shape or residual.dtype != tensor.dtype or residual.device != dev:
                raise ValueError("residual must match the input's shape, dtype and device")
            residual = residual.reshape(-1, d).contiguous()
            res_ptr = residual.data_ptr()
        gw, gb = self.gate.weight, self.gate.bias
        if gw.device != dev or _dtype_code(gw) != dtype:
            raise ValueError("gate parameters must share the input's device and dtype")
        if not as_it_lies:
            done = native.forward(x, residual, norm, self.top_k)      # bound for these rows, contiguous
            if done is not None:
                return done[0].reshape(shape), done[1]
        nw = nb = None
        eps = 0.0
        if norm is not None:
            if (tuple(norm.normalized_shape) != (d,) or norm.weight is None or norm.bias is None
                    or norm.weight.device != dev or _dtype_code(norm.weight) != dtype):
                raise ValueError("norm must be an affine LayerNorm over the last dimension with "
                                 "the input's device and dtype")
            nw, nb, eps = norm.weight.data_ptr(), norm.bias.data_ptr(), float(norm.eps)
        out = torch.empty_like(x)
        with torch.cuda.device(dev):
            if fine_tuning:
                plan = self._plan_ft.get(self._lora.get(list(self.experts), dtype, dev), d, f, dtype, dev)
            else:
                plan = self._plan.get(self.experts, d, f, dtype, dev)
            _, base, nbytes, _ = self._workspace(N, dtype, dev)
            check(lib.moe_b200_forward(x.data_ptr(), gw.data_ptr(), gb.data_ptr(), plan, res_ptr,
                                       nw, nb, eps, N, d, f, E, k, dtype, _cabi.FLAG_WS_CLEAN, base, nbytes,
                                       out.data_ptr(), _stream(dev)), "forward")
        aux = self._view("aux", torch.float32, (1,))[0].clone()
        scales = tuple(ex.lora_scale for ex in self.experts) if fine_tuning else ()
        if self._calls.bind_now(fine_tuning, (N, dtype, str(dev), plan, gw.data_ptr(), gb.data_ptr(), k, scales)):
            self._bind(native, fine_tuning, plan, N, dtype, dev)
        return out.reshape(shape), aux

    def _watch(self, fine_tuning: bool) -> list:
        """Everything in the module tree a prepared call depends on; empty for trees that do not hold
        their parameters under the usual names (those calls are prepared every time)."""
        watch = [(self._modules, "gate"), (self._modules, "experts"),
                 (self.gate._parameters, "weight"), (self.gate._parameters, "bias")]
        for name, ex in self.experts._modules.items():
            watch.append((self.experts._modules, name))
            watch += _expert_watch(ex, fine_tuning)
            if fine_tuning:
                watch.append((ex.__dict__, "lora_scale"))
        usual = len(self.experts) == self.num_experts and all(name in table for table, name in watch)
        return watch if usual else []

    def _bind(self, native, fine_tuning: bool, plan: int, N: int, dtype: int, dev: torch.device) -> None:
        """Hand the prepared call to the native path."""
        d, f, E, k = self.hidden_size, self.d_ff, self.num_experts, self.top_k
        native.unbind()
        watch = self._watch(fine_tuning)
        merged, scales, owner = ((self._lora.native, [float(ex.lora_scale) for ex in self.experts], self._plan_ft)
                                 if fine_tuning else (None, [], self._plan))
        buf, base, nbytes, _ = self._ws
        native.bind(watch, merged, scales, plan, [owner.buf], buf, base, nbytes, N, d, f, E, k, dtype, dev.index)

    # -- training mode -------------------------------------------------------
    def _train_workspace(self, N: int, device: torch.device):
        d, f, E, k = self.hidden_size, self.d_ff, self.num_experts, self.top_k
        key = (N, str(device), E, k)
        if key != self._tws_key:
            nbytes = lib.moe_b200_train_workspace_bytes(N, d, f, E, k, _cabi.BF16)
            if nbytes == 0:
                raise _cabi.MoeB200Error(lib.moe_b200_last_error_string().decode())
            buf = torch.empty(nbytes + 1024, dtype=torch.uint8, device=device)
            base = (buf.data_ptr() + 1023) & ~1023
            check(lib.moe_b200_train_setup(N, d, f, E, k, _cabi.BF16, base, nbytes, _stream(device)), "train_setup")
            self._tws = (buf, base, nbytes)
            self._generation = _host.Generation()
            self._tws_key = key
            self._native_train.unbind()
            self._native_train_ft.unbind()
        return self._tws

    def _prepare_train(self, tensor, residual, fine_tuning: bool, native):
        """Training forward of a call that differs from the one ``native`` was bound for: checks the arguments,
        prepares plan, workspaces and merged weights, binds them and runs. Gradients: the kernels run on the merged
        weights W' = W + s B A, b' = b + s (B a + b_lora) (model.py:175-179,185-189), whose gradients are the
        base Linear's own; the LoRA tensors' are formed from them (csrc/lora_bwd.cu)."""
        dtype = _dtype_code(tensor)
        shape = tensor.shape
        d, f, E, k = self.hidden_size, self.d_ff, self.num_experts, self.top_k
        if shape[-1] != d:
            raise ValueError(f"last dimension {shape[-1]} != hidden_size {d}")
        x = tensor.reshape(-1, d).contiguous()
        N = x.shape[0]
        dev = x.device
        as_it_lies = tensor.is_contiguous() and (residual is None or residual.is_contiguous())
        if residual is not None:
            if residual.shape != shape or residual.dtype != tensor.dtype or residual.device != dev:
                raise ValueError("residual must match the input's shape, dtype and device")
            residual = residual.reshape(-1, d).contiguous()
        if not as_it_lies:
            done = native.train(x, residual, self.experts[0].dropout.p, None, self.top_k)
            if done is not None:
                return done[0].reshape(shape), done[1], done[2]
        with torch.cuda.device(dev):
            if fine_tuning:
                plan = self._plan_ft.get(self._lora.get(list(self.experts), dtype, dev), d, f, dtype, dev)
            else:
                plan = self._plan.get(self.experts, d, f, dtype, dev)
            self._workspace(N, dtype, dev)
            buf, tbase, tbytes = self._train_workspace(N, dev)
            self._bind(native, fine_tuning, plan, N, dtype, dev)
            table = _lora_table(self.experts, dev) if fine_tuning else None
            native.bind_train(buf, tbase, tbytes, table, _lora_ranks(self.experts) if fine_tuning else [], self._generation)
            # the tensors themselves, wherever the module tree keeps them
            params = [self.gate.weight, self.gate.bias]
            for ex in self.experts:
                params += _expert_params(ex, fine_tuning)
            out, aux, seed = native.train(x, residual, float(self.experts[0].dropout.p), params, k)
        if type(tensor) not in (torch.Tensor, nn.Parameter):
            out = out.as_subclass(type(tensor))
        return out.reshape(shape), aux, seed

    def device_status(self) -> int:
        """Status word of the most recent call (0 = ok); synchronises. A non-zero status is
        returned once: the status region is zeroed again so that later calls start clean."""
        if self._ws is None or self._last_seed is False:
            return 0
        code = int(self._view("status", torch.int32, (16,))[0].item())
        if code != 0:
            self._view("status", torch.int32, (_cabi.READY_OFFSET + _cabi.READY_INTS,)).zero_()
        return code
