"""The modules' native host path (csrc/host/host.cpp): calls bound to a prepared state, in sequences of calls that
change that state. What a sequence gives is compared with the same last call on a module built afresh from the same
parameters, which has nothing to remember: the kernels are the same, so the results are equal bit for bit."""
import gc
import weakref

import pytest
import torch

from gemmallm_b200 import MOE, Attention, FeedForward, LLMLayer, _host
from gemmallm_b200._cabi import MoeB200Error, check, lib
from gemmallm_b200.attention import _linear_rows
from gemmallm_b200.layer import _layernorm

DT = torch.bfloat16
D, F, E, RANK = 64, 128, 4, 16


def build(kind, dev, seed=0, rank=RANK, p=0.1):
    torch.manual_seed(seed)
    m = (MOE(D, num_experts=E, d_ff=F, dropout_ratio=p, lora_rank=rank, device="cuda") if kind == "moe"
         else FeedForward(D, d_ff=F, dropout_ratio=p, lora_rank=rank))
    return m.to(device=dev, dtype=DT)


def fresh_copy(m, kind, dev, **kw):
    new = build(kind, dev, **kw)
    new.load_state_dict(m.state_dict())
    return new


def rows(n, dev, seed=1):
    return torch.randn(n, D, generator=torch.Generator().manual_seed(seed)).to(DT).to(dev)


def forward(m, x, fine_tuning=False, **kw):
    out = m(x, fine_tuning=fine_tuning, **kw)
    return out if isinstance(out, tuple) else (out,)


def train_step(m, x, fine_tuning=False, mask_seed=5):
    """Output and every gradient of one training step."""
    m.train()
    x = x.detach().clone().requires_grad_(True)
    for p in m.parameters():
        p.grad = None
    torch.manual_seed(mask_seed)
    out = forward(m, x, fine_tuning)
    sum((o.float() ** 2).sum() for o in out).backward()
    return [*(o.detach() for o in out), x.grad, *(p.grad for p in m.parameters() if p.grad is not None)]


def same(got, want):
    assert len(got) == len(want)
    for i, (a, b) in enumerate(zip(got, want)):
        assert torch.equal(a, b), f"tensor {i}: {float((a.float() - b.float()).abs().max())}"


KINDS = ["moe", "ffn"]


# ---- who owns what a bound call has the address of --------------------------------------------

@pytest.mark.parametrize("train", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_a_bound_call_owns_its_buffers(kind, train):
    """Plan, merged weights and workspaces belong to the binding until it is released, whatever the Python side drops."""
    table = {"weight": torch.zeros(1), "bias": torch.zeros(1)}
    watch = [(table, "weight"), (table, "bias")]
    buffers = [torch.zeros(8, dtype=torch.uint8) for _ in range(4)]
    refs = [weakref.ref(t) for t in buffers]
    if kind == "moe":
        native = _host.Block()
        native.bind(watch, None, [], 0, buffers[:2], buffers[2], 0, 0, 1, D, F, E, 2, 1, 0)
    else:
        native = _host.Ffn()
        native.bind(watch, None, [], 0, buffers[:2], buffers[2], buffers[2], 1, D, F, 1, 0)
    if train:
        native.bind_train(buffers[3], 0, 0, None, [], _host.Generation())
    else:
        del refs[3]
    del buffers
    gc.collect()
    assert all(r() is not None for r in refs)
    native.unbind()
    gc.collect()
    assert refs[0]() is None and refs[1]() is None


def test_nothing_is_bound_after_an_error():
    table = {"weight": torch.zeros(1)}
    native = _host.Ffn()
    status = torch.zeros(16, dtype=torch.int32)
    with pytest.raises(KeyError):
        native.bind([(table, "weight"), (table, "bias")], None, [], 0, [status], status, status, 1, D, F, 1, 0)
    assert native.forward(torch.zeros(1, D, dtype=DT), 1.0) is None


def exchange(params, others):
    for p, q in zip(params, others):
        p.data, q.data = q.data, p.data


@pytest.mark.gpu
@pytest.mark.parametrize("fine_tuning", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_weights_exchanged_for_an_evaluation_and_back(cuda_device, kind, fine_tuning):
    """Averaged weights by .data for an evaluation: the training call bound before it is right afterwards."""
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    averaged = [torch.empty_like(p).normal_(0, 0.1) for p in m.parameters()]
    for _ in range(3):
        train_step(m, x, fine_tuning)
    with torch.no_grad():
        exchange(list(m.parameters()), averaged)
        m.eval()
        for _ in range(3):
            got = forward(m, x, fine_tuning)
        fresh = fresh_copy(m, kind, cuda_device).eval()
        same(got, forward(fresh, x, fine_tuning))
        exchange(list(m.parameters()), averaged)
    for p in averaged:
        p.fill_(float("nan"))
    want = train_step(fresh_copy(m, kind, cuda_device), x, fine_tuning)
    same(train_step(m, x, fine_tuning), want)


@pytest.mark.gpu
@pytest.mark.parametrize("fine_tuning", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_backward_after_the_module_and_its_weights_are_gone(cuda_device, kind, fine_tuning):
    """Between forward and backward a node keeps everything it reads: plan, weights, merged weights, workspaces."""
    x = rows(48, cuda_device)
    xs, grads = [], []
    for drop in (False, True):
        m = build(kind, cuda_device).train().requires_grad_(False)
        xd = x.clone().requires_grad_(True)
        for i in range(2):       # prepared, then bound
            torch.manual_seed(i)
            out = forward(m, xd, fine_tuning)
        if drop:
            del m
            gc.collect()
            junk = [torch.full((1 << 20,), float("nan"), device=cuda_device) for _ in range(8)]
        out[0].float().sum().backward()
        torch.cuda.synchronize()
        xs.append(out[0].detach())
        grads.append(xd.grad)
    del junk
    assert torch.equal(xs[0], xs[1]) and torch.equal(grads[0], grads[1])


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_a_module_that_ran_can_be_freed(cuda_device, kind):
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    for fine_tuning in (False, True):
        for _ in range(2):
            train_step(m, x, fine_tuning)
            with torch.no_grad():
                forward(m.eval(), x, fine_tuning)
    ref = weakref.ref(m)
    weight = weakref.ref(next(m.parameters()))
    gc.collect()
    gc.disable()            # no cycle through a binding: the memory is free at once
    try:
        del m
        assert ref() is None and weight() is None
    finally:
        gc.enable()


# ---- a backward belongs to the last training forward of its module ---------------------------

def other_layout(x):
    """The same values in a tensor that is not contiguous."""
    return x.t().contiguous().t()


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("what", ["fine_tuning", "not contiguous", "no_grad"])
def test_a_second_forward_before_the_backward_is_refused(cuda_device, kind, what):
    m = build(kind, cuda_device).train()
    x1, x2 = rows(48, cuda_device, 1), rows(48, cuda_device, 2)
    for _ in range(2):          # every form of the call prepared and bound
        for ft in (False, True):
            forward(m, x1.clone().requires_grad_(True), ft)[0].sum().backward()
    if what == "not contiguous":
        x1, x2 = other_layout(x1), other_layout(x2)
    first = forward(m, x1.requires_grad_(True))[0]
    if what == "no_grad":
        with torch.no_grad():
            forward(m, x2)
    else:
        forward(m, x2, what == "fine_tuning")
    with pytest.raises(RuntimeError, match="another training forward"):
        first.sum().backward()
    # and the module is usable afterwards
    same(train_step(m, x2), train_step(fresh_copy(m, kind, cuda_device), x2))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_forwards_of_two_sizes_before_their_backwards(cuda_device, kind):
    """Another number of rows has workspaces of its own: both backwards are right, in either order."""
    m = build(kind, cuda_device).train().requires_grad_(False)
    xs = [rows(n, cuda_device, n).requires_grad_(True) for n in (48, 32)]
    want = []
    for x in xs:
        torch.manual_seed(3)
        want += torch.autograd.grad(forward(m, x)[0].float().square().sum(), x)
    for order in ((0, 1), (1, 0)):
        outs = []
        for x in xs:
            torch.manual_seed(3)
            outs.append(forward(m, x)[0])
        for i in order:
            (g,) = torch.autograd.grad(outs[i].float().square().sum(), xs[i])
            assert torch.equal(g, want[i])


# ---- merged weights: one record of what they hold ----------------------------------------------

def adapters(m):
    return [p for n, p in m.named_parameters() if "lora" in n]


@pytest.mark.gpu
@pytest.mark.parametrize("size", [48, 20])
@pytest.mark.parametrize("kind", KINDS)
def test_adapters_exchanged_for_an_evaluation_and_back(cuda_device, kind, size):
    """.data moves no version counter: what the merged weights hold is told by addresses and versions together."""
    m, x, other = build(kind, cuda_device), rows(48, cuda_device), rows(size, cuda_device, 2)
    adapters_b = [torch.empty_like(p).normal_(0, 0.3) for p in adapters(m)]
    for _ in range(2):
        train_step(m, x, True)
    for _ in range(2):
        with torch.no_grad():
            exchange(adapters(m), adapters_b)
            got = forward(m.eval(), other, True)
            same(got, forward(fresh_copy(m, kind, cuda_device).eval(), other, True))
            exchange(adapters(m), adapters_b)
        want = train_step(fresh_copy(m, kind, cuda_device), x, True)
        same(train_step(m, x, True), want)


@pytest.mark.gpu
def test_adapters_of_another_rank_for_an_evaluation(cuda_device):
    """Adapters of rank 8 and back: the merged buffers of the bound training call belong to it."""
    m, x = build("ffn", cuda_device), rows(48, cuda_device)
    small = build("ffn", cuda_device, seed=3, rank=8)
    names = ("lora_gate_and_up_a", "lora_gate_and_up_b", "lora_down_a", "lora_down_b")

    def swap():
        for n in names:
            a, b = getattr(m, n), getattr(small, n)
            setattr(m, n, b), setattr(small, n, a)
    for _ in range(2):
        train_step(m, x, True)
    swap()
    with torch.no_grad():
        got = forward(m.eval(), x, True)
    fresh = fresh_copy(m, "ffn", cuda_device, rank=8).eval()
    fresh.lora_scale = m.lora_scale
    with torch.no_grad():
        same(got, forward(fresh, x, True))
    swap()
    gc.collect()
    want = train_step(fresh_copy(m, "ffn", cuda_device), x, True)
    same(train_step(m, x, True), want)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_adapters_exchanged_between_forward_and_backward(cuda_device, kind):
    """An evaluation with other adapters in between merges them into the same buffers: the backward merges its own again.
    (Another number of rows: the block's workspace holds the training forward's tensors.)"""
    m, x, other = build(kind, cuda_device), rows(48, cuda_device), rows(20, cuda_device, 2)
    want = train_step(fresh_copy(m, kind, cuda_device), x, True)
    adapters_b = [torch.empty_like(p).normal_(0, 0.3) for p in adapters(m)]
    for _ in range(2):
        train_step(m, x, True)
    m.train()
    for p in m.parameters():
        p.grad = None
    xd = x.clone().requires_grad_(True)
    torch.manual_seed(5)
    out = forward(m, xd, True)
    with torch.no_grad():
        exchange(adapters(m), adapters_b)
        forward(m.eval(), other, True)
        exchange(adapters(m), adapters_b)
    sum((o.float() ** 2).sum() for o in out).backward()
    same([*(o.detach() for o in out), xd.grad, *(p.grad for p in m.parameters() if p.grad is not None)], want)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_adapters_written_in_place(cuda_device, kind):
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    for i in range(3):
        want = train_step(fresh_copy(m, kind, cuda_device), x, True)
        same(train_step(m, x, True), want)
        with torch.no_grad():
            same(forward(m.eval(), x, True), forward(fresh_copy(m, kind, cuda_device).eval(), x, True))
            for p in adapters(m):
                p.mul_(1.25)


# ---- what a new workspace holds ------------------------------------------------------------------

@pytest.mark.gpu
def test_training_with_tokens_that_have_no_expert(cuda_device):
    """A token of NaN has no expert and no sorted row: the step reports it and gives the other tokens' gradients,
    whatever the new workspaces held (0x7f bytes here: as an index of a pair, far outside)."""
    m, x = build("moe", cuda_device, p=0.0), rows(200, cuda_device)
    m.train()
    with torch.no_grad():
        x[[3, 77, 199]] = float("nan")
    clean = torch.ones(200, dtype=torch.bool, device=cuda_device)
    clean[[3, 77, 199]] = False
    junk = [torch.full((1 << 24,), 0x7F, dtype=torch.uint8, device=cuda_device) for _ in range(4)]
    del junk
    xd = x.clone().requires_grad_(True)
    out, _ = m(xd)
    grad = torch.zeros_like(out)
    grad[clean] = 1.0
    out.backward(grad)
    torch.cuda.synchronize()
    assert m.device_status() != 0
    assert torch.isfinite(out[clean]).all() and torch.isfinite(xd.grad[clean]).all()
    assert all(torch.isfinite(p.grad).all() for n, p in m.named_parameters() if p.grad is not None and "gate." not in n)
    # the clean tokens' part is what the same step without the others gives
    only = fresh_copy(m, "moe", cuda_device, p=0.0).train()
    xo = x[clean].clone().requires_grad_(True)
    oo, _ = only(xo)
    oo.backward(torch.ones_like(oo))
    assert torch.equal(out[clean], oo)
    for (n, p), q in zip(m.named_parameters(), only.parameters()):
        if p.grad is not None and "experts" in n:
            assert (p.grad.float() - q.grad.float()).norm() <= 1e-3 * q.grad.float().norm(), n


# ---- what an autograd function in Python refused, kept or passed on --------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_forward_mode_derivatives_are_refused(cuda_device, kind):
    import torch.autograd.forward_ad as fw
    m, x = build(kind, cuda_device).train(), rows(48, cuda_device)
    for _ in range(3):           # unbound, then bound
        with fw.dual_level():
            with pytest.raises(NotImplementedError):
                m(fw.make_dual(x, torch.ones_like(x)))
            with torch.no_grad(), pytest.raises(NotImplementedError):
                m(fw.make_dual(x, torch.ones_like(x)))
        train_step(m, x)
    for transform in (lambda f: torch.func.grad(lambda z: f(z).float().sum())(x), lambda f: torch.func.vmap(f)(x[None]),
                      lambda f: torch.func.jvp(f, (x,), (torch.ones_like(x),))):
        with pytest.raises(RuntimeError):
            transform(lambda z: forward(m, z)[0])


@pytest.mark.gpu
def test_traced_training_forward(cuda_device):
    """torch.jit.trace of the feed-forward in training mode (no dropout, so that runs agree) computes and has gradients;
    the block's was refused and is."""
    m, x = build("ffn", cuda_device, p=0.0).train(), rows(48, cuda_device)
    for _ in range(2):
        train_step(m, x)
    traced = torch.jit.trace(m, (x,), check_trace=False)
    other = rows(48, cuda_device, 2)
    want = train_step(fresh_copy(m, "ffn", cuda_device, p=0.0), other)
    same(_traced_step(traced, m, other), want)
    block = build("moe", cuda_device).train()
    for _ in range(2):
        train_step(block, x)
        with pytest.raises(RuntimeError):
            torch.jit.trace(block, (x,), check_trace=False)


def _traced_step(traced, m, x):
    for p in m.parameters():
        p.grad = None
    x = x.clone().requires_grad_(True)
    y = traced(x)
    (y.float() ** 2).sum().backward()
    return [y.detach(), x.grad, *(p.grad for p in m.parameters() if p.grad is not None)]


@pytest.mark.gpu
def test_the_block_keeps_the_class_of_its_input(cuda_device):
    class Rows(torch.Tensor):
        pass
    m, x = build("moe", cuda_device, p=0.0), rows(48, cuda_device)
    for module in (m.train(), m.eval()):
        for _ in range(3):
            assert type(module(x)[0]) is torch.Tensor and type(module(x.as_subclass(Rows))[0]) is Rows
            assert torch.equal(module(x)[0], module(x.as_subclass(Rows))[0])


@pytest.mark.gpu
def test_saved_tensor_hooks_see_what_is_saved(cuda_device):
    """Input and, for the feed-forward, h: moved to the host and back between forward and backward."""
    from torch.autograd.graph import saved_tensors_hooks
    for kind, shapes in (("moe", [(48, D)]), ("ffn", [(48, D), (48, F)])):
        m, x = build(kind, cuda_device), rows(48, cuda_device)
        want = train_step(fresh_copy(m, kind, cuda_device), x)
        for _ in range(3):
            seen = []
            m.train()
            for p in m.parameters():
                p.grad = None
            xd = x.clone().requires_grad_(True)
            torch.manual_seed(5)
            with saved_tensors_hooks(lambda t: (seen.append(tuple(t.shape)), t.cpu())[1], lambda t: t.to(cuda_device)):
                out = forward(m, xd)
            assert seen == shapes
            sum((o.float() ** 2).sum() for o in out).backward()
            same([*(o.detach() for o in out), xd.grad, *(p.grad for p in m.parameters() if p.grad is not None)], want)


# ---- plain attributes are read by every call -----------------------------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_lora_scale_set_between_calls(cuda_device, kind):
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    for scale in (2.0, 0.5, 2.0):
        for ex in (m.experts if kind == "moe" else [m]):
            ex.lora_scale = scale
        new = fresh_copy(m, kind, cuda_device)
        for ex in (new.experts if kind == "moe" else [new]):
            ex.lora_scale = scale
        want = train_step(new, x, True)
        for _ in range(3):
            same(train_step(m, x, True), want)
        with torch.no_grad():
            want = forward(new.eval(), x, True)
            for _ in range(3):
                same(forward(m.eval(), x, True), want)


@pytest.mark.gpu
def test_slots_set_between_calls(cuda_device):
    m, x = build("moe", cuda_device), rows(48, cuda_device)
    for k in (2, 1, 3, 2):
        m.top_k = k
        new = fresh_copy(m, "moe", cuda_device)
        new.top_k = k
        want = train_step(new, x)
        for _ in range(3):
            same(train_step(m, x), want)
        with torch.no_grad():
            want = forward(new.eval(), x)
            for _ in range(3):
                same(forward(m.eval(), x), want)
        assert m.last["idx"].shape == (48, k)


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["ranks", "scales"])
def test_experts_with_ranks_and_scales_of_their_own(cuda_device, what):
    """Replaced adapters: every expert's, and each of its Linears', at a rank of its own. The gradients follow from those of
    the merged weights (one rounding behind fp32 sums)."""
    torch.manual_seed(0)
    m, x = build("moe", cuda_device, p=0.0), rows(200, cuda_device)
    for e, ex in enumerate(m.experts):
        if what == "scales":
            ex.lora_scale = 0.5 + e
            continue
        ra, rb = (4, 16, 33, 8)[e], (16, 5, 16, 24)[e]
        ex.lora_gate_and_up_a, ex.lora_gate_and_up_b = torch.nn.Linear(D, ra), torch.nn.Linear(ra, 2 * F)
        ex.lora_down_a, ex.lora_down_b = torch.nn.Linear(F, rb), torch.nn.Linear(rb, D)
    m.to(device=cuda_device, dtype=DT)
    for _ in range(3):
        train_step(m, x, True)
        for ex in m.experts:
            for w, a, b in ((ex.gate_and_up, ex.lora_gate_and_up_a, ex.lora_gate_and_up_b),
                            (ex.down, ex.lora_down_a, ex.lora_down_b)):
                G, g, A, av, B = (t.detach().cpu().double() for t in (w.weight.grad, w.bias.grad, a.weight, a.bias, b.weight))
                s = ex.lora_scale
                for got, ref in ((a.weight.grad, s * B.t() @ G), (b.weight.grad, s * (G @ A.t() + torch.outer(g, av))),
                                 (a.bias.grad, s * B.t() @ g), (b.bias.grad, s * g)):
                    ref = ref.to(DT).double()
                    assert (got.cpu().double() - ref).norm() <= 1e-3 * ref.norm()


@pytest.mark.gpu
def test_only_a_layernorm_is_folded_in(cuda_device):
    """Norms with as many weights that are none, on a call that is bound for a LayerNorm."""
    m, x = build("moe", cuda_device).eval(), rows(48, cuda_device)
    put = lambda norm: norm.to(device=cuda_device, dtype=DT)
    ln = put(torch.nn.LayerNorm(D))
    with torch.no_grad():
        want = fresh_copy(m, "moe", cuda_device).eval()(x, norm=ln)
        for _ in range(3):
            same(m(x, norm=ln), want)
            for norm in (torch.nn.GroupNorm(8, D), torch.nn.BatchNorm1d(D), torch.nn.LayerNorm((48, D)),
                         torch.nn.LayerNorm(D, elementwise_affine=False), torch.nn.LayerNorm(D, bias=False)):
                with pytest.raises((ValueError, AttributeError)):
                    m(x, norm=put(norm))


@pytest.mark.gpu
def test_output_gradients_at_any_address(cuda_device):
    """A gradient that starts two bytes behind a 16-byte boundary, as a slice of a concatenation does: the feed-forward
    takes it, the block refuses it."""
    x = rows(48, cuda_device)
    g = torch.randn(48, D, generator=torch.Generator().manual_seed(4)).to(DT).to(cuda_device)
    shifted = torch.zeros(48 * D + 8, dtype=DT, device=cuda_device)[1:1 + 48 * D].view(48, D)
    shifted.copy_(g)
    for kind in KINDS:
        m, got = build(kind, cuda_device, p=0.0).train(), []
        for grad in (g, shifted):
            xd = x.clone().requires_grad_(True)
            out = forward(m, xd)[0]
            if kind == "moe" and grad is shifted:
                with pytest.raises(MoeB200Error, match="backward failed with code -3: buffers must be 16-byte aligned"):
                    out.backward(grad)
                continue
            m.zero_grad(set_to_none=True)
            out.backward(grad)
            got.append([xd.grad, *(p.grad for p in m.parameters() if p.grad is not None)])
        if kind == "ffn":
            same(*got)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_device_status_is_that_of_the_last_large_call(cuda_device, dtype):
    """An error that nobody asked for does not stay with the calls after it."""
    m = build("moe", cuda_device).to(dtype).eval()
    good = torch.randn(3000, D, generator=torch.Generator().manual_seed(1)).to(device=cuda_device, dtype=dtype)
    bad = good.clone()
    bad[7] = float("nan")
    with torch.no_grad():
        for _ in range(2):
            m(good)
            assert m.device_status() == 0
            m(bad)
            m(good)
            assert m.device_status() == 0
            m(bad)
            assert m.device_status() != 0


# ---- copies ----------------------------------------------------------------------------------------

def test_copies_hold_no_state_of_calls():
    import copy
    import pickle
    for kind in KINDS:
        m = MOE(D, num_experts=E, d_ff=F) if kind == "moe" else FeedForward(D, d_ff=F)
        m._tws, m._tws_key = (torch.zeros(4), 4711, 16), (48, "cpu")
        for new in (copy.deepcopy(m), copy.copy(m), pickle.loads(pickle.dumps(m))):
            assert new._tws is None and new._tws_key is None and new._native is not m._native and new._plan is not m._plan
            assert all(torch.equal(a, b) for a, b in zip(new.state_dict().values(), m.state_dict().values()))


@pytest.mark.gpu
@pytest.mark.parametrize("fine_tuning", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_a_copy_of_a_module_that_ran(cuda_device, kind, fine_tuning):
    """Forwards and backwards of the module and its copy in turn: each has its own workspaces."""
    import copy
    m, x, z = build(kind, cuda_device), rows(48, cuda_device, 1), rows(48, cuda_device, 2)
    want = [train_step(fresh_copy(m, kind, cuda_device), t, fine_tuning) for t in (x, z)]
    for _ in range(2):
        train_step(m, x, fine_tuning)
    new = copy.deepcopy(m)
    for _ in range(3):
        outs, xs = [], []
        for module, t in ((m, x), (new, z)):
            for p in module.parameters():
                p.grad = None
            xs.append(t.clone().requires_grad_(True))
            torch.manual_seed(5)
            outs.append(forward(module.train(), xs[-1], fine_tuning))
        for module, out, xd, ref in zip((m, new), outs, xs, want):
            sum((o.float() ** 2).sum() for o in out).backward()
            same([*(o.detach() for o in out), xd.grad, *(p.grad for p in module.parameters() if p.grad is not None)], ref)


# ---- what is bound, and when ------------------------------------------------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_a_call_is_bound_when_it_comes_again(cuda_device, kind):
    m = build(kind, cuda_device).eval()
    bound = lambda x: (m._native.forward(x, None, None, 2) if kind == "moe" else m._native.forward(x, 1.0)) is not None
    with torch.no_grad():
        for n in (1, 2, 3, 48, 4):
            x = rows(n, cuda_device)
            same(forward(m, x), forward(fresh_copy(m, kind, cuda_device).eval(), x))
            assert not bound(x)
        forward(m, x)
        assert bound(x)
        for _ in range(5):       # other weights: another call
            for p in m.parameters():
                p.data = p.data * 0.5
            forward(m, x)
            assert not bound(x)
            same(forward(m, x), forward(fresh_copy(m, kind, cuda_device).eval(), x))
            assert bound(x)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_inputs_that_are_not_contiguous_take_the_bound_call(cuda_device, kind):
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    z = other_layout(x)
    assert not z.is_contiguous()
    want = train_step(fresh_copy(m, kind, cuda_device), x)
    train_step(m, z)
    prepare = m._plan.get
    m._plan.get = None           # from here on nothing is prepared
    for _ in range(2):
        xd = z.detach().requires_grad_(True)
        for p in m.parameters():
            p.grad = None
        torch.manual_seed(5)
        out = forward(m.train(), xd)
        sum((o.float() ** 2).sum() for o in out).backward()
        same([*(o.detach() for o in out), xd.grad, *(p.grad for p in m.parameters() if p.grad is not None)], want)
    m._plan.get = prepare
    with torch.no_grad():
        want = forward(fresh_copy(m, kind, cuda_device).eval(), x)
        for _ in range(2):
            same(forward(m.eval(), z), want)
        m._plan.get = None
        for _ in range(2):
            same(forward(m, z), want)
            if kind == "moe":
                same(forward(m, z, residual=z), forward(m, x, residual=x))
                same(forward(m, x, residual=z), forward(m, x, residual=x))


@pytest.mark.gpu
def test_the_last_call_can_be_cleared(cuda_device):
    m, x = build("moe", cuda_device).eval(), rows(48, cuda_device)
    assert m.last is None
    for train in (False, True):
        m.train(train)
        for _ in range(3):
            with torch.no_grad():
                m(x)
            kept = m.last
            assert kept["idx"].shape == (48, 2) and ("seed" in kept) == train
            m.last = None
            assert m.last is None and m.device_status() == 0
            with pytest.raises(ValueError):
                m.last = {}


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_gradients_that_are_wanted_are_those_of_all(cuda_device, kind):
    """Frozen base weights, frozen adapters, a frozen router, a frozen expert: what is left gets the gradient it gets when
    everything does."""
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    for fine_tuning in (False, True):
        m.requires_grad_(True)
        train_step(m, x, fine_tuning)
        want = {n: p.grad for n, p in m.named_parameters()}
        for frozen in (lambda n: "lora" not in n, lambda n: "lora" in n, lambda n: "gate." in n, lambda n: "experts.1" in n,
                       lambda n: "bias" in n, lambda n: "gate_and_up" in n, lambda n: True):
            for n, p in m.named_parameters():
                p.requires_grad_(not frozen(n))
            for _ in range(2):
                train_step(m, x, fine_tuning)
                for n, p in m.named_parameters():
                    assert (p.grad is None) == (frozen(n) or want[n] is None), n
                    assert p.grad is None or torch.equal(p.grad, want[n]), n


# ---- other ways to run a call ----------------------------------------------------------------------

@pytest.mark.gpu
@pytest.mark.parametrize("warm", [1, 3])
@pytest.mark.parametrize("n", [1, 48, 3000])
@pytest.mark.parametrize("kind", KINDS)
def test_calls_under_stream_capture(cuda_device, kind, n, warm):
    """Captured after one warm-up call (not bound yet) or three, replayed on other inputs."""
    m, x = build(kind, cuda_device).eval(), rows(n, cuda_device)
    side = torch.cuda.Stream()
    with torch.no_grad():
        with torch.cuda.stream(side):
            for _ in range(warm):
                forward(m, x)
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = forward(m, x)
        for seed in (5, 6):
            x.copy_(rows(n, cuda_device, seed))
            graph.replay()
            same(out, forward(fresh_copy(m, kind, cuda_device).eval(), x))


@pytest.mark.gpu
@pytest.mark.parametrize("fine_tuning", [False, True])
def test_a_training_step_under_stream_capture(cuda_device, fine_tuning):
    m, x = build("ffn", cuda_device, p=0.0).train(), rows(48, cuda_device).requires_grad_(True)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        for _ in range(2):
            m.zero_grad(set_to_none=True)
            m(x, fine_tuning=fine_tuning).float().square().sum().backward()
    torch.cuda.current_stream().wait_stream(side)
    m.zero_grad(set_to_none=True)
    x.grad = None
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = m(x, fine_tuning=fine_tuning)
        y.float().square().sum().backward()
    with torch.no_grad():
        x.copy_(rows(48, cuda_device, 7))
    graph.replay()
    got = [y.detach(), x.grad, *(p.grad for p in m.parameters() if p.grad is not None)]
    got = [t.clone() for t in got]
    same(got, train_step(fresh_copy(m, "ffn", cuda_device, p=0.0), x, fine_tuning))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_calls_in_inference_mode(cuda_device, kind):
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    for fine_tuning in (False, True):
        with torch.no_grad():
            want = forward(fresh_copy(m, kind, cuda_device).eval(), x, fine_tuning)
        for _ in range(3):
            with torch.inference_mode():
                z = x.clone()
                same(forward(m.eval(), z, fine_tuning), want)
                torch.manual_seed(5)
                trained = forward(m.train(), z, fine_tuning)
            same(trained, train_step(fresh_copy(m, kind, cuda_device), x, fine_tuning)[:len(trained)])


@pytest.mark.gpu
@pytest.mark.parametrize("fine_tuning", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_parts_replaced_and_sizes_back_and_forth(cuda_device, kind, fine_tuning):
    """A Linear, a Parameter, and the storage of one replaced under bound calls, at two sizes in turn."""
    m, xs = build(kind, cuda_device), [rows(n, cuda_device, n) for n in (48, 20)]
    ex = m.experts[1] if kind == "moe" else m

    def linear():
        ex.down = torch.nn.Linear(F, D).to(device=cuda_device, dtype=DT)

    def parameter():
        ex.gate_and_up.weight = torch.nn.Parameter(torch.randn_like(ex.gate_and_up.weight) * 0.1)

    def storage():
        ex.lora_down_b.weight.data = torch.randn_like(ex.lora_down_b.weight)
        ex.down.bias.data = torch.randn_like(ex.down.bias)

    def router():
        if kind == "moe":
            m.gate = torch.nn.Linear(D, E).to(device=cuda_device, dtype=DT)

    def written():
        with torch.no_grad():
            ex.lora_gate_and_up_a.weight.mul_(2.0)
            ex.down.weight.mul_(0.5)

    for change in (lambda: None, linear, parameter, storage, router, written):
        change()
        new = fresh_copy(m, kind, cuda_device)
        want = [train_step(new, x, fine_tuning) for x in xs]
        with torch.no_grad():
            want_eval = [forward(new.eval(), x, fine_tuning) for x in xs]
        for _ in range(3):
            for x, a, b in zip(xs, want, want_eval):
                same(train_step(m, x, fine_tuning), a)
                with torch.no_grad():
                    same(forward(m.eval(), x, fine_tuning), b)
                    same(forward(m, x, fine_tuning), b)


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_rows_of_another_width_are_refused(cuda_device, kind):
    """(The feed-forward in inference took them for rows of its own width, past the end of the input.)"""
    m = build(kind, cuda_device)
    for train in (True, False):
        m.train(train)
        for _ in range(3):
            with torch.no_grad():
                forward(m, rows(48, cuda_device))
                for width in (D // 2, D * 2, D - 8):
                    with pytest.raises(ValueError):
                        forward(m, torch.zeros(48, width, dtype=DT, device=cuda_device))


@pytest.mark.gpu
@pytest.mark.parametrize("kind", KINDS)
def test_adapters_at_an_address_that_others_had(cuda_device, kind):
    """A tensor's storage replaced twice between two calls, the second time by one that lies where the first call's lay:
    address and version are as before, the values are not."""
    m, x = build(kind, cuda_device), rows(48, cuda_device)
    ex = m.experts[2] if kind == "moe" else m
    p = ex.lora_gate_and_up_b.weight
    for _ in range(3):
        with torch.no_grad():
            want = forward(fresh_copy(m, kind, cuda_device).eval(), x, True)
            for _ in range(3):
                same(forward(m.eval(), x, True), want)
            address, held = p.data_ptr(), []
            p.data = torch.randn_like(p)
            while len(held) < 1000 and p.data_ptr() != address:
                new = torch.randn_like(p)
                if new.data_ptr() == address:
                    p.data = new
                held.append(new)
            assert p.data_ptr() == address


# ---- the decoder layer's attention and LayerNorm ----------------------------------------------

class Table(torch.nn.Module):
    def __init__(self, n, hd):
        super().__init__()
        self.register_buffer("pos_emb", torch.randn(n, 2 * hd, generator=torch.Generator().manual_seed(2)))


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,heads,kv,ft", [(1, 1, 2, 1, False), (2, 37, 4, 4, True), (3, 128, 4, 2, False)])
def test_attention_native_and_python_paths_agree(cuda_device, monkeypatch, B, S, heads, kv, ft):
    torch.manual_seed(S)
    m = Attention(D, 64, heads, kv, Table(128, 64)).to(device=cuda_device, dtype=DT).eval()
    m.embedding.float()
    x = rows(B * S, cuda_device).view(B, S, D)
    causal = torch.full((S, S), float("-inf"), device=cuda_device).triu(1)
    masks = [None, causal, causal.view(1, 1, S, S), causal.double(), causal.t().contiguous().t(), causal.cpu()]
    inputs = [x, x.transpose(0, 1).contiguous().transpose(0, 1)]
    with torch.no_grad():
        native = [m(i, mask, ft) for i in inputs for mask in masks]
        monkeypatch.setattr(_host, "attention", lambda *a: None)
        same(native, [m(i, mask, ft) for i in inputs for mask in masks])
        monkeypatch.undo()
        with pytest.raises(NotImplementedError):
            m(x, torch.zeros(S, S + 1, device=cuda_device))
        with pytest.raises(ValueError):                                     # a table that is too short
            m.embedding = Table(S - 1, 64).to(cuda_device)
            m(x)


@pytest.mark.gpu
@pytest.mark.parametrize("B,S,hidden,heads,kv,ft", [(1, 1, 64, 2, 1, False), (1, 16, 200, 4, 2, True), (17, 1, 1024, 16, 1, False),
                                                    (1, 65, 1032, 2, 2, False), (4, 32, 2048, 4, 1, False), (3, 7, 2056, 8, 8, False),
                                                    (3, 43, 256, 2, 1, False), (3, 43, 200, 8, 1, False), (4, 64, 1024, 16, 1, True),
                                                    (3, 100, 1032, 24, 2, False), (40, 63, 512, 8, 4, False)])
def test_attention_of_a_layer_in_one_call(cuda_device, B, S, hidden, heads, kv, ft):
    """LayerNorm, attention and skip connection in one call, and step by step: the same to the bit, on both sides of 128 rows,
    where the Linears become tiles (whole, and with K in two or four ranges). What the call cannot do is left to the steps."""
    torch.manual_seed(S)
    layer = LLMLayer(hidden, 64, heads, kv, Table(128, 64), expansion_factor=1, use_moe=False, device="cuda")
    layer = layer.to(device=cuda_device, dtype=DT).eval()
    layer.mqa.embedding.float()
    torch.nn.init.normal_(layer.norm1.weight)
    torch.nn.init.normal_(layer.norm1.bias)
    x = torch.randn(B, S, hidden, generator=torch.Generator().manual_seed(B)).to(device=cuda_device, dtype=DT)
    mask = torch.full((S, S), float("-inf"), device=cuda_device).triu(1)
    with torch.no_grad():
        args = layer.mqa._arguments(x, mask, ft)
        norm = (layer.norm1.weight, layer.norm1.bias, layer.norm1.eps)
        want = layer.mqa(_layernorm(layer.norm1, x), mask, ft) + x
        # torch's Linears around the same core: sums in another order, and bf16 between the steps
        xn = _layernorm(layer.norm1, x)
        lib_qkv, own_qkv = torch.nn.functional.linear(xn, args[1], args[2]), _linear_rows(args[13], xn, *args[1:5])[0] \
            if layer.mqa._own_linears(args, B * S, hidden, heads * 64) else None
        if own_qkv is not None:
            assert (lib_qkv.float() - own_qkv.float()).norm() <= 2.0 ** -8 * lib_qkv.float().norm()
        one = _host.attention(*args, *norm)
        assert (one is None) == (B * S > 128 and heads % 8 != 0)
        if one is not None:
            assert torch.equal(one, want)
        assert torch.equal(layer._attend(x, mask, ft), want)
        seen = []
        handle = layer.mqa.register_forward_hook(lambda *a: seen.append(a))
        assert torch.equal(layer._attend(x, mask, ft), want) and len(seen) == 1
        handle.remove()
        assert layer.mqa.device_status() == 0
        odd = torch.empty(x.numel() + 1, device=cuda_device, dtype=DT)[1:].view_as(x).copy_(x)
        assert _host.attention(odd, *args[1:], *norm) is None
        assert _host.attention(*args, norm[0][:8], *norm[1:]) is None
    assert _host.attention(*args, *norm) is None                            # gradients are wanted


def test_own_linears_of_the_attention_give_no_derivatives():
    """The attention's Linears are torch's where gradients or tangents of one of their tensors are wanted."""
    import torch.autograd.forward_ad as fw
    m = Attention(D, 64, 8, 1, Table(16, 64)).to(dtype=DT).eval().requires_grad_(False)
    x = rows(32, "cpu").view(2, 16, D)
    own = lambda: m._own_linears(m._arguments(x, None, False), 32, D, 8 * 64)
    assert own()
    for p in (m.o.weight, m.o.bias, m.gate.bias):
        p.requires_grad_(True)
        assert not own()
        with torch.no_grad():
            assert own()
        p.requires_grad_(False)
    with fw.dual_level():
        x = fw.make_dual(x, torch.ones_like(x))
        assert not own()


def test_sizes_of_the_own_linears():
    """Products that are over before a library's have begun, and tiles that fill the chip; the native call and the module
    give the same answer."""
    own = lambda N, *a: lib.moe_b200_attention_linears(N, *a, 64)
    assert [own(N, 1024, 16, 1) for N in (1, 37, 64, 128, 129, 512, 32768)] == [1] * 7
    assert [own(N, 2048, 32, 8) for N in (1, 16, 17, 128, 129, 4095, 4096)] == [1, 1, 0, 0, 0, 0, 1]
    assert [own(N, 1024, 16, 16) for N in (64, 65, 128, 129)] == [1, 0, 0, 1]
    assert [own(N, 1536, 24, 6) for N in (32, 33, 129)] == [1, 0, 1] and own(129, 1544, 24, 6) == 0 and own(129, 1536, 25, 5) == 0
    assert own(0, 1024, 16, 1) == 0 and own(1, 1024, 0, 1) == 0 and own(1, 1 << 30, 1, 1) == 0
    m = Attention(2048, 64, 32, 8, Table(128, 64)).to(dtype=DT).eval().requires_grad_(False)
    for N in (16, 17):
        x = torch.zeros(1, N, 2048, dtype=DT)
        assert m._own_linears(m._arguments(x, None, False), N, 2048, 2048) is (N == 16)


@pytest.mark.gpu
@pytest.mark.parametrize("B,S", [(1, 17), (1, 128), (3, 50)])
def test_large_attentions_keep_torchs_linears(cuda_device, monkeypatch, B, S):
    torch.manual_seed(S)
    layer = LLMLayer(2048, 64, 32, 8, Table(128, 64), expansion_factor=1, use_moe=False, device="cuda")
    layer = layer.to(device=cuda_device, dtype=DT).eval().requires_grad_(False)
    m, x = layer.mqa, torch.randn(B, S, 2048, generator=torch.Generator().manual_seed(B)).to(device=cuda_device, dtype=DT)
    m.embedding.float()
    qkv, gate = [torch.nn.functional.linear(x, lin.weight, lin.bias) for lin in (m.qkv, m.gate)]
    core = torch.empty(B, S, 2048, device=cuda_device, dtype=DT)
    check(lib.moe_b200_attention(qkv.data_ptr(), gate.data_ptr(), m._pos_table(cuda_device).data_ptr(), None, B, S, 32, 8, 64,
                                 float(m.scaler), core.data_ptr(), torch.cuda.current_stream().cuda_stream), "attention")
    want = torch.nn.functional.linear(core, m.o.weight, m.o.bias)
    assert torch.equal(m(x), want)
    args = m._arguments(x, None, False)
    assert _host.attention(*args, layer.norm1.weight, layer.norm1.bias, layer.norm1.eps) is None
    assert torch.equal(layer._attend(x, None, False), m(_layernorm(layer.norm1, x)) + x)
    monkeypatch.setattr(_host, "attention", lambda *a: None)
    assert torch.equal(m(x), want)


def test_status_of_a_layer():
    """Of its attention or of its block, each returned once; and of an attention that was saved before it had any."""
    layer = LLMLayer(D, 64, 2, 1, Table(16, 64), expansion_factor=1, use_moe=True, num_experts=E, device="cuda")
    assert layer.device_status() == 0 and layer.mqa.device_status() == 0
    words = layer.mqa._status_words(torch.device("cpu"))
    words[:3] = torch.tensor([1, 34, 5], dtype=torch.int32)
    assert layer.device_status() == 1 and layer.device_status() == 0 and not words.any()
    words[0] = 1
    layer.moe.device_status = lambda: 2
    assert [layer.device_status(), layer.device_status()] == [1, 2]
    old = Attention(D, 64, 2, 1, Table(16, 64))
    old.__dict__.pop("_status", None)
    assert old.device_status() == 0 and old._status_words(torch.device("cpu")).numel() == 16
    plain = LLMLayer(D, 64, 2, 1, Table(16, 64), use_moe=False)
    plain.mqa = torch.nn.Identity()
    assert plain.device_status() == 0


class Scaled(torch.Tensor):
    """A weight that is half of what it stands for, and keeps it elsewhere."""

    @staticmethod
    def __new__(cls, half):
        return torch.Tensor._make_wrapper_subclass(cls, half.shape, dtype=half.dtype, device=half.device)

    def __init__(self, half):
        self.half_ = half

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        if func is torch.nn.functional.linear:
            x, w, b = args
            return torch.nn.functional.linear(x, w.half_ * 2, b)
        return super().__torch_function__(func, types, args, kwargs or {})

    @classmethod
    def __torch_dispatch__(cls, func, types, args=(), kwargs=None):
        raise NotImplementedError(func)


def test_own_linears_of_the_attention_leave_other_weights_alone():
    m = Attention(D, 64, 8, 1, Table(16, 64)).to(dtype=DT).eval().requires_grad_(False)
    args = m._arguments(rows(32, "cpu").view(2, 16, D), None, False)
    assert m._own_linears(args, 32, D, 8 * 64)
    for i in (1, 3, 5):
        assert not m._own_linears((*args[:i], Scaled(args[i]), *args[i + 1:]), 32, D, 8 * 64)


@pytest.mark.gpu
def test_attention_with_weights_of_a_class_of_their_own(cuda_device):
    m = Attention(D, 64, 8, 1, Table(16, 64)).to(device=cuda_device, dtype=DT).eval().requires_grad_(False)
    m.embedding.float()
    x = rows(32, cuda_device).view(2, 16, D)
    want = m(x)
    for lin in (m.qkv, m.gate, m.o):
        half = lin.weight.detach() / 2
        del lin.weight
        lin.weight = Scaled(half)
    # the library's Linears against torch's: sums in another order, rounded to bf16
    assert (m(x).float() - want.float()).norm() <= 2.0 ** -7 * want.float().norm()


@pytest.mark.gpu
@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("B,S", [(1, 1), (3, 17), (5, 64)])
def test_gradients_of_the_output_projection(cuda_device, monkeypatch, B, S, native):
    """With all but the output projection frozen it receives torch's gradients, from the attention and from a layer."""
    torch.manual_seed(S)
    layer = LLMLayer(256, 64, 8, 2, Table(128, 64), expansion_factor=1, use_moe=False, device="cuda")
    layer = layer.to(device=cuda_device, dtype=DT).eval().requires_grad_(False)
    m = layer.mqa
    m.embedding.float()
    m.o.requires_grad_(True)
    if not native:
        monkeypatch.setattr(_host, "attention", lambda *a: None)
    x = torch.randn(B, S, 256, generator=torch.Generator().manual_seed(B)).to(device=cuda_device, dtype=DT)
    g = torch.randn(B, S, 256, generator=torch.Generator().manual_seed(9)).to(device=cuda_device, dtype=DT)
    for whole in (False, True):
        xn = _layernorm(layer.norm1, x) if whole else x
        with torch.no_grad():
            qkv, gate = [torch.nn.functional.linear(xn, lin.weight, lin.bias) for lin in (m.qkv, m.gate)]
            core = torch.empty(B, S, 512, device=cuda_device, dtype=DT)
            check(lib.moe_b200_attention(qkv.data_ptr(), gate.data_ptr(), m._pos_table(cuda_device).data_ptr(), None, B, S, 8, 2, 64,
                                         float(m.scaler), core.data_ptr(), torch.cuda.current_stream().cuda_stream), "attention")
        want = torch.nn.functional.linear(core, m.o.weight, m.o.bias)
        want = want + x if whole else want
        wanted = torch.autograd.grad(want, [m.o.weight, m.o.bias], g)
        got = layer._attend(x, None, False) if whole else m(x)
        same((got, *torch.autograd.grad(got, [m.o.weight, m.o.bias], g)), (want, *wanted))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [DT, torch.float32])
def test_layernorm_native_and_left_alone(cuda_device, dtype):
    norm = torch.nn.LayerNorm(72).to(device=cuda_device, dtype=dtype)
    torch.nn.init.normal_(norm.weight)
    x = torch.randn(5, 3, 72, generator=torch.Generator().manual_seed(3)).to(device=cuda_device, dtype=dtype)
    args = (norm.weight, norm.bias, norm.eps)
    assert _host.layernorm(x, *args) is None                                # gradients are wanted
    with torch.no_grad():
        got, want = _host.layernorm(x, *args), norm(x)
        # a rounding of the result, and of the statistics
        assert (got.float() - want.float()).abs().max() <= (2.0 ** -7 if dtype == DT else 1e-5) * want.abs().max()
        assert _host.layernorm(x[..., :64], *args) is None                  # another width
        assert _host.layernorm(x.half(), *args) is None
        assert _host.layernorm(x[:0], *args) is None
        odd = torch.empty(15 * 72 + 1, device=cuda_device, dtype=dtype)[1:].view(5, 3, 72).copy_(x)
        assert _host.layernorm(odd, *args) is None                          # not on a 16-byte boundary
        with torch.autocast("cuda"):
            assert _host.layernorm(x, *args) is None


@pytest.mark.gpu
def test_decoder_layer_in_the_modes_that_see_its_calls(cuda_device):
    """Under autocast and torch function modes the layer runs the same kernels."""
    from torch.overrides import TorchFunctionMode

    class Watching(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    torch.manual_seed(4)
    layer = LLMLayer(D, 64, 2, 1, Table(128, 64), expansion_factor=2, use_moe=True, num_experts=E, device="cuda")
    layer = layer.to(device=cuda_device, dtype=DT).eval()
    layer.mqa.embedding.float()
    torch.nn.init.normal_(layer.norm1.weight)
    x = rows(2 * 37, cuda_device).view(2, 37, D)
    mask = torch.full((37, 37), float("-inf"), device=cuda_device).triu(1)
    with torch.no_grad():
        want = layer(x, mask)
        with torch.autocast("cuda", dtype=DT):
            same(layer(x, mask), want)
        with torch.device("cuda"):
            same(layer(x, mask), want)
        with Watching():
            same(layer(x, mask), want)
        norm = layer.norm1
        native = _host.layernorm(x, norm.weight, norm.bias, norm.eps)
        for args in ((x,), (x.transpose(0, 1).contiguous().transpose(0, 1),)):
            with torch.autocast("cuda", dtype=DT):
                assert torch.equal(_layernorm(norm, *args), native)
            assert torch.equal(_layernorm(norm, *args), native)
        # what the row kernel cannot read stays torch's: rows at an odd place, none at all
        odd = torch.empty(x.numel() + 1, device=cuda_device, dtype=DT)[1:].view_as(x).copy_(x)
        same([_layernorm(norm, odd), _layernorm(norm, x[:0])], [norm(odd), norm(x[:0])])
    assert _layernorm(norm, x).requires_grad
