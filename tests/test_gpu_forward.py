"""The whole block through the drop-in module (which calls moe_b200_forward)
against the CPU oracle and the fixtures generated from the reference class."""
import hashlib
import json
from pathlib import Path

import numpy as np
import pytest
import torch

import helpers
from gemmallm_b200 import MOE, _cabi, synthetic
from gemmallm_b200._cabi import check, lib
from oracle import moe_oracle

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"


def sha(t):
    return hashlib.sha256(t.contiguous().numpy().tobytes()).hexdigest()


def build(params, d, E, f, k, dtype, dev):
    m = MOE(d, num_experts=E, d_ff=f, top_k=k, device="cuda").eval()
    synthetic.load_into(m, params, dtype, dev)
    return m


def check_against_oracle(m, params, x, k, dtype, dev, residual=None):
    """Routing bit-exact given the kernel's logits; output within the block's
    tolerance under identical routing: fp32 max-abs 1e-4, bf16 relative 2e-2."""
    N, d = x.shape
    xin = x.to(dtype).to(dev).view(1, N, d)
    res = None if residual is None else residual.to(dtype).to(dev).view(1, N, d)
    with torch.no_grad():
        out, aux = m(xin, residual=res)
    torch.cuda.synchronize()
    assert m.device_status() == 0
    last = {n: t.cpu() for n, t in m.last.items()}
    with torch.no_grad():
        o = moe_oracle.moe_forward(x, params, k, logits=last["logits"])
    ties = moe_oracle.tie_rows(o["probs"], k)
    ok = ~ties
    assert torch.equal(last["idx"][ok].long(), o["idx"][ok])
    if not ties.any():
        assert torch.equal(last["cnt_slot"].long(), o["cnt_slot"])
    assert int(last["offsets"][-1]) == N * k
    assert torch.allclose(last["w"][ok], o["w"][ok], atol=2e-6, rtol=0)
    assert abs(float(aux) - float(o["aux"])) <= 1e-5 * abs(float(o["aux"])) + 1e-7
    ref = o["out"] if residual is None else o["out"] + residual
    got = out.view(N, d).float().cpu()
    err = (got - ref)[ok].abs().max()
    if dtype == torch.float32:
        assert err <= 1e-4, f"max-abs {err}"
    else:
        assert err <= 2e-2 * ref.abs().max(), f"max-abs {err} vs scale {ref.abs().max()}"
        assert (got - ref)[ok].norm() <= 2e-2 * ref[ok].norm()
    return last, o


def test_tiny_fixture_from_reference(cuda_device):
    z = np.load(GOLDEN / "tiny_k2.npz")
    z = {n: torch.from_numpy(z[n]) for n in z.files}
    params = {n: z[n] for n in ("gate_w", "gate_b", "w1", "b1", "w2", "b2")}
    m = build(params, 32, 4, 64, 2, torch.float32, cuda_device)
    with torch.no_grad():
        out, aux = m(z["x"].to(cuda_device).view(2, 12, 32))
    torch.cuda.synchronize()
    assert torch.equal(m.last["idx"].cpu(), z["idx"])
    assert torch.equal(m.last["cnt_slot"].cpu(), z["cnt_slot"])
    assert (out.view(24, 32).cpu() - z["out"]).abs().max() <= 1e-4
    assert abs(float(aux) - float(z["aux"])) <= 1e-6


@pytest.mark.parametrize("N,d,E,k", [(1, 8, 5, 2), (16, 72, 8, 2), (17, 512, 9, 1), (129, 264, 16, 5), (300, 2048, 32, 4),
                                     (2047, 64, 8, 2), (2048, 64, 17, 2)])
def test_fp32_routing_in_one_launch(cuda_device, N, d, E, k):
    """Rows, counts and copies as the dispatch kernel lays the same choices out, twice on one workspace; logits against
    64 bits (chains of at most 32 products and a tree: 2^-24 times a few)."""
    params = synthetic.make_params(d, E, 8, seed=N + E)
    params["gate_b"] = torch.randn(E, generator=torch.Generator().manual_seed(E)) * 0.3
    x = torch.randn(N, d, generator=torch.Generator().manual_seed(N))
    m = build(params, d, E, 8, k, torch.float32, cuda_device)
    for _ in range(2):
        last, _ = check_against_oracle(m, params, x, k, torch.float32, cuda_device)
    ref = torch.nn.functional.linear(x.double(), params["gate_w"].double(), params["gate_b"].double())
    assert (last["logits"].double() - ref).norm() <= 3e-7 * ref.norm()
    disp = helpers.dispatch(x.to(cuda_device), m.last["idx"], E)
    perm = m._view("perm", torch.float32, (N * k, d))
    assert torch.equal(perm, disp["perm"])
    for name in ("offsets", "row_of", "cnt_slot"):
        assert torch.equal(m.last[name], disp[name]), name


# Tokens in planes: one to 160 tokens a tile (and an expert of more), the down product whole and in two to eight ranges of K
# that end early, boxes of 32 to 160 rows, widths that are no multiple of 32, 64 or 128.
@pytest.mark.parametrize("N,d,f,E,k,special", [(1, 64, 264, 8, 2, ""), (7, 264, 1096, 4, 3, ""), (80, 512, 2048, 1, 1, ""),
                                               (161, 72, 1024, 2, 1, ""), (160, 1032, 200, 2, 2, ""), (400, 264, 512, 3, 2, ""),
                                               (2048, 128, 72, 17, 2, ""), (1300, 1024, 136, 8, 3, ""),
                                               (50, 264, 1024, 4, 2, "inf"), (700, 512, 2048, 8, 2, "inf"),
                                               (40, 264, 1024, 4, 2, "end"), (512, 512, 2048, 8, 2, "end")])
def test_fp32_calls_on_planes(cuda_device, N, d, f, E, k, special):
    """The whole call against the products that split their own activations, on the same routing: the products are the same,
    the sums of the ranges of K are added in another order."""
    params = synthetic.make_params(d, E, f, seed=N + f)
    g = torch.Generator().manual_seed(N)
    x = torch.randn(N, d, generator=g)
    if special == "inf":
        params["w1"][0, 9, 7], params["w2"][1, 11, 100], params["w1"][1, f + 2, 1] = 1e4, float("inf"), -float("inf")
        params["w2"].view(torch.int32)[0, 13, 5] = 0x7F800001      # NaN whose upper half alone would be an infinity
    if special == "end":
        # h = 64 up: products of h and w2 whose first parts cancel while the others sum up to more than the largest number
        top, near = 2.0 ** 127, 1 + 2.0 ** -7 - 2.0 ** -23
        params["w1"].zero_(), params["b1"].zero_(), params["w2"].zero_()
        params["b1"][:, :f] = 64.0
        params["b1"][:, f:f + 256] = torch.tensor([1.9921875 * top, near * top, near * top, 0.03125 * top] * 64) / 64
        params["w2"][:, ::2, :256] = torch.tensor([-1.0, near, near, -1.0] * 64)
    m = build(params, d, E, f, k, torch.float32, cuda_device)
    with torch.no_grad():
        out, _ = m(x.to(cuda_device).view(1, N, d))
    assert m.device_status() == 0
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    disp = helpers.dispatch(x.to(cuda_device), m.last["idx"], E)
    _, y, status = helpers.experts(disp["perm"], disp["offsets"], plan)
    assert status.cpu()[0] == 0
    want = helpers.combine(y, disp["row_of"], m.last["w"]).cpu()
    got = out.view(N, d).cpu()
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.isinf(), want.isinf()) and torch.equal(got[got.isinf()], want[want.isinf()])
    ok = want.isfinite()
    assert ok.any()
    if special == "end":
        # 256 sums of at most 2^128, each rounded, on both sides: 2^10 2^-24 2^127, where the result is 2^126
        assert want[:, ::2].abs().max() > 1e37
        assert (got[ok] - want[ok]).abs().max() <= 1.3e-4 * want[ok].abs().max()
    else:
        # sums of at most eight ranges and a read-out per 64 of K, each rounded to 2^-24
        assert (got[ok].double() - want[ok].double()).norm() <= 5e-7 * want[ok].double().norm()


# four, six and nine tokens a block, the last block with fewer, one to four of a warp's tokens side by side, a row's pieces over
# two to eight warps
@pytest.mark.parametrize("N,d,E,k", [(18, 8, 3, 2), (513, 1032, 8, 2), (645, 72, 9, 3), (1150, 264, 24, 1)])
def test_fp32_routing_by_tokens_of_a_block(cuda_device, N, d, E, k):
    test_fp32_routing_in_one_launch(cuda_device, N, d, E, k)


@pytest.mark.parametrize("N,fold", [(1, False), (40, False), (2048, False), (2049, False), (300, True), (2049, True)])
def test_fp32_tokens_of_nan(cuda_device, N, fold):
    """On both sides of 2048 tokens, with and without a folded LayerNorm: a token of NaN has no expert, its output is the
    residual, the status says so, and the other tokens are as without it. The status is that of the last call."""
    d, E, f, k = 64, 8, 128, 2
    params = synthetic.make_params(d, E, f, seed=N)
    m = build(params, d, E, f, k, torch.float32, cuda_device)
    x = torch.randn(1, N, d, generator=torch.Generator().manual_seed(N)).to(cuda_device)
    norm = torch.nn.LayerNorm(d, device=cuda_device) if fold else None
    bad = x.clone()
    rows = sorted({0, N // 3, N - 1})
    bad[0, rows, 5] = float("nan")
    other = torch.ones(N, dtype=torch.bool, device=cuda_device)
    other[rows] = False
    with torch.no_grad():
        for _ in range(2):
            want, _ = m(x, residual=x, norm=norm)
            m(bad, residual=x, norm=norm)
            m(x, residual=x, norm=norm)
            assert m.device_status() == 0
            got, aux = m(bad, residual=x, norm=norm)
            assert m.device_status() == 2 and m.device_status() == 0
            assert torch.equal(got[0, rows], x[0, rows]) and aux.isnan()
            assert m.last["row_of"][rows].eq(-1).all() and int(m.last["offsets"][-1]) == (N - len(rows)) * k
            assert torch.allclose(got[0, other], want[0, other], atol=1e-5, rtol=0)
            assert m(bad, norm=norm)[0][0, rows].eq(0).all() and m.device_status() == 2


# past the rows of the small calls: blocks of one group of 16 tokens and of one token more, a last block of one token, the most
# tokens and one more, rows of one piece and of several rounds, one expert and 64, one slot and eight
@pytest.mark.parametrize("N,d,E,k", [(2049, 8, 1, 1), (2500, 1032, 8, 2), (2369, 2056, 16, 8), (18944, 64, 9, 2), (18945, 64, 9, 2),
                                     (4737, 520, 3, 3), (1025, 2056, 64, 4), (3001, 64, 40, 2), (6000, 72, 32, 1), (2200, 40, 17, 2)])
def test_routing_of_thousands_of_tokens(cuda_device, N, d, E, k):
    """As the general router and dispatch give it, also where tokens or logits are not finite (up to 16 experts)."""
    x = torch.randn(N, d, generator=torch.Generator().manual_seed(E + N)).bfloat16().to(cuda_device)
    params = synthetic.make_params(d, E, 8, seed=N)
    m = build(params, d, E, 8, k, torch.bfloat16, cuda_device)
    gate = (m.gate.weight.detach(), m.gate.bias.detach())
    mag = x.float().abs() @ gate[0].float().abs().T + gate[1].float().abs()
    nan, inf = float("nan"), float("inf")
    for values in [(), (nan,), (-inf,), (inf, -inf), (nan,) * E, (-inf,) * (E - 1)][:6 if E <= 16 else 1]:
        if len(values) <= E:
            m.gate.bias.data.copy_(params["gate_b"])
            m.gate.bias.data[:len(values)] = torch.tensor(values, dtype=torch.bfloat16)
        with torch.no_grad():
            m(x.view(1, N, d))
        last = {n: t.clone() for n, t in m.last.items()}
        status = m.device_status()
        logits, idx, w, psum_part = helpers.router(x, *gate, k)
        # fp32 sums of d products in another order: d 2^-24 of their sum of magnitudes, at the worst
        diff = (last["logits"] - logits).abs()
        assert bool(((diff <= 2 * d * 2.0 ** -24 * mag) | ~logits.isfinite()).all()), values
        same = (last["idx"] == idx).all(1).cpu()
        if not values:
            r = moe_oracle.route_from_logits(last["logits"].cpu(), k)
            assert bool(same[~moe_oracle.tie_rows(r["probs"], k)].all())
        assert int((~same).sum()) <= N // 500, values      # near-ties
        assert torch.allclose(last["w"].cpu()[same], w.cpu()[same], atol=4e-6, rtol=0, equal_nan=True), values
        disp = helpers.dispatch(x, last["idx"], E, psum_part)
        for name in ("offsets", "row_of", "cnt_slot"):
            assert torch.equal(last[name], disp[name]), (values, name)
        assert torch.allclose(last["psum"], disp["psum"], rtol=1e-5, atol=1e-6, equal_nan=True), values
        assert status == int(disp["status"][0]), values


# router and dispatch in one launch, up to 2048 tokens and 4096 rows and beyond
@pytest.mark.parametrize("N,d,E,k", [(1, 64, 64, 4), (130, 1024, 40, 2), (700, 64, 33, 8), (2048, 72, 64, 2), (2200, 64, 17, 2),
                                     (3000, 128, 32, 4), (3001, 64, 40, 8), (1025, 2056, 64, 4)])
def test_logits_of_many_experts_that_are_not_finite(cuda_device, N, d, E, k):
    """As the general router of 17 to 64 experts has it: NaN is not chosen while there are numbers, and the weights are those of
    the chosen alone. Where a token has fewer than k logits above minus infinity its slots still have experts of their own."""
    x = torch.randn(N, d, generator=torch.Generator().manual_seed(E + N)).bfloat16().to(cuda_device)
    params = synthetic.make_params(d, E, 8, seed=N)
    m = build(params, d, E, 8, k, torch.bfloat16, cuda_device)
    gate = (m.gate.weight.detach(), m.gate.bias.detach())
    nan, inf = float("nan"), float("inf")
    for values, token in [({0: nan}, 0.), ({E - 1: nan, 9: nan}, 0.), ({3: -inf}, 0.), ({0: inf, 1: -inf}, 0.), ({2: inf, 5: inf}, 0.),
                          (dict.fromkeys(range(E), nan), 0.), (dict.fromkeys(range(E - 1), -inf), 0.),
                          (dict.fromkeys(range(E), -inf), 0.), ({}, nan), ({}, inf)]:
        m.gate.bias.data.copy_(params["gate_b"])
        for e, v in values.items():
            m.gate.bias.data[e] = v
        xx = x.clone()
        if token != 0.:
            xx[N // 2, 3] = token
        with torch.no_grad():
            m(xx.view(1, N, d))
        got_idx, got_w = m.last["idx"].cpu(), m.last["w"].cpu()
        assert m.device_status() == 0, values
        logits, idx, w = [t.cpu() for t in helpers.router(xx, *gate, k)[:3]]
        enough = (logits > -inf).sum(1) >= k
        same = (got_idx == idx).all(1)
        assert int((enough & ~same).sum()) <= N // 500, values      # near-ties
        assert got_idx.min() >= 0 and got_idx.max() < E
        ordered = got_idx.sort(1).values
        assert (ordered[:, 1:] != ordered[:, :-1]).all(), values
        # fp32 sums of the logits in another order, as above; without k numbers the choice is another one, the weights are the same
        assert torch.allclose(got_w[same | ~enough], w[same | ~enough], atol=4e-6, rtol=0, equal_nan=True), values


@pytest.mark.parametrize("N,E,k,norm", [(3000, 8, 2, False), (2300, 40, 2, False), (3000, 8, 2, True), (300, 8, 2, None)])
def test_large_calls_take_nothing_from_a_call_that_timed_out(cuda_device, N, E, k, norm):
    """Status words and counters as a wait that ran out leaves them: the next large call, and the next training step (norm:
    None) of any size, gives what a call on a clean workspace gives, and its own status."""
    d, f = 64, 128
    m = build(synthetic.make_params(d, E, f, seed=N), d, E, f, k, torch.bfloat16, cuda_device).train(norm is None)
    x = torch.randn(1, N, d, generator=torch.Generator().manual_seed(E)).bfloat16().to(cuda_device)
    ln = torch.nn.LayerNorm(d).to(device=cuda_device, dtype=torch.bfloat16) if norm else None

    def call():
        torch.manual_seed(3)
        with torch.set_grad_enabled(norm is None):
            out, aux = m(x, norm=ln) if norm else m(x)
        return out.detach().clone(), aux.detach().clone(), *(m.last[n].clone() for n in ("logits", "idx", "w", "row_of", "psum"))

    want = call()
    assert m.device_status() == 0
    region = m._view("status", torch.int32, (_cabi.READY_OFFSET + _cabi.READY_INTS,))
    for left in (1, 16, 1 << 20, -5):
        region.fill_(left)
        assert all(torch.equal(a, b) for a, b in zip(call(), want)) and m.device_status() == 0


@pytest.mark.parametrize("N,E,k", [(2049, 8, 2), (2500, 16, 3), (5000, 9, 8)])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_tokens_that_are_not_finite_behind_a_folded_layernorm(cuda_device, N, E, k, value):
    """Routed as by the general folded router, whichever experts that leaves: with any the output is NaN, and it is reported
    where there are fewer than k. The other tokens are as without them."""
    d, dev = 128, cuda_device
    params = synthetic.make_params(d, E, 32, seed=N)
    m = build(params, d, E, 32, k, torch.bfloat16, dev)
    norm = torch.nn.LayerNorm(d).to(device=dev, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(E)
    with torch.no_grad():
        norm.weight.copy_(1 + torch.randn(d, generator=g) / 4), norm.bias.copy_(torch.randn(d, generator=g) / 4)
    x = torch.randn(N, d, generator=g).bfloat16().to(dev)
    rows = torch.arange(0, N, 97, device=dev)
    bad = x.clone()
    bad[rows, torch.arange(len(rows), device=dev) % d] = value      # (with an infinity in the first column no logit is left)
    wn, c = torch.empty(E, d, dtype=torch.bfloat16, device=dev), torch.empty(2 * E, device=dev)
    gate, s = (m.gate.weight.detach(), m.gate.bias.detach()), helpers.stream(dev)
    check(lib.moe_b200_norm_fold(gate[0].data_ptr(), gate[1].data_ptr(), norm.weight.data_ptr(), norm.bias.data_ptr(), E, d,
                                 _cabi.BF16, wn.data_ptr(), c.data_ptr(), s), "norm_fold")
    logits, idx = torch.empty(N, E, device=dev), torch.empty(N, k, dtype=torch.int32, device=dev)
    w, part = torch.empty(N, k, device=dev), torch.empty(lib.moe_b200_router_blocks(N), E, device=dev)
    stats, status = torch.empty(N, 2, device=dev), torch.zeros(16, dtype=torch.int32, device=dev)
    check(lib.moe_b200_router_norm(bad.data_ptr(), wn.data_ptr(), c.data_ptr(), float(norm.eps), N, d, E, k, _cabi.BF16,
                                   logits.data_ptr(), idx.data_ptr(), w.data_ptr(), part.data_ptr(), stats.data_ptr(),
                                   status.data_ptr(), s), "router_norm")
    with torch.no_grad():
        want = m(x.view(1, N, d), norm=norm)[0][0]
        got = m(bad.view(1, N, d), norm=norm)[0][0]
    assert torch.equal(m.last["idx"][rows], idx[rows])
    new = m.last["logits"][rows]
    assert torch.equal(new.isnan(), logits[rows].isnan()) and torch.equal(new.isposinf(), logits[rows].isposinf())
    assert m.device_status() == (2 if (idx >= E).any() else 0)
    routed = (idx[rows] < E).any(1)
    assert got[rows[routed]].isnan().all() and (value != value or routed.any())
    others = torch.ones(N, dtype=torch.bool, device=dev)
    others[rows] = False
    assert torch.equal(got[others], want[others])


# a whole bf16 call of 33 to 64 experts: one token, a block of one and of all 16, streaming and sorted-row sizes, one slot and eight
@pytest.mark.parametrize("N,d,E,k", [(1, 64, 33, 1), (16, 2056, 64, 4), (33, 72, 63, 8), (130, 1024, 40, 2), (511, 520, 64, 8),
                                     (2048, 64, 64, 2)])
def test_routing_of_many_experts(cuda_device, N, d, E, k):
    """As the general router and dispatch give it; a token of NaN is routed to experts and its output is NaN."""
    x = torch.randn(N, d, generator=torch.Generator().manual_seed(E + N)).bfloat16().to(cuda_device)
    params = synthetic.make_params(d, E, 64, seed=N)
    m = build(params, d, E, 64, k, torch.bfloat16, cuda_device)
    gate = (m.gate.weight.detach(), m.gate.bias.detach())
    with torch.no_grad():
        out = m(x.view(1, N, d))[0]
    last = {n: t.clone() for n, t in m.last.items()}
    assert m.device_status() == 0 and bool(out.isfinite().all())
    logits, idx, w, psum_part = helpers.router(x, *gate, k)
    # fp32 sums of d products in another order: d 2^-24 of their sum of magnitudes, at the worst
    mag = x.float().abs() @ gate[0].float().abs().T + gate[1].float().abs()
    assert bool(((last["logits"] - logits).abs() <= 2 * d * 2.0 ** -24 * mag).all())
    r = moe_oracle.route_from_logits(last["logits"].cpu(), k)
    ok = ~moe_oracle.tie_rows(r["probs"], k)
    assert torch.equal(last["idx"].cpu()[ok].long(), r["idx"][ok])
    assert torch.allclose(last["w"].cpu()[ok], r["w"][ok], atol=2e-6, rtol=0)
    disp = helpers.dispatch(x, last["idx"], E, psum_part)
    for name in ("offsets", "row_of", "cnt_slot"):
        assert torch.equal(last[name], disp[name]), name
    bad = x.clone()
    bad[N // 2, 3] = float("nan")
    with torch.no_grad():
        got = m(bad.view(1, N, d))[0][0]
    assert m.device_status() == 0 and bool(got[N // 2].isnan().all())
    others = torch.arange(N, device=cuda_device) != N // 2
    assert bool(got[others].isfinite().all())


# fronts whose blocks meet: 8 and 16 tokens a block, up to 32 experts and more, and a block an SM
@pytest.mark.parametrize("N,E,k", [(512, 8, 2), (2048, 8, 2), (1000, 40, 2), (3000, 8, 2), (2500, 40, 2)])
def test_bf16_calls_on_three_streams_and_in_a_graph(cuda_device, N, E, k):
    """Three calls at once, whose fronts together have more blocks than there are SMs; then all from one graph. Words of the
    status region that no kernel of such a call uses may hold anything."""
    d, f = 64, 128
    params = synthetic.make_params(d, E, f, seed=3)
    mods = [build(params, d, E, f, k, torch.bfloat16, cuda_device) for _ in range(3)]
    xs = [torch.randn(1, N, d, generator=torch.Generator().manual_seed(i)).bfloat16().to(cuda_device) for i in range(3)]
    with torch.no_grad():
        want = [m(x)[0] for m, x in zip(mods, xs)]
        for m in mods:      # (where the blocks met before: one left there let the next call's blocks pass at once)
            m._view("status", torch.int32, (_cabi.READY_OFFSET + _cabi.READY_INTS,))[-4] = 7
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in range(3)]
        got = [[], [], []]
        for _ in range(50):
            for i, st in enumerate(streams):
                with torch.cuda.stream(st):
                    got[i].append(mods[i](xs[i])[0])
        torch.cuda.synchronize()
        for i in range(3):
            assert mods[i].device_status() == 0
            assert all(torch.equal(o, want[i]) for o in got[i])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = [m(x)[0] for m, x in zip(mods, xs)]
        for _ in range(3):
            for o in captured:
                o.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(o, w) for o, w in zip(captured, want))


@pytest.mark.parametrize("E,k", [(8, 2), (9, 8), (17, 3), (32, 4)])
def test_fp32_logits_that_are_not_finite(cuda_device, E, k):
    """Routing in one launch as the general kernel gives it: gate biases of NaN and both infinities, for some experts up
    to all of them."""
    d, f, N = 64, 8, 50
    x = torch.randn(N, d, generator=torch.Generator().manual_seed(E)).to(cuda_device)
    nan, inf = float("nan"), float("inf")
    for i, values in enumerate([(nan,), (inf,), (-inf,), (nan, inf, -inf), (-inf,) * (E - 1), (nan,) * (E - 1),
                                (nan,) * (E - k // 2), (nan,) * E, (inf,) * E, (-inf,) * E, (-nan, nan, -inf) * (E // 3)]):
        params = synthetic.make_params(d, E, f, seed=i)
        at = torch.randperm(E, generator=torch.Generator().manual_seed(i))[:len(values)]
        params["gate_b"][at] = torch.tensor(values)
        m = build(params, d, E, f, k, torch.float32, cuda_device)
        with torch.no_grad():
            m(x.view(1, N, d))
        _, idx, w, _ = helpers.router(x, m.gate.weight.detach(), m.gate.bias.detach(), k)
        last = m.last
        assert torch.equal(last["idx"], idx), values
        assert torch.allclose(last["w"], w, atol=2e-6, rtol=0, equal_nan=True), values
        disp = helpers.dispatch(x, idx, E)
        for name in ("offsets", "row_of", "cnt_slot"):
            assert torch.equal(last[name], disp[name]), (values, name)
        assert m.device_status() == int(disp["status"][0])


def test_fp32_calls_on_two_streams_and_in_a_graph(cuda_device):
    """Two calls at once, each with a grid whose blocks wait on one another and nearly as many blocks as there are SMs; then
    both from one graph."""
    N, d, E, f, k = 2048, 64, 8, 128, 2
    params = synthetic.make_params(d, E, f, seed=3)
    mods = [build(params, d, E, f, k, torch.float32, cuda_device) for _ in range(2)]
    xs = [torch.randn(1, N, d, generator=torch.Generator().manual_seed(i)).to(cuda_device) for i in range(2)]
    with torch.no_grad():
        want = [m(x)[0] for m, x in zip(mods, xs)]
        torch.cuda.synchronize()
        streams = [torch.cuda.Stream() for _ in range(2)]
        got = [[], []]
        for _ in range(50):
            for i, st in enumerate(streams):
                with torch.cuda.stream(st):
                    got[i].append(mods[i](xs[i])[0])
        torch.cuda.synchronize()
        for i in range(2):
            assert mods[i].device_status() == 0
            assert all(torch.equal(o, want[i]) for o in got[i])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            captured = [m(x)[0] for m, x in zip(mods, xs)]
        for _ in range(3):
            for o in captured:
                o.zero_()
            graph.replay()
            torch.cuda.synchronize()
            assert all(torch.equal(o, w) for o, w in zip(captured, want))


SMALL = [
    # N, d, E, f, k
    (1, 64, 8, 128, 2), (2, 64, 8, 128, 2), (3, 64, 8, 128, 2), (127, 64, 8, 128, 2),
    (128, 64, 8, 128, 2), (129, 64, 8, 128, 2), (1000, 128, 16, 200, 4), (513, 256, 5, 264, 3),
    (2048, 64, 8, 128, 2), (2049, 64, 8, 128, 2),
]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,d,E,f,k", SMALL)
def test_small_shapes(cuda_device, N, d, E, f, k, dtype):
    """bf16 with N*k <= 256 takes the small-N weight-streaming kernels, up to 4096 rows the
    streaming kernel on sorted rows, beyond that the prefill kernels: the sizes straddle
    every switch."""
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N), dtype)
    params["w1"] *= 2.0
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 1), dtype)
    m = build(params, d, E, f, k, dtype, cuda_device)
    check_against_oracle(m, params, x, k, dtype, cuda_device)
    res = synthetic.round_to(synthetic.make_input(N, d, seed=N + 2), dtype)
    check_against_oracle(m, params, x, k, dtype, cuda_device, residual=res)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_empty_expert_and_one_hot_expert(cuda_device, dtype):
    d, E, f, k, N = 64, 8, 128, 2, 300
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=4), dtype)
    params["gate_b"] = torch.tensor([8.0, 4.0, -60.0, -60.0, -60.0, -60.0, -60.0, -60.0])
    x = synthetic.round_to(synthetic.make_input(N, d, seed=5), dtype)
    m = build(params, d, E, f, k, dtype, cuda_device)
    last, _ = check_against_oracle(m, params, x, k, dtype, cuda_device)
    assert last["cnt_slot"][0].tolist() == [N, 0, 0, 0, 0, 0, 0, 0]
    assert last["cnt_slot"][1].tolist() == [0, N, 0, 0, 0, 0, 0, 0]


# calls of 192 and more rows an expert, up to 4096 in all: widths that are no multiple of a tile, an uneven routing, and 64
# tiles of the down product in one round
@pytest.mark.parametrize("N,d,bias0", [(767, 264, 0.0), (768, 264, 0.0), (1000, 72, 2.0), (2048, 1024, 0.0)])
def test_between_streaming_and_prefill(cuda_device, N, d, bias0):
    E, f, k = 8, 136, 2
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N), torch.bfloat16)
    params["w1"] *= 2.0
    params["gate_b"][0] = bias0
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 1), torch.bfloat16)
    res = synthetic.round_to(synthetic.make_input(N, d, seed=N + 2), torch.bfloat16)
    m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
    for _ in range(2):
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device, residual=res)


# one to three experts: 1536 rows, where one or two leave the streaming kernel, and below
@pytest.mark.parametrize("N,E,k", [(1535, 1, 1), (1536, 1, 1), (767, 3, 2), (768, 3, 2), (300, 2, 1)])
def test_between_streaming_and_prefill_with_few_experts(cuda_device, N, E, k):
    d, f = 136, 264
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N), torch.bfloat16)
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 1), torch.bfloat16)
    res = synthetic.round_to(synthetic.make_input(N, d, seed=N + 2), torch.bfloat16)
    m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
    for _ in range(2):
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device, residual=res)


def test_c0_full_size_fp32(cuda_device):
    wl = synthetic.WORKLOADS["c0"]
    pins = json.loads((GOLDEN / "routing_pins.json").read_text())["c0"]
    params = synthetic.make_params(wl.d_model, wl.n_experts, wl.d_ff, seed=0)
    x = synthetic.make_input(wl.tokens, wl.d_model, seed=1)
    m = build(params, wl.d_model, wl.n_experts, wl.d_ff, wl.top_k, torch.float32, cuda_device)
    last, o = check_against_oracle(m, params, x, wl.top_k, torch.float32, cuda_device)
    # routing equals the reference's routing on its own logits at this seed
    assert sha(last["idx"]) == pins["idx_sha256"]
    assert sha(last["cnt_slot"]) == pins["cnt_slot_sha256"]
    assert abs(float(o["aux"]) - pins["aux"]) < 1e-5


@pytest.mark.parametrize("name", ["c1_uniform", "c1_skew"])
def test_c1_full_size_bf16(cuda_device, name):
    wl = synthetic.WORKLOADS[name]
    pins = json.loads((GOLDEN / "routing_pins.json").read_text())[name]
    params = helpers.rounded_params(
        synthetic.make_params(wl.d_model, wl.n_experts, wl.d_ff, seed=0, gate_bias_kind=wl.gate_bias),
        torch.bfloat16)
    x = synthetic.round_to(synthetic.make_input(wl.tokens, wl.d_model, seed=1), torch.bfloat16)
    m = build(params, wl.d_model, wl.n_experts, wl.d_ff, wl.top_k, torch.bfloat16, cuda_device)
    last, _ = check_against_oracle(m, params, x, wl.top_k, torch.bfloat16, cuda_device)
    assert sha(last["idx"]) == pins["idx_sha256"]
    assert sha(last["cnt_slot"]) == pins["cnt_slot_sha256"]
    if name == "c1_skew":
        share = float(last["cnt_slot"][:, 0].sum()) / (wl.tokens * wl.top_k)
        assert abs(share - pins["expert0_share"]) < 1e-9


@pytest.mark.parametrize("name", ["c2_t1", "c2_t8", "c2_t32", "c2_t64"])
def test_c2_decode_shapes_bf16(cuda_device, name):
    wl = synthetic.WORKLOADS[name]
    params = helpers.rounded_params(
        synthetic.make_params(wl.d_model, wl.n_experts, wl.d_ff, seed=0), torch.bfloat16)
    x = synthetic.round_to(synthetic.make_input(wl.tokens, wl.d_model, seed=1), torch.bfloat16)
    m = build(params, wl.d_model, wl.n_experts, wl.d_ff, wl.top_k, torch.bfloat16, cuda_device)
    res = synthetic.round_to(synthetic.make_input(wl.tokens, wl.d_model, seed=7), torch.bfloat16)
    check_against_oracle(m, params, x, wl.top_k, torch.bfloat16, cuda_device)
    check_against_oracle(m, params, x, wl.top_k, torch.bfloat16, cuda_device, residual=res)


@pytest.mark.parametrize("d,E,f,k", [(1024, 8, 4096, 2), (256, 16, 200, 4), (2048, 8, 1408, 2),
                                     (128, 5, 264, 3), (64, 32, 136, 8), (72, 8, 24, 1)])
def test_one_to_eight_tokens_single_launch(cuda_device, d, E, f, k):
    """bf16 calls of one to eight tokens with fewer rows than experts run routing, both products and
    the weighted sum in one cooperative launch: every token count, shapes whose output columns
    per block need one and two column groups, feature counts that are no multiple of 16, all
    tokens equal (every row on the same k experts), with and without a residual, call after call."""
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=d + f), torch.bfloat16)
    m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
    for N in range(1, 9):
        x = synthetic.round_to(synthetic.make_input(N, d, seed=31 * N + k), torch.bfloat16)
        res = synthetic.round_to(synthetic.make_input(N, d, seed=31 * N + 7), torch.bfloat16)
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device)
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device, residual=res)
        same = x[:1].repeat(N, 1).contiguous()
        check_against_oracle(m, params, same, k, torch.bfloat16, cuda_device, residual=res)


@pytest.mark.parametrize("N,d,E,f,k", [(129, 64, 8, 128, 2), (300, 256, 8, 1024, 2), (512, 512, 8, 2048, 2),
                                       (400, 1024, 8, 4096, 2), (250, 128, 16, 200, 4), (1500, 256, 8, 1024, 2),
                                       (2048, 128, 8, 256, 2)])
def test_mid_sizes_rows_path(cuda_device, N, d, E, f, k):
    """Between the decode and the prefill sizes (257 to 4096 rows) the forward streams the
    weights over the sorted rows: the block's tolerance, with and without a residual, call
    after call."""
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N), torch.bfloat16)
    res = synthetic.round_to(synthetic.make_input(N, d, seed=N + 2), torch.bfloat16)
    m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
    for call in range(2):
        x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 10 + call), torch.bfloat16)
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device)
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device, residual=res)


# both products in one launch: either side of its lines (96 and 2048 rows an expert, 1536 and 4096 rows of one or two
# experts, 33 experts); blocks of 256 tokens and a token more, remainders of 32; more blocks than take turns on a tile of
# weights (16); experts without rows; widths that are no multiple of a tile; K of one block; one token; 200 experts
@pytest.mark.parametrize("N,d,E,f,k,bias0", [
    (383, 264, 8, 136, 2, 0.0), (384, 264, 8, 136, 2, 0.0), (512, 64, 2, 264, 1, 9.0), (1537, 136, 2, 264, 1, 0.7),
    (256 * 5 + 1, 72, 4, 200, 1, 40.0), (4400, 128, 8, 72, 1, 40.0), (8193, 64, 4, 64, 1, 0.0), (1, 256, 33, 136, 4, 0.0),
    (40, 136, 64, 264, 4, 3.0), (700, 64, 200, 72, 8, 0.0), (1100, 1024, 8, 1032, 2, 0.0),
    (143, 136, 3, 264, 2, 0.0), (144, 136, 3, 264, 2, 0.0), (8192, 64, 4, 64, 1, 0.0), (4096, 136, 2, 264, 1, 0.0),
    (4097, 136, 2, 264, 1, 0.0), (384, 256, 8, 4096, 2, 0.0), (2049, 136, 8, 1032, 2, 0.0)])
def test_both_products_in_one_launch(cuda_device, N, d, E, f, k, bias0):
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N), torch.bfloat16)
    params["w1"] *= 2.0
    params["gate_b"][0] = bias0
    m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
    for call in range(2):
        x = synthetic.round_to(synthetic.make_input(N, d, seed=N + call), torch.bfloat16)
        res = synthetic.round_to(synthetic.make_input(N, d, seed=N + 7), torch.bfloat16) if call else None
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device, residual=res)


def test_calls_of_every_size_share_their_counters(cuda_device):
    """The kernels of small calls and the one that takes both products count in the same words of a workspace, and each finds
    them zero: sizes in turn on one module, up to one whose call clears them itself."""
    d, E, f, k = 128, 8, 264, 2
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=3), torch.bfloat16)
    m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
    for N in (2300, 64, 512, 1, 300, 512, 40, 2300, 512, 512, 3, 2047, 64):
        x = synthetic.round_to(synthetic.make_input(N, d, seed=N), torch.bfloat16)
        check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device)


def test_calls_in_one_launch_on_two_streams(cuda_device):
    """Two such calls at once: tiles are claimed by pairs of CTAs that run, so that neither waits for one that does not.
    The outputs are those of the calls one after the other, to the bit."""
    N, d, E, f, k = 1200, 512, 8, 1024, 2
    ms = []
    for seed in (1, 2):
        params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=seed), torch.bfloat16)
        x = synthetic.round_to(synthetic.make_input(N, d, seed=seed + 5), torch.bfloat16).bfloat16().to(cuda_device)
        ms.append((build(params, d, E, f, k, torch.bfloat16, cuda_device), x.view(1, N, d), torch.cuda.Stream()))
    with torch.no_grad():
        want = [m(x)[0].clone() for m, x, _ in ms]
        torch.cuda.synchronize()
        for _ in range(20):
            got = []
            for m, x, s in ms:
                with torch.cuda.stream(s):
                    got.append(m(x)[0])
            torch.cuda.synchronize()
            assert all(torch.equal(g, w) for g, w in zip(got, want))
    assert all(m.device_status() == 0 for m, _, _ in ms)


def test_small_n_fresh_workspace_and_changing_inputs(cuda_device):
    """The small-N expert kernel runs while the routing kernel is still writing idx/offsets, and
    the combine may become resident before either has finished: every call on a fresh, zeroed
    workspace, and every call whose routing differs from the call before, must still come out
    right (a read of the routing that is served too early shows up here as a time-out or as
    the previous call's routing)."""
    N, d, E, f, k = 128, 64, 8, 128, 2
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=0), torch.bfloat16)
    for trial in range(12):
        m = build(params, d, E, f, k, torch.bfloat16, cuda_device)
        for call in range(3):
            x = synthetic.round_to(synthetic.make_input(N, d, seed=100 * trial + call), torch.bfloat16)
            check_against_oracle(m, params, x, k, torch.bfloat16, cuda_device)


@pytest.mark.parametrize("N", [4, 64])
def test_small_n_layers_back_to_back(cuda_device, N):
    """Several blocks launched back to back with no host synchronisation, each one's output the
    next one's input: the first kernel of a block becomes resident while the last kernel of the
    block before it is still running, and has to wait for it before it reads x."""
    d, E, f, k, L = 256, 8, 512, 2, 5
    layers, params = [], []
    for l in range(L):
        p = helpers.rounded_params(synthetic.make_params(d, E, f, seed=10 + l), torch.bfloat16)
        params.append(p)
        layers.append(build(p, d, E, f, k, torch.bfloat16, cuda_device))
    x0 = synthetic.round_to(synthetic.make_input(N, d, seed=3), torch.bfloat16)
    for rep in range(3):      # the first pass also creates plans and workspaces
        xs = [(x0 * (1.0 + 0.25 * rep)).to(torch.bfloat16).to(cuda_device).view(1, N, d)]
        with torch.no_grad():
            for m in layers:
                out, _aux = m(xs[-1], residual=xs[-1])
                xs.append(out)
        torch.cuda.synchronize()
        for l, m in enumerate(layers):
            assert m.device_status() == 0
            xin = xs[l].view(N, d).float().cpu()
            with torch.no_grad():
                o = moe_oracle.moe_forward(xin, params[l], k, logits=m.last["logits"].cpu())
            ok = ~moe_oracle.tie_rows(o["probs"], k)
            assert torch.equal(m.last["idx"].cpu()[ok].long(), o["idx"][ok])
            ref = o["out"] + xin
            got = xs[l + 1].view(N, d).float().cpu()
            assert (got - ref)[ok].abs().max() <= 2e-2 * ref.abs().max()


def test_c4_router_pin(cuda_device):
    wl = synthetic.WORKLOADS["c4"]
    pins = json.loads((GOLDEN / "routing_pins.json").read_text())["c4"]
    g = torch.Generator().manual_seed(0)
    gate_w = (torch.randn(wl.n_experts, wl.d_model, generator=g) * 0.02).to(torch.bfloat16)
    gate_b = synthetic.gate_bias(wl.gate_bias, wl.n_experts).to(torch.bfloat16)
    x = synthetic.make_input(wl.tokens, wl.d_model, seed=1).to(torch.bfloat16)
    _, idx, _, _ = helpers.router(x.to(cuda_device), gate_w.to(cuda_device), gate_b.to(cuda_device),
                                  wl.top_k)
    torch.cuda.synchronize()
    assert sha(idx.cpu()) == pins["idx_sha256"]


def test_c4_shape_bf16(cuda_device):
    """The expert-parallel workload's block on one GPU at its full size: d 2048, f 1408 (eleven
    128-feature GEGLU tiles, not a multiple of 256), 64 experts, top-4, Zipf(1.1) router bias
    (tail experts of a few dozen rows next to one of tens of thousands), 65536 tokens. Routing
    and counts are compared on every token; outputs on a 4096-token slice (tokens are
    independent, model.py:201) under the kernel's own logits."""
    wl = synthetic.WORKLOADS["c4"]
    pins = json.loads((GOLDEN / "routing_pins.json").read_text())["c4"]
    N, d, f, E, k = wl.tokens, wl.d_model, wl.d_ff, wl.n_experts, wl.top_k
    dt = torch.bfloat16
    m = MOE(d, num_experts=E, d_ff=f, top_k=k, device="cuda").eval().to(device=cuda_device, dtype=dt)
    gate_w, gate_b = synthetic.make_gate(d, E, 0, wl.gate_bias)
    w1, w2 = [], []
    with torch.no_grad():
        m.gate.weight.copy_(gate_w)
        m.gate.bias.copy_(gate_b)
        for e, ex in enumerate(m.experts):
            pe = synthetic.make_expert(d, f, e, 0)
            ex.gate_and_up.weight.copy_(pe["w1"]); ex.gate_and_up.bias.zero_()
            ex.down.weight.copy_(pe["w2"]); ex.down.bias.zero_()
            w1.append(synthetic.round_to(pe["w1"], dt))
            w2.append(synthetic.round_to(pe["w2"], dt))
    params = {"gate_w": synthetic.round_to(gate_w, dt), "gate_b": synthetic.round_to(gate_b, dt),
              "w1": w1, "b1": torch.zeros(E, 2 * f), "w2": w2, "b2": torch.zeros(E, d)}
    x = synthetic.round_to(synthetic.make_input(N, d, seed=1), dt)
    with torch.no_grad():
        out, aux = m(x.to(dt).to(cuda_device).view(N // 64, 64, d))
    torch.cuda.synchronize()
    assert m.device_status() == 0
    last = {n: t.cpu() for n, t in m.last.items()}
    # routing on all tokens: bit-exact against topk(softmax(logits)) on the kernel's logits,
    # and equal to the pinned routing of the oracle on its own logits
    r = moe_oracle.route_from_logits(last["logits"], k)
    good = ~moe_oracle.tie_rows(r["probs"], k)
    assert torch.equal(last["idx"][good].long(), r["idx"][good])
    if good.all():
        assert torch.equal(last["cnt_slot"].long(), r["cnt_slot"])
    assert int(last["offsets"][-1]) == N * k
    assert sha(last["idx"]) == pins["idx_sha256"]
    assert abs(float(aux) - float(r["aux"])) <= 1e-5 * abs(float(r["aux"])) + 1e-7
    # outputs on a slice that holds rows of the hot experts and of the tail
    sl = slice(30000, 30000 + 4096)
    with torch.no_grad():
        o = moe_oracle.moe_forward(x[sl], params, k, logits=last["logits"][sl])
    ok = ~moe_oracle.tie_rows(o["probs"], k)
    got = out.view(N, d)[sl].float().cpu()
    err = (got - o["out"])[ok].abs().max()
    assert err <= 2e-2 * o["out"].abs().max(), f"max-abs {err} vs scale {o['out'].abs().max()}"
    assert (got - o["out"])[ok].norm() <= 2e-2 * o["out"][ok].norm()
    assert len(set(o["idx"].flatten().tolist())) >= 48      # the slice reaches the tail experts


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,d,E,f,k", [(5000, 256, 8, 512, 2), (3000, 1024, 64, 264, 4), (100, 128, 8, 256, 2),
                                       (1, 64, 8, 128, 2), (1500, 512, 16, 384, 2)])
def test_layernorm_folded_into_the_block(cuda_device, N, d, E, f, k, dtype):
    """The caller's norm2 (model.py:298,311-312) inside the block: the router forms the row
    statistics and the logits of the normalised row, the dispatch normalises while it copies
    (calls of up to 4096 rows normalise their few rows in a kernel of their own). Reference:
    F.layer_norm in fp32 on the same values, then the oracle; the residual is the tensor
    before the norm (model.py:310,319). Input rows get a mean far from zero and a per-row
    scale, as a residual stream has."""
    import torch.nn.functional as F
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N + 3), dtype)
    params["w1"] *= 2.0
    g = torch.Generator().manual_seed(N + d)
    x = synthetic.make_input(N, d, seed=N + 4) * (0.5 + 2.0 * torch.rand(N, 1, generator=g)) \
        + 3.0 * torch.randn(N, 1, generator=g)
    x = synthetic.round_to(x, dtype)
    gamma = synthetic.round_to(1.0 + 0.2 * torch.randn(d, generator=g), dtype)
    beta = synthetic.round_to(0.1 * torch.randn(d, generator=g), dtype)
    m = build(params, d, E, f, k, dtype, cuda_device)
    norm = torch.nn.LayerNorm(d, eps=1e-5).to(device=cuda_device, dtype=dtype)
    with torch.no_grad():
        norm.weight.copy_(gamma)
        norm.bias.copy_(beta)
        xin = x.to(dtype).to(cuda_device).view(1, N, d)
        out, aux = m(xin, residual=xin, norm=norm)
        out2, _ = m(xin, residual=xin, norm=norm)
    torch.cuda.synchronize()
    assert m.device_status() == 0
    assert torch.equal(out, out2)
    xn = F.layer_norm(x, (d,), gamma, beta, 1e-5)
    last = {n: t.cpu() for n, t in m.last.items()}
    # the kernel's logits against the logits of the fp32-normalised rows
    ref_logits = F.linear(xn, params["gate_w"], params["gate_b"])
    tol = 1e-4 if dtype == torch.float32 else 3e-2
    assert (last["logits"] - ref_logits).abs().max() <= tol * max(1.0, float(ref_logits.abs().max()))
    with torch.no_grad():
        o = moe_oracle.moe_forward(xn, params, k, logits=last["logits"])
    ok = ~moe_oracle.tie_rows(o["probs"], k)
    assert torch.equal(last["idx"][ok].long(), o["idx"][ok])
    ref = o["out"] + x
    got = out.view(N, d).float().cpu()
    err = (got - ref)[ok].abs().max()
    if dtype == torch.float32:
        assert err <= 1e-4 * max(1.0, float(ref.abs().max())), f"max-abs {err}"
    else:
        assert err <= 2e-2 * ref.abs().max(), f"max-abs {err} vs scale {ref.abs().max()}"
        assert (got - ref)[ok].norm() <= 2e-2 * ref[ok].norm()


# routed in one launch: a block of one group of tokens and of one more, the most tokens, rows of several rounds
@pytest.mark.parametrize("N,d,E,f,k", [(2305, 264, 16, 64, 8), (2500, 2056, 3, 64, 2), (18944, 72, 8, 64, 1)])
def test_layernorm_folded_into_thousands_of_tokens(cuda_device, N, d, E, f, k):
    test_layernorm_folded_into_the_block(cuda_device, N, d, E, f, k, torch.bfloat16)


def test_state_survives_dtype_change_and_repeat_calls(cuda_device):
    d, E, f, k, N = 64, 8, 128, 2, 200
    params = synthetic.make_params(d, E, f, seed=9)
    m = build(params, d, E, f, k, torch.float32, cuda_device)
    x = synthetic.make_input(N, d, seed=10).to(cuda_device).view(1, N, d)
    with torch.no_grad():
        a, _ = m(x)
        b, _ = m(x)
        assert torch.equal(a, b)                      # deterministic
        m.to(torch.bfloat16)                          # parameter storage moves: plan is rebuilt
        c, _ = m(x.to(torch.bfloat16))
    assert c.dtype == torch.bfloat16
    assert (c.float() - a).abs().max() < 0.05 * a.abs().max() + 1e-3


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_fine_tuning_lora_branch(cuda_device, dtype):
    """fine_tuning=True (model.py:175-179,185-189): LoRA folded into merged weights."""
    from test_oracle import lora_dicts
    d, E, f, k, N = 128, 8, 256, 2, 600
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=40), dtype)
    x = synthetic.round_to(synthetic.make_input(N, d, seed=41), dtype)
    torch.manual_seed(42)
    m = build(params, d, E, f, k, dtype, cuda_device)
    with torch.no_grad():
        for ex in m.experts:          # LoRA tensors of a size that matters
            for lin in (ex.lora_gate_and_up_a, ex.lora_gate_and_up_b, ex.lora_down_a, ex.lora_down_b):
                lin.weight.normal_(0, 0.05)
                lin.bias.normal_(0, 0.05)
        out, aux = m(x.to(dtype).to(cuda_device).view(1, N, d), fine_tuning=True)
        plain, _ = m(x.to(dtype).to(cuda_device).view(1, N, d))
    torch.cuda.synchronize()
    logits = m.last["logits"].cpu()
    with torch.no_grad():
        o = moe_oracle.moe_forward(x, params, k, logits=logits, lora=lora_dicts(m))
    ok = ~moe_oracle.tie_rows(o["probs"], k)
    err = (out.view(N, d).float().cpu() - o["out"])[ok].abs().max()
    if dtype == torch.float32:
        assert err <= 1e-4
    else:
        assert err <= 2e-2 * o["out"].abs().max()
    assert (out.float() - plain.float()).abs().max() > 10 * err   # not the plain forward


def test_empty_batch(cuda_device):
    m = build(synthetic.make_params(64, 8, 128, seed=1), 64, 8, 128, 2, torch.bfloat16, cuda_device)
    with torch.no_grad():
        out, aux = m(torch.zeros(0, 4, 64, dtype=torch.bfloat16, device=cuda_device))
    torch.cuda.synchronize()
    assert out.shape == (0, 4, 64)
    assert m.last["offsets"].cpu().tolist() == [0] * 9


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows", [1, 200, 1000])
def test_feedforward_alone(cuda_device, dtype, rows):
    """The expert module on its own (the reference's dense FeedForward, model.py:154-190)
    runs through the grouped kernels with a single group."""
    from gemmallm_b200 import FeedForward
    d, f = 128, 384
    p = helpers.rounded_params(synthetic.make_params(d, 1, f, seed=rows), dtype)
    g = torch.Generator().manual_seed(rows + 1)
    p["b1"] = synthetic.round_to(torch.randn(1, 2 * f, generator=g) * 0.05, dtype)
    p["b2"] = synthetic.round_to(torch.randn(1, d, generator=g) * 0.05, dtype)
    ff = FeedForward(d, d_ff=f).eval().to(device=cuda_device, dtype=dtype)
    with torch.no_grad():
        ff.gate_and_up.weight.copy_(p["w1"][0]); ff.gate_and_up.bias.copy_(p["b1"][0])
        ff.down.weight.copy_(p["w2"][0]); ff.down.bias.copy_(p["b2"][0])
        x = synthetic.round_to(synthetic.make_input(rows, d, seed=rows + 2), dtype)
        y = ff(x.to(dtype).to(cuda_device).view(1, rows, d))
        y2 = ff(x.to(dtype).to(cuda_device).view(1, rows, d))
        ref = moe_oracle.expert_ffn(x, p["w1"][0], p["b1"][0], p["w2"][0], p["b2"][0])
    torch.cuda.synchronize()
    assert torch.equal(y, y2)
    err = (y.view(rows, d).float().cpu() - ref).abs().max()
    assert err <= (1e-4 if dtype == torch.float32 else 2e-2 * ref.abs().max())


def test_two_devices_in_one_process():
    """One process driving two GPUs: kernel attributes, occupancy results and SM counts are
    cached per device, so the second device gets its own (a per-process cache would leave its
    kernels without their shared-memory limit)."""
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    for dtype, N in ((torch.bfloat16, 6000), (torch.bfloat16, 40), (torch.bfloat16, 700), (torch.float32, 300)):
        d, E, f, k = 256, 8, 512, 2
        params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N), dtype)
        x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 1), dtype)
        for index in (0, 1, 0):
            dev = torch.device("cuda", index)
            m = build(params, d, E, f, k, dtype, dev)
            check_against_oracle(m, params, x, k, dtype, dev)
