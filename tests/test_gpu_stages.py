"""Parity of each C-ABI stage with the CPU oracle on the same seeded inputs:
routing indices and counts bit-exact, floating point within stated tolerances."""
import pytest
import torch
import torch.nn.functional as F

import helpers
from gemmallm_b200 import _cabi, synthetic
from oracle import moe_oracle
from gemmallm_b200._cabi import lib, check  # noqa: E402

pytestmark = pytest.mark.gpu

ROUTER_CASES = [
    # N, d, E, k, dtype
    (1, 64, 8, 2, torch.float32), (2, 64, 8, 2, torch.float32), (3, 64, 8, 2, torch.float32),
    (31, 64, 8, 2, torch.float32), (32, 64, 8, 2, torch.float32), (33, 64, 8, 2, torch.float32),
    (127, 64, 8, 2, torch.bfloat16), (128, 64, 8, 2, torch.bfloat16), (129, 64, 8, 2, torch.bfloat16),
    (512, 512, 8, 2, torch.float32), (1000, 256, 64, 4, torch.bfloat16),
    (300, 128, 256, 8, torch.bfloat16), (77, 72, 5, 3, torch.float32), (50, 40, 1, 1, torch.float32),
    (4096, 2048, 64, 4, torch.bfloat16), (20000, 264, 32, 4, torch.bfloat16), (9000, 1024, 24, 2, torch.bfloat16),
    (5, 72, 40, 3, torch.bfloat16), (129, 64, 17, 1, torch.bfloat16), (40000, 512, 64, 8, torch.bfloat16),
]


def make_gate(N, d, E, dtype, seed):
    g = torch.Generator().manual_seed(seed)
    gate_w = synthetic.round_to(torch.randn(E, d, generator=g) * 0.05, dtype)
    gate_b = synthetic.round_to(torch.randn(E, generator=g) * 0.3, dtype)
    x = synthetic.round_to(torch.randn(N, d, generator=g), dtype)
    return x, gate_w, gate_b


@pytest.mark.parametrize("N,d,E,k,dtype", ROUTER_CASES)
def test_router_matches_oracle(cuda_device, N, d, E, k, dtype):
    x, gw, gb = make_gate(N, d, E, dtype, seed=N + d + E)
    logits, idx, w, psum_part = helpers.router(x.to(dtype).to(cuda_device), gw.to(dtype).to(cuda_device),
                                               gb.to(dtype).to(cuda_device), k)
    torch.cuda.synchronize()
    logits, idx, w, psum_part = logits.cpu(), idx.cpu(), w.cpu(), psum_part.cpu()
    ref_logits = F.linear(x, gw, gb)
    assert (logits - ref_logits).abs().max() <= 2e-5 * max(1.0, float(ref_logits.abs().max()))
    # bit-exact routing given the kernel's own fp32 logits
    r = moe_oracle.route_from_logits(logits, k)
    ties = moe_oracle.tie_rows(r["probs"], k)
    ok = ~ties
    assert torch.equal(idx[ok].long(), r["idx"][ok]), "routing indices differ from topk(softmax(logits))"
    assert torch.allclose(w[ok], r["w"][ok], atol=2e-6, rtol=0)
    assert torch.allclose(psum_part.sum(0), r["probs"].sum(0), rtol=1e-5, atol=1e-5)
    assert ((idx >= 0) & (idx < E)).all()
    # no expert twice for one token
    assert (idx.sort(dim=1).values.diff(dim=1) > 0).all() if k > 1 else True


@pytest.mark.parametrize("N,d,E,k", [(1, 1024, 8, 2), (8, 1024, 8, 2), (17, 256, 16, 4), (64, 1024, 8, 2),
                                     (100, 72, 5, 2), (128, 128, 32, 2), (33, 64, 24, 7),
                                     (129, 256, 8, 2), (300, 1024, 8, 2), (512, 512, 32, 2), (200, 128, 16, 5),
                                     (1000, 256, 8, 2), (2048, 128, 16, 4)])
@pytest.mark.parametrize("split", [False, True])
def test_front_small_equals_router_plus_dispatch(cuda_device, N, d, E, k, split):
    """The single-launch front end gives what the two general kernels give, whether every block
    repeats the routing or (beyond 128 tokens) the blocks share it and meet at a counter."""
    if N > 512 and not split:
        pytest.skip("every block repeating the routing is limited to 512 tokens")
    dt = torch.bfloat16
    x, gw, gb = make_gate(N, d, E, dt, seed=N + E)
    xd, gwd, gbd = x.to(dt).to(cuda_device), gw.to(dt).to(cuda_device), gb.to(dt).to(cuda_device)
    logits, idx, w, psum_part = helpers.router(xd, gwd, gbd, k)
    ref = helpers.dispatch(xd, idx, E, psum_part)
    dev = cuda_device
    got = {"logits": torch.empty(N, E, dtype=torch.float32, device=dev),
           "idx": torch.empty(N, k, dtype=torch.int32, device=dev),
           "w": torch.empty(N, k, dtype=torch.float32, device=dev),
           "cnt_slot": torch.empty(k, E, dtype=torch.int32, device=dev),
           "offsets": torch.empty(E + 1, dtype=torch.int32, device=dev),
           "row_of": torch.empty(N, k, dtype=torch.int32, device=dev),
           "perm": torch.empty(N * k, d, dtype=dt, device=dev),
           "psum": torch.empty(E, dtype=torch.float32, device=dev),
           "aux": torch.zeros(1, dtype=torch.float32, device=dev)}
    outs = [got[n].data_ptr() for n in ("logits", "idx", "w", "cnt_slot", "offsets", "row_of", "perm",
                                        "psum", "aux")]
    if split:
        xch = torch.full((helpers.lib.moe_b200_front_exchange_ints(N, E, k),), 0x5A5A5A5A,
                         dtype=torch.int32, device=dev)
        counter = torch.full((1,), 77, dtype=torch.int32, device=dev)    # the call zeroes it
        status = torch.zeros(16, dtype=torch.int32, device=dev)
        for _ in range(2):       # twice: the counter has to be back at zero after a call
            helpers.check(helpers.lib.moe_b200_front_small_split(
                xd.data_ptr(), gwd.data_ptr(), gbd.data_ptr(), N, d, E, k, _cabi.BF16, *outs,
                xch.data_ptr(), counter.data_ptr(), status.data_ptr(), helpers.stream(dev)),
                "front_small_split")
            torch.cuda.synchronize()
            assert status.cpu().tolist()[0] == 0 and int(counter.item()) == 0
    else:
        helpers.check(helpers.lib.moe_b200_front_small(
            xd.data_ptr(), gwd.data_ptr(), gbd.data_ptr(), N, d, E, k, _cabi.BF16, *outs,
            helpers.stream(dev)), "front_small")
    torch.cuda.synchronize()
    assert (got["logits"] - logits).abs().max() <= 2e-5 * max(1.0, float(logits.abs().max()))
    r = moe_oracle.route_from_logits(got["logits"].cpu(), k)
    ok = ~moe_oracle.tie_rows(r["probs"], k)
    assert torch.equal(got["idx"].cpu()[ok].long(), r["idx"][ok])
    assert torch.allclose(got["w"].cpu()[ok], r["w"][ok], atol=2e-6, rtol=0)
    if torch.equal(got["idx"], idx):     # same routing (always, unless a near-tie flips): same layout
        for name in ("cnt_slot", "offsets", "row_of", "perm"):
            assert torch.equal(got[name], ref[name]), name
        assert torch.allclose(got["psum"], ref["psum"], rtol=1e-5, atol=1e-6)
        assert abs(float(got["aux"]) - float(ref["aux"])) <= 1e-5 * abs(float(ref["aux"])) + 1e-7
    else:
        assert torch.equal(got["cnt_slot"].cpu().long(), r["cnt_slot"])


# more than 128 tokens: a last block of one token, rows of fewer and more pieces than a warp has under way, chunks of K for a few
# warps and for several rounds, one expert and as many as there can be, all slots
@pytest.mark.parametrize("N,d,E,k", [(129, 8, 1, 1), (145, 4104, 8, 2), (600, 1032, 9, 8), (1041, 40, 32, 8), (2047, 2048, 17, 1)])
def test_front_of_many_tokens(cuda_device, N, d, E, k):
    test_front_small_equals_router_plus_dispatch(cuda_device, N, d, E, k, True)


DISPATCH_CASES = [(1, 64, 8, 2), (2, 64, 8, 2), (63, 64, 8, 2), (64, 64, 8, 2), (65, 64, 8, 2),
                  (129, 128, 8, 2), (1000, 256, 64, 4), (5000, 512, 8, 2), (333, 72, 5, 3),
                  (4097, 64, 256, 8), (40000, 64, 8, 2)]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,d,E,k", DISPATCH_CASES)
def test_dispatch_is_a_stable_counting_sort(cuda_device, N, d, E, k, dtype):
    g = torch.Generator().manual_seed(N * 7 + E)
    x = torch.randn(N, d, generator=g).to(dtype)
    # k distinct experts per token, skewed popularity
    score = torch.rand(N, E, generator=g) + torch.linspace(0.5, 0, E)
    idx = score.topk(k, dim=1).indices.to(torch.int32)
    psum_part = torch.rand(max(1, _cabi.lib.moe_b200_router_blocks(N)), E, generator=g)
    out = helpers.dispatch(x.to(cuda_device), idx.to(cuda_device), E, psum_part.to(cuda_device))
    torch.cuda.synchronize()
    cnt_slot, offsets, row_of, perm = (out[n].cpu() for n in ("cnt_slot", "offsets", "row_of", "perm"))
    assert int(out["status"][0]) == 0
    ref_cnt = torch.stack([torch.bincount(idx[:, j].long(), minlength=E) for j in range(k)])
    assert torch.equal(cnt_slot.long(), ref_cnt)
    total = ref_cnt.sum(0)
    assert torch.equal(offsets.long(), torch.cat([torch.zeros(1, dtype=torch.long), total.cumsum(0)]))
    flat = row_of.long().flatten()
    assert torch.equal(flat.sort().values, torch.arange(N * k))          # a permutation
    e_of_row = torch.bucketize(flat, offsets.long()[1:], right=True)
    assert torch.equal(e_of_row, idx.long().flatten())                  # rows land in their expert
    assert torch.equal(perm[flat].view(N, k, d), x[:, None, :].expand(N, k, d))  # rows are copies
    # stable: inside one expert, rows follow token order
    tok_of_row = torch.empty(N * k, dtype=torch.long)
    tok_of_row[flat] = torch.arange(N).repeat_interleave(k)
    for e in range(E):
        seg = tok_of_row[offsets[e]:offsets[e + 1]]
        assert (seg.diff() > 0).all()
    # load-balancing loss from the partial sums, fixed-order reduction
    psum = psum_part.sum(0)
    aux = (psum / N * (ref_cnt[0].float() / N)).mean() * float(E * E)
    assert torch.allclose(out["psum"].cpu(), psum, rtol=1e-5)
    assert abs(float(out["aux"][0]) - float(aux)) <= 1e-5 * abs(float(aux)) + 1e-7


# rows of one 16-byte piece, of odd counts of pieces, and on both sides of 8192 pieces
@pytest.mark.parametrize("dtype,d", [(torch.bfloat16, 8), (torch.bfloat16, 24), (torch.float32, 8), (torch.float32, 1016),
                                     (torch.bfloat16, 8 * 8191), (torch.bfloat16, 8 * 8192), (torch.float32, 4 * 8190)])
def test_dispatch_copies_rows_of_any_width(cuda_device, dtype, d):
    N, E, k = (20000, 8, 2) if d < 2000 else (150, 8, 2)     # chunks of more than four tokens where rows are short
    g = torch.Generator().manual_seed(d)
    x = torch.randn(N, d, generator=g).to(dtype).to(cuda_device)
    idx = torch.rand(N, E, generator=g).topk(k, dim=1).indices.to(torch.int32).to(cuda_device)
    out = helpers.dispatch(x, idx, E)
    flat = out["row_of"].long().flatten()
    assert torch.equal(flat.sort().values, torch.arange(N * k, device=cuda_device))
    assert torch.equal(out["perm"][flat].view(N, k, d), x[:, None, :].expand(N, k, d))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("aligned", [True, False])
def test_dispatch_normalises_with_weights_at_any_address(cuda_device, dtype, aligned):
    """The folded LayerNorm with gamma and beta on and off a 16-byte boundary; statistics as given."""
    N, d, E, k = 700, 136, 8, 2
    g = torch.Generator().manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dtype)
    x, gamma, beta = rnd(N, d), rnd(d), rnd(d)
    stats = torch.stack([torch.randn(N, generator=g), torch.rand(N, generator=g) + 0.5], dim=1)
    at = 0 if aligned else 1
    place = lambda t: torch.cat([torch.zeros(at, dtype=dtype), t]).to(cuda_device)[at:]
    gd, bd, xd, sd = place(gamma), place(beta), x.to(cuda_device), stats.to(cuda_device)
    assert (gd.data_ptr() % 16 == 0) == aligned
    idx = torch.rand(N, E, generator=g).topk(k, dim=1).indices.to(torch.int32).to(cuda_device)
    i32 = dict(dtype=torch.int32, device=cuda_device)
    scratch = torch.empty(lib.moe_b200_dispatch_scratch_bytes(N, E, k) // 4, **i32)
    cnt, offsets, row_of = torch.empty(k, E, **i32), torch.empty(E + 1, **i32), torch.empty(N, k, **i32)
    perm, status = torch.empty(N * k, d, dtype=dtype, device=cuda_device), torch.zeros(16, **i32)
    check(lib.moe_b200_dispatch_norm(xd.data_ptr(), idx.data_ptr(), sd.data_ptr(), gd.data_ptr(), bd.data_ptr(), N, d, E, k,
                                     helpers.CODE[dtype], scratch.data_ptr(), cnt.data_ptr(), offsets.data_ptr(),
                                     row_of.data_ptr(), perm.data_ptr(), None, None, None, status.data_ptr(),
                                     helpers.stream(cuda_device)), "dispatch_norm")
    assert status.cpu()[0] == 0
    want = (x.double() - stats[:, :1].double()) * stats[:, 1:].double() * gamma.double() + beta.double()
    got = perm[row_of.long().flatten()].view(N, k, d).cpu().double()
    # three rounded operations, and the rounding of the result
    size = ((x.double() - stats[:, :1].double()) * stats[:, 1:].double() * gamma.double()).abs() + beta.double().abs()
    bound = 2.0 ** -22 * size + (2.0 ** -8 if dtype == torch.bfloat16 else 0.0) * want.abs()
    assert ((got - want[:, None]).abs() <= bound[:, None]).all()


# rows kept in registers (up to 1024, up to 2048 wide) and read again, a lane's last piece missing
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("N,d", [(9, 8), (3, 1024), (17, 1032), (8, 2040), (5, 2048), (3, 2056), (2, 8200)])
def test_layernorm_rows_of_any_width(cuda_device, dtype, N, d):
    g = torch.Generator().manual_seed(d)
    rnd = lambda *s: torch.randn(*s, generator=g).to(dtype)
    x, gamma, beta = rnd(N, d) * 2 + 1, rnd(d), rnd(d)
    dev = [t.to(cuda_device) for t in (x, gamma, beta)]
    out = torch.full_like(dev[0], float("nan"))
    check(lib.moe_b200_layernorm(*[t.data_ptr() for t in dev], 1e-5, N, d, helpers.CODE[dtype], out.data_ptr(),
                                 helpers.stream(cuda_device)), "layernorm")
    want = F.layer_norm(x.double(), (d,), gamma.double(), beta.double(), 1e-5)
    # sums of d / 32 terms a lane and five of the lanes' in fp32, against a deviation of 2: 2^-24 (d / 32 + 5) of the values
    eps = (2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    bound = eps * want.abs() + 2.0 ** -24 * (d / 32 + 16) * (want.abs() + gamma.double().abs() + 1)
    assert ((out.cpu().double() - want).abs() <= bound).all()


def test_dispatch_reports_bad_index(cuda_device):
    x = torch.randn(10, 64, device=cuda_device)
    idx = torch.zeros(10, 2, dtype=torch.int32, device=cuda_device)
    idx[:, 1] = 1
    idx[4, 1] = 99
    out = helpers.dispatch(x, idx, 8)
    torch.cuda.synchronize()
    assert int(out["status"][0]) == _cabi.DEV_BAD_INDEX
    assert int(out["row_of"][4, 1]) == -1
    assert int(out["offsets"][-1]) == 19


EXPERT_CASES = [
    # rows per expert, d, f
    ([5, 0, 130, 1], 64, 128), ([128, 128], 128, 256), ([127, 129, 0, 0, 300], 256, 384),
    ([1], 64, 64), ([0, 0, 7], 72, 88), ([700, 3, 0, 513, 64, 1, 255, 256], 512, 1024),
]


def expert_inputs(rows, d, f, dtype, seed):
    E = len(rows)
    params = synthetic.make_params(d, E, f, seed=seed)
    g = torch.Generator().manual_seed(seed + 1)
    params["b1"] = torch.randn(E, 2 * f, generator=g) * 0.05
    params["b2"] = torch.randn(E, d, generator=g) * 0.05
    params["w1"] *= 3.0
    params["w2"] *= 3.0
    params = helpers.rounded_params(params, dtype)
    M = sum(rows)
    x = synthetic.round_to(torch.randn(M, d, generator=g), dtype)
    offsets = torch.tensor([0] + rows).cumsum(0).to(torch.int32)
    return params, x, offsets


def oracle_experts(params, x, offsets):
    hs, ys = [], []
    for e in range(len(offsets) - 1):
        seg = x[offsets[e]:offsets[e + 1]]
        gu = F.linear(seg, params["w1"][e], params["b1"][e])
        gate, up = gu.chunk(2, dim=-1)
        hs.append(F.gelu(gate, approximate="tanh") * up)
        ys.append(moe_oracle.expert_ffn(seg, params["w1"][e], params["b1"][e], params["w2"][e],
                                        params["b2"][e]))
    return torch.cat(hs), torch.cat(ys)


@pytest.mark.parametrize("rows,d,f", EXPERT_CASES)
def test_experts_fp32(cuda_device, rows, d, f):
    params, x, offsets = expert_inputs(rows, d, f, torch.float32, seed=len(rows) + d)
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, y, status = helpers.experts(x.to(cuda_device), offsets.to(cuda_device), plan)
    torch.cuda.synchronize()
    h_ref, y_ref = oracle_experts(params, x, offsets)
    assert (h.cpu() - h_ref).abs().max() <= 1e-4     # fp32 tolerance of the block: max-abs 1e-4
    assert (y.cpu() - y_ref).abs().max() <= 1e-4


# edges of the fp32 tiles: 4 and 8 rows (short products), 32 (a warp's rows), 64 (a block's); widths that are no
# multiple of 32, 64 or 128; K split over a cluster of up to eight blocks, with ranges that end early
@pytest.mark.parametrize("rows,d,f", [([1, 4, 5, 8, 9, 0, 31], 72, 200), ([64, 65, 32, 33], 264, 136), ([2], 1024, 2056),
                                      ([129, 0, 0, 1], 2056, 8)])
def test_experts_fp32_tile_edges(cuda_device, rows, d, f):
    params, x, offsets = expert_inputs(rows, d, f, torch.float32, seed=3 * len(rows) + d)
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, y, status = helpers.experts(x.to(cuda_device), offsets.to(cuda_device), plan)
    assert status.cpu()[0] == 0
    h_ref, y_ref = oracle_experts({n: t.double() for n, t in params.items()}, x.double(), offsets)
    # sums of at most 2056 fp32 products: a few ulp (2^-24) times the square root of their number
    assert (h.cpu().double() - h_ref).norm() <= 2e-6 * h_ref.norm()
    assert (y.cpu().double() - y_ref).norm() <= 4e-6 * y_ref.norm()


# tiles of 64 rows x 256 columns that end early, one tile and several, ranks up to the largest
@pytest.mark.parametrize("out_f,in_f,rank", [(1, 8, 1), (64, 256, 16), (65, 264, 5), (200, 520, 24), (63, 1032, 64)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_lora_merge(cuda_device, out_f, in_f, rank, dtype):
    g = torch.Generator().manual_seed(out_f + rank)
    rnd = lambda *s: synthetic.round_to(torch.randn(*s, generator=g), dtype)
    W, b, A, a, B, bl = rnd(out_f, in_f), rnd(out_f), rnd(rank, in_f), rnd(rank), rnd(out_f, rank), rnd(out_f)
    dev = [t.to(dtype).to(cuda_device) for t in (W, b, A, a, B, bl)]
    oW, ob = torch.full_like(dev[0], float("nan")), torch.full_like(dev[1], float("nan"))
    check(lib.moe_b200_lora_merge(*[t.data_ptr() for t in dev], 1.3, out_f, in_f, rank, helpers.CODE[dtype],
                                  oW.data_ptr(), ob.data_ptr(), helpers.stream(cuda_device)), "lora_merge")
    scale = float(torch.tensor(1.3))
    ref, refb = W.double() + scale * (B.double() @ A.double()), b.double() + scale * (B.double() @ a.double() + bl.double())
    # fp32 sums of at most 65 products of size 1, then one rounding: to bf16's 8 bits half an ulp, at most 2^-8 of the value
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 0.0
    for got, want in ((oW, ref), (ob, refb)):
        assert ((got.cpu().double() - want).abs() <= eps * want.abs() + 2e-5).all()


# bf16: units of 16 rows x 128 columns, more of them than warps, ranks in steps of 16
@pytest.mark.parametrize("out_f,in_f,rank", [(16, 128, 16), (17, 136, 17), (5000, 1032, 33)])
def test_lora_merge_by_units(cuda_device, out_f, in_f, rank):
    test_lora_merge(cuda_device, out_f, in_f, rank, torch.bfloat16)


@pytest.mark.parametrize("E", [1, 16, 17])      # 2, 32 and 34 Linears: one launch takes 32
def test_lora_merges_of_many_experts(cuda_device, E):
    """The merged weights of all experts are those of a call for each Linear, also when one adapter changed since."""
    from gemmallm_b200 import FeedForward
    from gemmallm_b200.moe import _MergedLora
    with torch.device(cuda_device):
        experts = [FeedForward(72, lora_rank=5, d_ff=264).bfloat16().requires_grad_(False) for _ in range(E)]
    for ex in experts:
        for p in ex.parameters():
            p.normal_(0.0, 0.1)
    lora = _MergedLora()
    for change in (False, True):
        if change:
            experts[-1].lora_down_b.weight.mul_(2.0)
        merged = lora.get(experts, _cabi.BF16, experts[0].gate_and_up.weight.device)
        for ex, mg in zip(experts, merged):
            for lin, a, b, out in ((ex.gate_and_up, ex.lora_gate_and_up_a, ex.lora_gate_and_up_b, mg.gate_and_up),
                                   (ex.down, ex.lora_down_a, ex.lora_down_b, mg.down)):
                W, bias = torch.empty_like(lin.weight), torch.empty_like(lin.bias)
                check(lib.moe_b200_lora_merge(
                    *[t.data_ptr() for m in (lin, a, b) for t in (m.weight, m.bias)], float(ex.lora_scale), lin.out_features,
                    lin.in_features, a.out_features, _cabi.BF16, W.data_ptr(), bias.data_ptr(), helpers.stream(cuda_device)),
                    "lora_merge")
                assert torch.equal(out.weight, W) and torch.equal(out.bias, bias)


# blocks of 16 rows and 16 or 32 tokens that end early, K that ends within a chunk of 32, a round of chunks more, one Linear
# and two; from 129 tokens on tiles of 256 x 2 times 128, the second Linear in either half, K whole and in two and four ranges
@pytest.mark.parametrize("N,K,r,r2", [(1, 8, 1, 0), (15, 40, 17, 2), (16, 1024, 1152, 16), (17, 1032, 72, 5), (33, 264, 2400, 1),
                                      (128, 3080, 48, 31), (129, 8, 8, 0), (255, 264, 128, 8), (300, 1032, 1152, 16),
                                      (257, 2056, 264, 136), (5000, 72, 1152, 16), (3000, 1024, 1024, 0)])
def test_linear_rows(cuda_device, N, K, r, r2):
    g = torch.Generator().manual_seed(N + K)
    rnd = lambda *s: (torch.randn(*s, generator=g) / 4).to(torch.bfloat16)
    x, W, b, W2, b2 = rnd(N, K), rnd(r, K), rnd(r), rnd(max(r2, 1), K), rnd(max(r2, 1))
    dev = [t.to(cuda_device) for t in (x, W, b, W2, b2)]
    out = torch.full((N + 1, r), 7.0, dtype=torch.bfloat16, device=cuda_device)
    out2 = torch.full((N + 1, max(r2, 1)), 7.0, dtype=torch.bfloat16, device=cuda_device)
    ptr, status = [t.data_ptr() for t in dev], torch.zeros(16, dtype=torch.int32, device=cuda_device)
    check(lib.moe_b200_linear_rows(ptr[0], ptr[1], ptr[2], r, ptr[3], ptr[4], r2, N, K, out.data_ptr(), out2.data_ptr(),
                                   status.data_ptr(), helpers.stream(cuda_device)), "linear_rows")
    assert status.cpu()[0] == 0
    for got, w, bias, wanted in ((out, W, b, True), (out2, W2, b2, r2 > 0)):
        assert (got[N:] == 7.0).all()
        if wanted:
            want = x.double() @ w.double().t() + bias.double()
            # K products of size 1/16 in fp32, in whatever order: 2^-24 K of their sum of sizes; half an ulp of bf16
            slack = 2.0 ** -24 * K * (x.double().abs() @ w.double().abs().t() + bias.double().abs())
            assert ((got[:N].cpu().double() - want).abs() <= 2.0 ** -8 * want.abs() + slack).all()
        else:
            assert (got == 7.0).all()


# edges of the fp32 token tiles (16 and 160 tokens) and of the read-outs (64 and 256 of K), whole and with K over clusters
# of two, four and eight CTAs, more tiles than SMs
@pytest.mark.parametrize("rows,d,f", [([15, 16, 17, 159], 512, 2048), ([160, 161, 0, 321], 1024, 512), ([7], 1024, 136),
                                      ([40, 3], 64, 1024), ([33] * 64, 288, 264), ([1] * 9, 264, 1096)])
def test_experts_fp32_against_64_bits(cuda_device, rows, d, f):
    params, x, offsets = expert_inputs(rows, d, f, torch.float32, seed=5 * len(rows) + d)
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, y, status = helpers.experts(x.to(cuda_device), offsets.to(cuda_device), plan)
    assert status.cpu()[0] == 0
    p64 = {n: t.double() for n, t in params.items()}
    h_ref, _ = oracle_experts(p64, x.double(), offsets)
    assert (h.cpu().double() - h_ref).norm() <= 5e-7 * h_ref.norm()
    # the second product of the h it was given; four truncated steps of 2^-23 per read-out, then rounded sums
    y_ref = torch.cat([F.linear(h[offsets[e]:offsets[e + 1]].cpu().double(), p64["w2"][e], p64["b2"][e])
                       for e in range(len(rows))])
    assert (y.cpu().double() - y_ref).norm() <= 3e-7 * y_ref.norm()


@pytest.mark.parametrize("rows,d,f", [([40, 170], 512, 2048), ([3, 2], 1024, 1024)])
def test_experts_fp32_not_finite(cuda_device, rows, d, f):
    """Infinities, NaN and sums that overflow come out as fp32 arithmetic gives them, and nowhere else."""
    params, x, offsets = expert_inputs(rows, d, f, torch.float32, seed=d)
    x[0, 3], x[1, d - 1], x[rows[0] + 1, 5], x[2, 7] = float("inf"), float("nan"), -float("inf"), 3e38
    params["w1"][0, 9, 7], params["w2"][1, 11, 100], params["w1"][1, f + 2, 1] = 1e4, float("inf"), -float("inf")
    # NaN whose upper half alone would be an infinity
    for t, at in ((x, (rows[0], d // 2)), (params["w2"], (0, 13, 5))):
        t.view(torch.int32)[at] = 0x7F800001
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, y, status = helpers.experts(x.to(cuda_device), offsets.to(cuda_device), plan)
    assert status.cpu()[0] == 0
    h_ref, _ = oracle_experts(params, x, offsets)
    y_ref = torch.cat([F.linear(h[offsets[e]:offsets[e + 1]].cpu(), params["w2"][e], params["b2"][e])
                       for e in range(len(rows))])
    for got, ref in ((h.cpu(), h_ref), (y.cpu(), y_ref)):
        assert torch.equal(got.isnan(), ref.isnan())
        assert torch.equal(got.isinf(), ref.isinf()) and torch.equal(got[got.isinf()], ref[ref.isinf()])
        ok = ref.isfinite() & (ref.abs() < 1e6)
        assert torch.allclose(got[ok], ref[ok], atol=1e-4, rtol=1e-5)


@pytest.mark.parametrize("E,K", [(80, 256), (40, 512), (1, 1024)])        # K in one CTA, over two and over eight
def test_experts_fp32_near_the_end_of_the_range(cuda_device, E, K):
    """Products whose first parts cancel while the others, 2^-6 of them, sum up to more than the largest number: finite as
    fp32 arithmetic is. Terms of one sign (1 + 2^-7 - 2^-23)^2 2^127, of the other two that outweigh them."""
    f, top = 64, 2.0 ** 127
    near = 1 + 2.0 ** -7 - 2.0 ** -23
    a = torch.tensor([1.9921875 * top, near * top, near * top, 0.03125 * top] * 64)
    b = torch.tensor([-1.0, near, near, -1.0] * 64)
    params = synthetic.make_params(K, E, f, seed=1)
    for t in params.values():
        t.zero_()
    params["b1"][:, :f] = 1.0                                   # gelu(1) as the factor of the up sums
    params["w1"][:, f:, :256] = b
    x = torch.zeros(2 * E, K)
    x[:, :256] = a
    offsets = torch.arange(E + 1, dtype=torch.int32) * 2
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, _, status = helpers.experts(x.to(cuda_device), offsets.to(cuda_device), plan)
    assert status.cpu()[0] == 0
    want = float(F.gelu(torch.tensor(1.0, dtype=torch.float64), approximate="tanh") * (a.double() @ b.double()))
    # 256 sums of at most 2^128, each rounded: 2^9 2^-24 2^127, where the result is 2^126
    assert (h.cpu().double() - want).abs().max() <= 6.2e-5 * abs(want)


def test_experts_fp32_infinities_take_no_longer(cuda_device):
    """With an infinite weight, and an infinity in every token, within a few times the time without (85 and 200 times as
    long when each sum that was not finite was formed again)."""
    rows, d, f = [128] * 8, 512, 2048
    params, x, offsets = expert_inputs(rows, d, f, torch.float32, seed=4)
    offsets = offsets.to(cuda_device)

    def best(params, x):
        dp = helpers.device_params(params, torch.float32, cuda_device)
        plan, xd, times = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"]), x.to(cuda_device), []
        for _ in range(6):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            helpers.experts(xd, offsets, plan)
            end.record()
            torch.cuda.synchronize()
            times.append(start.elapsed_time(end))
        return min(times)

    clean = best(params, x)
    params["w1"][:, 9, 7] = float("inf")
    assert best(params, x) < 8 * clean
    params["w1"][:, 9, 7] = 0.5
    x[:, 5] = float("inf")
    assert best(params, x) < 8 * clean


def test_experts_fp32_small_operands(cuda_device):
    """Down to 2^-110 an operand is the sum of its three parts; below, what is left out is under 2^-133 of one. Rows around
    2^-104 and 2^-112, results normal numbers."""
    d, f, n = 256, 64, 48
    params, x, offsets = expert_inputs([n, n], d, f, torch.float32, seed=2)
    for t in (params["w1"][:, :f], params["b1"], params["b2"]):
        t.zero_()
    params["b1"][:, :f] = 1.0
    scale = torch.cat([torch.full((n, 1), 2.0 ** -104), torch.full((n, 1), 2.0 ** -112)])
    x *= scale
    dp = helpers.device_params(params, torch.float32, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, _, status = helpers.experts(x.to(cuda_device), offsets.to(cuda_device), plan)
    assert status.cpu()[0] == 0
    up = torch.cat([F.linear(x[:n].double(), params["w1"][0, f:].double()), F.linear(x[n:].double(), params["w1"][1, f:].double())])
    want = F.gelu(torch.ones_like(up), approximate="tanh") * up
    weight = torch.cat([params["w1"][e, f:].double().abs().sum(1).expand(n, f) for e in range(2)])
    err = (h.cpu().double() - want).abs()
    # the sums' rounding (as in test_experts_fp32_against_64_bits, elementwise and not in the 2-norm), and 2^-133 an operand
    assert (err <= 2e-6 * want.abs().mean(1, keepdim=True) + 2.0 ** -133 * weight).all()


def test_gelu_of_the_fp32_experts(cuda_device):
    """Element by element against 64 bits: where the exponential underflows, where it no longer counts beside 1, where the
    quotient's correction ends (a denominator of 1e37), very large arguments, infinities and NaN."""
    inf = float("inf")
    g = torch.cat([torch.linspace(-15, 15, 6001), torch.linspace(-10.2, -9.2, 4001), torch.linspace(4, 7, 2001),
                   torch.logspace(-42, 2, 500), -torch.logspace(-42, 2, 500),
                   torch.tensor([0.0, -0.0, 1e30, -1e30, 3e38, -3e38, inf, -inf, float("nan")])])
    f = (g.numel() + 7) // 8 * 8
    b1 = torch.ones(1, 2 * f)
    b1[0, :g.numel()] = g
    dev = [t.to(cuda_device) for t in (torch.zeros(1, 2 * f, 8), b1, torch.zeros(1, 8, f), torch.zeros(1, 8))]
    h, _, status = helpers.experts(torch.zeros(1, 8, device=cuda_device),
                                   torch.tensor([0, 1], dtype=torch.int32, device=cuda_device), helpers.Plan(*dev))
    assert status.cpu()[0] == 0
    got, g = h[0, :g.numel()].cpu().double(), g.double()
    t = 2 * (2 / torch.pi) ** 0.5 * (g + 0.044715 * g ** 3)
    want = g * torch.sigmoid(t)          # g / 2 (1 + tanh(t / 2)) without its cancellation
    want[g == -inf] = float("nan")       # -inf * 0, as torch's own
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    ok = want.isfinite()
    # t is rounded five times (and its constants), which the exponential turns into |t| times that of its value; then the
    # exponential (2 ulp), the sum, the quotient; under 2^-120 the approximate reciprocal has become zero
    bound = (5 * t.abs().clamp(max=100) + 6) * 2.0 ** -24 * want.abs() + 2.0 ** -120
    assert ((got - want).abs() <= bound)[ok].all()


# the down product with its contraction split over the pairs of a cluster: four and two ranges, the last one shorter,
# K that is no multiple of 64, a last tile of 8 columns, odd CTAs without rows, an expert without rows; 33 tiles: none
@pytest.mark.parametrize("rows,d,f", [([700], 1024, 2056), ([300, 1, 0, 40], 520, 1032), ([2048], 1024, 1024),
                                      ([1], 64, 2048), ([2049], 1024, 1024)])
def test_experts_bf16_split_contraction(cuda_device, rows, d, f):
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=rows[0] + d)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, y, status = helpers.experts(x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device), plan)
    assert status.cpu()[0] == 0
    h_ref, y_ref = oracle_experts(params, x, offsets)
    # h and y are rounded to bf16 once each (2^-9 relative) and h enters the sums of y: within 2^-7 in the 2-norm
    assert (h.float().cpu() - h_ref).norm() <= 2 ** -7 * h_ref.norm()
    assert (y.float().cpu() - y_ref).norm() <= 2 ** -7 * y_ref.norm()


@pytest.mark.parametrize("rows,d,f", EXPERT_CASES)
def test_experts_bf16(cuda_device, rows, d, f):
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=len(rows) + d)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    h, y, status = helpers.experts(x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device),
                                   plan)
    torch.cuda.synchronize()
    assert status.cpu().tolist()[0] == 0, f"device status {status.cpu().tolist()[:4]}"
    h_ref, y_ref = oracle_experts(params, x, offsets)
    # bf16 tolerance of the block: relative error 2e-2 (max-abs over the largest reference value)
    assert (h.float().cpu() - h_ref).abs().max() <= 2e-2 * h_ref.abs().max()
    assert (y.float().cpu() - y_ref).abs().max() <= 2e-2 * y_ref.abs().max()
    assert (y.float().cpu() - y_ref).norm() <= 2e-2 * y_ref.norm()


DECODE_CASES = [
    ([1, 1], 64, 128), ([0, 2, 0, 5, 1], 72, 264), ([16, 0, 17, 15, 20, 30, 2, 28], 1024, 4096),
    ([1, 0, 0, 0, 0, 1, 0, 0], 1024, 4096), ([200, 56], 256, 1408), ([130], 128, 512),
]


@pytest.mark.parametrize("rows,d,f", DECODE_CASES)
def test_experts_decode_path_bf16(cuda_device, rows, d, f):
    """Small-N path: narrow tiles, split-K partial sums; h and sum(part)+bias
    against the oracle at the bf16 tolerance, and against the large-N kernels."""
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=len(rows) + f)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    xd, od = x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device)
    h, part, status = helpers.experts_decode_fused(xd, od, plan)
    h2, y2, _ = helpers.experts(xd, od, plan)
    torch.cuda.synchronize()
    assert status.cpu().tolist()[0] == 0
    assert not torch.isnan(part).any()
    # same products and fp32 accumulation; the MMA operand roles are swapped, so allow an ulp
    assert (h.float() - h2.float()).abs().max() <= 1e-2 * h2.float().abs().max()
    M = sum(rows)
    e_of_row = torch.bucketize(torch.arange(M), offsets.long()[1:], right=True)
    y = part.sum(0).cpu() + params["b2"][e_of_row]
    h_ref, y_ref = oracle_experts(params, x, offsets)
    assert (h.float().cpu() - h_ref).abs().max() <= 2e-2 * h_ref.abs().max()
    assert (y - y_ref).abs().max() <= 2e-2 * y_ref.abs().max()
    assert (y - y2.float().cpu()).abs().max() <= 1e-2 * y_ref.abs().max()
    # combine_decode == fixed-order sum of the partials, bias, bf16 rounding, weights
    k = 2 if (M % 2 == 0 and len(rows) >= 2) else 1
    N = M // k
    g = torch.Generator().manual_seed(M)
    row_of = torch.randperm(M, generator=g).view(N, k).to(torch.int32)
    idx = e_of_row[row_of.long()].to(torch.int32)
    w = torch.rand(N, k, generator=g)
    res = torch.randn(N, d, generator=g).to(torch.bfloat16)
    out = helpers.combine_decode(part, row_of.to(cuda_device), idx.to(cuda_device),
                                 w.to(cuda_device), plan, res.to(cuda_device))
    torch.cuda.synchronize()
    acc_s = torch.zeros(M, d)
    for sp in range(part.shape[0]):
        acc_s = acc_s + part[sp].cpu()
    yb = (acc_s + params["b2"][e_of_row]).to(torch.bfloat16).float()
    acc = torch.zeros(N, d)
    for j in range(k):
        acc = acc + w[:, j:j + 1] * yb[row_of[:, j].long()]
    assert torch.equal(out.cpu(), (acc + res.float()).to(torch.bfloat16))


@pytest.mark.parametrize("rows,d,f", DECODE_CASES)
def test_experts_decode_fused_repeats_bit_for_bit(cuda_device, rows, d, f):
    """The single-launch small-N kernel walks a static tile list with a fixed summation
    order: h and every partial sum come out bit-identical call after call, also when the
    completion counters it is handed are stale."""
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=len(rows) + f)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    xd, od = x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device)
    h, part, status = helpers.experts_decode_fused(xd, od, plan)
    for _ in range(2):
        hf, partf, statusf = helpers.experts_decode_fused(xd, od, plan)
        torch.cuda.synchronize()
        assert statusf.cpu().tolist()[0] == 0
        assert torch.equal(hf, h)
        assert torch.equal(partf, part)


@pytest.mark.parametrize("rows,d,f", DECODE_CASES + [([3, 0, 1, 0, 0, 0, 2, 0], 1024, 4096), ([40, 9], 72, 264)])
def test_experts_gemv_bf16(cuda_device, rows, d, f):
    """The matrix-vector streaming kernels for a few rows per expert (any count works):
    h and sum(part) + bias against the oracle and against the single-launch small-N kernel."""
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=len(rows) + f)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    xd, od = x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device)
    hf, partf, _ = helpers.experts_decode_fused(xd, od, plan)
    h_ref, y_ref = oracle_experts(params, x, offsets)
    M = sum(rows)
    e_of_row = torch.bucketize(torch.arange(M), offsets.long()[1:], right=True)
    for _ in range(2):
        h, part = helpers.experts_gemv(xd, od, plan)
        torch.cuda.synchronize()
        assert not torch.isnan(part).any() and not torch.isnan(h.float()).any()
        assert (h.float().cpu() - h_ref).abs().max() <= 2e-2 * h_ref.abs().max()
        assert (h.float() - hf.float()).abs().max() <= 1e-2 * hf.float().abs().max()
        y = part.sum(0).cpu() + params["b2"][e_of_row]
        assert (y - y_ref).abs().max() <= 2e-2 * y_ref.abs().max()
        assert (part.sum(0) - partf.sum(0)).abs().max() <= 1e-2 * partf.sum(0).abs().max()


@pytest.mark.parametrize("N,d,f,E,k", [(8, 1024, 4096, 8, 2), (8, 256, 200, 8, 4), (5, 2048, 1408, 16, 4),
                                       (1, 64, 24, 4, 4), (8, 128, 264, 32, 8), (8, 64, 64, 8, 8),
                                       (7, 1024, 4096, 8, 2)])
def test_decode_tiny_entry_point(cuda_device, N, d, f, E, k):
    """The one-launch block for one to eight tokens, called directly at sizes where most or all
    experts are hit (more weight rows than its shared memory holds, several column groups per
    block): routing results and output against the oracle, twice in a row."""
    dt = torch.bfloat16
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=N + d), dt)
    dp = helpers.device_params(params, dt, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + f), dt)
    res = synthetic.round_to(synthetic.make_input(N, d, seed=N + f + 1), dt)
    xd, rd = x.to(dt).to(cuda_device), res.to(dt).to(cuda_device)
    for residual in (None, rd):
        r = helpers.decode_tiny(xd, dp["gate_w"], dp["gate_b"], plan, k, f, residual)
        torch.cuda.synchronize()
        assert int(r["status"][0]) == 0
        o = moe_oracle.moe_forward(x, params, k, logits=r["logits"].cpu())
        ok = ~moe_oracle.tie_rows(o["probs"], k)
        assert torch.equal(r["idx"].cpu()[ok].long(), o["idx"][ok])
        assert int(r["offsets"][-1]) == N * k
        assert torch.allclose(r["w"].cpu()[ok], o["w"][ok], atol=2e-6, rtol=0)
        ref = o["out"] if residual is None else o["out"] + res
        got = r["out"].float().cpu()
        assert (got - ref)[ok].abs().max() <= 2e-2 * ref.abs().max()
        assert (got - ref)[ok].norm() <= 2e-2 * ref[ok].norm()


def test_decode_tiny_copies_rows_wider_than_the_grid(cuda_device):
    """More 16-byte pieces of rows than the grid has threads: the rest is copied ahead of the grid barrier."""
    N, d, f, E, k, dt = 4, 43304, 8, 32, 7, torch.bfloat16
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=7), dt)
    dp = helpers.device_params(params, dt, cuda_device)
    x = synthetic.round_to(synthetic.make_input(N, d, seed=8), dt)
    r = helpers.decode_tiny(x.to(dt).to(cuda_device), dp["gate_w"], dp["gate_b"],
                            helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"]), k, f)
    torch.cuda.synchronize()
    assert N * k * d // 8 > torch.cuda.get_device_properties(cuda_device).multi_processor_count * 1024
    rows = r["row_of"].long()
    assert int(r["status"][0]) == 0 and torch.equal(rows.flatten().sort().values, torch.arange(N * k, device=cuda_device))
    assert torch.equal(r["perm"][rows].cpu(), x.to(dt)[:, None, :].expand(N, k, d))
    o = moe_oracle.moe_forward(x, params, k, logits=r["logits"].cpu())
    assert torch.equal(r["idx"].cpu().long(), o["idx"])
    assert (r["out"].float().cpu() - o["out"]).norm() <= 2e-2 * o["out"].norm()


@pytest.mark.parametrize("N,d,E", [(1, 1024, 8), (3, 2048, 16), (2, 264, 32), (20, 1024, 8), (100, 264, 32)])
def test_routing_behind_the_kernel_that_writes_the_router_weights(cuda_device, N, d, E):
    """The kernel in front writes the weights and lets its dependents go early: the routing (one-launch decode, and beyond
    eight tokens the single-launch front) is that of the new weights. (A kernel that spins in front of both has them in
    the queue together.)"""
    dt, f, k = torch.bfloat16, 64, 2
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=d), dt)
    dp = helpers.device_params(params, dt, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    x = synthetic.make_input(N, d, seed=N).to(dt).to(cuda_device)

    def route(gate):
        if N <= 8:
            return helpers.decode_tiny(x, gate, dp["gate_b"], plan, k, f)["logits"]
        i32, f32 = dict(dtype=torch.int32, device=cuda_device), dict(dtype=torch.float32, device=cuda_device)
        outs = [torch.empty(N, E, **f32), torch.empty(N, k, **i32), torch.empty(N, k, **f32), torch.empty(k, E, **i32),
                torch.empty(E + 1, **i32), torch.empty(N, k, **i32), torch.empty(N * k, d, dtype=dt, device=cuda_device),
                torch.empty(E, **f32), torch.empty(1, **f32)]
        check(lib.moe_b200_front_small(x.data_ptr(), gate.data_ptr(), dp["gate_b"].data_ptr(), N, d, E, k, _cabi.BF16,
                                       *(t.data_ptr() for t in outs), helpers.stream(cuda_device)), "front_small")
        return outs[0]

    row_of = torch.arange(E, dtype=torch.int32, device=cuda_device).view(E, 1)
    idx, w = torch.zeros_like(row_of), torch.ones(E, 1, device=cuda_device)
    g = torch.Generator().manual_seed(E)
    parts = [torch.randn(1, E, d, generator=g).to(cuda_device) for _ in range(8)]
    gates = [helpers.combine_decode(p, row_of, idx, w, plan) for p in parts]
    torch.cuda.synchronize()
    want = [route(gate) for gate in gates]
    torch.cuda.synchronize()
    for i, p in enumerate(parts):
        torch.cuda._sleep(2_000_000)
        gate = helpers.combine_decode(p, row_of, idx, w, plan)
        got = route(gate)
        torch.cuda.synchronize()
        assert torch.equal(got, want[i]), i
        gate.zero_()          # what the next round's weights, at this address, hold before they are written


SPEC_CASES = [(1, 64, 128, 2, 2), (8, 1024, 4096, 8, 2), (17, 72, 264, 5, 3), (32, 256, 1408, 32, 4),
              (64, 1024, 4096, 8, 2), (100, 128, 512, 3, 2), (128, 256, 384, 16, 2), (64, 128, 256, 8, 1)]


@pytest.mark.parametrize("N,d,f,E,k", SPEC_CASES)
def test_experts_decode_spec_equals_sorted_path(cuda_device, N, d, f, E, k):
    """The routing-independent small-N kernel works on the unsorted tokens and all
    experts; its partial sums, stored in dispatch row order, match the kernel that
    works on the sorted rows, and sum(part)+bias matches the oracle."""
    dt = torch.bfloat16
    params = synthetic.make_params(d, E, f, seed=N + E)
    g = torch.Generator().manual_seed(N + f)
    params["b1"] = torch.randn(E, 2 * f, generator=g) * 0.05
    params["b2"] = torch.randn(E, d, generator=g) * 0.05
    params["w1"] *= 3.0
    params["w2"] *= 3.0
    params = helpers.rounded_params(params, dt)
    x = synthetic.round_to(torch.randn(N, d, generator=g), dt)
    # random routing with k distinct experts per token; expert E-1 never chosen when E > k
    pool = E - 1 if E > k else E
    idx = torch.stack([torch.randperm(pool, generator=g)[:k] for _ in range(N)]).to(torch.int32)
    dp = helpers.device_params(params, dt, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    xd, idxd = x.to(dt).to(cuda_device), idx.to(cuda_device)
    disp = helpers.dispatch(xd, idxd, E)
    h, part, status = helpers.experts_decode_fused(disp["perm"], disp["offsets"], plan)
    for _ in range(2):
        h_all, part_s, status_s = helpers.experts_decode_spec(xd, idxd, disp["offsets"], plan)
        torch.cuda.synchronize()
        assert status_s.cpu().tolist()[0] == 0
        assert not torch.isnan(part_s).any()
        assert (part_s.sum(0) - part.sum(0)).abs().max() <= 1e-3 * part.sum(0).abs().max()
    # h rows of the routed pairs, against the sorted kernel's h
    row_of = disp["row_of"].cpu().long()
    assert h_all.shape[1] == helpers.lib.moe_b200_decode_spec_rows(N)
    for t in range(0, N, max(1, N // 8)):
        for j in range(k):
            got = h_all[int(idx[t, j]), t].float().cpu()
            ref = h[row_of[t, j]].float().cpu()
            assert (got - ref).abs().max() <= 1e-2 * max(1e-3, float(ref.abs().max()))
    # against the oracle
    offsets = disp["offsets"].cpu()
    e_of_row = torch.bucketize(torch.arange(N * k), offsets.long()[1:], right=True)
    _, y_ref = oracle_experts(params, disp["perm"].float().cpu(), offsets)
    y = part_s.sum(0).cpu() + params["b2"][e_of_row]
    assert (y - y_ref).abs().max() <= 2e-2 * y_ref.abs().max()


@pytest.mark.parametrize("rows,d,f,ksplit", [([100, 0, 300, 57], 256, 1024, 2), ([128] * 8, 1024, 4096, 8),
                                             ([513, 1, 255, 256, 0, 700, 31, 64], 512, 2048, 4),
                                             ([40, 50], 72, 520, 1), ([0, 0, 129], 64, 128, 2),
                                             ([20, 33, 1, 40, 7, 64, 0, 65], 256, 1024, 3)])
def test_experts_rows_matches_prefill_kernels(cuda_device, rows, d, f, ksplit):
    """The streaming pipeline on sorted rows (calls between the decode and the prefill sizes):
    h and sum(part) + bias against the prefill kernels and against the oracle, twice in a row."""
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=len(rows) + f)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    xd, od = x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device)
    h2, y2, _ = helpers.experts(xd, od, plan)
    M = sum(rows)
    e_of_row = torch.bucketize(torch.arange(M), offsets.long()[1:], right=True)
    h_ref, y_ref = oracle_experts(params, x, offsets)
    for _ in range(2):
        h, part, status = helpers.experts_rows(xd, od, plan, ksplit)
        torch.cuda.synchronize()
        assert status.cpu().tolist()[0] == 0
        assert not torch.isnan(part).any() and not torch.isnan(h.float()).any()
        assert (h.float() - h2.float()).abs().max() <= 1e-2 * h2.float().abs().max()
        assert (h.float().cpu() - h_ref).abs().max() <= 2e-2 * h_ref.abs().max()
        y = part.sum(0).cpu() + params["b2"][e_of_row]
        assert (y - y_ref).abs().max() <= 2e-2 * y_ref.abs().max()
        assert (y - y2.float().cpu()).abs().max() <= 1e-2 * y_ref.abs().max()


# 18 blocks of an expert, more than the 16 that take turns on a tile of weights, with several tiles of features in both
# products; blocks of 256 and a row more; one row; few tiles of a long down product; experts without rows
@pytest.mark.parametrize("rows,d,f", [([4400, 3], 520, 264), ([513, 1, 255, 256, 0, 700, 31, 64], 512, 1024),
                                      ([1], 72, 200), ([96, 0, 300], 256, 4096), ([0, 2] * 40, 136, 264)])
def test_experts_mid_matches_prefill_kernels(cuda_device, rows, d, f):
    """Both products in one launch against the prefill kernels and the oracle, twice in a row; the counters are left zero."""
    params, x, offsets = expert_inputs(rows, d, f, torch.bfloat16, seed=len(rows) + f)
    dp = helpers.device_params(params, torch.bfloat16, cuda_device)
    plan = helpers.Plan(dp["w1"], dp["b1"], dp["w2"], dp["b2"])
    xd, od = x.to(torch.bfloat16).to(cuda_device), offsets.to(cuda_device)
    h2, y2, _ = helpers.experts(xd, od, plan)
    h_ref, y_ref = oracle_experts(params, x, offsets)
    for _ in range(2):
        h, y, status, ready = helpers.experts_mid(xd, od, plan)
        torch.cuda.synchronize()
        assert status.cpu().tolist()[0] == 0 and not ready.any()
        # where a sum was formed in another order a last bit of bf16 (2^-7) apart; y by that of h and by its own
        assert (h.float() - h2.float()).abs().max() <= 2 ** -7 * h2.float().abs().max()
        assert (y.float() - y2.float()).abs().max() <= 2 ** -6 * y2.float().abs().max()
        assert (h.float().cpu() - h_ref).abs().max() <= 2e-2 * h_ref.abs().max()
        assert (y.float().cpu() - y_ref).abs().max() <= 2e-2 * y_ref.abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,d,k", [(1, 64, 2), (130, 128, 2), (1000, 512, 4), (33, 72, 1)])
def test_combine_is_exact(cuda_device, N, d, k, dtype):
    g = torch.Generator().manual_seed(N + d)
    y = torch.randn(N * k, d, generator=g).to(dtype)
    row_of = torch.randperm(N * k, generator=g).view(N, k).to(torch.int32)
    w = torch.rand(N, k, generator=g)
    res = torch.randn(N, d, generator=g).to(dtype)
    acc = torch.zeros(N, d)
    for j in range(k):
        acc = acc + w[:, j:j + 1] * y[row_of[:, j].long()].float()
    for residual, expect in ((None, acc), (res, acc + res.float())):
        out = helpers.combine(y.to(cuda_device), row_of.to(cuda_device), w.to(cuda_device),
                              None if residual is None else residual.to(cuda_device))
        torch.cuda.synchronize()
        assert torch.equal(out.cpu(), expect.to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 8])      # one, two and four slots have kernels of their own
def test_combine_of_slots_without_rows(cuda_device, k, dtype):
    """A slot whose row is -1 adds nothing; the others are added in order."""
    N, d, g = 97, 72, torch.Generator().manual_seed(k)
    y = torch.randn(N * k, d, generator=g).to(dtype)
    row_of = torch.randperm(N * k, generator=g).view(N, k).to(torch.int32)
    row_of[torch.rand(N, k, generator=g) < 0.3] = -1
    w, res = torch.rand(N, k, generator=g), torch.randn(N, d, generator=g).to(dtype)
    acc = torch.zeros(N, d)
    for j in range(k):
        has = row_of[:, j] >= 0
        acc[has] = acc[has] + w[has, j:j + 1] * y[row_of[has, j].long()].float()
    out = helpers.combine(y.to(cuda_device), row_of.to(cuda_device), w.to(cuda_device), res.to(cuda_device))
    assert torch.equal(out.cpu(), (acc + res.float()).to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("N,d,E,k", [(777, 256, 8, 2), (64, 1024, 64, 4), (4100, 72, 5, 3)])
def test_layernorm_stage_entry_points(cuda_device, N, d, E, k, dtype):
    """moe_b200_norm_fold + moe_b200_router_norm + moe_b200_dispatch_norm against
    F.layer_norm: row statistics, logits, and the normalised rows in the sorted buffer;
    moe_b200_layernorm against F.layer_norm."""
    import torch.nn.functional as F
    g = torch.Generator().manual_seed(N + d + E)
    x = synthetic.round_to(torch.randn(N, d, generator=g) * (0.3 + torch.rand(N, 1, generator=g) * 3)
                           + 5.0 * torch.randn(N, 1, generator=g), dtype)
    gw = synthetic.round_to(torch.randn(E, d, generator=g) * 0.05, dtype)
    gb = synthetic.round_to(torch.randn(E, generator=g) * 0.1, dtype)
    gamma = synthetic.round_to(1.0 + 0.3 * torch.randn(d, generator=g), dtype)
    beta = synthetic.round_to(0.2 * torch.randn(d, generator=g), dtype)
    dev = cuda_device
    xd, gwd, gbd, gd, bd = (t.to(dtype).to(dev) for t in (x, gw, gb, gamma, beta))
    code = helpers.CODE[dtype]
    s = helpers.stream(dev)
    wn = torch.empty(E, d, dtype=dtype, device=dev)
    c = torch.empty(2 * E, dtype=torch.float32, device=dev)
    check(lib.moe_b200_norm_fold(gwd.data_ptr(), gbd.data_ptr(), gd.data_ptr(), bd.data_ptr(), E, d, code,
                                 wn.data_ptr(), c.data_ptr(), s), "norm_fold")
    logits = torch.empty(N, E, dtype=torch.float32, device=dev)
    idx = torch.empty(N, k, dtype=torch.int32, device=dev)
    w = torch.empty(N, k, dtype=torch.float32, device=dev)
    psum_part = torch.empty(max(1, lib.moe_b200_router_blocks(N)), E, dtype=torch.float32, device=dev)
    stats = torch.empty(N, 2, dtype=torch.float32, device=dev)
    status = torch.zeros(16, dtype=torch.int32, device=dev)
    check(lib.moe_b200_router_norm(xd.data_ptr(), wn.data_ptr(), c.data_ptr(), 1e-5, N, d, E, k, code,
                                   logits.data_ptr(), idx.data_ptr(), w.data_ptr(), psum_part.data_ptr(),
                                   stats.data_ptr(), status.data_ptr(), s), "router_norm")
    torch.cuda.synchronize()
    mean = x.mean(1)
    rstd = torch.rsqrt(x.var(1, unbiased=False) + 1e-5)
    assert torch.allclose(stats[:, 0].cpu(), mean, rtol=1e-5, atol=1e-5)
    assert torch.allclose(stats[:, 1].cpu(), rstd, rtol=2e-5, atol=0)
    xn = F.layer_norm(x, (d,), gamma, beta, 1e-5)
    ref_logits = F.linear(xn, gw, gb)
    tol = 1e-4 if dtype == torch.float32 else 3e-2
    assert (logits.cpu() - ref_logits).abs().max() <= tol * max(1.0, float(ref_logits.abs().max()))
    r = moe_oracle.route_from_logits(logits.cpu(), k)
    good = ~moe_oracle.tie_rows(r["probs"], k)
    assert torch.equal(idx.cpu()[good].long(), r["idx"][good])
    # dispatch: rows of the sorted buffer are the normalised rows
    nbytes = lib.moe_b200_dispatch_scratch_bytes(N, E, k)
    scratch = torch.empty(nbytes // 4, dtype=torch.int32, device=dev)
    cnt_slot = torch.empty(k, E, dtype=torch.int32, device=dev)
    offsets = torch.empty(E + 1, dtype=torch.int32, device=dev)
    row_of = torch.empty(N, k, dtype=torch.int32, device=dev)
    perm = torch.empty(N * k, d, dtype=dtype, device=dev)
    check(lib.moe_b200_dispatch_norm(xd.data_ptr(), idx.data_ptr(), stats.data_ptr(), gd.data_ptr(),
                                     bd.data_ptr(), N, d, E, k, code, scratch.data_ptr(), cnt_slot.data_ptr(),
                                     offsets.data_ptr(), row_of.data_ptr(), perm.data_ptr(), None, None, None,
                                     status.data_ptr(), s), "dispatch_norm")
    out = torch.empty(N, d, dtype=dtype, device=dev)
    check(lib.moe_b200_layernorm(xd.data_ptr(), gd.data_ptr(), bd.data_ptr(), 1e-5, N, d, code, out.data_ptr(), s),
          "layernorm")
    torch.cuda.synchronize()
    assert int(status[0]) == 0
    rtol = 2e-5 if dtype == torch.float32 else 1e-2
    scale = float(xn.abs().max())
    assert (out.float().cpu() - xn).abs().max() <= rtol * scale
    ro = row_of.cpu().long()
    for j in range(k):
        assert (perm.float().cpu()[ro[:, j]] - xn).abs().max() <= rtol * scale


# rounds of two, four and eight tiles, blocks whose share ends within a sequence and of one round; contexts at the edges of the
# 16-token tiles; a position table at an address that is no multiple of 16; masks with -inf, with none
@pytest.mark.parametrize("B,S,H,KV,masked,shift", [(1, 37, 16, 1, True, 0), (1, 1, 16, 1, True, 0), (3, 16, 6, 2, False, 1),
                                                   (2, 17, 4, 4, True, 0), (400, 48, 3, 1, True, 0),
                                                   (300, 15, 2, 1, False, 3), (1, 128, 5, 1, True, 0),
                                                   (97, 64, 16, 1, True, 0), (131, 50, 6, 3, False, 0), (37, 80, 9, 3, True, 1)])
def test_attention_core(cuda_device, B, S, H, KV, masked, shift):
    hd, g = 64, torch.Generator().manual_seed(B + S)
    qkv = synthetic.round_to(torch.randn(B, S, H + 2 * KV, hd, generator=g), torch.bfloat16)
    gate = synthetic.round_to(torch.randn(B, S, H, generator=g), torch.bfloat16)
    table = torch.randn(S, 2 * hd, generator=g)
    mask = torch.full((S, S), float("-inf")).triu(1) if masked else None
    table_d = torch.empty(S * 2 * hd + shift, device=cuda_device)[shift:].view(S, 2 * hd)
    table_d.copy_(table)
    mask_d = None if mask is None else mask.to(cuda_device)
    qkv_d, gate_d = qkv.bfloat16().to(cuda_device), gate.bfloat16().to(cuda_device)
    out = torch.empty(B, S, H * hd, dtype=torch.bfloat16, device=cuda_device)
    check(lib.moe_b200_attention(qkv_d.data_ptr(), gate_d.data_ptr(), table_d.data_ptr(),
                                 None if mask is None else mask_d.data_ptr(), B, S, H, KV, hd, hd ** -0.5,
                                 out.data_ptr(), helpers.stream(cuda_device)), "attention")
    swap = lambda t: t.view(*t.shape[:-1], hd // 2, 2).flip(-1).flatten(-2)
    rope = lambda t: t * table[:, None, :hd] + swap(t) * table[:, None, hd:]
    q, kk, v = qkv.split((H, KV, KV), dim=2)
    q, kk, v = rope(q), rope(kk).repeat_interleave(H // KV, 2), v.repeat_interleave(H // KV, 2)
    scores = torch.einsum("bshd,bthd->bhst", q, kk) * hd ** -0.5
    probs = torch.softmax(scores if mask is None else scores + mask, dim=-1)
    want = (torch.einsum("bhst,bthd->bshd", probs, v) * torch.sigmoid(gate)[..., None]).flatten(2)
    # rotated q and k are rounded to bf16, 2^-9 relative each, which moves scores (of about 2) by about 2^-8 and
    # probabilities by as much of themselves; probabilities and outputs are rounded once more: about 2^-7 in the
    # 2-norm, twice that allowed
    assert (out.float().cpu() - want).norm() <= 2 ** -6 * want.norm()


# 81 to 96 tokens: two blocks an SM without a mask, one with it; shares that end within a sequence
@pytest.mark.parametrize("B,S,H,KV,masked", [(131, 96, 6, 3, False), (61, 81, 6, 3, True), (300, 90, 2, 2, False)])
def test_attention_core_by_blocks_of_an_sm(cuda_device, B, S, H, KV, masked):
    test_attention_core(cuda_device, B, S, H, KV, masked, 0)


# up to 32 router blocks of 64 tokens a warp sums an expert's partial probabilities, beyond them a block
@pytest.mark.parametrize("N,E", [(1, 64), (64, 200), (2048, 17), (2049, 17), (2049, 64)])
def test_dispatch_probability_sums(cuda_device, N, E):
    g = torch.Generator().manual_seed(N + E)
    blocks = (N + 63) // 64
    part = torch.rand(blocks, E, generator=g)
    idx = torch.randint(E, (N, 1), generator=g, dtype=torch.int32)
    got = helpers.dispatch(torch.zeros(N, 8, device=cuda_device).bfloat16(), idx.to(cuda_device), E, part.to(cuda_device))
    want = part.double().sum(0)
    # sums of at most 33 terms in fp32: six roundings on a path of the tree, 2^-24 each
    assert ((got["psum"].cpu().double() - want).abs() <= 6 * 2.0 ** -24 * want).all()
    freq = torch.bincount(idx[:, 0].long(), minlength=E).double() / N
    aux = float((want / N * freq).sum() * E)
    assert abs(float(got["aux"]) - aux) <= 1e-5 * aux
