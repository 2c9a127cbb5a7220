"""Training mode: dropout on h (model.py:164,183) with a mask the CPU oracle can reproduce,
and the backward pass against torch.autograd on the oracle (the reference trains through this
block with loss.backward(), train.py:140-141)."""
import numpy as np
import pytest
import torch

import helpers
import philox_ref
from gemmallm_b200 import MOE, synthetic
from oracle import moe_oracle

DT = torch.bfloat16


def test_philox_known_answer():
    """Published Philox4x32-10 vectors (Random123 kat_vectors): zero counter and key; all-ones
    counter and key."""
    z = np.zeros(1, np.uint64)
    got = [int(a[0]) for a in philox_ref.philox4x32_10(z, z, 0, 0)]
    assert got == [0x6627E8D5, 0xE169C58D, 0xBC57AC4C, 0x9B00DBD8]


def make_block(d, E, f, k, p, dev, seed):
    params = helpers.rounded_params(synthetic.make_params(d, E, f, seed=seed), DT)
    g = torch.Generator().manual_seed(seed + 1)
    params["w1"] = synthetic.round_to(params["w1"] * 2.0, DT)
    params["b1"] = synthetic.round_to(torch.randn(E, 2 * f, generator=g) * 0.05, DT)
    params["b2"] = synthetic.round_to(torch.randn(E, d, generator=g) * 0.05, DT)
    params["gate_w"] = synthetic.round_to(params["gate_w"] * 10.0, DT)   # routing with real preferences
    m = MOE(d, num_experts=E, d_ff=f, top_k=k, dropout_ratio=p, device="cuda")
    synthetic.load_into(m, params, DT, dev)
    return m, params


def oracle_run(x, params, k, mask, grad_out, grad_aux):
    """fp32 forward and torch.autograd backward of the oracle; returns outputs and gradients."""
    leaves = {n: t.clone().requires_grad_(True) for n, t in params.items()}
    xl = x.clone().requires_grad_(True)
    o = moe_oracle.moe_forward(xl, leaves, k, h_mask=mask)
    loss = (o["out"] * grad_out).sum() + grad_aux * o["aux"]
    loss.backward()
    return o, xl.grad, {n: t.grad for n, t in leaves.items()}


def close(got, ref, rel, what):
    got, ref = got.float().cpu(), ref.float()
    scale = float(ref.abs().max())
    err = float((got - ref).abs().max())
    assert err <= rel * scale + 1e-6, f"{what}: max-abs {err:.4g} vs scale {scale:.4g}"
    assert float((got - ref).norm()) <= rel * float(ref.norm()) + 1e-6, f"{what}: Frobenius"


@pytest.mark.gpu
@pytest.mark.parametrize("N,d,E,f,k,p", [(300, 128, 8, 256, 2, 0.1), (1000, 256, 4, 264, 2, 0.25),
                                         (64, 64, 8, 128, 2, 0.0), (700, 128, 16, 192, 4, 0.1)])
def test_training_forward_applies_the_reproducible_dropout_mask(cuda_device, N, d, E, f, k, p):
    m, params = make_block(d, E, f, k, p, cuda_device, seed=N)
    m.train()
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 5), DT)
    with torch.no_grad():
        out, aux = m(x.to(DT).to(cuda_device).view(1, N, d))
    torch.cuda.synchronize()
    assert m.device_status() == 0
    seed = m.last.get("seed", 0)      # p = 0 without gradients is the inference path: no seed
    mult = torch.from_numpy(philox_ref.dropout_multiplier(N * k, f, p, seed)).view(N, k, f)
    if p > 0:
        kept = float((mult > 0).float().mean())
        assert abs(kept - (1 - p)) < 0.01
    logits = m.last["logits"].cpu()
    with torch.no_grad():
        o = moe_oracle.moe_forward(x, params, k, logits=logits, h_mask=mult)
        plain = moe_oracle.moe_forward(x, params, k, logits=logits)
    ok = ~moe_oracle.tie_rows(o["probs"], k)
    assert torch.equal(m.last["idx"].cpu()[ok].long(), o["idx"][ok])
    got = out.view(N, d).float().cpu()
    err = (got - o["out"])[ok].abs().max()
    assert err <= 2e-2 * o["out"].abs().max()
    if p > 0:   # and it is not the forward without dropout
        assert (got - plain["out"])[ok].abs().max() > 5 * err
    # eval mode: no mask
    m.eval()
    with torch.no_grad():
        out_e, _ = m(x.to(DT).to(cuda_device).view(1, N, d))
    torch.cuda.synchronize()
    assert (out_e.view(N, d).float().cpu() - plain["out"])[ok].abs().max() <= 2e-2 * plain["out"].abs().max()


@pytest.mark.gpu
@pytest.mark.parametrize("N,d,E,f,k,p", [(600, 128, 8, 256, 2, 0.1), (1500, 256, 4, 264, 2, 0.0),
                                         (320, 64, 8, 128, 4, 0.2), (2500, 512, 8, 1024, 2, 0.1)])
def test_backward_matches_autograd_on_the_oracle(cuda_device, N, d, E, f, k, p):
    """All gradients of the block (input, gate, both expert Linears with their biases) against
    torch.autograd on the fp32 oracle with the same dropout mask, the same output gradient
    and a load-balancing loss weight. bf16 storage of the intermediate gradients: relative 3e-2."""
    m, params = make_block(d, E, f, k, p, cuda_device, seed=N + 1)
    m.train()
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 6), DT)
    g = torch.Generator().manual_seed(N + 7)
    grad_out = synthetic.round_to(torch.randn(N, d, generator=g), DT)
    grad_aux = 0.5
    xd = x.to(DT).to(cuda_device).view(1, N, d).requires_grad_(True)
    res = synthetic.round_to(synthetic.make_input(N, d, seed=N + 8), DT).to(DT).to(cuda_device).view(1, N, d)
    res.requires_grad_(True)
    out, aux = m(xd, residual=res)
    loss = (out.float() * grad_out.to(cuda_device).view(1, N, d)).sum() + grad_aux * aux
    loss.backward()
    torch.cuda.synchronize()
    assert m.device_status() == 0
    seed = m.last["seed"]
    mult = torch.from_numpy(philox_ref.dropout_multiplier(N * k, f, p, seed)).view(N, k, f)
    o, gx, gp = oracle_run(x, params, k, mult, grad_out, grad_aux)
    # the gradients only compare under the same routing: the seeds are chosen so that it is
    assert torch.equal(m.last["idx"].cpu().long(), o["idx"]), "routing differs from the oracle's own"
    close(out.view(N, d), o["out"].detach() + res.detach().view(N, d).float().cpu(), 2e-2, "forward")
    assert torch.equal(res.grad.view(N, d).float().cpu(), grad_out)          # the residual's gradient
    close(xd.grad.view(N, d), gx, 3e-2, "grad x")
    close(m.gate.weight.grad, gp["gate_w"], 3e-2, "grad gate.weight")
    close(m.gate.bias.grad, gp["gate_b"], 3e-2, "grad gate.bias")
    for e, ex in enumerate(m.experts):
        close(ex.gate_and_up.weight.grad, gp["w1"][e], 3e-2, f"grad experts.{e}.gate_and_up.weight")
        close(ex.gate_and_up.bias.grad, gp["b1"][e], 3e-2, f"grad experts.{e}.gate_and_up.bias")
        close(ex.down.weight.grad, gp["w2"][e], 3e-2, f"grad experts.{e}.down.weight")
        close(ex.down.bias.grad, gp["b2"][e], 3e-2, f"grad experts.{e}.down.bias")
    # a second step on the same module: buffers are reused, gradients accumulate
    out2, aux2 = m(xd, residual=res)
    ((out2.float() * grad_out.to(cuda_device).view(1, N, d)).sum() + grad_aux * aux2).backward()
    torch.cuda.synchronize()
    assert torch.isfinite(m.experts[0].down.weight.grad.float()).all()


LORA_NAMES = (("lora_gate_and_up_a", "gu_a"), ("lora_gate_and_up_b", "gu_b"),
              ("lora_down_a", "dn_a"), ("lora_down_b", "dn_b"))


@pytest.mark.gpu
@pytest.mark.parametrize("N,k", [(37, 2), (38, 2), (39, 3)])
def test_backward_of_token_counts_that_are_no_multiple_of_four(cuda_device, N, k):
    """The gather of the input gradient takes four tokens a thread, with two slots all of them at once: same comparison
    and tolerance as above."""
    test_backward_matches_autograd_on_the_oracle(cuda_device, N, 72, 8, 136, k, 0.1)


@pytest.mark.gpu
@pytest.mark.parametrize("N,E,k", [(33, 3, 2), (31, 9, 3), (70, 16, 2), (40, 17, 2), (40, 33, 4)])
def test_backward_by_the_number_of_experts(cuda_device, N, E, k):
    """A warp of the router's backward pass takes four tokens of up to 8 experts, two of up to 16, else one: same comparison
    and tolerance as above."""
    test_backward_matches_autograd_on_the_oracle(cuda_device, N, 72, E, 136, k, 0.1)


@pytest.mark.gpu
@pytest.mark.parametrize("N,d,E,f,k,p", [(600, 128, 8, 256, 2, 0.1), (900, 256, 4, 264, 2, 0.0)])
def test_fine_tuning_trains_the_lora_tensors(cuda_device, N, d, E, f, k, p):
    """fine_tuning=True under .train() (what the reference's fine-tuning loop runs,
    model.py:175-179,185-189 with train.py's backward): the gradients of the four LoRA Linears
    of every expert, of the base Linears, the gate and the input against torch.autograd on the
    fp32 oracle with the same dropout mask."""
    m, params = make_block(d, E, f, k, p, cuda_device, seed=N + 11)
    g = torch.Generator().manual_seed(N + 12)
    with torch.no_grad():
        for ex in m.experts:
            for name, _ in LORA_NAMES:
                lin = getattr(ex, name)
                lin.weight.copy_(synthetic.round_to(torch.randn(lin.weight.shape, generator=g) * 0.05, DT))
                lin.bias.copy_(synthetic.round_to(torch.randn(lin.bias.shape, generator=g) * 0.05, DT))
    m.train()
    x = synthetic.round_to(synthetic.make_input(N, d, seed=N + 13), DT)
    grad_out = synthetic.round_to(torch.randn(N, d, generator=g), DT)
    grad_aux = 0.25
    xd = x.to(DT).to(cuda_device).view(1, N, d).requires_grad_(True)
    out, aux = m(xd, fine_tuning=True)
    ((out.float() * grad_out.to(cuda_device).view(1, N, d)).sum() + grad_aux * aux).backward()
    torch.cuda.synchronize()
    assert m.device_status() == 0
    mult = torch.from_numpy(philox_ref.dropout_multiplier(N * k, f, p, m.last["seed"])).view(N, k, f)
    leaves = {n: t.clone().requires_grad_(True) for n, t in params.items()}
    lora = []
    for ex in m.experts:
        dct = {"scale": ex.lora_scale}
        for name, short in LORA_NAMES:
            lin = getattr(ex, name)
            dct[short + "_w"] = lin.weight.detach().float().cpu().requires_grad_(True)
            dct[short + "_b"] = lin.bias.detach().float().cpu().requires_grad_(True)
        lora.append(dct)
    xl = x.clone().requires_grad_(True)
    o = moe_oracle.moe_forward(xl, leaves, k, lora=lora, h_mask=mult)
    ((o["out"] * grad_out).sum() + grad_aux * o["aux"]).backward()
    assert torch.equal(m.last["idx"].cpu().long(), o["idx"]), "routing differs from the oracle's own"
    close(out.view(N, d), o["out"].detach(), 2e-2, "forward")
    close(xd.grad.view(N, d), xl.grad, 3e-2, "grad x")
    close(m.gate.weight.grad, leaves["gate_w"].grad, 3e-2, "grad gate.weight")
    for e, ex in enumerate(m.experts):
        close(ex.gate_and_up.weight.grad, leaves["w1"].grad[e], 3e-2, f"grad experts.{e}.gate_and_up.weight")
        close(ex.down.bias.grad, leaves["b2"].grad[e], 3e-2, f"grad experts.{e}.down.bias")
        for name, short in LORA_NAMES:
            lin = getattr(ex, name)
            close(lin.weight.grad, lora[e][short + "_w"].grad, 4e-2, f"grad experts.{e}.{name}.weight")
            close(lin.bias.grad, lora[e][short + "_b"].grad, 4e-2, f"grad experts.{e}.{name}.bias")


@pytest.mark.gpu
def test_training_mode_limits(cuda_device):
    m, _ = make_block(64, 8, 128, 2, 0.1, cuda_device, seed=3)
    m.train()
    x = torch.zeros(1, 16, 64, dtype=DT, device=cuda_device)
    with pytest.raises(NotImplementedError):
        m(x, norm=torch.nn.LayerNorm(64).to(device=cuda_device, dtype=DT))
    with pytest.raises(NotImplementedError):
        m.float()(x.float())


@pytest.mark.gpu
@pytest.mark.parametrize("rows,d,f,p", [(700, 128, 384, 0.1), (64, 64, 128, 0.0), (3000, 256, 520, 0.2)])
def test_dense_feedforward_trains(cuda_device, rows, d, f, p):
    """The reference's dense FeedForward (use_moe=False, model.py:302,316) under .train(): forward
    with the reproducible dropout mask and every gradient against torch.autograd on the oracle's
    expert_ffn (model.py:173-184)."""
    from gemmallm_b200 import FeedForward
    prm = helpers.rounded_params(synthetic.make_params(d, 1, f, seed=rows), DT)
    g = torch.Generator().manual_seed(rows + 1)
    prm["w1"] = synthetic.round_to(prm["w1"] * 2.0, DT)
    prm["b1"] = synthetic.round_to(torch.randn(1, 2 * f, generator=g) * 0.05, DT)
    prm["b2"] = synthetic.round_to(torch.randn(1, d, generator=g) * 0.05, DT)
    ff = FeedForward(d, dropout_ratio=p, d_ff=f).to(device=cuda_device, dtype=DT).train()
    with torch.no_grad():
        ff.gate_and_up.weight.copy_(prm["w1"][0]); ff.gate_and_up.bias.copy_(prm["b1"][0])
        ff.down.weight.copy_(prm["w2"][0]); ff.down.bias.copy_(prm["b2"][0])
    x = synthetic.round_to(synthetic.make_input(rows, d, seed=rows + 2), DT)
    grad_y = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    xd = x.to(DT).to(cuda_device).view(1, rows, d).requires_grad_(True)
    y = ff(xd)
    (y.float() * grad_y.to(cuda_device).view(1, rows, d)).sum().backward()
    torch.cuda.synchronize()
    mult = torch.from_numpy(philox_ref.dropout_multiplier(rows, f, p, ff.last_seed))
    leaves = [t.clone().requires_grad_(True) for t in (x, prm["w1"][0], prm["b1"][0], prm["w2"][0], prm["b2"][0])]
    ref = moe_oracle.expert_ffn(*leaves, h_mask=mult)
    (ref * grad_y).sum().backward()
    close(y.view(rows, d), ref.detach(), 2e-2, "forward")
    close(xd.grad.view(rows, d), leaves[0].grad, 3e-2, "grad x")
    close(ff.gate_and_up.weight.grad, leaves[1].grad, 3e-2, "grad gate_and_up.weight")
    close(ff.gate_and_up.bias.grad, leaves[2].grad, 3e-2, "grad gate_and_up.bias")
    close(ff.down.weight.grad, leaves[3].grad, 3e-2, "grad down.weight")
    close(ff.down.bias.grad, leaves[4].grad, 3e-2, "grad down.bias")


@pytest.mark.gpu
def test_dense_feedforward_fine_tuning_trains_the_lora_tensors(cuda_device):
    """The dense FeedForward with fine_tuning=True under .train(): LoRA gradients against
    torch.autograd on the oracle's expert_ffn with the same dropout mask."""
    from gemmallm_b200 import FeedForward
    rows, d, f, p = 900, 128, 264, 0.1
    g = torch.Generator().manual_seed(77)
    ff = FeedForward(d, dropout_ratio=p, d_ff=f).to(device=cuda_device, dtype=DT).train()
    with torch.no_grad():
        for prm in ff.parameters():
            prm.copy_(synthetic.round_to(torch.randn(prm.shape, generator=g) * 0.05, DT))
    x = synthetic.round_to(synthetic.make_input(rows, d, seed=78), DT)
    grad_y = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    xd = x.to(DT).to(cuda_device).view(1, rows, d).requires_grad_(True)
    y = ff(xd, fine_tuning=True)
    (y.float() * grad_y.to(cuda_device).view(1, rows, d)).sum().backward()
    torch.cuda.synchronize()
    mult = torch.from_numpy(philox_ref.dropout_multiplier(rows, f, p, ff.last_seed))
    cpu = lambda t: t.detach().float().cpu().requires_grad_(True)
    lora = {"scale": ff.lora_scale}
    for name, short in LORA_NAMES:
        lora[short + "_w"], lora[short + "_b"] = cpu(getattr(ff, name).weight), cpu(getattr(ff, name).bias)
    xl = x.clone().requires_grad_(True)
    base = [cpu(ff.gate_and_up.weight), cpu(ff.gate_and_up.bias), cpu(ff.down.weight), cpu(ff.down.bias)]
    ref = moe_oracle.expert_ffn(xl, *base, lora, mult)
    (ref * grad_y).sum().backward()
    close(y.view(rows, d), ref.detach(), 2e-2, "forward")
    close(xd.grad.view(rows, d), xl.grad, 3e-2, "grad x")
    close(ff.down.weight.grad, base[2].grad, 3e-2, "grad down.weight")
    for name, short in LORA_NAMES:
        close(getattr(ff, name).weight.grad, lora[short + "_w"].grad, 4e-2, f"grad {name}.weight")
        close(getattr(ff, name).bias.grad, lora[short + "_b"].grad, 4e-2, f"grad {name}.bias")


@pytest.mark.gpu
@pytest.mark.parametrize("rank,rows,f", [(5, 65, 520), (8, 129, 136), (24, 300, 1032)])
def test_lora_gradients_at_other_ranks(cuda_device, rank, rows, f):
    """LoRA weights whose rows allow 16-byte loads (ranks that are multiples of 8) and those that do not, one and two
    rank steps of 16, contraction ranges of 512 that end early; dx = dgu W with its contraction over 2 f in one, two and
    four ranges. Tolerance as in the test above: bf16 activations and
    gradients, fp32 sums."""
    from gemmallm_b200 import FeedForward
    d, g = 72, torch.Generator().manual_seed(rank)
    ff = FeedForward(d, dropout_ratio=0.0, d_ff=f, lora_rank=rank).to(device=cuda_device, dtype=DT).train()
    with torch.no_grad():
        for prm in ff.parameters():
            prm.copy_(synthetic.round_to(torch.randn(prm.shape, generator=g) * 0.05, DT))
    x = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    grad_y = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    xd, xl = x.to(DT).to(cuda_device).requires_grad_(True), x.clone().requires_grad_(True)
    (ff(xd.view(1, rows, d), fine_tuning=True).float() * grad_y.to(cuda_device)).sum().backward()
    cpu = lambda t: t.detach().float().cpu().requires_grad_(True)
    lora = {"scale": ff.lora_scale}
    for name, short in LORA_NAMES:
        lora[short + "_w"], lora[short + "_b"] = cpu(getattr(ff, name).weight), cpu(getattr(ff, name).bias)
    base = [cpu(ff.gate_and_up.weight), cpu(ff.gate_and_up.bias), cpu(ff.down.weight), cpu(ff.down.bias)]
    (moe_oracle.expert_ffn(xl, *base, lora, None) * grad_y).sum().backward()
    close(xd.grad, xl.grad, 3e-2, "grad x")
    for name, short in LORA_NAMES:
        close(getattr(ff, name).weight.grad, lora[short + "_w"].grad, 4e-2, f"grad {name}.weight")
        close(getattr(ff, name).bias.grad, lora[short + "_b"].grad, 4e-2, f"grad {name}.bias")


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 15, 16, 17, 63, 64, 65, 129, 255, 257])
def test_weight_gradients_at_the_edges_of_a_block_of_rows(cuda_device, rows):
    """The weight-gradient product contracts over the rows in blocks of 64 (sixteen at a time) and cuts the last
    block; the input-gradient product works on 256-row tiles: gradients around those sizes, d and f that are no
    multiples of 64. bf16 products of bf16 operands with fp32 sums: relative 3e-2 as in the tests above."""
    from gemmallm_b200 import FeedForward
    d, f = 72, 136
    g = torch.Generator().manual_seed(rows)
    ff = FeedForward(d, dropout_ratio=0.25, d_ff=f).to(device=cuda_device, dtype=DT).train()
    with torch.no_grad():
        for prm in ff.parameters():
            prm.copy_(synthetic.round_to(torch.randn(prm.shape, generator=g) * 0.1, DT))
    x = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    grad_y = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    xd = x.to(DT).to(cuda_device).requires_grad_(True)
    (ff(xd).float() * grad_y.to(cuda_device)).sum().backward()
    torch.cuda.synchronize()
    mult = torch.from_numpy(philox_ref.dropout_multiplier(rows, f, 0.25, ff.last_seed))
    params = (ff.gate_and_up.weight, ff.gate_and_up.bias, ff.down.weight, ff.down.bias)
    leaves = [t.clone().requires_grad_(True) for t in (x, *(p.detach().float().cpu() for p in params))]
    (moe_oracle.expert_ffn(*leaves, h_mask=mult) * grad_y).sum().backward()
    for got, ref, what in zip((xd, *params), leaves, ("x", "w1", "b1", "w2", "b2")):
        close(got.grad, ref.grad, 3e-2, f"grad {what}")


@pytest.mark.gpu
def test_experts_without_tokens_get_zero_gradients(cuda_device):
    d, E, f, k = 64, 8, 128, 2
    m, _ = make_block(d, E, f, k, 0.1, cuda_device, seed=9)
    with torch.no_grad():
        m.gate.bias[3:] = -100.0
    m.train()
    x = torch.randn(1, 40, d, generator=torch.Generator().manual_seed(1)).to(DT).to(cuda_device)
    for _ in range(2):
        m.zero_grad(set_to_none=True)
        m(x)[0].float().square().sum().backward()
    torch.cuda.synchronize()
    assert m.device_status() == 0 and m.last["cnt_slot"].sum(0)[3:].eq(0).all()
    for e, ex in enumerate(m.experts):
        for p in (ex.gate_and_up.weight, ex.gate_and_up.bias, ex.down.weight, ex.down.bias):
            assert torch.isfinite(p.grad).all()
            assert bool((p.grad != 0).any()) == (e < 3 and bool(m.last["cnt_slot"].sum(0)[e] > 0))


@pytest.mark.gpu
@pytest.mark.parametrize("rows,d,f,rank", [(300, 136, 264, 16), (64, 72, 520, 5), (1632, 256, 1032, 24)])
def test_lora_step_keeps_its_rounding_points(cuda_device, rows, d, f, rank):
    """A LoRA step rounds to bf16 where a step through the merged weights' own gradients does: pre-activations, dh, dg and
    du, and G = dL/dW', from which the LoRA gradients are formed (an SGD step on them feeds the next pass, so other
    rounding points drift apart from step to step). The same arithmetic in 64 bits with these roundings gives what the
    kernels give, but for values that lie at a rounding boundary: a sum's fp32 error (about 2^-20 of it) and that of the
    GELU's exponential (2^-21) turn less than one value in 200 of bf16's 2^-8, below 3e-4 of a 2-norm, and pass through at
    most two further products. Without the rounding of dh the gradients differ by 3.6e-3."""
    from gemmallm_b200 import FeedForward
    g = torch.Generator().manual_seed(rows)
    ff = FeedForward(d, dropout_ratio=0.0, d_ff=f, lora_rank=rank).to(device=cuda_device, dtype=DT).train()
    with torch.no_grad():
        for prm in ff.parameters():
            prm.copy_(synthetic.round_to(torch.randn(prm.shape, generator=g) * 0.05, DT))
    x = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    dy = synthetic.round_to(torch.randn(rows, d, generator=g), DT)
    xd = x.to(DT).to(cuda_device).requires_grad_(True)
    ff(xd, fine_tuning=True).backward(dy.to(DT).to(cuda_device))
    cpu = lambda t: t.detach().cpu().double()
    bf = lambda t: t.to(DT).double()
    s = ff.lora_scale
    lins = [tuple(cpu(t) for lin in (w, a, b) for t in (lin.weight, lin.bias))
            for w, a, b in ((ff.gate_and_up, ff.lora_gate_and_up_a, ff.lora_gate_and_up_b),
                            (ff.down, ff.lora_down_a, ff.lora_down_b))]
    (w1, b1), (w2, _) = [(bf(W + s * B @ A), bf(b + s * (B @ a + bl))) for W, b, A, a, B, bl in lins]
    x, dy = x.double(), dy.double()
    z, u = bf(x @ w1.t() + b1).split(f, dim=1)
    beta, alpha = 0.7978845608028654, 0.044715
    t = torch.tanh(beta * (z + alpha * z ** 3))
    dgelu = 0.5 * (1 + t) + 0.5 * z * (1 - t * t) * beta * (1 + 3 * alpha * z * z)
    dh = bf(dy @ w2)
    dgu = bf(torch.cat((dh * u * dgelu, dh * 0.5 * z * (1 + t)), dim=1))
    off = lambda got, ref: float((cpu(got) - ref).norm() / ref.norm())
    assert off(xd.grad, bf(dgu @ w1)) <= 1e-3
    assert off(ff.gate_and_up.weight.grad, bf(dgu.t() @ x)) <= 1e-3
    assert off(ff.gate_and_up.bias.grad, bf(dgu.sum(0))) <= 1e-3
    assert off(ff.down.bias.grad, bf(dy.sum(0))) <= 1e-3
    # the LoRA gradients from the kernels' own G and g: one rounding behind fp32 sums
    for (_, _, A, a, B, _), w, la, lb in zip(lins, (ff.gate_and_up, ff.down), (ff.lora_gate_and_up_a, ff.lora_down_a),
                                             (ff.lora_gate_and_up_b, ff.lora_down_b)):
        G, gb = cpu(w.weight.grad), cpu(w.bias.grad)
        assert off(la.weight.grad, bf(s * B.t() @ G)) <= 5e-4
        assert off(la.bias.grad, bf(s * B.t() @ gb)) <= 1e-3        # a few values: one at a boundary counts more
        assert off(lb.weight.grad, bf(s * (G @ A.t() + torch.outer(gb, a)))) <= 5e-4
        assert off(lb.bias.grad, bf(s * gb)) == 0.0


@pytest.mark.gpu
def test_bias_gradients_of_more_row_tiles_than_a_grid_dimension(cuda_device):
    """65536 tiles of 256 rows: tiles lie along the grid dimension that goes beyond 65535. Rows of ones and a gradient that is
    one in the last row alone (the other rows' sums are zero and exact)."""
    from gemmallm_b200 import FeedForward
    rows, d, f = 65535 * 256 + 1, 8, 8
    torch.manual_seed(0)
    ff = FeedForward(d, dropout_ratio=0.0, d_ff=f).to(device=cuda_device, dtype=DT).train()
    x = torch.ones(rows, d, dtype=DT, device=cuda_device).requires_grad_(True)
    y = ff(x)
    grad = torch.zeros_like(y)
    grad[-1] = 1.0
    y.backward(grad)
    assert torch.equal(ff.down.bias.grad, torch.ones_like(ff.down.bias))
    assert (x.grad[:-1] == 0).all() and (x.grad[-1] != 0).any() and (ff.gate_and_up.bias.grad != 0).any()
