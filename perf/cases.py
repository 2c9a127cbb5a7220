"""The work a user has this framework do, as cases that can be timed and compared.

Every case is one pass through the public modules: the Mixture-of-Experts block
(``MOE``) in inference and in training, the dense feed-forward (``FeedForward``)
and the decoder layer (``LLMLayer``). Shapes are the repository's own workloads
(gemmallm_b200/synthetic.py): the 1024-wide block with 8 experts of width 4096
and top-2 routing, the 512-wide block in fp32, and the 2048-wide block with 64
experts of width 1408 and top-4 routing. Weights are N(0, 0.02^2), activations
N(0, 1). What is random comes from the case's seed alone.
"""
import math

import torch

from gemmallm_b200 import MOE, FeedForward, LLMLayer

# d_model, experts, expert width, slots
SHAPES = {"d1024": (1024, 8, 4096, 2), "d512": (512, 8, 2048, 2), "e64": (2048, 64, 1408, 4)}
HEAD_DIM, Q_HEADS, KV_HEADS = 64, 16, 1
DROPOUT = 0.1
AUX_WEIGHT = 0.01     # weight of the load-balancing loss in the training loss
LORA_RANK, LORA_LR = 16, 1e-3


def _case(name, kind, batch, seq, shape="d1024", dtype="bf16", gate="zero", residual=False, lora=False):
    c = {"kind": kind, "batch": batch, "seq": seq, "shape": shape, "dtype": dtype, "gate": gate,
         "residual": residual, "lora": lora}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one sequence generating its next token: the block alone, latency and launches count
        _case("block_1", "block", 1, 1),
        # 48 sequences generating together: every expert's weights are read for a few rows each
        _case("block_48", "block", 48, 1, residual=True),
        # a few prompts of uneven length, between the decode and the prefill sizes
        _case("block_6x50", "block", 6, 50),
        # a small batch of 51-token sequences (the length the dense model was trained with)
        _case("block_23x51", "block", 23, 51, residual=True),
        # prefill / evaluation batch, uniform routing: the headline workload
        _case("block_256x64", "block", 256, 64),
        # an odd batch whose router prefers one expert (+2.0 on its bias), skip connection fused
        _case("block_257x51_skew", "block", 257, 51, gate="expert0+2", residual=True),
        # many small experts with Zipf popularity on one GPU, the largest forward
        _case("block_e64_1024x64", "block", 1024, 64, shape="e64", gate="zipf1.1", residual=True),
        # the same block in fp32: the size at which the reference runs on a CPU
        _case("block_fp32_8x64", "block", 8, 64, shape="d512", dtype="f32"),
        # one training step of the block: forward with dropout, backward for x and every parameter
        _case("train_256x64", "train", 256, 64),
        # one LoRA fine-tuning step of the dense feed-forward: base weights frozen, SGD on the LoRA tensors
        _case("finetune_ffn_32x51", "ffn_train", 32, 51, lora=True),
        # one short sequence through a decoder layer (no KV cache: generation re-runs the context)
        _case("layer_1x37", "layer", 1, 37),
        # the decoder's evaluation batch through one layer: attention, folded LayerNorm, block, skips
        _case("layer_512x64", "layer", 512, 64),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _tokens(rng, lo, hi):
    """A token count spread over the logarithm of [lo, hi], as batch x sequence."""
    n = _log_int(rng, lo, hi)
    seq = rng.choice([1, 1, 51, 64, rng.randint(2, 128)]) if n > 1 else 1
    seq = min(seq, n)
    return max(1, n // seq), seq


def draw(rng):
    what = rng.choice(["block", "block", "block", "block", "e64", "fp32", "train", "train", "ffn", "ffn_train",
                       "layer", "layer"])
    if what == "block":
        b, s = _tokens(rng, 1, 32768)
        return _case(None, "block", b, s, gate=rng.choice(["zero", "expert0+2"]), residual=rng.random() < 0.5,
                     lora=rng.random() < 0.2)
    if what == "e64":
        b, s = _tokens(rng, 1, 65536)
        return _case(None, "block", b, s, shape="e64", gate=rng.choice(["zero", "zipf1.1"]),
                     residual=rng.random() < 0.5)
    if what == "fp32":
        b, s = _tokens(rng, 1, 2048)
        return _case(None, "block", b, s, shape="d512", dtype="f32", residual=rng.random() < 0.5)
    if what == "train":
        b, s = _tokens(rng, 64, 16384)
        return _case(None, "train", b, s, shape=rng.choice(["d1024", "d1024", "d512"]),
                     gate=rng.choice(["zero", "expert0+2"]))
    if what == "ffn":
        b, s = _tokens(rng, 1, 32768)
        return _case(None, "ffn", b, s, lora=rng.random() < 0.3)
    if what == "ffn_train":
        b, s = _tokens(rng, 64, 16384)
        return _case(None, "ffn_train", b, s, lora=rng.random() < 0.6)
    return _case(None, "layer", _log_int(rng, 1, 512), rng.choice([1, 51, 64, rng.randint(2, 64)]))


class _Rope(torch.nn.Module):
    """The model's position table: row m = [cos | signed sin] of position m, base 10000."""

    def __init__(self, device):
        super().__init__()
        inv = 10000.0 ** (-torch.arange(0, HEAD_DIM, 2, device=device).float() / HEAD_DIM)
        ang = torch.arange(128, device=device).float()[:, None] * inv[None]
        cos = ang.cos().repeat_interleave(2, dim=1)
        sin = torch.stack((-ang.sin(), ang.sin()), dim=-1).flatten(1)
        self.register_buffer("pos_emb", torch.cat((cos, sin), dim=1))


def _fill(module, gen, gate=None):
    """Weights and biases N(0, 0.02^2), LayerNorms near the identity, the router bias of the case."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.normal_(0.0, 0.02, generator=gen)
            if "norm" in name and name.endswith("weight"):
                p.add_(1.0)
        if gate is not None:
            lin, kind = gate
            lin.bias.zero_()
            if kind == "expert0+2":
                lin.bias[0] = 2.0
            elif kind == "zipf1.1":
                n = lin.bias.numel()
                lin.bias.copy_(torch.tensor([-1.1 * math.log(e + 1) for e in range(n)]))


def _build(make, dtype, device):
    with torch.device("meta"):
        module = make()
    return module.to(dtype).to_empty(device=device)


def prepare(case, seed):
    dev = torch.device("cuda")
    dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
    d, E, f, k = SHAPES[case["shape"]]
    gen = torch.Generator(device=dev).manual_seed(seed)
    kind = case["kind"]
    if kind in ("block", "train"):
        module = _build(lambda: MOE(d, num_experts=E, d_ff=f, top_k=k, dropout_ratio=DROPOUT, device="cuda"), dt, dev)
        _fill(module, gen, (module.gate, case["gate"]))
    elif kind in ("ffn", "ffn_train"):
        module = _build(lambda: FeedForward(d, d_ff=f, dropout_ratio=DROPOUT), dt, dev)
        _fill(module, gen)
    else:
        module = _build(lambda: LLMLayer(d, HEAD_DIM, Q_HEADS, KV_HEADS, torch.nn.Identity(), expansion_factor=f // d,
                                         use_moe=True, num_experts=E, device="cuda"), dt, dev)
        _fill(module, gen, (module.moe.gate, case["gate"]))
        module.mqa.embedding = _Rope(dev)
    x = torch.randn(case["batch"], case["seq"], d, device=dev, generator=gen).to(dt)
    st = {"kind": kind, "module": module, "x": x, "lora": case["lora"]}
    if kind in ("train", "ffn_train"):
        module.train()
        frozen = kind == "ffn_train" and case["lora"]
        named = [(n, p) for n, p in module.named_parameters() if case["lora"] or "lora" not in n]
        for n, p in module.named_parameters():
            p.requires_grad_(not frozen or "lora" in n)
        st["params"] = {n: p for n, p in named if p.requires_grad}
        st["x"] = x.requires_grad_(True)
        st["grad"] = torch.randn(x.shape, device=dev, generator=gen).to(dt)
        st["grad_aux"] = torch.tensor(AUX_WEIGHT, device=dev)
        # the dropout mask is drawn from torch's CPU generator
        st["mask_seed"] = seed
        st["optimizer"] = torch.optim.SGD(st["params"].values(), lr=LORA_LR) if frozen else None
    else:
        module.eval().requires_grad_(False)
        st["residual"] = (torch.randn(x.shape, device=dev, generator=gen).to(dt) if case["residual"] else None)
        if kind == "layer":
            s = case["seq"]
            st["mask"] = torch.full((s, s), float("-inf"), device=dev).triu(1)
    return st


def run(st):
    kind, m, x = st["kind"], st["module"], st["x"]
    if kind in ("train", "ffn_train"):
        torch.default_generator.manual_seed(st["mask_seed"])
        x.grad = None
        for p in st["params"].values():
            p.grad = None
        if kind == "train":
            out, aux = m(x, fine_tuning=st["lora"])
            torch.autograd.backward((out, aux), (st["grad"], st["grad_aux"]))
        else:
            out, aux = m(x, fine_tuning=st["lora"]), None
            torch.autograd.backward(out, st["grad"])
        if st["optimizer"] is not None:
            st["optimizer"].step()
        return out, aux, x.grad, {n: p.grad for n, p in st["params"].items()}
    with torch.no_grad():
        if kind == "block":
            return m(x, fine_tuning=st["lora"], residual=st["residual"])
        if kind == "ffn":
            return m(x, fine_tuning=st["lora"])
        return m(x, attention_mask=st["mask"])


def work(case):
    d, E, f, k = SHAPES[case["shape"]]
    N, S, kind = case["batch"] * case["seq"], case["seq"], case["kind"]
    es = 2 if case["dtype"] == "bf16" else 4
    if kind in ("ffn", "ffn_train"):
        E, k, hit = 1, 1, 1.0
    else:
        hit = E * (1.0 - (1.0 - k / E) ** N)          # experts that uniform routing reaches
    weights = (3 * d * f + 2 * f + d) * es            # one expert
    lora = LORA_RANK * (2 * d + 3 * f) * es           # its four LoRA matrices
    fwd = 6.0 * N * k * d * f
    gate = 2.0 * N * d * E if E > 1 else 0.0
    act = N * d * es
    moved = hit * (weights + (lora if case["lora"] else 0)) + E * d * es + 2 * act
    flops = fwd + gate
    lora_flops = 2.0 * N * k * LORA_RANK * (2 * d + 3 * f)
    if case["lora"] and kind != "block":
        flops += lora_flops
    if case["residual"]:
        moved += act
    if kind == "train" or (kind == "ffn_train" and not case["lora"]):
        # input and weight gradients; the gradients of every parameter are written
        flops += 2 * (fwd + gate)
        moved += 2 * act + E * weights + E * d * es
    elif kind == "ffn_train":
        # frozen base: input gradients, the LoRA tensors' gradients and their update
        flops += fwd + 2 * lora_flops
        moved += 2 * act + 3 * lora
    elif kind == "layer":
        cols = (Q_HEADS + 2 * KV_HEADS) * HEAD_DIM
        flops += 2.0 * N * d * (cols + Q_HEADS * HEAD_DIM + Q_HEADS) + 4.0 * N * S * Q_HEADS * HEAD_DIM
        moved += d * (cols + Q_HEADS * HEAD_DIM + Q_HEADS) * es + 4 * d * es
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    if case["kind"] == "layer":
        # the attention's bf16 output decides the routing behind it: a last-bit difference there
        # moves about one token in five hundred, whose two best experts nearly tie, to another
        # expert, by a part of its row
        return {"rel": 1.5e-2, "max": 0.9}
    return {"rel": 1e-2}
