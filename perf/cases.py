"""The work that a user of this package has it do on one B200, as timed cases: routing, expert layers in inference
and in training, the language-model head, prefill logits and whole training steps.

Every case is a dict of plain values; ``prepare`` makes what a program holds before the call (weights, optimizer,
inputs), ``run`` makes one pass through the public entry points.  All tensors are bf16, the compute type of the
CUDA path.  Sizes come from the shipped configurations (``configs/``), the micro-benchmark suite
(``benchmarks/run_benchmark.py``) and ``bench.py``; ``draw`` spreads the same kinds over their whole ranges.
"""

from __future__ import annotations

import math

import torch

from composed_mixture_of_experts_engine_b200.engine import Trainer
from composed_mixture_of_experts_engine_b200.models import build_model
from composed_mixture_of_experts_engine_b200.models.decoder import lm_head_loss
from composed_mixture_of_experts_engine_b200.ops.moe_router import MoERouter, moe_topk_route
from composed_mixture_of_experts_engine_b200.ops.optim import build_optimizer
from composed_mixture_of_experts_engine_b200.parallel import DistributedMoELayer, ParallelTopology
from composed_mixture_of_experts_engine_b200.utils.config import MoEConfig

BF16 = torch.bfloat16


def listed():
    return [
        # the smallest router shape of the micro-benchmark suite: a call whose time is latency and host work
        dict(name="route_small", kind="route", tokens=512, hidden=256, experts=16, top_k=2),
        # the router shape of the benchmark specification: one pass over 16384 tokens of width 4096
        dict(name="route_spec", kind="route", tokens=16384, hidden=4096, experts=64, top_k=2),
        # router training at the widest configuration (256 experts, top-8), with the load-balance and z losses that
        # configuration turns on; a token count that fills no tile
        dict(name="router_train_256", kind="router_train", tokens=8190, hidden=4096, experts=256, top_k=8),
        # one decode batch: 64 sequences, one token each, through an OLMoE-shaped expert layer
        dict(name="layer_decode", kind="layer_infer", tokens=64, hidden=2048, ffn=1024, experts=64, top_k=8,
             dropping=False),
        # a prefill of odd length through a layer of the single-GPU smoke configuration
        dict(name="layer_prefill_ragged", kind="layer_infer", tokens=3001, hidden=1024, ffn=512, experts=16, top_k=2,
             dropping=False),
        # forward and backward of the expert layer of the headline configuration at its microbatch (4 x 4096 tokens)
        dict(name="layer_train_olmoe", kind="layer_train", tokens=16384, hidden=2048, ffn=1024, experts=64, top_k=8,
             dropping=False, main_grad=False),
        # the same of a Mixtral-shaped layer under the fused optimizer: gradients added into its fp32 buffers
        dict(name="layer_train_mixtral", kind="layer_train", tokens=8192, hidden=4096, ffn=14336, experts=8, top_k=2,
             dropping=False, main_grad=True),
        # the large-scale configuration's experts (H 4096, F 2048, top-8, capacity factor 1.5 with dropping), the 32 of
        # them that one GPU of a group holds, on an odd number of tokens
        dict(name="layer_train_dropping", kind="layer_train", tokens=3333, hidden=4096, ffn=2048, experts=32, top_k=8,
             dropping=True, main_grad=True),
        # the LM head and its loss (forward and both gradients) on two and a half chunks of rows
        dict(name="lm_head", kind="lm_head", tokens=10000, hidden=2048, vocab=50304),
        # prefill logits of a two-layer decoder of the headline widths, one prompt of 1000 tokens
        dict(name="prefill_logits", kind="logits", batch=1, seq=1000, hidden=2048, layers=2, heads=16, kv_heads=16,
             ffn=1024, experts=64, top_k=8, vocab=50304),
        # a whole optimizer step of the single-GPU smoke configuration (two microbatches): launches and host work count
        dict(name="train_small", kind="train", micro=4, accum=2, seq=1024, hidden=1024, layers=4, heads=8, kv_heads=8,
             ffn=512, experts=16, top_k=2, vocab=8192),
        # a whole optimizer step at the headline widths and microbatch, two of its layers, two microbatches
        dict(name="train_olmoe", kind="train", micro=4, accum=2, seq=4096, hidden=2048, layers=2, heads=16, kv_heads=16,
             ffn=1024, experts=64, top_k=8, vocab=50304),
    ]


# -------------------------------------------------------------------------------------------------- drawn cases
def _log(rng, lo, hi, multiple=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return min(hi, max(lo, int(round(v / multiple)) * multiple))


def draw(rng):
    kind = rng.choice(("route", "router_train", "layer_infer", "layer_infer", "layer_train", "layer_train", "lm_head",
                       "logits", "train"))
    if kind in ("route", "router_train"):
        experts = rng.choice((8, 16, 32, 64, 128, 256))
        return dict(kind=kind, tokens=_log(rng, 33, 16384), hidden=_log(rng, 256, 4096, 8), experts=experts,
                    top_k=rng.choice([k for k in (1, 2, 4, 6, 8) if k < experts]))
    if kind in ("layer_infer", "layer_train"):
        experts = rng.choice((8, 16, 32, 64))
        hidden, ffn = _log(rng, 512, 4096, 64), _log(rng, 256, 4096, 64)
        while experts * hidden * ffn > 64 * 2048 * 2048:
            ffn = max(256, ffn // 2 // 64 * 64)
            if ffn == 256:
                hidden = 512
        case = dict(kind=kind, tokens=_log(rng, 5, 16384), hidden=hidden, ffn=ffn, experts=experts,
                    top_k=rng.choice((1, 2, 4, 6)) if experts < 64 else rng.choice((2, 4, 8)),
                    dropping=rng.random() < 0.3)
        if kind == "layer_train":
            case["tokens"] = _log(rng, 500, 16384)
            case["main_grad"] = rng.random() < 0.5
        return case
    if kind == "lm_head":
        return dict(kind=kind, tokens=_log(rng, 500, 16384), hidden=_log(rng, 512, 4096, 64),
                    vocab=_log(rng, 8192, 50304, 8))
    hd = rng.choice((64, 128))
    heads = rng.choice((8, 16)) if hd == 128 else 16
    case = dict(kind=kind, hidden=hd * heads, layers=rng.choice((1, 2)), heads=heads,
                kv_heads=rng.choice((heads, heads // 4)), ffn=rng.choice((256, 512, 1024)),
                experts=rng.choice((8, 16, 64)), top_k=rng.choice((2, 4)), vocab=_log(rng, 8192, 50304, 64))
    if kind == "logits":
        case.update(batch=rng.choice((1, 2, 4)), seq=_log(rng, 65, 2048))
    else:
        case.update(micro=rng.choice((1, 2, 4)), accum=rng.choice((1, 2)), seq=_log(rng, 256, 4096, 64))
    return case


# -------------------------------------------------------------------------------------------------- states
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _tokens(g, n, hidden):
    """Normalised activations: unit variance with a component common to all tokens, as residual streams have; it
    loads the experts unevenly (the busiest gets about three times the mean)."""
    x = torch.randn(n, hidden, generator=g, device="cuda")
    x += 0.5 * torch.randn(1, hidden, generator=g, device="cuda")
    return x.mul_(1.0 / math.sqrt(1.25)).to(BF16)


def _config(c, seed, accum):
    return MoEConfig.from_dict({
        "model": dict(arch="moe_decoder", hidden_dim=c["hidden"], num_layers=c["layers"], num_heads=c["heads"],
                      num_kv_heads=c["kv_heads"], num_experts=c["experts"], top_k=c["top_k"], ffn_dim=c["ffn"],
                      vocab_size=c["vocab"], sequence_length=c["seq"], dtype="bfloat16", aux_loss_coeff=0.01,
                      init_std=0.02),
        "training": dict(micro_batch_size=c.get("micro", c.get("batch", 1)), gradient_accumulation_steps=accum,
                         max_steps=100000, warmup_steps=0, learning_rate=4.0e-4, weight_decay=0.1, grad_clip=1.0,
                         seed=seed),
        "parallelism": dict(data_parallel=1, expert_parallel=1),
    })


def prepare(case, seed):
    c, g = case, _gen(seed)
    kind = c["kind"]
    torch.manual_seed(seed)  # the layers draw their weights from the global generators
    if kind == "route":
        w = torch.randn(c["hidden"], c["experts"], generator=g, device="cuda") / math.sqrt(c["hidden"])
        return dict(c, x=_tokens(g, c["tokens"], c["hidden"]), w=w.to(BF16))
    if kind == "router_train":
        with torch.device("cuda"):
            router = MoERouter(c["hidden"], c["experts"], c["top_k"], dtype=BF16)
        x = _tokens(g, c["tokens"], c["hidden"]).requires_grad_()
        gw = torch.randn(c["tokens"], c["top_k"], generator=g, device="cuda").to(BF16)
        return dict(c, router=router, x=x, gw=gw)
    if kind in ("layer_infer", "layer_train"):
        with torch.device("cuda"):
            layer = DistributedMoELayer(c["hidden"], c["ffn"], c["experts"], c["top_k"], capacity_factor=1.5,
                                        capacity_dropping=c["dropping"], dtype=BF16)
        s = dict(c, layer=layer, x=_tokens(g, c["tokens"], c["hidden"]))
        if kind == "layer_train":
            s["x"].requires_grad_()
            s["dy"] = torch.randn(c["tokens"], c["hidden"], generator=g, device="cuda").to(BF16)
            s["opt"] = build_optimizer(layer, lr=1e-4, max_grad_norm=1.0) if c["main_grad"] else None
        return s
    if kind == "lm_head":
        h = _tokens(g, c["tokens"], c["hidden"]).requires_grad_()
        w = torch.randn(c["vocab"], c["hidden"], generator=g, device="cuda").mul_(0.02).to(BF16).requires_grad_()
        return dict(c, h=h, w=w, targets=torch.randint(0, c["vocab"], (c["tokens"],), generator=g, device="cuda"))
    if kind == "logits":
        model = build_model(_config(c, seed, 1), ParallelTopology(1, 0, 1, 1, device=torch.device("cuda", 0)))
        return dict(c, model=model,
                    ids=torch.randint(0, c["vocab"], (c["batch"], c["seq"]), generator=g, device="cuda"))
    trainer = Trainer(_config(c, seed, c["accum"]))
    ids, targets = trainer.synthetic_batch(torch.Generator().manual_seed(seed))
    return dict(c, trainer=trainer, ids=ids, targets=targets)


# -------------------------------------------------------------------------------------------------- passes
def run(state):
    s, kind = state, state["kind"]
    if kind == "route":
        with torch.no_grad():
            return moe_topk_route(s["x"], s["w"], s["top_k"])
    if kind == "router_train":
        router, x = s["router"], s["x"]
        x.grad = router.gate_w.grad = None
        idx, w, _counts = router(x)
        loss = (w * s["gw"]).sum().float() + 0.01 * router.last_aux_loss + 0.001 * router.last_z_loss
        loss.backward()
        # the counts are read off idx, and the load-balance loss is made of them
        return [idx, w, router.last_aux_loss, router.last_z_loss, x.grad, router.gate_w.grad]
    if kind == "layer_infer":
        with torch.no_grad():
            return s["layer"](s["x"])
    if kind == "layer_train":
        layer, x = s["layer"], s["x"]
        params = [layer.router.gate_w, layer.w13, layer.w2]
        x.grad = None
        if s["opt"] is not None:
            s["opt"].zero_grad()
        for p in params:
            p.grad = None
        y = layer(x)
        y.backward(s["dy"])
        # under the fused optimizer the expert gradients are in its fp32 buffers, the gate's is autograd's
        grads = [p.grad if p.grad is not None else p.main_grad for p in params]
        return [y, x.grad] + grads
    if kind == "lm_head":
        s["h"].grad = s["w"].grad = None
        loss = lm_head_loss(s["h"], s["w"], s["targets"], 1.0 / s["tokens"])
        loss.backward()
        return [loss, s["h"].grad, s["w"].grad]
    if kind == "logits":
        with torch.no_grad():
            return s["model"](s["ids"])
    trainer = s["trainer"]
    loss = trainer.train_step(s["ids"], s["targets"])
    groups = trainer.optimizer.state_dict()["groups"]
    # the updated weights: as the model holds them, and the optimizer's master copies
    return [loss, [p.data for p in trainer.model.parameters()], [g["master"] for g in groups.values()]]


# -------------------------------------------------------------------------------------------------- what a pass needs
def _expert_flops(rows, hidden, ffn):
    return 6.0 * rows * hidden * ffn  # gate, up and down projections


def _decoder_work(c, sequences):
    """(forward flops without the LM head, parameters without embedding and head) of ``sequences`` sequences."""
    n, h, hd = sequences * c["seq"], c["hidden"], c["hidden"] // c["heads"]
    qkv = (c["heads"] + 2 * c["kv_heads"]) * hd
    per_layer = (2.0 * n * h * (qkv + h) + 2.0 * n * c["seq"] * h + 2.0 * n * h * c["experts"]
                 + _expert_flops(n * c["top_k"], h, c["ffn"]))
    params = c["layers"] * (h * (qkv + h) + h * c["experts"] + 3.0 * c["experts"] * h * c["ffn"] + 2 * h)
    return c["layers"] * per_layer, params


def work(case):
    c, kind = case, case["kind"]
    if kind in ("route", "router_train"):
        n, h, e, k = c["tokens"], c["hidden"], c["experts"], c["top_k"]
        nbytes = 2.0 * (n * h + h * e) + n * k * 10
        if kind == "route":
            return dict(bytes=nbytes, flops=2.0 * n * h * e)
        # tokens read and their gradient written, gate weights read and their gradient written, the gate weights'
        # upstream gradient read
        return dict(bytes=nbytes + 2.0 * (n * h + h * e + n * k), flops=6.0 * n * h * e)
    if kind in ("layer_infer", "layer_train"):
        n, h, e = c["tokens"], c["hidden"], c["experts"]
        rows = n * c["top_k"]
        touched = min(1.0, rows / e) * 3.0 * e * h * c["ffn"] if rows < e else 3.0 * e * h * c["ffn"]
        flops = _expert_flops(rows, h, c["ffn"]) + 2.0 * n * h * e
        if kind == "layer_infer":
            return dict(bytes=2.0 * (touched + 2 * n * h + h * e), flops=flops)
        # weights read, gradients written (fp32 under the fused optimizer), x, y, dy, dx
        return dict(bytes=touched * (2.0 + (4.0 if c["main_grad"] else 2.0)) + 8.0 * n * h + 4.0 * h * e, flops=3 * flops)
    if kind == "lm_head":
        n, h, v = c["tokens"], c["hidden"], c["vocab"]
        return dict(bytes=4.0 * (n * h + v * h) + 8.0 * n, flops=6.0 * n * h * v)
    head = float(c["vocab"] * c["hidden"])
    if kind == "logits":
        fwd, params = _decoder_work(c, c["batch"])
        n = c["batch"] * c["seq"]
        return dict(bytes=2.0 * (params + head + n * c["hidden"] + n * c["vocab"]), flops=fwd + 2.0 * n * head)
    sequences = c["micro"] * c["accum"]
    fwd, params = _decoder_work(c, sequences)
    params += 2 * head
    n = sequences * c["seq"]
    # master weights and both moments read and written, bf16 weights written and read once per microbatch
    return dict(bytes=params * (26.0 + 2.0 * c["accum"]) + 16.0 * n, flops=3 * (fwd + 2.0 * n * head))


def tolerance(case):
    """About four times what the kernels differ from this package's PyTorch path (``CMOE_FORCE_LIBRARY=1``: fp64 router,
    cuBLAS experts, eager norms) on the same inputs.  Where two experts are all but tied for the last pick, the paths
    may pick either one, and that token's values then differ throughout (``max``)."""
    kind = case["kind"]
    if kind == "route":  # gate weights differ by single roundings to bf16: rel 1e-4, max 8e-3
        return {"rel": 5e-4, "max": 3e-2, "differ": 2e-4}
    if kind == "router_train":  # rel 1.1e-2 with 5e-5 of the picks another, 2.7e-3 with none
        return {"rel": 3e-2, "max": 0.99, "differ": 2e-4}
    if kind in ("layer_infer", "layer_train"):  # rel 5e-3 to 7e-3
        return {"rel": 2.5e-2, "max": 0.99}
    if kind == "lm_head":  # gradients differ by single roundings to bf16
        return {"rel": 5e-3, "max": 0.1}
    if kind == "logits":  # rel 2.3e-2: the second layer's picks depend on the first one's roundings
        return {"rel": 3e-2, "max": 0.99}
    # weights after the step: rel 5e-3, max 4e-2 (Adam's first steps turn a gradient near zero into a whole step of
    # either sign; the step itself moves the weights by rel 2e-2)
    return {"rel": 2e-2, "max": 0.2}
