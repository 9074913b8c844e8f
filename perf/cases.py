"""The work that a user of this package has its GPU do, as cases that can be timed and compared.

A case is one call of a layer class (``elmo_b200.xmc_classifiers``), the way the training loop and the
evaluator make it, or one training step that starts from label lists on the host (``elmo_b200.glue``):

    step    ``xfc_forward_backward``: forward, loss gradient, embedding gradient, weight update
    host    the same behind ``collate_labels``, ``StepStager`` and ``xmc_train_step``
    logits  ``xfc_forward``
    topk    ``xfc_topk``

over the layer classes (``layer``): ``fp8`` and ``simfp8`` (e4m3 weights, real and simulated FP8 arithmetic),
``kahan`` (e4m3 with compensated head rows) and ``bf16`` (dense bfloat16 weights).  Sizes are those of
``elmo_b200.synth.WORKLOADS``, of the tests, and generic ones around them.
"""
import math
from types import SimpleNamespace as NS

import torch

from elmo_b200.glue import StepStager, collate_labels, xmc_train_step
from elmo_b200.xmc_classifiers import (Fp8XMCBCEChunkedHeadKahanLayer, Fp8XMCBCEChunkedLayer,
                                       XMCBCECHUNKEDLayer)

LR = 0.05                      # learning rate of the layer's SGD (elmo_b200.synth.Workload)
HEAD_RATIO = 0.1               # share of the label rows that the Kahan layer compensates
ZIPF = 1.1                     # label popularity: p(rank k) ~ k^-1.1
LARGEST_WORK = 2812281 * 768 * 1024      # labels x features x batch of the largest listed step
LARGEST_WEIGHTS = 2812281 * 768          # bytes of weights that one layer holds
LARGEST_OUTPUT = 671744 * 512            # logits that one xfc_forward call writes


def _case(name, op, layer, labels, dim, batch, chunks, *, rounding="sr", positives=5, loss=False, k=0,
          embed="bf16"):
    return {"name": name, "op": op, "layer": layer, "labels": labels, "dim": dim, "batch": batch,
            "chunks": chunks, "rounding": rounding, "positives": positives, "loss": loss, "k": k, "embed": embed}


def listed():
    return [
        # a data set of a few thousand labels and a small batch: every launch and host line shows
        _case("step small", "step", "fp8", 4001, 768, 16, 1),
        # the usual small data set, odd batch, with the loss read back every step for logging
        _case("step ragged with loss", "step", "fp8", 31003, 512, 100, 3, loss=True),
        # bfloat16 weights, the layer's default precision
        _case("step bf16", "step", "bf16", 131072, 768, 256, 4),
        # e4m3 weights with a compensated head
        _case("step kahan", "step", "kahan", 312330, 768, 128, 5),
        # simulated FP8 arithmetic, rounding to nearest, many positives per row
        _case("step simulated fp8", "step", "simfp8", 500000, 768, 256, 10, rounding="rn", positives=20),
        # the headline training configuration
        _case("step fp8", "step", "fp8", 670091, 768, 512, 11),
        # millions of labels on one GPU, the batch of a two- or four-GPU encoder
        _case("step largest", "step", "fp8", 2812281, 768, 1024, 8, positives=30),
        # a whole training step from label lists on the host, the way the training loop runs it
        _case("step from host labels", "host", "fp8", 131072, 768, 256, 2),
        # full evaluation scores of the bfloat16 layer
        _case("logits bf16", "logits", "bf16", 131072, 768, 256, 4),
        # evaluation of the headline configuration: the 100 best labels of every row, e4m3 embeddings
        _case("topk evaluation", "topk", "fp8", 670091, 768, 512, 11, k=100, embed="e4m3"),
        # online prediction: one query, the 5 best labels
        _case("topk one query", "topk", "fp8", 131072, 768, 1, 2, k=5),
        # offline prediction in odd batches with the simulated arithmetic
        _case("topk simulated fp8", "topk", "simfp8", 320003, 384, 300, 5, k=10),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: 1 000 to 2.8 million labels, 64 to 1024 features, 1 to 2048 rows."""
    while True:
        op = rng.choice(["step"] * 6 + ["host"] + ["logits"] * 2 + ["topk"] * 3)
        layer = rng.choice({"step": ["fp8", "fp8", "simfp8", "bf16", "kahan"], "host": ["fp8", "bf16"],
                            "logits": ["fp8", "simfp8", "bf16"], "topk": ["fp8", "fp8", "simfp8"]}[op])
        labels = _log_uniform(rng, 1000, 2812281)
        dim = rng.choice([768] * 6 + [1024, 1024, 512, 512, 384, 320, 256, 192, 128, 64])
        batch = _log_uniform(rng, 1, 2048)
        if labels * dim * (2 if layer == "bf16" else 1) > LARGEST_WEIGHTS or labels * dim * batch > LARGEST_WORK:
            continue
        if op == "logits" and labels * batch > LARGEST_OUTPUT:
            continue
        per_chunk = rng.choice([32768, 50000, 65536, 131072])
        return {"op": op, "layer": layer, "labels": labels, "dim": dim, "batch": batch,
                "chunks": max(1, round(labels / per_chunk)), "rounding": rng.choice(["sr", "sr", "rn"]),
                "positives": rng.choice([1, 5, 5, 8, 20, 30]), "loss": op == "step" and rng.random() < 0.25,
                "k": rng.choice([1, 5, 5, 10, 20, 50, 100]) if op == "topk" else 0,
                "embed": rng.choice(["bf16", "e4m3"]) if op in ("logits", "topk") and layer == "fp8" else "bf16"}


# --- inputs ------------------------------------------------------------------------------------------

def _layer(case):
    """The layer a training program builds once.  Built on the GPU; the weights are then those of a layer in
    mid-training, U(+-1/sqrt(d)) as in ``elmo_b200.synth``."""
    cfg = NS(environment=NS(device="cuda:0"),
             model=NS(xmc=NS(dtype="bfloat16", num_chunks=case["chunks"], input_features=case["dim"])),
             training=NS(precision=NS(mode="mixed", purelp_dtype="bfloat16"),
                         xmc=NS(momentum=0, wd=0.0, simulated_fp8=case["layer"] == "simfp8",
                                rounding=case["rounding"]),
                         FP8=NS(using_head_kahan=case["layer"] == "kahan", fp8_head_kahan=False,
                                head_ratio=min(HEAD_RATIO, 0.9 / case["chunks"]))),
             data=NS(num_labels=case["labels"], batch_size=case["batch"]))
    cls = {"bf16": XMCBCECHUNKEDLayer, "kahan": Fp8XMCBCEChunkedHeadKahanLayer}.get(case["layer"],
                                                                                Fp8XMCBCEChunkedLayer)
    with torch.device("cuda:0"):
        layer = cls(cfg)
    return layer


def _weights(layer):
    return [layer.xfc_weight] if isinstance(layer.xfc_weight, torch.Tensor) else [p.data for p in layer.xfc_weight]


def _positives(case, gen):
    """(batch row, label id) pairs: Poisson-many positives per row, popular labels first, none twice in a row."""
    cdf = torch.arange(1, case["labels"] + 1, device="cuda:0", dtype=torch.float64).pow_(-ZIPF).cumsum_(0)
    rate = torch.full((case["batch"],), float(case["positives"]), device="cuda:0")
    counts = torch.poisson(rate, generator=gen).clamp_(1, 200).long()
    rows = torch.repeat_interleave(torch.arange(case["batch"], device="cuda:0"), counts)
    u = torch.rand(rows.numel(), generator=gen, device="cuda:0", dtype=torch.float64) * cdf[-1]
    ids = torch.searchsorted(cdf, u).clamp_(max=case["labels"] - 1)
    pairs = torch.unique(rows * case["labels"] + ids)          # sorted by row, then label
    return torch.stack([pairs // case["labels"], pairs % case["labels"]], 1).to(torch.int32)


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device="cuda:0").manual_seed(seed)
    layer = _layer(case)
    for w in _weights(layer):
        for part in w.split(1 << 18):                           # bounded fp32 temporaries
            part.copy_((torch.rand(part.shape, generator=gen, device="cuda:0") * 2 - 1) / case["dim"] ** 0.5)
    x = torch.randn(case["batch"], case["dim"], generator=gen, device="cuda:0") / case["dim"] ** 0.5
    state = {"case": dict(case), "layer": layer,
             "x": x.to(torch.float8_e4m3fn if case["embed"] == "e4m3" else torch.bfloat16)}
    if case["op"] == "step":
        state["labels"] = _positives(case, gen)
    if case["op"] == "host":
        lists = [[] for _ in range(case["batch"])]
        for row, label in _positives(case, gen).tolist():
            lists[row].append(label)
        state["lists"] = lists
        state["stager"] = StepStager("cuda:0", label_capacity=200 * case["batch"])
    return state


def run(state):
    case, layer, x = state["case"], state["layer"], state["x"]
    if case["op"] == "logits":
        return layer.xfc_forward(x)
    if case["op"] == "topk":
        return layer.xfc_topk(x, case["k"])
    if case["op"] == "host":
        stager = state["stager"]
        stager.put(collate_labels(state["lists"]))
        labels, _ = stager.get()
        loss = xmc_train_step(layer, x, labels, [LR])
        stager.release()
    else:
        loss = layer.xfc_forward_backward(x, state["labels"], [LR], skip_loss=not case["loss"])
    out = {"grad_input": layer.grad_input, "weights": _weights(layer)}
    if case["loss"]:
        out["loss"] = loss
    if case["layer"] == "kahan":
        out["head_kahan"] = layer.head_kahan
    return out


# --- what a pass cannot do without, and how far apart two correct results may be ---------------------------

def work(case):
    labels, dim, batch = case["labels"], case["dim"], case["batch"]
    weights = labels * dim * (2 if case["layer"] == "bf16" else 1)
    embed = batch * dim * (1 if case["embed"] == "e4m3" else 2)
    product = 2.0 * labels * dim * batch
    if case["op"] == "logits":
        return {"bytes": weights + embed + 2 * labels * batch, "flops": product}
    if case["op"] == "topk":
        return {"bytes": weights + embed + 8 * batch * case["k"], "flops": product}
    moved = 2 * weights + 2 * embed + 8 * batch * case["positives"]
    if case["layer"] == "kahan":
        moved += 4 * int(min(HEAD_RATIO, 0.9 / case["chunks"]) * labels) * dim
    return {"bytes": moved, "flops": 3 * product}


def tolerance(case):
    """Logits and gradients are bfloat16 (one rounding: 2^-8).  A weight whose exact update lies at the edge between
    two e4m3 values may land on either, which are up to an eighth of the value apart; a logit that lies
    between two bfloat16 values likewise, which exchanges neighbours among the best labels."""
    if case["op"] == "logits":
        return {"rel": 4e-3, "max": 0.02}
    if case["op"] == "topk":
        return {"rel": 4e-3, "max": 0.02, "differ": 0.01}
    return {"rel": 5e-3, "max": 0.15}
