"""The work that users of this package have it do, as cases to time: the operators that stand in for the reference's
own (scan, linear cross-entropy), one recurrent block, whole training steps, prompt prefill and cached decoding.

Every case goes through the public entry points: `fused_linear_scan`, `fused_cross_entropy`, `model.Hawk`,
`train.Trainer.step`, `generate.GraphedDecoder.prefill` / `.step`.  Two model shapes set the range: the README
model (hidden = recurrent = 512, intermediate 1024, vocabulary 32000, 16 gate blocks) and the 1.35 B model (hidden =
recurrent = 2048, intermediate 6144, 24 layers).  Training cases run 4 layers of a shape: the layers are alike, and
4 leave room for every gradient among the outputs.
"""
import math
import os
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "hawk-pytorch_b200"))

from hawk_b200 import fused_cross_entropy, fused_linear_scan  # noqa: E402
from hawk_b200.generate import GraphedDecoder  # noqa: E402
from hawk_b200.model import Hawk, HawkConfig, HawkModel, ring_init_  # noqa: E402
from hawk_b200.train import Trainer  # noqa: E402

DEV = "cuda"
VOCAB, BLOCKS, CONV = 32000, 16, 4
DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16}


def listed():
    return [
        # the scan operator as the reference's users call it, forward and backward: a small fp32 call, where launches
        # and latency count; many tokens of uneven length in a middling width; one very long sequence of a wide model
        dict(name="scan_f32_small", kind="scan", batch=2, seq=2048, width=512, dtype="f32"),
        dict(name="scan_bf16_ragged", kind="scan", batch=5, seq=3001, width=1536, dtype="bf16"),
        dict(name="scan_bf16_long", kind="scan", batch=1, seq=65536, width=4096, dtype="bf16"),
        # the loss operator at the 1.35 B model's training shape: 8 sequences of 4096 tokens, next-token targets
        dict(name="loss_large", kind="loss", rows=8 * 4095, hidden=2048, vocab=VOCAB, act="f32"),
        # one recurrent block of the README model under bf16 autocast, forward and backward
        dict(name="block_readme", kind="block", batch=8, seq=2048, width=512),
        # training steps (forward, loss, backward, AdamW): a few short sequences of odd length, as in fine-tuning or
        # on a small card's share; the README configuration's batch; the 1.35 B model's per-GPU batch
        dict(name="train_ragged", kind="train", hidden=512, inter=1024, layers=4, batch=3, seq=517),
        dict(name="train_readme", kind="train", hidden=512, inter=1024, layers=4, batch=16, seq=2048),
        dict(name="train_1b", kind="train", hidden=2048, inter=6144, layers=4, batch=8, seq=4096),
        # serving the 1.35 B model in bf16: a handful of prompts of odd length into the caches
        dict(name="prefill_1b", kind="prefill", hidden=2048, inter=6144, layers=24, batch=4, seq=777, weights="bf16"),
        # one cached token: the README model with the decoder's default options (fp32 weights under autocast), then
        # the 1.35 B model in bf16 for one user and for a full batch
        dict(name="decode_readme", kind="decode", hidden=512, inter=1024, layers=8, batch=16, weights="f32"),
        dict(name="decode_1b_single", kind="decode", hidden=2048, inter=6144, layers=24, batch=1, weights="bf16"),
        dict(name="decode_1b_batch", kind="decode", hidden=2048, inter=6144, layers=24, batch=256, weights="bf16"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges.  Widths are those of the tests, the benchmark and between; lengths and batch
    sizes are any whole number; no case costs more than the largest listed one of its kind."""
    kind = rng.choice(["scan", "scan", "loss", "block", "train", "train", "prefill", "decode", "decode"])
    if kind == "scan":
        width = 64 * _log_int(rng, 1, 64)
        batch = _log_int(rng, 1, 16)
        most = min(65536, (1 << 27) // (batch * width))
        return dict(kind=kind, batch=batch, seq=_log_int(rng, min(64, most), most), width=width,
                    dtype=rng.choice(["bf16", "bf16", "f32"]))
    if kind == "loss":
        return dict(kind=kind, rows=_log_int(rng, 256, 32760), hidden=64 * _log_int(rng, 4, 32),
                    vocab=rng.choice([VOCAB, VOCAB, _log_int(rng, 1000, VOCAB)]), act=rng.choice(["bf16", "f32"]))
    hidden = rng.choice([256, 512, 768, 1024, 1536, 2048])
    inter = hidden * rng.choice([2, 3])
    if kind == "block":
        batch = _log_int(rng, 1, 16)
        return dict(kind=kind, batch=batch, seq=_log_int(rng, 128, 32768 // batch), width=hidden)
    if kind == "train":
        batch = _log_int(rng, 1, 16)
        return dict(kind=kind, hidden=hidden, inter=inter, layers=rng.randint(1, 4), batch=batch,
                    seq=_log_int(rng, 64, min(4096, 32768 // batch)))
    layers = rng.randint(4, 24)
    if kind == "prefill":
        batch = _log_int(rng, 1, 16)
        return dict(kind=kind, hidden=hidden, inter=inter, layers=layers, batch=batch,
                    seq=_log_int(rng, 4, min(2048, 3108 // batch)), weights="bf16")
    return dict(kind=kind, hidden=hidden, inter=inter, layers=layers, batch=_log_int(rng, 1, 256),
                weights=rng.choice(["bf16", "bf16", "f32"]))


# ---- inputs ----------------------------------------------------------------------------------------------------
def _config(case):
    return HawkConfig(VOCAB, case["hidden"], case["inter"], case["layers"], case["hidden"], BLOCKS, CONV)


def _trained_scale_(module, layers):
    """The branch outputs and the head start at zero and the embeddings at 1/sqrt(width); give them the proportions of
    a trained model: unit embeddings and branches that together add about as much again to the residual stream."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if name.endswith("resid_proj.weight"):
                p.normal_(0.0, 1.0 / math.sqrt(2 * layers * p.shape[1]))
            elif name.endswith("lm_head.weight"):
                p.normal_(0.0, 1.0 / math.sqrt(p.shape[1]))
            elif name.endswith("embed_tokens.weight"):
                p.normal_()


def _tokens(case, seq):
    return torch.randint(1, VOCAB, (case["batch"], seq), device=DEV)


def _decoder(case):
    half = case["weights"] == "bf16"
    with torch.device(DEV):
        model = HawkModel(_config(case), use_cache=True)
    _trained_scale_(model, case["layers"])
    if half:
        model = model.bfloat16()
    return GraphedDecoder(model, case["batch"], **({"autocast": False} if half else {}))


def prepare(case, seed):
    torch.manual_seed(seed)
    kind = case["kind"]
    if kind == "scan":
        shape = (case["batch"], case["seq"], case["width"])
        x, gx, ga, go = (torch.randn(shape, device=DEV).to(DTYPES[case["dtype"]]) for _ in range(4))
        lam = ring_init_(torch.empty(case["width"], device=DEV))
        return dict(kind=kind, go=go, ins=[t.requires_grad_() for t in (x, gx, ga, lam)])
    if kind == "loss":
        w = torch.randn(case["vocab"], case["hidden"], device=DEV) / math.sqrt(case["hidden"])
        act = torch.randn(case["rows"], case["hidden"], device=DEV).to(DTYPES[case["act"]])
        labels = torch.randint(0, case["vocab"], (case["rows"],), device=DEV)
        return dict(kind=kind, labels=labels, ins=[w.requires_grad_(), act.requires_grad_()])
    if kind == "block":
        width = case["width"]
        with torch.device(DEV):
            block = Hawk(HawkConfig(VOCAB, width, 2 * width, 1, width, BLOCKS, CONV))
        _trained_scale_(block, 1)
        x, go = (torch.randn(case["batch"], case["seq"], width, device=DEV).bfloat16() for _ in range(2))
        return dict(kind=kind, block=block, go=go, ins=[x.requires_grad_()] + list(block.parameters()))
    if kind == "train":
        with torch.device(DEV):
            trainer = Trainer(_config(case), DEV, seed=seed)
        _trained_scale_(trainer.model, case["layers"])
        return dict(kind=kind, trainer=trainer, params=list(trainer.model.parameters()), ids=_tokens(case, case["seq"]))
    dec = _decoder(case)
    if kind == "prefill":
        return dict(kind=kind, dec=dec, ids=_tokens(case, case["seq"]))
    dec.prefill(_tokens(case, 16))
    dec.step(_tokens(case, 1))  # a serving loop is past its first token: the step has been captured
    return dict(kind=kind, dec=dec, ids=_tokens(case, 1))


# ---- one pass --------------------------------------------------------------------------------------------------
def _caches(dec):
    return [t for c in dec.caches for t in (c.recc_state, c.conv_state)]


def run(state):
    kind = state["kind"]
    if kind == "scan":
        h = fused_linear_scan(*state["ins"])
        return [h, *torch.autograd.grad(h, state["ins"], state["go"])]
    if kind == "loss":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = fused_cross_entropy(*state["ins"], state["labels"])
        return [loss, *torch.autograd.grad(loss, state["ins"])]
    if kind == "block":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            out, _ = state["block"](state["ins"][0])
        return [out, *torch.autograd.grad(out, state["ins"], state["go"])]
    if kind == "train":
        grads = []
        loss = state["trainer"].step(state["ids"], after_backward=lambda _: grads.extend(p.grad for p in state["params"]))
        return [loss, *grads]
    dec = state["dec"]
    logits = dec.prefill(state["ids"]) if kind == "prefill" else dec.step(state["ids"])
    return [logits, *_caches(dec)]


# ---- what a pass cannot do without -----------------------------------------------------------------------------
def _weights(case):
    """Parameters of the model in matrices that every token is multiplied with: per layer, and the head."""
    h, i = case["hidden"], case["inter"]
    layer = 2 * h * h + h * h + 2 * h * i + i * h + 2 * h * (h // BLOCKS)
    return layer, VOCAB * h


def work(case):
    kind = case["kind"]
    if kind == "scan":
        n, es = case["batch"] * case["seq"] * case["width"], 2 if case["dtype"] == "bf16" else 4
        return {"bytes": 8 * es * n, "flops": 60 * n}  # read x, gx, ga, go; write h and three gradients
    if kind == "loss":
        n, h, v = case["rows"], case["hidden"], case["vocab"]
        return {"bytes": 8 * v * h + (4 if case["act"] == "bf16" else 8) * n * h + 8 * n, "flops": 6 * n * h * v}
    if kind == "block":
        n, r = case["batch"] * case["seq"], case["width"]
        par = 3 * r * r + 2 * r * (r // BLOCKS)
        return {"bytes": 8 * n * r + 8 * par, "flops": 6 * n * par}
    layer, head = _weights(case)
    total = case["layers"] * layer + head
    if kind == "train":
        n = case["batch"] * case["seq"]
        # AdamW reads and writes p, m, v in fp32; the gradients are among the results
        return {"bytes": 28 * (total + VOCAB * case["hidden"]) + 8 * n, "flops": 6 * n * total}
    tokens = case["batch"] * (case["seq"] if kind == "prefill" else 1)
    size = 2 if case["weights"] == "bf16" else 4
    caches = 2 * case["layers"] * case["batch"] * case["hidden"] * CONV * (2 if kind == "decode" else 1)
    return {"bytes": size * total + caches + 2 * tokens * VOCAB, "flops": 2 * tokens * total}


def tolerance(case):
    """About four times what two correct computations differ by, measured: the scan and the loss against the same in 64
    bits (5e-7 in fp32, 2e-3 and 2.5e-3 in bf16), the block (5e-3) and three training steps (8e-3) with the gate
    products in another order and against fp32 activations, serving (1.3e-2) against fp32 activations and caches."""
    kind = case["kind"]
    if kind == "scan":
        return {"rel": 4e-6 if case["dtype"] == "f32" else 8e-3}
    return {"rel": {"loss": 1e-2, "block": 2e-2}.get(kind, 3e-2)}
