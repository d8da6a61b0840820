"""The work that users have this framework do, as cases that can be timed and compared.

Three kinds, each through the public entry points:

* ``train``  one ``XCTrainer.train_step`` on a page-locked host batch: host-to-device copies, encoder forward, the
  label-sharded classifier step, encoder backward, both optimizers.  The trainer is what a program keeps between steps;
  it is some hundred steps into the learning-rate warm-up, as a resumed run would be.
* ``embed``  ``XCTrainer.embed_eval`` on a host batch: the encoder in evaluation mode, as prediction calls it.
* ``topk``   ``XFCClassifier.topk`` of a batch of embeddings against a label shard: the other half of prediction.

Sizes are those of ``bench.py``'s workloads, of the recipes in ``docs/train_commands.md`` and of the tests.  Row lengths are
uniform in ``[len_lo, seq]`` as in those workloads (titles and documents shorter than ``--maxlen`` are padded).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from renee_b200.data import xcrepo
from renee_b200.data.collate import XCCollator
from renee_b200.data.synthetic import SyntheticSpec, SyntheticXC
from renee_b200.models.encoder import ENCODER_PRESETS
from renee_b200.models.xfc import XFCClassifier
from renee_b200.parallel.dist import DistContext
from renee_b200.train import TrainConfig, XCTrainer
from renee_b200.utils.sharding import shard_labels

MAX_TOKENS = 16384                 # padded tokens of the largest training step
MAX_LOGITS = 512 * 1310720         # batch x labels of the largest classifier step


def _train(name, enc, batch, seq, len_lo, labels, lam=1.3, zipf=1.1, pooling="cls", bottleneck=0, accum=1, dtype="bf16",
           dropout=0.85):
    return dict(name=name, kind="train", enc=enc, batch=batch, seq=seq, len_lo=len_lo, labels=labels, lam=lam, zipf=zipf,
                pooling=pooling, bottleneck=bottleneck, accum=accum, dtype=dtype, dropout=dropout)


def listed():
    return [
        # the plumbing workload on a GPU: a two-layer encoder and 4 K labels, where launches and latency are everything
        _train("train_tiny", "tiny", 32, 32, 8, 4096, lam=2.0, dropout=0.5),
        # what each of 8 GPUs sees of the 131 K-label workload: 32 rows and a 16 K-label shard
        _train("train_rank_share", "distilbert", 32, 32, 6, 16384),
        # the headline workload: LF-AmazonTitles-131K's shape, short titles
        _train("train_131k_s32", "distilbert", 256, 32, 6, 131072),
        # the same labels with longer text
        _train("train_131k_s128", "distilbert", 128, 128, 32, 131072, lam=4.5),
        # 1.3 M labels: the classifier carries half of the step
        _train("train_1p3m_s32", "distilbert", 512, 32, 6, 1310720, lam=21.0, zipf=1.05),
        # nothing a power of two: fp16 encoder, mean pooling, split accumulation
        _train("train_ragged_fp16", "distilbert", 90, 48, 8, 312330, lam=3.0, pooling="mean", accum=2, dtype="fp16"),
        # full documents at --maxlen 256 on a RoBERTa-style encoder
        _train("train_documents_s256", "distilroberta", 64, 256, 64, 670091, lam=4.5, pooling="mean"),
        # the small encoder with a 64-wide bottleneck and a large batch of very short titles
        _train("train_bottleneck_s16", "minilm-l3", 1024, 16, 4, 1310720, lam=21.0, pooling="mean", bottleneck=64),
        # prediction: the encoder in evaluation mode
        dict(name="embed_s32", kind="embed", enc="distilbert", batch=256, seq=32, len_lo=6, pooling="cls", dtype="bf16"),
        # prediction during training (K = 5) and of the final evaluation (K = 100)
        dict(name="topk5_131k", kind="topk", batch=256, labels=131072, dims=768, k=5),
        dict(name="topk100_1p3m", kind="topk", batch=512, labels=1310720, dims=768, k=100),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(("train", "embed", "topk"), (8, 1, 2))[0]
    if kind == "topk":
        batch = _log_int(rng, 16, 1024)
        return dict(kind="topk", batch=batch, labels=_log_int(rng, 2000, min(1310720, MAX_LOGITS // batch)),
                    dims=rng.choice((768, 768, 384, 64)), k=rng.choice((1, 5, 5, 10, 100)))
    enc = rng.choices(("distilbert", "distilroberta", "minilm-l6", "minilm-l3", "tiny"), (5, 2, 1, 1, 1))[0]
    # sequences beyond 128 tokens belong to the base-sized encoders
    seq = _log_int(rng, 8, 128 if enc.startswith("minilm") else 256)
    batch = _log_int(rng, 8, min(1024, MAX_TOKENS // seq))
    case = dict(kind=kind, enc=enc, batch=batch, seq=seq, len_lo=rng.randint(max(1, seq // 6), seq),
                pooling=rng.choice(("cls", "mean")), dtype=rng.choice(("bf16", "bf16", "bf16", "fp16")))
    if kind == "train":
        case.update(labels=_log_int(rng, 1000, min(1310720, MAX_LOGITS // batch)), lam=rng.choice((1.3, 3.0, 4.5, 21.0)),
                    zipf=rng.choice((1.05, 1.1)), bottleneck=rng.choice((0, 0, 0, 64)), accum=rng.choice((1, 1, 1, 2, 4)),
                    dropout=rng.choice((0.5, 0.75, 0.85)))
    return case


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    if case["kind"] == "topk":
        xfc = XFCClassifier(case["labels"], case["dims"], dev, True, seed=seed, max_batch=case["batch"])
        g = torch.Generator(device=dev).manual_seed(seed + 1)
        return dict(kind="topk", xfc=xfc, k=case["k"],
                    X=torch.randn(case["batch"], case["dims"], generator=g, device=dev).to(xfc.dtype))
    train = case["kind"] == "train"
    enc = ENCODER_PRESETS[case["enc"]]
    B, S = case["batch"], case["seq"]
    labels = case["labels"] if train else 1024
    sharding = shard_labels(labels, 1)
    spec = SyntheticSpec(num_labels=labels, seq_len=S, len_lo=case["len_lo"], len_hi=S, vocab=30522,
                         poisson_lam=case["lam"] if train else 1.3, zipf_s=case["zipf"] if train else 1.1, seed=seed)
    data = xcrepo.InMemoryDataset(*SyntheticXC(spec).rows(np.arange(B)))
    batch = XCCollator(sharding, data, 0, case["accum"] if train else 1, B, train)(np.arange(B)).pin()
    cfg = TrainConfig(batch_size=B, epochs=1, seed=seed, dropout=case["dropout"] if train else 0.5,
                      bottleneck_dims=case["bottleneck"] if train else 0, lr1=0.05, lr2=1e-5, warmup=5000, wd1=1e-4,
                      noloss=True, fp16xfc=True, maxlen=S, pooling=case["pooling"], accum=case["accum"] if train else 1,
                      encoder_dtype=case["dtype"])
    trainer = XCTrainer(cfg, enc, sharding, DistContext(device=dev), steps_per_epoch=100000)
    trainer.xfc_sched.last_step = trainer.tf_sched.last_step = 500
    if case["dtype"] == "fp16":
        trainer.hp.load_state_dict({"scale": 2.0 ** -7})    # where the back-off settles with fp16 gradients of these sizes
    return dict(kind=case["kind"], trainer=trainer, batch=batch)


def run(state):
    if state["kind"] == "topk":
        return state["xfc"].topk(state["X"], state["k"])
    trainer = state["trainer"]
    if state["kind"] == "embed":
        return trainer.embed_eval(state["batch"])
    trainer.train_step(state["batch"])
    enc = trainer.encoder
    # all updated weights, and the gradients of everything behind the embeddings (theirs are a few rows of a large, otherwise
    # empty table, which no single measure of distance suits; they are seen through the updated weights)
    layers = enc.slots["transformer.layer.0.attention.q_lin.weight"].offset
    return {"W": trainer.xfc.W, "momentum": trainer.xfc.M, "encoder": enc.p32, "gradient": enc.g[layers:]}


def _encoder_counts(case):
    """(parameters, parameters of the linear layers) of the case's encoder."""
    c = ENCODER_PRESETS[case["enc"]]
    linear = c.n_layers * (4 * c.dim * c.dim + 2 * c.dim * c.hidden_dim)
    vectors = c.n_layers * (9 * c.dim + c.hidden_dim) + 2 * c.dim
    total = linear + vectors + (c.vocab_size + c.max_position_embeddings) * c.dim
    bottleneck = case.get("bottleneck", 0) * c.dim
    return total + bottleneck, linear + bottleneck


def work(case):
    if case["kind"] == "topk":
        B, L, D, k = case["batch"], case["labels"], case["dims"], case["k"]
        return {"bytes": 2 * (L + B) * D + 12 * B * k, "flops": 2 * B * L * D}
    c = ENCODER_PRESETS[case["enc"]]
    B, lo, hi = case["batch"], case["len_lo"], case["seq"]
    tokens = B * (lo + hi) / 2                                           # expected over the uniform row lengths
    pairs = B * sum(n * n for n in range(lo, hi + 1)) / (hi - lo + 1)    # query-key pairs of one head
    total, linear = _encoder_counts(case)
    forward = 2 * linear * tokens + 4 * pairs * c.dim * c.n_layers
    if case["kind"] == "embed":
        return {"bytes": 2 * linear + 2 * c.dim * (tokens + B), "flops": forward}
    D = case["bottleneck"] or c.dim
    L = case["labels"]
    # encoder: fp32 weights and both moments read and written, 16-bit copy read and written, gradient written;
    # classifier: fp16 weights and momentum read and written
    return {"bytes": total * (24 + 4 + 2) + 8 * L * D, "flops": 3 * forward + 6 * B * L * D}


def tolerance(case):
    if case["kind"] == "topk":
        # fp32 sums of the same fp16 products in another order; neighbours closer than that may change places
        return {"rel": 1e-5, "max": 1e-4, "differ": 4e-3}
    if case["kind"] == "embed":
        # 16-bit activations between the layers: fused and separate epilogues, two correct orders, differ by 0.008
        return {"rel": 2e-2, "max": 0.3}
    # 16-bit activations and gradients between the layers, both ways: the same two orders differ in bf16 by 0.012 with CLS
    # pooling, where all gradient enters through one token of a row, and by 0.005 with mean pooling; fp16 has three more bits
    if case["dtype"] == "fp16":
        return {"rel": 1e-2, "max": 0.3}
    return {"rel": 3e-2, "max": 0.9} if case["pooling"] == "cls" else {"rel": 2e-2, "max": 0.6}
