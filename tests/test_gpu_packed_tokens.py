"""Packed tokens against the padded layout on the same own-GEMM engine: same weights, same dropout counters."""
from __future__ import annotations

import os

import pytest
import torch

pytestmark = pytest.mark.gpu


def _engine(cfg, dtype, pooling):
    from renee_b200.models.flat_encoder import FlatEncoder
    os.environ["RENEE_B200_OWN_GEMM"] = "1"
    try:
        return FlatEncoder(cfg, torch.device("cuda", 0), dtype, pooling, 0, seed=3)
    finally:
        os.environ.pop("RENEE_B200_OWN_GEMM", None)


def _mask(kind, b, S, gen):
    m = torch.zeros(b, S, dtype=torch.int32)
    if kind == "full":
        m += 1
    elif kind == "prefix":
        for i in range(b):
            m[i, : int(torch.randint(1, S + 1, (1,), generator=gen))] = 1
    elif kind == "holes":           # any mask is accepted: gaps, a masked first token, values other than 1
        m = (torch.rand(b, S, generator=gen) < 0.4).to(torch.int32) * 3
        m[0, 0] = 0
        m[0, -1] = 1
    if kind == "empty_rows" or kind == "holes":
        m[b // 2] = 0               # a wholly masked row: uniform softmax over all its keys
    if kind == "empty_rows":
        m[0] = 1
    return m.cuda()


@pytest.mark.parametrize("S,b,kind,pooling,dt", [
    (32, 24, "prefix", "cls", torch.bfloat16), (32, 24, "full", "mean", torch.bfloat16),
    (20, 7, "holes", "mean", torch.float16), (20, 7, "holes", "cls", torch.bfloat16), (1, 5, "full", "cls", torch.bfloat16),
    (7, 9, "empty_rows", "mean", torch.bfloat16), (64, 6, "prefix", "mean", torch.bfloat16),
    (128, 5, "holes", "mean", torch.bfloat16), (100, 3, "prefix", "cls", torch.float16),
    (256, 4, "prefix", "mean", torch.bfloat16), (201, 3, "holes", "mean", torch.bfloat16), (130, 2, "empty_rows", "cls", torch.bfloat16),
])
@pytest.mark.parametrize("hint", [0, 64])
def test_packed_equals_padded(S, b, kind, pooling, dt, hint):
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.ops import StepRNG, cuda as cu
    cfg = EncoderConfig(dim=256, n_layers=2, n_heads=4, hidden_dim=512, attn_output_dropout=0.1, vocab_size=2000)
    gen = torch.Generator().manual_seed(S * 100 + b)
    mask = _mask(kind, b, S, gen)
    ids = torch.randint(5, 2000, (b, S), generator=gen, dtype=torch.int32).cuda()
    d_emb = (torch.randn(b, 256, generator=gen) * 0.1).cuda()
    rng = StepRNG(7, torch.tensor([7], dtype=torch.int32, device="cuda"))
    outs, grads = [], []
    for pack in (True, False):
        enc = _engine(cfg, dt, pooling)
        enc.pack_tokens, enc.rows_hint = pack, hint
        for rep in range(2):        # the second pass finds the buffers as the first one left them
            if rep == 0:            # a batch that fills every row first: the packed rows behind the kept ones are stale then
                m, i = torch.ones_like(mask), torch.flip(ids, (0,))
            else:
                m, i = mask, ids
            e = enc.forward(i, m, rng, train=True)
            enc.backward(d_emb)
        outs.append(e.clone())
        grads.append(enc.g.float().clone())
        if pack:
            t = enc._acts["tmap"]
            keep = (mask != 0) | (torch.arange(S, device="cuda") == 0) | (mask != 0).any(1).logical_not()[:, None]
            n = int(keep.sum())
            assert t.meta.tolist()[:3] == [n, min(b * S, (n + 63) // 64 * 64), 0]
            assert torch.equal(t.tok[:n].long(), keep.flatten().nonzero().flatten())
            assert torch.equal(t.slot[: b * S].view(b, S) >= 0, keep)
    cu.check_status()
    # no sum over features or keys changes its order or loses a non-zero term: the forward pass agrees to the bit
    assert torch.equal(outs[0], outs[1])
    assert torch.isfinite(grads[0]).all()
    for name, slot in enc.slots.items():
        x, y = (g[slot.offset: slot.offset + slot.numel] for g in grads)
        # sums over tokens are fp32 in another order and are rounded to 16 bits once: one ulp (2^-8 of the value in bf16)
        # and fp32 noise at the scale of the largest; the embedding tables are summed by 16-bit atomics in any order
        scale = float(y.abs().max().clamp_min(1e-6))
        tol = 2.0 ** -7 * y.abs() + (3e-2 if name.startswith("embeddings") else 1e-4) * scale
        assert bool(((x - y).abs() <= tol).all()), (name, float((x - y).abs().max()), scale)


def test_embed_eval_graph_equals_the_eager_pass():
    """Several shapes, new batches of a shape after its capture, more shapes than graphs are kept, weights changed in between."""
    from types import SimpleNamespace

    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.parallel.dist import DistContext
    from renee_b200.train import EMBED_GRAPHS, TrainConfig, XCTrainer
    from renee_b200.utils.sharding import shard_labels
    dev = torch.device("cuda", 0)
    enc = EncoderConfig(dim=128, n_layers=2, n_heads=2, hidden_dim=256, vocab_size=500)
    cfg = TrainConfig(batch_size=40, epochs=1, maxlen=24, pooling="mean", fp16xfc=True, noloss=True)
    tr = XCTrainer(cfg, enc, shard_labels(512, 1), DistContext(device=dev), steps_per_epoch=4)
    gen = torch.Generator().manual_seed(5)
    kept = []
    for rep in range(4):
        for b in list(range(40, 40 - EMBED_GRAPHS - 2, -1)):
            mask = _mask("prefix", b, 24, gen).cpu()
            ids = torch.randint(5, 500, (b, 24), generator=gen, dtype=torch.int32) * mask
            got = tr.embed_eval(SimpleNamespace(input_ids=ids, attention_mask=mask))
            kept.append((got, got.clone()))
            want = tr.encoder.forward(ids.cuda(), mask.cuda(), tr.step_rng, train=False).to(got.dtype)
            assert torch.equal(got, want)
        tr.encoder.p16.mul_(1.01)
    assert len(tr._embed_graphs) == EMBED_GRAPHS and all(g["graph"] is not None for g in tr._embed_graphs.values())
    assert all(torch.equal(a, c) for a, c in kept)         # a result is not overwritten by later batches
