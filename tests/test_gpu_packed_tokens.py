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
    (256, 4, "prefix", "mean", torch.bfloat16), (300, 3, "prefix", "mean", torch.bfloat16), (16, 9, "prefix", "cls", torch.float16),
    (257, 2, "holes", "cls", torch.float16), (64, 5, "empty_rows", "cls", torch.bfloat16), (201, 3, "holes", "mean", torch.bfloat16), (130, 2, "empty_rows", "cls", torch.bfloat16),
])
@pytest.mark.parametrize("hint,heads", [(0, 4), (64, 8)])
def test_packed_equals_padded(S, b, kind, pooling, dt, hint, heads):
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.ops import StepRNG, cuda as cu
    cfg = EncoderConfig(dim=256, n_layers=2, n_heads=heads, hidden_dim=512, attn_output_dropout=0.1, vocab_size=2000)
    if heads == 8 and S > 128:
        pytest.skip("head dim 32 has own kernels up to 128 tokens")
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
    assert torch.isfinite(grads[0]).all()
    if S <= 128:
        # no sum over features or keys changes its order or loses a non-zero term: the forward pass agrees to the bit
        assert torch.equal(outs[0], outs[1])
    else:
        # sequences of at most 128 tokens take the smaller tile, whose fp32 row sums are in another order: a probability
        # may round to the neighbouring 16-bit value, which moves each activation by at most one rounding (2^-8 in bf16)
        assert float((outs[0] - outs[1]).norm() / outs[1].norm()) < 2.0 ** -8
    for name, slot in enc.slots.items():
        x, y = (g[slot.offset: slot.offset + slot.numel] for g in grads)
        # sums over tokens are fp32 in another order and are rounded to 16 bits once: one ulp (2^-8 of the value in bf16)
        # and fp32 noise at the scale of the largest; the embedding tables are summed by 16-bit atomics in any order
        scale = float(y.abs().max().clamp_min(1e-6))
        if S > 64:                  # other tile, other order in the softmax gradient: 16-bit roundings differ here and there
            # (the key bias has gradient zero, and what is left of it is rounding alone)
            assert float((x - y).norm()) <= 2.0 ** -7 * float(y.norm()) + 1e-6 or name.endswith("k_lin.bias"), name
            continue
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


@pytest.mark.parametrize("S,b,nh,hd,dt", [(256, 3, 2, 64, torch.bfloat16), (193, 2, 3, 64, torch.float16), (130, 2, 1, 64, torch.bfloat16),
                                          (128, 3, 4, 32, torch.float16), (65, 2, 2, 32, torch.bfloat16), (33, 2, 2, 32, torch.float16),
                                          (16, 5, 2, 64, torch.bfloat16), (9, 4, 4, 32, torch.bfloat16), (97, 2, 2, 64, torch.float16)])
@pytest.mark.parametrize("p", [0.0, 0.2])
def test_attention_tile_sizes_against_the_oracle(S, b, nh, hd, dt, p):
    """Every tile size and head dim of the register-resident kernels, masked keys included, against the fp32 oracle."""
    from renee_b200 import ops
    from renee_b200.ops import StepRNG, cuda as cu, reference as ref
    H = nh * hd
    gen = torch.Generator().manual_seed(S + hd)
    r = lambda *s: (torch.randn(*s, generator=gen) * 0.5).to(dt).cuda()
    qkv, bias, dctx = r(b * S, 3 * H), r(3 * H), r(b * S, H)
    mask = _mask("prefix", b, S, gen)
    mask[0] = 0
    rng = StepRNG(11, torch.tensor([11], dtype=torch.int32, device="cuda"))
    ws = ops.attention_workspace(b, S, nh, torch.device("cuda"), dt)
    ctx, dqkv, db = torch.empty_like(dctx), torch.empty_like(qkv), torch.empty_like(bias)
    ops.attention_fwd(qkv, bias, mask, nh, p, rng, 5, ctx, ws)
    ops.attention_bwd(dctx, qkv, bias, mask, nh, p, rng, 5, ws, dqkv, db)
    cu.check_status()
    # q, k, v after the bias are 16-bit numbers in the kernels
    q16 = (qkv.float() + bias.float()).to(dt).float()
    z = torch.zeros_like(bias).float()
    ctx_r, probs_r = ref.attention_fwd(q16, z, mask, nh, p, 11, 5)
    d_r = ref.attention_bwd(dctx.float(), q16, z, mask, probs_r, nh, p, 11, 5)
    # 16-bit probabilities, softmax gradients and results: three roundings of relative size eps each, over sums of S terms
    eps = 2.0 ** -8 if dt == torch.bfloat16 else 2.0 ** -11
    for got, want in ((ctx, ctx_r), (dqkv, d_r)):
        rel = float((got.float() - want).norm() / want.norm())
        assert rel < 3 * eps, rel
        assert float((got.float() - want).abs().max()) < 16 * eps * float(want.abs().max())
    torch.testing.assert_close(db.float(), d_r.sum(0), rtol=8 * eps, atol=8 * eps * float(d_r.sum(0).abs().max()) + 1e-3)


def test_capture_after_a_backward_pass_that_raised(monkeypatch):
    """A backward pass that ended in a host exception leaves no event behind that a later pass, or its capture, waits for."""
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.ops import StepRNG, cuda as cu
    cfg = EncoderConfig(dim=128, n_layers=3, n_heads=2, hidden_dim=256, vocab_size=500)
    enc = _engine(cfg, torch.bfloat16, "mean")
    gen = torch.Generator().manual_seed(1)
    mask = _mask("prefix", 8, 32, gen)
    ids = torch.randint(5, 500, (8, 32), generator=gen, dtype=torch.int32).cuda()
    d_emb = (torch.randn(8, 128, generator=gen) * 0.1).cuda()
    rng = StepRNG(7, torch.tensor([7], dtype=torch.int32, device="cuda"))

    def step():
        enc.forward(ids, mask, rng, train=True)
        enc.backward(d_emb)

    step()
    want = enc.g.float().clone()
    dgrad, n = cu.linear_dgrad, [0]

    def failing(*a, **k):
        n[0] += 1
        if n[0] == 5:                        # in the second layer of the pass: the first one's weight gradients are under way
            raise RuntimeError("stop")
        return dgrad(*a, **k)

    monkeypatch.setattr(cu, "linear_dgrad", failing)
    with pytest.raises(RuntimeError, match="stop"):
        step()
    monkeypatch.setattr(cu, "linear_dgrad", dgrad)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    enc.g.zero_()
    graph.replay()
    cu.check_status()
    for name, slot in enc.slots.items():     # the matrices; the column sums still hold what the failed pass had added
        if name.startswith("transformer") and name.endswith(("_lin.weight", "lin1.weight", "lin2.weight")):
            at = slice(slot.offset, slot.offset + slot.numel)
            assert torch.equal(enc.g[at].float(), want[at]), name
