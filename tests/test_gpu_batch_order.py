"""What a batch gives does not depend on which batch of its shape a trainer met first."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _trainer(dim, B, S, pooling):
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.parallel.dist import DistContext
    from renee_b200.train import TrainConfig, XCTrainer
    from renee_b200.utils.sharding import shard_labels
    enc = EncoderConfig(dim=dim, n_layers=2, n_heads=dim // 64, hidden_dim=2 * dim, vocab_size=2000)
    cfg = TrainConfig(batch_size=B, epochs=1, maxlen=S, pooling=pooling, fp16xfc=True, noloss=True, dropout=0.5)
    return XCTrainer(cfg, enc, shard_labels(512, 1), DistContext(device=torch.device("cuda", 0)), steps_per_epoch=4)


def _batch(B, S, lens, seed):
    from renee_b200.data import xcrepo
    from renee_b200.data.collate import XCCollator
    from renee_b200.data.synthetic import SyntheticSpec, SyntheticXC
    from renee_b200.utils.sharding import shard_labels
    spec = SyntheticSpec(num_labels=512, seq_len=S, len_lo=lens[0], len_hi=lens[1], vocab=2000, poisson_lam=2.0, seed=seed)
    data = xcrepo.InMemoryDataset(*SyntheticXC(spec).rows(np.arange(B)))
    return XCCollator(shard_labels(512, 1), data, 0, 1, B, True)(np.arange(B))


@pytest.mark.parametrize("dim,B,S,pooling", [(256, 128, 32, "mean"), (256, 40, 150, "cls"), (128, 96, 32, "mean"), (256, 256, 32, "mean")])
def test_first_batch_does_not_choose_the_path(dim, B, S, pooling):
    short, full, typical = (_batch(B, S, l, k) for k, l in enumerate([(2, 3), (S, S), (S // 4, S)]))
    outs = []
    for first in (short, full):
        tr = _trainer(dim, B, S, pooling)
        tr.embed_eval(first)
        own = tr.encoder.own_gemm
        outs.append([tr.embed_eval(typical) for _ in range(3)][-1])
        tr.train_step(typical)
        assert tr.encoder.own_gemm == own
        outs[-1] = (outs[-1], own)
    assert outs[0][1] == outs[1][1]
    assert torch.equal(outs[0][0], outs[1][0])


def test_frequent_shapes_take_the_place_of_rare_ones():
    """The shapes met first do not keep the graphs for good, shapes of like frequency do not evict one another, and every
    result is the eager one."""
    from renee_b200.train import EMBED_GRAPHS
    S, tr = 24, _trainer(128, 40, 24, "mean")
    batches = {b: _batch(b, S, (2, S), b) for b in range(40, 40 - EMBED_GRAPHS - 3, -1)}

    def ask(b):
        got = tr.embed_eval(batches[b])
        want = tr.encoder.forward(batches[b].input_ids.cuda(), batches[b].attention_mask.cuda(), tr.step_rng, train=False)
        assert torch.equal(got, want.to(got.dtype))

    for _ in range(3):
        for b in batches:
            ask(b)
    first = set(tr._embed_graphs)
    assert first == {(b, S) for b in list(batches)[:EMBED_GRAPHS]}
    late = list(batches)[-1]
    for _ in range(5):
        ask(late)
    assert (late, S) in tr._embed_graphs and len(tr._embed_graphs) == EMBED_GRAPHS
    for b in batches:
        ask(b)
    assert len(tr._embed_graphs) == EMBED_GRAPHS


def test_embed_eval_inside_a_callers_graph():
    """A caller that captures embed_eval into a graph of its own gets the eager launches, also after the shape has a graph."""
    from types import SimpleNamespace
    S, tr = 24, _trainer(128, 40, 24, "cls")
    a, b = (SimpleNamespace(**{n: getattr(x, n).to("cuda", torch.int32) for n in ("input_ids", "attention_mask")})
            for x in (_batch(40, S, (2, S), 1), _batch(40, S, (2, S), 2)))
    want = [[tr.embed_eval(x) for _ in range(3)][-1] for x in (a, b)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = tr.embed_eval(a)
    for x, w in zip((a, b), want):
        a.input_ids.copy_(x.input_ids); a.attention_mask.copy_(x.attention_mask)
        graph.replay()
        assert torch.equal(out, w)
