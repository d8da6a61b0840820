"""A step's inputs in one launch from page-locked memory, and the calls that go back to single copies."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,offset", [((1, 3, 5, 0), 0), ((4096, 4096, 1, 7), 0), ((100003, 17, 64, 63), 1), ((8, 8), 3)])
def test_staged_arrays_arrive_whole(sizes, offset):
    from renee_b200.ops import cuda as cu
    gen = torch.Generator().manual_seed(sum(sizes))
    pairs, want, around = [], [], []
    for n in sizes:
        host = torch.randint(-2 ** 31, 2 ** 31 - 1, (n + offset,), generator=gen, dtype=torch.int64).int().pin_memory()[offset:]
        dev = torch.full((n + 8,), 7, dtype=torch.int32, device="cuda")
        pairs.append((host, dev[4: 4 + n]))
        around.append(dev)
        want.append(host.clone())
    hp_host, hp = torch.arange(8, dtype=torch.float32) + 0.5, torch.zeros(16, device="cuda")
    nnz = torch.zeros(2, dtype=torch.int32, device="cuda")
    assert cu.stage_inputs(pairs, hp_host, hp, 123, nnz)
    torch.cuda.synchronize()
    for (_, dev), w, a in zip(pairs, want, around):
        assert torch.equal(dev.cpu(), w)
        assert bool((a[:4] == 7).all()) and bool((a[-4:] == 7).all())
    assert hp.tolist() == hp_host.tolist() + [0.0] * 8 and nnz.tolist() == [123, 0]


def test_other_memory_is_left_to_single_copies():
    from renee_b200.ops import cuda as cu
    dev = torch.zeros(4, 6, dtype=torch.int32, device="cuda")
    pinned = torch.ones(4, 6, dtype=torch.int32).pin_memory()
    for host in (torch.ones(4, 6, dtype=torch.int32), pinned.long().pin_memory(), pinned.t(), pinned[:, :3], dev):
        assert not cu.stage_inputs([(host, dev)])
    assert not dev.any()


def test_steps_from_batches_that_are_dropped_at_once():
    """Page-locked batches of which only the trainer keeps hold give the weights that kept, pageable ones give."""
    import numpy as np
    from renee_b200.data import xcrepo
    from renee_b200.data.collate import XCCollator
    from renee_b200.data.synthetic import SyntheticSpec, SyntheticXC
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.parallel.dist import DistContext
    from renee_b200.train import TrainConfig, XCTrainer
    from renee_b200.utils.sharding import shard_labels
    enc, L, B, S = EncoderConfig(dim=128, n_layers=1, n_heads=2, hidden_dim=256, vocab_size=3000), 700, 12, 10
    sh = shard_labels(L, 1)
    spec = SyntheticSpec(num_labels=L, seq_len=S, len_lo=2, len_hi=S, vocab=3000, poisson_lam=2.0, seed=0)
    data = xcrepo.InMemoryDataset(*SyntheticXC(spec).rows(np.arange(8 * B)))
    out = []
    for pin in (False, True):
        cfg = TrainConfig(batch_size=B, epochs=1, seed=0, dropout=0.5, lr1=0.05, lr2=1e-3, warmup=10, wd1=1e-4, noloss=True,
                          fp16xfc=True, maxlen=S, pooling="cls")
        tr = XCTrainer(cfg, enc, sh, DistContext(device=torch.device("cuda", 0)), steps_per_epoch=8)
        col = XCCollator(sh, data, 0, 1, B, True)
        for k in range(8):
            batch = col(np.arange(k * B, (k + 1) * B))
            tr.train_step(batch.pin() if pin else batch)
            del batch
            if pin:
                torch.full((64 * 1024,), -1, dtype=torch.int32).pin_memory()      # takes page-locked memory that is free
        torch.cuda.synchronize()
        out.append((tr.xfc.W.clone(), tr.encoder.p32.clone()))
    # the steps are the same; the embedding gradients are summed by 16-bit atomics in any order
    for a, b in zip(*out):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2.0 ** -9


def _trainer(cuda_graph=True, B=12, S=10):
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.parallel.dist import DistContext
    from renee_b200.train import TrainConfig, XCTrainer
    from renee_b200.utils.sharding import shard_labels
    enc = EncoderConfig(dim=128, n_layers=1, n_heads=2, hidden_dim=256, vocab_size=3000)
    cfg = TrainConfig(batch_size=B, epochs=1, seed=0, dropout=0.5, lr1=0.05, lr2=1e-3, warmup=10, wd1=1e-4, noloss=True,
                      fp16xfc=True, maxlen=S, pooling="cls", cuda_graph=cuda_graph)
    return XCTrainer(cfg, enc, shard_labels(700, 1), DistContext(device=torch.device("cuda", 0)), steps_per_epoch=8)


def test_an_embedding_outlives_its_trainer():
    """The trainer and the batch are dropped while the launch that reads the batch is still queued, and their page-locked memory is
    handed out again at once."""
    import gc
    import weakref
    from types import SimpleNamespace
    gen = torch.Generator().manual_seed(2)
    ids, mask = torch.randint(5, 3000, (12, 10), generator=gen, dtype=torch.int32), torch.ones(12, 10, dtype=torch.int32)
    mask[:, 7:] = 0

    def pinned():
        return SimpleNamespace(input_ids=ids.clone().pin_memory(), attention_mask=mask.clone().pin_memory())
    tr = _trainer()
    for _ in range(3):                                     # eager, captured, staged
        want = tr.embed_eval(pinned())
    batch = pinned()
    torch.cuda.synchronize()
    torch.cuda._sleep(200_000_000)                         # some 0.1 s
    got = tr.embed_eval(batch)
    gone = weakref.ref(tr)
    del tr, batch
    gc.collect()
    assert gone() is None
    taken = [torch.full((12, 10), 7, dtype=torch.int32).pin_memory() for _ in range(16)]
    torch.cuda.synchronize()
    assert torch.equal(got, want) and len(taken) == 16


def test_training_step_in_a_graph_of_the_callers():
    """``cuda_graph=False`` leaves capturing to the caller: a captured step and an eager one behind it, against eager steps."""
    import numpy as np
    from renee_b200.data import xcrepo
    from renee_b200.data.collate import XCCollator
    from renee_b200.data.synthetic import SyntheticSpec, SyntheticXC
    from renee_b200.utils.sharding import shard_labels
    spec = SyntheticSpec(num_labels=700, seq_len=10, len_lo=2, len_hi=10, vocab=3000, poisson_lam=2.0, seed=0)
    data = xcrepo.InMemoryDataset(*SyntheticXC(spec).rows(np.arange(12)))
    batch = XCCollator(shard_labels(700, 1), data, 0, 1, 12, True)(np.arange(12)).pin()
    out = []
    for capture in (False, True):
        tr = _trainer(cuda_graph=False)
        for _ in range(3):
            tr.train_step(batch)
        if capture:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                tr.train_step(batch)
            graph.replay()
        else:
            tr.train_step(batch)
        tr.train_step(batch)
        torch.cuda.synchronize()
        out.append((tr.xfc.W.clone(), tr.encoder.p32.clone()))
    # the steps are the same; the embedding gradients are summed by 16-bit atomics in any order
    for a, b in zip(*out):
        assert float((a.float() - b.float()).norm() / b.float().norm()) < 2.0 ** -9


def test_steps_beside_a_capture_of_another_thread():
    """A thread that captures in the default mode forbids every thread a query of an event; a step on pinned batches needs none."""
    import threading
    import numpy as np
    from renee_b200.data import xcrepo
    from renee_b200.data.collate import XCCollator
    from renee_b200.data.synthetic import SyntheticSpec, SyntheticXC
    from renee_b200.utils.sharding import shard_labels
    spec = SyntheticSpec(num_labels=700, seq_len=10, len_lo=2, len_hi=10, vocab=3000, poisson_lam=2.0, seed=0)
    data = xcrepo.InMemoryDataset(*SyntheticXC(spec).rows(np.arange(12)))
    batch = XCCollator(shard_labels(700, 1), data, 0, 1, 12, True)(np.arange(12)).pin()
    tr = _trainer()
    for _ in range(6):
        tr.train_step(batch)
        tr.embed_eval(batch)
    torch.cuda.synchronize()
    raised = []

    def steps():
        try:
            for _ in range(3):
                tr.train_step(batch)
        except Exception as exc:
            raised.append(exc)
    x, graph = torch.zeros(8, device="cuda"), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.add_(1.0)
        thread = threading.Thread(target=steps)
        thread.start()
        thread.join()
    assert not raised
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 8 and tr.count == 9
