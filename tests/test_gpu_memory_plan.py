"""The meta-device plan against what a trainer allocates on a GPU, on both GEMM paths and every attention regime."""
from __future__ import annotations

import numpy as np
import pytest
import torch


def _enc(S):
    from renee_b200.models.encoder import EncoderConfig
    return EncoderConfig(vocab_size=2000, dim=128, n_layers=2, n_heads=2, hidden_dim=256, max_position_embeddings=max(S, 64))


SHAPES = [(256, 32), (16, 24), (64, 160), (8, 160), (32, 300), (4, 300)]


@pytest.mark.parametrize("B,S", SHAPES)
def test_plan_has_the_buffers_of_the_path(B, S):
    from renee_b200.models import flat_encoder as fe
    from renee_b200.utils.memory_plan import plan
    p = plan(labels=3000, gpus=1, global_batch=B, seq=S, enc_cfg=_enc(S), pooling="mean")
    gb = p["per_gpu_gb"]
    own = B * S >= fe.OWN_GEMM_MIN_TOKENS
    # own: two sets of 4 H + F and 3 H columns and the 39 MB of partial tiles; library: 4 H + 2 F columns
    rows = (B + 1) * S
    scratch = 74 * 4 * 128 * 256 * 4
    bwd = rows * 2 * (2 * (5 * 128 + 256) if own else 4 * 128 + 2 * 256)
    known = sum(v for k, v in gb.items() if k in ("encoder", "encoder.activations", "attention")) * 1e9
    assert known >= bwd + (scratch if own else 0)
    ds = (B + 1) * 2 * S * S * 2
    probs = 2 * ds                                  # two layers
    att = gb.get("attention", 0) * 1e9
    assert abs(att - probs - (ds if S > 256 else 0)) < 1e6


@pytest.mark.gpu
@pytest.mark.parametrize("B,S", SHAPES)
def test_plan_is_what_a_trainer_allocates(B, S):
    from renee_b200.data import xcrepo
    from renee_b200.data.collate import XCCollator
    from renee_b200.data.synthetic import SyntheticSpec, SyntheticXC
    from renee_b200.ops import cuda as cu
    from renee_b200.parallel.dist import DistContext
    from renee_b200.train import TrainConfig, XCTrainer
    from renee_b200.utils import guard
    from renee_b200.utils.memory_plan import plan
    from renee_b200.utils.sharding import shard_labels
    L = 3000
    want = plan(labels=L, gpus=1, global_batch=B, seq=S, enc_cfg=_enc(S), pooling="mean")["framework_total_bytes"]
    data = xcrepo.InMemoryDataset(*SyntheticXC(SyntheticSpec(num_labels=L, seq_len=S, len_lo=4, len_hi=S, vocab=2000,
                                                             poisson_lam=2.0, seed=1)).rows(np.arange(B)))
    batch = XCCollator(shard_labels(L, 1), data, 0, 1, B, True)(np.arange(B))
    cfg = TrainConfig(batch_size=B, epochs=1, seed=0, dropout=0.5, lr1=0.05, lr2=1e-5, warmup=10, wd1=1e-4, noloss=True,
                      fp16xfc=True, maxlen=S, pooling="mean")
    with guard.enabled_for_test():
        tr = XCTrainer(cfg, _enc(S), shard_labels(L, 1), DistContext(device=torch.device("cuda", 0)), steps_per_epoch=10)
        tr.encoder.allocate(B, S, capacity=B + 1)
        for _ in range(4):                          # eager passes, then a graph: nothing beyond the plan
            tr.train_step(batch)
        torch.cuda.synchronize()
        guard.assert_clean()
        cu.check_status()
        assert sum(e.hi - e.lo for e in guard._registry) == want
