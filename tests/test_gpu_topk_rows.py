"""Fused top-k where every row of the batch has its own scores: lanes of a warp insert at different columns, and for large k
rows recompute different lists, often more labels than fit beside the candidates at once."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("B,D,L,k", [(40, 64, 20000, 5), (257, 64, 9000, 256), (129, 128, 1000, 256), (200, 64, 60000, 200),
                                     (600, 192, 5003, 8), (31, 64, 300, 17)])
@pytest.mark.parametrize("order", ["random", "clustered"])
def test_rows_with_scores_of_their_own(B, D, L, k, order, dt):
    from renee_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(L + k)
    # small integers: every score is an exact fp32 sum in any order
    W = torch.randint(-3, 4, (L, D), generator=g, device="cuda").to(dt)
    X = torch.randint(-3, 4, (B, D), generator=g, device="cuda").to(dt)
    if order == "clustered":            # the labels that most rows score best stand together
        mean = X.float().mean(0)
        W = W[torch.argsort(W.float() @ mean)].contiguous()
    v, i = cu.xfc_topk8(W, X, k)
    cu.check_status()
    Z = X.float() @ W.float().t()
    want = torch.topk(Z, k, dim=1)[0]
    assert torch.equal(v, want)
    assert torch.equal(torch.gather(Z, 1, i), want)
    assert all(len(set(r)) == k for r in i.tolist())


@pytest.mark.parametrize("k", [1, 5, 30, 200])
def test_nan_ranks_above_infinity(k):
    from renee_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(k)
    W = torch.randint(-3, 4, (4000, 64), generator=g, device="cuda").half()
    X = torch.randint(1, 4, (70, 64), generator=g, device="cuda").half()
    W[[11, 12, 13, 2500], 7] = float("inf")
    W[[14, 3999], 9] = float("nan")
    W[100:120, 3] = float("-inf")
    v, i = cu.xfc_topk8(W, X, k)
    cu.check_status()
    Z = X.float() @ W.float().t()
    want = torch.topk(Z, k, dim=1)[0]              # NaN first, then +inf
    assert torch.equal(torch.isnan(v), torch.isnan(want))
    assert torch.equal(v.nan_to_num(nan=0.0, posinf=1e9), want.nan_to_num(nan=0.0, posinf=1e9))
    assert torch.equal(torch.gather(Z, 1, i).nan_to_num(nan=0.0, posinf=1e9), want.nan_to_num(nan=0.0, posinf=1e9))
