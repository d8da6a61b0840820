"""Fused top-k (GEMM candidates + row selection) against exact scores, for label orders that crowd the best into few lists."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _weights(scores, D, dt=torch.float16):
    """W [L, D], x [D] with x . W[l] == scores[l] exactly (integers below 2^21 as two fp16 integers)."""
    W = torch.zeros(len(scores), D, dtype=dt)
    s = torch.as_tensor(scores, dtype=torch.int64)
    W[:, 3] = (s // 1024).to(dt)
    W[:, D - 1] = (s % 1024).to(dt)
    x = torch.zeros(D, dtype=dt)
    x[3], x[D - 1] = 1024.0, 1.0
    return W.cuda(), x.cuda()


def _scores(order, L, rng):
    if order == "ascending":
        return np.arange(L)
    if order == "descending":
        return np.arange(L)[::-1].copy()
    if order == "block":            # the best share one run of labels, so one or a few lists see all of them
        s = rng.permutation(L)
        a = L // 3
        w = min(300, L - a)
        top = np.sort(s)[-w:]
        rest = np.setdiff1d(s, top, assume_unique=True)
        return np.concatenate([rest[:a], rng.permutation(top), rest[a:]])
    if order == "ties":
        return rng.permutation(L) // 7
    return rng.permutation(L)


@pytest.mark.parametrize("B,D,L,k", [(300, 64, 40000, 100), (33, 128, 1000, 256), (513, 64, 20011, 10), (1, 768, 130, 100),
                                     (700, 64, 9000, 1), (128, 64, 70000, 9), (5, 64, 100, 100)])
@pytest.mark.parametrize("order", ["random", "ascending", "descending", "block", "ties"])
def test_topk_is_exact_for_any_label_order(B, D, L, k, order):
    from renee_b200.ops import cuda as cu
    rng = np.random.default_rng(L + k)
    s = _scores(order, L, rng)
    W, x = _weights(s, D)
    X = x[None].repeat(B, 1)
    X[B // 2] = 0                       # a row of equal logits: any labels are right, each once
    v, i = cu.xfc_topk8(W, X, k)
    cu.check_status()
    want = np.sort(s)[::-1][:k].astype(np.float32)
    v, i = v.cpu().numpy(), i.cpu().numpy()
    assert i.min() >= 0 and i.max() < L
    for b in range(B):
        assert len(set(i[b])) == k
        if b == B // 2:
            assert (v[b] == 0).all()
            continue
        np.testing.assert_array_equal(v[b], want)
        np.testing.assert_array_equal(s[i[b]], want)


def test_topk_through_the_classifier_and_non_finite_logits():
    """XFCClassifier.topk for every k up to the limit of the fused path and beyond it; -inf and NaN logits rank as in torch.topk."""
    from renee_b200.models.xfc import XFCClassifier
    torch.manual_seed(1)
    xfc = XFCClassifier(3000, 128, torch.device("cuda"), True)
    X = (torch.randn(40, 128, device="cuda")).half()
    Z = X.float() @ xfc.W.float().t()
    for k in (1, 8, 9, 100, 256, 257, 3000, 5000):
        v, i = xfc.topk(X, k)
        kk = min(k, 3000)
        # fp32 sums of the same products in another order: 128 terms, each of the size of the result
        torch.testing.assert_close(v, torch.topk(Z, kk, dim=1)[0], rtol=1e-5, atol=1e-5)
        torch.testing.assert_close(torch.gather(Z, 1, i), v, rtol=1e-5, atol=1e-5)
    X = X.abs()
    xfc.W.abs_()
    xfc.W[:2950, 5] = float("-inf")     # fewer finite logits than k
    xfc.W[17, 5] = float("nan")
    v, i = xfc.topk(X, 100)
    assert bool(torch.isnan(v[:, 0]).all()) and bool((i[:, 0] == 17).all())
    assert bool(torch.isfinite(v[:, 1:51]).all()) and bool((i[:, 1:51] >= 2950).all())
    assert bool((v[:, 51:] == float("-inf")).all())
    assert all(len(set(r.tolist())) == 100 for r in i.cpu())
