"""Non-finite logits stay where they are: a NaN embedding in its own batch column, infinities at the ends of the sigmoid."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,L,D", [(64, 300, 64), (90, 1000, 128), (7, 130, 64)])
@pytest.mark.parametrize("bad", [0, 5, 6])
def test_nan_row_of_the_batch_keeps_its_neighbours(B, L, D, bad):
    from renee_b200.ops import cuda as cu
    g = torch.Generator(device="cuda").manual_seed(B)
    W = (torch.randn(L, D, generator=g, device="cuda") * 0.05).half()
    X = torch.randn(B, D, generator=g, device="cuda").half()
    W[3] = 1000.0                                  # logits of some thousands either way
    zero = torch.zeros(1, dtype=torch.int32, device="cuda")
    ld = (B + 7) // 8 * 8
    clean, got = (torch.empty(L, ld, dtype=torch.float16, device="cuda") for _ in range(2))
    cu.xfc_logits_grad_v2(W, X, clean, ld, zero, zero, zero, 0)
    X[bad] = float("nan")
    cu.xfc_logits_grad_v2(W, X, got, ld, zero, zero, zero, 0)
    cu.check_status()
    others = [c for c in range(B) if c != bad]
    assert bool(torch.isnan(got[:, bad]).all())
    # a pair with a NaN takes the two reciprocals apart: each may round the other way in its last fp16 bit
    torch.testing.assert_close(got[:, others].float(), clean[:, others].float(), rtol=2.0 ** -10, atol=2.0 ** -24)
    assert bool((got[:, B:] == 0).all())
    want = torch.sigmoid(X.float() @ W.float().t()).t()
    torch.testing.assert_close(got[:, others].float(), want[:, others], rtol=2.0 ** -9, atol=1e-6)
