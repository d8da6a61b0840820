"""Logit gradients where a few labels have most of the positives, or all of them, against fp32 matmul + sigmoid."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Lc,B,D", [(130, 64, 64), (700, 200, 64), (700, 90, 128), (3000, 520, 64), (40000, 256, 64)])
@pytest.mark.parametrize("heavy", [(0,), (31, 32, 33), (5, 64, 129)])
def test_logit_gradient_with_heavy_labels(Lc, B, D, heavy):
    from renee_b200.ops import cuda as cu
    gen = torch.Generator().manual_seed(Lc + B + len(heavy))
    W, X = (torch.randn(Lc, D, generator=gen) * 0.05).half(), torch.randn(B, D, generator=gen).half()
    Y = torch.rand(Lc, B, generator=gen) < 2.0 / Lc              # sparse ones everywhere
    for l in heavy:
        Y[l] = True                                              # every row has these labels
    labels, rows = Y.nonzero(as_tuple=True)
    shuffled = torch.argsort(labels * B + torch.randperm(B, generator=gen)[rows])     # sorted by label, rows in any order
    labels, rows = labels[shuffled].int().cuda(), rows[shuffled].int().cuda()
    ldG = (B + 7) // 8 * 8
    Gt = torch.full((Lc, ldG), 9.0, dtype=torch.float16, device="cuda")
    nnz = torch.tensor([labels.numel()], dtype=torch.int32, device="cuda")
    label0 = 1000
    cu.xfc_logits_grad_v2(W.cuda(), X.cuda(), Gt, ldG, rows, labels + label0, nnz, label0)
    cu.check_status()
    want = torch.sigmoid(W.float() @ X.float().t())
    # sigmoid in 16 bits (2^-11), minus 1 in 16 bits where there is a positive
    err = (Gt[:, :B].float().cpu() - (want - Y.float())).abs()
    assert float(err.max()) < 2.0 ** -10
    assert not Gt[:, B:].any()


def test_a_wait_that_runs_out_before_heavy_labels():
    """A peer whose flag never comes: the launch ends with a status although its warps have meetings ahead, and the next one is right."""
    from renee_b200.ops import cuda as cu
    gen = torch.Generator().manual_seed(1)
    Lc, B, D = 3000, 200, 64
    W, X = (torch.randn(Lc, D, generator=gen) * 0.05).half(), torch.randn(B, D, generator=gen).half()
    labels, rows = (torch.rand(Lc, B, generator=gen) < 0.5).nonzero(as_tuple=True)         # 3200 positives per 32 labels
    Gt = torch.empty(Lc, B, dtype=torch.float16, device="cuda")
    nnz = torch.tensor([labels.numel()], dtype=torch.int32, device="cuda")
    flags, step = (torch.full((1,), v, dtype=torch.int32, device="cuda") for v in (0, 1))
    args = (W.cuda(), X.cuda(), Gt, B, rows.int().cuda(), labels.int().cuda(), nnz, 0)
    cu.xfc_logits_grad_v2(*args, wait=(flags, 1, step))
    with pytest.raises(cu.KernelError, match="timed out"):
        cu.check_status()
    cu.xfc_logits_grad_v2(*args, wait=(step, 1, step))
    cu.check_status()
    want = torch.sigmoid(W.float() @ X.float().t())
    want[labels, rows] -= 1.0
    assert float((Gt.float().cpu() - want).abs().max()) < 2.0 ** -10          # two roundings to 16 bits, as above
