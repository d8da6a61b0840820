"""Stochastic rounding of the fp16 classifier weights: every element draws its noise from the hash of its own number."""
import numpy as np
import pytest
import torch

from renee_b200.ops import reference as ref

SR_STREAM = 0x5152


def _mix32(seed, stream, idx):
    """The counter-based hash, restated in numpy."""
    x = np.asarray(idx, dtype=np.uint32)
    with np.errstate(over="ignore"):
        x = x * np.uint32(0x9E3779B1) + np.uint32(seed)
        x ^= x >> np.uint32(16); x *= np.uint32(0x85EBCA6B); x ^= x >> np.uint32(13); x *= np.uint32(0xC2B2AE35); x ^= x >> np.uint32(16)
        x += np.uint32((stream * 0x27D4EB2F) & 0xFFFFFFFF)
        x ^= x >> np.uint32(15); x *= np.uint32(0x2C1B3C6D); x ^= x >> np.uint32(12); x *= np.uint32(0x297A2D39); x ^= x >> np.uint32(15)
    return x


def _expected(w, seed, dtype=np.float16):
    """fp32 ``w`` (numpy) with 13 bits of noise per element, cut to fp16's mantissa."""
    noise = _mix32(seed, SR_STREAM, np.arange(w.size)).reshape(w.shape) & np.uint32(0x1FFF)
    with np.errstate(over="ignore"):
        bits = (w.view(np.uint32) + noise) & np.uint32(0xFFFFE000)
    return bits.view(np.float32).astype(dtype)


def _truncate_subnormal(w):
    """To fp16 as the kernels do it: exact in the normal range, towards zero below it (steps of 2^-24)."""
    return np.where(np.abs(w) < 2.0 ** -14, np.trunc(w * 2.0 ** 24) * 2.0 ** -24, w).astype(np.float16)


@pytest.mark.parametrize("n", [1, 2, 7, 4096])
def test_oracle_noise_is_the_hash_of_the_element(n):
    w = np.random.default_rng(n).standard_normal(n).astype(np.float32) * 0.03
    got = ref.stochastic_round_fp16(torch.from_numpy(w), 12345)
    np.testing.assert_array_equal(got.numpy().view(np.uint16), _expected(w, 12345).view(np.uint16))


@pytest.mark.gpu
@pytest.mark.parametrize("v2", [False, True])
@pytest.mark.parametrize("Lc,D", [(128, 64), (130, 128), (517, 768)])
def test_kernels_round_with_the_oracles_noise(Lc, D, v2):
    from renee_b200.ops import cuda as cu
    from renee_b200.optim.hparams import HyperParams
    dev, B, lr, seed = torch.device("cuda"), 64, 3e-3, 987654321
    g = torch.Generator(device=dev).manual_seed(Lc)
    W = (torch.randn(Lc, D, generator=g, device=dev) * 0.03).half()
    M = torch.randn(Lc, D, generator=g, device=dev).half()
    X = torch.randn(B, D, generator=g, device=dev).half()
    Gt = torch.zeros(Lc, B, dtype=torch.float16, device=dev)
    hp = HyperParams(dev)
    hp.set_step(lr, 0.0, seed)
    hp.upload()
    # no gradient, no decay: m stays, w becomes w - lr m with one fp32 rounding (fp16 factors: exact in fp64 up to then)
    want = (W.double() - float(np.float32(lr)) * M.double()).float()
    want = _truncate_subnormal(_expected(want.cpu().numpy(), seed, np.float32))
    M0 = M.clone()
    cu.xfc_dw_sgd(Gt, B, X, W, M, hp.buf, 1.0, 0.0, stochastic_round=True, v2=v2)
    cu.check_status()
    assert torch.equal(M, M0)
    np.testing.assert_array_equal(W.cpu().numpy(), want)
