"""GELU and its derivative at every 16-bit number (both zeros, subnormals, the largest, infinities, NaNs), element by element against
64 bits: in the GEMM epilogues and in the stand-alone kernels."""
from __future__ import annotations

import pytest
import torch

from renee_b200 import ops

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float16]


def _all_numbers(dt):
    return torch.arange(-2 ** 15, 2 ** 15, dtype=torch.int32).to(torch.int16).view(dt)


def _check(got, want):
    """One rounding to 16 bits of a value that the published approximation of erfc (1.5e-7 of 0.5 erfc, times |z| up to 6 where the
    tail is not yet smaller) and fp32 arithmetic give to 2e-6.  With p significant bits the rounding moves a value of [2^e, 2^(e+1))
    by half of its spacing 2^(e+1-p), at most 2^-p of it (p = 8 in bf16, 11 in fp16), and a subnormal by half of the smallest one."""
    got, dt = got.double().cpu(), got.dtype
    assert torch.equal(got.isnan(), want.isnan()), got[got.isnan() != want.isnan()]
    unit, tiny = (2.0 ** -8, 2.0 ** -134) if dt == torch.bfloat16 else (2.0 ** -11, 2.0 ** -25)
    inf = want.isinf()
    assert torch.equal(got[inf], want[inf])
    ok = ~(inf | want.isnan())
    over = (got[ok] - want[ok]).abs() - (unit * want[ok].abs() + tiny + 2e-6)
    assert float(over.max()) <= 0.0, (got[ok][over.argmax()], want[ok][over.argmax()])


def _derivative(z):
    z = z.double().requires_grad_(True)
    torch.nn.functional.gelu(z).sum().backward()
    return z.grad


@pytest.mark.parametrize("ncta", [1, 2])
@pytest.mark.parametrize("dt", DTYPES)
def test_derivative_in_the_gemm_epilogue(dt, ncta):
    from renee_b200.ops import cuda as cu
    T, N, z = 64, 64, _all_numbers(dt)
    f = z.cuda().expand(T, -1).contiguous()
    dy, W = torch.zeros(T, N, device="cuda", dtype=dt), torch.zeros(N, z.numel(), device="cuda", dtype=dt)
    dy[:, 0], W[0] = 1.0, 1.0                                    # a gradient of exactly 1 everywhere
    out, dbias = torch.empty_like(f), torch.empty(z.numel(), device="cuda", dtype=dt)
    cu.linear_dgrad(dy, W, out, "gelu_bwd", pre=f, dbias=dbias, ncta=ncta)
    cu.check_status()
    _check(out[0], _derivative(z))
    assert torch.equal(torch.nan_to_num(out, 9.0), torch.nan_to_num(out[:1].expand(T, -1), 9.0))
    assert torch.equal(torch.nan_to_num(dbias.float(), 9.0), torch.nan_to_num(T * out[0].float(), 9.0))    # 64 equal rows: exact


@pytest.mark.parametrize("dt", DTYPES)
def test_derivative_in_the_kernel_of_its_own(dt):
    z = _all_numbers(dt).view(16, 4096)
    x, bias = z.cuda(), torch.full((4096,), -0.0, device="cuda", dtype=dt)                               # x + -0 is x, -0 included
    dx, dbias = torch.empty_like(x), torch.empty_like(bias)
    ops.bias_gelu_bwd(torch.ones_like(x), x, bias, dbias, dx)
    _check(dx.flatten(), _derivative(z).flatten())


@pytest.mark.parametrize("ncta", [1, 2])
@pytest.mark.parametrize("dt", DTYPES)
def test_gelu_in_the_gemm_epilogue(dt, ncta):
    from renee_b200.ops import cuda as cu
    T, K, z = 64, 64, _all_numbers(dt)
    x, W = torch.zeros(T, K, device="cuda", dtype=dt), torch.zeros(z.numel(), K, device="cuda", dtype=dt)
    x[:, 0], W[:, 0] = 1.0, z.cuda()
    act, pre = (torch.empty(T, z.numel(), device="cuda", dtype=dt) for _ in range(2))
    cu.linear_fwd(x, W, act, "bias_gelu", bias=torch.zeros(z.numel(), device="cuda", dtype=dt), pre_out=pre, ncta=ncta)
    cu.check_status()
    # the stored pre-activations are these numbers (fp32 subnormals, which bf16's are, become 0 on the way)
    stored = torch.where(z.float().abs() < torch.finfo(torch.float32).tiny, 0.0, z.float())
    assert torch.equal(torch.nan_to_num(pre[0].float().cpu(), 9.0), torch.nan_to_num(stored, 9.0))
    _check(act[0], torch.nn.functional.gelu(z.double()))
    assert torch.equal(torch.nan_to_num(act, 9.0), torch.nan_to_num(act[:1].expand(T, -1), 9.0))


@pytest.mark.parametrize("dt", DTYPES)
def test_gelu_in_the_kernel_of_its_own(dt):
    z = _all_numbers(dt).view(16, 4096)
    x, out = z.cuda(), torch.empty(16, 4096, device="cuda", dtype=dt)
    ops.bias_gelu_fwd(x, torch.full((4096,), -0.0, device="cuda", dtype=dt), out)
    _check(out.flatten(), torch.nn.functional.gelu(z.double()).flatten())
