"""The grouped weight-gradient launch against fp32 products: runs that end inside tiles, ragged edges, device-side row counts."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu

LAYER = [(2304, 768), (768, 768), (3072, 768), (768, 3072)]


@pytest.mark.parametrize("T,shapes", [
    (4864, LAYER), (8192, LAYER), (64, LAYER), (1, LAYER), (100, LAYER), (513, [(384, 128), (128, 128), (512, 128), (128, 512)]),
    (16384, [(384, 128), (128, 128), (512, 128), (128, 512)]), (1000, [(264, 520)]), (3000, [(8, 8), (72, 1024), (256, 256)]),
    (6400, [(1152, 384), (384, 384), (1536, 384), (384, 1536)]), (700, [(768, 768)]),
])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16])
def test_group_equals_products(T, shapes, dt):
    from renee_b200.ops import cuda as cu
    gen = torch.Generator(device="cuda").manual_seed(T)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda", dtype=torch.float32).to(dt)
    group = cu.WgradGroup(shapes, torch.device("cuda", 0))
    group.scratch.fill_(float("nan"))            # the scratch needs no initial value
    for rows in {T, max(1, T - 37), (T + 1) // 2}:
        items = [(r(T, m) * 0.1, r(T, n), torch.full((m, n), 7.0, dtype=dt, device="cuda")) for m, n in shapes]
        tmap = None
        if rows != T:                            # packed rows: multiples of 64 (or all), what lies behind is not read
            rows = min(T, (rows + 63) // 64 * 64)
            tmap = cu.TokenMap(1, T, "cuda")
            tmap.meta[1] = rows
            for dy, x, _ in items:
                dy[rows:] = float("nan")
                x[rows:] = float("nan")
        for _ in range(2):
            cu.wgrad_group(items, group, tmap=tmap)
        cu.check_status()
        assert int(group.counters.abs().max()) == 0
        for dy, x, dW in items:
            want = dy[:rows].float().t() @ x[:rows].float()
            # fp32 accumulation, one rounding to 16 bits: relative 2^-9 (bf16) or 2^-12 on average
            rel = float((dW.float() - want).norm() / want.norm())
            assert rel < (4e-3 if dt == torch.bfloat16 else 1e-3), rel
            assert float((dW.float() - want).abs().max()) <= 2.0 ** -7 * float(want.abs().max())
