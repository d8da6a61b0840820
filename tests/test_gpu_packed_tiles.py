"""Packed rows at sizes where the persistent GEMMs give a unit several tiles: each layer op on its own against the padded rows."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _map(b, S, len_lo, seed):
    """A token map and the kept positions (padded index per packed row) of lengths uniform in len_lo..S."""
    from renee_b200.ops import cuda as cu
    g = torch.Generator().manual_seed(seed)
    lens = torch.randint(len_lo, S + 1, (b,), generator=g)
    mask = (torch.arange(S)[None] < lens[:, None]).to(torch.int32)
    tmap = cu.TokenMap(b, S, "cuda")
    tmap.update(mask.cuda())
    kept = mask.flatten().nonzero().flatten().cuda()
    tmap.tok[: len(kept)] = kept.to(torch.int32)
    rows = int(tmap.meta[1])
    tmap.tok[len(kept): rows] = -1
    return tmap, kept, rows


@pytest.mark.parametrize("hint", [0, 1, 0.6])
@pytest.mark.parametrize("b,S,len_lo,K,N,dt", [
    (640, 32, 6, 256, 768, torch.bfloat16),       # 80 M tiles of 256 rows at most, 48 kept, 3 N tiles: two tiles per SM pair
    (1024, 32, 31, 128, 1024, torch.float16),     # 128 x 4 tiles, nearly all kept: up to seven per pair
    (64, 256, 64, 768, 3072, torch.bfloat16),     # 40 x 12
    (333, 32, 1, 192, 448, torch.bfloat16)])      # ragged in both directions
def test_packed_gemms_with_several_tiles_per_unit(b, S, len_lo, K, N, dt, hint):
    from renee_b200.ops import StepRNG, cuda as cu
    tmap, kept, rows = _map(b, S, len_lo, b + K)
    tmap.rows_hint = hint if hint in (0, 1) else int(hint * b * S)
    T, n = b * S, len(kept)
    g = torch.Generator(device="cuda").manual_seed(N)
    r = lambda *s, sc=1.0: (torch.randn(*s, generator=g, device="cuda") * sc).to(dt)
    rng = StepRNG(7, torch.tensor([7], dtype=torch.int32, device="cuda"))
    x, W, bias, res, dy = r(T, K), r(N, K, sc=K ** -0.5), r(N), r(T, N), r(T, N)

    def pack(t):                                   # capacity as the padded rows have it; what lies behind the rows is NaN
        p = torch.full_like(t, float("nan"))
        p[:n], p[n:rows] = t[kept], 0
        return p

    def both(run):
        """run(rows of x / dy, residual, token map) on the padded and on the packed rows."""
        want, got = run(lambda t: t, None), run(pack, tmap)
        cu.check_status()
        for w, p in zip(want, got):
            assert torch.equal(p[:n], w[kept])     # the same products in the same order, and the same dropout decisions
            assert bool(torch.isfinite(p[:rows].float()).all())

    new = lambda *s: torch.full(s, 7.0, dtype=dt, device="cuda")

    def fwd(epi, **kw):
        def run(at, tm):
            out, pre = new(T, N), new(T, N)
            args = dict(bias=bias) if epi != "store" else {}
            if epi == "bias_gelu":
                args["pre_out"] = pre
            if epi == "bias_dropout_resid":
                args.update(resid=at(res), p=0.1, rng=rng, stream=11)
            cu.linear_fwd(at(x), W, out, epi, tmap=tm, **args)
            return (out, pre) if epi == "bias_gelu" else (out,)
        return run

    for epi in ("store", "bias_gelu", "bias_dropout_resid"):
        both(fwd(epi))
    f, dres = r(T, K), r(T, K)
    both(lambda at, tm: (cu.linear_dgrad(at(dy), W, new(T, K), "add", resid=at(dres), tmap=tm),))
    cols = []

    def gelu_bwd(at, tm):
        db = new(K)
        rows_dy = torch.zeros_like(dy)
        rows_dy[kept] = dy[kept]                   # padded rows have no gradient
        out = cu.linear_dgrad(at(rows_dy), W, new(T, K), "gelu_bwd", pre=at(f), dbias=db, tmap=tm)
        cols.append(db.float())
        return (out,)

    both(gelu_bwd)
    # fp32 sums of the same rounded values in another order, rounded once: one ulp and fp32 noise at the largest sum's scale
    eps = 2.0 ** -7 if dt == torch.bfloat16 else 2.0 ** -10
    assert bool(((cols[0] - cols[1]).abs() <= eps * cols[0].abs() + 1e-4 * cols[0].abs().max()).all())
