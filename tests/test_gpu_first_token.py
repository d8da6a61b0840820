"""CLS pooling: the last layer on first tokens only against the same layer on all tokens."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,b,heads,dt", [(1, 3, 4, torch.bfloat16), (16, 9, 8, torch.float16), (17, 130, 4, torch.bfloat16),
                                          (33, 5, 4, torch.float16), (65, 4, 8, torch.bfloat16), (128, 70, 4, torch.bfloat16),
                                          (129, 3, 4, torch.bfloat16), (256, 2, 4, torch.float16)])
@pytest.mark.parametrize("layers,p,po", [(1, 0.0, 0.0), (3, 0.1, 0.1), (2, 0.1, 0.0)])
def test_first_tokens_only_equals_all_tokens(monkeypatch, S, b, heads, dt, layers, p, po):
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.models.flat_encoder import FlatEncoder
    from renee_b200.ops import StepRNG, cuda as cu
    monkeypatch.setenv("RENEE_B200_OWN_GEMM", "1")
    cfg = EncoderConfig(dim=256, n_layers=layers, n_heads=heads, hidden_dim=512, dropout=p, attention_dropout=p,
                        attn_output_dropout=po, vocab_size=2000)
    gen = torch.Generator().manual_seed(S * 10 + b)
    mask = (torch.rand(b, S, generator=gen) < 0.6).to(torch.int32)
    mask[b // 2] = 0                                   # gaps, a masked first token, a wholly masked row
    mask = mask.cuda()
    ids = torch.randint(5, 2000, (b, S), generator=gen, dtype=torch.int32).cuda()
    d_emb = (torch.randn(b, 256, generator=gen) * 0.1).cuda()
    rng = StepRNG(7, torch.tensor([7], dtype=torch.int32, device="cuda"))
    outs, grads = [], []
    for on in (True, False):
        enc = FlatEncoder(cfg, torch.device("cuda", 0), dt, "cls", 0, seed=3)
        enc.first_token_layer = on
        for m in (torch.ones_like(mask), mask):        # the second pass finds the buffers as the first one left them
            e = enc.forward(ids, m, rng, train=True)
            assert (enc._fw["first"] is not None) == on
            enc.backward(d_emb)
        outs.append(e.clone())
        grads.append(enc.g.float().clone())
    cu.check_status()
    # one row's sums over features and keys are the same ones in the same order
    assert torch.equal(outs[0], outs[1])
    for name, slot in enc.slots.items():
        x, y = (g[slot.offset: slot.offset + slot.numel] for g in grads)
        # only zero terms are left out of the sums over rows, whose other terms are added in fp32 in another order and rounded
        # once: one ulp, and fp32 noise at the scale of the largest (embeddings: 16-bit atomics in any order)
        scale = float(y.abs().max().clamp_min(1e-6))
        tol = 2.0 ** -7 * y.abs() + (3e-2 if name.startswith("embeddings") else 1e-4) * scale
        assert bool(((x - y).abs() <= tol).all()), (name, float((x - y).abs().max()), scale)


@pytest.mark.parametrize("S,b,heads,dt", [(16, 9, 8, torch.float16), (33, 70, 4, torch.bfloat16)])
@pytest.mark.parametrize("layers", [1, 3, 4])
@pytest.mark.parametrize("side,callback", [(False, True), (True, False), (True, True)])
def test_weight_gradients_left_to_the_next_launch(monkeypatch, S, b, heads, dt, layers, side, callback):
    """Weight gradients on a stream of their own, where the backward buffers of two layers take turns, and the caller's callback, which
    reads a layer's gradients as soon as it is told of them: against one stream without a callback."""
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.models.flat_encoder import FlatEncoder
    from renee_b200.ops import StepRNG, cuda as cu
    monkeypatch.setenv("RENEE_B200_OWN_GEMM", "1")
    cfg = EncoderConfig(dim=256, n_layers=layers, n_heads=heads, hidden_dim=512, vocab_size=2000)
    gen = torch.Generator().manual_seed(S * 10 + b)
    mask = (torch.rand(b, S, generator=gen) < 0.6).to(torch.int32).cuda()
    ids = torch.randint(5, 2000, (b, S), generator=gen, dtype=torch.int32).cuda()
    d_emb = (torch.randn(b, 256, generator=gen) * 0.1).cuda()
    rng = StepRNG(7, torch.tensor([7], dtype=torch.int32, device="cuda"))
    grads = []
    for on in (False, True):
        enc = FlatEncoder(cfg, torch.device("cuda", 0), dt, "cls", 0, seed=3)
        enc._wgrad_stream = torch.cuda.Stream() if on and side else None
        seen = {}

        def done(l):
            for name, slot in enc.slots.items():
                if l >= 0 and name.startswith(f"transformer.layer.{l}.") and len(slot.shape) == 2:
                    seen[name] = enc.g[slot.offset: slot.offset + slot.numel].clone()
        for _ in range(2):
            enc.forward(ids, mask, rng, train=True)
            assert enc._fw["first"] is not None
            enc.g.fill_(float("nan"))
            enc.backward(d_emb, on_layer_done=done if on and callback else None)
        grads.append(enc.g.float().clone())
        torch.cuda.synchronize()
        assert len(seen) == (6 * layers if on and callback else 0)
        for name, g in seen.items():
            slot = enc.slots[name]
            assert torch.equal(g, enc.g[slot.offset: slot.offset + slot.numel]), name
    cu.check_status()
    for name, slot in enc.slots.items():
        x, y = (g[slot.offset: slot.offset + slot.numel] for g in grads)
        # the products are cut into pieces in other places, whose fp32 sums are rounded once: one ulp, and fp32 noise at the scale
        # of the largest (embeddings: 16-bit atomics in any order)
        scale = float(y.abs().max().clamp_min(1e-6))
        tol = 2.0 ** -7 * y.abs() + (3e-2 if name.startswith("embeddings") else 1e-4) * scale
        assert bool(((x - y).abs() <= tol).all()), (name, float((x - y).abs().max()), scale)
