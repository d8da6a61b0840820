"""Which attention kernel a call reaches: packed rows only the kernels that know them, whatever the environment says."""
import pytest
import torch

from renee_b200.ops import StepRNG, cuda as cu


@pytest.fixture
def calls(monkeypatch):
    seen = []
    monkeypatch.setattr(cu, "_call", lambda name, *a, launches=1: seen.append((name, launches, len(a))))
    monkeypatch.setattr(cu, "_stream", lambda: None)
    monkeypatch.setattr(cu, "colsum", lambda x, out: None)
    return seen


class _Map:
    pointers = dict.fromkeys(("slot", "len", "meta"))


def _attend(S, hd, dtype, tmap, b=2, nh=2):
    H = nh * hd
    z = lambda *s: torch.zeros(*s, dtype=dtype)
    mask = torch.ones(b, S, dtype=torch.int32)
    rng = StepRNG(1, torch.tensor([1], dtype=torch.int32))
    ws = {"probs": z(b, nh, S, S), "ds": z(1)}
    cu.attention_fwd(z(b * S, 3 * H), z(3 * H), mask, nh, 0.0, rng, 1, z(b * S, H), ws, tmap=tmap)
    cu.attention_bwd(z(b * S, H), z(b * S, 3 * H), z(3 * H), mask, nh, 0.0, rng, 1, ws, z(b * S, 3 * H), z(3 * H), tmap=tmap)


ENVS = [{}, {"RENEE_B200_ATTENTION": "tiles"}, {"RENEE_B200_ATTENTION_LONG": "0"}]


@pytest.mark.parametrize("env", ENVS, ids=["default", "tiles", "no_long"])
@pytest.mark.parametrize("S,hd,dtype,kind,launches", [
    (1, 64, torch.bfloat16, "mma", (1, 1)), (32, 32, torch.float16, "mma", (1, 1)), (33, 64, torch.float16, "mma", (2, 2)),
    (128, 32, torch.bfloat16, "mma", (2, 2)), (129, 64, torch.bfloat16, "mma", (2, 2)), (256, 64, torch.float16, "mma", (2, 2)),
    (257, 64, torch.bfloat16, "long", (1, 2)), (512, 64, torch.bfloat16, "long", (1, 2)),
    (129, 32, torch.bfloat16, None, None), (513, 64, torch.bfloat16, None, None), (32, 64, torch.float32, None, None),
    (64, 16, torch.bfloat16, None, None)])
def test_packed_rows_reach_only_kernels_that_know_them(calls, monkeypatch, env, S, hd, dtype, kind, launches):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    if kind is None:
        assert not cu.attention_packs(dtype, S, 2 * hd, 2)
        with pytest.raises(cu.KernelError):
            _attend(S, hd, dtype, _Map)
        assert calls == []
        return
    _attend(S, hd, dtype, _Map)
    got = [(n, l) for n, l, _ in calls if n.startswith("rb_attention")]
    assert got == [(f"rb_attention_fwd_{kind}", launches[0]), (f"rb_attention_bwd_{kind}", launches[1])]
    if not env:
        assert cu.attention_packs(dtype, S, 2 * hd, 2)


@pytest.mark.parametrize("S,hd,dtype,env,fwd,bwd", [
    (32, 64, torch.bfloat16, ENVS[0], "rb_attention_fwd_mma", "rb_attention_bwd_mma"),
    (200, 64, torch.bfloat16, ENVS[0], "rb_attention_fwd_mma", "rb_attention_bwd_mma"),
    (32, 64, torch.bfloat16, ENVS[1], "rb_attention_fwd_tc", "rb_attention_bwd_tc"),
    (200, 64, torch.bfloat16, ENVS[1], "rb_attention_fwd_long", "rb_attention_bwd_long"),
    (300, 64, torch.float16, ENVS[0], "rb_attention_fwd_long", "rb_attention_bwd_long"),
    (100, 16, torch.float16, ENVS[0], "rb_attention_fwd_tc", "rb_attention_bwd_tc"),
    (32, 64, torch.float32, ENVS[0], "rb_attention_fwd", "rb_attention_bwd")])
def test_padded_rows_follow_the_environment(calls, monkeypatch, S, hd, dtype, env, fwd, bwd):
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    _attend(S, hd, dtype, None)
    long = 2 if bwd.endswith("_long") else 1
    assert [(n, l) for n, l, _ in calls if n.startswith("rb_attention")] == [(fwd, 1), (bwd, long)]
    # arguments of the C entries: 14, 3 more where packed rows are known; the backward's bias accumulator (16-bit kernels) and
    # softmax-gradient scratch (streaming kernels)
    n_fwd, n_bwd = (a for n, _, a in calls if n.startswith("rb_attention"))
    known = 3 if fwd.endswith(("_mma", "_long")) else 0
    assert n_fwd == 14 + known
    assert n_bwd == 14 + known + (dtype != torch.float32) + (long == 2)


@pytest.mark.gpu
@pytest.mark.parametrize("S,env", [(32, ENVS[1]), (100, ENVS[1]), (160, ENVS[1]), (160, ENVS[2])])
def test_switch_set_after_the_first_pass_is_followed(monkeypatch, S, env):
    """An engine that has packed tokens before goes back to the padded layout when the environment asks for kernels that only
    know that one; a switch between forward and backward leaves the pass on the kernels it began with."""
    from renee_b200.models.encoder import EncoderConfig
    from renee_b200.models.flat_encoder import FlatEncoder
    cfg = EncoderConfig(dim=256, n_layers=2, n_heads=4, hidden_dim=512, vocab_size=2000)
    gen = torch.Generator().manual_seed(S)
    lens = torch.randint(1, S + 1, (6,), generator=gen)
    mask = (torch.arange(S)[None] < lens[:, None]).to(torch.int32).cuda()
    ids = torch.randint(5, 2000, (6, S), generator=gen, dtype=torch.int32).cuda()
    d_emb = (torch.randn(6, 256, generator=gen) * 0.1).cuda()
    rng = StepRNG(7, torch.tensor([7], dtype=torch.int32, device="cuda"))
    monkeypatch.setenv("RENEE_B200_OWN_GEMM", "1")

    def run(switch):
        enc = FlatEncoder(cfg, torch.device("cuda", 0), torch.bfloat16, "mean", 0, seed=3)
        out = []
        for at in ("first pass", "between", "later pass"):
            e = enc.forward(ids, mask, rng, train=True)
            if switch and at == "between":
                for k, v in env.items():
                    monkeypatch.setenv(k, v)
            enc.backward(d_emb)
            out += [e.clone(), enc.g.float().clone()]
        for k in env:
            monkeypatch.delenv(k, raising=False)
        return out

    for got, want in zip(run(True), run(False)):
        # other kernels: 16-bit probabilities and activations round differently here and there (2^-8 each)
        assert float((got - want).norm() / want.norm()) < 2.0 ** -7
    cu.check_status()
