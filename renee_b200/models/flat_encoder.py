"""Flat-buffer encoder engine with a hand-written forward and backward pass.

The reference runs the HF encoder under autograd, DDP and apex FusedAdam (main.py:160-161,
177-181; dl_base.py:299-300, 360, 372).  On B200 the 131K-label configurations are launch-bound,
so this engine is built for CUDA-graph capture instead:

* every parameter is a view into ONE flat fp32 master buffer (decayed parameters first, then the
  no-decay group), with a low-precision compute copy, a flat gradient buffer and flat Adam moments —
  the gradient all-reduce and the fused AdamW each touch one contiguous range;
* the q/k/v projections are adjacent in the buffer, so one GEMM computes all three;
* forward and backward are explicit sequences of GEMMs and fused kernels from :mod:`renee_b200.ops`
  (attention, LayerNorm, embedding gather+LayerNorm, pooling), writing into pre-allocated activations;
  no autograd graph, no allocator calls inside the step.  With 16-bit activations on a GPU every
  linear layer is an own tcgen05 GEMM (``ops/csrc/gemm.cu``) whose epilogue carries its element-wise
  neighbours: bias + GELU (storing the pre-activation), bias + dropout + residual (producing the
  LayerNorm input), GELU backward + bias-gradient column sums, the residual-gradient add of the
  data-gradient GEMMs; the weight gradients of a layer are one launch (``ops/csrc/wgrad.cu``).  fp32 activations (CPU, debugging mode) use
  library GEMMs and stand-alone element-wise ops;
* on that path padded tokens are left out: the activations hold packed rows (``ops/csrc/token_map.cuh``), whose number
  the kernels read from the device, so one captured graph serves every batch of its padded shape.  Texts are shorter
  than the padded length (uniform lengths in the benchmark workloads: 38 to 42 % padding).  What leaving it out gave when
  it went in: training steps of 256 x 32 tokens 3.90 -> 2.92 ms, 128 x 128 7.41 -> 5.50, 512 x 32 with 1.3 M labels
  10.53 -> 8.60, 64 x 256 16.58 -> 11.36;
* with CLS pooling on that path the last layer goes on with first tokens only behind its attention (``_first_tokens``), as do
  their gradients up to it: training steps of 256 x 32 tokens 2.58 -> 2.46 ms, 128 x 128 4.60 -> 4.26, 512 x 32 with 1.3 M
  labels 7.83 -> 7.54; evaluation of 256 x 32 tokens 695 -> 664 us;
* dropout masks are recomputed from a counter-based RNG in the backward pass.

State-dict keys are those of HF DistilBERT (see :mod:`renee_b200.models.encoder`).
"""
from __future__ import annotations

import math
import os
from dataclasses import dataclass

import torch

from .. import ops
from ..utils import guard
from .encoder import EncoderConfig

ALIGN = 128  # elements; keeps every parameter 256-byte aligned in bf16


# dropout stream ids (call sites); layer l uses base + 8*l
_S_EMB, _S_ATTN, _S_FFN, _S_PROBS, _S_CLS = 1, 2, 3, 4, 5


def _no_decay(name: str) -> bool:
    """The reference's no-decay filter is a substring match on ``bias``, ``LayerNorm.bias`` and
    ``LayerNorm.weight`` (dl_base.py:229).  DistilBERT names its block norms ``sa_layer_norm`` /
    ``output_layer_norm``, so only biases and ``embeddings.LayerNorm.weight`` escape weight decay."""
    return any(nd in name for nd in ("bias", "LayerNorm.bias", "LayerNorm.weight"))


# Padded tokens per step and GPU from which the own GEMMs are used in "auto" mode.  The rule looks at nothing but the padded
# shape: the two paths round differently, and a step must not depend on which batch a run happened to begin with.  At small
# sizes the fixed cost per launch of a persistent kernel (TMEM allocation, cluster start-up, a serial K loop on the few SMs the
# tiles cover) outweighs the fused epilogues where most tokens are kept.  Training steps with 16384 labels on one B200, us, own
# (packed) / library GEMMs, all tokens kept; about 60 % kept:
#   DistilBERT, bf16, CLS, S = 32:   1024 padded tokens 1274 / 1167; 1170 / 1166     2048: 1431 / 1358; 1317 / 1356
#                                    3072: 1568 / 1578; 1430 / 1572   4096: 1826 / 1912; 1551 / 1963   6144: 2226 / 2536; 1823 / 2491
#   mean:                            1024: 1298 / 1120; 1180 / 1172   2048: 1486 / 1425; 1352 / 1419   4096: 1954 / 1982; 1615 / 1917
#   fp16, mean, S = 48:              960: 1288 / 1114; 1233 / 1168    2160: 1520 / 1392; 1462 / 1388   4320: 2072 / 2045; 1733 / 2050
#   MiniLM (384-wide), bf16, CLS:    1024: 796 / 735; 696 / 682       2048: 884 / 813; 781 / 867       4096: 1035 / 1137; 924 / 1134
# So with the present kernels the paths cross between 2000 and 4300 tokens even where all are kept.  8192 is where they crossed
# when the rule was made; steps between have run on the library since, and moving the line changes how they round.
OWN_GEMM_MIN_TOKENS = int(os.environ.get("RENEE_B200_OWN_GEMM_MIN_TOKENS", "8192"))


@dataclass
class _Slot:
    offset: int
    shape: tuple
    numel: int


class FlatEncoder:
    def __init__(self, cfg: EncoderConfig, device, act_dtype=torch.bfloat16, pooling: str = "mean",
                 bottleneck_dims: int = 0, seed: int = 0, grad_alloc=None, p16_alloc=None):
        self.cfg = cfg
        self.device = torch.device(device)
        self.act_dtype = act_dtype
        self.pooling = pooling
        self.bottleneck_dims = int(bottleneck_dims)
        self.out_dims = self.bottleneck_dims if self.bottleneck_dims > 0 else cfg.dim
        H, Fd = cfg.dim, cfg.hidden_dim
        names = [("embeddings.word_embeddings.weight", (cfg.vocab_size, H)),
                 ("embeddings.position_embeddings.weight", (cfg.max_position_embeddings, H)),
                 ("embeddings.LayerNorm.weight", (H,)), ("embeddings.LayerNorm.bias", (H,))]
        for l in range(cfg.n_layers):
            p = f"transformer.layer.{l}."
            names += [(p + "attention.q_lin.weight", (H, H)), (p + "attention.k_lin.weight", (H, H)),
                      (p + "attention.v_lin.weight", (H, H)),
                      (p + "attention.q_lin.bias", (H,)), (p + "attention.k_lin.bias", (H,)),
                      (p + "attention.v_lin.bias", (H,)),
                      (p + "attention.out_lin.weight", (H, H)), (p + "attention.out_lin.bias", (H,)),
                      (p + "sa_layer_norm.weight", (H,)), (p + "sa_layer_norm.bias", (H,)),
                      (p + "ffn.lin1.weight", (Fd, H)), (p + "ffn.lin1.bias", (Fd,)),
                      (p + "ffn.lin2.weight", (H, Fd)), (p + "ffn.lin2.bias", (H,)),
                      (p + "output_layer_norm.weight", (H,)), (p + "output_layer_norm.bias", (H,))]
        self.encoder_param_names = [n for n, _ in names]
        if self.bottleneck_dims > 0:
            names.append(("__bottleneck__.transformer_weight", (self.bottleneck_dims, H)))
        decay = [(n, s) for n, s in names if not _no_decay(n)]
        nodecay = [(n, s) for n, s in names if _no_decay(n)]
        # the (decayed) block LayerNorm weights go behind the last layer's matrices: a layer's matrices are then one
        # contiguous range whose gradients are final as soon as the backward pass leaves the layer, while every
        # vector-shaped gradient (LayerNorm, biases: converted by one launch at the end of the pass) sits in the
        # tail of the buffer — which is what lets the gradient reduction start layer by layer under the backward pass
        ln_w = [(n, s) for n, s in decay if n.endswith("layer_norm.weight")]
        decay = [(n, s) for n, s in decay if not n.endswith("layer_norm.weight") and not n.startswith("__bottleneck__")] \
            + ln_w + [(n, s) for n, s in decay if n.startswith("__bottleneck__")]
        self.slots: dict[str, _Slot] = {}
        off = 0
        for n, s in decay:
            numel = math.prod(s)
            self.slots[n] = _Slot(off, s, numel)
            # q/k/v must stay adjacent (no padding between them): H*H and H are multiples of ALIGN
            off += (numel + ALIGN - 1) // ALIGN * ALIGN
        self.n_decay = off
        for n, s in nodecay:
            numel = math.prod(s)
            self.slots[n] = _Slot(off, s, numel)
            off += (numel + ALIGN - 1) // ALIGN * ALIGN
        self.numel = off
        if H % ALIGN != 0:
            raise ValueError(f"hidden size must be a multiple of {ALIGN}")
        dev = self.device
        self.p32 = guard.zeros(off, dtype=torch.float32, device=dev, name="encoder.p32")
        if act_dtype == torch.float32:
            self.p16 = self.p32
        elif p16_alloc is not None:
            self.p16 = p16_alloc(off, act_dtype)[:off]
        else:
            self.p16 = guard.zeros(off, dtype=act_dtype, device=dev, name="encoder.p16")
        if grad_alloc is not None and act_dtype != torch.float32:
            # the gradient buffer lives where the collective backend wants it (symmetric peer memory)
            self.g = grad_alloc(off, act_dtype)[:off]
        else:
            self.g = guard.zeros(off, dtype=act_dtype, device=dev, name="encoder.grad")
        self.m = guard.zeros(off, dtype=torch.float32, device=dev, name="encoder.adam_m")
        self.v = guard.zeros(off, dtype=torch.float32, device=dev, name="encoder.adam_v")
        self._init_params(seed)
        self._acts = None
        self._acts_key = None
        self._plan = None
        self.generation = 0
        self.own_gemm = False          # whether the current step's linears run on the own GEMM kernels
        self._own_mode = "0"
        self._own_supported = False
        self._wgrad_stream = None
        self._wgrad_group = None
        self._wgrad_done = [None, None]
        self._wgrad_left = None        # (parity, weight gradients that the next layer's launch takes along)
        self.pack_tokens = True        # own GEMM path: leave padded tokens out (TokenMap); a comparison may switch it off
        self.first_token_layer = True  # packed tokens, CLS pooling: last layer on first tokens only; a comparison may switch it off
        self.rows_hint = 0             # caller's estimate of the kept tokens of the coming batches (tile planning only)
        if self.device.type in ("cuda", "meta") and act_dtype != torch.float32:
            from ..ops import cuda as cu
            # RENEE_B200_OWN_GEMM: 1 = the own tcgen05 GEMMs with fused epilogues always, 0 = library GEMMs + separate
            # element-wise kernels, auto (default) = own from OWN_GEMM_MIN_TOKENS tokens per step and GPU upwards
            self._own_mode = os.environ.get("RENEE_B200_OWN_GEMM", "auto")
            self._own_supported = cu.enc_gemm_supported(self.p16, H, Fd)
            self.own_gemm = self._own_supported and self._own_mode != "auto"
            if self._own_supported and self.device.type == "cuda" and os.environ.get("RENEE_B200_WGRAD_STREAM", "1") != "0":
                # weight gradients are off the critical path of the backward pass (nothing reads them before the
                # optimizer): a layer's launch runs on a second stream, where it fills the SMs that the next layer's
                # kernels leave idle.  Captured into the step's CUDA graph as parallel branches.
                self._wgrad_stream = torch.cuda.Stream(device=self.device)

    # ------------------------------------------------------------------ parameter views
    def view(self, buf: torch.Tensor, name: str) -> torch.Tensor:
        s = self.slots[name]
        return buf[s.offset: s.offset + s.numel].view(s.shape)

    def _qkv(self, buf, l, kind):
        p = f"transformer.layer.{l}.attention.q_lin.{kind}"
        s = self.slots[p]
        H = self.cfg.dim
        n = 3 * s.numel
        return buf[s.offset: s.offset + n].view((3 * H, H) if kind == "weight" else (3 * H,))

    def _init_params(self, seed: int) -> None:
        g = torch.Generator(device="cpu").manual_seed(int(seed))
        std = self.cfg.initializer_range
        for n, s in self.slots.items():
            if n.endswith("LayerNorm.weight") or n.endswith("layer_norm.weight"):
                t = torch.ones(s.shape)
            elif n.endswith("bias"):
                t = torch.zeros(s.shape)
            elif n.startswith("__bottleneck__"):
                stdv = 1.0 / math.sqrt(s.shape[1])
                t = (torch.rand(s.shape, generator=g) * 2 - 1) * stdv
            else:
                t = torch.randn(s.shape, generator=g) * std
                if n == "embeddings.word_embeddings.weight":
                    t[self.cfg.pad_token_id].zero_()
            self.view(self.p32, n).copy_(t)
        self.sync_compute_copy()

    def sync_compute_copy(self) -> None:
        if self.p16 is not self.p32:
            self.p16.copy_(self.p32)

    def encoder_state_dict(self) -> dict:
        return {n: self.view(self.p32, n).detach().clone() for n in self.encoder_param_names}

    def load_encoder_state_dict(self, sd: dict, strict: bool = True) -> None:
        missing = [n for n in self.encoder_param_names if n not in sd]
        if strict and missing:
            raise KeyError(f"missing encoder keys: {missing[:4]} ...")
        for n in self.encoder_param_names:
            if n in sd:
                self.view(self.p32, n).copy_(sd[n].to(self.p32.device, torch.float32))
        self.sync_compute_copy()

    def bottleneck_weight(self, buf=None):
        return self.view(self.p32 if buf is None else buf, "__bottleneck__.transformer_weight")

    # ------------------------------------------------------------------ activations
    def _alloc(self, b: int, S: int):
        key = (b, S)
        if self._acts_key is not None and self._acts_key[0] >= b and self._acts_key[1] == S:
            return
        cfg, dev, dt = self.cfg, self.device, self.act_dtype
        T, H, Fd, nh = b * S, cfg.dim, cfg.hidden_dim, cfg.n_heads
        e = lambda *shape, dtype=dt: guard.empty(*shape, dtype=dtype, device=dev, name=f"encoder.act{guard.registered()}")
        layers = []
        # long sequences: one softmax-gradient scratch serves every layer (it lives within one attention backward)
        att_ds = ops.attention_ds(b, S, nh, dev, dt)
        for _ in range(cfg.n_layers):
            layers.append(dict(qkv=e(T, 3 * H), ctx=e(T, H), ao=e(T, H), pre1=e(T, H), h1=e(T, H),
                               mean1=e(T, dtype=torch.float32), rstd1=e(T, dtype=torch.float32),
                               f1=e(T, Fd), a1=e(T, Fd), f2=e(T, H), pre2=e(T, H), h2=e(T, H),
                               mean2=e(T, dtype=torch.float32), rstd2=e(T, dtype=torch.float32),
                               att=ops.attention_workspace(b, S, nh, dev, dt, ds=att_ds)))
        self._acts = dict(h0=e(T, H), mean0=e(T, dtype=torch.float32), rstd0=e(T, dtype=torch.float32),
                          layers=layers, pooled=e(b, H, dtype=torch.float32),
                          dh=e(T, H), dctx=e(T, H), att_ds=att_ds,
                          emb=e(b, self.out_dims, dtype=torch.float32), tmap=None, own=None, lib=None)
        self._acts_key = key
        self.generation += 1      # activation addresses changed: graphs captured over the old ones are stale

    def _choose_path(self, T: int) -> None:
        if self._own_mode == "auto":
            self.own_gemm = self._own_supported and T >= OWN_GEMM_MIN_TOKENS

    def allocate(self, b: int, S: int, capacity: int = 0) -> None:
        """Everything that training steps of ``[b, S]`` batches hold (buffers for ``capacity`` >= b rows): what the first
        forward and backward passes would allocate."""
        self._alloc(max(b, capacity), S)
        self._choose_path(b * S)
        self._token_map(S)
        self._ensure_backward_buffers()
        if self._acts["att_ds"] is not None:
            from ..ops import cuda as cu
            if cu.attention_streams(self.act_dtype, S, self.cfg.dim, self.cfg.n_heads):
                self._acts["att_ds"].get()

    def _token_map(self, S: int):
        """The token map of a pass that packs, made by the first one, or ``None``.  Asked on every pass: the environment may
        have sent attention to kernels that read the padded layout."""
        if not (self.own_gemm and self.pack_tokens):
            return None
        from ..ops import cuda as cu
        if not cu.attention_packs(self.act_dtype, S, self.cfg.dim, self.cfg.n_heads):
            return None
        if self._acts["tmap"] is None:
            self._acts["tmap"] = cu.TokenMap(self._acts_key[0], S, self.device)
        return self._acts["tmap"]

    def _first_tokens(self, tmap, S: int):
        """CLS pooling reads one row per sequence, so behind the attention of the last layer (whose keys and values are all
        tokens) only first tokens count: its output projection, LayerNorms and FFN, and their gradients, run on ``b`` rows
        instead of all.  Nothing that is left out reaches the embedding, and the rows' gradients were exact zeros.  For
        packed tokens with attention kernels that know it, else ``None``."""
        if tmap is None or self.pooling != "cls" or not self.first_token_layer:
            return None
        from ..ops import cuda as cu
        return tmap.first if cu.attention_first_token(self.act_dtype, S, self.cfg.dim, self.cfg.n_heads) else None

    # ------------------------------------------------------------------ forward
    def forward(self, input_ids: torch.Tensor, attention_mask: torch.Tensor, rng, train: bool = True) -> torch.Tensor:
        """ids/mask ``[b, S]`` int32 on the device → pooled embedding ``[b, D]`` fp32 (before the
        classifier-input dropout)."""
        cfg = self.cfg
        b, S = input_ids.shape
        self._alloc(b, S)
        A = self._acts
        T, H = b * S, cfg.dim
        self._choose_path(T)
        P = self.p16
        pd = cfg.dropout if train else 0.0
        pa = cfg.attention_dropout if train else 0.0
        po = cfg.attn_output_dropout if train else 0.0
        tmap = self._token_map(S)
        packed = {}
        if tmap is not None:
            tmap.rows_hint = min(self.rows_hint, T)
            tmap.update(attention_mask)
            packed = dict(tmap=tmap)
        first = self._first_tokens(tmap, S)
        self._fw = dict(ids=input_ids, mask=attention_mask, b=b, S=S, pd=pd, pa=pa, po=po, rng=rng, packed=packed, first=first)
        h = A["h0"][:T]
        ops.embed_ln_fwd(input_ids, self.view(P, "embeddings.word_embeddings.weight"),
                         self.view(P, "embeddings.position_embeddings.weight"),
                         self.view(P, "embeddings.LayerNorm.weight"), self.view(P, "embeddings.LayerNorm.bias"),
                         cfg.layer_norm_eps, S, pd, rng, _S_EMB, h, A["mean0"][:T], A["rstd0"][:T],
                         **(dict(mask=attention_mask, **packed) if packed else {}))
        if self.own_gemm:
            h = self._forward_layers_fused(h, attention_mask, T, pd, pa, po, rng, packed, first)
        for l, L in enumerate(A["layers"] if not self.own_gemm else ()):
            pre = f"transformer.layer.{l}."
            sb = 8 * (l + 1)
            qkv = L["qkv"][:T]
            torch.mm(h, self._qkv(P, l, "weight").t(), out=qkv)
            ctx = L["ctx"][:T]
            ops.attention_fwd(qkv, self._qkv(P, l, "bias"), attention_mask, cfg.n_heads, pa, rng, sb + _S_PROBS,
                              ctx, L["att"])
            ao = L["ao"][:T]
            torch.mm(ctx, self.view(P, pre + "attention.out_lin.weight").t(), out=ao)
            h1 = L["h1"][:T]
            # HF DistilBERT applies no dropout to the attention output projection; BERT-family encoders do
            ops.bias_dropout_add_ln_fwd(ao, self.view(P, pre + "attention.out_lin.bias"), h,
                                        self.view(P, pre + "sa_layer_norm.weight"), self.view(P, pre + "sa_layer_norm.bias"),
                                        cfg.layer_norm_eps, po, rng, sb + _S_ATTN,
                                        h1, L["pre1"][:T], L["mean1"][:T], L["rstd1"][:T])
            f1 = L["f1"][:T]
            torch.mm(h1, self.view(P, pre + "ffn.lin1.weight").t(), out=f1)
            a1 = L["a1"][:T]
            ops.bias_gelu_fwd(f1, self.view(P, pre + "ffn.lin1.bias"), a1)
            f2 = L["f2"][:T]
            torch.mm(a1, self.view(P, pre + "ffn.lin2.weight").t(), out=f2)
            h2 = L["h2"][:T]
            ops.bias_dropout_add_ln_fwd(f2, self.view(P, pre + "ffn.lin2.bias"), h1,
                                        self.view(P, pre + "output_layer_norm.weight"),
                                        self.view(P, pre + "output_layer_norm.bias"),
                                        cfg.layer_norm_eps, pd, rng, sb + _S_FFN,
                                        h2, L["pre2"][:T], L["mean2"][:T], L["rstd2"][:T])
            L["h_in"] = h
            h = h2
        pooled = A["pooled"][:b]
        if first is not None:
            ops.pool_fwd(h.view(b, 1, H), attention_mask, self.pooling, pooled)
        else:
            ops.pool_fwd(h.view(b, S, H), attention_mask, self.pooling, pooled, **packed)
        if self.bottleneck_dims > 0:
            emb = A["emb"][:b]
            torch.mm(pooled, self.bottleneck_weight().t(), out=emb)   # fp32, master weights
            return emb
        return pooled

    def _forward_layers_fused(self, h, attention_mask, T, pd, pa, po, rng, packed, first):
        """The transformer blocks on the own GEMMs: 4 GEMMs, 1 attention and 2 LayerNorm launches per layer.  With a
        token map in ``packed`` the activations hold kept tokens only; the buffers keep their padded capacity.  With ``first``
        the last layer goes on with first tokens only behind its attention (its buffers then hold one row per sequence)."""
        from ..ops import cuda as cu
        cfg, A, P = self.cfg, self._acts, self.p16
        for l, L in enumerate(A["layers"]):
            pre = f"transformer.layer.{l}."
            sb = 8 * (l + 1)
            qkv = L["qkv"][:T]
            L["h_in"] = h
            cu.linear_fwd(h, self._qkv(P, l, "weight"), qkv, **packed)
            last = {}
            if first is not None and l == cfg.n_layers - 1:
                T = attention_mask.shape[0]
                last = dict(first=(h, L["ao"][:T]))
            ctx = L["ctx"][:T]
            ops.attention_fwd(qkv, self._qkv(P, l, "bias"), attention_mask, cfg.n_heads, pa, rng, sb + _S_PROBS,
                              ctx, L["att"], **packed, **last)
            if last:
                h, packed = L["ao"][:T], dict(tmap=first)
            pre1 = L["pre1"][:T]
            cu.linear_fwd(ctx, self.view(P, pre + "attention.out_lin.weight"), pre1, "bias_dropout_resid",
                          bias=self.view(P, pre + "attention.out_lin.bias"), resid=h, p=po, rng=rng, stream=sb + _S_ATTN,
                          **packed)
            h1 = L["h1"][:T]
            cu.ln_fwd(pre1, self.view(P, pre + "sa_layer_norm.weight"), self.view(P, pre + "sa_layer_norm.bias"),
                      cfg.layer_norm_eps, h1, L["mean1"][:T], L["rstd1"][:T], **packed)
            a1 = L["a1"][:T]
            cu.linear_fwd(h1, self.view(P, pre + "ffn.lin1.weight"), a1, "bias_gelu",
                          bias=self.view(P, pre + "ffn.lin1.bias"), pre_out=L["f1"][:T], **packed)     # f1 holds x W^T + bias here
            pre2 = L["pre2"][:T]
            cu.linear_fwd(a1, self.view(P, pre + "ffn.lin2.weight"), pre2, "bias_dropout_resid",
                          bias=self.view(P, pre + "ffn.lin2.bias"), resid=h1, p=pd, rng=rng, stream=sb + _S_FFN,
                          **packed)
            h2 = L["h2"][:T]
            cu.ln_fwd(pre2, self.view(P, pre + "output_layer_norm.weight"), self.view(P, pre + "output_layer_norm.bias"),
                      cfg.layer_norm_eps, h2, L["mean2"][:T], L["rstd2"][:T], **packed)
            h = h2
        return h

    # ------------------------------------------------------------------ backward
    def backward(self, d_emb: torch.Tensor, on_layer_done=None) -> None:
        """``d_emb [b, D]`` fp32 → gradients of every parameter written into the flat ``g`` buffer
        (overwritten, not accumulated).  ``on_layer_done(l)`` is called when the gradients of layer ``l``'s
        matrices (one contiguous range of the flat buffer) have become final, and ``on_layer_done(-1)`` at the
        end of the pass (embeddings, bottleneck, LayerNorm parameters and biases), so a caller can reduce the
        buffer across ranks piece by piece while the remaining layers are still being differentiated."""
        if self.g.is_cuda:
            # column sums (LN gammas/betas, all bias gradients) are accumulated by the kernels and converted
            # by ONE launch at the end of the pass instead of a serial tail inside each kernel
            from ..ops import cuda as cu
            if self._plan is None:
                self._plan = cu.DeferredColumns(self.device, self.act_dtype)
            with cu.deferred_columns(self._plan):
                self._backward(d_emb, on_layer_done)
            self._plan.finalize()
        else:
            self._backward(d_emb, on_layer_done)
        if on_layer_done is not None:
            on_layer_done(-1)       # embeddings and every vector-shaped gradient are final: the whole buffer is

    def _wgrad_layer(self, par: int, items, packed) -> None:
        """Weight gradients in one launch, their rows numbered by the token map in ``packed``, on the weight-gradient stream (ordered
        after everything issued so far on the current one).  Their inputs live in the backward buffers of parity ``par``, which the
        layer after the next overwrites: :meth:`_wgrad_wait` comes before that."""
        from ..ops import cuda as cu
        side = self._wgrad_stream
        if side is None:
            cu.wgrad_group(items, self._wgrad_group, **packed)
            return
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            cu.wgrad_group(items, self._wgrad_group, **packed)
            self._wgrad_done[par] = side.record_event()

    def _wgrad_wait(self, par: int) -> None:
        """The current stream waits for the weight gradients last issued with parity ``par``."""
        if self._wgrad_done[par] is not None:
            torch.cuda.current_stream().wait_event(self._wgrad_done[par])
            self._wgrad_done[par] = None

    def _backward(self, d_emb: torch.Tensor, on_layer_done=None) -> None:
        cfg, A, fw = self.cfg, self._acts, self._fw
        b, S, pd, pa, rng = fw["b"], fw["S"], fw["pd"], fw["pa"], fw["rng"]
        T, H = b * S, cfg.dim
        P, G = self.p16, self.g
        mask, packed = fw["mask"], fw["packed"]
        self._wgrad_done = [None, None]      # a pass that ended in an exception may have left an event of its own (or its capture's)
        self._wgrad_left = None
        if self.bottleneck_dims > 0:
            gw = self.view(G, "__bottleneck__.transformer_weight")
            pooled = A["pooled"][:b]
            if gw.dtype == torch.float32:
                torch.mm(d_emb.t(), pooled, out=gw)
            else:
                gw.copy_(torch.mm(d_emb.t(), pooled))
            d_pool = torch.mm(d_emb, self.bottleneck_weight())
        else:
            d_pool = d_emb
        self._ensure_backward_buffers()
        dh = A["dh"][:T]
        if fw["first"] is not None:
            ops.pool_bwd(d_pool, mask, self.pooling, 1, dh[:b].view(b, 1, H))
        else:
            ops.pool_bwd(d_pool, mask, self.pooling, S, dh.view(b, S, H), **packed)
        for l in reversed(range(cfg.n_layers)):
            L = A["layers"][l]
            pre = f"transformer.layer.{l}."
            sb = 8 * (l + 1)
            h_in = L["h_in"]
            if self.own_gemm:
                self._backward_layer_fused(l, L, dh, on_layer_done)
                continue
            buf = A["lib"][0]
            # ---- output LN + FFN
            d_pre2, d_f2 = ops.bias_dropout_add_ln_bwd(
                dh, L["pre2"][:T], self.view(P, pre + "output_layer_norm.weight"), L["mean2"][:T], L["rstd2"][:T],
                pd, rng, sb + _S_FFN,
                self.view(G, pre + "output_layer_norm.weight"), self.view(G, pre + "output_layer_norm.bias"),
                self.view(G, pre + "ffn.lin2.bias"), buf["dh_b"][:T], L["f2"][:T])
            torch.mm(d_f2.t(), L["a1"][:T], out=self.view(G, pre + "ffn.lin2.weight"))
            da1 = buf["da1"][:T]
            torch.mm(d_f2, self.view(P, pre + "ffn.lin2.weight"), out=da1)
            df1 = buf["df1"][:T]
            ops.bias_gelu_bwd(da1, L["f1"][:T], self.view(P, pre + "ffn.lin1.bias"),
                              self.view(G, pre + "ffn.lin1.bias"), df1)
            torch.mm(df1.t(), L["h1"][:T], out=self.view(G, pre + "ffn.lin1.weight"))
            # dh1 = d_pre2 (residual) + df1 @ W1
            dh1 = d_pre2.addmm_(df1, self.view(P, pre + "ffn.lin1.weight"))      # in place: no copy of the addend
            # ---- attention LN + attention
            d_pre1, d_ao = ops.bias_dropout_add_ln_bwd(
                dh1, L["pre1"][:T], self.view(P, pre + "sa_layer_norm.weight"), L["mean1"][:T], L["rstd1"][:T],
                fw["po"], rng, sb + _S_ATTN,
                self.view(G, pre + "sa_layer_norm.weight"), self.view(G, pre + "sa_layer_norm.bias"),
                self.view(G, pre + "attention.out_lin.bias"), dh, L["ao"][:T])
            torch.mm(d_ao.t(), L["ctx"][:T], out=self.view(G, pre + "attention.out_lin.weight"))
            dctx = A["dctx"][:T]
            torch.mm(d_ao, self.view(P, pre + "attention.out_lin.weight"), out=dctx)
            dqkv = buf["dqkv"][:T]
            ops.attention_bwd(dctx, L["qkv"][:T], self._qkv(P, l, "bias"), mask, cfg.n_heads, pa, rng,
                              sb + _S_PROBS, L["att"], dqkv, self._qkv(G, l, "bias"))
            torch.mm(dqkv.t(), h_in, out=self._qkv(G, l, "weight"))
            d_pre1.addmm_(dqkv, self._qkv(P, l, "weight"))                       # d_pre1 is dh
            if on_layer_done is not None:
                on_layer_done(l)
        ops.embed_ln_bwd(dh, fw["ids"], self.view(P, "embeddings.word_embeddings.weight"),
                         self.view(P, "embeddings.position_embeddings.weight"),
                         self.view(P, "embeddings.LayerNorm.weight"), A["mean0"][:T], A["rstd0"][:T],
                         S, pd, rng, _S_EMB, cfg.pad_token_id,
                         self.view(G, "embeddings.word_embeddings.weight"),
                         self.view(G, "embeddings.position_embeddings.weight"),
                         self.view(G, "embeddings.LayerNorm.weight"), self.view(G, "embeddings.LayerNorm.bias"), **packed)
        self._wgrad_wait(0)
        self._wgrad_wait(1)

    def _ensure_backward_buffers(self) -> None:
        """The gradient buffers of one block, allocated by the first backward pass of the path that uses them.  Library path:
        one set.  Own GEMMs: two sets of the gradients that the weight-gradient launch of a layer still reads while the next
        layer is differentiated, and that launch's scratch."""
        which = "own" if self.own_gemm else "lib"
        if self._acts[which] is not None:
            return
        (b, S), H, Fd = self._acts_key, self.cfg.dim, self.cfg.hidden_dim
        widths = (("dpre2", H), ("dpre1", H), ("df1", Fd), ("dqkv", 3 * H)) if self.own_gemm else \
            (("dh_b", H), ("dqkv", 3 * H), ("df1", Fd), ("da1", Fd))
        sets = 2 if self.own_gemm else 1
        sizes = [b * S * n for _, n in widths] * sets
        flat = guard.empty(sum(sizes), dtype=self.act_dtype, device=self.device, name="encoder.activations.bwd").split(sizes)
        self._acts[which] = [{k: flat[len(widths) * i + j].view(b * S, n) for j, (k, n) in enumerate(widths)}
                             for i in range(sets)]
        if self.own_gemm and self._wgrad_group is None:
            from ..ops import cuda as cu
            self._wgrad_group = cu.WgradGroup([(3 * H, H), (H, H), (Fd, H), (H, Fd), (3 * H, H)], self.device)

    def _backward_layer_fused(self, l: int, L: dict, dh, on_layer_done) -> None:
        """One transformer block on the own GEMMs: ``dh`` (gradient of its output) becomes the gradient of its input."""
        from ..ops import cuda as cu
        cfg, A, P, G, fw = self.cfg, self._acts, self.p16, self.g, self._fw
        T, packed, pd, po, rng = fw["b"] * fw["S"], fw["packed"], fw["pd"], fw["po"], fw["rng"]
        pre, sb, par = f"transformer.layer.{l}.", 8 * (l + 1), l & 1
        # n rows, numbered by `rows`: all tokens, or first tokens only up to the attention of the last layer
        n, rows = T, packed
        if fw["first"] is not None and l == cfg.n_layers - 1:
            n, rows = fw["b"], dict(tmap=fw["first"])
        one_row = rows is not packed
        buf = A["own"][par]
        self._wgrad_wait(par)
        d_pre2, d_f2 = ops.bias_dropout_add_ln_bwd(
            dh[:n], L["pre2"][:n], self.view(P, pre + "output_layer_norm.weight"), L["mean2"][:n], L["rstd2"][:n],
            pd, rng, sb + _S_FFN,
            self.view(G, pre + "output_layer_norm.weight"), self.view(G, pre + "output_layer_norm.bias"),
            self.view(G, pre + "ffn.lin2.bias"), buf["dpre2"][:n], L["f2"][:n], **rows)
        df1 = cu.linear_dgrad(d_f2, self.view(P, pre + "ffn.lin2.weight"), buf["df1"][:n], "gelu_bwd", pre=L["f1"][:n],
                              dbias=self.view(G, pre + "ffn.lin1.bias"), **rows)
        dh1 = cu.linear_dgrad(df1, self.view(P, pre + "ffn.lin1.weight"), dh[:n], "add", resid=d_pre2, **rows)
        d_pre1, d_ao = ops.bias_dropout_add_ln_bwd(
            dh1, L["pre1"][:n], self.view(P, pre + "sa_layer_norm.weight"), L["mean1"][:n], L["rstd1"][:n],
            po, rng, sb + _S_ATTN,
            self.view(G, pre + "sa_layer_norm.weight"), self.view(G, pre + "sa_layer_norm.bias"),
            self.view(G, pre + "attention.out_lin.bias"), buf["dpre1"][:n], L["ao"][:n], **rows)
        dctx = cu.linear_dgrad(d_ao, self.view(P, pre + "attention.out_lin.weight"), A["dctx"][:n], **rows)
        dqkv = buf["dqkv"][:T]
        # with one row per sequence the attention kernel lays the residual's gradient out for all tokens (h2 is free by now)
        resid = L["h2"][:T] if one_row else d_pre1
        ops.attention_bwd(dctx, L["qkv"][:T], self._qkv(P, l, "bias"), fw["mask"], cfg.n_heads, fw["pa"], rng,
                          sb + _S_PROBS, L["att"], dqkv, self._qkv(G, l, "bias"), **packed,
                          **(dict(first=(d_pre1, resid)) if one_row else {}))
        dense = [(df1, L["h1"][:n], self.view(G, pre + "ffn.lin1.weight")),
                 (d_f2, L["a1"][:n], self.view(G, pre + "ffn.lin2.weight"))]
        qkv = [(dqkv, L["h_in"], self._qkv(G, l, "weight"))]
        out = [(d_ao, L["ctx"][:n], self.view(G, pre + "attention.out_lin.weight"))]
        if one_row:
            # all tokens behind q/k/v, one row per sequence behind the others: two launches, unless the next layer's can take q/k/v
            # along (27 tiles on their own are cut into pieces for 74 SM pairs: 32 us at 4900 tokens, 13 in its company)
            self._wgrad_layer(par, dense + out, {})
            if l > 0 and on_layer_done is None:
                self._wgrad_left = (par, qkv)
            else:
                self._wgrad_layer(par, qkv, packed)
        else:
            left, self._wgrad_left = self._wgrad_left, None
            self._wgrad_layer(par, dense + qkv + out + (left[1] if left else []), packed)
            if left:
                self._wgrad_done[left[0]] = self._wgrad_done[par]
        cu.linear_dgrad(dqkv, self._qkv(P, l, "weight"), dh, "add", resid=resid, **packed)
        if on_layer_done is not None:
            self._wgrad_wait(par)           # the caller may reduce the layer's gradients from here on
            on_layer_done(l)
