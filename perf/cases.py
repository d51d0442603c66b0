"""The work that a user of this framework has it do, as cases to be timed and compared.

Four kinds, each through the public entry points a program calls:

  block      one attention block + residual + LayerNorm (`Encoder.forward` of a configuration without the feed-forward)
  encoder    a BERT encoder stack, fp32 activations in and out (`Encoder.forward`)
  reader     reading comprehension / pooled classification from token ids: embedding front-end, key mask, encoder stack,
             span-extraction head and pooler head (`ops.*` and `Encoder.forward_hidden`)
  attention  the attention operator alone on a packed QKV activation (`ops.attention`)

`cfg` is "base" (12 layers, hidden 768, 12 heads, FFN 3072) or "large" (24 layers, 1024, 16, 4096), the two geometries
of `tnn_b200.model_synth`.  `lo` is the shortest sequence of a padded batch: lengths ~ Uniform[lo, S]; lo = S means that
every sequence is full.  The key mask is always passed, as the graph's mask input always is.
"""
import math

import numpy as np
import torch

from tnn_b200 import ops
from tnn_b200.encoder import Encoder
from tnn_b200.model_synth import BERT_BASE, BERT_LARGE, EncoderConfig, LayerWeights

CFGS = {"base": BERT_BASE, "large": BERT_LARGE}
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16}
VOCAB = 30522          # BERT's word-piece vocabulary, two segment types, 512 positions
MAX_POS = 512
# No drawn case costs more than the largest listed one (1024 sequences x 128 tokens, base).
MAX_FLOPS = 2.29e13


def _case(kind, B, S, lo, dtype, cfg="base", heads=0, name=None):
    c = {"kind": kind, "B": B, "S": S, "lo": lo, "dtype": dtype, "cfg": cfg, "heads": heads}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one attention block for one sentence (benchmark configuration 1)
        _case("block", 1, 128, 128, "f16", name="block_b1_s128_f16"),
        # interactive serving: one short sentence, an odd number of tokens
        _case("encoder", 1, 41, 41, "f16", name="base_b1_s41_f16"),
        # the reading-comprehension demo: one question + paragraph, padded to the tokenizer's 256 tokens
        _case("reader", 1, 256, 64, "f16", name="reader_base_b1_s256_f16"),
        # a few requests gathered by a server: ragged, odd padded length
        _case("encoder", 4, 77, 9, "bf16", name="base_b4_s77_ragged_bf16"),
        # a small full batch: a quarter of configuration 2
        _case("encoder", 16, 128, 128, "f16", name="base_b16_s128_f16"),
        # benchmark configuration 2: ordinary batch, full length
        _case("encoder", 64, 128, 128, "f16", name="base_b64_s128_f16"),
        # benchmark configuration 3: padded variable-length batch
        _case("encoder", 32, 256, 16, "f16", name="base_b32_s256_ragged_f16"),
        # benchmark configuration 4: BERT-large, long padded sequences, bf16
        _case("encoder", 64, 384, 128, "bf16", cfg="large", name="large_b64_s384_ragged_bf16"),
        # benchmark configuration 5: the full throughput batch
        _case("encoder", 1024, 128, 128, "f16", name="base_b1024_s128_f16"),
        # the attention sweep of configuration 5 (16 heads x 64, batch 16): shortest, a padded middle one, longest
        _case("attention", 16, 512, 512, "f16", heads=16, name="attn_b16_h16_s512_f16"),
        _case("attention", 16, 1024, 200, "bf16", heads=16, name="attn_b16_h16_s1024_ragged_bf16"),
        _case("attention", 16, 2048, 2048, "f16", heads=16, name="attn_b16_h16_s2048_f16"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: kinds by how often a program meets them, sizes spread over the logarithm of their ranges."""
    while True:
        kind = rng.choices(["block", "encoder", "reader", "attention"], [1, 5, 2, 3])[0]
        dtype = rng.choice(["f16", "bf16"])
        ragged = rng.random() < 0.6
        if kind == "attention":
            S = _log_int(rng, 64, 2048)
            B = _log_int(rng, 1, max(1, 32768 // S))
            heads, cfg = rng.choice([12, 16]), "base"
        else:
            S = _log_int(rng, 16, MAX_POS)
            tokens = _log_int(rng, S, 131072)
            B = max(1, tokens // S)
            heads, cfg = 0, ("base" if kind != "encoder" or rng.random() < 0.7 else "large")
        if rng.random() < 0.5 and S >= 32:
            S = S // 16 * 16          # callers often pad to a round length, others do not
        lo = max(1, int(S * rng.uniform(0.05, 0.7))) if ragged else S
        c = _case(kind, B, S, lo, dtype, cfg, heads)
        if work(c)["flops"] <= MAX_FLOPS:
            return c


# ---------------------------------------------------------------------------------------------------- preparation
class _Weights:
    """What `Encoder.from_workload` reads of a workload: the geometry and the host weights of every layer."""

    def __init__(self, cfg, gen, dev):
        def normal(shape, std, mean=0.0):
            return (torch.randn(shape, device=dev, generator=gen) * std + mean).cpu().numpy()

        H, F = cfg.hidden, cfg.ffn
        self.cfg = cfg
        self.weights = []
        for _ in range(cfg.layers):
            lw = LayerWeights(*[normal((H, H), 0.02) for _ in range(4)], *[normal((H,), 0.05) for _ in range(4)],
                              normal((H,), 0.1, 1.0), normal((H,), 0.1))
            if cfg.with_ffn:
                lw.w1, lw.b1 = normal((H, F), 0.02), normal((F,), 0.05)
                lw.w2, lw.b2 = normal((F, H), 0.02), normal((H,), 0.05)
                lw.ln2_g, lw.ln2_b = normal((H,), 0.1, 1.0), normal((H,), 0.1)
            self.weights.append(lw)


def prepare(case, seed):
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    B, S, kind = case["B"], case["S"], case["kind"]
    dt = DTYPES[case["dtype"]]
    lengths = np.random.default_rng(seed).integers(case["lo"], S + 1, B)
    valid = torch.arange(S, device=dev)[None, :] < torch.from_numpy(lengths).to(dev)[:, None]
    st = {"kind": kind}
    if kind == "attention":
        heads = case["heads"]
        st["heads"] = heads
        st["qkv"] = torch.randn((B, S, 3 * heads * 64), device=dev, generator=gen).to(dt)
        st["mask"] = torch.where(valid, 0.0, -10000.0).contiguous()
        return st
    cfg = CFGS[case["cfg"]]
    if kind == "block":
        cfg = EncoderConfig(1, cfg.hidden, cfg.heads, cfg.ffn, with_ffn=False)
    st["enc"] = Encoder.from_workload(_Weights(cfg, gen, dev), dt, dev)
    H = cfg.hidden
    if kind == "reader":
        st["ids"] = torch.randint(0, VOCAB, (B, S), device=dev, generator=gen, dtype=torch.int32)
        split = torch.from_numpy(lengths // 4).to(dev)[:, None]            # question, then paragraph
        st["segments"] = (torch.arange(S, device=dev)[None, :] >= split).to(torch.int32).contiguous()
        st["input_mask"] = valid.to(torch.int32).contiguous()
        for k, rows in (("word", VOCAB), ("type", 2), ("pos", MAX_POS)):
            st[k] = (torch.randn((rows, H), device=dev, generator=gen) * 0.02).to(dt)
        st["gamma"] = 1.0 + 0.1 * torch.randn(H, device=dev, generator=gen)
        st["beta"] = 0.1 * torch.randn(H, device=dev, generator=gen)
        st["dtype"] = dt
        st["w_qa"] = 0.02 * torch.randn((H, 2), device=dev, generator=gen)
        st["b_qa"] = 0.02 * torch.randn(2, device=dev, generator=gen)
        st["w_pool"] = ops.pack_weight(0.02 * torch.randn((H, H), device=dev, generator=gen), dt)
        st["b_pool"] = 0.02 * torch.randn(H, device=dev, generator=gen)
    else:
        st["x"] = torch.randn((B, S, H), device=dev, generator=gen)
        st["mask"] = torch.where(valid, 0.0, -10000.0).reshape(B, 1, 1, S).contiguous()
    return st


# ---------------------------------------------------------------------------------------------------- one pass
def run(st):
    kind = st["kind"]
    if kind == "attention":
        kv_len = ops.mask_to_kv_len(st["mask"])
        return ops.attention(st["qkv"], st["heads"], st["mask"], kv_len)
    enc = st["enc"]
    if kind != "reader":
        return enc.forward(st["x"], st["mask"])
    hidden = ops.embedding_layernorm(st["ids"], st["segments"], st["word"], st["type"], st["pos"], st["gamma"],
                                     st["beta"], enc.cfg.ln_eps, out_dtype=st["dtype"])
    mask, kv_len = ops.mask_from_input_mask(st["input_mask"])
    hidden = enc.forward_hidden(hidden, mask, kv_len)
    logits = ops.qa_head(hidden, st["w_qa"], st["b_qa"])
    pooled = ops.linear(hidden[:, 0], st["w_pool"], st["b_pool"], epilogue=ops.EPI_BIAS_TANH)
    return {"hidden": hidden, "logits": logits, "pooled": pooled}


# ---------------------------------------------------------------------------------------------------- work, tolerance
def work(case):
    """Every query row is part of the result, padded ones too; keys beyond a sequence's end weigh exactly nothing, so
    the attention's share counts the mean length's keys only."""
    B, S = case["B"], case["S"]
    keys = (case["lo"] + S) / 2.0
    T = B * S
    if case["kind"] == "attention":
        H = case["heads"] * 64
        return {"flops": 4.0 * T * keys * H, "bytes": 2.0 * T * H * 2 + 2.0 * B * keys * H * 2 + 4.0 * T}
    cfg = CFGS[case["cfg"]]
    H, F = cfg.hidden, cfg.ffn
    L = 1 if case["kind"] == "block" else cfg.layers
    per_layer = 4 * H * H + (0 if case["kind"] == "block" else 2 * H * F)
    flops = L * (2.0 * T * per_layer + 4.0 * T * keys * H)
    n_bytes = 2.0 * L * per_layer + 4.0 * T
    if case["kind"] == "reader":
        # ids, segments, mask; the embedding rows in use; the pooler's weight; hidden state, logits and pooled rows
        flops += 2.0 * T * H * 2 + 2.0 * B * H * H
        n_bytes += 8.0 * T + 2.0 * (min(T, VOCAB) + min(S, MAX_POS)) * H + 2.0 * H * H + 2.0 * T * H + 8.0 * T + 2.0 * B * H
    else:
        n_bytes += 8.0 * T * H     # fp32 activations in and out
    return {"flops": flops, "bytes": n_bytes}


def tolerance(case):
    """About four times what the path was seen to differ from the same computation in 64-bit floating point (weights
    rounded to the compute type, nothing else): attention and one block f16 3.6e-4 / 1.8e-3, bf16 2.9e-3 / 1.5e-2;
    whole stacks f16 1.3e-3 / 1.2e-2, bf16 1.05e-2 / 6.0e-2 (relative 2-norm / largest difference)."""
    half = case["dtype"] == "f16"
    if case["kind"] in ("block", "attention"):
        return {"rel": 1.5e-3, "max": 8e-3} if half else {"rel": 1.2e-2, "max": 6e-2}
    return {"rel": 5e-3, "max": 5e-2} if half else {"rel": 3e-2, "max": 0.25}


# ---------------------------------------------------------------------------------------------------- 64-bit result
def _exact_layernorm(x, gamma, beta, eps):
    mean = x.mean(-1, keepdim=True)
    var = ((x - mean) ** 2).mean(-1, keepdim=True)
    return (x - mean) / torch.sqrt(var + eps) * gamma + beta


def _exact_attention(qkv, heads, valid):
    """softmax(Q K^T / 8) V over the valid keys, one sequence at a time (the scores of a whole batch need not fit)."""
    B, S, W = qkv.shape
    H = W // 3
    out = torch.empty((B, S, H), dtype=qkv.dtype, device=qkv.device)
    for b in range(B):
        n = int(valid[b].sum())
        q, k, v = (qkv[b, :, i * H:(i + 1) * H].reshape(S, heads, 64).transpose(0, 1) for i in range(3))
        p = torch.softmax(q @ k[:, :n].transpose(1, 2) * 0.125, dim=-1)
        out[b] = (p @ v[:, :n]).transpose(0, 1).reshape(S, H)
    return out


def exact(case, seed):
    """`run`'s outputs in 64-bit floating point: the same inputs, matrix weights rounded to the compute type (the type
    they are given to the path in), nothing else rounded."""
    dev = torch.device("cuda")
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    B, S, kind = case["B"], case["S"], case["kind"]
    dt = DTYPES[case["dtype"]]
    lengths = np.random.default_rng(seed).integers(case["lo"], S + 1, B)
    valid = torch.arange(S, device=dev)[None, :] < torch.from_numpy(lengths).to(dev)[:, None]
    if kind == "attention":
        heads = case["heads"]
        return _exact_attention(torch.randn((B, S, 3 * heads * 64), device=dev, generator=gen).to(dt).double(), heads, valid)
    cfg = CFGS[case["cfg"]]
    if kind == "block":
        cfg = EncoderConfig(1, cfg.hidden, cfg.heads, cfg.ffn, with_ffn=False)
    weights = _Weights(cfg, gen, dev).weights
    H, eps = cfg.hidden, cfg.ln_eps

    def full(a):
        return torch.from_numpy(a).to(dev).double()

    def half(a):
        return torch.from_numpy(a).to(dev).to(dt).double()

    if kind == "reader":
        ids = torch.randint(0, VOCAB, (B, S), device=dev, generator=gen, dtype=torch.int32)
        segments = torch.arange(S, device=dev)[None, :] >= torch.from_numpy(lengths // 4).to(dev)[:, None]
        word, typ, pos = ((torch.randn((rows, H), device=dev, generator=gen) * 0.02).to(dt).double()
                          for rows in (VOCAB, 2, MAX_POS))
        gamma = 1.0 + 0.1 * torch.randn(H, device=dev, generator=gen)
        beta = 0.1 * torch.randn(H, device=dev, generator=gen)
        w_qa = 0.02 * torch.randn((H, 2), device=dev, generator=gen)
        b_qa = 0.02 * torch.randn(2, device=dev, generator=gen)
        w_pool = 0.02 * torch.randn((H, H), device=dev, generator=gen)
        b_pool = 0.02 * torch.randn(H, device=dev, generator=gen)
        x = _exact_layernorm(word[ids.long()] + typ[segments.long()] + pos[:S], gamma.double(), beta.double(), eps)
    else:
        x = torch.randn((B, S, H), device=dev, generator=gen).double()
    for lw in weights:
        qkv = torch.cat([x @ half(w) + full(b) for w, b in ((lw.wq, lw.bq), (lw.wk, lw.bk), (lw.wv, lw.bv))], -1)
        x = _exact_layernorm(_exact_attention(qkv, cfg.heads, valid) @ half(lw.wo) + full(lw.bo) + x, full(lw.ln1_g),
                             full(lw.ln1_b), eps)
        if cfg.with_ffn:
            f = x @ half(lw.w1) + full(lw.b1)
            f = 0.5 * f * (1.0 + torch.erf(f * math.sqrt(0.5)))
            x = _exact_layernorm(f @ half(lw.w2) + full(lw.b2) + x, full(lw.ln2_g), full(lw.ln2_b), eps)
    if kind != "reader":
        return x
    logits = (x.reshape(-1, H) @ w_qa.double() + b_qa.double()).T.contiguous()
    pooled = torch.tanh(x[:, 0] @ w_pool.to(dt).double() + b_pool.double())
    return {"hidden": x, "logits": logits, "pooled": pooled}
