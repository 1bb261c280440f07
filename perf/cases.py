"""Performance cases: the work that programs built on helix_b200 have it do, each through an entry point that such a program calls.

Kernel-level cases go through the C ABI of include/helix_b200_kernels.h at the layer sizes of this repository's configurations
(helix_b200/configs.py: the 8B and 1B decoders, the bge-base encoder); whole calls go through helix_b200.Engine: a batch of chunks
embedded, and driven sequences of a state-space layer stack (prompt portions, a turn of prompt and decoded tokens, the exact mode).
"""
import math

import numpy as np
import torch

from helix_b200 import Engine, EngineConfig, configs, lib
from helix_b200 import engine as E

BF = torch.bfloat16
EPI = {"none": 0, "bias_gelu": 2, "resid": 3, "swiglu": 5}


def listed():
    return [
        # the down projection of a step in which running sequences decode beside a prompt portion (512 tokens: the serving default)
        dict(name="proj_mixed_step", kind="gemm", m=512, n=4096, k=14336, epi="resid"),
        # the gate / up projection of a prompt step, the largest product of a decoder layer
        dict(name="proj_gate_up", kind="gemm", m=8000, n=28672, k=4096, epi="swiglu"),
        # prompts of a chat batch: causal grouped-query attention over packed sequences of unequal length
        dict(name="attn_prompts", kind="attn", seqs=6, shortest=300, longest=3000, hq=32, hkv=8, d=128, causal=True),
        # the encoder's attention over chunks of documents
        dict(name="attn_encoder", kind="attn", seqs=64, shortest=64, longest=512, hq=12, hkv=12, d=64, causal=False),
        # a long prompt taken in portions: queries of one portion against the cached pages of everything before them
        dict(name="attn_portion", kind="portion", seqs=2, rows=777, ctx=6000, hq=32, hkv=8, d=128),
        # one decode step of 32 sequences with about 2k positions each
        dict(name="attn_tokens", kind="tokens", seqs=32, shortest=1500, longest=2176, hq=32, hkv=8, d=128, splits=1),
        # sampling of a decode step whose requests carry temperature, top_p and top_k
        dict(name="sample_filtered", kind="sample", rows=32, vocab=128256),
        # log-probabilities of the sampled token and of five alternatives for every row of a decode step
        dict(name="logprobs", kind="logprobs", rows=32, vocab=128256, width=6),
        # document chunks to embeddings: the whole encoder call
        dict(name="embed_chunks", kind="embed", chunks=48, shortest=64, longest=512),
        # prompts through one state-space layer with its feed-forward
        dict(name="ssm_prompts", kind="ssm", width=2048, layers=1, seqs=8, shortest=700, longest=2048, steps=0, f32=False),
        # a turn: short prompts, then decoded tokens one step at a time
        dict(name="ssm_turn", kind="ssm", width=1024, layers=2, seqs=16, shortest=40, longest=200, steps=12, f32=False),
        # a trace replayed in the exact number format
        dict(name="ssm_exact", kind="ssm", width=1024, layers=1, seqs=2, shortest=200, longest=400, steps=2, f32=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "attn", "encoder", "portion", "tokens", "sample", "logprobs", "embed", "ssm", "turn", "exact"])
    if kind == "gemm":
        n, k, epi = rng.choice([(4096, 4096, "resid"), (4096, 14336, "resid"), (28672, 4096, "swiglu"), (6144, 4096, "none"),
                                (2048, 8192, "resid"), (3072, 768, "bias_gelu"), (16384, 2048, "swiglu")])
        return dict(kind="gemm", m=_log_int(rng, 257, 8000), n=n, k=k, epi=epi)
    if kind == "attn":
        hq, hkv, d = rng.choice([(32, 8, 128), (32, 8, 64), (12, 2, 128)])
        longest = _log_int(rng, 65, 3000)
        return dict(kind="attn", seqs=rng.randint(1, 8), shortest=max(1, longest // 8), longest=longest, hq=hq, hkv=hkv, d=d, causal=True)
    if kind == "encoder":
        return dict(kind="attn", seqs=_log_int(rng, 1, 96), shortest=rng.randint(1, 64), longest=rng.randint(65, 512), hq=12, hkv=12, d=64, causal=False)
    if kind == "portion":
        hq, hkv, d = rng.choice([(32, 8, 128), (32, 8, 64)])
        return dict(kind="portion", seqs=rng.randint(1, 3), rows=_log_int(rng, 64, 2048), ctx=_log_int(rng, 2100, 7000), hq=hq, hkv=hkv, d=d)
    if kind == "tokens":
        hq, hkv, d = rng.choice([(32, 8, 128), (32, 8, 64)])
        seqs, longest = _log_int(rng, 1, 64), _log_int(rng, 200, 8000)
        longest = min(longest, 100000 // seqs)
        return dict(kind="tokens", seqs=seqs, shortest=max(1, longest // 2), longest=longest, hq=hq, hkv=hkv, d=d,
                    splits=max(1, min(16, -(-237 // (seqs * hkv)))))
    if kind == "sample":
        return dict(kind="sample", rows=_log_int(rng, 1, 128), vocab=rng.choice([128256, 151936, 32768]))
    if kind == "logprobs":
        return dict(kind="logprobs", rows=_log_int(rng, 1, 128), vocab=rng.choice([128256, 151936, 32768]), width=rng.randint(1, 21))
    if kind == "embed":
        return dict(kind="embed", chunks=_log_int(rng, 1, 64), shortest=rng.randint(1, 64), longest=rng.randint(65, 512))
    if kind == "ssm":
        longest = _log_int(rng, 300, 2048)
        return dict(kind="ssm", width=rng.choice([1024, 2048]), layers=1, seqs=rng.randint(1, 8), shortest=longest // 2, longest=longest, steps=0, f32=False)
    if kind == "turn":
        longest = rng.randint(10, 200)
        return dict(kind="ssm", width=1024, layers=rng.randint(1, 2), seqs=_log_int(rng, 1, 32), shortest=longest // 2, longest=longest, steps=rng.randint(2, 12),
                    f32=False)
    longest = rng.randint(20, 400)
    return dict(kind="ssm", width=rng.choice([512, 1024]), layers=1, seqs=rng.randint(1, 2), shortest=longest // 2, longest=longest, steps=rng.randint(1, 3),
                f32=True)


# ------------------------------------------------------------------ inputs
def _gen(seed, salt):
    return torch.Generator(device="cuda").manual_seed((int(seed) * 1000003 + salt * 7919) & 0x7FFFFFFF)


def _randn(seed, salt, shape, scale=1.0, mean=0.0, dtype=BF):
    return (torch.randn(shape, generator=_gen(seed, salt), device="cuda", dtype=torch.float32) * scale + mean).to(dtype)


def _lengths(case):
    """Unequal lengths between shortest and longest: part of the case, not of the seed, so that every seed is the same work."""
    n, lo, hi = case["seqs"] if "seqs" in case else case["chunks"], case["shortest"], case["longest"]
    return [lo + (hi - lo) * ((i * 7 + 3) % n) // max(1, n - 1) if n > 1 else hi for i in range(n)]


def _p(t):
    return t.data_ptr()


def _ok(rc):
    if rc != 0:
        raise RuntimeError(f"status {rc}: {lib().hbk_last_error().decode()}")


def _kernels():
    _ok(lib().hbk_init())


def _gemm_inputs(case, seed):
    m, n, k, epi = case["m"], case["n"], case["k"], case["epi"]
    s = dict(case=case, a=_randn(seed, 1, (m, k)), w=_randn(seed, 2, (n, k), k ** -0.5))
    s["r"] = _randn(seed, 3, (m, n)) if epi == "resid" else None
    s["bias"] = _randn(seed, 4, (n,), 0.5) if epi == "bias_gelu" else None
    s["out"] = torch.empty((m, n // 2 if epi == "swiglu" else n), device="cuda", dtype=BF)
    return s


def _attn_inputs(case, seed):
    lens, hq, hkv, d = _lengths(case), case["hq"], case["hkv"], case["d"]
    t = sum(lens)
    qkv = _randn(seed, 1, (t, (hq + 2 * hkv) * d))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), device="cuda", dtype=torch.int32)
    return dict(case=case, lens=lens, t=t, qkv=qkv, cu=cu, out=torch.empty((t, hq * d), device="cuda", dtype=BF))


def _paged_inputs(case, seed, ctx, rows):
    """ctx[b] cached positions per sequence in pages of 64 spread over the pool; q rows of `rows` tokens per sequence."""
    hq, hkv, d, b = case["hq"], case["hkv"], case["d"], len(ctx)
    pages = [(c + 63) // 64 for c in ctx]
    total = sum(pages)
    perm = torch.randperm(total, generator=_gen(seed, 9), device="cuda").to(torch.int32)
    table = torch.zeros((b, max(pages)), device="cuda", dtype=torch.int32)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = perm[at:at + n]
        at += n
    return dict(case=case, ctx=ctx, table=table, num_pages=total, k=_randn(seed, 2, (total, hkv, 64, d)), v=_randn(seed, 3, (total, hkv, 64, d)),
                q=_randn(seed, 1, (b * rows, hq * d)), lens=torch.tensor(ctx, device="cuda", dtype=torch.int32),
                out=torch.empty((b * rows, hq * d), device="cuda", dtype=BF))


def _logits(case, seed):
    """A decode step's logits: a broad bulk and a few dozen tokens that stand out."""
    rows, vocab = case["rows"], case["vocab"]
    x = _randn(seed, 1, (rows, vocab), 2.0, dtype=torch.float32)
    at = torch.randint(0, vocab, (rows, 40), generator=_gen(seed, 2), device="cuda")
    return x.scatter_add_(1, at, _randn(seed, 3, (rows, 40), 1.0, 6.0, dtype=torch.float32))


def _sample_inputs(case, seed):
    rows = case["rows"]
    kinds = [i % 4 for i in range(rows)]  # requests of a batch ask for different things
    f = lambda v, t: torch.tensor(v, device="cuda", dtype=t)  # noqa: E731
    return dict(case=case, logits=_logits(case, seed), temperature=f([0.7 if k != 3 else 0.1 for k in kinds], torch.float32),
                top_k=f([40 if k == 1 else 0 for k in kinds], torch.int32), top_p=f([0.95 if k == 0 else 0.9 if k == 1 else 1.0 if k == 2 else 0.8 for k in kinds], torch.float32),
                seeds=torch.randint(0, 1 << 62, (rows,), generator=_gen(seed, 5), device="cuda"), out=torch.empty(rows, device="cuda", dtype=torch.int32))


def _logprob_inputs(case, seed):
    rows, width = case["rows"], case["width"]
    x = _logits(case, seed)
    return dict(case=case, logits=x, sampled=x.argmax(1).to(torch.int32), width=torch.full((rows,), width, device="cuda", dtype=torch.int32),
                ids=torch.empty((rows, width), device="cuda", dtype=torch.int32), lps=torch.empty((rows, width), device="cuda", dtype=torch.float32))


class _Held:
    """A loaded engine that gives its memory back with the state that holds it."""

    def __init__(self, cfg, desc, weights):
        self.engine = Engine(cfg)
        self.engine.load_state_dict(desc, {k: v.float().cpu().numpy() for k, v in weights.items()})

    def __del__(self):
        self.engine.close()


def _tokens(seed, lens, vocab):
    rng = np.random.default_rng(seed)
    return [rng.integers(0, vocab, n).astype(np.int32) for n in lens]


def _encoder_weights(seed):
    d = configs.bge_base()
    h, f = d.hidden, d.ffn
    w = {"embeddings.word_embeddings.weight": _randn(seed, 1, (d.vocab, h), 0.05), "embeddings.position_embeddings.weight": _randn(seed, 2, (d.max_pos, h), 0.05),
         "embeddings.token_type_embeddings.weight": _randn(seed, 3, (d.type_vocab, h), 0.05), "embeddings.LayerNorm.weight": _randn(seed, 4, (h,), 0.05, 1.0),
         "embeddings.LayerNorm.bias": _randn(seed, 5, (h,), 0.02)}
    for i in range(d.layers):
        p, s = f"encoder.layer.{i}.", 100 * (i + 1)
        for j, (name, rows, cols) in enumerate((("attention.self.query", h, h), ("attention.self.key", h, h), ("attention.self.value", h, h),
                                                ("attention.output.dense", h, h), ("intermediate.dense", f, h), ("output.dense", h, f))):
            w[p + name + ".weight"] = _randn(seed, s + j, (rows, cols), 0.03)
            w[p + name + ".bias"] = _randn(seed, s + 20 + j, (rows,), 0.02)
        for j, name in enumerate(("attention.output.LayerNorm", "output.LayerNorm")):
            w[p + name + ".weight"] = _randn(seed, s + 40 + j, (h,), 0.05, 1.0)
            w[p + name + ".bias"] = _randn(seed, s + 50 + j, (h,), 0.02)
    return d, w


SSM_VOCAB = 4096


def _ssm_desc(case):
    w = case["width"]
    layers = [E.LayerDesc(mixer=E.MIXER_MAMBA2, heads=2 * w // 64, vdim=64, dim=128, kv_heads=8, norm_groups=8, conv_taps=4, ff_kind=E.FF_RELU2, ff=4 * w)
              for _ in range(case["layers"])]
    return E.StackDesc(width=w, vocab=SSM_VOCAB, layers=layers, compute_f32=int(case["f32"]), norm_eps=1e-5, resid_alpha=1.0, norm_place=E.NORM_PARALLEL,
                       embed_norm=1, plain_gains=1, tie_head=1)


def _ssm_weights(case, seed):
    w, d = case["width"], _ssm_desc(case)
    out = {"embed": _randn(seed, 1, (SSM_VOCAB, w), 0.5), "embed.norm": _randn(seed, 2, (w,), 0.1, 1.0), "final.norm": _randn(seed, 3, (w,), 0.1, 1.0)}
    for i, l in enumerate(d.layers):
        p, s = f"l{i}.", 100 * (i + 1)
        inner, ch = l.heads * l.vdim, l.heads * l.vdim + 2 * l.kv_heads * l.dim
        out[p + "norm1"], out[p + "norm2"] = _randn(seed, s, (w,), 0.1, 1.0), _randn(seed, s + 1, (w,), 0.1, 1.0)
        out[p + "mix.in"] = _randn(seed, s + 2, (inner + ch + l.heads, w), 1.5 * w ** -0.5)
        out[p + "mix.conv"], out[p + "mix.conv.b"] = _randn(seed, s + 3, (ch, l.conv_taps), 0.5), _randn(seed, s + 4, (ch,), 0.2)
        out[p + "mix.dt_bias"], out[p + "mix.A_log"] = _randn(seed, s + 5, (l.heads,), 0.5, -1.0), _randn(seed, s + 6, (l.heads,), 0.5, -1.0)
        out[p + "mix.D"], out[p + "mix.norm"] = _randn(seed, s + 7, (l.heads,), 0.3, 1.0), _randn(seed, s + 8, (inner,), 0.1, 1.0)
        out[p + "mix.o"] = _randn(seed, s + 9, (w, inner), inner ** -0.5)
        out[p + "mlp.up"], out[p + "mlp.down"] = _randn(seed, s + 10, (l.ff, w), 1.5 * w ** -0.5), _randn(seed, s + 11, (w, l.ff), l.ff ** -0.5)
    return d, out


def _ssm_wanted(n):
    return list(range(max(0, n - 4), n))  # a prompt's last positions


def _ssm_inputs(case, seed):
    lens = _lengths(case)
    desc, weights = _ssm_weights(case, seed)
    longest = -(-(max(lens) + case["steps"]) // 64) * 64
    cfg = EngineConfig(max_seqs=len(lens), max_ctx=longest, max_batched_tokens=max(512, sum(lens)), kv_pool_tokens=longest * len(lens))
    return dict(case=case, held=_Held(cfg, desc, weights), prompts=_tokens(seed, lens, SSM_VOCAB),
                follow=_tokens(seed + 1000003, [len(lens)] * case["steps"], SSM_VOCAB))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "embed":
        desc, weights = _encoder_weights(seed)
        lens = _lengths(case)
        held = _Held(EngineConfig(max_seqs=64, max_ctx=512, max_batched_tokens=16384), desc, weights)
        return dict(case=case, held=held, seqs=_tokens(seed, lens, desc.vocab))
    if kind == "ssm":
        return _ssm_inputs(case, seed)
    _kernels()
    if kind == "gemm":
        return _gemm_inputs(case, seed)
    if kind == "attn":
        return _attn_inputs(case, seed)
    if kind == "portion":
        ctx = [case["ctx"] - 61 * i for i in range(case["seqs"])]
        s = _paged_inputs(case, seed, ctx, case["rows"])
        s["cu"] = torch.arange(case["seqs"] + 1, device="cuda", dtype=torch.int32) * case["rows"]
        return s
    if kind == "tokens":
        s = _paged_inputs(case, seed, _lengths(case), 1)
        n = lib().hbk_attn_decode_workspace_floats(case["seqs"], case["hq"], case["d"], case["splits"])
        s["ws"] = torch.empty(max(1, n), device="cuda", dtype=torch.float32)
        return s
    if kind == "sample":
        return _sample_inputs(case, seed)
    return _logprob_inputs(case, seed)


# ------------------------------------------------------------------ one pass
def run(state):
    c, l = state["case"], lib()
    kind = c["kind"]
    if kind == "gemm":
        r, bias, out = state["r"], state["bias"], state["out"]
        _ok(l.hbk_gemm(_p(state["a"]), c["k"], _p(state["w"]), c["k"], _p(out), out.shape[1], _p(r) if r is not None else None, c["n"],
                       _p(bias) if bias is not None else None, c["m"], c["n"], c["k"], EPI[c["epi"]], 0))
        return out
    if kind == "attn":
        hq, hkv, d = c["hq"], c["hkv"], c["d"]
        ld, q = (hq + 2 * hkv) * d, _p(state["qkv"])
        _ok(l.hbk_attn_prefill(q, ld, q + 2 * hq * d, ld, q + 2 * (hq + hkv) * d, ld, _p(state["out"]), hq * d, _p(state["cu"]), len(state["lens"]), state["t"],
                               max(state["lens"]), hq, hkv, d, int(c["causal"]), d ** -0.5))
        return state["out"]
    if kind == "portion":
        hq, hkv, d, b = c["hq"], c["hkv"], c["d"], c["seqs"]
        _ok(l.hbk_attn_prefill_paged(_p(state["q"]), hq * d, _p(state["k"]), _p(state["v"]), _p(state["table"]), state["table"].shape[1], _p(state["lens"]),
                                     _p(state["out"]), hq * d, _p(state["cu"]), b, b * c["rows"], c["rows"], hq, hkv, d, 1, d ** -0.5, state["num_pages"]))
        return state["out"]
    if kind == "tokens":
        hq, hkv, d = c["hq"], c["hkv"], c["d"]
        _ok(l.hbk_attn_decode(_p(state["q"]), hq * d, _p(state["k"]), _p(state["v"]), _p(state["table"]), state["table"].shape[1], _p(state["lens"]),
                              _p(state["out"]), hq * d, _p(state["ws"]), c["seqs"], hq, hkv, d, 64, c["splits"], d ** -0.5, state["num_pages"]))
        return state["out"]
    if kind == "sample":
        _ok(l.hbk_sample_filtered(_p(state["logits"]), c["vocab"], _p(state["temperature"]), _p(state["seeds"]), _p(state["top_k"]), _p(state["top_p"]),
                                  _p(state["out"]), c["rows"], c["vocab"]))
        return state["out"]
    if kind == "logprobs":
        _ok(l.hbk_logprob_topk(_p(state["logits"]), c["vocab"], c["vocab"], _p(state["sampled"]), _p(state["width"]), _p(state["ids"]), _p(state["lps"]),
                               c["rows"], c["width"]))
        return dict(ids=state["ids"], logprobs=state["lps"])
    e = state["held"].engine
    if kind == "embed":
        return e.embed(state["seqs"])
    seqs = [e.seq_open() for _ in state["prompts"]]
    out = [e.seq_step([(s, t, _ssm_wanted(len(t))) for s, t in zip(seqs, state["prompts"])])]
    for toks in state["follow"]:
        out.append(e.seq_step([(s, toks[i:i + 1], [0]) for i, s in enumerate(seqs)]))
    for s in seqs:
        e.seq_close(s)
    return out


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        outs = n // 2 if case["epi"] == "swiglu" else n * (2 if case["epi"] == "resid" else 1)
        return {"bytes": 2 * (m * k + n * k + m * outs), "flops": 2.0 * m * n * k}
    if kind == "attn":
        lens, hq, hkv, d = _lengths(case), case["hq"], case["hkv"], case["d"]
        pairs = sum(x * (x + 1) // 2 if case["causal"] else x * x for x in lens)
        return {"bytes": 2 * sum(lens) * (2 * hq + 2 * hkv) * d, "flops": 4.0 * pairs * d * hq}
    if kind == "portion":
        hq, hkv, d, r = case["hq"], case["hkv"], case["d"], case["rows"]
        ctx = [case["ctx"] - 61 * i for i in range(case["seqs"])]
        pairs = sum(r * c - r * (r - 1) // 2 for c in ctx)
        return {"bytes": 2 * d * (2 * hq * r * len(ctx) + 2 * hkv * sum(ctx)), "flops": 4.0 * pairs * d * hq}
    if kind == "tokens":
        ctx, d = sum(_lengths(case)), case["d"]
        return {"bytes": 2 * d * (2 * case["hkv"] * ctx + 2 * case["hq"] * case["seqs"]), "flops": 4.0 * ctx * d * case["hq"]}
    if kind in ("sample", "logprobs"):
        return {"bytes": 4 * case["rows"] * case["vocab"], "flops": 0}
    lens = _lengths(case)
    if kind == "embed":
        d = configs.bge_base()
        per = 2 * d.layers * (4 * d.hidden * d.hidden + 2 * d.hidden * d.ffn)
        weights = 2 * (per // 2 + sum(lens) * d.hidden)
        return {"bytes": weights, "flops": float(per * sum(lens) + 4 * d.layers * d.hidden * sum(x * x for x in lens))}
    w, n = case["width"], sum(lens) + len(lens) * case["steps"]
    l = _ssm_desc(case).layers[0]
    inner = l.heads * l.vdim
    weights = w * (2 * inner + 2 * l.kv_heads * l.dim + l.heads) + w * inner + 2 * w * l.ff
    head = SSM_VOCAB * w * sum(min(4, x) + case["steps"] for x in lens)
    state = 2 * 4 * inner * l.dim * len(lens) * case["steps"]
    byte = (4 if case["f32"] else 2) * (weights * case["layers"] + SSM_VOCAB * w) * (1 + case["steps"]) + state * case["layers"]
    return {"bytes": byte, "flops": float(case["layers"] * n * (2 * weights + 6 * inner * l.dim) + 2 * head)}


def tolerance(case):
    kind = case["kind"]
    # about four times the distance from exact() that was seen: one rounding of bf16 outputs, bf16 probabilities, a whole encoder
    if kind == "gemm":
        return {"rel": 7e-3}
    if kind in ("attn", "portion", "tokens"):
        return {"rel": 1e-2}
    if kind == "sample":
        return "exact"
    if kind == "logprobs":
        return {"rel": 5e-7}
    if kind == "embed":
        return {"rel": 3e-2}
    return {"rel": 8e-6} if case["f32"] else {"rel": 1.5e-2}


# ------------------------------------------------------------------ the same in 64 bits
def _softmax_attention(q, k, v, scale, first):
    """q [n, H, D], k / v [m, G, D] in 64 bits; query i sees the keys up to position first + i (all of them: first None)."""
    n, hq, d = q.shape
    out = torch.empty_like(q)
    for h in range(hq):
        g = h // (hq // k.shape[1])
        s = q[:, h] @ k[:, g].T * scale
        if first is not None:
            s.masked_fill_(torch.arange(k.shape[0], device=s.device)[None] > first + torch.arange(n, device=s.device)[:, None], -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, g]
    return out


def _pages_of(s, b):
    """Keys and values of sequence b in order of position, 64 bits."""
    n = s["ctx"][b]
    at = s["table"][b, :(n + 63) // 64].long()
    flat = lambda t: t[at].permute(0, 2, 1, 3).reshape(-1, t.shape[1], t.shape[3])[:n].double()  # noqa: E731
    return flat(s["k"]), flat(s["v"])


def _norm_rows(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _ssm_layer(x, p, l, eps):
    """One layer over padded rows x [B, T, W]."""
    b, t, _ = x.shape
    f = torch.nn.functional
    inner, gn, h, n = l.heads * l.vdim, l.kv_heads * l.dim, l.heads, l.dim
    zx = _norm_rows(x, p["norm1"], eps) @ p["mix.in"].T
    z, u, dt = zx[..., :inner], zx[..., inner:2 * inner + 2 * gn], zx[..., 2 * inner + 2 * gn:]
    pad = f.pad(u, (0, 0, l.conv_taps - 1, 0))
    u = f.silu(sum(p["mix.conv"][:, j] * pad[:, j:j + t] for j in range(l.conv_taps)) + p["mix.conv.b"])
    v = u[..., :inner].reshape(b, t, h, l.vdim)
    rep = lambda m: m.reshape(b, t, l.kv_heads, n).repeat_interleave(h // l.kv_heads, 2)  # noqa: E731
    k, q = rep(u[..., inner:inner + gn]), rep(u[..., inner + gn:])
    dt = f.softplus(dt + p["mix.dt_bias"])
    a = torch.exp(-torch.exp(p["mix.A_log"]) * dt)
    s, y = torch.zeros((b, h, n, l.vdim), device=x.device, dtype=x.dtype), torch.empty_like(v)
    for i in range(t):
        s.mul_(a[:, i, :, None, None]).add_((dt[:, i, :, None] * k[:, i])[..., None] * v[:, i, :, None, :])
        y[:, i] = torch.einsum("bhn,bhnv->bhv", q[:, i], s)
    y = (y + p["mix.D"][:, None] * v).reshape(b, t, inner) * f.silu(z)
    y = _norm_rows(y.reshape(b, t, l.norm_groups, -1), 1.0, eps).reshape(b, t, inner) * p["mix.norm"]
    m = torch.relu(_norm_rows(x, p["norm2"], eps) @ p["mlp.up"].T) ** 2
    return x + y @ p["mix.o"].T + m @ p["mlp.down"].T


def _ssm_exact(case, seed):
    lens = _lengths(case)
    desc, weights = _ssm_weights(case, seed)
    w = {k: v.double() for k, v in weights.items()}
    prompts, follow = _tokens(seed, lens, SSM_VOCAB), _tokens(seed + 1000003, [len(lens)] * case["steps"], SSM_VOCAB)
    whole = [np.concatenate([t] + [f[i:i + 1] for f in follow]) for i, t in enumerate(prompts)]
    t = max(len(x) for x in whole)
    toks = torch.tensor(np.stack([np.pad(x, (0, t - len(x))) for x in whole]), device="cuda", dtype=torch.long)
    x = _norm_rows(w["embed"][toks], w["embed.norm"], desc.norm_eps)
    for i, l in enumerate(desc.layers):
        x = _ssm_layer(x, {k[len(f"l{i}."):]: v for k, v in w.items() if k.startswith(f"l{i}.")}, l, desc.norm_eps)
    x = _norm_rows(x, w["final.norm"], desc.norm_eps)
    out = [torch.cat([x[i, _ssm_wanted(n)] @ w["embed"].T for i, n in enumerate(lens)])]
    for j in range(case["steps"]):
        out.append(torch.stack([x[i, n + j] for i, n in enumerate(lens)]) @ w["embed"].T)
    return out


def _embed_exact(case, seed):
    d, weights = _encoder_weights(seed)
    w = {k: v.double() for k, v in weights.items()}
    f = torch.nn.functional
    norm = lambda x, p: f.layer_norm(x, (d.hidden,), w[p + ".weight"], w[p + ".bias"], d.norm_eps)  # noqa: E731
    lin = lambda x, p: x @ w[p + ".weight"].T + w[p + ".bias"]  # noqa: E731
    out = []
    for toks in _tokens(seed, _lengths(case), d.vocab):
        n = len(toks)
        x = w["embeddings.word_embeddings.weight"][torch.tensor(toks, device="cuda", dtype=torch.long)] + w["embeddings.position_embeddings.weight"][:n] + \
            w["embeddings.token_type_embeddings.weight"][0]
        x = norm(x, "embeddings.LayerNorm")
        for i in range(d.layers):
            p = f"encoder.layer.{i}."
            q, k, v = (lin(x, p + "attention.self." + m).reshape(n, d.heads, -1).transpose(0, 1) for m in ("query", "key", "value"))
            a = torch.softmax(q @ k.transpose(1, 2) * d.head_dim ** -0.5, -1) @ v
            x = norm(lin(a.transpose(0, 1).reshape(n, -1), p + "attention.output.dense") + x, p + "attention.output.LayerNorm")
            x = norm(lin(f.gelu(lin(x, p + "intermediate.dense")), p + "output.dense") + x, p + "output.LayerNorm")
        out.append(x[0] / x[0].norm())
    return torch.stack(out)


def exact(case, seed):
    kind = case["kind"]
    if kind == "gemm":
        s = _gemm_inputs(case, seed)
        out = []
        for rows in range(0, case["m"], 1024):  # in pieces: the 64-bit copies of the largest product stay small
            x = s["a"][rows:rows + 1024].double() @ s["w"].double().T
            if case["epi"] == "resid":
                x += s["r"][rows:rows + 1024].double()
            elif case["epi"] == "bias_gelu":
                x = torch.nn.functional.gelu(x + s["bias"].double())
            elif case["epi"] == "swiglu":
                g = x.view(x.shape[0], -1, 2, 128)
                x = (torch.nn.functional.silu(g[:, :, 0]) * g[:, :, 1]).reshape(x.shape[0], -1)
            out.append(x)
        return torch.cat(out)
    if kind == "attn":
        s, hq, hkv, d = _attn_inputs(case, seed), case["hq"], case["hkv"], case["d"]
        out, at = [], 0
        for n in s["lens"]:
            x = s["qkv"][at:at + n].double().view(n, hq + 2 * hkv, d)
            out.append(_softmax_attention(x[:, :hq], x[:, hq:hq + hkv], x[:, hq + hkv:], d ** -0.5, 0 if case["causal"] else None).reshape(n, -1))
            at += n
        return torch.cat(out)
    if kind in ("portion", "tokens"):
        rows = case["rows"] if kind == "portion" else 1
        s = prepare(case, seed)
        q = s["q"].double().view(case["seqs"], rows, case["hq"], case["d"])
        return torch.cat([_softmax_attention(q[b], *_pages_of(s, b), case["d"] ** -0.5, s["ctx"][b] - rows).reshape(rows, -1) for b in range(case["seqs"])])
    if kind == "sample":
        return None
    if kind == "logprobs":
        s = _logprob_inputs(case, seed)
        lp = torch.log_softmax(s["logits"].double(), -1)
        top = torch.topk(lp, max(1, case["width"] - 1), dim=-1).values[:, :case["width"] - 1]
        return dict(ids=None, logprobs=torch.cat([lp.gather(1, s["sampled"].long()[:, None]), top], 1))
    return _embed_exact(case, seed) if kind == "embed" else _ssm_exact(case, seed)
