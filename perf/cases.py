"""The work this engine is measured on: requests through the engine, and the operators that carry them, at the sizes of its named models.

Kinds of case (field ``kind``):
  serve      requests through :class:`LLMEngine`: prompts of one batch, then decoding with given tokens, logits of every step.  Layers
             of the named dense models (two of them, so that layers and not the head are the work), bf16 or Q4_K / Q6_K weights.
  attention  ``ops.attention`` over a paged cache with shuffled pages: prompts (also behind a cached prefix) and decode batches, the head geometries
             of gpt-oss (64 / 8 heads of 64 with sinks, alternately with a window of 128), Llama-3-8B (32 / 8 of 128) and Qwen3-Next (16 / 2 of 256)
  linear     ``ops.linear``: projections of those models for one row, for the rows of a decode batch and for prompts
  moe        an expert layer (``MoEFFN``: router, packing, experts, sum) with the residual norm that consumes it: MXFP4 experts of gpt-oss, Q8_0
             experts of Qwen3-Next / Qwen3-MoE
  deltanet   the mixer of a Qwen3-Next linear layer between its projections: convolution, gated delta rule, gated head norm
"""
import math

import torch

from machx_inference_engine_b200 import ops
from machx_inference_engine_b200.formats.gguf import GGMLType
from machx_inference_engine_b200.formats.model_config import ModelConfig
from machx_inference_engine_b200.models.transformer import MoEFFN, TransformerModel
from machx_inference_engine_b200.ops.cuda import rmsnorm_combine
from machx_inference_engine_b200.parallel.comm import ParallelCtx
from machx_inference_engine_b200.runtime.engine import EngineOptions, LLMEngine

PAGE = 128
DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    small = dict(hidden=2048, heads=32, kv_heads=8, head_dim=64, ffn=8192, vocab=32768, layers=2)
    large = dict(hidden=4096, heads=32, kv_heads=8, head_dim=128, ffn=14336, vocab=32768, layers=2)
    oss = dict(heads=64, kv_heads=8, head_dim=64, sinks=True)
    llama = dict(heads=32, kv_heads=8, head_dim=128, sinks=False)
    return [
        # one short chat turn on a small model: launches and latencies
        dict(name="serve_chat_small", kind="serve", **small, quant="bf16", seqs=1, prompt_lo=75, prompt_hi=75, steps=16),
        # one user of a quantised 8B-class model: a prompt of some hundred tokens, then single-token steps
        dict(name="serve_q4_one_user", kind="serve", **large, quant="q4_k_m", seqs=1, prompt_lo=700, prompt_hi=700, steps=24),
        # sixteen requests of different lengths arriving together at an 8B-class model
        dict(name="serve_batch", kind="serve", **large, quant="bf16", seqs=16, prompt_lo=64, prompt_hi=640, steps=16),
        # a whole 4096-token prompt on a full-attention layer of gpt-oss
        dict(name="attn_prompt_oss", kind="attention", **oss, seqs=1, new_lo=4096, new_hi=4096, past_lo=0, past_hi=0, window=0, kv="bf16"),
        # prompts of different lengths, some behind a cached prefix
        dict(name="attn_prompts_ragged", kind="attention", **llama, seqs=6, new_lo=200, new_hi=3000, past_lo=0, past_hi=4096, window=0, kv="bf16"),
        # the decode step of 64 concurrent gpt-oss requests
        dict(name="attn_decode_64", kind="attention", **oss, seqs=64, new_lo=1, new_hi=1, past_lo=256, past_hi=4096, window=0, kv="bf16"),
        # a few users with long documents
        dict(name="attn_decode_long", kind="attention", **llama, seqs=4, new_lo=1, new_hi=1, past_lo=16000, past_hi=32000, window=0, kv="bf16"),
        # gate and up projection of a 4096-token prompt, Llama-3-8B
        dict(name="linear_prompt", kind="linear", rows=4096, n=28672, k=4096, quant="bf16", act="swiglu"),
        # qkv projection of a decode batch of 40
        dict(name="linear_batch", kind="linear", rows=40, n=6144, k=4096, quant="bf16", act="none"),
        # expert layer of gpt-oss-20b over a 2048-token prompt
        dict(name="moe_prompt_mxfp4", kind="moe", tokens=2048, hidden=2880, ffn=2880, experts=32, topk=4, quant="mxfp4"),
        # expert layer of Qwen3-Next-80B (Q8_0) over a 1000-token prompt
        dict(name="moe_prompt_q8", kind="moe", tokens=1000, hidden=2048, ffn=512, experts=512, topk=10, quant="q8_0"),
        # linear layer of Qwen3-Next-80B over two prompts
        dict(name="deltanet_prompt", kind="deltanet", seqs=2, new_lo=1500, new_hi=2600, n_k=16, n_v=32),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["serve"] * 3 + ["prompt"] * 2 + ["decode"] * 2 + ["linear"] * 2 + ["moe"] * 2 + ["deltanet"])
    if kind == "serve":
        size = rng.choice([dict(hidden=2048, heads=32, kv_heads=8, head_dim=64, ffn=8192), dict(hidden=4096, heads=32, kv_heads=8, head_dim=128, ffn=14336)])
        seqs = rng.choice([1, 1, 2, 3, 5, 8, 13, 16])
        hi = min(2048, max(40, _log_int(rng, 40, 8000) // seqs))
        return dict(kind="serve", **size, vocab=32768, layers=2, quant=rng.choice(["bf16", "q4_k_m"]), seqs=seqs, prompt_lo=max(17, hi // rng.choice([1, 4])),
                    prompt_hi=max(17, hi), steps=rng.randint(8, 24))
    if kind in ("prompt", "decode"):
        heads, kv_heads, hd, sinks = rng.choice([(64, 8, 64, True), (32, 8, 128, False), (16, 2, 256, False)])
        window = rng.choice([0, 128]) if sinks else 0
        base = dict(kind="attention", heads=heads, kv_heads=kv_heads, head_dim=hd, sinks=sinks, window=window)
        if kind == "prompt":
            seqs = rng.choice([1, 1, 2, 4, 7])
            new = max(65, _log_int(rng, 100, 6000) // seqs)
            past = rng.choice([0, 0, rng.randint(1, 4000)])
            return dict(base, seqs=seqs, new_lo=max(65, new // rng.choice([1, 5])), new_hi=new, past_lo=past // 2, past_hi=past, kv="bf16")
        seqs = rng.choice([1, 2, 4, 7, 16, 31, 64])
        past = min(40000, _log_int(rng, 60, 200000 // seqs))
        return dict(base, seqs=seqs, new_lo=1, new_hi=1, past_lo=max(1, past // rng.choice([1, 8])), past_hi=past, kv=rng.choice(["bf16", "bf16", "bf16", "int8"]))
    if kind == "linear":
        n, k, act = rng.choice([(6144, 4096, "none"), (4096, 4096, "none"), (28672, 4096, "swiglu"), (4096, 14336, "none"), (5120, 2880, "none"),
                                (2880, 4096, "none"), (12288, 2048, "none"), (2048, 8192, "none")])
        quant = rng.choice(["bf16", "bf16", "bf16", "q8_0", "q4_k"])
        if quant == "q4_k" and k % 256:
            quant = "q8_0"
        return dict(kind="linear", rows=_log_int(rng, 1, 4096), n=n, k=k, quant=quant, act=act)
    if kind == "moe":
        hidden, ffn, experts, topk, quant = rng.choice([(2880, 2880, 32, 4, "mxfp4"), (2880, 2880, 128, 4, "mxfp4"), (2048, 512, 512, 10, "q8_0"),
                                                        (2048, 768, 128, 8, "q8_0")])
        return dict(kind="moe", tokens=_log_int(rng, 1, 4096), hidden=hidden, ffn=ffn, experts=experts, topk=topk, quant=quant)
    seqs = rng.choice([1, 2, 3, 8, 30])
    new = rng.choice([1, max(2, _log_int(rng, 64, 5000) // seqs)])
    return dict(kind="deltanet", seqs=seqs, new_lo=max(1, new // rng.choice([1, 3])), new_hi=new, n_k=16, n_v=rng.choice([32, 48]))


# ------------------------------------------------------------------ weights: ggml payloads, as a checkpoint holds them, and their values in 64 bits
def _gen(seed, name):
    h = 14695981039346656037
    for ch in f"{seed}/{name}".encode():
        h = ((h ^ ch) * 1099511628211) & ((1 << 62) - 1)
    return torch.Generator(device=DEV).manual_seed(h)


def _randn(g, *shape, std=1.0):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float32) * std


def _bytes(g, *shape):
    return torch.randint(0, 256, shape, generator=g, device=DEV, dtype=torch.uint8)


def _half_bytes(v):
    return v.to(torch.float16).unsqueeze(-1).view(torch.uint8)


FORMATS = {"bf16": GGMLType.BF16, "q8_0": GGMLType.Q8_0, "q4_k": GGMLType.Q4_K, "q6_k": GGMLType.Q6_K, "mxfp4": GGMLType.MXFP4}
BLOCK_BYTES = {"bf16": (1, 2), "q8_0": (32, 34), "q4_k": (256, 144), "q6_k": (256, 210), "mxfp4": (32, 17)}
FP4 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0)


def weight_payload(g, quant, rows, k):
    """uint8 [rows, bytes per row]: random blocks whose values have a standard deviation near 0.02."""
    if quant == "bf16":
        return _randn(g, rows, k, std=0.02).to(torch.bfloat16).view(torch.uint8)
    if quant == "q8_0":
        codes = _randn(g, rows, k // 32, 32, std=42.0).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
        d = _half_bytes(torch.rand(rows, k // 32, generator=g, device=DEV) * 2e-4 + 3.8e-4)
        return torch.cat([d, codes], dim=-1).reshape(rows, -1)
    if quant == "mxfp4":
        e = torch.randint(119, 122, (rows, k // 32, 1), generator=g, device=DEV, dtype=torch.uint8)
        return torch.cat([e, _bytes(g, rows, k // 32, 16)], dim=-1).reshape(rows, -1)
    if quant == "q4_k":            # minima in step with the scales, so that blocks are centred as fitted ones are
        nb = k // 256
        s = torch.randint(16, 64, (rows, nb, 8), generator=g, device=DEV, dtype=torch.uint8)
        d = torch.rand(rows, nb, generator=g, device=DEV) * 4e-5 + 9e-5
        lo, hi = s[..., :4], s[..., 4:]
        a = lo | ((hi >> 4) << 6)
        return torch.cat([_half_bytes(d), _half_bytes(7.5 * d.to(torch.float16).float()), a, a, (hi & 15) | ((hi & 15) << 4), _bytes(g, rows, nb, 128)], dim=-1).reshape(rows, -1)
    nb = k // 256                  # q6_k
    sc = torch.randint(20, 110, (rows, nb, 16), generator=g, device=DEV, dtype=torch.int8).view(torch.uint8)
    d = torch.rand(rows, nb, generator=g, device=DEV) * 8e-6 + 1.2e-5
    return torch.cat([_bytes(g, rows, nb, 192), sc, _half_bytes(d)], dim=-1).reshape(rows, -1)


def weight_values(raw, quant, rows, k):
    """The same rows in 64 bits (the public ggml block formats)."""
    if quant == "bf16":
        return raw.view(torch.bfloat16).double()
    f16 = lambda b: b.contiguous().view(torch.float16).double()
    if quant == "q8_0":
        b = raw.reshape(rows, k // 32, 34)
        return (f16(b[..., :2]) * b[..., 2:].contiguous().view(torch.int8).double()).reshape(rows, k)
    if quant == "mxfp4":
        b = raw.reshape(rows, k // 32, 17)
        table = torch.tensor(FP4, dtype=torch.float64, device=raw.device)
        q = b[..., 1:].long()
        return (torch.cat([table[q & 15], table[q >> 4]], dim=-1) * torch.exp2(b[..., :1].double() - 127.0)).reshape(rows, k)
    nb = k // 256
    if quant == "q4_k":
        b = raw.reshape(rows, nb, 144)
        d, dm, s = f16(b[..., 0:2]), f16(b[..., 2:4]), b[..., 4:16].int()
        lo, hi, tail = s[..., 0:4], s[..., 4:8], s[..., 8:12]
        sc = torch.cat([lo & 63, (tail & 15) | ((lo >> 6) << 4)], dim=-1).double()
        mn = torch.cat([hi & 63, (tail >> 4) | ((hi >> 6) << 4)], dim=-1).double()
        q = b[..., 16:].reshape(rows, nb, 4, 32)
        q = torch.stack([q & 15, q >> 4], dim=-2).reshape(rows, nb, 8, 32).double()
        return (q * (d * sc).unsqueeze(-1) - (dm * mn).unsqueeze(-1)).reshape(rows, k)
    b = raw.reshape(rows, nb, 210)
    ql, qh = b[..., :128].int().reshape(rows, nb, 2, 2, 32), b[..., 128:192].int().reshape(rows, nb, 2, 1, 32)
    low = torch.cat([ql & 15, ql >> 4], dim=-2)
    high = (qh >> torch.tensor([0, 2, 4, 6], device=raw.device).reshape(4, 1)) & 3
    q = ((low | (high << 4)) - 32).double().reshape(rows, nb, 16, 16)
    sc = b[..., 192:208].contiguous().view(torch.int8).double()
    return (q * (f16(b[..., 208:210]) * sc).unsqueeze(-1)).reshape(rows, k)


class Weights:
    """A checkpoint of random blocks under the names the graphs ask for: payloads for the engine, the same in 64 bits for the comparison."""

    def __init__(self, seed, recipe):
        self.seed, self.recipe = seed, recipe

    def quant(self, name):
        if self.recipe == "q4_k_m":        # Q6_K head, and Q6_K values and down projections in the first layers
            more = name == "output.weight" or (name.startswith("blk.0.") and name.split(".")[2] in ("attn_v", "ffn_down"))
            return "q6_k" if more else "q4_k"
        if self.recipe in ("mxfp4", "q8_0"):
            return self.recipe if "_exps" in name else "bf16"
        return self.recipe

    def has(self, name):
        return True

    def payload(self, name, n, k, e=0):
        return weight_payload(_gen(self.seed, f"{name}#{e}"), self.quant(name), n, k)

    def matrix(self, name, n, k, E=1, experts=None):
        raw = torch.cat([self.payload(name, n, k, e) for e in range(E)]) if E > 1 else self.payload(name, n, k)
        return ops.from_ggml(raw.reshape(-1), FORMATS[self.quant(name)], n, k, E)

    def values(self, name, n, k, e=0):
        return weight_values(self.payload(name, n, k, e), self.quant(name), n, k)

    def vector(self, name, n):
        g = _gen(self.seed, name)
        return 1.0 + _randn(g, n, std=0.05) if "norm" in name else _randn(g, n, std=0.02)

    def table(self, name, shape):
        return _randn(_gen(self.seed, name), *shape, std=0.1)


def weight_bytes(quant, elements):
    n, size = BLOCK_BYTES[quant]
    return elements // n * size


def _spread(lo, hi, n, seed):
    """n lengths between lo and hi, the longest at hi: the same for every seed's inputs would time one batch only, so the order follows the seed."""
    v = [hi - (hi - lo) * i // max(n - 1, 1) for i in range(n)]
    order = torch.randperm(n, generator=torch.Generator().manual_seed(seed)).tolist()
    return [v[i] for i in order]


# ------------------------------------------------------------------ serve
def _serve_config(c):
    return ModelConfig(arch="llama", n_layers=c["layers"], hidden=c["hidden"], n_heads=c["heads"], n_kv_heads=c["kv_heads"], head_dim=c["head_dim"],
                       ffn=c["ffn"], vocab=c["vocab"], rms_eps=1e-5, rope_theta=500000.0, n_rot=c["head_dim"], ctx_train=8192)


def _serve_tokens(c, seed):
    g = torch.Generator().manual_seed(seed)
    lens = _spread(c["prompt_lo"], c["prompt_hi"], c["seqs"], seed)
    return [(torch.randint(0, c["vocab"], (n,), generator=g).tolist(), torch.randint(0, c["vocab"], (c["steps"],), generator=g).tolist()) for n in lens]


def _serve_prepare(c, seed):
    ctx = (c["prompt_hi"] + c["steps"] + 16 + PAGE - 1) // PAGE * PAGE
    model = TransformerModel(_serve_config(c), Weights(seed, c["quant"]), DEV, max_ctx=ctx)
    eng = LLMEngine(model, EngineOptions(max_ctx=ctx, max_batch_tokens=8192, max_seqs=c["seqs"]))
    return dict(kind="serve", eng=eng, tokens=_serve_tokens(c, seed))


def _serve_run(s):
    eng = s["eng"]
    seqs = [eng.open_sequence() for _ in s["tokens"]]
    first = eng.feed([(q, list(prompt), [len(prompt) - 1]) for q, (prompt, _) in zip(seqs, s["tokens"])])
    steps = [eng.feed([(q, [given[i]], [0]) for q, (_, given) in zip(seqs, s["tokens"])]) for i in range(len(s["tokens"][0][1]))]
    for q in seqs:
        eng.abort(q)
    return [first, torch.stack(steps)]


def _rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w.double()


def _serve_exact(c, seed):
    W, H, hd, nq, nkv = Weights(seed, c["quant"]), c["hidden"], c["head_dim"], c["heads"], c["kv_heads"]
    toks = _serve_tokens(c, seed)
    V, F = c["vocab"], c["ffn"]
    lens = [len(p) + len(g) for p, g in toks]
    ids = torch.tensor([t for p, g in toks for t in p + g], device=DEV)
    x = W.values("token_embd.weight", V, H)[ids]
    inv = 500000.0 ** (-torch.arange(0, hd, 2, device=DEV).double() / hd)

    def rope(t, n):
        a = torch.arange(n, device=DEV).double()[:, None, None] * inv
        lo, hi = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], dim=-1)

    for l in range(c["layers"]):
        p = f"blk.{l}"
        h = _rms(x, W.vector(f"{p}.attn_norm.weight", H), 1e-5)
        q, k, v = (h @ W.values(f"{p}.attn_{n}.weight", m * hd, H).T for n, m in (("q", nq), ("k", nkv), ("v", nkv)))
        outs = []
        for qs, ks, vs in zip(q.split(lens), k.split(lens), v.split(lens)):
            n = qs.shape[0]
            qs, ks, vs = rope(qs.view(n, nq, hd), n), rope(ks.view(n, nkv, hd), n), vs.view(n, nkv, hd)
            o = torch.nn.functional.scaled_dot_product_attention(qs.transpose(0, 1), ks.repeat_interleave(nq // nkv, 1).transpose(0, 1),
                                                                 vs.repeat_interleave(nq // nkv, 1).transpose(0, 1), is_causal=True)
            outs.append(o.transpose(0, 1).reshape(n, nq * hd))
        x = x + torch.cat(outs) @ W.values(f"{p}.attn_output.weight", H, nq * hd).T
        h = _rms(x, W.vector(f"{p}.ffn_norm.weight", H), 1e-5)
        a = torch.nn.functional.silu(h @ W.values(f"{p}.ffn_gate.weight", F, H).T) * (h @ W.values(f"{p}.ffn_up.weight", F, H).T)
        x = x + a @ W.values(f"{p}.ffn_down.weight", H, F).T
    hs = _rms(x, W.vector("output_norm.weight", H), 1e-5).split(lens)
    want = torch.stack([h[len(p) - 1:] for h, (p, _) in zip(hs, toks)], dim=1)          # [1 + steps, seqs, H]
    logits = want @ W.values("output.weight", V, H).T
    return [logits[0], logits[1:]]


def _serve_work(c):
    W, H, hd, nq, nkv, F = Weights(0, c["quant"]), c["hidden"], c["head_dim"], c["heads"], c["kv_heads"], c["ffn"]
    lens = _spread(c["prompt_lo"], c["prompt_hi"], c["seqs"], 0)
    wb = params = 0
    for l in range(c["layers"]):
        for n, el in (("attn_q", nq * hd * H), ("attn_k", nkv * hd * H), ("attn_v", nkv * hd * H), ("attn_output", nq * hd * H), ("ffn_gate", F * H),
                      ("ffn_up", F * H), ("ffn_down", F * H)):
            wb += weight_bytes(W.quant(f"blk.{l}.{n}.weight"), el)
            params += el
    head = c["vocab"] * H
    passes = 1 + c["steps"]
    cached = 4 * nkv * hd * c["layers"]
    kv = sum(cached * ((n + i) if i else n) for n in lens for i in range(passes))
    rows = sum(lens) + c["seqs"] * c["steps"]
    scores = sum(n * (n + 1) // 2 + sum(n + i for i in range(1, passes)) for n in lens)
    return {"bytes": passes * (wb + weight_bytes(W.quant("output.weight"), head)) + kv + passes * c["seqs"] * c["vocab"] * 4,
            "flops": 2.0 * params * rows + 2.0 * head * c["seqs"] * passes + 4.0 * nq * hd * scores * c["layers"]}


# ------------------------------------------------------------------ attention
def _attn_lens(c, seed):
    new, past = _spread(c["new_lo"], c["new_hi"], c["seqs"], seed), _spread(c["past_lo"], c["past_hi"], c["seqs"], seed + 1)
    return new, past


def _attn_inputs(c, seed):
    g = _gen(seed, "attention")
    new, past = _attn_lens(c, seed)
    lens = [a + b for a, b in zip(new, past)]
    pages = [(n + PAGE - 1) // PAGE for n in lens]
    total = sum(pages) + 1
    order = (torch.randperm(total - 1, generator=g, device=DEV) + 1).int()
    table = torch.zeros(len(lens), max(pages), dtype=torch.int32, device=DEV)
    at = 0
    for i, n in enumerate(pages):
        table[i, :n] = order[at:at + n]
        at += n
    shape = (total, c["kv_heads"], PAGE, c["head_dim"])
    s = dict(q=_randn(g, sum(new), c["heads"], c["head_dim"]).to(torch.bfloat16), table=table, lens=torch.tensor(lens, dtype=torch.int32, device=DEV),
             cu=torch.tensor([0] + new, device=DEV).cumsum(0).int(), longest=max(new), max_kv=max(lens), scales=None)
    if c["kv"] == "int8":
        s["k"], s["v"] = (_randn(g, *shape, std=40.0).round_().clamp_(-127, 127).to(torch.int8) for _ in "kv")
        s["scales"] = tuple(torch.rand(*shape[:3], generator=g, device=DEV) * 0.01 + 0.02 for _ in "kv")
    else:
        s["k"], s["v"] = (_randn(g, *shape).to(torch.bfloat16) for _ in "kv")
    s["sinks"] = _randn(g, c["heads"]) if c["sinks"] else None
    return s


def _attn_prepare(c, seed):
    return dict(_attn_inputs(c, seed), kind="attention", window=c["window"])


def _attn_run(s):
    return ops.attention(s["q"], s["k"], s["v"], s["table"], s["lens"], s["cu"], s["longest"], sinks=s["sinks"], window=s["window"], kv_scales=s["scales"],
                         max_kv_len=s["max_kv"])


def _attn_exact(c, seed):
    s = _attn_inputs(c, seed)
    new, past = _attn_lens(c, seed)
    hd, nkv = c["head_dim"], c["kv_heads"]
    gqa = c["heads"] // nkv
    out, t0 = [], 0
    for i, (n, p) in enumerate(zip(new, past)):
        L = n + p
        pages = s["table"][i, :(L + PAGE - 1) // PAGE].long()
        kv = []
        for j, t in enumerate((s["k"], s["v"])):
            t = t[pages].double()
            if s["scales"] is not None:
                t = t * s["scales"][j][pages].double().unsqueeze(-1)
            kv.append(t.transpose(0, 1).reshape(nkv, -1, hd)[:, :L])
        q = s["q"][t0:t0 + n].double().view(n, nkv, gqa, hd)
        for lo in range(0, n, 512):
            m = min(512, n - lo)
            sc = torch.einsum("qhgd,hkd->hgqk", q[lo:lo + m], kv[0]) / math.sqrt(hd)
            qp, kp = torch.arange(p + lo, p + lo + m, device=DEV)[:, None], torch.arange(L, device=DEV)[None]
            seen = (kp <= qp) & (kp > qp - c["window"]) if c["window"] else kp <= qp
            sc = sc.masked_fill(~seen, -math.inf)
            if s["sinks"] is not None:
                sk = s["sinks"].double().view(nkv, gqa, 1, 1).expand(-1, -1, m, 1)
                pr = torch.softmax(torch.cat([sc, sk], dim=-1), dim=-1)[..., :-1]
            else:
                pr = torch.softmax(sc, dim=-1)
            out.append(torch.einsum("hgqk,hkd->qhgd", pr, kv[1]).reshape(m, c["heads"], hd))
        t0 += n
    return torch.cat(out)


def _attn_work(c):
    new, past = _attn_lens(c, 0)
    w = c["window"] or 1 << 30
    keys = pairs = 0
    for n, p in zip(new, past):
        keys += min(n + p, n + w)
        full = max(0, min(n, w - 1 - p))            # queries whose window is not full yet
        pairs += sum(range(p + 1, p + full + 1)) + (n - full) * w if c["window"] else n * p + n * (n + 1) // 2
    row = c["kv_heads"] * (c["head_dim"] + 4 if c["kv"] == "int8" else c["head_dim"] * 2)
    return {"bytes": 2.0 * keys * row + 4.0 * sum(new) * c["heads"] * c["head_dim"], "flops": 4.0 * pairs * c["heads"] * c["head_dim"]}


# ------------------------------------------------------------------ linear
def _linear_x(c, seed):
    return _randn(_gen(seed, "x"), c["rows"], c["k"]).to(torch.bfloat16)


def _linear_prepare(c, seed):
    W = Weights(seed, c["quant"])
    if c["act"] == "swiglu":
        w = ops.QuantWeight.interleave_gate_up(*(ops.from_ggml(weight_payload(_gen(seed, n), c["quant"], c["n"] // 2, c["k"]).reshape(-1), FORMATS[c["quant"]],
                                                               c["n"] // 2, c["k"]) for n in ("gate", "up")))
    else:
        w = ops.from_ggml(weight_payload(_gen(seed, "w"), c["quant"], c["n"], c["k"]).reshape(-1), FORMATS[c["quant"]], c["n"], c["k"])
    return dict(kind="linear", x=_linear_x(c, seed), w=w, act=ops.ACT_SWIGLU if c["act"] == "swiglu" else ops.ACT_NONE)


def _linear_run(s):
    return ops.linear(s["x"], s["w"], act=s["act"])


def _linear_exact(c, seed):
    x = _linear_x(c, seed).double()
    value = lambda name, n: weight_values(weight_payload(_gen(seed, name), c["quant"], n, c["k"]), c["quant"], n, c["k"])
    if c["act"] == "swiglu":
        return torch.nn.functional.silu(x @ value("gate", c["n"] // 2).T) * (x @ value("up", c["n"] // 2).T)
    return x @ value("w", c["n"]).T


def _linear_work(c):
    out = c["n"] // 2 if c["act"] == "swiglu" else c["n"]
    return {"bytes": weight_bytes(c["quant"], c["n"] * c["k"]) + 2.0 * c["rows"] * (c["k"] + out), "flops": 2.0 * c["rows"] * c["n"] * c["k"]}


# ------------------------------------------------------------------ moe
def _moe_config(c):
    return ModelConfig(arch="gpt-oss" if c["quant"] == "mxfp4" else "qwen3moe", n_layers=1, hidden=c["hidden"], n_heads=64, n_kv_heads=8, head_dim=64,
                       ffn=c["ffn"], vocab=1024, n_experts=c["experts"], n_experts_used=c["topk"], expert_ffn=c["ffn"])


def _moe_inputs(c, seed):
    """Residual rows, what the block reads, and the next norm's weight.  The rows share a common part, so that some experts are chosen more often."""
    g = _gen(seed, "moe")
    x = _randn(g, c["tokens"], c["hidden"]) + 0.3 * _randn(g, 1, c["hidden"])
    return x, x.to(torch.bfloat16), 1.0 + _randn(g, c["hidden"], std=0.05)


def _moe_prepare(c, seed):
    oss = c["quant"] == "mxfp4"
    block = MoEFFN(_moe_config(c), 0, Weights(seed, c["quant"]), ParallelCtx(), ops.ACT_SWIGLU_OAI if oss else ops.ACT_SWIGLU, with_bias=oss)
    x, h, w = _moe_inputs(c, seed)
    return dict(kind="moe", block=block, par=ParallelCtx(), x=x, h=h, w=w)


def _moe_run(s):
    x = s["x"].clone()               # the residual stream of this pass: the norm adds the expert sum to it in place
    y = s["block"](s["h"], s["par"])
    n = ops.rmsnorm(x, s["w"], 1e-5, delta=y) if isinstance(y, torch.Tensor) else rmsnorm_combine(x, s["w"], 1e-5, y)
    return [x, n]


def _e4m3(x):
    """Rows as the block-scaled product takes them: e4m3 with a power-of-two scale per 32, the smallest that keeps the block in range."""
    b = x.reshape(*x.shape[:-1], -1, 32)
    amax = b.abs().amax(-1, keepdim=True).clamp_min(1e-38)
    ex = torch.floor(torch.log2(amax)) - 8.0
    ex = torch.where(amax * torch.exp2(-ex) > 448.0, ex + 1.0, ex)
    return ((b * torch.exp2(-ex)).float().to(torch.float8_e4m3fn).double() * torch.exp2(ex)).reshape(x.shape)


def _moe_exact(c, seed):
    W, (x, h, w) = Weights(seed, c["quant"]), _moe_inputs(c, seed)
    H, F, E, K, oss = c["hidden"], c["ffn"], c["experts"], c["topk"], c["quant"] == "mxfp4"
    p = "blk.0"
    logits = h.double() @ W.values(f"{p}.ffn_gate_inp.weight", E, H).T
    if oss:
        logits = logits + W.vector(f"{p}.ffn_gate_inp.bias", E).double()
        gb, ub, db = (W.table(f"{p}.ffn_{n}_exps.bias", (E, m)).double() for n, m in (("gate", F), ("up", F), ("down", H)))
    best, idx = torch.sort(logits, dim=-1, descending=True, stable=True)
    prob = torch.softmax(best[:, :K], dim=-1)
    idx = idx[:, :K]
    xin = _e4m3(h.double()) if oss else h.double()
    y = x.double()
    for e in range(E):
        t, slot = (idx == e).nonzero(as_tuple=True)
        if t.numel() == 0:
            continue
        g, u = (xin[t] @ W.values(f"{p}.ffn_{n}_exps.weight", F, H, e).T for n in ("gate", "up"))
        if oss:
            g, u = (g + gb[e]).clamp(max=7.0), (u + ub[e]).clamp(-7.0, 7.0)
            a = _e4m3(g * torch.sigmoid(1.702 * g) * (u + 1.0))
        else:
            a = torch.nn.functional.silu(g) * u
        o = a @ W.values(f"{p}.ffn_down_exps.weight", H, F, e).T
        if oss:
            o = o + db[e]
        y.index_add_(0, t, o * prob[t, slot, None])
    return [y, _rms(y, w, 1e-5)]


def _moe_work(c):
    H, F, E, T, K = c["hidden"], c["ffn"], c["experts"], c["tokens"], c["topk"]
    live = E * (1.0 - (1.0 - K / E) ** T)
    return {"bytes": live * weight_bytes(c["quant"], 3 * H * F) + 2.0 * E * H + T * H * (2.0 + 4.0 + 4.0 + 2.0), "flops": 2.0 * T * K * 3 * H * F + 2.0 * T * E * H}


# ------------------------------------------------------------------ deltanet
DN = 128


def _dn_inputs(c, seed):
    g = _gen(seed, "deltanet")
    new = _spread(c["new_lo"], c["new_hi"], c["seqs"], seed)
    T, B, nk, nv = sum(new), c["seqs"], c["n_k"], c["n_v"]
    C = (2 * nk + nv) * DN
    s = dict(new=new, x=_randn(g, T, C).to(torch.bfloat16), conv_w=_randn(g, C, 4, std=0.4), conv=_randn(g, B, 3, C).to(torch.bfloat16),
             ab=_randn(g, T, 2 * nv).to(torch.bfloat16), state=_randn(g, B, nv, DN, DN, std=0.05), z=_randn(g, T, nv * DN).to(torch.bfloat16),
             a=-torch.exp(_randn(g, nv, std=0.5)), dt=_randn(g, nv, std=0.2) - 1.0, w=1.0 + _randn(g, DN, std=0.05))
    at = torch.arange(nv, dtype=torch.int32, device=DEV)
    s.update(ai=at, bi=at + nv, kv=(at // (nv // nk)).int(), slots=torch.randperm(B, generator=g, device=DEV).int(),
             cu=torch.tensor([0] + new, device=DEV).cumsum(0).int(), longest=max(new), n_k=nk, n_v=nv)
    return s


def _dn_prepare(c, seed):
    return dict(_dn_inputs(c, seed), kind="deltanet")


def _dn_run(s):
    conv, state = s["conv"].clone(), s["state"].clone()          # the recurrent state of this pass: both operators advance theirs in place
    y = ops.conv1d_silu(s["x"], s["conv_w"], conv, s["slots"], s["cu"], s["longest"])
    o = ops.deltanet_scan(y, s["n_k"], s["ab"], s["ai"], s["bi"], s["kv"], s["a"], s["dt"], state, s["slots"], s["cu"], s["n_v"])
    return [ops.gated_rmsnorm_heads(o, s["z"], s["w"], 1e-6, DN), conv, state]


def _dn_exact(c, seed):
    s = _dn_inputs(c, seed)
    nk, nv, B = c["n_k"], c["n_v"], c["seqs"]
    conv, state = s["conv"].clone().double(), s["state"].double()
    S = state[s["slots"].long()]
    n_max = max(s["new"])
    C = s["x"].shape[1]
    y = torch.zeros(B, n_max, C, dtype=torch.float64, device=DEV)
    pad = lambda t: torch.stack([torch.nn.functional.pad(u.double(), (0, 0, 0, n_max - u.shape[0])) for u in t.split(s["new"])])
    for i, (slot, xs) in enumerate(zip(s["slots"].tolist(), s["x"].split(s["new"]))):
        full = torch.cat([conv[slot], xs.double()])
        y[i, :xs.shape[0]] = torch.nn.functional.silu((full.unfold(0, 4, 1) * s["conv_w"].double()).sum(-1))
        conv[slot] = full[-3:]
    unit = lambda t: t * torch.rsqrt(t.pow(2).sum(-1, keepdim=True) + 1e-6)
    heads = lambda lo, n: y[..., lo * DN:(lo + n) * DN].reshape(B, n_max, n, DN)
    pick = s["kv"].long()
    q, k, v = unit(heads(0, nk))[:, :, pick] / math.sqrt(DN), unit(heads(nk, nk))[:, :, pick], heads(2 * nk, nv)
    ab = pad(s["ab"])
    decay = torch.exp(s["a"].double() * torch.nn.functional.softplus(ab[..., :nv] + s["dt"].double()))
    beta = torch.sigmoid(ab[..., nv:])
    live = torch.arange(n_max, device=DEV)[None] < torch.tensor(s["new"], device=DEV)[:, None]
    decay, beta = torch.where(live[..., None], decay, 1.0), torch.where(live[..., None], beta, 0.0)
    out = torch.empty(B, n_max, nv, DN, dtype=torch.float64, device=DEV)
    for t in range(n_max):
        S = S * decay[:, t, :, None, None]
        d = (v[:, t] - (S @ k[:, t].unsqueeze(-1)).squeeze(-1)) * beta[:, t, :, None]
        S = S + d.unsqueeze(-1) * k[:, t].unsqueeze(-2)
        out[:, t] = (S @ q[:, t].unsqueeze(-1)).squeeze(-1)
    state[s["slots"].long()] = S
    o = _rms(torch.cat([out[i, :n] for i, n in enumerate(s["new"])]), s["w"], 1e-6)
    return [(o * torch.nn.functional.silu(s["z"].double().view(-1, nv, DN))).reshape(-1, nv * DN), conv, state]


def _dn_work(c):
    new = _spread(c["new_lo"], c["new_hi"], c["seqs"], 0)
    T, nv = sum(new), c["n_v"]
    C = (2 * c["n_k"] + nv) * DN
    return {"bytes": T * (2.0 * C + 4.0 * nv + 4.0 * nv * DN) + c["seqs"] * (8.0 * nv * DN * DN + 12.0 * C), "flops": 6.0 * T * nv * DN * DN + 8.0 * T * C}


# ------------------------------------------------------------------ the interface
_KINDS = {"serve": (_serve_prepare, _serve_run, _serve_exact, _serve_work), "attention": (_attn_prepare, _attn_run, _attn_exact, _attn_work),
          "linear": (_linear_prepare, _linear_run, _linear_exact, _linear_work), "moe": (_moe_prepare, _moe_run, _moe_exact, _moe_work),
          "deltanet": (_dn_prepare, _dn_run, _dn_exact, _dn_work)}


def prepare(case, seed):
    return _KINDS[case["kind"]][0](case, seed)


def run(state):
    return _KINDS[state["kind"]][1](state)


def exact(case, seed):
    with torch.no_grad():
        return _KINDS[case["kind"]][2](case, seed)


def work(case):
    return _KINDS[case["kind"]][3](case)


def tolerance(case):
    """About four times what the path is off from 64 bits (serve 0.009 to 0.017, attention and linear 0.0017 to 0.0022, deltanet 0.0038, experts 0.0017;
    MXFP4 experts 0.014, since a sum that rounds to another e4m3 neighbour moves by 6 %), at most 0.03."""
    if case["kind"] == "moe":
        return {"rel": 0.03 if case["quant"] == "mxfp4" else 0.007}
    return {"rel": {"serve": 0.03, "attention": 0.009, "linear": 0.007, "deltanet": 0.015}[case["kind"]]}
