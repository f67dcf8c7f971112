"""The work that a user of this engine has a B200 do, as cases that can be timed and compared.

Every case goes through an entry point that a program calls: a decode step of the model runner, or one block of a model
(`Attention`, `MLAAttention`, `DenseMLP`, the routed experts, a recurrent mixer) on a loaded batch and a paged cache or
state slots. Sizes are those of the presets and of the side benchmarks' configurations; `draw` spreads them over what
the engine serves: one sequence to full batches, one token to long chunked prompts, ragged lengths, scattered pages.

`listed()`, `draw(rng)`, `prepare(case, seed)`, `run(state)`, `work(case)`, `tolerance(case)`, `exact(case, seed)`.
`exact` states the result in 64 bits in plain torch; it takes the tensors from the same seeded makers as `prepare`.
"""
import math
import random

import numpy as np
import torch

DEV = "cuda"
BF16, F32, F64, F8 = torch.bfloat16, torch.float32, torch.float64, torch.float8_e4m3fn
PAGE = 16
EPS = 1e-6
KINDS = ("model", "gqa", "mlp", "experts", "mla", "delta", "mamba")

# attention blocks: preset shapes (Qwen3-8B, Llama-3-70B, Llama-2-7B, Qwen3-0.6B) and a generic one with heads of 64
GQA = {"qwen3-8b": (4096, 32, 8, 128, True, 1e6), "llama-3-70b": (8192, 64, 8, 128, False, 5e5),
       "llama-2-7b": (4096, 32, 32, 128, False, 1e4), "qwen3-0.6b": (1024, 16, 8, 128, True, 1e6),
       "generic-64": (2048, 32, 8, 64, False, 5e5)}
# feed-forwards: (width, inner)
MLP = {"qwen3-8b": (4096, 12288), "llama-3-70b": (8192, 28672), "deepseek-v3": (7168, 18432), "qwen3-0.6b": (1024, 3072)}
# routed experts: (width, inner, experts, held by this rank, chosen per token)
EXPERTS = {"mixtral-8x7b": (4096, 14336, 8, 8, 2), "qwen3-30b-a3b": (2048, 768, 128, 128, 8),
           "deepseek-v3-ep8": (7168, 2048, 256, 32, 8)}
MODEL_LAYERS = 8


def listed():
    return [
        # a lone chat: one token of one sequence through a whole small model (CUDA graph), where launches and latency count
        {"name": "model_decode_1", "kind": "model", "seqs": 1, "ctx": 500, "mix": 1},
        # a chunked-prefill step of the throughput workload: decoding sequences beside ragged prompts, one attention block
        {"name": "gqa_step_4096", "kind": "gqa", "shape": "qwen3-8b", "decodes": 32, "seqs": 19, "tokens": 4064, "ctx": 1500,
         "prior": 0, "mix": 2},
        # the second half of a long prompt: 8192 new tokens over 8192 cached ones
        {"name": "gqa_long_8192", "kind": "gqa", "shape": "llama-3-70b", "decodes": 0, "seqs": 1, "tokens": 8192, "ctx": 0,
         "prior": 8192, "mix": 3},
        # a full decode batch over ragged contexts
        {"name": "gqa_decode_256", "kind": "gqa", "shape": "qwen3-8b", "decodes": 256, "seqs": 0, "tokens": 0, "ctx": 2048,
         "prior": 0, "mix": 4},
        # the feed-forward of a decode batch: weights are the traffic
        {"name": "mlp_decode_64", "kind": "mlp", "shape": "qwen3-8b", "rows": 64, "fp8": False},
        # the dense feed-forward of a block-scaled fp8 checkpoint on a prefill chunk
        {"name": "mlp_fp8_4096", "kind": "mlp", "shape": "deepseek-v3", "rows": 4096, "fp8": True},
        # many small experts on a decode batch
        {"name": "experts_decode_48", "kind": "experts", "shape": "qwen3-30b-a3b", "rows": 48, "fp8": False, "mix": 5},
        # one expert-parallel rank's share of a block-scaled fp8 mixture on a prefill chunk
        {"name": "experts_fp8_4096", "kind": "experts", "shape": "deepseek-v3-ep8", "rows": 4096, "fp8": True, "mix": 6},
        # latent attention, decoding: one tensor-parallel rank's 16 heads
        {"name": "mla_decode_128", "kind": "mla", "heads": 16, "decodes": 128, "seqs": 0, "tokens": 0, "ctx": 4096,
         "prior": 0, "mix": 7},
        # latent attention, ragged prompts, some with cached prefixes
        {"name": "mla_prefill_4096", "kind": "mla", "heads": 16, "decodes": 0, "seqs": 5, "tokens": 4096, "ctx": 0,
         "prior": 2048, "mix": 8},
        # a gated-delta-rule mixer on ragged prompts
        {"name": "delta_prefill_6000", "kind": "delta", "width": 4096, "heads": 32, "dim": 128, "vdim": 128, "seqs": 4,
         "tokens": 6000, "mix": 9},
        # a Mamba-1 mixer on ragged prompts
        {"name": "mamba_prefill_8192", "kind": "mamba", "width": 4096, "inner": 8192, "state": 16, "seqs": 4, "tokens": 8192,
         "mix": 10},
    ]


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        case = _draw(rng)
        if _cost(case) <= most:
            return case


def _draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind, mix = rng.choice(KINDS), rng.randrange(1 << 20)
    if kind == "model":
        return {"kind": kind, "seqs": log(1, 64), "ctx": log(16, 1500), "mix": mix}
    if kind in ("gqa", "mla"):
        form = rng.choice(("decode", "prefill", "step"))
        decodes = log(1, 512 if kind == "gqa" else 256) if form != "prefill" else 0
        seqs = 0 if form == "decode" else log(1, 16)
        tokens = 0 if form == "decode" else max(seqs, log(32, 8192 if kind == "gqa" else 4096))
        case = {"kind": kind, "decodes": decodes, "seqs": seqs, "tokens": tokens, "ctx": log(16, 4096) if decodes else 0,
                "prior": rng.choice((0, log(16, 8192))) if seqs else 0, "mix": mix}
        case.update({"shape": rng.choice(sorted(GQA))} if kind == "gqa" else {"heads": rng.choice((8, 16, 32, 128))})
        return case
    if kind == "mlp":
        return {"kind": kind, "shape": rng.choice(sorted(MLP)), "rows": log(1, 8192), "fp8": rng.random() < 0.4}
    if kind == "experts":
        shape = rng.choice(sorted(EXPERTS))
        return {"kind": kind, "shape": shape, "rows": log(1, 4096),
                "fp8": shape.startswith("deepseek") or rng.random() < 0.25, "mix": mix}
    seqs = log(1, 8)
    tokens = max(seqs, log(64, 16384))
    if kind == "delta":
        heads = rng.choice((8, 16, 32))
        return {"kind": kind, "width": heads * 128, "heads": heads, "dim": rng.choice((64, 128)),
                "vdim": rng.choice((64, 128, 256)), "seqs": seqs, "tokens": tokens, "mix": mix}
    width = rng.choice((1024, 2048, 4096))
    return {"kind": kind, "width": width, "inner": 2 * width, "state": 16, "seqs": seqs, "tokens": tokens, "mix": mix}


# -- batches ---------------------------------------------------------------------------------------------------
def _lengths(case):
    """(new tokens, cached tokens) of every sequence, decoding ones first: one new token over a ragged context, then
    `tokens` new ones cut raggedly into `seqs` prompts, over up to `prior` cached ones."""
    r = random.Random(case["mix"])
    q, ctx = [], []
    for i in range(case.get("decodes", 0)):
        q.append(1)
        ctx.append(case["ctx"] - 1 if i == 0 else int(math.exp(r.uniform(math.log(max(case["ctx"] / 16, 1.0)),
                                                                         math.log(case["ctx"])))) - 1)
    n, left = case.get("seqs", 0), case.get("tokens", 0)
    share = [math.exp(r.gauss(0.0, 0.7)) for _ in range(n)]
    for i in range(n):
        took = left - (n - 1 - i) if i == n - 1 else max(1, min(left - (n - 1 - i), int(left * share[i] / sum(share[i:]))))
        left -= took
        q.append(took)
        prior = case.get("prior", 0)
        ctx.append(prior if n == 1 else r.randint(0, prior))
    return q, [max(c, 0) for c in ctx]


def _pages(q, ctx, seed):
    """Block table over pages in scattered order, and the number of pages."""
    need = [-(-(a + b) // PAGE) for a, b in zip(q, ctx)]
    total = sum(need)
    order = np.random.RandomState(seed % (1 << 31)).permutation(total).astype(np.int32)
    table, at = np.zeros((len(q), max(need)), np.int32), 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    return table, total


def _batch(q, ctx, table, tokens=None):
    from gllm_b200.input_data import BatchArrays
    q, ctx = np.asarray(q, np.int32), np.asarray(ctx, np.int32)
    qsl = np.zeros(len(q) + 1, np.int32)
    np.cumsum(q, out=qsl[1:])
    pos = np.concatenate([np.arange(c, c + n, dtype=np.int32) for n, c in zip(q, ctx)])
    row = np.repeat(np.arange(len(q)), q)
    slots = table[row, pos // PAGE] * PAGE + pos % PAGE
    e = len(q)
    i32, f32 = np.int32, np.float32
    dec = int((q == 1).cumprod().sum()) if (q == 1).any() and q[0] == 1 else 0
    return BatchArrays(tokens=np.zeros(int(qsl[-1]), i32) if tokens is None else tokens.astype(i32), positions=pos,
                       slot_mapping=slots.astype(i32), block_table=table, seq_lens=q + ctx, query_start_loc=qsl,
                       logits_idx=qsl[1:] - 1, emit_seq=np.arange(e, dtype=i32), temperature=np.ones(e, f32),
                       top_k=np.ones(e, i32), top_p=np.ones(e, f32), rep_penalty=np.ones(e, f32),
                       state_slot=np.zeros(e, i32), num_decode_seqs=dec, num_seqs=e, num_tokens=int(qsl[-1]),
                       max_q_len=int(q.max()), max_seq_len=int((q + ctx).max()), rec_slots=np.arange(e, dtype=i32))


def _input(q, ctx, table):
    from gllm_b200.input_data import InputData
    inp = InputData(sum(q), len(q), table.shape[1], DEV)
    inp.need_tok_seq = True
    inp.load(_batch(q, ctx, table))
    return inp


def _pairs(q, ctx):
    """(query, visible key) pairs under the causal mask, and cached rows read or written."""
    return sum(a * c + a * (a + 1) // 2 for a, c in zip(q, ctx)), sum(a + c for a, c in zip(q, ctx))


class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator(DEV).manual_seed(int(seed))

    def normal(self, *shape, std=1.0, dtype=BF16):
        return torch.empty(shape, dtype=F32, device=DEV).normal_(0.0, std, generator=self.g).to(dtype)

    def uniform(self, *shape, lo=0.0, hi=1.0):
        return torch.empty(shape, dtype=F32, device=DEV).uniform_(lo, hi, generator=self.g)


def _set(param, value):
    assert param.shape == value.shape, (param.shape, value.shape)
    param.data.copy_(value)


def _interleave(w, block):
    """[.., 2 I, K] = gate rows, then up rows -> blocks of gate and up rows in turn (the gated product's layout)."""
    gate, up = (x.reshape(*x.shape[:-2], -1, block, x.shape[-1]) for x in w.chunk(2, -2))
    return torch.cat([gate, up], -2).reshape(w.shape).contiguous()


def _spec(width, heads, kv_heads, dim, inner, vocab=64, layers=1, qk_norm=False, theta=1e4, **more):
    from gllm_b200.models.decoder import ModelSpec
    return ModelSpec(arch="perf", hidden_size=width, num_layers=layers, num_heads=heads, num_kv_heads=kv_heads, head_dim=dim,
                     intermediate_size=inner, vocab_size=vocab, rms_eps=EPS, qk_norm=qk_norm, rope_theta=theta,
                     max_position=32768, **more)


def _tpc():
    from gllm_b200.parallel.tp import make_tp_comm
    return make_tp_comm(False)


# -- 64-bit building blocks ------------------------------------------------------------------------------------
def _rms(x, w=None):
    y = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w.to(F64)


def _rotate(x, pos, theta, adjacent=False):
    """x [T, H, D]; pairs (i, i + D / 2), or adjacent ones."""
    d = x.shape[-1]
    ang = pos.to(F64)[:, None] * theta ** (-torch.arange(0, d, 2, dtype=F64, device=x.device) / d)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    if adjacent:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _attend(q, k, v, ctx, scale):
    """q [n, H, D] at positions ctx .. ctx + n - 1 over k, v [L, Hkv, *]; -> [n, H, Dv]."""
    n, heads, length, rep = q.shape[0], q.shape[1], k.shape[0], q.shape[1] // k.shape[1]
    out = torch.empty(n, heads, v.shape[-1], dtype=F64, device=q.device)
    step = max(1, (1 << 27) // length)
    for g in range(k.shape[1]):
        kg, vg = k[:, g], v[:, g]
        rows = q[:, g * rep:(g + 1) * rep].reshape(n * rep, -1)
        at = torch.arange(n, device=q.device).repeat_interleave(rep) + ctx
        res = torch.empty(n * rep, v.shape[-1], dtype=F64, device=q.device)
        for a in range(0, n * rep, step):
            s = (rows[a:a + step] @ kg.T) * scale
            s.masked_fill_(torch.arange(length, device=q.device)[None] > at[a:a + step, None], -math.inf)
            res[a:a + step] = torch.softmax(s, -1) @ vg
        out[:, g * rep:(g + 1) * rep] = res.view(n, rep, -1)
    return out


def _slots(q, ctx, table):
    pos = np.concatenate([np.arange(c, c + n) for n, c in zip(q, ctx)])
    row = np.repeat(np.arange(len(q)), q)
    return torch.as_tensor(pos, device=DEV), torch.as_tensor(table[row, pos // PAGE].astype(np.int64), device=DEV), \
        torch.as_tensor(pos % PAGE, device=DEV)


def _rows(cache, table, i, length):
    """Cached rows of sequence i, [length, heads, width], from the paged layout [pages, heads, slabs, PAGE, 64]."""
    pages = torch.as_tensor(table[i, :-(-length // PAGE)].astype(np.int64), device=DEV)
    return cache[pages].permute(0, 3, 1, 2, 4).reshape(-1, cache.shape[1], cache.shape[2] * 64)[:length]


def _fp8(x):
    """x as e4m3 with one scale per row and 128 columns."""
    g = x.reshape(*x.shape[:-1], -1, 128)
    s = g.abs().amax(-1, keepdim=True) / 448.0
    s = torch.where(s > 0, s, torch.ones_like(s))
    return ((g / s).float().to(F8).to(F64) * s).reshape(x.shape)


# -- whole model: one decode step ------------------------------------------------------------------------------
def _model_lens(case):
    r = random.Random(case["mix"])
    return [case["ctx"]] + [r.randint(max(1, case["ctx"] // 4), case["ctx"]) for _ in range(case["seqs"] - 1)]


def _model_tensors(case, seed):
    h, heads, kv, d, _, _ = GQA["qwen3-0.6b"]
    inner, vocab = MLP["qwen3-0.6b"][1], 151936
    r = _Rand(seed)
    w = {"embed": r.normal(vocab, h, std=1.0)}
    for i in range(MODEL_LAYERS):
        w[i] = {"qkv": r.normal((heads + 2 * kv) * d, h, std=h ** -0.5),
                "o": r.normal(h, heads * d, std=(heads * d) ** -0.5),
                "gu": r.normal(2 * inner, h, std=h ** -0.5), "down": r.normal(h, inner, std=inner ** -0.5)}
    lens = _model_lens(case)
    ids = np.random.RandomState(seed % (1 << 31)).randint(0, vocab, sum(lens))
    return w, lens, ids


def _model_prepare(case, seed):
    from gllm_b200.config import EngineConfig
    from gllm_b200.model_runner import ModelRunner
    from gllm_b200.models.presets import PRESETS
    w, lens, ids = _model_tensors(case, seed)
    q = [n - 1 for n in lens]
    table, pages = _pages([1] * len(lens), q, seed)
    chunk = max(sum(lens), 64)
    cfg = EngineConfig(model_path=dict(PRESETS["qwen3-0.6b"], num_hidden_layers=MODEL_LAYERS), load_format="dummy",
                       page_size=PAGE, maxp=chunk, maxd=64, num_gpu_pages=pages + 1, model_max_length=max(lens) + PAGE,
                       enable_prefix_caching=False, max_cuda_graph_bs=1 << (len(lens) - 1).bit_length(), log_stats=False,
                       launch_mode="inproc", device="cuda:0")
    runner = ModelRunner(cfg).init("cuda:0")
    m = runner.model
    _set(m.embed_w, w["embed"])
    for i, layer in enumerate(m.layers):
        _set(layer.attn.qkv_w, w[i]["qkv"])
        _set(layer.attn.o_w, w[i]["o"])
        layer.mlp.set_gate_up(w[i]["gu"])
        _set(layer.mlp.down_w, w[i]["down"])
    first = np.cumsum([0] + lens[:-1])
    if any(q):
        some = [i for i in range(len(q)) if q[i]]
        toks = np.concatenate([ids[first[i]:first[i] + q[i]] for i in some])
        runner.step(_batch([q[i] for i in some], [0] * len(some), table[some], toks))
    last = ids[first + np.asarray(q)]
    return {"runner": runner, "batch": _batch([1] * len(q), q, table, last), "n": len(q)}


def _model_run(s):
    runner = s["runner"]
    runner.step(s["batch"])            # greedy tokens come back as well; equal logits of random weights make them moot
    bucket = min(b for b in runner.graphs if b >= s["n"])
    return runner.graph_logits[bucket][:s["n"]]


def _model_exact(case, seed):
    w, lens, ids = _model_tensors(case, seed)
    h, heads, kv, d, _, theta = GQA["qwen3-0.6b"]
    x = w["embed"][torch.as_tensor(ids, device=DEV)].to(F64)
    pos = torch.as_tensor(np.concatenate([np.arange(n) for n in lens]), device=DEV)
    ends = np.cumsum(lens)
    for i in range(MODEL_LAYERS):
        t = _rms(x) @ w[i]["qkv"].to(F64).T
        qq, kk, vv = (y.reshape(len(ids), -1, d) for y in t.split([heads * d, kv * d, kv * d], -1))
        qq, kk = _rotate(_rms(qq), pos, theta), _rotate(_rms(kk), pos, theta)
        a = torch.cat([_attend(qq[e - n:e], kk[e - n:e], vv[e - n:e], 0, d ** -0.5) for e, n in zip(ends, lens)])
        x = x + a.reshape(len(ids), -1) @ w[i]["o"].to(F64).T
        g, u = (_rms(x) @ w[i]["gu"].to(F64).T).chunk(2, -1)
        x = x + (torch.nn.functional.silu(g) * u) @ w[i]["down"].to(F64).T
    return _rms(x[torch.as_tensor(ends - 1, device=DEV)]) @ w["embed"].to(F64).T


# -- grouped-query attention block -----------------------------------------------------------------------------
def _gqa_tensors(case, seed):
    h, heads, kv, d, norm, theta = GQA[case["shape"]]
    q, ctx = _lengths(case)
    table, pages = _pages(q, ctx, seed)
    r = _Rand(seed)
    return {"h": r.normal(sum(q), h), "qkv": r.normal((heads + 2 * kv) * d, h, std=h ** -0.5),
            "qn": (1 + r.normal(d, std=0.2)) if norm else None, "kn": (1 + r.normal(d, std=0.2)) if norm else None,
            "k": r.normal(pages, kv, d // 64, PAGE, 64), "v": r.normal(pages, kv, d // 64, PAGE, 64)}, q, ctx, table, pages


def _gqa_prepare(case, seed):
    from gllm_b200.layers.rotary import build_rope
    from gllm_b200.memory_manager import KVCache
    from gllm_b200.models.decoder import Attention
    x, q, ctx, table, pages = _gqa_tensors(case, seed)
    h, heads, kv, d, norm, theta = GQA[case["shape"]]
    att = Attention(_spec(h, heads, kv, d, h, qk_norm=norm, theta=theta), 0, build_rope(d, 32768, theta, device=DEV), DEV)
    _set(att.qkv_w, x["qkv"])
    if norm:
        _set(att.q_norm_w, x["qn"])
        _set(att.k_norm_w, x["kn"])
    cache = KVCache(1, pages, PAGE, kv, d, BF16, DEV)
    cache.k_cache[0].copy_(x["k"])
    cache.v_cache[0].copy_(x["v"])
    return {"block": att, "inp": _input(q, ctx, table), "h": x["h"], "cache": cache, "tpc": _tpc()}


def _block_run(s):
    out = s["block"](s["inp"], s["h"], s["cache"], s["tpc"])
    c = s["cache"]
    return {"out": out, "k": c.k_cache[0], "v": c.v_cache[0]} if c.v_cache else {"out": out, "k": c.k_cache[0]}


def _gqa_exact(case, seed):
    x, q, ctx, table, _ = _gqa_tensors(case, seed)
    _, heads, kv, d, _, theta = GQA[case["shape"]]
    t = x["h"].to(F64) @ x["qkv"].to(F64).T
    n = t.shape[0]
    qq, kk, vv = (y.reshape(n, -1, d) for y in t.split([heads * d, kv * d, kv * d], -1))
    if x["qn"] is not None:
        qq, kk = _rms(qq, x["qn"]), _rms(kk, x["kn"])
    pos, page, off = _slots(q, ctx, table)
    qq, kk = _rotate(qq, pos, theta), _rotate(kk, pos, theta)
    k, v = x["k"].to(F64), x["v"].to(F64)
    k[page, :, :, off] = kk.reshape(n, kv, d // 64, 64)
    v[page, :, :, off] = vv.reshape(n, kv, d // 64, 64)
    out, at = torch.empty(n, heads * d, dtype=F64, device=DEV), 0
    for i, (a, c) in enumerate(zip(q, ctx)):
        out[at:at + a] = _attend(qq[at:at + a], _rows(k, table, i, a + c), _rows(v, table, i, a + c), c,
                                 d ** -0.5).reshape(a, -1)
        at += a
    return {"out": out, "k": k, "v": v}


# -- multi-head latent attention block -------------------------------------------------------------------------
MLA_WIDTH, Q_RANK, KV_RANK, NOPE, ROT, MLA_V = 7168, 1536, 512, 128, 64, 128


def _mla_tensors(case, seed):
    heads = case["heads"]
    q, ctx = _lengths(case)
    table, pages = _pages(q, ctx, seed)
    r = _Rand(seed)
    return {"h": r.normal(sum(q), MLA_WIDTH), "q_a": r.normal(Q_RANK, MLA_WIDTH, std=MLA_WIDTH ** -0.5),
            "q_b": r.normal(heads * (NOPE + ROT), Q_RANK, std=Q_RANK ** -0.5),
            "kv_a": r.normal(KV_RANK + ROT, MLA_WIDTH, std=MLA_WIDTH ** -0.5),
            "kv_b": r.normal(heads * (NOPE + MLA_V), KV_RANK, std=KV_RANK ** -0.5), "qn": 1 + r.normal(Q_RANK, std=0.2),
            "kvn": 1 + r.normal(KV_RANK, std=0.2), "k": r.normal(pages, 1, (KV_RANK + ROT) // 64, PAGE, 64)}, \
        q, ctx, table, pages


def _mla_prepare(case, seed):
    from gllm_b200.layers.rotary import build_rope
    from gllm_b200.memory_manager import KVCache
    from gllm_b200.models.deepseek_v2 import MLAAttention
    x, q, ctx, table, pages = _mla_tensors(case, seed)
    spec = _spec(MLA_WIDTH, case["heads"], case["heads"], NOPE + ROT, MLA_WIDTH, use_mla=True,
                 extra={"qk_nope_head_dim": NOPE, "qk_rope_head_dim": ROT, "v_head_dim": MLA_V, "kv_lora_rank": KV_RANK,
                        "q_lora_rank": Q_RANK})
    att = MLAAttention(spec, 0, build_rope(ROT, 32768, 1e4, None, ROT, False, device=DEV), DEV)
    for name, p in (("q_a", att.q_a_w), ("q_b", att.q_b_w), ("kv_a", att.kv_a_w), ("kv_b", att.kv_b_w),
                    ("qn", att.q_a_norm_w), ("kvn", att.kv_a_norm_w)):
        _set(p, x[name])
    att.process_weights()
    cache = KVCache(1, pages, PAGE, 1, KV_RANK + ROT, BF16, DEV, use_mla=True)
    cache.k_cache[0].copy_(x["k"])
    return {"block": att, "inp": _input(q, ctx, table), "h": x["h"], "cache": cache, "tpc": _tpc()}


def _mla_exact(case, seed):
    x, q, ctx, table, _ = _mla_tensors(case, seed)
    heads = case["heads"]
    h = x["h"].to(F64)
    n = h.shape[0]
    qq = (_rms(h @ x["q_a"].to(F64).T, x["qn"]) @ x["q_b"].to(F64).T).view(n, heads, NOPE + ROT)
    kv = h @ x["kv_a"].to(F64).T
    pos, page, off = _slots(q, ctx, table)
    new = torch.cat([_rms(kv[:, :KV_RANK], x["kvn"]), _rotate(kv[:, None, KV_RANK:], pos, 1e4, True)[:, 0]], -1)
    q_rot = _rotate(qq[:, :, NOPE:], pos, 1e4, True)
    lat = x["k"].to(F64)
    lat[page, :, :, off] = new.view(n, 1, -1, 64)
    uk, uv = x["kv_b"].to(F64).view(heads, NOPE + MLA_V, KV_RANK).split([NOPE, MLA_V], 1)
    full = torch.cat([torch.einsum("nhd,hdr->nhr", qq[:, :, :NOPE], uk), q_rot], -1)
    out, at = torch.empty(n, heads * MLA_V, dtype=F64, device=DEV), 0
    for i, (a, c) in enumerate(zip(q, ctx)):
        rows = _rows(lat, table, i, a + c)
        o = _attend(full[at:at + a], rows, rows[..., :KV_RANK], c, (NOPE + ROT) ** -0.5)
        out[at:at + a] = torch.einsum("nhr,hdr->nhd", o, uv).reshape(a, -1)
        at += a
    return {"out": out, "k": lat}


# -- feed-forward ----------------------------------------------------------------------------------------------
def _fp8_weight(r, n, k):
    """e4m3 weight with one scale per 128 x 128 block, of the size that keeps a unit input a unit output."""
    w = (r.normal(n, k, std=100.0, dtype=F32)).clamp_(-448.0, 448.0).to(F8)
    return w, r.uniform(-(-n // 128), k // 128, lo=0.5, hi=1.5) * (k ** -0.5 / 100.0)


def _wide(w, s):
    return w.to(F64) * s.to(F64).repeat_interleave(128, 0)[:w.shape[0]].repeat_interleave(128, 1)


def _mlp_tensors(case, seed):
    h, inner = MLP[case["shape"]]
    r = _Rand(seed)
    x = {"h": r.normal(case["rows"], h)}
    if case["fp8"]:
        x["gu"], x["gu_s"] = _fp8_weight(r, 2 * inner, h)
        x["down"], x["down_s"] = _fp8_weight(r, h, inner)
    else:
        x["gu"], x["down"] = r.normal(2 * inner, h, std=h ** -0.5), r.normal(h, inner, std=inner ** -0.5)
    return x


def _mlp_prepare(case, seed):
    from gllm_b200.models.decoder import DenseMLP
    x = _mlp_tensors(case, seed)
    h, inner = MLP[case["shape"]]
    mlp = DenseMLP(h, inner, BF16, DEV, spec=_spec(h, 1, 1, 64, inner, quant="fp8" if case["fp8"] else None))
    if case["fp8"]:
        _set(mlp.gate_up_w, x["gu"])
        _set(mlp.gate_up_ws, x["gu_s"])
        _set(mlp.down_ws, x["down_s"])
    else:
        mlp.set_gate_up(x["gu"])
    _set(mlp.down_w, x["down"])
    return {"mlp": mlp, "h": x["h"], "tpc": _tpc()}


def _mlp_run(s):
    return s["tpc"].row_linear(s["mlp"].act(s["h"], s["tpc"]), s["mlp"].down_weight())


def _mlp_exact(case, seed):
    x = _mlp_tensors(case, seed)
    h = x["h"].to(F64)
    if not case["fp8"]:
        g, u = (h @ x["gu"].to(F64).T).chunk(2, -1)
        return (torch.nn.functional.silu(g) * u) @ x["down"].to(F64).T
    g, u = (_fp8(h) @ _wide(x["gu"], x["gu_s"]).T).chunk(2, -1)
    return _fp8(torch.nn.functional.silu(g) * u) @ _wide(x["down"], x["down_s"]).T


# -- routed experts --------------------------------------------------------------------------------------------
def _experts_tensors(case, seed):
    h, inner, experts, held, top = EXPERTS[case["shape"]]
    r = _Rand(seed)
    x = {"h": r.normal(case["rows"], h)}
    scores = r.normal(case["rows"], experts, dtype=F32) + r.normal(experts, std=0.5, dtype=F32)   # some experts are liked
    best, ids = scores.topk(top, -1)
    x["w"], x["ids"] = torch.softmax(best, -1), ids.to(torch.int32)
    gu, down, gu_s, down_s = [], [], [], []
    for _ in range(held):
        if case["fp8"]:
            a, b = _fp8_weight(r, 2 * inner, h), _fp8_weight(r, h, inner)
            gu_s.append(a[1])
            down_s.append(b[1])
            a, b = a[0], b[0]
        else:
            a, b = r.normal(2 * inner, h, std=h ** -0.5), r.normal(h, inner, std=inner ** -0.5)
        gu.append(a)
        down.append(b)
    x["gu"], x["down"], x["gu_s"], x["down_s"] = gu, down, gu_s, down_s
    return x


def _experts_prepare(case, seed):
    x = _experts_tensors(case, seed)
    h, inner, experts, held, top = EXPERTS[case["shape"]]
    s = {"h": x["h"], "w": x["w"], "ids": x["ids"], "down": torch.stack(x["down"]), "map": None}
    gu = torch.stack(x["gu"])
    del x["gu"], x["down"]
    if case["fp8"]:
        # the loader's layout: gate and up rows in blocks of 64, one scale per 64 rows
        s["gu"] = _interleave(gu.view(torch.uint8), 64).view(F8)
        s["gu_s"] = _interleave(torch.stack(x["gu_s"]).repeat_interleave(2, 1), 1)
        s["down_s"] = torch.stack(x["down_s"]).repeat_interleave(2, 1).contiguous()
        if held < experts:
            s["map"] = torch.full((experts,), -1, dtype=torch.int32, device=DEV)
            s["map"][:held] = torch.arange(held, dtype=torch.int32, device=DEV)
    else:
        s["gu"] = _interleave(gu, 64)
    return s


def _experts_run(s):
    if "gu_s" in s:
        from gllm_b200.ops import sm100_moe
        return sm100_moe.fused_experts_fp8(s["h"], s["gu"], s["gu_s"], s["down"], s["down_s"], s["w"], s["ids"], s["map"])
    from gllm_b200.layers import functional as Fn
    return Fn.routed_experts(s["h"], s["gu"], s["down"], s["w"], s["ids"], True)


def _experts_exact(case, seed):
    x = _experts_tensors(case, seed)
    held = EXPERTS[case["shape"]][3]
    h, out = x["h"].to(F64), torch.zeros(x["h"].shape, dtype=F64, device=DEV)
    for e in range(held):
        row, slot = (x["ids"] == e).nonzero(as_tuple=True)
        if not len(row):
            continue
        if case["fp8"]:
            g, u = (_fp8(h[row]) @ _wide(x["gu"][e], x["gu_s"][e]).T).chunk(2, -1)
            y = _fp8(torch.nn.functional.silu(g) * u) @ _wide(x["down"][e], x["down_s"][e]).T
        else:
            g, u = (h[row] @ x["gu"][e].to(F64).T).chunk(2, -1)
            y = (torch.nn.functional.silu(g) * u) @ x["down"][e].to(F64).T
        out.index_add_(0, row, y * x["w"][row, slot].to(F64)[:, None])
    return out


# -- recurrent mixers ------------------------------------------------------------------------------------------
TAPS = 4


def _step_bias(r, n):
    """softplus^-1 of steps spread over 0.001 .. 0.1, as such mixers are initialised."""
    dt = torch.exp(r.uniform(n, lo=math.log(1e-3), hi=math.log(0.1)))
    return dt + torch.log(-torch.expm1(-dt))


def _mixer_state(case, block, q):
    from gllm_b200.memory_manager import HybridCache
    cache = HybridCache([block.cache_entry()], 1, PAGE, len(q), BF16, DEV)
    return {"mixer": block, "inp": _input(q, [0] * len(q), np.zeros((len(q), -(-max(q) // PAGE)), np.int32)), "cache": cache}


def _mixer_run(s):
    out = s["mixer"](s["inp"], s["h"], s["cache"], 0)
    return {"out": out, "state": s["cache"].ssm_state[0], "conv": s["cache"].conv_state[0]}


def _padded(x, q):
    """[T, ...] -> [len(q), max(q), ...], zeros behind each sequence."""
    out = torch.zeros(len(q), max(q), *x.shape[1:], dtype=x.dtype, device=x.device)
    for i, (n, e) in enumerate(zip(q, np.cumsum(q))):
        out[i, :n] = x[e - n:e]
    return out


def _unpadded(x, q):
    return torch.cat([x[i, :n] for i, n in enumerate(q)])


def _convolved(x, w, b):
    """Causal depthwise convolution + SiLU of x [S, L, C]; w [C, TAPS]."""
    y = torch.nn.functional.pad(x, (0, 0, TAPS - 1, 0))
    acc = sum(y[:, j:j + x.shape[1]] * w[:, j].to(F64) for j in range(TAPS))
    return torch.nn.functional.silu(acc if b is None else acc + b.to(F64))


def _tail(x, q):
    """The last TAPS - 1 inputs of every sequence, zeros before its start."""
    y = torch.nn.functional.pad(x, (0, 0, TAPS - 1, 0))
    return torch.stack([y[i, n:n + TAPS - 1] for i, n in enumerate(q)])


def _delta_tensors(case, seed):
    hd, d, dv, width = case["heads"], case["dim"], case["vdim"], case["width"]
    g = hd // 2
    r = _Rand(seed)
    q, _ = _lengths(case)
    rows = 2 * g * d + 2 * hd * dv
    w_in = torch.cat([r.normal(rows, width, std=2 * width ** -0.5), r.normal(hd, width, std=2 * width ** -0.5),
                      r.normal(hd, width, std=0.5 * width ** -0.5)])
    return {"h": r.normal(sum(q), width), "in": w_in, "conv": r.normal(2 * g * d + hd * dv, TAPS, std=0.6, dtype=F32),
            "neg_a": -r.uniform(hd, lo=1.0, hi=16.0), "dt_bias": _step_bias(r, hd), "norm": 1 + r.normal(dv, std=0.2),
            "o": r.normal(width, hd * dv, std=(hd * dv) ** -0.5)}, q


def _delta_prepare(case, seed):
    from gllm_b200.layers.linear_attention import GatedDeltaCore
    from gllm_b200.layers.parallel_mixer import CoreMixer
    x, q = _delta_tensors(case, seed)
    core = GatedDeltaCore(case["heads"], case["heads"] // 2, case["dim"], case["vdim"], TAPS, EPS, BF16, DEV)
    m = CoreMixer(case["width"], [core], [""], [1.0], BF16, DEV)
    m.in_w.data[:x["in"].shape[0]].copy_(x["in"])
    for name, p in (("conv", core.conv_w), ("neg_a", core.neg_a), ("dt_bias", core.dt_bias), ("norm", core.norm_w),
                    ("o", m.o_w)):
        _set(p, x[name])
    return dict(_mixer_state(case, m, q), h=x["h"])


def _delta_exact(case, seed):
    x, q = _delta_tensors(case, seed)
    hd, d, dv = case["heads"], case["dim"], case["vdim"]
    g = hd // 2
    nq, nv = g * d, hd * dv
    proj = _padded(x["h"].to(F64) @ x["in"].to(F64).T, q)
    s, length = proj.shape[:2]
    xc = _convolved(proj[..., :2 * nq + nv], x["conv"], None)
    qq, kk = (y.reshape(s, length, g, d) for y in (xc[..., :nq], xc[..., nq:2 * nq]))
    qq, kk = (y / torch.sqrt((y * y).sum(-1, keepdim=True) + 1e-6) for y in (qq, kk))
    qq, kk = ((y * f).repeat_interleave(2, 2) for y, f in ((qq, d ** -0.5), (kk, 1.0)))
    vv = xc[..., 2 * nq:].reshape(s, length, hd, dv)
    at = 2 * nq + nv
    gate, beta = proj[..., at:at + nv], torch.sigmoid(proj[..., at + nv:at + nv + hd])
    dec = torch.exp(x["neg_a"].to(F64) * torch.nn.functional.softplus(proj[..., at + nv + hd:] + x["dt_bias"].to(F64)))
    live = (torch.arange(length, device=DEV)[None] < torch.as_tensor(q, device=DEV)[:, None]).to(F64)
    beta, kk = beta * live[..., None], kk * live[..., None, None]
    dec = torch.where(live[..., None] > 0, dec, torch.ones_like(dec))
    st, o = torch.zeros(s, hd, d, dv, dtype=F64, device=DEV), torch.empty(s, length, hd, dv, dtype=F64, device=DEV)
    for t in range(length):
        st = st * dec[:, t, :, None, None]
        u = beta[:, t, :, None] * (vv[:, t] - (kk[:, t, :, None] @ st)[:, :, 0])
        st = st + kk[:, t, :, :, None] * u[:, :, None]
        o[:, t] = (qq[:, t, :, None] @ st)[:, :, 0]
    y = _rms(o, x["norm"]).reshape(s, length, nv) * torch.nn.functional.silu(gate)
    return {"out": _unpadded(y, q) @ x["o"].to(F64).T, "state": st, "conv": _tail(proj[..., :at], q)}


def _mamba_tensors(case, seed):
    width, inner, n = case["width"], case["inner"], case["state"]
    rank = width // 16
    r = _Rand(seed)
    q, _ = _lengths(case)
    return {"h": r.normal(sum(q), width), "in": r.normal(2 * inner, width, std=width ** -0.5),
            "conv": r.normal(inner, TAPS, std=0.5, dtype=F32), "conv_b": r.normal(inner, std=0.1, dtype=F32),
            "x": r.normal(rank + 2 * n, inner, std=2 * inner ** -0.5), "dt": r.normal(inner, rank, std=rank ** -0.5),
            "dt_b": _step_bias(r, inner), "a": -torch.arange(1, n + 1, dtype=F32, device=DEV).repeat(inner, 1),
            "d": 1 + r.normal(inner, std=0.1, dtype=F32), "o": r.normal(width, inner, std=inner ** -0.5)}, q


def _mamba_prepare(case, seed):
    from gllm_b200.layers.ssm import Mamba1Mixer
    x, q = _mamba_tensors(case, seed)
    m = Mamba1Mixer(case["width"], case["inner"], case["state"], case["width"] // 16, TAPS, BF16, DEV)
    for name, p in (("in", m.in_w), ("conv", m.conv_w), ("conv_b", m.conv_b), ("x", m.x_w), ("dt", m.dt_w), ("dt_b", m.dt_b),
                    ("a", m.a), ("d", m.d_skip), ("o", m.o_w)):
        _set(p, x[name])
    return dict(_mixer_state(case, m, q), h=x["h"])


def _mamba_exact(case, seed):
    x, q = _mamba_tensors(case, seed)
    inner, n, rank = case["inner"], case["state"], case["width"] // 16
    xz = _padded(x["h"].to(F64) @ x["in"].to(F64).T, q)
    s, length = xz.shape[:2]
    xc = _convolved(xz[..., :inner], x["conv"], x["conv_b"])
    p = xc @ x["x"].to(F64).T
    dt = torch.nn.functional.softplus(p[..., :rank] @ x["dt"].to(F64).T + x["dt_b"].to(F64))
    dt = dt * (torch.arange(length, device=DEV)[None] < torch.as_tensor(q, device=DEV)[:, None])[..., None]
    a, bm, cm = x["a"].to(F64), p[..., rank:rank + n], p[..., rank + n:]
    st, y = torch.zeros(s, inner, n, dtype=F64, device=DEV), torch.empty(s, length, inner, dtype=F64, device=DEV)
    for t in range(length):
        st = torch.exp(dt[:, t, :, None] * a) * st + (dt[:, t] * xc[:, t])[..., None] * bm[:, t, None]
        y[:, t] = (st @ cm[:, t, :, None])[..., 0]
    y = (y + x["d"].to(F64) * xc) * torch.nn.functional.silu(xz[..., inner:])
    return {"out": _unpadded(y, q) @ x["o"].to(F64).T, "state": st.transpose(1, 2), "conv": _tail(xz[..., :inner], q)}


# -- what the cases have in common -----------------------------------------------------------------------------
_PREPARE = {"model": _model_prepare, "gqa": _gqa_prepare, "mla": _mla_prepare, "mlp": _mlp_prepare,
            "experts": _experts_prepare, "delta": _delta_prepare, "mamba": _mamba_prepare}
_RUN = {"model": _model_run, "gqa": _block_run, "mla": _block_run, "mlp": _mlp_run, "experts": _experts_run,
        "delta": _mixer_run, "mamba": _mixer_run}
_EXACT = {"model": _model_exact, "gqa": _gqa_exact, "mla": _mla_exact, "mlp": _mlp_exact, "experts": _experts_exact,
          "delta": _delta_exact, "mamba": _mamba_exact}


def prepare(case, seed):
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)


@torch.no_grad()
def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def work(case):
    """Bytes of every input and output once, and the multiply-adds (twice) of the products and of the attention or
    recurrence over what is visible."""
    kind = case["kind"]
    if kind == "model":
        h, heads, kv, d, _, _ = GQA["qwen3-0.6b"]
        inner, vocab = MLP["qwen3-0.6b"][1], 151936
        rows = sum(_model_lens(case))
        layer = (heads + 2 * kv) * d * h + heads * d * h + 3 * inner * h
        return {"bytes": 2.0 * (MODEL_LAYERS * (layer + rows * 2 * kv * d) + vocab * h + case["seqs"] * vocab),
                "flops": 2.0 * (case["seqs"] * (MODEL_LAYERS * layer + vocab * h) + MODEL_LAYERS * rows * 2 * heads * d)}
    if kind == "gqa":
        h, heads, kv, d, _, _ = GQA[case["shape"]]
        q, ctx = _lengths(case)
        pairs, rows = _pairs(q, ctx)
        t, n = sum(q), (heads + 2 * kv) * d
        return {"bytes": 2.0 * (t * h + n * h + rows * 2 * kv * d + t * heads * d),
                "flops": 2.0 * (t * n * h + pairs * 2 * heads * d)}
    if kind == "mla":
        q, ctx = _lengths(case)
        pairs, rows = _pairs(q, ctx)
        t, hd = sum(q), case["heads"]
        lin = Q_RANK * MLA_WIDTH + hd * (NOPE + ROT) * Q_RANK + (KV_RANK + ROT) * MLA_WIDTH + hd * (NOPE + MLA_V) * KV_RANK
        # scores and values per visible pair in the expanded form (key 192, value 128 wide), the cheaper one for prompts
        return {"bytes": 2.0 * (t * MLA_WIDTH + lin + rows * (KV_RANK + ROT) + t * hd * MLA_V),
                "flops": 2.0 * (t * lin + pairs * hd * (NOPE + ROT + MLA_V))}
    if kind == "mlp":
        h, inner = MLP[case["shape"]]
        return {"bytes": 3.0 * h * inner * (1 if case["fp8"] else 2) + 4.0 * case["rows"] * h,
                "flops": 6.0 * case["rows"] * h * inner}
    if kind == "experts":
        h, inner, experts, held, top = EXPERTS[case["shape"]]
        slots = case["rows"] * top * held / experts
        hit = held * (1 - (1 - top / experts) ** case["rows"])
        return {"bytes": hit * 3.0 * h * inner * (1 if case["fp8"] else 2) + 4.0 * case["rows"] * h,
                "flops": 6.0 * slots * h * inner}
    t, width = case["tokens"], case["width"]
    if kind == "delta":
        hd, d, dv = case["heads"], case["dim"], case["vdim"]
        lin = width * (hd * d + 2 * hd * dv + 2 * hd) + width * hd * dv
        return {"bytes": 4.0 * t * width + 2.0 * lin + 4.0 * case["seqs"] * hd * d * dv,
                "flops": 2.0 * t * lin + 8.0 * t * hd * d * dv}
    inner, n, rank = case["inner"], case["state"], width // 16
    lin = 3 * width * inner + inner * (rank + 2 * n) + rank * inner
    return {"bytes": 4.0 * t * width + 2.0 * lin + 4.0 * case["seqs"] * inner * n,
            "flops": 2.0 * t * lin + 7.0 * t * inner * n}


def tolerance(case):
    """bf16 (or e4m3) operands with fp32 sums: what another order of the sums and another place of the 16-bit rounding
    between two products change; about four times what was measured against `exact` (model 0.01, gqa 0.004, mla 0.0045,
    bf16 products 0.003, fp8 0.018, delta 0.004, mamba 0.006), at most 0.03."""
    fp8 = case.get("fp8")
    return {"rel": {"model": 0.03, "gqa": 0.015, "mla": 0.018, "mlp": 0.03 if fp8 else 0.01,
                    "experts": 0.03 if fp8 else 0.012, "delta": 0.016, "mamba": 0.024}[case["kind"]]}
