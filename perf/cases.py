"""The work whose time counts: what programs on top of this library have it do, as measurable cases.

Ten kinds of work over the ranges below, in the types they are used in.  The models are those of the repository's own
benchmark of layers (width 4096, feed-forward 14336, 8 layers, vocabulary 32000: `bench_layered.py`), with random weights:
  decode     one token for each of a batch of sequences, driven by a scheduler's block tables (bf16; f16, which is the
             default type of the project that this library serves; contexts from a few to a few thousand tokens)
  prefill    the logits after a whole prompt (`Engine.forward_with_cache`)
  verify     the logits of a few drafted tokens behind a long context (speculative decoding)
  mixed      a step of continuous batching: decoded tokens and portions of prompts in one batch
  serve      a batch of prompts and some decoded tokens through the layered family (Latarax: windowed attention, two linear
             recurrences, several residual streams)
  sample     the next token of every row of logits on the device: temperature, nucleus, penalties; without a nucleus the
             distribution itself, as the acceptance test of speculative decoding reads it
  attention  paged attention of decoded tokens as an operation of its own (bf16, f16; with a sliding window or without)
  gemm       a projection as an operation of its own (bf16, f16)
  experts    the feed-forward of a mixture of experts: routing, sorted rows, two grouped products, the weighted sum
  glue       the small operations between the products of a layer: add + norm, rotation, cache write, gate
"""
import ctypes
import math

import numpy as np
import torch

import __graft_entry__

MODEL = dict(hidden_size=4096, intermediate_size=14336, num_hidden_layers=8, num_attention_heads=32, num_key_value_heads=8,
             vocab_size=32000, rms_norm_eps=1e-6, rope_theta=500000.0)
H, FF, LAYERS, HEADS, KV, DIM, VOCAB = 4096, 14336, 8, 32, 8, 128, 32000
PARAMS = LAYERS * ((HEADS + 2 * KV) * DIM * H + H * H + 3 * FF * H)  # of the layers
BLOCK = 16
ROWS = 512       # rows of a step
STD = 0.01       # of the random weights (twice as much and the rounding of bf16 grows to 3 % of the logits over the layers)
DEVICE = "cuda"
TYPES = {"bf16": torch.bfloat16, "f16": torch.float16}


def listed():
    return [
        # one person at a chat window; a server under load; the default type of the served project
        dict(name="decode 1 sequence", kind="decode", dtype="bf16", batch=1, ctx=700),
        dict(name="decode 64 sequences", kind="decode", dtype="bf16", batch=64, ctx=900),
        dict(name="decode 16 sequences in f16", kind="decode", dtype="f16", batch=16, ctx=100),
        # a document to read; a draft of eight tokens to check; a scheduler's step with newcomers in it
        dict(name="prefill 2000 tokens", kind="prefill", dtype="bf16", tokens=2000),
        dict(name="verify 8 tokens", kind="verify", dtype="bf16", tokens=8, ctx=1500),
        dict(name="mixed step", kind="mixed", dtype="bf16", batch=40, ctx=600, prompts=3, tokens=437),
        dict(name="serve Latarax", kind="serve", dtype="bf16", batch=12, tokens=250, steps=6),
        # sampling at the vocabulary of the flagship model; a long context; a product with a ragged batch
        dict(name="sample 64 rows", kind="sample", rows=64, vocab=128256, top_p=0.9, penalties=False),
        dict(name="attention long contexts", kind="attention", dtype="bf16", batch=20, heads=32, kv=8, ctx=9000, splits=1, window=0),
        dict(name="gemm 1500 rows", kind="gemm", dtype="bf16", rows=1500, n=14336, k=4096),
        dict(name="experts 600 rows", kind="experts", rows=600, experts=8, top=2, width=4096, ff=7168),
        # the smallest calls: between the products of one layer for one token
        dict(name="glue 1 token", kind="glue", dtype="f16", tokens=1),
    ]


def draw(rng):
    def size(lo, hi):  # spread over the logarithm
        return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))

    kind = rng.choice(("decode", "decode", "decode", "prefill", "prefill", "verify", "mixed", "serve", "sample", "attention", "gemm",
                       "experts", "glue"))
    if kind == "decode":
        if rng.random() < 0.3:
            return dict(kind=kind, dtype="f16", batch=size(1, 32), ctx=size(8, 120))
        batch = size(1, 128)
        return dict(kind=kind, dtype="bf16", batch=batch, ctx=size(8, min(3000, 60000 // batch)))
    if kind == "prefill":
        if rng.random() < 0.25:
            return dict(kind=kind, dtype="f16", tokens=size(5, 200))
        return dict(kind=kind, dtype="bf16", tokens=size(5, 2000))
    if kind == "verify":
        return dict(kind=kind, dtype="bf16", tokens=size(2, 16), ctx=size(16, 3000))
    if kind == "mixed":
        prompts = size(1, 4)
        return dict(kind=kind, dtype="bf16", batch=size(2, 80), ctx=size(16, 700), prompts=prompts, tokens=size(8, 1300 // prompts))
    if kind == "serve":
        batch = size(1, 16)
        return dict(kind=kind, dtype="bf16", batch=batch, tokens=size(4, 2500 // batch), steps=size(1, 6))
    if kind == "sample":
        return dict(kind=kind, rows=size(1, 128), vocab=rng.choice((32000, 32768, 50257, 128256)),
                    top_p=rng.choice((0.5, 0.9, 0.95, 1.0)), penalties=rng.random() < 0.4)
    if kind == "attention":
        batch, heads = size(1, 128), rng.choice((8, 16, 32, 64))
        return dict(kind=kind, dtype=rng.choice(("bf16", "bf16", "f16")), batch=batch, heads=heads,
                    kv=heads // rng.choice((1, 4, 8)), ctx=size(30, min(20000, 100000 // batch)), splits=rng.choice((1, 1, 2, 4, 8)),
                    window=rng.choice((0, 0, 0, 1000)))
    if kind == "gemm":
        if rng.random() < 0.25:
            return dict(kind=kind, dtype="f16", rows=size(1, 100), n=rng.choice((4096, 6144)), k=4096)
        n, k = rng.choice(((4096, 4096), (6144, 4096), (28672, 4096), (4096, 14336), (32000, 4096), (11000, 2048), (1408, 2048)))
        return dict(kind=kind, dtype="bf16", rows=size(1, 3000), n=n, k=k)
    if kind == "experts":
        if rng.random() < 0.5:
            return dict(kind=kind, rows=size(1, 1500), experts=16, top=4, width=2048, ff=1408)
        return dict(kind=kind, rows=size(1, 800), experts=8, top=2, width=4096, ff=7168)
    return dict(kind=kind, dtype=rng.choice(("f16", "f16", "bf16")), tokens=size(1, 2000))


# ------------------------------------------------------------------------------------- inputs
def library():
    return __graft_entry__.load_package()


def randn(gen, *shape, dtype=torch.float32, scale=1.0):
    return (torch.randn(*shape, generator=gen, device=DEVICE) * scale).to(dtype)


def context_lengths(case, seed):
    """Ragged: from a half to one and a half of the stated length, every sequence its own (one alone: the stated one)."""
    rng = np.random.default_rng([seed, 1])
    if case["batch"] == 1:
        return np.array([case["ctx"]])
    return rng.integers(max(1, case["ctx"] // 2), case["ctx"] + case["ctx"] // 2 + 1, case["batch"])


def token_ids(seed, place, n):
    return np.random.default_rng([seed, 2, place]).integers(0, VOCAB, n).astype(np.uint32)


def latarax():
    def gla():
        return {"type": "gla", "mixer": dict(heads=32, dim=64, vdim=128, tau=16.0), "mlp": {"kind": "dense", "ff": FF}}

    def parallel():
        decay = [1.0 - 2.0 ** (-3.0 - 5.0 * i / 15) for i in range(16)]
        return {"type": "parallel",
                "mixer": {"left": dict(heads=32, kv_heads=8, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=1024, keep_first=16)),
                          "right": dict(heads=16, dim=128, vdim=128, decay=decay)},
                "mlp": {"kind": "dense", "ff": FF}}

    return {"architecture": "Latarax", "width": H, "vocab": VOCAB, "streams": 4, "max_positions": 8192, "norm": {"eps": 1e-6},
            "layers": [gla() if i % 2 == 0 else parallel() for i in range(LAYERS)]}


def engine_for(case, seed, tokens, sequences):
    """tokens: of the longest sequence; sequences: as many of that length as the pool holds."""
    hb = library()
    longest = (tokens + BLOCK - 1) // BLOCK * BLOCK + BLOCK
    kw = dict(seed=seed % (1 << 31) + 1, std=STD, max_seq_len=longest, max_batch=ROWS, num_kv_blocks=sequences * (longest // BLOCK))
    if case["kind"] == "serve":
        return hb.Engine.create_random_config(latarax(), max_seqs=sequences, **kw)
    return hb.Engine.create_random(MODEL, bf16=case["dtype"] == "bf16", **kw)


def pinned(*shape):
    return torch.empty(*shape, dtype=torch.float32, pin_memory=True).numpy()


def prepare(case, seed):
    return globals()["prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["run_" + state["kind"]](state)


def prepare_decode(case, seed):
    lens = context_lengths(case, seed)
    most = int(lens.max()) + 1
    eng = engine_for(case, seed, most, case["batch"])
    per = (most + BLOCK - 1) // BLOCK
    tables = np.random.default_rng([seed, 3]).permutation(case["batch"] * per).reshape(case["batch"], per).astype(np.int64)
    for b, n in enumerate(lens):  # the contexts are in the cache before the step
        eng.forward_tables(token_ids(seed, b, n), 0, tables[b])
    last = np.array([token_ids(seed, b, n + 1)[-1] for b, n in enumerate(lens)], dtype=np.uint32)
    return dict(kind="decode", eng=eng, last=last, positions=lens.astype(np.int64), tables=tables, logits=pinned(case["batch"], VOCAB))


def run_decode(s):
    s["eng"].decode_batch_tables(s["last"], s["positions"], s["tables"], logits=s["logits"])
    return s["logits"]


def prepare_prefill(case, seed):
    return dict(kind="prefill", eng=engine_for(case, seed, case["tokens"], 1), ids=token_ids(seed, 0, case["tokens"]))


def run_prefill(s):
    cache = s["eng"].create_kv_cache()
    logits = s["eng"].forward_with_cache(s["ids"], 0, cache)
    cache.free()
    return logits


def prepare_verify(case, seed):
    eng = engine_for(case, seed, case["ctx"] + case["tokens"], 1)
    cache = eng.create_kv_cache()
    ids = token_ids(seed, 0, case["ctx"] + case["tokens"])
    eng.forward_with_cache(ids[:case["ctx"]], 0, cache)
    return dict(kind="verify", eng=eng, cache=cache, ctx=case["ctx"], draft=ids[case["ctx"]:])


def run_verify(s):
    logits = s["eng"].forward_all_positions(s["draft"], s["ctx"], s["cache"])
    s["eng"].truncate(s["cache"], s["ctx"])  # nothing of the draft is accepted here
    return logits


def prepare_mixed(case, seed):
    lens = context_lengths(case, seed)
    eng = engine_for(case, seed, max(int(lens.max()) + 1, case["tokens"]), case["batch"] + case["prompts"])
    caches = []
    for b, n in enumerate(lens):
        caches.append(eng.create_kv_cache())
        eng.forward_with_cache(token_ids(seed, b, n), 0, caches[-1])
    return dict(kind="mixed", eng=eng, caches=caches, lens=lens.tolist(), last=[token_ids(seed, b, n + 1)[-1:] for b, n in enumerate(lens)],
                prompts=[token_ids(seed, case["batch"] + i, case["tokens"]) for i in range(case["prompts"])])


def run_mixed(s):
    eng = s["eng"]
    new = [eng.create_kv_cache() for _ in s["prompts"]]
    entries = [(c, t, [0]) for c, t in zip(s["caches"], s["last"])] + [(c, p, [len(p) - 1]) for c, p in zip(new, s["prompts"])]
    _, logits = eng.step(entries)
    for c, n in zip(s["caches"], s["lens"]):  # the next pass starts where this one did
        eng.truncate(c, n)
    for c in new:
        c.free()
    return logits


def prepare_serve(case, seed):
    eng = engine_for(case, seed, case["tokens"] + case["steps"], case["batch"])
    ids = np.stack([token_ids(seed, b, case["tokens"] + case["steps"]) for b in range(case["batch"])])
    return dict(kind="serve", eng=eng, ids=ids, tokens=case["tokens"], steps=case["steps"], logits=pinned(case["steps"], case["batch"], VOCAB))


def run_serve(s):
    eng, ids, n = s["eng"], s["ids"], s["tokens"]
    caches = [eng.create_kv_cache() for _ in ids]
    per = ROWS // len(ids)
    for at in range(0, n, per):
        end = min(n, at + per)
        _, first = eng.step([(c, t[at:end], [end - at - 1] if end == n else []) for c, t in zip(caches, ids)])
    for i in range(s["steps"]):
        eng.decode_batch(caches, ids[:, n + i], logits=s["logits"][i])
    for c in caches:
        c.free()
    return first, s["logits"]


def prepare_sample(case, seed):
    g = torch.Generator(DEVICE).manual_seed(seed)
    n, v = case["rows"], case["vocab"]
    counts = None
    if case["penalties"]:  # the tokens of a conversation so far
        at = torch.randint(0, v, (n, 400), generator=g, device=DEVICE)
        counts = torch.zeros(n, v, dtype=torch.int32, device=DEVICE).scatter_add_(1, at, torch.ones_like(at, dtype=torch.int32))
    # a language model's distribution: probabilities fall with the rank of a token, some tens make up nine tenths
    logits = -1.2 * torch.log(torch.rand(n, v, generator=g, device=DEVICE) * v + 1) + randn(g, n, v, scale=0.3)
    return dict(kind="sample", logits=logits, counts=counts, seeds=torch.randint(0, 1 << 62, (n,), generator=g, device=DEVICE),
                top_p=case["top_p"], presence=0.4 if case["penalties"] else 0.0, frequency=0.3 if case["penalties"] else 0.0)


TEMPERATURE = 0.8


def run_sample(s):
    if s["top_p"] == 1.0:
        return library().logits_to_probs(s["logits"], TEMPERATURE, s["top_p"], s["counts"], s["presence"], s["frequency"])
    return library().sample(s["logits"], s["seeds"], TEMPERATURE, s["top_p"], s["counts"], s["presence"], s["frequency"])


def prepare_attention(case, seed):
    g = torch.Generator(DEVICE).manual_seed(seed)
    t = TYPES[case["dtype"]]
    lens = context_lengths(case, seed)
    per = (int(lens.max()) + BLOCK - 1) // BLOCK
    held = -(-lens // BLOCK)
    blocks = int(held.sum())
    order = np.random.default_rng([seed, 3]).permutation(blocks).astype(np.int32)
    tables = np.zeros((case["batch"], per), dtype=np.int32)
    at = 0
    for b, n in enumerate(held):
        tables[b, :n] = order[at:at + n]
        at += n
    return dict(kind="attention", q=randn(g, case["batch"], case["heads"], DIM, dtype=t), k=randn(g, blocks, case["kv"], BLOCK, DIM, dtype=t),
                v=randn(g, blocks, case["kv"], BLOCK, DIM, dtype=t), tables=torch.from_numpy(tables).to(DEVICE),
                lens=torch.from_numpy(lens.astype(np.int32)).to(DEVICE), splits=case["splits"], window=case["window"])


def run_attention(s):
    return library().paged_decode_attention(s["q"], s["k"], s["v"], s["tables"], s["lens"], n_splits=s["splits"], sliding_window=s["window"])


def prepare_gemm(case, seed):
    g = torch.Generator(DEVICE).manual_seed(seed)
    t = TYPES[case["dtype"]]
    return dict(kind="gemm", x=randn(g, case["rows"], case["k"], dtype=t), w=randn(g, case["n"], case["k"], dtype=t, scale=0.02))


def run_gemm(s):
    return library().gemm(s["x"], s["w"])


def prepare_experts(case, seed):
    hb = library()
    g = torch.Generator(DEVICE).manual_seed(seed)
    rows, E, top, w, ff = (case[k] for k in ("rows", "experts", "top", "width", "ff"))
    picks = rows * top
    m_pad = min(128, max(16, -(-math.ceil(picks * 1.5 / E) // 16) * 16))
    tiles = min(E, picks) + picks // m_pad
    bf = torch.bfloat16
    s = dict(kind="experts", rows=rows, width=w, h=randn(g, rows, w, dtype=bf), router=randn(g, E, w, dtype=bf, scale=w ** -0.5),
             up=randn(g, E, 2 * ff, w, dtype=bf, scale=w ** -0.5), down=randn(g, E, w, ff, dtype=bf, scale=ff ** -0.5),
             norm=1 + randn(g, w, scale=0.1), one=torch.ones(1, device=DEVICE), zero=torch.zeros(1, device=DEVICE),
             residual=torch.zeros(rows, w, device=DEVICE), out=torch.empty(rows, w, dtype=bf, device=DEVICE),
             x=torch.zeros(tiles * m_pad, w, dtype=bf, device=DEVICE), act=torch.zeros(tiles * m_pad, ff, dtype=bf, device=DEVICE),
             y=torch.zeros(tiles * m_pad, w, dtype=bf, device=DEVICE), weight=torch.zeros(rows, top, device=DEVICE))
    ints = [torch.zeros(*n, dtype=torch.int32, device=DEVICE) for n in ((rows, top), (rows, top), (rows, top), (E + 1,), (E,), (tiles,))]
    ids, rank, place, count, first, group = (t.data_ptr() for t in ints)
    silu = hb.GatedActSpec(1.0, 0.0, math.inf, 0.0)
    likely = max(1, min(tiles, round(min(E, picks) * max(1.0, math.ceil(picks / min(E, picks) / m_pad)))))
    s.update(ints=ints, routing=hb.MoeRouting(E, top, m_pad, tiles, ids, rank, place, s["weight"].data_ptr(), count, first, group),
             gate_up=hb.GroupedGemm(E, 2 * ff, w, m_pad, tiles, likely, group, w, ff, 1, 0, silu),
             down_gemm=hb.GroupedGemm(E, w, ff, m_pad, tiles, likely, group, ff, w, 0, 0, silu),
             # one residual stream that takes the mixture's output alone
             mix=hb.StreamMixArgs(s["zero"].data_ptr(), s["one"].data_ptr(), s["one"].data_ptr(), s["norm"].data_ptr(), None, None, 0.0,
                                  None, s["y"].data_ptr(), place, s["weight"].data_ptr(), top))
    return s


def run_experts(s):
    hb = library()
    st, rows, w, ref = torch.cuda.current_stream().cuda_stream, s["rows"], s["width"], ctypes.byref
    ptr = lambda name: s[name].data_ptr()  # noqa: E731
    hb.check(hb.lib.hb_moe_route_top(st, ref(s["routing"]), ptr("h"), w, ptr("router"), None, rows, w, hb.BF16))
    hb.check(hb.lib.hb_moe_gather(st, ref(s["routing"]), ptr("x"), ptr("h"), w, rows, hb.BF16))
    hb.check(hb.lib.hb_gemm_grouped(st, ptr("act"), ptr("x"), ptr("up"), ref(s["gate_up"]), hb.BF16))
    hb.check(hb.lib.hb_gemm_grouped(st, ptr("y"), ptr("act"), ptr("down"), ref(s["down_gemm"]), hb.BF16))
    hb.check(hb.lib.hb_streams_mix_ex(st, ptr("residual"), ptr("out"), None, None, w, ref(s["mix"]), rows, 1, w, w, 1e-6, hb.BF16))
    return s["residual"], s["out"], s["weight"]


def prepare_glue(case, seed):
    g = torch.Generator(DEVICE).manual_seed(seed)
    t, n = TYPES[case["dtype"]], case["tokens"]
    inv = torch.from_numpy(library().kernels.rope.inv_freq(MODEL["rope_theta"], DIM)).to(DEVICE)
    angle = torch.arange(100, 100 + n, device=DEVICE).float()[:, None] * inv
    blocks = (n + BLOCK - 1) // BLOCK + 4
    slots = torch.randperm(blocks * BLOCK, generator=g, device=DEVICE)[:n].contiguous()
    return dict(kind="glue", x=randn(g, n, H, dtype=t), residual=randn(g, n, H, dtype=t), norm=randn(g, H, dtype=t, scale=0.1) + 1,
                q=randn(g, 1, HEADS, n, DIM, dtype=t), k=randn(g, 1, KV, n, DIM, dtype=t), cos=angle.cos().to(t), sin=angle.sin().to(t),
                new_k=randn(g, n, KV, DIM, dtype=t), new_v=randn(g, n, KV, DIM, dtype=t), slots=slots,
                kc=torch.zeros(blocks, KV, BLOCK, DIM, dtype=t, device=DEVICE), vc=torch.zeros(blocks, KV, BLOCK, DIM, dtype=t, device=DEVICE),
                gate_up=randn(g, n, 2 * FF, dtype=t))


def run_glue(s):
    hb = library()
    k = hb.kernels
    normed, residual = k.rms_norm.add_apply(s["x"], s["residual"], s["norm"], 1e-6)
    q, key = k.rope.apply(s["q"], s["k"], s["cos"], s["sin"])
    k.kv_assign.assign_paged(s["kc"], s["vc"], s["new_k"], s["new_v"], s["slots"])
    return dict(normed=normed, residual=residual, q=q, k=key, kc=s["kc"], vc=s["vc"], gated=hb.silu_mul(s["gate_up"]))


# --------------------------------------------------------------------------------------- work
def work(case):
    """Weights, cached keys and values, inputs and outputs once; the products' and the attention's operations."""
    kind = case["kind"]
    kv_token = 2 * KV * DIM * 2.0  # bytes of a token in one layer's cache
    attn_flops = 4.0 * HEADS * DIM
    if kind in ("decode", "verify", "mixed", "prefill"):
        if kind == "decode":
            rows, seen, read, wanted = case["batch"], case["batch"] * (case["ctx"] + 1.0), case["batch"] * (case["ctx"] + 1.0), case["batch"]
        elif kind == "prefill":
            rows = case["tokens"]
            seen, read, wanted = rows * (rows + 1) / 2.0, rows, 1
        elif kind == "verify":
            rows = case["tokens"]
            seen, read, wanted = rows * (case["ctx"] + (rows + 1) / 2.0), case["ctx"] + rows, rows
        else:
            n = case["prompts"] * case["tokens"]
            rows, wanted = case["batch"] + n, case["batch"] + case["prompts"]
            seen = case["batch"] * (case["ctx"] + 1.0) + n * (case["tokens"] + 1) / 2.0
            read = case["batch"] * (case["ctx"] + 1.0) + n
        return {"bytes": 2.0 * (PARAMS + VOCAB * H) + 2.0 * rows * H + LAYERS * kv_token * (read + rows) + 4.0 * wanted * VOCAB,
                "flops": 2.0 * PARAMS * rows + 2.0 * VOCAB * H * wanted + LAYERS * attn_flops * seen}
    if kind == "serve":
        b, n, steps = case["batch"], case["tokens"], case["steps"]
        pairs = LAYERS // 2
        params = pairs * (H * (32 * 64 * 2 + 32 * 128 * 3 + 16) + H * ((32 + 16) * DIM + 16 * 128 * 4 + 16 * 128 + 32 * DIM) + 6 * FF * H)
        state = pairs * 4.0 * (32 * 64 * 128 + 16 * 128 * 128)
        seen = pairs * sum(min(p + 1, 1040) for p in range(n + steps))
        return {"bytes": (1 + steps) * (2.0 * params + 2.0 * VOCAB * H + 2 * b * state) + 2.0 * b * (n + steps) * H + 4.0 * (1 + steps) * b * VOCAB
                + pairs * kv_token * b * (n + sum(min(n + i, 1040) for i in range(steps))),
                "flops": b * (n + steps) * (2.0 * params + 6.0 * state / 4) + 2.0 * VOCAB * H * b * (1 + steps) + b * attn_flops * seen}
    if kind == "sample":
        n = case["rows"] * case["vocab"]
        return {"bytes": n * (12.0 if case["penalties"] else 8.0), "flops": 4.0 * n}
    if kind == "attention":
        span = min(case["ctx"], case["window"] or case["ctx"]) * float(case["batch"])
        return {"bytes": 4.0 * span * case["kv"] * DIM + 4.0 * case["batch"] * case["heads"] * DIM, "flops": 4.0 * span * case["heads"] * DIM}
    if kind == "gemm":
        m, n, k = case["rows"], case["n"], case["k"]
        return {"bytes": 2.0 * (m * k + n * k + m * n), "flops": 2.0 * m * n * k}
    if kind == "experts":
        rows, E, top, w, ff = (case[k] for k in ("rows", "experts", "top", "width", "ff"))
        active = E * (1.0 - (1.0 - top / E) ** rows)
        return {"bytes": 6.0 * active * ff * w + 2.0 * E * w + rows * w * 8.0, "flops": rows * (6.0 * top * ff * w + 2.0 * E * w)}
    n = case["tokens"]
    return {"bytes": n * 2.0 * (4 * H + 2 * (HEADS + KV) * DIM + 4 * KV * DIM + 3 * FF) + 2.0 * H + 2.0 * n * DIM + 8.0 * n, "flops": 8.0 * n * FF}


def tolerance(case):
    """Four times the distance between two correct forms of the same precision, as measured: products on CUDA cores and on
    tensor cores, norms before and after a product (models: 1.1 % in bf16, an eighth of that in f16), else from `exact`."""
    kind, half = case["kind"], case.get("dtype") == "f16"
    if kind in ("decode", "prefill", "verify", "mixed", "serve"):
        return {"rel": 0.006 if half else 0.03}
    if kind == "sample":
        return {"rel": 1e-6, "max": 1e-4}
    return {"rel": 0.012 / (8 if half else 1)}


# -------------------------------------------------------------------------- the same in 64 bits
def signed(v):
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


def splitmix(x):
    """The splitmix64 finaliser on int64 tensors (products wrap, shifts bring in zeros)."""
    shift = lambda v, n: (v >> n) & ((1 << (64 - n)) - 1)  # noqa: E731
    x = x + signed(0x9E3779B97F4A7C15)
    x = (x ^ shift(x, 30)) * signed(0xBF58476D1CE4E5B9)
    x = (x ^ shift(x, 27)) * signed(0x94D049BB133111EB)
    return x ^ shift(x, 31)


def weight(seed, tensor, rows, cols, dtype):
    """The random matrix that an engine of this seed draws for a tensor (its number, or its name), in 64 bits."""
    if isinstance(tensor, str):
        name, tensor = tensor, 1469598103934665603
        for c in name.encode():
            tensor = ((tensor ^ c) * 1099511628211) & ((1 << 64) - 1)
    key = signed((seed % (1 << 31) + 1) * 0xD1342543DE82EF95 + tensor * 0x9E3779B97F4A7C15 + 1)
    out = torch.empty(rows * cols, dtype=torch.float64, device=DEVICE)
    for at in range(0, rows * cols, 1 << 26):
        z = splitmix(key ^ splitmix(torch.arange(at, min(rows * cols, at + (1 << 26)), device=DEVICE)))
        u1 = (((z >> 40) & 0xFFFFFF) + 1).float() / 16777216.0
        u2 = (((z >> 16) & 0xFFFFFF).float() + 0.5) / 16777216.0
        value = torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2) * STD
        out[at:at + len(z)] = value.to(dtype).double()
    return out.view(rows, cols)


def rms(x, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def silu(x):
    return x * torch.sigmoid(x)


def causal(q, k, v, visible=None):
    """q [n, heads, d], k and v [n, kv, d] of one sequence: softmax over what `visible` (or the past) allows."""
    n, rep = len(q), q.shape[1] // k.shape[1]
    mask = torch.ones(n, n, dtype=torch.bool, device=DEVICE).tril() if visible is None else visible
    out = torch.empty_like(q)
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // rep].T) * q.shape[2] ** -0.5
        out[:, h] = torch.softmax(s.masked_fill(~mask, -math.inf), dim=-1) @ v[:, h // rep]
    return out


def in_pieces(f, x, rows=8192):
    return torch.cat([f(x[i:i + rows]) for i in range(0, len(x), rows)])


def model_in_64_bits(seed, dtype, sequences, wanted):
    """Logits of the last wanted[i] tokens of every sequence."""
    t = TYPES[dtype]
    lens = [len(s) for s in sequences]
    ids = torch.from_numpy(np.concatenate(sequences).astype(np.int64)).to(DEVICE)
    pos = torch.cat([torch.arange(n, device=DEVICE) for n in lens]).double()
    angle = pos[:, None] * MODEL["rope_theta"] ** (-torch.arange(0, DIM, 2, device=DEVICE).double() / DIM)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rotated(x):
        a, b = x[..., :DIM // 2], x[..., DIM // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    x = weight(seed, 0, VOCAB, H, t)[ids]
    for layer in range(LAYERS):
        w = lambda i, rows, cols: weight(seed, 16 + 16 * layer + i, rows, cols, t)  # noqa: E731
        h = rms(x)
        q, k, v = ((h @ w(i, n * DIM, H).T).view(-1, n, DIM) for i, n in ((0, HEADS), (1, KV), (2, KV)))
        q, k = rotated(q), rotated(k)
        at, parts = 0, []
        for n in lens:
            parts.append(causal(q[at:at + n], k[at:at + n], v[at:at + n]))
            at += n
        x = x + torch.cat(parts).view(-1, H) @ w(3, H, H).T
        gate, up, down = w(4, FF, H), w(5, FF, H), w(6, H, FF)
        x = in_pieces(lambda y: y + (silu(rms(y) @ gate.T) * (rms(y) @ up.T)) @ down.T, x)
    at, rows = 0, []
    for n, some in zip(lens, wanted):
        at += n
        rows += range(at - some, at)
    return rms(x[rows]) @ weight(seed, 1, VOCAB, H, t).T


def latarax_in_64_bits(seed, ids, wanted):
    """Logits of the last `wanted` tokens of sequences of one length: [batch, wanted, vocab]."""
    t = torch.bfloat16
    batch, n = ids.shape
    w = lambda name, rows, cols: weight(seed, name, rows, cols, t)  # noqa: E731
    x = w("embed", VOCAB, H)[torch.from_numpy(ids.astype(np.int64)).to(DEVICE)] + w("pos", 8192, H)[:n]
    x = x[None].repeat(4, 1, 1, 1)  # streams; neutral mixing: read the mean, add to every one
    i = torch.arange(n, device=DEVICE)
    far = i[:, None] - i[None, :]
    visible = (far >= 0) & ((far < 1024) | (i[None, :] < 16))

    def recurrence(q, k, v, decay):
        state = torch.zeros(batch, q.shape[2], q.shape[3], v.shape[3], dtype=torch.float64, device=DEVICE)
        out = torch.empty_like(v)
        for at in range(n):
            state = decay[:, at, :, :, None] * state + k[:, at, :, :, None] * v[:, at, :, None, :]
            out[:, at] = torch.einsum("bhdv,bhd->bhv", state, q[:, at])
        return out

    for layer, spec in enumerate(latarax()["layers"]):
        p = "l%d." % layer
        h, m = rms(x.mean(0)), spec["mixer"]
        rows = lambda name, heads, dim: (h @ w(p + "mix." + name, heads * dim, H).T).view(batch, n, heads, dim)  # noqa: E731
        if spec["type"] == "gla":
            low = h @ w(p + "mix.a1", 16, H).T @ weight(seed, p + "mix.a2", 32 * 64, 16, torch.float32).T + 1.0
            decay = torch.sigmoid(low).pow(1.0 / 16.0).view(batch, n, 32, 64)
            o = rms(recurrence(rows("q", 32, 64) * 64 ** -0.5, rows("k", 32, 64), rows("v", 32, 128), decay))
            y = (o * silu(rows("g", 32, 128))).view(batch, n, H) @ w(p + "mix.o", H, 32 * 128).T
        else:
            q, k, v = rows("left.q", 32, 128), rows("left.k", 8, 128), rows("left.v", 8, 128)
            left = torch.stack([causal(q[b], k[b], v[b], visible) for b in range(batch)]).view(batch, n, H) @ w(p + "mix.left.o", H, H).T
            decay = torch.tensor(np.float32(m["right"]["decay"]), device=DEVICE).double()[None, None, :, None].expand(batch, n, 16, 128)
            o = recurrence(*(silu(rows("right." + name, 16, 128)) for name in "qkv"), decay)
            o = rms(o.reshape(batch, n, 2048)) * torch.sigmoid(rows("right.g", 16, 128).view(batch, n, 2048))
            y = 0.5 * (rms(left) + rms(o @ w(p + "mix.right.o", H, 2048).T))
        x = x + y
        h = rms(x.mean(0))
        x = x + (silu(h @ w(p + "mlp.gate", FF, H).T) * (h @ w(p + "mlp.up", FF, H).T)) @ w(p + "mlp.down", H, FF).T
    return rms(x.sum(0)[:, n - wanted:]) @ w("head", VOCAB, H).T


def exact(case, seed):
    kind = case["kind"]
    if kind in ("decode", "mixed"):
        lens = context_lengths(case, seed)
        sequences = [token_ids(seed, b, n + 1) for b, n in enumerate(lens)]
        if kind == "mixed":
            sequences += [token_ids(seed, case["batch"] + i, case["tokens"]) for i in range(case["prompts"])]
        return model_in_64_bits(seed, case["dtype"], sequences, [1] * len(sequences))
    if kind == "prefill":
        return model_in_64_bits(seed, case["dtype"], [token_ids(seed, 0, case["tokens"])], [1])[0]
    if kind == "verify":
        return model_in_64_bits(seed, case["dtype"], [token_ids(seed, 0, case["ctx"] + case["tokens"])], [case["tokens"]])
    if kind == "serve":
        n, steps = case["tokens"], case["steps"]
        ids = np.stack([token_ids(seed, b, n + steps) for b in range(case["batch"])])
        logits = latarax_in_64_bits(seed, ids, steps + 1)
        return logits[:, 0].contiguous(), logits[:, 1:].transpose(0, 1).contiguous()
    s = prepare(case, seed)
    if kind == "sample":
        z = s["logits"].double()
        if s["counts"] is not None:
            c = s["counts"].double()
            z = z - (c > 0) * s["presence"] - s["frequency"] * c / c.sum(1, keepdim=True).clamp(min=1)
        p = torch.softmax(z / TEMPERATURE, dim=1)
        if case["top_p"] < 1:
            down = p.sort(dim=1, descending=True).values
            last = (down.cumsum(1) < case["top_p"]).sum(1, keepdim=True).clamp(max=p.shape[1] - 1)
            p = p * (p >= down.gather(1, last))
        p = p / p.sum(1, keepdim=True)
        return p if case["top_p"] == 1.0 else (None, p)  # the draws themselves are whole numbers
    if kind == "attention":
        out, rep = torch.empty(s["q"].shape, dtype=torch.float64, device=DEVICE), case["heads"] // case["kv"]
        for b, n in enumerate(s["lens"].tolist()):
            first = max(0, n - case["window"]) if case["window"] else 0
            at = s["tables"][b, :(n + BLOCK - 1) // BLOCK].long()
            k, v = (s[c][at].transpose(1, 2).reshape(-1, case["kv"], DIM)[first:n].double().transpose(0, 1) for c in ("k", "v"))
            q = s["q"][b].double().view(case["kv"], rep, DIM)
            out[b] = (torch.softmax(q @ k.transpose(1, 2) * DIM ** -0.5, -1) @ v).reshape(case["heads"], DIM)
        return out
    if kind == "gemm":
        return s["x"].double() @ s["w"].double().T
    if kind == "experts":
        h, ff = s["h"].double(), case["ff"]
        best, chosen = (h @ s["router"].double().T).topk(case["top"], dim=1)
        share = torch.softmax(best, dim=1)
        y = torch.zeros_like(h)
        for e in range(case["experts"]):
            row, k = (chosen == e).nonzero(as_tuple=True)
            up = h[row] @ s["up"][e].double().T
            y.index_add_(0, row, share[row, k, None] * ((silu(up[:, :ff]) * up[:, ff:]) @ s["down"][e].double().T))
        return y, rms(y) * s["norm"].double(), share
    if kind == "glue":
        x = s["x"].double() + s["residual"].double()
        turn = []
        for a in (s["q"].double(), s["k"].double()):
            u, v = a[..., :DIM // 2], a[..., DIM // 2:]
            c, n = s["cos"].double(), s["sin"].double()
            turn.append(torch.cat([u * c - v * n, u * n + v * c], -1))
        cache = {}
        for name, new in (("kc", "new_k"), ("vc", "new_v")):
            cache[name] = s[name].double()
            cache[name][s["slots"] // BLOCK, :, s["slots"] % BLOCK] = s[new].double()
        gate, up = s["gate_up"].double().chunk(2, dim=1)
        return dict(normed=rms(x) * s["norm"].double(), residual=x, q=turn[0], k=turn[1], gated=silu(gate) * up, **cache)
    return None
