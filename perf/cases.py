"""Performance cases of the framework: the work a user has it do, through its public entry points.

Three families. Batch-1 sessions (`InferenceSession`: chat and scoring, f32 parity mode and bf16), continuous batching
(`Engine`: bf16 serving of ragged sequences, three model sizes), and the fused kernels called on their own (`ops`).
Sizes are those of the model configurations, the benchmark and the microbenchmarks, with odd and small ones beside them.

Lengths (prompts, KV lengths) belong to the case, token ids and tensor values come from the seed, so a case does the
same work for every seed. The engine's and sessions' handles and the weights are built once per configuration and kept,
as a serving program keeps them.
"""
import collections
import math

import numpy as np
import torch

import __graft_entry__ as entry

ak = entry.load_package()
ops = ak.ops

MODELS = {"hall_162m": ak.ModelConfig.akasha_hall_1, "pidgeon": ak.ModelConfig.pidgeon, "scaled_1p4b": ak.ModelConfig.scaled_1p4b}
CHAT = dict(temperature=0.8, top_k=40, top_p=0.95, repetition_penalty=1.15)   # the chat command's sampler settings
SESSION_CTX = 1024
ESZ = {"f32": 4, "bf16": 2}
DT = {"f32": ak.AK_F32, "bf16": ak.AK_BF16}
EPI = {"store_f32": ak.EPI_STORE_F32, "add_f32": ak.EPI_ADD_F32, "store_bf16": ak.EPI_STORE_BF16, "silu_bf16": ak.EPI_SILU_BF16}


def listed():
    return [
        # A chat turn on the 162M model in parity mode, the reference's own configuration: 64-token prompt, 128 greedy tokens.
        {"name": "chat_greedy_f32", "kind": "chat", "model": "hall_162m", "dtype": "f32", "prompt": 64, "new": 128, "sampled": False},
        # Scoring a text in parity mode: a full 512-token context prefilled, then given tokens, logits back on the host each time.
        {"name": "score_f32", "kind": "score", "model": "hall_162m", "dtype": "f32", "prompt": 512, "new": 16},
        # The chat command: short odd prompt, sampled with its temperature / top-k / top-p / repetition penalty.
        {"name": "chat_sampled_f32", "kind": "chat", "model": "hall_162m", "dtype": "f32", "prompt": 23, "new": 64, "sampled": True},
        # One user on the bf16 model: prefill of an odd-length prompt, then single-token steps with logits.
        {"name": "score_bf16", "kind": "score", "model": "hall_162m", "dtype": "bf16", "prompt": 201, "new": 24},
        # The serving benchmark's shape at half its queue: 64 in flight, prompts U[16,448], each run to length 512.
        {"name": "serve_162m_64", "kind": "serve", "model": "hall_162m", "slots": 64, "seqs": 128, "lo": 16, "hi": 448, "total": 512,
         "gen": 0, "eos": False, "lens": 2},
        # A lightly loaded server: 8 in flight, 64 tokens each.
        {"name": "serve_162m_8", "kind": "serve", "model": "hall_162m", "slots": 8, "seqs": 12, "lo": 16, "hi": 448, "total": 512,
         "gen": 64, "eos": False, "lens": 3},
        # The small model, sequences that end at their end-of-sequence token (each step's tokens are read before the next).
        {"name": "serve_pidgeon_eos", "kind": "serve", "model": "pidgeon", "slots": 21, "seqs": 40, "lo": 1, "hi": 300, "total": 512,
         "gen": 128, "eos": True, "lens": 4},
        # The 1.4B model: long ragged prompts, short answers.
        {"name": "serve_1p4b", "kind": "serve", "model": "scaled_1p4b", "slots": 16, "seqs": 24, "lo": 128, "hi": 3072, "total": 3200,
         "gen": 24, "eos": False, "lens": 5},
        # Decode attention of a large ragged batch (the attention microbenchmark).
        {"name": "attn_decode_1024", "kind": "attn_decode", "rows": 1024, "heads": 12, "head_dim": 64, "lo": 1, "hi": 512, "dtype": "bf16",
         "append": False, "lens": 3},
        # Prefill projection of the 162M model over 32768 prompt tokens: ffn-up with its SiLU.
        {"name": "gemm_prefill", "kind": "gemm", "m": 32768, "n": 3072, "k": 768, "epilogue": "silu_bf16"},
        # Causal prefill attention of 16 ragged prompts, head size of the 1.4B model.
        {"name": "attn_prefill", "kind": "attn_prefill", "seqs": 16, "heads": 16, "head_dim": 128, "lo": 128, "hi": 3072, "lens": 5},
        # Fused RMSNorm + RoPE over the rows of a large prefill.
        {"name": "norm_rope", "kind": "norm", "rows": 32768, "size": 768, "head_dim": 64, "residual": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chat", "score", "serve", "serve", "attn_decode", "gemm", "attn_prefill", "norm"])
    if kind == "chat":
        dtype = rng.choice(["f32", "f32", "bf16"])
        return {"kind": kind, "model": rng.choice(["hall_162m", "pidgeon"]), "dtype": dtype, "prompt": _log(rng, 1, 512), "new": _log(rng, 4, 128),
                "sampled": rng.random() < 0.4}
    if kind == "score":
        return {"kind": kind, "model": rng.choice(["hall_162m", "pidgeon"]), "dtype": rng.choice(["f32", "bf16"]), "prompt": _log(rng, 1, 512),
                "new": rng.randint(1, 48)}
    if kind == "serve":
        model = rng.choice(["hall_162m", "hall_162m", "pidgeon", "scaled_1p4b"])
        big = model == "scaled_1p4b"
        slots = _log(rng, 1, 16 if big else 64)
        lo = _log(rng, 1, 256)
        hi = rng.randint(lo, 3072 if big else 448)
        return {"kind": kind, "model": model, "slots": slots, "seqs": slots + rng.randint(0, slots // 2 + 1), "lo": lo, "hi": hi,
                "total": 3200 if big else 512, "gen": _log(rng, 4, 24 if big else 64), "eos": rng.random() < 0.3, "lens": rng.randrange(1 << 20)}
    if kind == "attn_decode":
        heads, hd = rng.choice([(12, 64), (5, 64), (16, 128)])
        rows, hi = _log(rng, 1, 1024), _log(rng, 16, 512)
        return {"kind": kind, "rows": rows, "heads": heads, "head_dim": hd, "lo": 1, "hi": hi, "dtype": rng.choice(["bf16", "bf16", "f32"]),
                "append": rng.random() < 0.5, "lens": rng.randrange(1 << 20)}
    if kind == "gemm":
        n, k = rng.choice([(2304, 768), (768, 768), (3072, 768), (768, 3072), (960, 320), (1280, 320), (320, 1280), (6144, 2048), (2048, 2048), (8192, 2048),
                           (2048, 8192), (50257, 768)])
        m = _log(rng, 1, 2048 if n * k > 1 << 22 else 32768)
        return {"kind": kind, "m": m, "n": n, "k": k, "epilogue": rng.choice(sorted(EPI))}
    if kind == "attn_prefill":
        heads, hd = rng.choice([(12, 64), (5, 64), (16, 128)])
        hi = _log(rng, 16, 3072)
        return {"kind": kind, "seqs": rng.randint(1, 16), "heads": heads, "head_dim": hd, "lo": rng.randint(1, hi), "hi": hi, "lens": rng.randrange(1 << 20)}
    return {"kind": kind, "rows": _log(rng, 1024, 32768), "size": rng.choice([320, 768, 2048]), "head_dim": rng.choice([0, 64]), "residual": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------- kept handles
_kept = {}                              # the context and the weights of each (model, dtype, confident)
_handles = collections.OrderedDict()    # the last few engines and sessions


def _ctx():
    if "ctx" not in _kept:
        _kept["ctx"] = ak.Context(0)
    return _kept["ctx"]


def _successor(vocab):
    """The fixed permutation a confident model follows (see _weights)."""
    return torch.randperm(vocab, generator=torch.Generator().manual_seed(17))


def _weights(model, dtype, confident):
    """Seeded random-init weights. `confident`: the embedding carries more of the residual stream and the lm_head's column
    for a token's successor is aligned with that token's embedding, so that the greedy choice stands well clear of the
    rest, as a trained model's does. (Random-init logits have top-2 margins near bf16's rounding error: one rounding
    then decides a token, and with it every later one.)"""
    key = (model, dtype, confident)
    if key not in _kept:
        cfg = MODELS[model]()
        w = ak.ModelWeights(_ctx(), cfg, DT[dtype])
        w.init_synthetic(0, 0.02)
        if confident:
            V, D = cfg.vocab_size, cfg.dim
            emb = 2.0 * torch.randn(V, D, device="cuda", generator=torch.Generator(device="cuda").manual_seed(11))
            head = torch.empty(V, D, device="cuda")
            head[_successor(V).cuda()] = emb / (2.0 * math.sqrt(D))     # logits of the other tokens: standard deviation 1
            for index, t in ((0, emb), (len(cfg.param_shapes()) - 1, head.T.contiguous())):
                a = t.cpu().numpy()
                ak.check(ak.lib().ak_weights_set_param(w.h, index, a.ctypes.data_as(ak.f32p), a.size))
        _kept[key] = w
    return _kept[key]


def _handle(key, make):
    if key not in _handles:
        while len(_handles) >= 3:
            _handles.popitem(last=False)[1].close()
        _handles[key] = make()
    return _handles[key]


def _session(c):
    # free-running bf16 generation follows its own choices, so it gets the confident weights; scoring is given its tokens
    confident = c["kind"] == "chat" and c["dtype"] == "bf16"
    return _handle(("session", c["model"], c["dtype"], confident),
                   lambda: ak.InferenceSession(_ctx(), _weights(c["model"], c["dtype"], confident), SESSION_CTX))


def _engine(c):
    big = c["model"] == "scaled_1p4b"
    return _handle(("engine", c["model"], c["slots"], c["total"], c["eos"]),
                   lambda: ak.Engine(_ctx(), _weights(c["model"], "bf16", True), max_seqs=c["slots"], max_seq_len=c["total"],
                                     max_batch_tokens=c["slots"] + 16384 if big else 0, use_cuda_graph=True, stop_on_eos=c["eos"],
                                     async_steps=not c["eos"]))


# ---------------------------------------------------------------------------------------------- inputs
def _lens(c, n):
    return ak.uniform_ints(n, c["lo"], c["hi"], seed=c["lens"])


def _serve_limits(c):
    """(prompt length, total length limit, tokens until the end-of-sequence token) of every sequence."""
    plen = _lens(c, c["seqs"])
    limit = np.minimum(plen + c["gen"], c["total"]) if c["gen"] else np.full(c["seqs"], c["total"])
    until = ak.uniform_ints(c["seqs"], 1, 2 * max(1, c["gen"]), seed=c["lens"] + 1)
    return plen, limit, until


def _bf16(g, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).bfloat16()


def _values(g, dtype, *shape):
    t = torch.randn(*shape, device="cuda", generator=g)
    return t.bfloat16() if dtype == "bf16" else t


def _rope_table(length, head_dim):
    freq = 1.0 / torch.pow(torch.tensor(10000.0), torch.arange(0, head_dim, 2, dtype=torch.float32) / head_dim)
    angle = torch.arange(length, dtype=torch.float32)[:, None] * freq[None, :]
    return torch.stack((torch.cos(angle), torch.sin(angle)), -1).contiguous().cuda()


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    rng = np.random.RandomState(seed % (1 << 31))
    s = {"c": c}
    if kind in ("chat", "score"):
        cfg = MODELS[c["model"]]()
        _session(c)
        s["prompt"] = rng.randint(0, cfg.vocab_size, c["prompt"]).astype(np.uint32)
        s["given"] = [int(t) for t in rng.randint(0, cfg.vocab_size, c["new"])]
        s["seed"] = int(seed)
        return s
    if kind == "serve":
        cfg = MODELS[c["model"]]()
        _engine(c)
        plen, limit, until = _serve_limits(c)
        s["prompts"] = [rng.randint(0, cfg.vocab_size - 1, int(n)).astype(np.uint32) for n in plen]
        s["limit"] = [int(v) for v in limit]
        if c["eos"]:   # the last prompt token lies `until` steps before the end-of-sequence token
            succ = _successor(cfg.vocab_size).numpy()
            pred = np.empty_like(succ)
            pred[succ] = np.arange(succ.size)
            for p, u in zip(s["prompts"], rng.permutation(until)):
                t = cfg.eos_token
                for _ in range(int(u)):
                    t = pred[t]
                p[-1] = t
        s["cap"] = int((limit - plen).max())
        return s
    g = torch.Generator(device="cuda").manual_seed(seed)
    if kind == "attn_decode":
        rows, H, hd = c["rows"], c["heads"], c["head_dim"]
        lens = _lens(c, rows)
        mb = (c["hi"] + 15) // 16
        nb = rows * mb
        s["k"], s["v"] = (_values(g, c["dtype"], nb, H, 16, hd) for _ in range(2))
        s["tables"] = torch.randperm(nb, device="cuda", generator=g).to(torch.int32).reshape(rows, mb)
        s["kv_lens"] = torch.from_numpy(lens.astype(np.int32)).cuda()
        if c["append"]:
            s["qkv"] = torch.randn(rows, 3 * H * hd, device="cuda", generator=g)
            s["rope"] = _rope_table(c["hi"], hd)
        else:
            s["q"] = _values(g, c["dtype"], rows, H * hd)
        s["out"] = torch.empty(rows, H * hd, device="cuda", dtype=s["k"].dtype)
        n = ops.attn_decode_scratch_bytes(rows, H, hd, mb, 0, DT[c["dtype"]])
        s["scratch"] = torch.zeros(max(n, 16), dtype=torch.uint8, device="cuda")
        s["mb"], s["nb"] = mb, nb
    elif kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        s["a"], s["wt"] = _bf16(g, m, k), _bf16(g, n, k, scale=0.02)
        s["ldc"] = (n + 7) // 8 * 8     # a row pitch of whole 16-byte vectors
        s["c_out"] = torch.zeros(m, s["ldc"], device="cuda", dtype=torch.bfloat16 if c["epilogue"].endswith("bf16") else torch.float32)
    elif kind == "attn_prefill":
        n, H, hd = c["seqs"], c["heads"], c["head_dim"]
        lens = _lens(c, n)
        mb = (int(lens.max()) + 15) // 16
        nb = n * mb
        s["k"], s["v"] = _bf16(g, nb, H, 16, hd), _bf16(g, nb, H, 16, hd)
        s["tables"] = torch.randperm(nb, device="cuda", generator=g).to(torch.int32).reshape(n, mb)
        cu = np.zeros(n + 1, np.int32)
        cu[1:] = np.cumsum(lens)
        s["rows"], s["max_len"] = int(cu[-1]), int(lens.max())
        s["q"] = _bf16(g, s["rows"], H * hd)
        s["out"] = torch.empty_like(s["q"])
        s["cu"] = torch.from_numpy(cu).cuda()
        s["slot"] = torch.arange(n, dtype=torch.int32, device="cuda")
        s["mb"], s["nb"] = mb, nb
    else:
        rows, size = c["rows"], c["size"]
        s["x"] = torch.randn(rows, size, device="cuda", generator=g)
        s["res"] = torch.randn(rows, size, device="cuda", generator=g) if c["residual"] else None
        s["w"] = 1.0 + 0.02 * torch.randn(size, device="cuda", generator=g)
        s["y"] = torch.empty(rows, size, device="cuda", dtype=torch.bfloat16)
        s["pos"] = (torch.arange(rows, device="cuda", dtype=torch.int32) % 512).contiguous() if c["head_dim"] else None
    return s


# ---------------------------------------------------------------------------------------------- one pass
def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "chat":
        ses = _session(c)
        ses.replace_cache()
        sampler = dict(CHAT, seed=s["seed"]) if c["sampled"] else {}
        return ses.generate(s["prompt"], c["new"], stop_on_eos=False, **sampler)
    if kind == "score":
        ses = _session(c)
        ses.replace_cache()
        got = [ses.prefill(s["prompt"])[0]]
        for t in s["given"]:
            got.append(ses.decode_step(t)[0])
        return got
    if kind == "serve":
        eng = _engine(c)
        ids = [eng.submit(p, n) for p, n in zip(s["prompts"], s["limit"])]
        eng.run_to_completion()
        out = np.full((len(ids), s["cap"]), -1, np.int64)
        for row, i in zip(out, ids):
            toks, _ = eng.poll(i, s["cap"])
            row[:toks.size] = toks
        eng.clear_finished()
        return out
    if kind == "attn_decode":
        rows, H, hd = c["rows"], c["heads"], c["head_dim"]
        scale = 1.0 / math.sqrt(hd)
        if c["append"]:
            ops.attn_decode_append_paged(s["qkv"], s["rope"], c["hi"], s["k"], s["v"], s["tables"], s["kv_lens"], s["out"], rows, H, hd, s["mb"], scale,
                                         DT[c["dtype"]], 0, s["nb"], s["scratch"])
            return s["out"], s["k"], s["v"]
        ops.attn_decode_paged(s["q"], s["k"], s["v"], s["tables"], s["kv_lens"], s["out"], rows, H, hd, s["mb"], scale, DT[c["dtype"]], 0, s["nb"],
                              s["scratch"])
        return s["out"]
    if kind == "gemm":
        ops.gemm_bf16(s["a"], s["wt"], s["c_out"], c["m"], c["n"], c["k"], EPI[c["epilogue"]], ldc=s["ldc"])
        return s["c_out"]
    if kind == "attn_prefill":
        ops.attn_prefill_paged(s["q"], s["k"], s["v"], s["tables"], s["mb"], s["cu"], s["slot"], s["out"], c["seqs"], s["max_len"], s["rows"], c["heads"],
                               c["head_dim"], 1.0 / math.sqrt(c["head_dim"]), ak.AK_BF16, s["nb"])
        return s["out"]
    ops.rmsnorm_rope_residual(s["x"], s["res"], s["w"], s["y"], s["pos"], c["rows"], c["size"], 1e-5, c["head_dim"], ak.AK_BF16)
    return (s["x"], s["y"]) if c["residual"] else s["y"]


# ---------------------------------------------------------------------------------------------- what a pass cannot do without
def _model_work(cfg, esz, plen, gen, steps, logits_rows):
    """A model's work on sequences with prompts `plen` that generate `gen` tokens in `steps` passes over the weights."""
    D, L, F, V = cfg.dim, cfg.num_layers, cfg.ffn_hidden, cfg.vocab_size
    layer = D * 3 * D + D * D + 2 * D * F
    plen, gen = np.asarray(plen, float), np.asarray(gen, float)
    fed = plen + np.maximum(gen - 1, 0)                     # tokens that go through the layers
    dec = np.maximum(gen - 1, 0)                            # of them one at a time, over a growing cache
    kv_read = dec * plen + dec * (dec + 1) / 2
    pairs = plen * (plen + 1) / 2 + kv_read
    nbytes = steps * (L * layer + D * V) * esz + L * 2 * D * esz * (kv_read.sum() + fed.sum()) + fed.sum() * D * esz + logits_rows * V * 4
    flops = 2.0 * L * layer * fed.sum() + 2.0 * D * V * gen.sum() + 4.0 * L * D * pairs.sum()
    return {"bytes": float(nbytes), "flops": float(flops)}


def work(case):
    c = case
    kind = c["kind"]
    if kind in ("chat", "score"):
        gen = c["new"] + (1 if kind == "score" else 0)
        return _model_work(MODELS[c["model"]](), ESZ[c["dtype"]], [c["prompt"]], [gen], gen, gen if kind == "score" else 0)
    if kind == "serve":
        plen, limit, until = _serve_limits(c)
        gen = limit - plen
        if c["eos"]:
            gen = np.minimum(gen, until)
        steps = max(int(gen.max()), -(-int(gen.sum()) // c["slots"]))
        return _model_work(MODELS[c["model"]](), 2, plen, gen, steps, 0)
    if kind == "attn_decode":
        lens = _lens(c, c["rows"]).astype(float)
        D, esz = c["heads"] * c["head_dim"], ESZ[c["dtype"]]
        extra = c["rows"] * D * (3 * 4 + 3 * esz) if c["append"] else c["rows"] * D * 2 * esz
        return {"bytes": lens.sum() * D * 2 * esz + extra + np.ceil(lens / 16).sum() * 4, "flops": 4.0 * D * lens.sum()}
    if kind == "gemm":
        m, n, k = c["m"], c["n"], c["k"]
        out = {"store_f32": 4, "add_f32": 8, "store_bf16": 2, "silu_bf16": 2}[c["epilogue"]]
        return {"bytes": 2.0 * (m * k + n * k) + float(out) * m * n, "flops": 2.0 * m * n * k}
    if kind == "attn_prefill":
        lens = _lens(c, c["seqs"]).astype(float)
        D = c["heads"] * c["head_dim"]
        return {"bytes": lens.sum() * D * 2 * 4, "flops": 4.0 * D * (lens * (lens + 1) / 2).sum()}
    n = c["rows"] * c["size"]
    return {"bytes": float(n * (4 + 2) + (n * 8 if c["residual"] else 0)), "flops": 6.0 * n}


def tolerance(case):
    kind = case["kind"]
    if kind in ("chat", "serve"):
        return {"rel": 0.0, "differ": 0.01}      # token ids
    if kind == "score":
        # 32-bit sums in another order, through 12 layers; bf16 roundings of every activation, through 12 layers
        return {"rel": 2e-5} if case["dtype"] == "f32" else {"rel": 2e-2}
    if kind == "attn_decode" and case["dtype"] == "f32":
        return {"rel": 1e-5}
    if kind == "gemm" and case["epilogue"].endswith("f32"):
        return {"rel": 1e-5}
    return {"rel": 1e-2}
