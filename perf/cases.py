"""What the engine's users have it do, as cases that can be timed and compared.

A case is one pass of a serving program over a loaded model: a few decode steps of a batch, a prompt, a
step that mixes both, or a whole call from prompts to tokens.  Models are those of ``bench.py``: LFM2 at
its three sizes, which is what the engine is for, in bfloat16 and on the true 32-bit path, and Vukavik's
eight layers, whose recurrences stand for the mixers that carry a state instead of a cache.  Weights and
token ids are random.  The mixtures of experts of the other architectures are left out: a router's choice
flips with the last bit of a bfloat16 activation, so their logits cannot be compared between two correct
programs.

``exact`` restates the two models in float64 with plain torch; positions times frequencies are the float32
products that the models define.
"""
import math
import random

import torch

from vapi_b200.config.model import resolve_architecture
from vapi_b200.engine.engine import Engine
from vapi_b200.engine.runner import ModelRunner
from vapi_b200.engine.scheduler import SchedulerConfig
from vapi_b200.engine.step import StepEntry
from vapi_b200.sampling.params import SamplingParams

PAGE = 64
#: decode steps in one pass: the last one reads what the others left in the caches and states
STEPS = 4


# ---- the cases ----------------------------------------------------------------------------------------

def listed():
    return [
        # one user's answer, deep in a long context: every weight is read for one token
        {"name": "decode-1.2b-1x4096", "kind": "decode", "model": "lfm2-1.2b", "dtype": "bfloat16",
         "requests": 1, "shortest": 4090, "longest": 4090},
        # the benchmark's configuration
        {"name": "decode-1.2b-8x4096", "kind": "decode", "model": "lfm2-1.2b", "dtype": "bfloat16",
         "requests": 8, "shortest": 4090, "longest": 4090},
        # a full server: 64 requests of lengths 128 to 2,048 on the largest size
        {"name": "decode-2.6b-64x128..2048", "kind": "decode", "model": "lfm2-2.6b", "dtype": "bfloat16",
         "requests": 64, "shortest": 128, "longest": 2048},
        # a few short chats, no power of two of them
        {"name": "decode-700m-19x33..700", "kind": "decode", "model": "lfm2-700m", "dtype": "bfloat16",
         "requests": 19, "shortest": 33, "longest": 700},
        # a question of a line: time to first token when nothing else runs
        {"name": "prefill-700m-57", "kind": "prefill", "model": "lfm2-700m", "dtype": "bfloat16",
         "requests": 1, "shortest": 57, "longest": 57, "portion": 2048},
        # the benchmark's prompt
        {"name": "prefill-1.2b-2048", "kind": "prefill", "model": "lfm2-1.2b", "dtype": "bfloat16",
         "requests": 1, "shortest": 2048, "longest": 2048, "portion": 2048},
        # a document, in the portions of the default configuration
        {"name": "prefill-2.6b-8000", "kind": "prefill", "model": "lfm2-2.6b", "dtype": "bfloat16",
         "requests": 1, "shortest": 8000, "longest": 8000, "portion": 2048},
        # continuous batching: a portion of one prompt beside the decoding requests
        {"name": "mixed-1.2b-31+777", "kind": "mixed", "model": "lfm2-1.2b", "dtype": "bfloat16",
         "requests": 31, "shortest": 100, "longest": 1900, "portion": 777},
        # the 32-bit path: decoding, a prompt, and a whole call from prompts to sampled tokens
        {"name": "decode-fp32-1.2b-8x1024", "kind": "decode", "model": "lfm2-1.2b", "dtype": "float32",
         "requests": 8, "shortest": 1000, "longest": 1024},
        {"name": "prefill-fp32-1.2b-1024", "kind": "prefill", "model": "lfm2-1.2b", "dtype": "float32",
         "requests": 1, "shortest": 1024, "longest": 1024, "portion": 2048},
        {"name": "generate-fp32-700m-5x12..90", "kind": "generate", "model": "lfm2-700m", "dtype": "float32",
         "requests": 5, "shortest": 12, "longest": 90, "new": 12},
        # the recurrences over a whole prompt
        {"name": "prefill-vukavik-2000", "kind": "prefill", "model": "vukavik-1.2b", "dtype": "bfloat16",
         "requests": 1, "shortest": 2000, "longest": 2000, "portion": 2048},
    ]


def draw(rng: random.Random):
    def log_between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["decode", "decode", "prefill", "prefill", "mixed", "decode-fp32", "prefill-fp32", "generate", "vukavik"])
    size = rng.choice(["700m", "1.2b", "2.6b"])
    if kind == "decode":
        n, longest = log_between(1, 64), log_between(24, 4090)
        if n * longest > 80000:
            longest = 80000 // n
        return {"kind": "decode", "model": "lfm2-" + size, "dtype": "bfloat16", "requests": n,
                "shortest": rng.randint(max(8, longest // 8), longest), "longest": longest}
    if kind == "prefill":
        n, longest = rng.choice([1, 1, 1, 2, 3, 5]), log_between(17, 8000)
        longest = min(longest, 8000 // n)
        return {"kind": "prefill", "model": "lfm2-" + size, "dtype": "bfloat16", "requests": n,
                "shortest": rng.randint(max(9, longest // 4), longest), "longest": longest, "portion": rng.choice([512, 2048, 4096])}
    if kind == "mixed":
        return {"kind": "mixed", "model": "lfm2-" + size, "dtype": "bfloat16", "requests": log_between(2, 60),
                "shortest": rng.randint(20, 300), "longest": rng.randint(300, 1900), "portion": log_between(40, 2000)}
    if kind == "decode-fp32":
        longest = log_between(24, 1024)
        return {"kind": "decode", "model": "lfm2-" + rng.choice(["700m", "1.2b"]), "dtype": "float32", "requests": log_between(1, 16),
                "shortest": rng.randint(max(8, longest // 8), longest), "longest": longest}
    if kind == "prefill-fp32":
        longest = log_between(17, 1024)
        return {"kind": "prefill", "model": "lfm2-" + rng.choice(["700m", "1.2b"]), "dtype": "float32", "requests": 1,
                "shortest": longest, "longest": longest, "portion": 2048}
    if kind == "generate":
        longest = rng.randint(20, 200)
        return {"kind": "generate", "model": "lfm2-700m", "dtype": "float32", "requests": rng.randint(1, 8),
                "shortest": rng.randint(8, longest), "longest": longest, "new": rng.randint(4, 16)}
    if rng.random() < 0.5:
        longest = log_between(40, 2000)
        return {"kind": "prefill", "model": "vukavik-1.2b", "dtype": "bfloat16", "requests": rng.choice([1, 1, 2]),
                "shortest": rng.randint(max(20, longest // 2), longest), "longest": longest, "portion": 2048}
    longest = log_between(40, 1000)
    return {"kind": "decode", "model": "vukavik-1.2b", "dtype": "bfloat16", "requests": log_between(1, 16),
            "shortest": rng.randint(longest // 2, longest), "longest": longest}


def lengths(case):
    """The requests' lengths: spread evenly from the shortest to the longest, long and short ones in turn."""
    n, lo, hi = case["requests"], case["shortest"], case["longest"]
    even = [hi if n == 1 else lo + (hi - lo) * i // (n - 1) for i in range(n)]
    return [even[i // 2] if i % 2 == 0 else even[n - 1 - i // 2] for i in range(n)]


# ---- models -------------------------------------------------------------------------------------------

SIZES = {"700m": (1536, 24, 10240, 16, (2, 5, 8, 10, 12, 14)),
         "1.2b": (2048, 32, 12288, 16, (2, 5, 8, 10, 12, 14)),
         "2.6b": (2048, 32, 10752, 30, (2, 6, 10, 14, 18, 21, 24, 27))}
VOCAB, KV_HEADS, HEAD, EPS, THETA, TAPS = 65536, 8, 64, 1e-5, 1000000.0, 3


def config(model):
    family, size = model.split("-", 1)
    hidden, heads, ff, layers, attention = SIZES[size]
    lfm2 = {"architectures": ["Lfm2ForCausalLM"], "model_type": "lfm2", "vocab_size": VOCAB, "hidden_size": hidden,
            "intermediate_size": ff, "block_auto_adjust_ff_dim": True, "block_ffn_dim_multiplier": 1.0, "block_multiple_of": 256,
            "num_hidden_layers": layers, "num_attention_heads": heads, "num_key_value_heads": KV_HEADS, "head_dim": HEAD,
            "conv_L_cache": TAPS, "conv_bias": False, "rope_theta": THETA, "norm_eps": EPS, "tie_word_embeddings": True,
            "max_position_embeddings": 128000,
            "layer_types": ["full_attention" if i in attention else "conv" for i in range(layers)]}
    if family == "lfm2":
        return lfm2
    mlp = {"kind": "dense", "ff": ff_width(ff)}
    att = {"type": "attention", "mlp": mlp, "mixer": {
        "heads": heads, "kv_heads": KV_HEADS, "dim": HEAD, "vdim": HEAD, "scale": 0.125, "mask": {"size": 8192},
        "rot": {"base": THETA, "dims": HEAD, "scaling": {"factor": 8.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": hidden // 128, "kv_heads": hidden // 128, "dim": 128, "vdim": 128, "conv": 4}}
    mamba = {"type": "mamba2", "mlp": mlp, "mixer": {"heads": 2 * hidden // 64, "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}}
    return {"architecture": "Vukavik", "vocab": VOCAB, "width": hidden, "residual_mult": 0.5, "logit_scale": 1.0,
            "norm": {"eps": EPS}, "layers": [delta, mamba, delta, att, delta, mamba, delta, att]}


MATRICES = ("matrix", "branch", "embedding")


def ff_width(ff):
    return -(-(2 * ff // 3) // 256) * 256


def shapes(cfg):
    """(name, shape, how it is drawn) of every tensor.  Matrices are in the model's type, vectors float32."""
    out = []
    if "layer_types" in cfg:
        H, nh, ff = cfg["hidden_size"], cfg["num_attention_heads"], ff_width(cfg["intermediate_size"])
        out.append(("model.embed_tokens.weight", (VOCAB, H), "embedding"))
        for i, kind in enumerate(cfg["layer_types"]):
            p = f"model.layers.{i}."
            out += [(p + "operator_norm.weight", (H,), "norm"), (p + "ffn_norm.weight", (H,), "norm"),
                    (p + "feed_forward.w1.weight", (ff, H), "matrix"), (p + "feed_forward.w3.weight", (ff, H), "matrix"),
                    (p + "feed_forward.w2.weight", (H, ff), "branch")]
            if kind == "conv":
                out += [(p + "conv.in_proj.weight", (3 * H, H), "matrix"), (p + "conv.conv.weight", (H, 1, TAPS), "taps"),
                        (p + "conv.out_proj.weight", (H, H), "branch")]
            else:
                a = p + "self_attn."
                out += [(a + "q_proj.weight", (nh * HEAD, H), "matrix"), (a + "k_proj.weight", (KV_HEADS * HEAD, H), "matrix"),
                        (a + "v_proj.weight", (KV_HEADS * HEAD, H), "matrix"), (a + "out_proj.weight", (H, nh * HEAD), "branch"),
                        (a + "q_layernorm.weight", (HEAD,), "norm"), (a + "k_layernorm.weight", (HEAD,), "norm")]
        return out + [("model.embedding_norm.weight", (H,), "norm")]
    H = cfg["width"]
    out.append(("embed", (VOCAB, H), "embedding"))
    for i, layer in enumerate(cfg["layers"]):
        p, m, ff = f"l{i}.", layer["mixer"], layer["mlp"]["ff"]
        out += [(p + "norm1", (H,), "norm"), (p + "norm2", (H,), "norm"), (p + "norm1b", (H,), "branch norm"), (p + "norm2b", (H,), "branch norm")]
        out += [(p + "mlp.gate", (ff, H), "matrix"), (p + "mlp.up", (ff, H), "matrix"), (p + "mlp.down", (H, ff), "matrix")]
        p += "mix."
        nh = m["heads"]
        if layer["type"] == "attention":
            out += [(p + "q", (nh * HEAD, H), "matrix"), (p + "k", (KV_HEADS * HEAD, H), "matrix"), (p + "v", (KV_HEADS * HEAD, H), "matrix"),
                    (p + "o", (H, nh * HEAD), "matrix"), (p + "g", (nh, H), "matrix"), (p + "sink", (nh,), "small"),
                    (p + "q.norm", (HEAD,), "norm"), (p + "k.norm", (HEAD,), "norm")]
        elif layer["type"] == "delta":
            qk, vv = m["kv_heads"] * m["dim"], nh * m["vdim"]
            out += [(p + "q", (qk, H), "matrix"), (p + "k", (qk, H), "matrix"), (p + "v", (vv, H), "matrix"),
                    (p + "q.conv", (qk, 4), "taps"), (p + "k.conv", (qk, 4), "taps"), (p + "v.conv", (vv, 4), "taps"),
                    (p + "a", (nh, H), "matrix"), (p + "b", (nh, H), "matrix"), (p + "A_log", (nh,), "A_log"), (p + "dt_bias", (nh,), "dt_bias"),
                    (p + "norm", (m["vdim"],), "norm"), (p + "g", (vv, H), "matrix"), (p + "o", (H, vv), "matrix")]
        else:
            inner, n2 = nh * m["vdim"], 2 * m["groups"] * m["state"]
            out += [(p + "in", (2 * inner + n2 + nh, H), "matrix"), (p + "conv", (inner + n2, 4), "taps"), (p + "conv.b", (inner + n2,), "small"),
                    (p + "dt_bias", (nh,), "dt_bias"), (p + "A_log", (nh,), "A_log"), (p + "D", (nh,), "norm"),
                    (p + "norm", (inner,), "norm"), (p + "o", (H, inner), "matrix")]
    return out + [("final.norm", (H,), "norm"), ("head", (VOCAB, H), "matrix")]


def weights(case, seed):
    """N(0, 0.02) as in the benchmark, but for what decides how a layer's rounding comes back in the logits: what writes
    into the stream is divided by the root of the number of sublayers (the usual initialisation of a deep stack), and the
    embedding is about as large as what all layers add to it, as in a trained model.  With everything at 0.02 each layer
    replaces the stream, two correct bfloat16 programs differ by 5 % of the logits, and nothing could be told from them.
    (Sampled tokens are float32's: there the small embedding stays, or every token would repeat its own.)"""
    cfg, dtype = config(case["model"]), torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    sublayers = 2 * len(cfg.get("layer_types") or cfg["layers"])
    embedding = 0.02 if case["kind"] == "generate" else 0.6
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(shape):
        return torch.randn(shape, generator=gen, device="cuda")

    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=gen, device="cuda") * (hi - lo) + lo

    out = {}
    for name, shape, how in shapes(cfg):
        if how in MATRICES:
            t = normal(shape).mul_({"matrix": 0.02, "branch": 0.02 * sublayers ** -0.5, "embedding": embedding}[how]).to(dtype)
        elif how == "norm":
            t = 1.0 + 0.1 * normal(shape)
        elif how == "branch norm":
            t = 0.3 + 0.03 * normal(shape)
        elif how == "taps":              # (what a depthwise convolution's default initialisation gives: +- 1/sqrt(taps))
            t = uniform(shape, -1.0, 1.0) * shape[-1] ** -0.5
        elif how == "A_log":             # (the recurrences' published initialisation: rates of 1 to 16 and steps of 0.001 to 0.1)
            t = uniform(shape, 1.0, 16.0).log()
        elif how == "dt_bias":
            t = uniform(shape, math.log(0.001), math.log(0.1)).exp().expm1().log()
        else:
            t = normal(shape).mul_(0.02)
        out[name] = t
    return out


def tokens_of(case, seed):
    """Per request: its prompt, and the tokens that the pass feeds behind it."""
    rng = torch.Generator().manual_seed(seed * 7919 + 1)
    more = {"decode": STEPS, "mixed": 1, "prefill": 0, "generate": 0}[case["kind"]]
    want = [n + more for n in lengths(case)]
    if case["kind"] == "mixed":          # the last request is the one whose prompt is under way
        want.append(case["longest"] // 2 + case["portion"])
    return [torch.randint(0, VOCAB, (n,), generator=rng).tolist() for n in want]


# ---- one pass -----------------------------------------------------------------------------------------

def fill(runner, request, tokens):
    """Computes a request's first positions, in portions."""
    assert runner.cache.reserve(request, len(tokens))
    for at in range(0, len(tokens), 4096):
        runner.step([StepEntry(request, tokens[at:at + 4096], [])])


def prepare(case, seed):
    cfg = config(case["model"])
    arch = resolve_architecture(cfg)
    tokens = tokens_of(case, seed)
    room = max(len(t) for t in tokens) + case.get("new", 0) + 1
    pages = sum(-(-(len(t) + case.get("new", 0) + 1) // PAGE) for t in tokens) + 2
    runner = ModelRunner(arch.plan(arch.parse(cfg)), weights(case, seed), dtype=case["dtype"], device="cuda", page_size=PAGE,
                         num_pages=pages, max_requests=len(tokens), max_batched_tokens=8192, max_context=room, validate=False)
    state = {"case": case, "runner": runner, "tokens": tokens}
    if case["kind"] == "generate":
        # greedy, at a temperature, and with the cuts of nucleus and top-k sampling
        kinds = [dict(temperature=0.0), dict(temperature=0.8), dict(temperature=0.7, top_k=50, top_p=0.95)]
        state["params"] = [SamplingParams(max_tokens=case["new"], seed=seed + i, ignore_eos=True, **kinds[i % 3]) for i in range(len(tokens))]
        state["engine"] = Engine(runner, SchedulerConfig(max_concurrent_seqs=len(tokens), max_batched_tokens=8192,
                                                         prefill_chunk_tokens=2048, max_context=room))
        state["round"] = 0
        run(state)                       # a server's decode graphs are captured before its first request
        return state
    # what every request has computed when the pass begins
    past = [len(t) for t in tokens]
    if case["kind"] == "decode":
        past = [n - STEPS for n in past]
    elif case["kind"] == "mixed":
        past = [n - 1 for n in past[:-1]] + [past[-1] - case["portion"]]
    else:
        past = [0 for _ in past]
    requests = [runner.cache.open(i) for i in range(len(tokens))]
    for request, toks, n in zip(requests, tokens, past):
        if n:
            fill(runner, request, toks[:n])
        assert runner.cache.reserve(request, len(toks))
    state.update(requests=requests, past=past, kept=[g.tensor.clone() for g in runner.cache.state] if any(past) else [])
    if case["kind"] == "decode":
        run(state)                       # (captures the batch's decode graph, as a server does when it starts)
    return state


def run(state):
    case, runner, tokens = state["case"], state["runner"], state["tokens"]
    if case["kind"] == "generate":
        engine, at = state["engine"], state["round"]
        state["round"] += 1
        for i, (prompt, params) in enumerate(zip(tokens, state["params"])):
            engine.admit((at, i), prompt, params)
        done = {f.request_id[1]: f.tokens for f in engine.run()}
        return {"tokens": torch.tensor([done[i] for i in range(len(tokens))])}
    # every pass starts from where the requests stood: positions set back, the rolling states as they were
    requests, cache = state["requests"], runner.cache
    rolling = [group.tensor[:len(requests)] for group in cache.state]
    for group, kept in zip(cache.state, state["kept"]):
        group.tensor.copy_(kept)
    for request, n in zip(requests, state["past"]):
        cache.commit(request, n)
    if case["kind"] == "decode":
        for s in range(STEPS):
            entries = [StepEntry(r, [t[n + s]], [0]) for r, t, n in zip(requests, tokens, state["past"])]
            logits = runner.step_decode_graph(entries)
            if logits is None:
                logits = runner.step(entries)
        return {"logits": logits, "rolling": rolling}
    if case["kind"] == "mixed":
        entries = [StepEntry(r, t[n:], [len(t) - n - 1]) for r, t, n in zip(requests, tokens, state["past"])]
        return {"logits": runner.step(entries), "rolling": rolling}
    # prompts: whole ones share a step as far as they fit, longer ones come in portions
    out, step, room = [], [], case["portion"]
    for request, toks in zip(requests, tokens):
        at = 0
        while at < len(toks):
            take = min(room, len(toks) - at)
            step.append(StepEntry(request, toks[at:at + take], [take - 1] if at + take == len(toks) else []))
            at, room = at + take, room - take
            if room == 0:
                out.append(runner.step(step))
                step, room = [], case["portion"]
    if step:
        out.append(runner.step(step))
    return {"logits": [x for x in out if x is not None], "rolling": rolling}


# ---- what a pass cannot do without ----------------------------------------------------------------------

def work(case):
    cfg = config(case["model"])
    size = 4 if case["dtype"] == "float32" else 2
    vectors = sum(math.prod(s) for _, s, how in shapes(cfg) if how not in MATRICES)
    matrices = {n: math.prod(s) for n, s, how in shapes(cfg) if how in MATRICES}
    head = matrices.pop("head", None)
    table = matrices.pop("embed", None) or matrices.pop("model.embed_tokens.weight")
    head = head or table
    body = sum(matrices.values())
    width = cfg.get("hidden_size") or cfg["width"]
    kinds = cfg.get("layer_types") or [layer["type"] for layer in cfg["layers"]]
    attention = sum(k in ("attention", "full_attention") for k in kinds)
    heads = SIZES[case["model"].split("-", 1)[1]][1]
    kv = attention * 2 * KV_HEADS * HEAD * size                        # bytes of cache per position
    state = {"conv": (TAPS - 1) * width * size, "delta": 4 * (width * 128 + 9 * width), "mamba2": 4 * (2 * width * 128 + 3 * (2 * width + 256))}
    rolling = sum(state.get(k, 0) for k in kinds)                      # bytes of rolling state per request
    scan = sum({"delta": 8 * width * 128, "mamba2": 6 * 2 * width * 128}.get(k, 0) for k in kinds)   # flops of the recurrences per token

    def step(entries, rows):
        """``entries``: (positions before, tokens) of each request in one step, ``rows``: how many rows of logits."""
        n = sum(q for _, q in entries)
        pairs = sum(q * p + q * (q + 1) // 2 for p, q in entries)
        b = body * size + vectors * 4 + (head * size if rows else 0) + n * width * size + rows * VOCAB * 4
        b += sum((p + q) * kv for p, q in entries) + sum(rolling * (2 if p else 1) for p, _ in entries)
        return b, 2.0 * body * n + 2.0 * head * rows + attention * 4.0 * heads * HEAD * pairs + scan * n

    ls = lengths(case)
    if case["kind"] == "decode":
        parts = [step([(n + s, 1) for n in ls], len(ls)) for s in range(STEPS)]
    elif case["kind"] == "mixed":
        parts = [step([(n, 1) for n in ls] + [(case["longest"] // 2, case["portion"])], len(ls) + 1)]
    elif case["kind"] == "generate":
        parts = [step([(0, n) for n in ls], len(ls))] + [step([(n + s, 1) for n in ls], len(ls)) for s in range(case["new"] - 1)]
    else:
        parts, entries, rows, room = [], [], 0, case["portion"]
        for n in ls:
            at = 0
            while at < n:
                take = min(room, n - at)
                entries.append((at, take))
                at, room, rows = at + take, room - take, rows + (at + take == n)
                if room == 0:
                    parts.append(step(entries, rows))
                    entries, rows, room = [], 0, case["portion"]
        if entries:
            parts.append(step(entries, rows))
    return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}


def tolerance(case):
    if case["kind"] == "generate":       # (tokens; in float32 the choices do not come near a tie)
        return "exact"
    # About four times what the outputs are off by in float64: bfloat16 up to 5.9e-3 (the largest value by 2.6e-2 of the
    # root mean square), float32 up to 2.3e-6 (9e-6).
    return {"rel": 1e-5, "max": 4e-5} if case["dtype"] == "float32" else {"rel": 0.024, "max": 0.1}


# ---- the models in float64 --------------------------------------------------------------------------------

def rms(x, eps=EPS):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def silu(z):
    return z * torch.sigmoid(z)


def causal_conv(x, taps):
    """x [T, C], taps [C, L]: the last column belongs to the current token; zeros before the start."""
    L = taps.shape[1]
    x = torch.cat([x.new_zeros(L - 1, x.shape[1]), x])
    return sum(x[j:x.shape[0] - L + 1 + j] * taps[:, j] for j in range(L))


def angles(T, freqs):
    return (torch.arange(T, device="cuda", dtype=torch.float32)[:, None] * freqs.to("cuda")[None, :]).double()


def attend(q, k, v, scale, sink=None):
    """Causal attention of q [T, heads, d] over k, v [T, kv heads, d], one kv head at a time."""
    T, nh, d = q.shape
    rep, out = nh // k.shape[1], torch.empty_like(q)
    hidden = torch.ones(T, T, dtype=torch.bool, device=q.device).triu(1)
    for h in range(nh):
        s = (q[:, h] @ k[:, h // rep].T).mul_(scale).masked_fill_(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T, 1)], 1)
        p = torch.softmax(s, -1)
        out[:, h] = p[:, :T] @ v[:, h // rep]
    return out.reshape(T, nh * d)


def lfm2_sequence(cfg, w, ids):
    """The last position's logits of one sequence, and the rows that its convolutions keep."""
    def m(name):
        return w[name].double()
    T, nh = len(ids), cfg["num_attention_heads"]
    x = w["model.embed_tokens.weight"][torch.tensor(ids, device="cuda")].double()
    freqs = 1.0 / torch.pow(torch.tensor(THETA), torch.arange(0, HEAD, 2, dtype=torch.float32) / HEAD)
    a = angles(T, freqs)
    cos, sin = a.cos()[:, None, :], a.sin()[:, None, :]

    def rope(z):
        z1, z2 = z[..., :HEAD // 2], z[..., HEAD // 2:]
        return torch.cat([z1 * cos - z2 * sin, z2 * cos + z1 * sin], -1)

    kept = []
    for i, kind in enumerate(cfg["layer_types"]):
        p = f"model.layers.{i}."
        h = rms(x) * m(p + "operator_norm.weight")
        if kind == "conv":
            b, c, z = (h @ m(p + "conv.in_proj.weight").T).chunk(3, -1)
            kept.append((b * z)[1 - TAPS:])
            x = x + (c * causal_conv(b * z, m(p + "conv.conv.weight")[:, 0])) @ m(p + "conv.out_proj.weight").T
        else:
            s = p + "self_attn."
            q = rope(rms((h @ m(s + "q_proj.weight").T).view(T, nh, HEAD)) * m(s + "q_layernorm.weight"))
            k = rope(rms((h @ m(s + "k_proj.weight").T).view(T, KV_HEADS, HEAD)) * m(s + "k_layernorm.weight"))
            v = (h @ m(s + "v_proj.weight").T).view(T, KV_HEADS, HEAD)
            x = x + attend(q, k, v, HEAD ** -0.5) @ m(s + "out_proj.weight").T
        h = rms(x) * m(p + "ffn_norm.weight")
        x = x + (silu(h @ m(p + "feed_forward.w1.weight").T) * (h @ m(p + "feed_forward.w3.weight").T)) @ m(p + "feed_forward.w2.weight").T
    return m("model.embed_tokens.weight") @ (rms(x[-1]) * m("model.embedding_norm.weight")), torch.stack(kept)


def yarn(rot):
    dims, base, sc = rot["dims"], rot["base"], rot["scaling"]

    def pair_of(turns):
        return dims * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(base))

    lo, hi = max(math.floor(pair_of(sc["fast"])), 0), min(math.ceil(pair_of(sc["slow"])), dims - 1)
    out = []
    for i in range(dims // 2):
        f, ramp = base ** (-2.0 * i / dims), min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0)
        out.append(f / sc["factor"] * ramp + f * (1.0 - ramp))
    return torch.tensor(out, dtype=torch.float64).float(), 0.1 * math.log(sc["factor"]) + 1.0


def delta_rule(q, k, v, beta, decay):
    """S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q, head by head; [T, heads, d]."""
    S, out = q.new_zeros(q.shape[1], q.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(q.shape[0]):
        S = S * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - torch.einsum("hij,hi->hj", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hij,hi->hj", S, q[t])
    return out


def state_space(x, B, C, dt, rate):
    """sum over s <= t of exp(-rate * (dt_{s+1} + ... + dt_t)) (C_t . B_s) dt_s x_s; x [T, heads, p], B, C [T, N]."""
    total, pairs, out = torch.cumsum(dt * rate, 0), C @ B.T, torch.empty_like(x)
    later = torch.ones_like(pairs, dtype=torch.bool).triu(1)
    for h in range(x.shape[1]):
        g = (total[None, :, h] - total[:, None, h]).masked_fill_(later, -math.inf).exp_()
        out[:, h] = (pairs * g) @ (dt[:, h, None] * x[:, h])
    return out


def vukavik_sequence(cfg, w, ids):
    def m(name):
        return w[name].double()
    T, x = len(ids), w["embed"][torch.tensor(ids, device="cuda")].double()
    for i, layer in enumerate(cfg["layers"]):
        p, e = f"l{i}.mix.", layer["mixer"]
        h, nh = rms(x) * m(f"l{i}.norm1"), e["heads"]
        if layer["type"] == "attention":
            freqs, mult = yarn(e["rot"])
            a = angles(T, freqs)
            cos, sin = a.cos()[:, None, :] * mult, a.sin()[:, None, :] * mult

            def turn(z):
                u, v = z[..., 0::2], z[..., 1::2]
                return torch.stack([u * cos - v * sin, v * cos + u * sin], -1).flatten(-2)

            q = turn(rms((h @ m(p + "q").T).view(T, nh, HEAD)) * m(p + "q.norm"))
            k = turn(rms((h @ m(p + "k").T).view(T, KV_HEADS, HEAD)) * m(p + "k.norm"))
            v = (h @ m(p + "v").T).view(T, KV_HEADS, HEAD)
            y = attend(q, k, v, e["scale"], m(p + "sink")).view(T, nh, HEAD) * torch.sigmoid(h @ m(p + "g").T)[:, :, None]
            y = y.reshape(T, -1) @ m(p + "o").T
        elif layer["type"] == "delta":
            d, dv = e["dim"], e["vdim"]
            q, k, v = (silu(causal_conv(h @ m(p + n).T, m(p + n + ".conv"))) for n in "qkv")
            q, k, v = q.view(T, nh, d), k.view(T, nh, d), v.view(T, nh, dv)
            q = q * torch.rsqrt(q.square().sum(-1, keepdim=True) + 1e-6) * d ** -0.5
            k = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
            decay = torch.exp(-m(p + "A_log").exp() * torch.nn.functional.softplus(h @ m(p + "a").T + m(p + "dt_bias")))
            o = rms(delta_rule(q, k, v, torch.sigmoid(h @ m(p + "b").T), decay)) * m(p + "norm")
            y = (o.reshape(T, nh * dv) * silu(h @ m(p + "g").T)) @ m(p + "o").T
        else:
            P, N = e["vdim"], e["state"]
            inner = nh * P
            z, xbc, dt = (h @ m(p + "in").T).split([inner, inner + 2 * N, nh], -1)
            xbc = silu(causal_conv(xbc, m(p + "conv")) + m(p + "conv.b"))
            u, B, C = xbc[:, :inner].view(T, nh, P), xbc[:, inner:inner + N], xbc[:, inner + N:]
            dt = torch.nn.functional.softplus(dt + m(p + "dt_bias"))
            o = state_space(u, B, C, dt, m(p + "A_log").exp()) + m(p + "D")[:, None] * u
            y = (rms(o.reshape(T, inner) * silu(z)) * m(p + "norm")) @ m(p + "o").T
        x = x + cfg["residual_mult"] * (rms(y) * m(f"l{i}.norm1b"))
        h, p = rms(x) * m(f"l{i}.norm2"), f"l{i}.mlp."
        y = (silu(h @ m(p + "gate").T) * (h @ m(p + "up").T)) @ m(p + "down").T
        x = x + cfg["residual_mult"] * (rms(y) * m(f"l{i}.norm2b"))
    return m("head") @ (rms(x[-1]) * m("final.norm")) * cfg["logit_scale"], None


def exact(case, seed):
    if case["kind"] == "generate":       # sampled tokens come from the engine's own random numbers
        return None
    cfg = config(case["model"])
    w = weights(case, seed)
    sequence = lfm2_sequence if "layer_types" in cfg else vukavik_sequence
    with torch.no_grad():
        rows, kept = zip(*(sequence(cfg, w, ids) for ids in tokens_of(case, seed)))
    # (how the recurrences lay their matrices out in a slot is theirs to say)
    rolling = None if kept[0] is None else [torch.stack(kept)]
    if case["kind"] != "prefill":
        return {"logits": torch.stack(rows), "rolling": rolling}
    # laid out as the steps are: a step's rows are those of the prompts that end in it
    out, room, ends = [], case["portion"], []
    for row, n in zip(rows, lengths(case)):
        while n > room:
            n, room = n - room, case["portion"]
            if ends:
                out.append(torch.stack(ends))
                ends = []
        room -= n
        ends.append(row)
        if room == 0:
            out.append(torch.stack(ends))
            ends, room = [], case["portion"]
    if ends:
        out.append(torch.stack(ends))
    return {"logits": out, "rolling": rolling}
