"""What this framework's users have it do, as cases that can be timed and compared.

Two kinds of work:

* `llama`: whole calls of `Engine.step` on a stack of decoder layers with the widths of the two configurations that the
  repository's benchmark quotes (2B-class and 0.5B-class): decoding a batch behind its prompts, filling prompts, filling a
  portion late in a prompt, in bfloat16 (serving) and in true 32-bit (verification).  They return the wanted logits and
  the first and the last layer's pages.
* one layer's mixer or feed-forward, through the part's own `forward` inside a step that has begun, at the widths of the
  benchmark's other architectures: attention through latents (three of the seven architectures), retention, gated linear
  attention, the selective scan, and a mixture of experts.  They return the part's output rows and the request's state
  after them (the pages' latents and rotated parts, or the recurrent state).

Sizes, head counts, ranks, windows and decays are those of `bench.py`; weights are N(0, 0.02) as the repository's random
models have them, inputs of a layer are normed rows, N(0, 1)."""
import math

import torch

F64 = torch.float64
DEVICE = "cuda:0"
PAGE = 16
STEP_TOKENS = 2048                       # most tokens of one step while a context is filled

LLAMA = {
    "2b": dict(hidden_size=2048, intermediate_size=6144, num_attention_heads=16, num_key_value_heads=2, head_dim=128),
    "0.5b": dict(hidden_size=1024, intermediate_size=4096, num_attention_heads=16, num_key_value_heads=2, head_dim=64),
}
WIDTHS = {
    "2b": dict(width=2048, heads=16, dim=128, rot_dim=64, kv_rank=512, q_rank=1024, inner=4096, state=16, dt_rank=128,
               expert_ff=2048, shared_ff=2048),
    "0.5b": dict(width=1024, heads=16, dim=64, rot_dim=32, kv_rank=256, q_rank=512, inner=2048, state=16, dt_rank=64,
                 expert_ff=1024, shared_ff=2048),
}


# ---- the cases ----

def listed():
    return [
        # one conversation: the smallest call, where a step's launches and hand-overs are everything
        llama("decode_1", "2b", "bfloat16", "decode", requests=1, context=2048, layers=8),
        # the benchmark's headline point: eight conversations behind 2,048-token prompts
        llama("decode_8", "2b", "bfloat16", "decode", requests=8, context=2048, layers=8),
        # a full batch: most of what is read is cache
        llama("decode_64", "2b", "bfloat16", "decode", requests=64, context=2048, layers=8),
        # one whole prompt of the benchmark's length
        llama("prefill_2048", "2b", "bfloat16", "prefill", requests=1, tokens=2048, layers=8),
        # the 32-bit path, as a reference run or a trace replay uses it: three ragged prompts
        llama("prefill_f32_600", "0.5b", "float32", "prefill", requests=3, tokens=600, layers=2),
        # attention through latents over a whole prompt, queries straight from the input, gated output, all keys
        latent("latent_prefill_2048", "2b", "gated", "prefill", requests=1, tokens=2048),
        # the same mechanism with a query latent and a window, two portions of unequal length late in their prompts
        latent("latent_portions_1111", "2b", "windowed", "prefill", requests=2, tokens=1111, context=1500),
        # and its decoding, thirty-two conversations
        latent("latent_decode_32", "2b", "gated", "decode", requests=32, context=2048),
        # a linear recurrence with a fixed decay a head over a whole prompt
        recurrence("retention_2048", "retention", "2b", requests=1, tokens=2048),
        # a linear recurrence with a decay per token and channel, three ragged prompts, smaller widths
        recurrence("gla_1500", "gla", "0.5b", requests=3, tokens=1500),
        # a selective scan over a whole prompt
        recurrence("scan_2048", "scan", "2b", requests=1, tokens=2048),
        # a mixture of eight experts, two chosen and one shared, a batch of ordinary size
        {"name": "experts_512", "kind": "experts", "size": "2b", "dtype": "bfloat16", "tokens": 512},
    ]


def llama(name, size, dtype, phase, requests, layers, tokens=0, context=0):
    case = {"kind": "llama", "size": size, "dtype": dtype, "phase": phase, "requests": requests, "layers": layers,
            "tokens": requests if phase == "decode" else tokens, "context": context}
    return {"name": name, **case} if name else case


def latent(name, size, form, phase, requests, tokens=0, context=0):
    case = {"kind": "latent", "size": size, "dtype": "bfloat16", "form": form, "phase": phase, "requests": requests,
            "tokens": requests if phase == "decode" else tokens, "context": context}
    return {"name": name, **case} if name else case


def recurrence(name, kind, size, requests, tokens):
    case = {"kind": kind, "size": size, "dtype": "bfloat16", "requests": requests, "tokens": tokens}
    return {"name": name, **case} if name else case


def spread(rng, low, high):
    """A whole number between `low` and `high`, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["llama", "llama", "llama", "llama", "latent", "latent", "latent", "retention", "gla", "scan", "experts"])
    size = rng.choice(["2b", "0.5b"])
    if kind == "llama":
        if rng.random() < 0.25:
            return llama(None, "0.5b", "float32", "prefill", rng.randint(1, 3), rng.randint(1, 2), tokens=spread(rng, 48, 600))
        if rng.random() < 0.5:
            return llama(None, size, "bfloat16", "decode", spread(rng, 1, 64), rng.randint(4, 8), context=spread(rng, 100, 2048))
        context = 0 if rng.random() < 0.6 else spread(rng, 100, 2048)
        return llama(None, size, "bfloat16", "prefill", rng.randint(1, 4), rng.randint(4, 8), tokens=spread(rng, 64, 1600),
                     context=context)
    if kind == "latent":
        form = rng.choice(["gated", "windowed"])
        if rng.random() < 0.35:
            return latent(None, size, form, "decode", spread(rng, 1, 32), context=spread(rng, 200, 2048))
        context = 0 if rng.random() < 0.5 else spread(rng, 100, 2048)
        return latent(None, size, form, "prefill", rng.randint(1, 4), tokens=spread(rng, 128, 2048), context=context)
    if kind == "experts":
        return {"kind": kind, "size": size, "dtype": "bfloat16", "tokens": spread(rng, 1, 2048)}
    return recurrence(None, kind, size, rng.randint(1, 4), spread(rng, 128, 2048))


def portions(case):
    """Tokens that each request brings: all alike when there is one a request, otherwise unequal (2 : 3 : 4 : ...)."""
    requests, tokens = case["requests"], case["tokens"]
    if case.get("phase") == "decode":
        return [1] * requests
    weights = [2 + i for i in range(requests)]
    out = [tokens * w // sum(weights) for w in weights]
    out[-1] += tokens - sum(out)
    return out


def generator(seed, stream):
    return torch.Generator(device=DEVICE).manual_seed(seed * 1000 + stream)


def normal(g, *shape, std=0.02, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=g, device=DEVICE, dtype=torch.float32) * std).to(dtype)


# ---- whole calls: the Llama decoder ----

def llama_config(case):
    return dict(LLAMA[case["size"]], architectures=["LlamaForCausalLM"], model_type="llama", num_hidden_layers=case["layers"],
                vocab_size=73448, rope_theta=10000.0, rms_norm_eps=1e-5, tie_word_embeddings=True, scale_emb=12,
                scale_depth=1.4, dim_model_base=256, max_position_embeddings=32768, initializer_range=0.02, hidden_act="silu",
                torch_dtype="bfloat16")


def llama_weights(case, seed):
    c, g = llama_config(case), generator(seed, 1)
    h, ff, nq, nkv, d = (c[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
    w = {"model.embed_tokens.weight": normal(g, c["vocab_size"], h), "model.norm.weight": 1 + normal(g, h, std=0.1)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for name, shape in [("self_attn.q_proj", (nq * d, h)), ("self_attn.k_proj", (nkv * d, h)), ("self_attn.v_proj", (nkv * d, h)),
                            ("self_attn.o_proj", (h, nq * d)), ("mlp.gate_proj", (ff, h)), ("mlp.up_proj", (ff, h)),
                            ("mlp.down_proj", (h, ff))]:
            w[p + name + ".weight"] = normal(g, *shape)
        w[p + "input_layernorm.weight"] = 1 + normal(g, h, std=0.1)
        w[p + "post_attention_layernorm.weight"] = 1 + normal(g, h, std=0.1)
    return w


def llama_tokens(case, seed):
    g = generator(seed, 2)
    return [torch.randint(0, 73448, (case["context"] + count,), generator=g, device=DEVICE).tolist() for count in portions(case)]


def prepare_llama(case, seed):
    from lia_rs_b200 import LlamaConfig
    from lia_rs_b200.engine import Engine, StepEntry
    counts, context = portions(case), case["context"]
    pages = sum((context + count + PAGE - 1) // PAGE for count in counts)
    engine = Engine.from_tensors(LlamaConfig.from_dict(llama_config(case)), llama_weights(case, seed), dtype=case["dtype"],
                                 page_size=PAGE, max_tokens=pages * PAGE, max_seqs=len(counts),
                                 max_batch_tokens=max(STEP_TOKENS, case["tokens"]), max_context=4096)
    entries = []
    for tokens, count in zip(llama_tokens(case, seed), counts):
        slot = engine.admit()
        assert engine.reserve(slot, 0, context + count)
        for at in range(0, context, STEP_TOKENS):
            engine.step([StepEntry(slot, tokens[at:min(at + STEP_TOKENS, context)], at, [])])
        entries.append(StepEntry(slot, tokens[context:], context, [count - 1]))
    engine.synchronize()
    views = [engine.cache.kv_view(layer, True) for layer in sorted({0, case["layers"] - 1})]
    return {"kind": "llama", "engine": engine, "entries": entries, "kept": [pages for v in views for pages in (v.k_pages, v.v_pages)]}


def exact_llama(case, seed):
    c, w = llama_config(case), llama_weights(case, seed)
    nq, nkv, d, eps = c["num_attention_heads"], c["num_key_value_heads"], c["head_dim"], c["rms_norm_eps"]
    scale = c["scale_depth"] / math.sqrt(case["layers"])
    f64 = lambda name: w[name].to(F64)
    rows = [f64("model.embed_tokens.weight")[torch.tensor(t, device=DEVICE)] * c["scale_emb"] for t in llama_tokens(case, seed)]
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        m = {n: f64(p + n + ".weight") for n in ("self_attn.q_proj", "self_attn.k_proj", "self_attn.v_proj", "self_attn.o_proj",
                                                 "mlp.gate_proj", "mlp.up_proj", "mlp.down_proj", "input_layernorm",
                                                 "post_attention_layernorm")}
        for r, h in enumerate(rows):
            n = h.shape[0]
            x = rms(h, eps) * m["input_layernorm"]
            freq = c["rope_theta"] ** (-2.0 * torch.arange(d // 2, device=DEVICE, dtype=F64) / d)
            q = rotate_halves((x @ m["self_attn.q_proj"].T).view(n, nq, d), freq)
            k = rotate_halves((x @ m["self_attn.k_proj"].T).view(n, nkv, d), freq)
            v = (x @ m["self_attn.v_proj"].T).view(n, nkv, d)
            o = torch.empty_like(q)
            for head in range(nq):
                o[:, head] = attend(q[:, head], k[:, head * nkv // nq], v[:, head * nkv // nq], d ** -0.5, None, 0)
            h = h + scale * (o.reshape(n, nq * d) @ m["self_attn.o_proj"].T)
            x = rms(h, eps) * m["post_attention_layernorm"]
            gate = x @ m["mlp.gate_proj"].T
            rows[r] = h + scale * ((x @ m["mlp.up_proj"].T) * gate * torch.sigmoid(gate) @ m["mlp.down_proj"].T)
    last = torch.stack([h[-1] for h in rows])
    last = rms(last, eps) * f64("model.norm.weight") * (c["dim_model_base"] / c["hidden_size"])
    return {"logits": last @ f64("model.embed_tokens.weight").T, "kept": [None] * (2 * len({0, case["layers"] - 1}))}


def rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def rotate_halves(x, freq, start=0):
    """x [T, heads, d]: element i with element i + d/2, by position * freq[i]."""
    angle = torch.arange(start, start + x.shape[0], device=DEVICE, dtype=F64)[:, None, None] * freq
    u, v = x.chunk(2, dim=-1)
    return torch.cat([u * torch.cos(angle) - v * torch.sin(angle), v * torch.cos(angle) + u * torch.sin(angle)], dim=-1)


def rotate_pairs(x, freq, start=0):
    """x [T, heads, d]: element 2i with element 2i + 1, by position * freq[i]."""
    angle = torch.arange(start, start + x.shape[0], device=DEVICE, dtype=F64)[:, None, None] * freq
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * torch.cos(angle) - v * torch.sin(angle), v * torch.cos(angle) + u * torch.sin(angle)], dim=-1).flatten(-2)


def attend(q, k, v, scale, window, start):
    """Causal softmax attention of one head: query i is at position start + i, key j at position j."""
    at = torch.arange(q.shape[0], device=DEVICE)[:, None] + start
    j = torch.arange(k.shape[0], device=DEVICE)[None, :]
    seen = j <= at
    if window:
        seen &= at - j < window
    return torch.softmax((q @ k.T * scale).masked_fill(~seen, -math.inf), dim=-1) @ v


# ---- one part inside a step that has begun ----

def part_spec(case):
    """(registry's kind, parameters, tensors) of the case's part; the tensors from a seed are made by `part_weights`."""
    s = WIDTHS[case["size"]]
    if case["kind"] == "latent":
        params = dict(hidden=s["width"], heads=s["heads"], head_dim=s["dim"], rot_dim=s["rot_dim"], v_head_dim=s["dim"],
                      kv_rank=s["kv_rank"], scale=(s["dim"] + s["rot_dim"]) ** -0.5, norm_eps=1e-5,
                      rot={"base": 10000.0, "dims": s["rot_dim"]})
        more = (dict(q_rank=None, gate="sigmoid", rot_pairs=True) if case["form"] == "gated" else
                dict(q_rank=s["q_rank"], window=1024))
        return "latent_attention", {**params, **more}
    if case["kind"] == "retention":
        return "retention", dict(hidden=s["width"], heads=s["heads"], head_dim=s["dim"], v_head_dim=s["dim"], norm_eps=1e-5,
                                 decay=[1.0 - 2.0 ** (-5 - 0.25 * h) for h in range(s["heads"])],
                                 rot={"base": 10000.0, "dims": s["dim"]})
    if case["kind"] == "gla":
        return "gated_linear_attention", dict(hidden=s["width"], heads=s["heads"], head_dim=s["dim"] // 2, v_head_dim=s["dim"],
                                              tau=16.0, decay_rank=16, norm_eps=1e-5)
    if case["kind"] == "scan":
        return "selective_scan", dict(hidden=s["width"], inner=s["inner"], state=s["state"], dt_rank=s["dt_rank"], taps=4)
    return "expert_mixture", dict(hidden=s["width"], experts=8, top=2, intermediate=s["expert_ff"],
                                  shared={"intermediate": s["shared_ff"]})


def part_weights(case, seed, specs):
    """Tensors by name for `specs` ([(name, shape)]): matrices N(0, 0.02), norms near one, and the few that a trained layer
    has elsewhere (a scan's decays and step sizes, a gated recurrence's bias)."""
    g = generator(seed, 1)
    out = {}
    for name, shape in sorted(specs):
        kind = name.split(".", 1)[1]
        if kind.endswith("norm"):
            out[name] = 1 + normal(g, *shape, std=0.1)
        elif kind == "A_log":
            out[name] = torch.log(torch.arange(1, shape[1] + 1, device=DEVICE, dtype=torch.float32)).repeat(shape[0], 1)
        elif kind == "dt.b":                          # softplus of it between 0.001 and 0.1
            dt = torch.exp(torch.rand(shape, generator=g, device=DEVICE) * math.log(100.0) + math.log(0.001))
            out[name] = torch.log(torch.expm1(dt))
        elif kind == "a2.b":                          # decays sigmoid(0..4)^(1/16)
            out[name] = torch.rand(shape, generator=g, device=DEVICE) * 4
        elif kind == "D":
            out[name] = torch.ones(shape, device=DEVICE)
        elif kind == "conv":
            out[name] = normal(g, *shape, std=0.3)
        else:
            out[name] = normal(g, *shape)
    return out


def part_specs(case):
    """The names and shapes of the part's tensors, as its architecture's checkpoints have them."""
    kind, p = part_spec(case)
    h = p["hidden"]
    if kind == "latent_attention":
        H, d, dr, dv, rank = p["heads"], p["head_dim"], p["rot_dim"], p["v_head_dim"], p["kv_rank"]
        out = {"dkv": (rank + dr, h), "dkv.norm": (rank,), "uk": (H * d, rank), "uv": (H * dv, rank), "o": (h, H * dv)}
        out.update({"dq": (p["q_rank"], h), "dq.norm": (p["q_rank"],), "uq": (H * (d + dr), p["q_rank"])} if p["q_rank"] else
                   {"q": (H * (d + dr), h)})
        if p.get("gate"):
            out["g"] = (H * dv, h)
    elif kind in ("retention", "gated_linear_attention"):
        H, d, dv = p["heads"], p["head_dim"], p["v_head_dim"]
        out = {"q": (H * d, h), "k": (H * d, h), "v": (H * dv, h), "g": (H * dv, h), "o": (h, H * dv)}
        if kind == "gated_linear_attention":
            out.update({"norm": (dv,), "a1": (p["decay_rank"], h), "a2": (H * d, p["decay_rank"]), "a2.b": (H * d,)})
    elif kind == "selective_scan":
        inner, n, rank = p["inner"], p["state"], p["dt_rank"]
        out = {"in": (2 * inner, h), "conv": (inner, p["taps"]), "conv.b": (inner,), "x": (rank + 2 * n, inner), "dt": (inner, rank),
               "dt.b": (inner,), "A_log": (inner, n), "D": (inner,), "o": (h, inner)}
    else:
        ff, ffs = p["intermediate"], p["shared"]["intermediate"]
        out = {"router": (p["experts"], h), "shared.gate": (ffs, h), "shared.up": (ffs, h), "shared.down": (h, ffs), "shared.sg": (1, h)}
        for e in range(p["experts"]):
            out.update({f"e{e}.gate": (ff, h), f"e{e}.up": (ff, h), f"e{e}.down": (h, ff)})
    return [("L." + name, shape) for name, shape in out.items()]


def part_rows(case, seed):
    """The layer's normed input rows of every request, from its first position to its last: [[context + count, hidden]]."""
    g, width = generator(seed, 2), WIDTHS[case["size"]]["width"]
    if case["kind"] == "experts":
        return [normal(g, case["tokens"], width, std=1.0)]
    return [normal(g, case.get("context", 0) + count, width, std=1.0) for count in portions(case)]


def prepare_part(case, seed):
    from lia_rs_b200.cache import CacheManager
    from lia_rs_b200.engine import StepEntry, StepRuntime
    from lia_rs_b200.parts import FEED_FORWARDS, MIXERS, Runtime
    kind, params = part_spec(case)
    feed_forward = kind in FEED_FORWARDS
    cls = (FEED_FORWARDS if feed_forward else MIXERS)[kind]
    dtype = getattr(torch, case["dtype"])
    cache_request = None if feed_forward else cls.cache_request(params)
    state_request = None if feed_forward else cls.state_request(params)
    counts = [case["tokens"]] if feed_forward else portions(case)
    context = case.get("context", 0)
    longest = context + max(counts)
    pages = sum((context + count + PAGE - 1) // PAGE for count in counts)
    cache = CacheManager({0: cache_request} if cache_request else {}, {0: state_request} if state_request else {}, pages, PAGE,
                         len(counts), longest, dtype, DEVICE)
    runtime = StepRuntime(cache, 1000, max(STEP_TOKENS, case["tokens"] + 8), DEVICE)
    part = cls(params, part_weights(case, seed, part_specs(case)), "L.", Runtime(DEVICE, dtype))
    rows = part_rows(case, seed)
    width = params["hidden"]

    def forward(ctx, x, out):
        if feed_forward:
            part.forward(ctx, x, out, 1.0, store=True)
        else:
            part.forward(ctx, x, out, 1.0, kv=ctx.kv_view(0, True) if cache_request else None,
                         state=ctx.state(0) if state_request else None, store=True)

    entries = []
    for x, count in zip(rows, counts):
        slot = cache.admit()
        assert cache.ensure(slot, 0, context + count)
        for at in range(0, context, STEP_TOKENS):
            end = min(at + STEP_TOKENS, context)
            ctx = runtime.begin([StepEntry(slot, [1] * (end - at), at, [])])
            forward(ctx, x[at:end].contiguous(), torch.empty(end - at, width, device=DEVICE))
            runtime.finish()
        entries.append(StepEntry(slot, [1] * count, context, []))
    x = torch.cat([r[context:] for r in rows])
    ctx = runtime.begin(entries)
    if ctx.n_tokens > x.shape[0]:                     # rows of nobody, as a step of single tokens has them
        x = torch.cat([x, torch.zeros(ctx.n_tokens - x.shape[0], width, dtype=dtype, device=DEVICE)])
    torch.cuda.synchronize()
    kept = []
    if cache_request:
        view = ctx.kv_view(0, True)
        kept = [view.k_pages, view.v_pages]
    elif state_request:
        kept = [ctx.state(0)]
    return {"kind": case["kind"], "forward": forward, "ctx": ctx, "x": x, "out": torch.empty(x.shape[0], width, device=DEVICE),
            "kept": kept, "runtime": runtime, "rows": sum(counts)}


def exact_part(case, seed):
    kind, p = part_spec(case)
    w = {name[2:]: t.to(F64) for name, t in part_weights(case, seed, part_specs(case)).items()}
    rows = [x.to(F64) for x in part_rows(case, seed)]
    if kind == "expert_mixture":
        return {"rows": exact_experts(p, w, rows[0]), "kept": []}
    outs, states = [], []
    for x, count in zip(rows, portions(case)):
        if kind == "latent_attention":
            outs.append(exact_latent(p, w, x, count))
        elif kind == "selective_scan":
            outs.append(exact_scan(p, w, x))
        else:
            out, state = exact_recurrence(kind, p, w, x)
            outs.append(out)
            states.append(state)
    kept = [None, None] if kind == "latent_attention" else [torch.stack(states)] if states else [None]
    return {"rows": torch.cat(outs), "kept": kept}


def exact_latent(p, w, x, count):
    n, H, d, dr, dv, rank = x.shape[0], p["heads"], p["head_dim"], p["rot_dim"], p["v_head_dim"], p["kv_rank"]
    start, new = n - count, x[n - count:]
    freq = p["rot"]["base"] ** (-2.0 * torch.arange(dr // 2, device=DEVICE, dtype=F64) / dr)
    rotate = rotate_pairs if p.get("rot_pairs") else rotate_halves
    both = x @ w["dkv"].T
    c = rms(both[:, :rank], p["norm_eps"]) * w["dkv.norm"]
    part = rotate(both[:, None, rank:], freq)[:, 0]
    q = (rms(new @ w["dq"].T, p["norm_eps"]) * w["dq.norm"]) @ w["uq"].T if p["q_rank"] else new @ w["q"].T
    q = q.view(count, H, d + dr)
    q = torch.cat([q[..., :d], rotate(q[..., d:], freq, start)], dim=-1)
    o = torch.empty(count, H, dv, device=DEVICE, dtype=F64)
    for h in range(H):
        k = torch.cat([c @ w["uk"][h * d:(h + 1) * d].T, part], dim=-1)
        o[:, h] = attend(q[:, h], k, c @ w["uv"][h * dv:(h + 1) * dv].T, p["scale"], p.get("window"), start)
    o = o.reshape(count, H * dv)
    if p.get("gate"):
        o = o * torch.sigmoid(new @ w["g"].T)
    return o @ w["o"].T


def exact_recurrence(kind, p, w, x):
    n, H, d, dv = x.shape[0], p["heads"], p["head_dim"], p["v_head_dim"]
    q, k, v = ((x @ w[name].T).view(n, H, -1) for name in ("q", "k", "v"))
    if kind == "retention":
        freq = p["rot"]["base"] ** (-2.0 * torch.arange(d // 2, device=DEVICE, dtype=F64) / d)
        q, k = rotate_halves(q, freq), rotate_halves(k, freq) * d ** -0.5
        decay = torch.tensor(p["decay"], device=DEVICE, dtype=F64)[None, :, None, None].expand(n, H, 1, 1)
    else:
        q = q * d ** -0.5
        z = (x @ w["a1"].T) @ w["a2"].T + w["a2.b"]
        decay = torch.exp(torch.nn.functional.logsigmoid(z) / p["tau"]).view(n, H, d, 1)
    S = torch.zeros(H, d, dv, device=DEVICE, dtype=F64)
    out = torch.empty(n, H, dv, device=DEVICE, dtype=F64)
    for t in range(n):
        S = decay[t] * S + k[t][:, :, None] * v[t][:, None, :]
        out[t] = (S * q[t][:, :, None]).sum(dim=1)
    out = rms(out, p["norm_eps"]) * (w["norm"] if "norm" in w else 1.0)
    gate = x @ w["g"].T
    return (out.reshape(n, H * dv) * gate * torch.sigmoid(gate)) @ w["o"].T, S


def exact_scan(p, w, x):
    n, inner, states, rank = x.shape[0], p["inner"], p["state"], p["dt_rank"]
    u, z = (x @ w["in"].T).chunk(2, dim=-1)
    padded = torch.cat([torch.zeros(p["taps"] - 1, inner, device=DEVICE, dtype=F64), u])
    u = w["conv.b"] + sum(padded[j:j + n] * w["conv"][:, j] for j in range(p["taps"]))
    u = u * torch.sigmoid(u)
    r, B, C = (u @ w["x"].T).split([rank, states, states], dim=-1)
    dt = torch.nn.functional.softplus(r @ w["dt"].T + w["dt.b"])
    A, S, y = -torch.exp(w["A_log"]), torch.zeros(inner, states, device=DEVICE, dtype=F64), torch.empty_like(u)
    for t in range(n):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * B[t]
        y[t] = S @ C[t]
    return ((y + w["D"] * u) * z * torch.sigmoid(z)) @ w["o"].T


def exact_experts(p, w, x):
    def mlp(rows, name):
        gate = rows @ w[name + "gate"].T
        return (rows @ w[name + "up"].T * gate * torch.sigmoid(gate)) @ w[name + "down"].T

    weights, chosen = torch.topk(torch.softmax(x @ w["router"].T, dim=-1), p["top"], dim=-1)
    out = torch.sigmoid(x @ w["shared.sg"].T) * mlp(x, "shared.")
    for e in range(p["experts"]):
        out = out + (weights * (chosen == e)).sum(dim=-1, keepdim=True) * mlp(x, f"e{e}.")
    return out


# ---- what is measured ----

def prepare(case, seed):
    return prepare_llama(case, seed) if case["kind"] == "llama" else prepare_part(case, seed)


def run(state):
    if state["kind"] == "llama":
        return {"logits": state["engine"].step(state["entries"]), "kept": state["kept"]}
    state["forward"](state["ctx"], state["x"], state["out"])
    return {"rows": state["out"][:state["rows"]], "kept": state["kept"]}


def exact(case, seed):
    return exact_llama(case, seed) if case["kind"] == "llama" else exact_part(case, seed)


def seen_keys(case):
    """(query, key) pairs of the case's new tokens, and the cached keys that they read, both over all requests."""
    window = 1024 if case.get("form") == "windowed" else None
    pairs = keys = 0
    for count in portions(case):
        last = case.get("context", 0) + count
        reach = [min(i + 1, window or i + 1) for i in range(last - count, last)]
        pairs += sum(reach)
        keys += min(last, (window or last) + count - 1)
    return pairs, keys


def work(case):
    """Bytes: every weight and every needed cache entry once, inputs and results once.  Flops: two a multiply-add of the
    products and of the visible (query, key) pairs, with keys and values of a latent expanded once."""
    n = case["tokens"]
    element = 4 if case["dtype"] == "float32" else 2
    if case["kind"] == "llama":
        c = llama_config(case)
        h, ff, nq, nkv, d = (c[k] for k in ("hidden_size", "intermediate_size", "num_attention_heads", "num_key_value_heads", "head_dim"))
        layer = (nq + 2 * nkv) * d * h + nq * d * h + 3 * ff * h
        pairs, keys = seen_keys(case)
        weights = case["layers"] * layer + c["vocab_size"] * h
        return {"bytes": element * (weights + case["layers"] * 2 * nkv * d * keys) + 4 * case["requests"] * c["vocab_size"],
                "flops": 2 * n * case["layers"] * layer + 2 * case["requests"] * c["vocab_size"] * h + case["layers"] * 4 * nq * d * pairs}
    kind, p = part_spec(case)
    matrices = {name: math.prod(shape) for name, shape in part_specs(case) if len(shape) == 2}
    rows = n * p["hidden"] * (element + 4)
    if kind == "expert_mixture":
        expert = 3 * p["hidden"] * p["intermediate"]
        shared = sum(matrices.values()) - p["experts"] * expert
        used = p["experts"] if n * p["top"] >= p["experts"] else n * p["top"]
        return {"bytes": element * (shared + used * expert) + rows, "flops": 2 * n * (shared + p["top"] * expert)}
    weights = sum(matrices.values())
    if kind == "latent_attention":
        pairs, keys = seen_keys(case)
        H, d, dr, dv, rank = p["heads"], p["head_dim"], p["rot_dim"], p["v_head_dim"], p["kv_rank"]
        expansion = H * (d + dv) * rank
        inputs = weights - expansion
        if case["phase"] == "decode":                 # the queries are taken into the latent's space instead
            attention = 2 * n * expansion + 2 * H * (2 * rank + dr) * pairs
        else:
            attention = 2 * keys * expansion + 2 * H * (d + dr + dv) * pairs
        return {"bytes": element * (weights + keys * (rank + dr)) + rows, "flops": 2 * n * inputs + attention}
    if kind == "selective_scan":
        state, recurrent = p["inner"] * (p["state"] + p["taps"] - 1), 6 * n * p["inner"] * p["state"]
    else:
        state = p["heads"] * p["head_dim"] * p["v_head_dim"]
        recurrent = 4 * n * state
    return {"bytes": element * weights + rows + 8 * state * case["requests"], "flops": 2 * n * weights + recurrent}


def tolerance(case):
    """Largest relative error between two correct implementations at the same precision: about four times what the cases
    show against `exact` (a stack of bfloat16 layers 0.0075, of 32-bit layers 1.7e-6; attention through latents 0.0039, the
    other parts 0.0017)."""
    if case["kind"] == "llama":
        return {"rel": 8e-6 if case["dtype"] == "float32" else 3e-2}
    return {"rel": 1.6e-2 if case["kind"] == "latent" else 7e-3}
