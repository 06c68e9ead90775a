"""What the engine's speed is measured on: the calls that a program makes, over the range of sizes it makes them for.

Two cases are whole steps of a Llama model of the 1B shape: a captured decode step and a long prompt.  The others
are single layers through the parts' own ``forward``, as a model calls them, at the layer sizes of the
configurations that the benchmark runs: feed-forwards (dense, routed experts) and mixers (paged attention,
latent attention, attention with a sink and a window, delta rule, gated linear attention, HGRN2, mLSTM).
Prompts come whole or as portions behind a cached context, several requests in a step, with lengths that are no
multiple of anything; decoding is one token per request.  Steps of up to 1,024 tokens are captured and replayed, longer
ones are launched one kernel at a time, as the engine does.
"""

from __future__ import annotations

import math
import zlib

import torch

DEVICE = "cuda"
PAGE = 16  # tokens per cache page
CAPTURED_TOKENS = 1024  # up to here the engine replays captured steps
EPS = 1e-5
THETA = 10000.0

LLAMA_1B = {
    "architectures": ["LlamaForCausalLM"], "vocab_size": 128256, "hidden_size": 2048, "intermediate_size": 8192,
    "num_hidden_layers": 16, "num_attention_heads": 32, "num_key_value_heads": 8, "head_dim": 64,
    "max_position_embeddings": 8192, "rms_norm_eps": 1e-5, "rope_theta": 500000.0, "tie_word_embeddings": True,
}
MODEL_KINDS = ("llama",)
FEED_FORWARDS = ("mlp", "experts")
RECURRENT = ("delta", "gla", "hgrn2", "mlstm")
ATTENTIONS = ("attention", "latent", "sink")


def listed():
    bf, f32 = "bfloat16", "float32"
    return [
        # a decode step of eight chats: the engine's headline
        {"name": "llama_decode_b8", "kind": "llama", "dtype": bf, "lens": "1,1,1,1,1,1,1,1",
         "starts": "1024,1024,1024,1024,1024,1024,1024,1024"},
        # a long prompt by itself
        {"name": "llama_prompt_2048", "kind": "llama", "dtype": bf, "lens": "2048", "starts": "0"},
        # a dense feed-forward on a step of odd size
        {"name": "mlp_1000", "kind": "mlp", "dtype": bf, "hidden": 2048, "ff": 8192, "lens": "1000", "starts": "0"},
        # attention of the 8B shape: a portion deep in a document, a new prompt and decoding requests in one step
        {"name": "attention_mixed", "kind": "attention", "dtype": bf, "hidden": 4096, "heads": 32, "kv_heads": 8, "dim": 128,
         "lens": "512,300,1,1,1,1", "starts": "8192,0,3000,517,1200,64"},
        # the 32-bit path: two short prompts
        {"name": "attention_f32", "kind": "attention", "dtype": f32, "hidden": 1024, "heads": 16, "kv_heads": 4, "dim": 64,
         "lens": "300,77", "starts": "0,150"},
        # routed experts: a prompt, and a decode step
        {"name": "experts_2048", "kind": "experts", "dtype": bf, "hidden": 2048, "ff": 1024, "experts": 32, "top": 4,
         "groups": 4, "keep": 2, "limit": 7.0, "scoring": "softmax", "lens": "2048", "starts": "0"},
        {"name": "experts_8", "kind": "experts", "dtype": bf, "hidden": 2048, "ff": 1024, "experts": 32, "top": 4,
         "groups": 1, "keep": 1, "limit": None, "scoring": "softmax", "lens": "1,1,1,1,1,1,1,1",
         "starts": "1024,1024,1024,1024,1024,1024,1024,1024"},
        # recurrent layers: a long prompt, two prompts of odd lengths, a short prompt of the smaller width
        {"name": "delta_2048", "kind": "delta", "dtype": bf, "hidden": 2048, "heads": 16, "dim": 128, "vdim": 128, "rank": 64,
         "lens": "2048", "starts": "0"},
        {"name": "gla_1337_663", "kind": "gla", "dtype": bf, "hidden": 2048, "heads": 16, "dim": 128, "vdim": 128, "rank": 32,
         "lens": "1337,663", "starts": "0,0"},
        {"name": "hgrn2_513", "kind": "hgrn2", "dtype": bf, "hidden": 1024, "heads": 8, "dim": 128, "vdim": 128, "rank": 0,
         "lens": "513", "starts": "0"},
        # attention over a shared latent and attention with a sink and a window: a long prompt each
        {"name": "latent_2048", "kind": "latent", "dtype": bf, "hidden": 2048, "heads": 16, "dim": 128, "rot": 64, "vdim": 128,
         "rank": 512, "lens": "2048", "starts": "0"},
        {"name": "sink_2048", "kind": "sink", "dtype": bf, "hidden": 2048, "heads": 16, "kv_heads": 4, "dim": 128, "vdim": 128,
         "window": 1024, "softcap": None, "lens": "2048", "starts": "0"},
    ]


def draw(rng):
    """A step of one of the kinds: decoding requests, whole prompts or portions behind a context, of any length."""
    kind = rng.choice(("llama",) + FEED_FORWARDS + RECURRENT + ATTENTIONS)
    small = rng.random() < 0.4  # which of the two layer sizes
    dtype = "float32" if kind != "llama" and rng.random() < 0.15 else "bfloat16"

    def log_uniform(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    most = 160 if dtype == "float32" else 2000
    if kind not in RECURRENT and rng.random() < 0.4:
        batch = log_uniform(1, 48)
        lens = [1] * batch
    else:
        lens = [log_uniform(2, most // 2) for _ in range(rng.choice((1, 1, 2, 3)))]
        while sum(lens) > most:
            lens.pop()
    starts = [0] * len(lens)
    if kind in ATTENTIONS or kind == "llama":
        starts = [rng.choice((0, 1)) * log_uniform(16, 4000) if n > 1 else log_uniform(16, 4000) for n in lens]
        if kind == "llama":
            lens, starts = lens[:16], starts[:16]
    case = {"kind": kind, "dtype": dtype, "lens": ",".join(map(str, lens)), "starts": ",".join(map(str, starts))}
    hidden = 1024 if small else 2048
    if kind == "mlp":
        case.update(hidden=hidden, ff=4 * hidden)
    elif kind == "experts":
        case.update(hidden=hidden, ff=512 if small else 1024, experts=16 if small else 32, top=rng.choice((2, 4)),
                    groups=4 if not small else 1, keep=2 if not small else 1, limit=rng.choice((None, 7.0)),
                    scoring=rng.choice(("softmax", "sigmoid")))
    elif kind in RECURRENT:
        dim = 64 if kind == "mlstm" else rng.choice((64, 128))
        case.update(hidden=hidden, heads=8 if small else 16, dim=dim, vdim=rng.choice((64, 128)),
                    rank=rng.choice((16, 32, 64)) if kind in ("delta", "gla") else 0)
    elif kind == "attention":
        hidden = rng.choice((1024, 2048, 4096))
        dim = 128 if hidden == 4096 else 64
        case.update(hidden=hidden, heads=hidden // dim, kv_heads=hidden // dim // 4, dim=dim)
    elif kind == "latent":
        case.update(hidden=hidden, heads=8 if small else 16, dim=64 if small else 128, rot=32 if small else 64,
                    vdim=64 if small else 128, rank=256 if small else 512)
    elif kind == "sink":
        dim = 64 if small else 128
        case.update(hidden=hidden, heads=16, kv_heads=4, dim=dim, vdim=dim, window=rng.choice((None, 512, 1024)),
                    softcap=rng.choice((None, 40.0)))
    return case


# --- what a case is made of ---------------------------------------------------------------------------


def _numbers(text):
    return [int(n) for n in str(text).split(",")]


def _generator(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) * 0x9E3779B1 + zlib.crc32(name.encode())) % (2**63 - 1))


def _normal(seed, name, shape, std=1.0, mean=0.0, dtype=torch.bfloat16):
    return (torch.randn(shape, generator=_generator(seed, name), device=DEVICE) * std + mean).to(dtype)


def _shapes(case):
    """name -> (shape, standard deviation, mean) of the layer's tensors."""
    kind, c, h = case["kind"], case, case["hidden"]
    if kind == "mlp":
        return {"gate": ((c["ff"], h), 0.02, 0), "up": ((c["ff"], h), 0.02, 0), "down": ((h, c["ff"]), 0.02, 0)}
    if kind == "experts":
        out = {"router": ((c["experts"], h), 0.02, 0)}
        if c["scoring"] == "sigmoid":
            out["correction"] = ((c["experts"],), 0.01, 0)
        for e in range(c["experts"]):
            out.update({f"e{e}.gate": ((c["ff"], h), 0.02, 0), f"e{e}.up": ((c["ff"], h), 0.02, 0),
                        f"e{e}.down": ((h, c["ff"]), 0.02, 0)})
        return out
    if kind == "attention":
        q, k = c["heads"] * c["dim"], c["kv_heads"] * c["dim"]
        return {"q": ((q, h), 0.02, 0), "k": ((k, h), 0.02, 0), "v": ((k, h), 0.02, 0), "o": ((h, q), 0.02, 0)}
    if kind == "latent":
        H, d, r, v, rank = c["heads"], c["dim"], c["rot"], c["vdim"], c["rank"]
        return {"q": ((H * (d + r), h), 0.02, 0), "dkv": ((rank + r, h), 0.02, 0), "latent_norm": ((rank,), 0.02, 1),
                "uk": ((H * d, rank), 0.03, 0), "uv": ((H * v, rank), 0.03, 0), "gate": ((H, h), 0.02, 0),
                "o": ((h, H * v), 0.02, 0)}
    if kind == "sink":
        H, G, d, v = c["heads"], c["kv_heads"], c["dim"], c["vdim"]
        return {"q": ((H * d, h), 0.02, 0), "k": ((G * d, h), 0.02, 0), "v": ((G * v, h), 0.02, 0),
                "q_bias": ((H * d,), 0.02, 0), "k_bias": ((G * d,), 0.02, 0), "v_bias": ((G * v,), 0.02, 0),
                "sink": ((H,), 1.0, 0), "head_gate": ((H, h), 0.02, 0), "o": ((h, H * v), 0.02, 0)}
    H, d, v, r = c["heads"], c["dim"], c["vdim"], c["rank"]
    if kind == "delta":  # (decays between about 0.8 and 0.99, as trained ones are)
        return {"q": ((H * d, h), 0.02, 0), "k": ((H * d, h), 0.02, 0), "v": ((H * v, h), 0.02, 0),
                "q_conv": ((H * d, 4), 0.3, 0.2), "k_conv": ((H * d, 4), 0.3, 0.2), "v_conv": ((H * v, 4), 0.3, 0.2),
                "beta": ((H, h), 0.02, 0), "A_log": ((H,), 0.5, 0), "dt_bias": ((H * d,), 1.0, -3.0),
                "a1": ((r, h), 0.02, 0), "a2": ((H * d, r), 0.1, 0), "g1": ((r, h), 0.02, 0), "g2": ((H * v, r), 0.1, 0),
                "out_norm": ((v,), 0.02, 1), "o": ((h, H * v), 0.02, 0)}
    if kind == "gla":
        return {"q": ((H * d, h), 0.02, 0), "k": ((H * d, h), 0.02, 0), "v": ((H * v, h), 0.02, 0), "g": ((H * v, h), 0.02, 0),
                "a1": ((r, h), 0.02, 0), "a2": ((H * d, r), 0.2, 0), "a2_bias": ((H * d,), 1.0, 1.0),
                "out_norm": ((v,), 0.02, 1), "o": ((h, H * v), 0.02, 0)}
    if kind == "hgrn2":
        return {"q": ((H * d, h), 0.02, 0), "f": ((H * d, h), 0.02, 0), "f_bias": ((H * d,), 1.0, 2.0),
                "lower": ((H * d,), 0.0, 0), "v": ((H * v, h), 0.02, 0), "out_norm": ((v,), 0.02, 1),
                "o": ((h, H * v), 0.02, 0)}
    return {"q": ((H * d, h), 0.02, 0), "k": ((H * d, h), 0.02, 0), "v": ((H * v, h), 0.02, 0), "g": ((H * v, h), 0.02, 0),
            "i": ((H, h), 0.02, 0), "i_bias": ((H,), 0.5, 0), "f": ((H, h), 0.02, 0), "f_bias": ((H,), 1.0, 3.0),
            "out_norm": ((H * v,), 0.02, 1), "o": ((h, H * v), 0.02, 0)}


def _tensors(case, seed):
    return {n: _normal(seed, n, shape, std, mean) for n, (shape, std, mean) in _shapes(case).items()}


def _inputs(case, seed):
    """The layer's normalised input rows, and for feed-forwards the residual stream they are added to."""
    n = sum(_numbers(case["lens"]))
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    return _normal(seed, "input", (n, case["hidden"]), dtype=dtype), _normal(seed, "residual", (n, case["hidden"]), dtype=torch.float32)


def _cached(case, seed, what, start, request, heads, dim, std=1.0):
    """``[start, heads, dim]``: what earlier steps left in the cache of a request."""
    dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
    return _normal(seed, f"{what}.{request}", (start, heads, dim), std, dtype=dtype)


def _cache_sizes(case):
    """(heads, key size, value size) of a cached token."""
    if case["kind"] == "latent":
        return 1, case["rank"] + case["rot"], 0
    return case["kv_heads"], case["dim"], case.get("vdim", case["dim"])


# --- the engine's side --------------------------------------------------------------------------------


def _spec(case):
    from inference_engine_b200.config.spec import LayerSpec, ModelSpec, PartSpec, ScheduleEntry

    c, kind = case, case["kind"]
    names = {n: n for n in _shapes(case)}
    attention = {"q_proj": "m.q", "k_proj": "m.k", "v_proj": "m.v", "o_proj": "m.o", "num_heads": 1, "num_kv_heads": 1,
                 "head_dim": 64, "position": "rotary", "window": None}
    feed_forward, positions = None, {"rotary": PartSpec("rotary", {"rotary_dim": 64, "theta": THETA})}
    mixer = PartSpec("paged_attention", attention)
    if kind == "mlp":
        feed_forward = PartSpec("swiglu", {"gate_proj": "gate", "up_proj": "up", "down_proj": "down", "intermediate_size": c["ff"]})
    elif kind == "experts":
        sigmoid = c["scoring"] == "sigmoid"
        feed_forward = PartSpec("routed_experts", {
            "router": "router", "expert_prefix": "e", "experts": c["experts"], "top": c["top"], "groups": c["groups"],
            "keep_groups": c["keep"], "intermediate_size": c["ff"], "limit": c["limit"], "alpha": 1.0, "up_offset": 0.0,
            "scoring": c["scoring"], "correction": "correction" if sigmoid else None})
    elif kind == "attention":
        positions = {"rotary": PartSpec("rotary", {"rotary_dim": c["dim"], "theta": THETA})}
        mixer = PartSpec("paged_attention", {"q_proj": "q", "k_proj": "k", "v_proj": "v", "o_proj": "o", "num_heads": c["heads"],
                                             "num_kv_heads": c["kv_heads"], "head_dim": c["dim"], "position": "rotary"})
    elif kind == "latent":
        positions = {"rotary": PartSpec("rotary", {"rotary_dim": c["rot"], "theta": THETA, "layout": "interleaved"})}
        mixer = PartSpec("latent_attention", {
            "names": names, "heads": c["heads"], "dim": c["dim"], "rot_dim": c["rot"], "vdim": c["vdim"], "kv_rank": c["rank"],
            "scale": (c["dim"] + c["rot"]) ** -0.5, "eps": EPS, "position": "rotary"})
    elif kind == "sink":
        positions = {}
        mixer = PartSpec("sink_attention", {
            "names": names, "heads": c["heads"], "kv_heads": c["kv_heads"], "dim": c["dim"], "vdim": c["vdim"],
            "scale": c["dim"] ** -0.5, "window": c["window"], "value_norm": True, "eps": EPS, "softcap": c["softcap"]})
    else:
        sizes = {"names": names, "heads": c["heads"], "dim": c["dim"], "vdim": c["vdim"], "eps": EPS}
        if kind == "delta":
            mixer = PartSpec("channel_delta", {**sizes, "kv_heads": c["heads"], "taps": 4, "decay_rank": c["rank"],
                                               "gate_rank": c["rank"]})
        elif kind == "gla":
            mixer = PartSpec("gla", {**sizes, "rank": c["rank"], "tau": 8.0})
        elif kind == "hgrn2":
            mixer = PartSpec("hgrn2", sizes)
        else:
            mixer = PartSpec("mlstm", {**sizes, "gate_cap": 15.0})
    norms = {"pre_mixer": PartSpec("rms", {"weight": "norm", "eps": EPS})}
    if feed_forward is not None:
        norms["pre_feed_forward"] = PartSpec("rms", {"weight": "norm2", "eps": EPS})
    return ModelSpec(
        architecture="one layer", vocab_size=64, hidden_size=c["hidden"], max_position_embeddings=16384,
        embedding=PartSpec("token", {"weight": "embed", "vocab_size": 64}), positions=positions,
        layers=(LayerSpec("l0", PartSpec("prenorm_residual"), mixer, feed_forward, norms),), schedule=(ScheduleEntry(0),),
        final_norm=PartSpec("rms", {"weight": "final", "eps": EPS}), head=PartSpec("linear", {"weight": "head", "vocab_size": 64}))


class _State:
    pass


def _fill(case, seed, runner, heads, k_size, v_size, request, start, layer):
    """The keys and values of ``start`` earlier tokens, into the request's pages."""
    if start == 0:
        return
    storage = runner.storage.paged[0]
    count = -(-start // PAGE)
    pages = torch.tensor(runner.cache.table(0, request)[:count], device=DEVICE)
    for what, store, size in (("keys", storage.k, k_size), ("values", storage.v, v_size)):
        if not size:
            continue
        rows = torch.zeros(count * PAGE, heads, size, dtype=store.dtype, device=DEVICE)
        rows[:start] = _cached(case, seed, f"{what}{layer}", start, request, heads, size)
        store[layer, pages] = rows.view(count, PAGE, heads, size).transpose(1, 2)


def _prepare_model(case, seed):
    from inference_engine_b200.engine.batch import StepEntry
    from inference_engine_b200.engine.graphs import DecodeGraphs, MixedGraphs
    from inference_engine_b200.engine.loading import random_model
    from inference_engine_b200.engine.runner import make_runner
    from inference_engine_b200.kernels import get_ops

    lens, starts = _numbers(case["lens"]), _numbers(case["starts"])
    s = _State()
    model, _ = random_model(LLAMA_1B, seed=seed, dtype=case["dtype"], device=DEVICE)
    pages = sum(-(-(a + n) // PAGE) for a, n in zip(starts, lens)) + 8
    s.runner = runner = make_runner(model, get_ops(DEVICE), DEVICE, PAGE, pages, max(len(lens) + 1, 8), max(sum(lens), 64))
    for group in runner.storage.paged:
        group.k.zero_()
        group.v.zero_()
    tokens = torch.randint(0, LLAMA_1B["vocab_size"], (sum(lens),), generator=_generator(seed, "tokens"), device=DEVICE).tolist()
    s.entries, at = [], 0
    for i, (a, n) in enumerate(zip(starts, lens)):
        runner.cache.add_request(i)
        runner.cache.grow(i, 0, a + n)
        for layer in range(LLAMA_1B["num_hidden_layers"]):
            _fill(case, seed, runner, 8, 64, 64, i, a, layer)
        s.entries.append(StepEntry(i, tokens[at: at + n], a, [n - 1]))
        at += n
    decode = DecodeGraphs(runner, runner.max_seqs, LLAMA_1B["max_position_embeddings"] // PAGE)
    if max(lens) == 1:
        s.step = lambda: decode.run(s.entries)
    elif sum(lens) <= CAPTURED_TOKENS:
        mixed = MixedGraphs(decode)
        s.step = lambda: mixed.run(s.entries)
    else:
        s.step = lambda: runner.step(s.entries)
    s.step()  # (captures where a step is captured)
    storage = runner.storage.paged[0]
    s.call = lambda: {"logits": s.step(), "keys": storage.k[:, : storage.num_pages], "values": storage.v[:, : storage.num_pages]}
    return s


def prepare(case, seed):
    if case["kind"] in MODEL_KINDS:
        return _prepare_model(case, seed)
    from inference_engine_b200.engine.batch import StepEntry
    from inference_engine_b200.engine.model import Model
    from inference_engine_b200.engine.runner import make_runner
    from inference_engine_b200.kernels import get_ops

    lens, starts = _numbers(case["lens"]), _numbers(case["starts"])
    n, h, kind = sum(lens), case["hidden"], case["kind"]
    s = _State()
    model = Model(_spec(case), case["dtype"], 16384, DEVICE)
    given, own = _tensors(case, seed), {}
    for name, decl in model.declared_weights().items():
        plain = name.removeprefix("m.") if kind in FEED_FORWARDS and name.startswith("m.") else None
        own[name] = torch.zeros(decl.shape, dtype=torch.bfloat16, device=DEVICE) if plain else given.get(name)
        if own[name] is None:  # (norms, embedding and head around the layer)
            own[name] = torch.ones(decl.shape, dtype=torch.bfloat16, device=DEVICE)
    model.load(own)
    pages = sum(-(-(a + q) // PAGE) for a, q in zip(starts, lens)) + 8
    s.runner = runner = make_runner(model, get_ops(DEVICE), DEVICE, PAGE, pages, max(len(lens) + 1, 8), max(n, 64))
    for group in runner.storage.paged:
        group.k.zero_()
        if group.v is not None:
            group.v.zero_()
    entries = []
    for i, (a, q) in enumerate(zip(starts, lens)):
        runner.cache.add_request(i)
        runner.cache.grow(i, 0, a + q)
        if runner.cache.state_slot(i) != i:
            raise RuntimeError("requests take the state slots in their order")
        if kind in ATTENTIONS:
            _fill(case, seed, runner, *_cache_sizes(case), i, a, 0)
        entries.append(StepEntry(i, [0] * q, a, []))
    ctx, _ = runner.build_context(entries)
    x, residual = _inputs(case, seed)
    block, binding = model.blocks[0], model.bindings[0]
    rows = torch.arange(n, dtype=torch.int32, device=DEVICE)

    def layer():
        if kind in FEED_FORWARDS:  # the slices of the result are added by the norm that follows, as in a model
            delta = block.feed_forward.forward(x, ctx)
            return {"out": model.final_norm.add_norm(residual, delta, ctx, rows=rows)}
        if kind in RECURRENT:  # requests that start at position 0 start from a zero state
            state = runner.storage.state[0][0]
            state[: len(lens)].zero_()
        delta = block.mixer.forward(x, ctx, binding)
        out = {"out": delta if delta.dim() == 2 else delta.sum(0)}
        if kind in RECURRENT:
            out["state"] = state[: len(lens)]
        else:
            storage = runner.storage.paged[0]
            out["keys"] = storage.k[0, : storage.num_pages]
            if storage.v is not None and kind != "latent":
                out["values"] = storage.v[0, : storage.num_pages]
        return out

    s.kept = (model, ctx, x, residual, rows)
    s.call = layer
    if n <= CAPTURED_TOKENS:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            layer()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            out = layer()
        s.graph, s.out = graph, out

        def replay():
            graph.replay()
            return out

        s.call = replay
    return s


def run(state):
    return state.call()


# --- what a pass cannot do without --------------------------------------------------------------------


def _seen(lens, starts, window=None):
    """(query, key) pairs and distinct cached rows read."""
    pairs = rows = 0
    for q, a in zip(lens, starts):
        if window is None:
            pairs += q * a + q * (q + 1) // 2
            rows += a + q
        else:
            pairs += sum(min(a + i + 1, window) for i in range(q))
            rows += min(a + q, window + q - 1)
    return pairs, rows


def work(case):
    lens, starts, kind = _numbers(case["lens"]), _numbers(case["starts"]), case["kind"]
    n, act = sum(lens), 2 if case["dtype"] == "bfloat16" else 4
    if kind == "llama":
        c = LLAMA_1B
        h, layers, vocab = c["hidden_size"], c["num_hidden_layers"], c["vocab_size"]
        per_layer = 2 * h * h + 2 * h * 512 + 3 * h * c["intermediate_size"]
        pairs, rows = _seen(lens, starts)
        return {"bytes": 2 * (layers * per_layer + vocab * h) + layers * rows * 2 * 512 * 2 + len(lens) * vocab * 4 + n * h * 2,
                "flops": 2 * n * layers * per_layer + 2 * len(lens) * vocab * h + layers * pairs * 4 * 2048}
    h = case["hidden"]
    if kind == "experts":
        used = min(case["experts"], n * case["top"])
        per_expert = 3 * h * case["ff"]
        # the stream is read, the normalised rows are written
        return {"bytes": 2 * used * per_expert + 4 * case["experts"] * h + n * h * (2 * act + 4),
                "flops": 2 * n * case["top"] * per_expert + 2 * n * case["experts"] * h}
    weights = sum(math.prod(shape) for shape, _, _ in _shapes(case).values())
    byte, flops = 2 * weights if act == 2 else 4 * weights, 2 * n * weights
    if kind == "mlp":
        return {"bytes": byte + n * h * (2 * act + 4), "flops": flops}
    byte += n * h * (act + 4)
    if kind in RECURRENT:
        state = case["heads"] * case["dim"] * case["vdim"]
        return {"bytes": byte + 4 * len(lens) * state, "flops": flops + n * state * (8 if kind == "delta" else 6)}
    heads, k_size, v_size = _cache_sizes(case)
    pairs, rows = _seen(lens, starts, case.get("window"))
    byte += act * rows * heads * (k_size + v_size)
    if kind == "latent":  # keys and values per head, as if they were at hand
        return {"bytes": byte, "flops": flops + 2 * pairs * case["heads"] * (case["dim"] + case["rot"] + case["vdim"])}
    return {"bytes": byte, "flops": flops + 2 * pairs * case["heads"] * (k_size + v_size)}


def tolerance(case):
    """About four times what another order of the sums at the same precision shows against 64 bits."""
    if case["kind"] == "llama":  # sixteen layers' roundings add up
        return {"rel": 0.03, "max": 0.3}
    if case["dtype"] == "float32":
        return {"rel": 2e-4, "max": 5e-3}
    return {"rel": 0.012, "max": 0.12}


# --- the same in 64 bits, in plain torch --------------------------------------------------------------


def _rms(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _rotate(x, positions, interleaved):
    """``x``: [tokens, heads, dim], all of it rotated."""
    dim = x.shape[-1]
    freq = THETA ** (-torch.arange(0, dim, 2, dtype=torch.float64, device=x.device) / dim)
    angle = positions.double()[:, None] * freq
    c, s = angle.cos()[:, None, :], angle.sin()[:, None, :]
    if interleaved:
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], dim=-1).flatten(-2)
    a, b = x[..., : dim // 2], x[..., dim // 2:]
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def _attend(q, k, v, start, scale, window=None, softcap=None, sink=None):
    """``q``: [tokens, heads, d]; ``k``, ``v``: [context, kv heads, d]."""
    n, heads = q.shape[:2]
    group = heads // k.shape[1]
    at = torch.arange(n, device=q.device)[:, None] + start
    key = torch.arange(k.shape[0], device=q.device)[None, :]
    hidden = key > at
    if window is not None:
        hidden |= key <= at - window
    out = []
    for h in range(heads):
        s = (q[:, h] @ k[:, h // group].T) * scale
        if softcap is not None:
            s = softcap * torch.tanh(s / softcap)
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], dim=1)
        p = torch.softmax(s, dim=-1)[:, : k.shape[0]]
        out.append(p @ v[:, h // group])
    return torch.stack(out, dim=1)


def _exact_experts(case, w, x, residual):
    logits = x @ w["router"].T
    n, experts, groups, keep, top = x.shape[0], case["experts"], case["groups"], case["keep"], case["top"]
    sigmoid = case["scoring"] == "sigmoid"
    scores = torch.sigmoid(logits) if sigmoid else torch.softmax(logits, dim=-1)
    choice = scores + w["correction"] if sigmoid else scores
    if keep < groups:
        best = choice.view(n, groups, -1).amax(-1).topk(keep, dim=-1).indices
        kept = torch.zeros(n, groups, dtype=torch.bool, device=x.device).scatter_(1, best, True)
        choice = choice.masked_fill(~kept.repeat_interleave(experts // groups, dim=1), -math.inf)
    ids = choice.topk(top, dim=-1).indices
    weight = scores.gather(1, ids)
    weight = weight / weight.sum(-1, keepdim=True)
    total = torch.zeros_like(x)
    for e in range(experts):
        token, place = (ids == e).nonzero(as_tuple=True)
        if token.numel() == 0:
            continue
        rows = x[token]
        g, u = rows @ w[f"e{e}.gate"].T, rows @ w[f"e{e}.up"].T
        if case["limit"] is not None:
            g, u = g.clamp(max=case["limit"]), u.clamp(-case["limit"], case["limit"])
        total.index_add_(0, token, (_silu(g) * u) @ w[f"e{e}.down"].T * weight[token, place][:, None])
    return _rms(residual + total)


def _recurrence(q, k, v, decay, beta=None):
    """S <- diag(decay) S; S <- S + k u^T with u = v, or beta (v - S^T k) of the decayed state; o = S^T q."""
    n, heads, dim = q.shape
    S = torch.zeros(heads, dim, v.shape[-1], dtype=torch.float64, device=q.device)
    out = torch.empty(n, heads, v.shape[-1], dtype=torch.float64, device=q.device)
    for t in range(n):
        S = decay[t][:, :, None] * S
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hkv,hk->hv", S, q[t])
    return out, S


def _exact_recurrent(case, w, x):
    """One request: the layer's output and what it leaves in the request's slot."""
    kind, n, H, d, v = case["kind"], x.shape[0], case["heads"], case["dim"], case["vdim"]
    lin = lambda name: x @ w[name].T  # noqa: E731
    heads = lambda t, size: t.view(n, H, size)  # noqa: E731
    if kind == "hgrn2":
        f = w["lower"] + (1 - w["lower"]) * torch.sigmoid(lin("f") + w["f_bias"])
        o, S = _recurrence(heads(_silu(lin("q")), d), heads(1 - f, d), heads(lin("v"), v), heads(f, d))
        y = (_rms(o) * w["out_norm"]).flatten(1)
    elif kind == "gla":
        decay = torch.exp(torch.nn.functional.logsigmoid(lin("a1") @ w["a2"].T + w["a2_bias"]) / 8.0)
        o, S = _recurrence(heads(lin("q") * d ** -0.5, d), heads(lin("k"), d), heads(lin("v"), v), heads(decay, d))
        y = (_rms(o) * w["out_norm"]).flatten(1) * _silu(lin("g"))
    elif kind == "mlstm":
        cap = 15.0
        logi = cap * torch.tanh((lin("i") + w["i_bias"]) / cap)
        logf = torch.nn.functional.logsigmoid(cap * torch.tanh((lin("f") + w["f_bias"]) / cap))
        m, a, b, ms = torch.zeros(H, dtype=torch.float64, device=x.device), [], [], []
        for t in range(n):
            new = torch.maximum(logf[t] + m, logi[t])
            a.append(torch.exp(logf[t] + m - new))
            b.append(torch.exp(logi[t] - new))
            m = new
            ms.append(m)
        a, b, ms = torch.stack(a), torch.stack(b), torch.stack(ms)
        value = torch.cat([heads(lin("v"), v), torch.ones(n, H, 1, dtype=torch.float64, device=x.device)], dim=-1) * b[..., None]
        o, S = _recurrence(heads(lin("q") * d ** -0.5, d), heads(lin("k"), d), value, a[..., None].expand(n, H, d))
        o = o[..., :v] / (torch.maximum(o[..., v].abs(), torch.exp(-ms)) + 1e-6)[..., None]
        y = _rms(o).flatten(1) * w["out_norm"] * torch.sigmoid(lin("g"))
        return y @ w["o"].T, torch.cat([S.transpose(1, 2).reshape(-1), m])
    else:
        raw = torch.cat([lin("q"), lin("k"), lin("v")], dim=1)
        taps = torch.cat([w["q_conv"], w["k_conv"], w["v_conv"]])
        before = torch.cat([torch.zeros(3, raw.shape[1], dtype=torch.float64, device=x.device), raw])
        mixed = _silu(sum(before[j: j + n] * taps[:, j] for j in range(4)))
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
        q, k = unit(heads(mixed[:, : H * d], d)) * d ** -0.5, unit(heads(mixed[:, H * d: 2 * H * d], d))
        a = lin("a1").bfloat16().double() if case["dtype"] == "bfloat16" else lin("a1")  # (the low-rank values' own precision)
        decay = torch.exp(-torch.exp(w["A_log"])[:, None] * heads(torch.nn.functional.softplus(a @ w["a2"].T + w["dt_bias"]), d))
        o, S = _recurrence(q, k, heads(mixed[:, 2 * H * d:], v), decay, torch.sigmoid(lin("beta")))
        y = (_rms(o) * w["out_norm"]).flatten(1) * torch.sigmoid(lin("g1") @ w["g2"].T)
        return y @ w["o"].T, torch.cat([S.transpose(1, 2).reshape(-1), before[n: n + 3].reshape(-1)])
    return y @ w["o"].T, S.transpose(1, 2).reshape(-1)


def _exact_attention(case, w, x, start, cached):
    """One request: the layer's output.  ``cached``: keys and values of its earlier tokens."""
    kind, n, H, d = case["kind"], x.shape[0], case["heads"], case["dim"]
    lin = lambda name: x @ w[name].T  # noqa: E731
    at = torch.arange(start, start + n, device=x.device)
    if kind == "attention":
        q, k = (_rotate(lin(t).view(n, -1, d), at, False) for t in ("q", "k"))
        k, v = torch.cat([cached[0], k]), torch.cat([cached[1], lin("v").view(n, -1, d)])
        return _attend(q, k, v, start, d ** -0.5).flatten(1) @ w["o"].T
    if kind == "sink":
        v = _rms((lin("v") + w["v_bias"]).view(n, -1, case["vdim"]))
        k = torch.cat([cached[0], (lin("k") + w["k_bias"]).view(n, -1, d)])
        o = _attend((lin("q") + w["q_bias"]).view(n, H, d), k, torch.cat([cached[1], v]), start, d ** -0.5, case["window"],
                    case["softcap"], w["sink"])
        return (o * torch.sigmoid(lin("head_gate"))[..., None]).flatten(1) @ w["o"].T
    r, rank, vd = case["rot"], case["rank"], case["vdim"]
    q, low = lin("q").view(n, H, d + r), lin("dkv")
    c = torch.cat([_rms(low[:, :rank]) * w["latent_norm"], _rotate(low[:, None, rank:], at, True)[:, 0]], dim=1)
    c = torch.cat([cached[0][:, 0], c])
    k = torch.cat([(c[:, :rank] @ w["uk"].T).view(-1, H, d), c[:, None, rank:].expand(-1, H, r)], dim=-1)
    v = (c[:, :rank] @ w["uv"].T).view(-1, H, vd)
    q = torch.cat([q[..., :d], _rotate(q[..., d:], at, True)], dim=-1)
    o = _attend(q, k, v, start, (d + r) ** -0.5)
    return (o * torch.sigmoid(lin("gate"))[..., None]).flatten(1) @ w["o"].T


def exact(case, seed):
    if case["kind"] == "llama":
        return None
    kind, lens, starts = case["kind"], _numbers(case["lens"]), _numbers(case["starts"])
    w = {n: t.double() for n, t in _tensors(case, seed).items()}
    x, residual = (t.double() for t in _inputs(case, seed))
    if kind == "mlp":
        return {"out": _rms(residual + (_silu(x @ w["gate"].T) * (x @ w["up"].T)) @ w["down"].T)}
    if kind == "experts":
        return {"out": _exact_experts(case, w, x, residual)}
    outs, states, at = [], [], 0
    for i, (n, start) in enumerate(zip(lens, starts)):
        rows = x[at: at + n]
        at += n
        if kind in RECURRENT:
            o, state = _exact_recurrent(case, w, rows)
            states.append(state)
        else:
            heads, k_size, v_size = _cache_sizes(case)
            cached = [_cached(case, seed, f"{t}0", start, i, heads, size).double() if size else None
                      for t, size in (("keys", k_size), ("values", v_size))]
            o = _exact_attention(case, w, rows, start, cached)
        outs.append(o)
    if kind in RECURRENT:
        return {"out": torch.cat(outs), "state": torch.stack(states)}
    return {"out": torch.cat(outs), "keys": None, "values": None} if kind != "latent" else {"out": torch.cat(outs), "keys": None}
