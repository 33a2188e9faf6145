"""The work that the engine's speed is measured on.

A case is a few steps of the step function (``ModelRunner.step``) on requests that hold given contexts, or one call of
``Engine.generate``.  The listed cases are what a serving engine does all day: decoding at small, ordinary and large batches
and at unequal contexts, whole prompts, a portion of a long prompt, a portion beside decoding requests, the float32 path, a
design with recurrent mixers, and a small model's generation, where only launches and the host count.  ``draw`` gives more of the
same ranges.

Weights are random (normal 0.02, norm weights 1 + normal 0.1: the engine's own random-weights mode), token ids uniform, contexts
normal: all made on the GPU from the seed.  ``exact`` computes the same in float64 with plain torch.
"""
import math
import zlib
from types import SimpleNamespace

import torch

F64 = torch.float64
DEVICE = "cuda"
# the caches of this many layers, the last ones, are outputs beside the logits: their rows depend on every layer before them
CACHES_RETURNED = 4

# Of the 36 or 40 layers of these models, which are all alike, as many as let two correct bfloat16 implementations be told from a
# wrong one: the logits of 12 layers move by 1.3 % when the order of the products' sums changes, those of 36 by 2.3 %.
LAYERS = 12
# layer sizes: width, query heads, key/value heads, feed-forward width (all heads are of 128, but for the tiny models)
SIZES = {"1b": (2048, 16, 4, 6144), "4b": (2560, 20, 4, 9728), "8b": (4096, 32, 8, 12288), "14b": (5120, 40, 8, 17408)}
# layers, width, query heads, key/value heads, head size, feed-forward width, vocabulary, rope base, tied head, page size
TINY = {"tiny-a": (2, 64, 4, 2, 16, 128, 256, 1e4, True, 16), "tiny-b": (3, 96, 8, 2, 32, 224, 320, 1e6, False, 8)}


# ------------------------------------------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------------------------------------------
def steps_case(size, *, design="qwen3", dtype="bfloat16", layers=LAYERS, vocab=151936, decoding=0, context=0, spread=0.0, prompts=0,
               prompt=0, past=0, steps=1):
    """``decoding`` requests bring one token a step for ``steps`` steps; their contexts go down from ``context`` tokens by the share
    ``spread``.  ``prompts`` requests bring a portion of ``prompt`` tokens each in the first step, ``past`` tokens already cached."""
    return {"kind": "steps", "design": design, "size": size, "dtype": dtype, "layers": layers, "vocab": vocab, "decoding": decoding,
            "context": context, "spread": spread, "prompts": prompts, "prompt": prompt, "past": past, "steps": steps}


def generate_case(size, prompts, longest, new_tokens):
    return {"kind": "generate", "design": "qwen3", "size": size, "dtype": "float32", "prompts": prompts, "longest": longest,
            "new_tokens": new_tokens}


def listed():
    cases = {
        # one user's stream of tokens: every weight is read for one token
        "decode-1": steps_case("8b", decoding=1, context=2048, steps=8),
        # a few users at once
        "decode-8": steps_case("8b", decoding=8, context=2048, steps=8),
        # a busy server: the cache's bytes pass the weights'
        "decode-64": steps_case("8b", decoding=64, context=2048, steps=4),
        # requests of all ages: an odd batch, contexts from 450 to 9,000 tokens
        "decode-ragged": steps_case("8b", decoding=21, context=9000, spread=0.95, steps=4),
        # a long prompt in one step
        "prefill-2048": steps_case("8b", prompts=1, prompt=2048),
        # a short question, an odd number of tokens
        "prefill-203": steps_case("8b", prompts=1, prompt=203),
        # a portion of a long document whose first 6,000 tokens are cached
        "prefill-portion": steps_case("8b", prompts=1, prompt=1733, past=6000),
        # continuous batching: a portion of a prompt beside requests that decode
        "mixed-14b": steps_case("14b", decoding=24, context=3072, spread=0.9, prompts=1, prompt=997),
        # the float32 path: what results are checked against
        "float32-prefill": steps_case("1b", dtype="float32", layers=4, vocab=32768, prompts=1, prompt=301),
        "float32-decode": steps_case("1b", dtype="float32", layers=4, vocab=32768, decoding=4, context=700, spread=0.5, steps=4),
        # recurrent mixers (delta rule, retention) beside softmax attention
        "recurrent-prefill": steps_case("8b", design="pugozen", layers=4, vocab=32768, prompts=1, prompt=1500),
        # the smallest calls: three short prompts to a model that fits the caches
        "generate-tiny": generate_case("tiny-a", 3, 17, 8),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "portion", "mixed", "float32", "recurrent", "generate"])
    if kind == "decode":
        batch = log_uniform(rng, 1, 64)
        context = log_uniform(rng, 100, min(9000, 131072 // batch))
        return steps_case("8b", decoding=batch, context=context, spread=rng.choice([0.0, 0.5, 0.95]), steps=4 if batch > 16 else 8)
    if kind == "prefill":
        prompts = rng.choice([1, 1, 1, 2, 3])
        return steps_case("8b", prompts=prompts, prompt=log_uniform(rng, 130, 2048 // prompts))
    if kind == "portion":
        return steps_case("8b", prompts=1, prompt=log_uniform(rng, 130, 1733), past=log_uniform(rng, 300, 6000))
    if kind == "mixed":
        return steps_case("14b", decoding=log_uniform(rng, 2, 24), context=log_uniform(rng, 130, 3072), spread=0.9,
                          prompts=1, prompt=log_uniform(rng, 130, 997))
    if kind == "float32":
        if rng.random() < 0.5:
            return steps_case("1b", dtype="float32", layers=4, vocab=32768, prompts=1, prompt=log_uniform(rng, 20, 301))
        return steps_case("1b", dtype="float32", layers=4, vocab=32768, decoding=log_uniform(rng, 1, 4), context=log_uniform(rng, 50, 700),
                          spread=0.5, steps=4)
    if kind == "recurrent":
        if rng.random() < 0.5:
            return steps_case("8b", design="pugozen", layers=4, vocab=32768, prompts=1, prompt=log_uniform(rng, 130, 1500))
        return steps_case(rng.choice(["1b", "8b"]), design="pugozen", layers=4, vocab=32768, decoding=log_uniform(rng, 1, 32),
                          context=log_uniform(rng, 100, 2048), spread=0.5, steps=4)
    return generate_case(rng.choice(["tiny-a", "tiny-b"]), rng.randint(1, 4), log_uniform(rng, 8, 40), rng.randint(4, 12))


def requests_of(case):
    """(tokens cached, tokens brought over all steps) of every request, in the order in which they are opened."""
    n = case["decoding"]
    share = [1.0 - case["spread"] * i / max(n - 1, 1) for i in range(n)]
    return ([(max(1, int(case["context"] * s)), case["steps"]) for s in share]
            + [(case["past"], case["prompt"])] * case["prompts"])


def prompt_lengths(case):
    return [max(1, round(case["longest"] * (i + 1) / case["prompts"])) for i in range(case["prompts"])]


def page_size(case):
    return TINY[case["size"]][-1] if case["size"] in TINY else 64


# ------------------------------------------------------------------------------------------------------------------------------
# configuration and weights
# ------------------------------------------------------------------------------------------------------------------------------
def config_of(case):
    """config.json as a dict."""
    if case["design"] == "qwen3":
        if case["size"] in TINY:
            layers, width, heads, kv, dim, ff, vocab, theta, tied, _ = TINY[case["size"]]
        else:
            (width, heads, kv, ff), layers, vocab = SIZES[case["size"]], case["layers"], case["vocab"]
            dim, theta, tied = 128, 1e6, False
        return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": layers, "hidden_size": width,
                "num_attention_heads": heads, "num_key_value_heads": kv, "head_dim": dim, "intermediate_size": ff,
                "vocab_size": vocab, "rope_theta": theta, "rms_norm_eps": 1e-6, "tie_word_embeddings": tied,
                "max_position_embeddings": 40960}
    width, heads, kv, ff = SIZES[case["size"]]
    n, mlp = width // 128, {"kind": "dense", "ff": ff}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": n, "kv_heads": n // 2, "dim": 128, "vdim": 128, "conv": 4}}
    pair = {"type": "parallel", "mlp": mlp,
            "mixer": {"left": {"heads": heads, "kv_heads": kv, "dim": 128, "vdim": 128, "scale": 128 ** -0.5,
                               "rot": {"dims": 32, "base": 1e6}},
                      "right": {"heads": n, "kv_heads": n, "dim": 128, "vdim": 128, "conv": 3, "a_rank": 64, "g_rank": 64},
                      "left_scale": 0.7, "right_scale": 0.6}}
    retention = {"type": "retention", "mlp": mlp,
                 "mixer": {"heads": n, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** (-5 - 6 * j // n) for j in range(n)],
                           "rot": {"dims": 128, "base": 1e6}}}
    kinds = (delta, pair, pair, retention)
    return {"architecture": "Pugozen", "vocab": case["vocab"], "width": width, "layers": [kinds[i % 4] for i in range(case["layers"])],
            "norm": {"eps": 1e-6}, "embedding": {"scale": float(width) ** 0.5}, "max_position_embeddings": 8192}


def tensors_of(cfg):
    """name -> (shape, mean, standard deviation, kept in float32)."""
    out = {}

    def matrix(name, *shape, std=0.02):
        out[name] = (shape, 0.0, std, False)

    def vector(name, *shape, mean=0.0, std=0.1):
        out[name] = (shape, mean, std, True)

    if "layers" not in cfg:
        W, d, ff, V = cfg["hidden_size"], cfg["head_dim"], cfg["intermediate_size"], cfg["vocab_size"]
        q, kv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
        matrix("model.embed_tokens.weight", V, W)
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}"
            vector(f"{p}.input_layernorm.weight", W, mean=1.0)
            vector(f"{p}.post_attention_layernorm.weight", W, mean=1.0)
            for n, rows, cols in (("q", q, W), ("k", kv, W), ("v", kv, W), ("o", W, q)):
                matrix(f"{p}.self_attn.{n}_proj.weight", rows, cols)
            for n in ("q", "k"):
                vector(f"{p}.self_attn.{n}_norm.weight", d, mean=1.0)
            for n, rows, cols in (("gate", ff, W), ("up", ff, W), ("down", W, ff)):
                matrix(f"{p}.mlp.{n}_proj.weight", rows, cols)
        vector("model.norm.weight", W, mean=1.0)
        if not cfg["tie_word_embeddings"]:
            matrix("lm_head.weight", V, W)
        return out
    W, V = cfg["width"], cfg["vocab"]
    matrix("embed", V, W)

    def recurrent_paths(p, m, per_channel):
        H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
        for n, rows in (("q", G * d), ("k", G * d), ("v", H * dv)):
            matrix(f"{p}.{n}", rows, W)
            vector(f"{p}.{n}.conv", rows, m["conv"], std=0.5)
        matrix(f"{p}.b", H, W)
        vector(f"{p}.A_log", H, std=0.5)
        vector(f"{p}.norm", dv, mean=1.0)
        vector(f"{p}.dt_bias", H * d if per_channel else H, std=0.05)
        if per_channel:
            for n, rank, rows in (("a", m["a_rank"], H * d), ("g", m["g_rank"], H * dv)):
                matrix(f"{p}.{n}1", rank, W)
                matrix(f"{p}.{n}2", rows, rank, std=0.3)
        else:
            matrix(f"{p}.a", H, W)
            matrix(f"{p}.g", H * dv, W)
        matrix(f"{p}.o", W, H * dv)

    for i, layer in enumerate(cfg["layers"]):
        p, m = f"l{i}.mix", layer["mixer"]
        vector(f"l{i}.norm1", W, mean=1.0)
        if layer["type"] == "delta":
            recurrent_paths(p, m, per_channel=False)
        elif layer["type"] == "retention":
            for n, size in (("q", m["dim"]), ("k", m["dim"]), ("v", m["vdim"]), ("g", m["vdim"])):
                matrix(f"{p}.{n}", m["heads"] * size, W)
            matrix(f"{p}.o", W, m["heads"] * m["vdim"])
        else:
            left = m["left"]
            matrix(f"{p}.left.q", left["heads"] * left["dim"], W)
            matrix(f"{p}.left.k", left["kv_heads"] * left["dim"], W)
            matrix(f"{p}.left.o", W, left["heads"] * left["dim"])
            for n in ("q", "k"):
                vector(f"{p}.left.{n}.norm", left["dim"], mean=1.0)
            vector(f"{p}.left.temp", left["heads"], mean=1.0, std=0.2)
            vector(f"{p}.left.sink", left["heads"], std=1.0)
            recurrent_paths(f"{p}.right", m["right"], per_channel=True)
        matrix(f"l{i}.mlp.up", layer["mlp"]["ff"], W)
        matrix(f"l{i}.mlp.down", W, layer["mlp"]["ff"])
    vector("final.norm", W, mean=1.0)
    matrix("head", V, W)
    return out


def generator(seed, *what):
    """A generator of its own for every tensor, so that each can be made alone."""
    return torch.Generator(device=DEVICE).manual_seed(zlib.crc32(repr((int(seed),) + what).encode()))


def weights(cfg, seed):
    """A function name -> tensor, as a checkpoint would hold it: matrices in bfloat16, vectors in float32."""
    table = tensors_of(cfg)

    def get(name):
        shape, mean, std, wide = table[name]
        t = torch.empty(shape, dtype=torch.float32 if wide else torch.bfloat16, device=DEVICE)
        return t.normal_(mean, std, generator=generator(seed, name))

    return get


def token_ids(case, seed):
    """The token ids that every request brings."""
    vocab = TINY[case["size"]][6] if case["size"] in TINY else case["vocab"]
    if case["kind"] == "generate":
        counts = prompt_lengths(case)
    else:
        counts = [n for _, n in requests_of(case)]
    g = generator(seed, "tokens")
    return [torch.randint(0, vocab, (n,), generator=g, device=DEVICE).tolist() for n in counts]


def fill_pool(pool, seed, layer, which):
    return pool.normal_(0.0, 1.0, generator=generator(seed, "cache", layer, which))


# ------------------------------------------------------------------------------------------------------------------------------
# what a user's program holds, and one pass
# ------------------------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    """The model with its weights, the cache with the requests' contexts, decode steps captured as CUDA graphs (as a server has them
    after its first step)."""
    from carbon_engine_b200 import models  # noqa: F401  (registers the architectures)
    from carbon_engine_b200.config.registry import resolve_architecture
    cfg = config_of(case)
    arch = resolve_architecture(cfg)
    config = arch.parse_config(cfg)
    get, tokens = weights(cfg, seed), token_ids(case, seed)
    if case["kind"] == "generate":
        from carbon_engine_b200.engine.engine import Engine
        from carbon_engine_b200.sampling.params import SamplingParams
        engine = Engine(config=config, dtype=case["dtype"], dummy_weight=True, kv_tokens=1024, page_size=page_size(case),
                        max_seq_len=128, max_running_requests=4, max_prefill_tokens=256, cuda_graphs=True)
        engine.model.load_weights(get, engine.device, engine.dtype)
        state = SimpleNamespace(kind="generate", engine=engine, prompts=tokens,
                                params=SamplingParams(max_tokens=case["new_tokens"], ignore_eos=True))
        run(state)
        return state
    from carbon_engine_b200.cache.storage import CacheStorage
    from carbon_engine_b200.engine.batch import StepEntry
    from carbon_engine_b200.engine.engine import parse_dtype
    from carbon_engine_b200.engine.runner import ModelRunner
    requests = requests_of(case)
    longest = max(past + n for past, n in requests)
    ps = page_size(case)
    dtype, device = parse_dtype(case["dtype"]), torch.device(DEVICE, torch.cuda.current_device())
    model = arch.build_model(config, longest)
    model.load_weights(get, device, dtype)
    storage = CacheStorage(model, dtype, device, ps, sum(-(-(past + n) // ps) for past, n in requests), len(requests), longest)
    for i, call in enumerate(model.schedule):
        view = storage.view(call)
        if view.kind == "paged" and any(past for past, _ in requests):
            fill_pool(view.k_pool, seed, i, "keys")
            fill_pool(view.v_pool, seed, i, "values")
    most = case["decoding"] + case["prompts"] * case["prompt"]
    runner = ModelRunner(model, storage, max(most, 64))
    runner.enable_graphs()
    n = case["decoding"]
    steps = [[StepEntry(r, [tokens[r][t]], [0]) for r in range(n)] for t in range(case["steps"])] if n else [[]]
    steps[0] = steps[0] + [StepEntry(r, tokens[r], [len(tokens[r]) - 1]) for r in range(n, len(requests))]
    views = [storage.view(call) for call in model.schedule[-CACHES_RETURNED:]]
    caches = [{k: v for k, v in {"keys": w.k_pool, "values": w.v_pool, "state": w.state, **(w.extra or {})}.items() if v is not None}
              for w in views]
    state = SimpleNamespace(kind="steps", runner=runner, requests=requests, steps=steps, caches=caches)
    run(state)
    return state


def run(state):
    if state.kind == "generate":
        outs = state.engine.generate(state.prompts, state.params)
        pools = [t for v in state.engine.storage.paged_views() for t in (v.k_pool, v.v_pool)]
        return {"tokens": [torch.tensor(o.token_ids) for o in outs], "caches": pools}
    runner, manager = state.runner, state.runner.storage.manager
    for r, (past, brought) in enumerate(state.requests):
        runner.open_request(r)
        manager.reserve(r, past + brought)        # (a request's pages for its whole life)
        manager.commit(r, past)
    for entries in state.steps:
        logits = runner.step(entries)
    for r in reversed(range(len(state.requests))):    # (slots are given out again last in, first out)
        runner.close_request(r)
    return {"logits": logits, "caches": state.caches}


# ------------------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------------------------
def work(case):
    """Every step reads every weight once (no cache holds them from one step to the next, but for the tiny models) and its requests'
    cached rows; a mixer's state is read and written once."""
    cfg = config_of(case)
    table = tensors_of(cfg)
    el = 4 if case["dtype"] == "float32" else 2
    matrices = {n: s[0] * s[1] for n, (s, _, _, wide) in table.items() if not wide and "embed" not in n}
    tied = cfg.get("tie_word_embeddings", False)
    if "layers" in cfg:
        vocab, width = cfg["vocab"], cfg["width"]
        head = matrices.pop("head")
        kinds = [layer["type"] for layer in cfg["layers"]]
        mixers = [layer["mixer"]["left"] for layer in cfg["layers"] if layer["type"] == "parallel"]
        score, row = (sum(m["heads"] * m["dim"] for m in mixers), sum(2 * m["kv_heads"] * m["dim"] for m in mixers))
        state = len(kinds) * width * 128
    else:
        vocab, width = cfg["vocab_size"], cfg["hidden_size"]
        head = vocab * width if tied else matrices.pop("lm_head.weight")
        layers = cfg["num_hidden_layers"]
        score, row = layers * cfg["num_attention_heads"] * cfg["head_dim"], layers * 2 * cfg["num_key_value_heads"] * cfg["head_dim"]
        state = 0
    body = sum(matrices.values())

    def step(portions):
        """``portions``: (tokens cached, tokens brought) of a step's requests, one logits row each."""
        tokens, rows = sum(n for _, n in portions), len(portions)
        seen = sum(n * past + n * (n + 1) // 2 for past, n in portions)
        return (el * (body + head + tokens * width + row * sum(past + 2 * n for past, n in portions)) + 4 * rows * (vocab + 2 * state),
                2 * tokens * body + 2 * rows * head + 4 * score * seen + 8 * tokens * state)

    if case["kind"] == "generate":
        lens = prompt_lengths(case)
        done = [step([(0, n) for n in lens])] + [step([(n + t, 1) for n in lens]) for t in range(case["new_tokens"] - 1)]
        # the weights stay in the caches of the chip over the steps: they are read once
        nbytes = sum(b for b, _ in done) - el * (body + head) * (len(done) - 1)
    else:
        requests, n = requests_of(case), case["decoding"]
        done = [step([(past + t, 1) for past, _ in requests[:n]] + (requests[n:] if t == 0 else [])) for t in range(case["steps"])]
        nbytes = sum(b for b, _ in done)
    return {"bytes": nbytes, "flops": sum(f for _, f in done)}


def tolerance(case):
    """float32: four times the error against ``exact``.  bfloat16: the outputs move by 0.013 when the order of the products' sums
    changes (other tiles, splits and attention kernels), and lie as far from ``exact`` as the same steps rounded elsewhere."""
    return {"rel": 2e-5 if case["dtype"] == "float32" else 3e-2}


# ------------------------------------------------------------------------------------------------------------------------------
# the same in float64
# ------------------------------------------------------------------------------------------------------------------------------
def rms(x, weight, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def silu(z):
    return z * torch.sigmoid(z)


def rotate(x, positions, dims, base):
    """x [T, heads, size]: element i of the first ``dims`` turns with element i + dims / 2."""
    half = dims // 2
    freq = base ** (-torch.arange(half, dtype=F64, device=x.device) * 2.0 / dims)
    ang = positions.to(F64)[:, None, None] * freq
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin(), x[..., dims:]], dim=-1)


def attend(q, k, v, past, scale, temp=None, sink=None):
    """q [n, H, d] at positions past .., k and v [past + n, G, d]."""
    n, H, d = q.shape
    G = k.shape[1]
    hidden = torch.arange(past + n, device=q.device)[None, :] > torch.arange(past, past + n, device=q.device)[:, None]
    out = torch.empty((n, H, v.shape[2]), dtype=F64, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T) * (scale if temp is None else scale * temp[h])
        s = s.masked_fill(hidden, float("-inf"))
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], dim=1)
        p = torch.softmax(s, dim=-1)
        out[:, h] = p[:, :past + n] @ v[:, g]
    return out


class Requests:
    """Where the rows of a pass's requests lie: in the joined tokens, in positions, in the cache's pages."""

    def __init__(self, requests, ps):
        self.ps, self.spans, at, page = ps, [], 0, 0
        for past, n in requests:
            self.spans.append((slice(at, at + n), past, n, page))
            at, page = at + n, page + -(-(past + n) // ps)
        self.pages = page
        self.positions = torch.cat([torch.arange(past, past + n, device=DEVICE) for past, n in requests])

    def flat(self, pool, span):
        """A request's rows of a pool [pages, heads, page size, size], in the order of their positions."""
        _, past, n, page = span
        rows = pool[page:page + -(-(past + n) // self.ps)].permute(0, 2, 1, 3)
        return rows.reshape(-1, *rows.shape[2:])

    def put(self, pool, span, rows):
        _, past, n, page = span
        at = torch.arange(past, past + n, device=DEVICE)
        pool[page + at // self.ps, :, at % self.ps] = rows


def cached(case, seed, where, layer, heads, size):
    """A layer's pools in float64, as they are before the pass."""
    shape, dtype = (where.pages, heads, where.ps, size), torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    pools = [torch.zeros(shape, dtype=dtype, device=DEVICE) for _ in range(2)]
    if any(past for _, past, _, _ in where.spans):
        for pool, which in zip(pools, ("keys", "values")):
            fill_pool(pool, seed, layer, which)
    return [pool.to(F64) for pool in pools]


def softmax_attention(q, k, v, pools, where, scale, temp=None, sink=None):
    """All requests of the pass over one layer's pools, which take the new rows."""
    out = torch.empty_like(q)
    for span in where.spans:
        rows, past, n, _ = span
        where.put(pools[0], span, k[rows])
        where.put(pools[1], span, v[rows])
        out[rows] = attend(q[rows], where.flat(pools[0], span)[:past + n], where.flat(pools[1], span)[:past + n], past, scale, temp, sink)
    return out


def recurrent_walk(q, k, v, decay, beta, where):
    """S <- decay S; u = beta (v - S^T k), or v where there is no beta; S <- S + k u^T; o = S^T q, all heads at once, from zeros.
    q, k [T, H, d], v [T, H, dv], decay [T, H, d or 1], beta [T, H] or None."""
    out, states = torch.empty_like(v), []
    for rows, _, n, _ in where.spans:
        S = torch.zeros((q.shape[1], q.shape[2], v.shape[2]), dtype=F64, device=q.device)
        for t in range(rows.start, rows.stop):
            S = decay[t][:, :, None] * S
            u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            out[t] = torch.einsum("hkv,hk->hv", S, q[t])
        states.append(S)
    return out, torch.stack(states)


def short_convolution(x, taps, where):
    y = torch.zeros_like(x)
    for rows, _, n, _ in where.spans:
        for j in range(min(taps.shape[1], n)):
            y[rows.start + j:rows.stop] += x[rows.start:rows.stop - j] * taps[:, taps.shape[1] - 1 - j]
    return silu(y)


def delta_rule(w, p, m, h, where, eps, per_channel):
    T, H, G, d, dv = h.shape[0], m["heads"], m["kv_heads"], m["dim"], m["vdim"]
    q, k, v = (short_convolution(h @ w(f"{p}.{n}").T, w(f"{p}.{n}.conv"), where) for n in ("q", "k", "v"))
    q, k = (x.reshape(T, G, d).repeat_interleave(H // G, dim=1) for x in (q, k))
    q, k = (x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    z = (h @ w(f"{p}.a1").T) @ w(f"{p}.a2").T if per_channel else h @ w(f"{p}.a").T
    g = torch.nn.functional.softplus(z + w(f"{p}.dt_bias")).reshape(T, H, -1)
    g = torch.exp(-torch.exp(w(f"{p}.A_log"))[None, :, None] * g)
    out, state = recurrent_walk(q * d ** -0.5, k, v.reshape(T, H, dv), g, torch.sigmoid(h @ w(f"{p}.b").T), where)
    out = rms(out, w(f"{p}.norm"), eps).reshape(T, H * dv)
    out = out * (torch.sigmoid((h @ w(f"{p}.g1").T) @ w(f"{p}.g2").T) if per_channel else silu(h @ w(f"{p}.g").T))
    return out @ w(f"{p}.o").T, state


def retention(w, p, m, h, where, eps):
    T, H, d, dv, rot = h.shape[0], m["heads"], m["dim"], m["vdim"], m["rot"]
    q, k = (rotate((h @ w(f"{p}.{n}").T).reshape(T, H, d), where.positions, rot["dims"], rot["base"]) for n in ("q", "k"))
    v = (h @ w(f"{p}.v").T).reshape(T, H, dv)
    decay = torch.tensor(m["decay"], dtype=F64, device=h.device)[None, :, None].expand(T, H, 1)
    out, state = recurrent_walk(q, k * d ** -0.5, v, decay, None, where)
    return (rms(out, None, eps).reshape(T, H * dv) * silu(h @ w(f"{p}.g").T)) @ w(f"{p}.o").T, state


def qwen3_layers(case, cfg, seed, w, x, where):
    eps, d = cfg["rms_norm_eps"], cfg["head_dim"]
    H, G, L = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["num_hidden_layers"]
    caches = []
    for i in range(L):
        p = f"model.layers.{i}"
        h = rms(x, w(f"{p}.input_layernorm.weight"), eps)
        q, k, v = ((h @ w(f"{p}.self_attn.{n}_proj.weight").T).reshape(len(h), heads, d) for n, heads in (("q", H), ("k", G), ("v", G)))
        q, k = (rotate(rms(y, w(f"{p}.self_attn.{n}_norm.weight"), eps), where.positions, d, cfg["rope_theta"]) for n, y in (("q", q), ("k", k)))
        pools = cached(case, seed, where, i, G, d)
        o = softmax_attention(q, k, v, pools, where, d ** -0.5)
        if i >= L - CACHES_RETURNED:
            caches.append({"keys": pools[0], "values": pools[1]})
        x = x + o.reshape(len(h), H * d) @ w(f"{p}.self_attn.o_proj.weight").T
        h = rms(x, w(f"{p}.post_attention_layernorm.weight"), eps)
        x = x + (silu(h @ w(f"{p}.mlp.gate_proj.weight").T) * (h @ w(f"{p}.mlp.up_proj.weight").T)) @ w(f"{p}.mlp.down_proj.weight").T
    return x, caches


def pugozen_layers(case, cfg, seed, w, x, where):
    eps, caches = cfg["norm"]["eps"], []
    for i, layer in enumerate(cfg["layers"]):
        p, m, cache = f"l{i}.mix", layer["mixer"], {}
        h = rms(x, w(f"l{i}.norm1"), eps)
        if layer["type"] == "delta":
            y, cache["state"] = delta_rule(w, p, m, h, where, eps, per_channel=False)
            cache["conv"] = None
        elif layer["type"] == "retention":
            y, cache["state"] = retention(w, p, m, h, where, eps)
        else:
            a = m["left"]
            q, v = ((h @ w(f"{p}.left.{n}").T).reshape(len(h), a[heads], a["dim"]) for n, heads in (("q", "heads"), ("k", "kv_heads")))
            q, k = (rotate(rms(y, w(f"{p}.left.{n}.norm"), eps), where.positions, a["rot"]["dims"], a["rot"]["base"])
                    for n, y in (("q", q), ("k", v)))
            pools = cached(case, seed, where, i, a["kv_heads"], a["dim"])
            left = softmax_attention(q, k, v, pools, where, a["scale"], w(f"{p}.left.temp"), w(f"{p}.left.sink"))
            right, state = delta_rule(w, f"{p}.right", m["right"], h, where, eps, per_channel=True)
            y = m["left_scale"] * (left.reshape(len(h), -1) @ w(f"{p}.left.o").T) + m["right_scale"] * right
            cache = {"keys": pools[0], "values": pools[1], "1.state": state, "1.conv": None}
        x = x + y + torch.relu(h @ w(f"l{i}.mlp.up").T) ** 2 @ w(f"l{i}.mlp.down").T
        caches.append(cache)
    return x, caches[-CACHES_RETURNED:]


def forward64(case, cfg, seed, tokens, requests):
    """(logits of every request's last token, caches) of requests that bring ``tokens`` on top of what they hold."""
    get, where = weights(cfg, seed), Requests(requests, page_size(case))
    w = lambda name: get(name).to(F64)
    ids = torch.tensor([t for row in tokens for t in row], device=DEVICE)
    last = [rows.stop - 1 for rows, _, _, _ in where.spans]
    if "layers" in cfg:
        x = get("embed")[ids].to(F64) * cfg["embedding"]["scale"]
        x, caches = pugozen_layers(case, cfg, seed, w, x, where)
        return rms(x[last], w("final.norm"), cfg["norm"]["eps"]) @ w("head").T, caches
    embed = get("model.embed_tokens.weight")
    x, caches = qwen3_layers(case, cfg, seed, w, embed[ids].to(F64), where)
    head = embed if cfg["tie_word_embeddings"] else get("lm_head.weight")
    return rms(x[last], w("model.norm.weight"), cfg["rms_norm_eps"]) @ head.to(F64).T, caches


@torch.no_grad()
def exact(case, seed):
    cfg, tokens = config_of(case), token_ids(case, seed)
    if case["kind"] == "generate":
        out = []
        for prompt in tokens:
            seq = list(prompt)
            for _ in range(case["new_tokens"]):
                seq.append(int(forward64(case, cfg, seed, [seq], [(0, len(seq))])[0].argmax()))
            out.append(torch.tensor(seq[len(prompt):]))
        # (which pages the engine gives which request is its own affair)
        return {"tokens": out, "caches": [None] * (2 * cfg["num_hidden_layers"])}
    logits, caches = forward64(case, cfg, seed, tokens, requests_of(case))
    return {"logits": logits, "caches": caches}
