"""The engine's measured work: steps of whole models through ``Engine`` and ``Sampler``, as a serving program runs them.

A case names a model shape and one kind of pass:

  decode     one more token for every request of a batch whose prompts are in the cache: the loop that generation spends
             its time in.  Requests move on by a position a pass and go back after ``SPAN`` passes.
  prompt     whole prompts of given total length, cut unevenly over the requests, the last row's logits wanted: the time to
             the first token.
  mixed      portions of prompts beside decoding requests in one step, as the scheduler packs them under load.
  generate   prompts, then decode steps to the end, then the requests leave: for models that carry a state from token to
             token, whose requests cannot go back by a few positions.

Every pass that ends in tokens samples them and reads them back, since the next step needs them; the ids that are fed are
fixed by the seed all the same, so that a tie between two logits cannot send two implementations different ways, and the
logits are what is returned.  Weights and tokens are made from the seed alone.
"""
from __future__ import annotations

import math
import zlib

import torch

from infinicore_infer_b200.config import MiniCPMConfig, SitelornConfig, VunelixConfig
from infinicore_infer_b200.engine import Engine, StepEntry
from infinicore_infer_b200.sampling import Sampler, SamplingParams
from infinicore_infer_b200.weights import WeightSource

DEVICE = "cuda:0"
SPAN = 64                     # decode positions that a request moves on by before it goes back
F64 = torch.float64

# The decoder's shapes: the three benchmark shapes and the small named configuration with grouped heads and pages of 8.
DECODERS = {
    "2b": dict(model_type="minicpm", num_hidden_layers=40, hidden_size=2304, num_attention_heads=36, num_key_value_heads=36,
               intermediate_size=5760, vocab_size=122753, max_position_embeddings=4096, rms_norm_eps=1e-5, rope_theta=10000.0,
               scale_emb=12, scale_depth=1.4, dim_model_base=256, tie_word_embeddings=True),
    "1b": dict(model_type="minicpm", num_hidden_layers=52, hidden_size=1536, num_attention_heads=24, num_key_value_heads=8,
               intermediate_size=3840, vocab_size=73440, max_position_embeddings=4096, rms_norm_eps=1e-5, rope_theta=10000.0,
               scale_emb=12, scale_depth=1.4, dim_model_base=256, tie_word_embeddings=True),
    "8b": dict(model_type="fm9g", num_hidden_layers=32, hidden_size=4096, num_attention_heads=32, num_key_value_heads=2,
               intermediate_size=16384, vocab_size=73448, max_position_embeddings=4096, rms_norm_eps=1e-5, rope_theta=10000.0,
               scale_emb=12, scale_depth=1.4, dim_model_base=256, tie_word_embeddings=False),
    "tiny": dict(model_type="fm9g", num_hidden_layers=3, hidden_size=96, num_attention_heads=3, num_key_value_heads=1,
                 intermediate_size=224, vocab_size=384, max_position_embeddings=96, rms_norm_eps=1e-6, rope_theta=1e6,
                 scale_emb=2.5, scale_depth=1.0, dim_model_base=48, tie_word_embeddings=False),
}
# The two layer-list designs at the benchmark's smaller real size: width, feed-forward, heads, key/value heads, head, vocabulary.
WIDTH, FF, HEADS, KV_HEADS, DIM, VOCAB = 2048, 5632, 16, 4, 128, 32000


def sitelorn():
    """Constant and projected decays beside windowed attention, one layer on another's keys."""
    mlp = {"kind": "dense", "ff": FF}
    light = {"type": "lightning", "mlp": mlp, "mixer": {"heads": HEADS, "dim": DIM, "vdim": DIM,
             "decay": [1.0 - 2.0 ** (-5 - 3 * h / (HEADS - 1)) for h in range(HEADS)]}}
    gla = {"type": "gla", "mlp": mlp, "mixer": {"heads": HEADS, "dim": DIM, "vdim": DIM, "tau": 16.0, "rank": 16}}
    att = {"heads": HEADS, "kv_heads": KV_HEADS, "dim": DIM, "vdim": DIM, "conv": 4, "rot": {"dims": DIM // 2, "base": 5e5},
           "scale": DIM ** -0.5, "mask": {"size": 1024}}
    layers = [light, gla, {"type": "attention", "mixer": att, "mlp": mlp}, light, light, gla,
              {"type": "attention", "mixer": dict(att, kv_from=2), "mlp": mlp}, light]
    return {"architecture": "Sitelorn", "embedding": {"scale": 1.0}, "norm": {"eps": 1e-5}, "vocab": VOCAB, "width": WIDTH,
            "layers": layers}


def vunelix():
    """Latent attention and selective scans; a dense feed-forward, then routed experts with a shared one; a layer that runs twice."""
    att = {"heads": HEADS, "dim": DIM, "rot_dim": DIM // 2, "vdim": DIM, "kv_rank": 4 * DIM, "scale": (1.5 * DIM) ** -0.5,
           "rot": {"base": 1e4, "dims": DIM // 2, "scaling": {"factor": 4.0, "original": 1024, "fast": 32.0, "slow": 1.0}}}
    ssm = {"inner": 2 * WIDTH, "state": 16, "dt_rank": WIDTH // 16, "conv": 4}
    moe = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": FF // 4}, "shared": {"ff": FF // 4}}
    lat = lambda mlp: {"type": "latent_attention", "mixer": att, "mlp": mlp}
    scan = {"type": "mamba1", "mixer": ssm, "mlp": moe}
    return {"architecture": "Vunelix", "norm": {"eps": 1e-5}, "vocab": VOCAB, "width": WIDTH, "logit_softcap": 30.0,
            "loop": {"start": 1, "stop": 2, "times": 2},
            "layers": [lat({"kind": "dense", "ff": FF}), lat(moe), scan, lat(moe), lat(moe), scan, lat(moe)]}


# ---- the cases ----------------------------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a small model in 32 bits, one prompt portion beside three decoding requests, as replays and checks run
        {"name": "tiny-f32-mixed", "kind": "mixed", "shape": "tiny", "dtype": "float32", "rows": 3, "context": 31, "portions": 1, "portion": 9, "held": 18},
        # one user's chat: a single request, a short history
        {"name": "2b-decode-b1", "kind": "decode", "shape": "2b", "dtype": "bfloat16", "requests": 1, "context": 512, "ragged": False},
        # the headline: eight requests at the full context
        {"name": "2b-decode-b8", "kind": "decode", "shape": "2b", "dtype": "bfloat16", "requests": 8, "context": 4031, "ragged": False},
        # a loaded server with short histories
        {"name": "2b-decode-b64", "kind": "decode", "shape": "2b", "dtype": "bfloat16", "requests": 64, "context": 512, "ragged": False},
        # the largest model under load: histories of unlike lengths, grouped heads 16:1
        {"name": "8b-decode-b32", "kind": "decode", "shape": "8b", "dtype": "bfloat16", "requests": 32, "context": 1150, "ragged": True},
        # time to the first token of a long prompt
        {"name": "2b-prompt-2048", "kind": "prompt", "shape": "2b", "dtype": "bfloat16", "requests": 1, "tokens": 2048},
        # the largest step: several prompts of odd lengths at once through the largest model
        {"name": "8b-prompts-5003", "kind": "prompt", "shape": "8b", "dtype": "bfloat16", "requests": 3, "tokens": 5003},
        # what the scheduler packs while requests come and go: two portions of 256 beside 20 decoding requests
        {"name": "1b-mixed-532", "kind": "mixed", "shape": "1b", "dtype": "bfloat16", "rows": 20, "context": 700, "portions": 2, "portion": 256, "held": 256},
        # the true 32-bit path at a real size: an ordinary prompt
        {"name": "1b-f32-prompt-301", "kind": "prompt", "shape": "1b", "dtype": "float32", "requests": 1, "tokens": 301},
        # decaying recurrences beside windowed attention: a long prompt
        {"name": "sitelorn-prompt-2048", "kind": "prompt", "shape": "sitelorn", "dtype": "bfloat16", "requests": 1, "tokens": 2048},
        # latent attention, selective scans and routed experts: a long prompt
        {"name": "vunelix-prompt-2048", "kind": "prompt", "shape": "vunelix", "dtype": "bfloat16", "requests": 1, "tokens": 2048},
        # the same, eight requests generated to their end
        {"name": "vunelix-generate-b8", "kind": "generate", "shape": "vunelix", "dtype": "bfloat16", "requests": 8, "tokens": 1500, "new": 24},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prompt", "prompt", "mixed", "generate"])
    if kind == "decode":
        shape = rng.choice(["1b", "2b", "8b"])
        requests = _spread(rng, 1, 64)
        context = _spread(rng, 64, min(4000, (26000 if shape == "8b" else 33000) // requests))
        return {"kind": kind, "shape": shape, "dtype": "bfloat16", "requests": requests, "context": context, "ragged": rng.random() < 0.7}
    if kind == "prompt":
        shape = rng.choice(["1b", "2b", "8b", "sitelorn", "vunelix", "tiny"])
        if shape == "tiny":
            return {"kind": kind, "shape": shape, "dtype": "float32", "requests": rng.randint(1, 4), "tokens": rng.randint(9, 90)}
        if shape == "1b" and rng.random() < 0.4:
            return {"kind": kind, "shape": shape, "dtype": "float32", "requests": rng.randint(1, 3), "tokens": _spread(rng, 24, 400)}
        return {"kind": kind, "shape": shape, "dtype": "bfloat16", "requests": rng.randint(1, 4), "tokens": _spread(rng, 40, 2048 if shape in ("sitelorn", "vunelix") else 4000)}
    if kind == "mixed":
        if rng.random() < 0.2:
            return {"kind": kind, "shape": "tiny", "dtype": "float32", "rows": rng.randint(1, 3), "context": rng.randint(8, 40), "portions": 1, "portion": rng.randint(2, 9), "held": rng.randint(0, 40)}
        return {"kind": kind, "shape": rng.choice(["1b", "2b"]), "dtype": "bfloat16", "rows": _spread(rng, 1, 40), "context": _spread(rng, 32, 1000),
                "portions": rng.randint(1, 3), "portion": _spread(rng, 16, 512), "held": rng.choice([0, rng.randint(1, 1000)])}
    return {"kind": kind, "shape": rng.choice(["sitelorn", "vunelix"]), "dtype": "bfloat16", "requests": _spread(rng, 1, 16), "tokens": _spread(rng, 200, 1600), "new": rng.randint(4, 24)}


def _cut(total, parts):
    """``total`` in ``parts`` uneven shares (weights 1, 2, 3, ...), each at least 1."""
    weights = [i + 1 for i in range(parts)]
    cut = [max(1, total * w // sum(weights)) for w in weights]
    cut[-1] += total - sum(cut)
    return cut


def _lengths(case):
    """How many tokens each request holds before the pass, and how many it is given by it."""
    if case["kind"] == "decode":
        n, c = case["requests"], case["context"]
        held = [max(1, c - (i * c // (2 * n) if case["ragged"] else 0)) for i in range(n)]
        return held, [1] * n
    if case["kind"] == "mixed":
        return [case["context"] + i for i in range(case["rows"])] + [case["held"]] * case["portions"], [1] * case["rows"] + [case["portion"]] * case["portions"]
    cut = _cut(case["tokens"], case["requests"])
    return [0] * len(cut), cut


# ---- weights and tokens from the seed ------------------------------------------------------------------------------------
def _config(shape):
    if shape in DECODERS:
        return dict(DECODERS[shape])
    return sitelorn() if shape == "sitelorn" else vunelix()


def _tensors(shape):
    """{checkpoint name: (shape, how it is drawn)}; matrices are held in 16 bits (m), vectors in 32 (v)."""
    c, t = _config(shape), {}
    if shape in DECODERS:
        d, h, ff, v = c["hidden_size"], c["num_attention_heads"], c["intermediate_size"], c["vocab_size"]
        dh = d // h
        kv = c["num_key_value_heads"] * dh
        t["model.embed_tokens.weight"] = ((v, d), "m0.02")
        if not c["tie_word_embeddings"]:
            t["lm_head.weight"] = ((v, d), "m0.02")
        t["model.norm.weight"] = ((d,), "one")
        for i in range(c["num_hidden_layers"]):
            p = f"model.layers.{i}."
            t[p + "input_layernorm.weight"] = t[p + "post_attention_layernorm.weight"] = ((d,), "one")
            for name, rows, cols in (("self_attn.q_proj", d, d), ("self_attn.k_proj", kv, d), ("self_attn.v_proj", kv, d), ("self_attn.o_proj", d, d),
                                     ("mlp.gate_proj", ff, d), ("mlp.up_proj", ff, d), ("mlp.down_proj", d, ff)):
                t[f"{p}{name}.weight"] = ((rows, cols), "m0.02")
        return t
    d, v = c["width"], c["vocab"]

    def unit(p, ff):
        for name, s in (("gate", (ff, d)), ("up", (ff, d)), ("down", (d, ff))):
            t[p + name] = (s, "m0.02")

    t["embed"], t["final.norm"] = ((v, d), "m0.02" if shape == "sitelorn" else "clusters"), ((d,), "one")
    if shape == "sitelorn":
        t["head"], t["final.norm.b"] = ((v, d), "m0.02"), ((d,), "zero")
    else:
        t["loop.in"], t["loop.step"] = ((d, 2 * d), "mix"), ((c["loop"]["times"], d), "zero")
    for i, layer in enumerate(c["layers"]):
        p, m, mlp = f"l{i}.", layer["mixer"], layer["mlp"]
        x = p + "mix."
        if shape == "sitelorn":
            for n in ("norm1", "norm2"):
                t[p + n], t[p + n + ".b"] = ((d,), "one"), ((d,), "zero")
            h, dk, dv = m["heads"], m["dim"], m["vdim"]
            if layer["type"] == "attention":
                g = m["kv_heads"]
                for n, rows in (("q", h * dk),) + ((("k", g * dk), ("v", g * dv)) if m.get("kv_from") is None else ()):
                    t[x + n], t[f"{x}{n}.conv"] = ((rows, d), "m0.02"), ((rows, m["conv"]), "taps")
                    if n != "v":
                        t[f"{x}{n}.norm"] = ((rows,), "one")
                t[x + "g"] = ((h, d), "m0.02")
            else:
                for n, rows in (("q", h * dk), ("k", h * dk), ("v", h * dv), ("g", h * dv)):
                    t[x + n] = ((rows, d), "m0.02")
                t[x + "norm"] = ((h * dv if layer["type"] == "lightning" else dv,), "one")
                if layer["type"] == "gla":
                    t[x + "a1"], t[x + "a2"], t[x + "a2.b"] = ((m["rank"], d), "m0.02"), ((h * dk, m["rank"]), "m0.3"), ((h * dk,), "zero")
            t[x + "o"] = ((d, h * dv), "m0.02")
            unit(p + "mlp.", mlp["ff"])
            continue
        for n in ("norm1", "norm2"):
            t[p + n], t[p + n + "b"] = ((d,), "one"), ((d,), "small")
        if layer["type"] == "latent_attention":
            h, dn, dr, dv, r = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            t[x + "q"], t[x + "dkv"], t[x + "dkv.norm"] = ((h * (dn + dr), d), "m0.02"), ((r + dr, d), "m0.02"), ((r,), "one")
            t[x + "uk"], t[x + "uv"] = ((h * dn, r), "m0.02"), ((h * dv, r), "m0.02")
            t[x + "g"], t[x + "o"] = ((h * dv, d), "m0.02"), ((d, h * dv), "m0.02")
        else:
            e, n, k = m["inner"], m["state"], m["dt_rank"]
            t[x + "in"], t[x + "conv"], t[x + "conv.b"] = ((2 * e, d), "m0.02"), ((e, m["conv"]), "taps"), ((e,), "zero")
            t[x + "x"], t[x + "dt"], t[x + "dt.b"] = ((k + 2 * n, e), "m0.02"), ((e, k), "m0.02"), ((e,), "step")
            t[x + "A_log"], t[x + "D"], t[x + "o"] = ((e, n), "log"), ((e,), "one"), ((d, e), "m0.02")
        if mlp["kind"] == "dense":
            unit(p + "mlp.", mlp["ff"])
        else:
            t[p + "mlp.router"] = ((mlp["router"]["experts"], d), "router")
            for j in range(mlp["router"]["experts"]):
                unit(f"{p}mlp.e{j}.", mlp["expert"]["ff"])
            unit(p + "mlp.shared.", mlp["shared"]["ff"])
    return t


def _gen(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))


def _centres(seed, size):
    """Eight directions that tokens gather around.  A trained router sends a row to its experts by a clear margin; a random one
    has ties that any rounding turns, and nothing could be compared behind them."""
    return torch.randn(8, size, generator=_gen(seed, "centres"), device=DEVICE)


def _make(seed, name, size, how):
    g = _gen(seed, name)
    if how[0] == "m" and how != "mix":
        return torch.empty(size, dtype=torch.bfloat16, device=DEVICE).normal_(0.0, float(how[1:]), generator=g)
    x = torch.randn(size, generator=g, device=DEVICE)
    if how == "clusters":
        own = torch.arange(size[0], device=DEVICE) % 8
        return (0.03 * x + 0.04 * _centres(seed, size[1])[own]).to(torch.bfloat16)
    if how == "mix":          # the stream and the embedding go on, each a little changed
        eye = torch.eye(size[0], device=DEVICE)
        return (torch.cat([0.8 * eye, 0.6 * eye], 1) + 0.1 * size[1] ** -0.5 * x).to(torch.bfloat16)
    if how == "router":       # cluster c prefers expert c, then expert 3 c + 1
        c = _centres(seed, size[1]) / size[1]
        first = torch.arange(8, device=DEVICE)
        w = 0.25 * size[1] ** -0.5 * x
        w[first] += 4.0 * c
        w.index_add_(0, (3 * first + 1) % 8, 2.4 * c)
        return w
    return {"one": 1.0 + 0.01 * x, "zero": 0.01 * x, "small": 0.05 * (1.0 + 0.1 * x), "taps": 0.5 * x, "step": -4.0 + x,
            "log": torch.arange(1, size[-1] + 1, device=DEVICE).log().expand(size) + 0.01 * x}[how].contiguous()


class SeededWeights(WeightSource):
    """Hands the engine's parts the tensors that the seed makes."""

    def __init__(self, shape, seed, dtype):
        super().__init__(dtype, DEVICE)
        self.seed, self.tensors = seed, _tensors(shape)

    def shapes(self):
        return {n: s for n, (s, _) in self.tensors.items()}

    def has(self, name):
        return name in self.tensors

    def get(self, name, role="matrix"):
        return _make(self.seed, name, *self.tensors[name]).to(torch.float32 if role == "vector" else self.compute_dtype)


def _tokens(case, seed, more):
    """Token ids of every request: what it holds, what the pass gives it, and ``more`` further ones."""
    c = _config(case["shape"])
    v = c.get("vocab_size") or c["vocab"]
    g = torch.Generator().manual_seed(seed * 7919 + 17)
    return [torch.randint(0, v, (h + n + more,), generator=g).tolist() for h, n in zip(*_lengths(case))]


# ---- the measured interface --------------------------------------------------------------------------------------------------
def prepare(case, seed):
    dtype = getattr(torch, case["dtype"])
    cfg = _config(case["shape"])
    held, given = _lengths(case)
    more = case.get("new", SPAN if case["kind"] == "decode" else 0)
    if case["shape"] in DECODERS:
        spec = MiniCPMConfig.from_dict(cfg).model_spec()
    else:
        spec = (SitelornConfig if case["shape"] == "sitelorn" else VunelixConfig).from_dict(cfg, max_tokens=4096).model_spec()
    page = 8 if case["shape"] == "tiny" else 16
    step_tokens = max(sum(given), 64 if case["shape"] == "tiny" else 4096)
    engine = Engine(spec, SeededWeights(case["shape"], seed, dtype), dtype=dtype, device=DEVICE, page_size=page, max_requests=max(2, len(held)),
                    cache_tokens=sum(h + g + more + 2 * page for h, g in zip(held, given)), max_step_tokens=step_tokens)
    tokens = _tokens(case, seed, more)
    greedy = case["kind"] != "mixed"         # the mixed steps draw their tokens, the others take the largest logit
    state = {"case": case, "engine": engine, "sampler": Sampler(DEVICE), "tokens": tokens, "held": held, "given": given, "turn": 0,
             "params": [SamplingParams(0.0 if greedy else 0.8, 0 if greedy else 50, 1.0 if greedy else 0.9, seed) for _ in held]}
    for i, h in enumerate(held):             # what the requests hold already
        if h:
            engine.begin(i)
        for at in range(0, h, step_tokens):
            engine.step([StepEntry(i, tokens[i][at: min(h, at + step_tokens)], [])])
    if case["kind"] == "decode":             # a program that decodes has done so before: the step's graph is there
        run(state)
        _back(state)
    torch.cuda.synchronize()
    return state


def _back(state):
    for i, h in enumerate(state["held"]):
        if h:
            state["engine"].cache.truncate(i, h)
        elif state["engine"].cache.is_live(i):
            state["engine"].end(i)
    state["turn"] = 0


def _sampled(state, logits, at):
    state["sampler"].sample(logits, state["params"], at)
    return logits


def run(state):
    case, engine, tokens, held, given = state["case"], state["engine"], state["tokens"], state["held"], state["given"]
    rows = range(len(held))
    if case["kind"] == "decode":
        if state["turn"] == SPAN:
            _back(state)
        t = state["turn"]
        state["turn"] = t + 1
        logits = engine.step([StepEntry(i, [tokens[i][held[i] + t]], [0]) for i in rows], stage_next=True)
        return _sampled(state, logits, [held[i] + t + 1 for i in rows])
    logits = engine.step([StepEntry(i, tokens[i][held[i]: held[i] + given[i]], [given[i] - 1]) for i in rows])
    _sampled(state, logits, [held[i] + given[i] for i in rows])
    seen = [logits]
    for t in range(case.get("new", 0)):
        logits = engine.step([StepEntry(i, [tokens[i][given[i] + t]], [0]) for i in rows], stage_next=True)
        seen.append(_sampled(state, logits, [given[i] + t + 1 for i in rows]))
    _back(state)
    return torch.stack(seen) if case["kind"] == "generate" else logits


def _per_token(shape):
    """(weights that a row's products read, among them those of the output matrix, multiply-adds of a row beside attention's)."""
    read = macs = 0
    c = _config(shape)
    for name, (size, _) in _tensors(shape).items():
        n = math.prod(size)
        times = 2 if shape == "vunelix" and name.startswith("l1.") else 1
        if len(size) == 1 or name.endswith(("embed", "embed_tokens.weight", "lm_head.weight", "head", "conv", "A_log", "loop.step")):
            continue
        read += n
        macs += times * n * (0.25 if ".mlp.e" in name else 1) * (2 if name == "loop.in" else 1)
    v, d = c.get("vocab_size") or c["vocab"], c.get("hidden_size") or c["width"]
    return read, macs, v * d


def work(case):
    """Every weight once, the cache and state that the pass reads and writes, ids in and logits out; all multiply-adds of the rows."""
    size = 4 if case["dtype"] == "float32" else 2
    c = _config(case["shape"])
    held, given = _lengths(case)
    read, macs, head = _per_token(case["shape"])
    new = case.get("new", 0)
    rows, wanted, steps = sum(given) + new * len(given), len(given) * (1 + new), 1 + new
    flops, nbytes = 2.0 * (rows * macs + wanted * head), steps * (read + head) * size + 4.0 * wanted * head / (c.get("hidden_size") or c["width"])
    spans = [(h, g) for h, g in zip(held, given)] + [(g + t, 1) for g in given for t in range(new)]
    for h, g in spans:
        pairs = g * h + g * (g + 1) / 2
        if case["shape"] in DECODERS:
            dh = c["hidden_size"] // c["num_attention_heads"]
            flops += c["num_hidden_layers"] * 4.0 * pairs * c["hidden_size"]
            nbytes += c["num_hidden_layers"] * 2.0 * (h + g) * c["num_key_value_heads"] * dh * size
            continue
        for i, layer in enumerate(c["layers"]):
            m, times = layer["mixer"], 2 if case["shape"] == "vunelix" and i == 1 else 1
            if layer["type"] == "attention":
                w = m["mask"]["size"]
                seen = sum(min(h + t + 1, w) for t in range(g))
                flops += 4.0 * seen * m["heads"] * m["dim"]
                nbytes += 2.0 * min(h + g, w + g) * m["kv_heads"] * m["dim"] * size
            elif layer["type"] == "latent_attention":
                flops += times * 2.0 * pairs * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
                nbytes += times * (h + g) * (m["kv_rank"] + m["rot_dim"]) * size
            elif layer["type"] == "mamba1":
                flops += 6.0 * g * m["inner"] * m["state"]
                nbytes += 8.0 * m["inner"] * m["state"]
            else:
                flops += 4.0 * g * m["heads"] * m["dim"] * m["vdim"]
                nbytes += 8.0 * m["heads"] * m["dim"] * m["vdim"]
    return {"bytes": float(nbytes), "flops": float(flops)}


def tolerance(case):
    """Four times what was measured against 64 bits, at most: 3.3e-6 in 32 bits; 0.0014 for Vunelix, whose logits come mostly from
    its embedding; 0.007 to 0.02 for the others, where 0.03 is as far as two runs may be apart (products cut along their inner
    dimension add up in another order each time)."""
    if case["dtype"] == "float32":
        return {"rel": 1.3e-5, "max": 2e-4}
    return {"rel": 0.006, "max": 0.1} if case["shape"] == "vunelix" else {"rel": 0.03, "max": 0.3}


# ---- the same in 64 bits ---------------------------------------------------------------------------------------------------
def _rms(x, w, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _layer_norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w + b


def _silu(x):
    return x * torch.sigmoid(x)


def _attend(q, k, v, scale, window=0, sink=False):
    """Causal attention of one request: q [T, H, d], k and v [T, G, .]; a few heads at a time."""
    T, H, _ = q.shape
    rep = H // k.shape[1]
    i, j = torch.arange(T, device=DEVICE)[:, None], torch.arange(T, device=DEVICE)[None, :]
    hidden = (j > i) | ((i - j >= window) if window else False)
    out = torch.empty(T, H, v.shape[-1], dtype=F64, device=DEVICE)
    for h in range(H):
        s = (q[:, h] @ k[:, h // rep].T * scale).masked_fill_(hidden, -math.inf)
        top = s.amax(-1, keepdim=True).clamp_(min=0.0 if sink else -math.inf)
        s = s.sub_(top).exp_()
        out[:, h] = (s @ v[:, h // rep]) / (s.sum(-1, keepdim=True) + (torch.exp(-top) if sink else 0.0))
    return out


def _apart(lens):
    """The rows of each request among the rows of all."""
    at = 0
    for n in lens:
        yield slice(at, at + n)
        at += n


def _decoder(case, W, x, lens):
    c = _config(case["shape"])
    d, H, G, eps = c["hidden_size"], c["num_attention_heads"], c["num_key_value_heads"], c["rms_norm_eps"]
    dh = d // H
    x = x * c["scale_emb"]
    res = c["scale_depth"] / math.sqrt(c["num_hidden_layers"])
    pos = torch.cat([torch.arange(n, device=DEVICE, dtype=F64) for n in lens])
    ang = pos[:, None, None] / float(c["rope_theta"]) ** (torch.arange(dh // 2, device=DEVICE, dtype=F64) / (dh // 2))
    cos, sin = ang.cos(), ang.sin()

    def turned(y):
        a, b = y[..., : dh // 2], y[..., dh // 2:]
        return torch.cat([a * cos - b * sin, a * sin + b * cos], -1)

    for i in range(c["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _rms(x, W(p + "input_layernorm.weight"), eps)
        q, k, v = (h @ W(f"{p}self_attn.{n}_proj.weight").T for n in "qkv")
        q, k, v = turned(q.view(-1, H, dh)), turned(k.view(-1, G, dh)), v.view(-1, G, dh)
        o = torch.cat([_attend(q[s], k[s], v[s], dh ** -0.5) for s in _apart(lens)])
        x = x + res * (o.reshape(-1, d) @ W(p + "self_attn.o_proj.weight").T)
        h = _rms(x, W(p + "post_attention_layernorm.weight"), eps)
        h = _silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)
        x = x + res * (h @ W(p + "mlp.down_proj.weight").T)
    return x, lambda y: _rms(y, W("model.norm.weight"), eps) * (d // c["dim_model_base"]) @ W("model.embed_tokens.weight" if c["tie_word_embeddings"] else "lm_head.weight").T


def _pairs(x, f, mag=1.0):
    """x [T, ..., n]: pairs (2 i, 2 i + 1), i < len(f), turned by position * f_i."""
    n = 2 * f.numel()
    ang = torch.arange(x.shape[0], device=DEVICE, dtype=F64).view(-1, *([1] * (x.dim() - 1))) * f
    c, s = ang.cos() * mag, ang.sin() * mag
    out = x.clone()
    out[..., 0:n:2], out[..., 1:n:2] = x[..., 0:n:2] * c - x[..., 1:n:2] * s, x[..., 1:n:2] * c + x[..., 0:n:2] * s
    return out


def _conv(u, taps):
    """y_t = sum_j taps[:, j] u_(t - J + 1 + j), zeros ahead of the start."""
    J = taps.shape[1]
    u = torch.cat([torch.zeros(J - 1, u.shape[1], dtype=F64, device=DEVICE), u])
    return sum(taps[:, j] * u[j: u.shape[0] - J + 1 + j] for j in range(J))


def _sitelorn(case, W, x, lens):
    c, kvs = sitelorn(), {}
    eps = c["norm"]["eps"]
    for i, layer in enumerate(c["layers"]):
        p, m = f"l{i}.", layer["mixer"]
        w = lambda n: W(f"{p}mix.{n}")
        H, dk, dv = m["heads"], m["dim"], m["vdim"]
        out = []
        for n, s in enumerate(_apart(lens)):
            h = x[s]
            T = h.shape[0]
            if layer["type"] == "attention":
                f = float(m["rot"]["base"]) ** (-2.0 * torch.arange(m["rot"]["dims"] // 2, device=DEVICE, dtype=F64) / m["rot"]["dims"])
                side = lambda name: _pairs(_rms(_conv(h @ w(name).T, w(name + ".conv")), w(name + ".norm"), eps).view(T, -1, dk), f)
                if m.get("kv_from") is None:
                    kvs[i, n] = side("k"), _conv(h @ w("v").T, w("v.conv")).view(T, -1, dv)
                k, v = kvs[m.get("kv_from", i), n]
                o = _attend(side("q"), k, v, m["scale"], m["mask"]["size"], sink=True) * torch.sigmoid(h @ w("g").T).unsqueeze(-1)
            else:
                light = layer["type"] == "lightning"
                act = _silu if light else (lambda y: y)
                q, k, v = (act(h @ w(name).T).view(T, H, -1) for name in "qkv")
                if light:
                    decay = torch.tensor(m["decay"], dtype=F64, device=DEVICE).view(1, H, 1).expand(T, H, dk)
                else:
                    q = q * dk ** -0.5
                    decay = torch.exp(torch.nn.functional.logsigmoid((h @ w("a1").T) @ w("a2").T + w("a2.b")) / m["tau"]).view(T, H, dk)
                S, o = torch.zeros(H, dk, dv, dtype=F64, device=DEVICE), torch.empty(T, H, dv, dtype=F64, device=DEVICE)
                for t in range(T):
                    S = torch.baddbmm(decay[t].unsqueeze(-1) * S, k[t].unsqueeze(-1), v[t].unsqueeze(-2))
                    o[t] = (q[t].unsqueeze(-2) @ S).squeeze(-2)
                if light:
                    o = _rms(o.reshape(T, -1), w("norm"), eps) * torch.sigmoid(h @ w("g").T)
                else:
                    o = _rms(o, w("norm"), eps).reshape(T, -1) * _silu(h @ w("g").T)
            out.append(o.reshape(T, -1) @ w("o").T)
        x = x + _layer_norm(torch.cat(out), W(p + "norm1"), W(p + "norm1.b"), eps)
        h = torch.nn.functional.gelu(x @ W(p + "mlp.gate").T, approximate="tanh") * (x @ W(p + "mlp.up").T)
        x = x + _layer_norm(h @ W(p + "mlp.down").T, W(p + "norm2"), W(p + "norm2.b"), eps)
    return x, lambda y: _layer_norm(y, W("final.norm"), W("final.norm.b"), eps) @ W("head").T


def _ramp(rot):
    """Frequencies whose long wavelengths are stretched, and the factor on cos and sin."""
    dims, base, s = rot["dims"], rot["base"], rot["scaling"]
    i = torch.arange(dims // 2, device=DEVICE, dtype=F64)
    f = float(base) ** (-2.0 * i / dims)
    where = lambda turns: dims * math.log(s["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
    lo, hi = max(math.floor(where(s["fast"])), 0), min(math.ceil(where(s["slow"])), dims - 1)
    r = ((i - lo) / max(hi - lo, 0.001)).clamp(0.0, 1.0)
    return f / s["factor"] * r + f * (1.0 - r), 0.1 * math.log(s["factor"]) + 1.0


def _vunelix(case, W, x, lens):
    c = vunelix()
    eps, x0 = c["norm"]["eps"], x
    unit = lambda h, p, act: (act(h @ W(p + "gate").T) * (h @ W(p + "up").T)) @ W(p + "down").T
    order = [(0, None), (1, 0), (1, 1)] + [(i, None) for i in range(2, len(c["layers"]))]
    for i, again in order:
        p, m, mlp = f"l{i}.", c["layers"][i]["mixer"], c["layers"][i]["mlp"]
        w = lambda n: W(f"{p}mix.{n}")
        if again is not None:
            x = torch.cat([x, x0], -1) @ W("loop.in").T + W("loop.step")[again]
        normed, out = _rms(x, W(p + "norm1"), eps), []
        for s in _apart(lens):
            h = normed[s]
            T = h.shape[0]
            if c["layers"][i]["type"] == "latent_attention":
                H, dn, R = m["heads"], m["dim"], m["kv_rank"]
                f, mag = _ramp(m["rot"])
                q, down = (h @ w("q").T).view(T, H, -1), h @ w("dkv").T
                latent = _rms(down[:, :R], w("dkv.norm"), eps)
                k = torch.cat([(latent @ w("uk").T).view(T, H, dn), _pairs(down[:, R:], f, mag).unsqueeze(1).expand(T, H, -1)], -1)
                q = torch.cat([q[..., :dn], _pairs(q[..., dn:], f, mag)], -1)
                o = _attend(q, k, (latent @ w("uv").T).view(T, H, -1), m["scale"]).reshape(T, -1) * torch.sigmoid(h @ w("g").T)
            else:
                E, N, K = m["inner"], m["state"], m["dt_rank"]
                u, z = (h @ w("in").T).split(E, -1)
                u = _silu(_conv(u, w("conv")) + w("conv.b"))
                low = u @ w("x").T
                dt = torch.nn.functional.softplus(low[:, :K] @ w("dt").T + w("dt.b"))
                A, B, C, D = -torch.exp(w("A_log")), low[:, K: K + N], low[:, K + N:], w("D")
                S, o = torch.zeros(E, N, dtype=F64, device=DEVICE), torch.empty(T, E, dtype=F64, device=DEVICE)
                for t in range(T):
                    S = torch.exp(dt[t].unsqueeze(1) * A) * S + (dt[t] * u[t]).unsqueeze(1) * B[t]
                    o[t] = S @ C[t]
                o = (o + D * u) * _silu(z)
            out.append(o @ w("o").T)
        x = x + _rms(torch.cat(out), W(p + "norm1b"), eps)
        h = _rms(x, W(p + "norm2"), eps)
        if mlp["kind"] == "dense":
            y = unit(h, p + "mlp.", torch.relu)
        else:
            score = torch.sigmoid(h @ W(p + "mlp.router").T)
            chosen = score.topk(mlp["router"]["top"], -1).indices
            y = unit(h, p + "mlp.shared.", _silu)
            for e in range(mlp["router"]["experts"]):
                rows = (chosen == e).any(-1).nonzero().squeeze(-1)
                y = y.index_add(0, rows, unit(score[rows, e].unsqueeze(-1) * h[rows], f"{p}mlp.e{e}.", _silu))
        x = x + _rms(y, W(p + "norm2b"), eps)
    cap = c["logit_softcap"]
    return x, lambda y: cap * torch.tanh(_rms(y, W("final.norm"), eps) @ W("embed").T / cap)


def exact(case, seed):
    new = case.get("new", 0)
    held, given = _lengths(case)
    lens = [h + g + new for h, g in zip(held, given)]
    if 2.0 * sum(lens) * _per_token(case["shape"])[1] > 4e14:      # over about twenty seconds of products in 64 bits
        return None
    tensors = _tensors(case["shape"])
    vectors = {}

    def W(name):
        if name not in vectors:
            t = _make(seed, name, *tensors[name]).to(F64)
            if t.numel() > 1 << 20:
                return t
            vectors[name] = t
        return vectors[name]

    more = case.get("new", SPAN if case["kind"] == "decode" else 0)
    ids = [t[:n] for t, n in zip(_tokens(case, seed, more), lens)]
    table = "model.embed_tokens.weight" if case["shape"] in DECODERS else "embed"
    x = W(table)[torch.tensor([t for r in ids for t in r], device=DEVICE)]
    x, head = {"sitelorn": _sitelorn, "vunelix": _vunelix}.get(case["shape"], _decoder)(case, W, x, lens)
    ends = torch.tensor(lens, device=DEVICE).cumsum(0) - 1 - new
    if case["kind"] == "generate":
        return torch.stack([head(x[ends + t]) for t in range(new + 1)])
    return head(x[ends])
