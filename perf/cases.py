"""What this engine is measured on: steps of decoding, of prompts and of both together through ``ModelRunner.step``, the one
function that generation, trace replay and the benchmark all call, at the sizes of the benchmark's models.

``listed`` gives the cases, ``draw`` more of the same ranges, ``prepare`` a bound model with its cache as a running server
holds it, ``run`` one step, ``work`` what a step cannot do without, ``exact`` the same logits in 64 bits.

A case: ``model`` ("3B" and "7B": the dense decoder; "mixed_layers": block-masked attention beside retention, and the gated
delta rule, in turn), ``dtype`` of the engine, ``decode`` requests with up to ``context`` cached tokens that get one token
each (``ragged``: spread evenly from an eighth of it), ``prompt`` tokens of ``portions`` prompts, each portion after
``history`` cached tokens, and ``sampled``: the step draws its tokens too.  A step with tokens drawn is only compared where
its logits are float32: in bfloat16 two correct results differ by more than the two largest logits of a row often do.
"""
import math
import zlib

import torch

from qwen_decoder_b200.config import config_from_dict, describe_model
from qwen_decoder_b200.engine import ModelRunner, StepEntry
from qwen_decoder_b200.parts.model import build_model
from qwen_decoder_b200.weights import TensorSource, load_into

DEVICE = "cuda:0"
PAGE = 16
DENSE = {
    "3B": dict(hidden_size=2048, intermediate_size=11008, num_hidden_layers=36, num_attention_heads=16, num_key_value_heads=2,
               vocab_size=151936, tie_word_embeddings=True),
    "7B": dict(hidden_size=3584, intermediate_size=18944, num_hidden_layers=28, num_attention_heads=28, num_key_value_heads=4,
               vocab_size=152064, tie_word_embeddings=False),
}
THETA, EPS = 1000000.0, 1e-6
WIDTH, FF, VOCAB, HEADS, KV_HEADS, DIM, BLOCK, LAYERS, GROUPS, MIXED_EPS = 2048, 5632, 32000, 16, 2, 128, 1024, 8, 8, 1e-5
# Random weights with the proportions of trained ones: what a branch adds is small against the sum it joins, whatever the depth.
# (With branches as large as the sum every rounding of an activation grows from layer to layer, and two correct bfloat16
# results differ by a tenth of the logits: nothing could be told from comparing them.)
EMBED, INTO_SUM = 0.5, 0.1
DECAY = [1.0 - 2.0 ** (-3.0 - 6.0 * i / 32) for i in range(32)]


def case(name, model, dtype="bfloat16", decode=0, context=0, ragged=False, prompt=0, portions=1, history=0, sampled=False):
    return {"name": name, "model": model, "dtype": dtype, "decode": decode, "context": context, "ragged": ragged,
            "prompt": prompt, "portions": portions, "history": history, "sampled": sampled}


def listed():
    return [
        # one person at a prompt: the smallest call, all latency
        case("decode_3b_b1", "3B", decode=1, context=2048),
        # a few users, the benchmark's headline
        case("decode_3b_b8", "3B", decode=8, context=2048),
        # a full server
        case("decode_3b_b64", "3B", decode=64, context=2048),
        # a server's ordinary moment: requests of every age decoding together
        case("decode_7b_b23_ragged", "7B", decode=23, context=4001, ragged=True),
        # a question's first token
        case("prompt_3b_101", "3B", prompt=101),
        # one step's default budget of prompt tokens, three prompts in it
        case("prompt_3b_512_of_3", "3B", prompt=512, portions=3),
        # a document in one step
        case("prompt_3b_2048", "3B", prompt=2048),
        # the usual step of a busy server: a portion of a long prompt beside the requests that decode
        case("serve_7b_489_and_23", "7B", decode=23, context=2048, ragged=True, prompt=489, history=1024),
        # the 32-bit engine, as one compares checkpoints with it: generation, some of it sampled, ...
        case("f32_decode_3b_b4", "3B", "float32", decode=4, context=1000, sampled=True),
        # ... and a prompt
        case("f32_prompt_3b_203", "3B", "float32", prompt=203),
        # the linear-attention design: decoding from a state per request ...
        case("mixed_decode_b8", "mixed_layers", decode=8, context=500, ragged=True),
        # ... and a prompt through the recurrence
        case("mixed_prompt_1500", "mixed_layers", prompt=1500),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode_3b", "decode_3b", "decode_7b", "prompt_3b", "prompt_3b", "prompt_7b", "serve", "f32_decode",
                       "f32_prompt", "mixed_decode", "mixed_prompt"])
    ragged = rng.random() < 0.5
    if kind in ("decode_3b", "decode_7b"):
        c = case("", kind[-2:].upper(), decode=_log(rng, 1, 64), context=_log(rng, 64, 4096), ragged=ragged)
    elif kind == "prompt_3b":
        c = case("", "3B", prompt=_log(rng, 9, 2048), portions=rng.randint(1, 4))
    elif kind == "prompt_7b":
        c = case("", "7B", prompt=_log(rng, 9, 800), portions=rng.randint(1, 4), history=rng.choice([0, 0, 300, 1500]))
    elif kind == "serve":
        c = case("", rng.choice(["3B", "7B"]), decode=_log(rng, 1, 48), context=_log(rng, 128, 4096), ragged=ragged,
                 prompt=_log(rng, 16, 512), portions=rng.randint(1, 2), history=_log(rng, 1, 2048))
    elif kind == "f32_decode":
        c = case("", "3B", "float32", decode=_log(rng, 1, 16), context=_log(rng, 64, 2048), ragged=ragged, sampled=True)
    elif kind == "f32_prompt":
        c = case("", "3B", "float32", prompt=_log(rng, 9, 400), portions=rng.randint(1, 3))
    elif kind == "mixed_decode":
        c = case("", "mixed_layers", decode=_log(rng, 1, 48), context=rng.randint(17, 600), ragged=ragged)
    else:
        c = case("", "mixed_layers", prompt=_log(rng, 9, 2048), portions=rng.randint(1, 3))
    del c["name"]
    return c


# ---- what a user's program holds ----------------------------------------------------------------------------------

def _config(c):
    if c["model"] in DENSE:
        return dict(DENSE[c["model"]], architectures=["Qwen2ForCausalLM"], max_position_embeddings=32768, rope_theta=THETA,
                    rms_norm_eps=EPS)
    attention = {"heads": HEADS, "kv_heads": KV_HEADS, "dim": DIM, "vdim": DIM, "scale": DIM ** -0.5, "mask": {"size": BLOCK},
                 "rot": {"base": 200000.0, "dims": DIM, "scaling": {"factor": 4.0}}}
    retention = {"heads": 32, "dim": 64, "vdim": 64, "decay": DECAY, "rot": {"base": 10000.0, "dims": 64}}
    mlp = {"kind": "dense", "ff": FF}
    both = {"type": "parallel", "mlp": mlp, "mixer": {"left": attention, "right": retention, "left_scale": 0.8,
                                                      "right_scale": 1.25}}
    delta = {"type": "delta", "mlp": mlp, "mixer": {"heads": 32, "kv_heads": 16, "dim": 128, "vdim": 128, "conv": 4}}
    return {"architecture": "Gopevik", "vocab": VOCAB, "width": WIDTH, "norm": {"eps": MIXED_EPS, "groups": GROUPS},
            "layers": [both, delta] * (LAYERS // 2)}


def _shapes(c):
    """{tensor: (shape, how it is filled)} of the model, in the names of its checkpoints."""
    out = {}
    if c["model"] in DENSE:
        z = DENSE[c["model"]]
        D, F, V = z["hidden_size"], z["intermediate_size"], z["vocab_size"]
        kv = z["num_key_value_heads"] * 128
        out["model.embed_tokens.weight"] = ((V, D), EMBED)
        for i in range(z["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for n, rows in (("q", D), ("k", kv), ("v", kv)):
                out[f"{p}self_attn.{n}_proj.weight"] = ((rows, D), 0.02)
                out[f"{p}self_attn.{n}_proj.bias"] = ((rows,), 0.02)
            out[f"{p}self_attn.o_proj.weight"] = ((D, D), 0.02 * INTO_SUM)
            for n in ("gate", "up"):
                out[f"{p}mlp.{n}_proj.weight"] = ((F, D), 0.02)
            out[f"{p}mlp.down_proj.weight"] = ((D, F), 0.02 * INTO_SUM)
            for n in ("input", "post_attention"):
                out[f"{p}{n}_layernorm.weight"] = ((D,), "one")
        out["model.norm.weight"] = ((D,), "one")
        if not z["tie_word_embeddings"]:
            out["lm_head.weight"] = ((V, D), 0.02)
        return out
    D, F = WIDTH, FF
    out["embed"], out["head"] = ((VOCAB, D), EMBED), ((VOCAB, D), 0.02)
    out["final.norm"] = ((D,), "one")
    for i in range(LAYERS):
        p = f"l{i}."
        for n in ("norm1", "norm2"):
            out[p + n] = ((D,), "one")
            out[p + n + "b"] = ((D,), (0.8 * INTO_SUM, 1.2 * INTO_SUM))
        for n in ("gate", "up"):
            out[f"{p}mlp.{n}"], out[f"{p}mlp.{n}.b"] = ((F, D), 0.02), ((F,), 0.02)
        out[f"{p}mlp.down"], out[f"{p}mlp.down.b"] = ((D, F), 0.02), ((D,), 0.02)
        if i % 2 == 0:
            for n, rows in (("q", D), ("k", 256), ("v", 256), ("g", D), ("o", D)):
                out[f"{p}mix.left.{n}"] = ((rows, D), 0.02)
            for n in "qkvgo":
                out[f"{p}mix.right.{n}"] = ((D, D), 0.02)
        else:
            for n, rows in (("q", 2048), ("k", 2048), ("v", 4096)):
                out[f"{p}mix.{n}"], out[f"{p}mix.{n}.conv"] = ((rows, D), 0.02), ((rows, 4), (-0.5, 0.5))
            out[f"{p}mix.g"], out[f"{p}mix.o"] = ((4096, D), 0.02), ((D, 4096), 0.02)
            out[f"{p}mix.a"] = out[f"{p}mix.b"] = ((32, D), 0.02)
            out[f"{p}mix.A_log"], out[f"{p}mix.dt_bias"] = ((32,), (-2.0, 1.0)), ((32,), (-3.0, 0.0))
            out[f"{p}mix.norm"] = ((128,), "one")
    return out


def _random(name, seed, shape, fill, dtype):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(zlib.crc32(name.encode()) + (int(seed) << 32))
    t = torch.empty(shape, dtype=torch.float32, device=DEVICE)
    if isinstance(fill, float):
        t.normal_(0.0, fill, generator=g)
    elif fill == "one":
        t.normal_(1.0, 0.1, generator=g)
    elif fill == "unit":
        t.normal_(0.0, 1.0, generator=g)
    else:
        t.uniform_(*fill, generator=g)
    return t.to(dtype)


def _tokens(c, seed, n, name):
    vocab = DENSE[c["model"]]["vocab_size"] if c["model"] in DENSE else VOCAB
    g = torch.Generator().manual_seed(zlib.crc32(name.encode()) + int(seed))
    return torch.randint(0, vocab, (n,), generator=g).tolist()


def _contexts(c):
    """Cached tokens of each request that decodes."""
    n, most = c["decode"], c["context"]
    if not c["ragged"] or n == 1:
        return [most] * n
    return [most // 8 + (most - most // 8) * i // (n - 1) for i in range(n)]


def _portions(c):
    """Tokens of each prompt: the first ones longer by what is left over."""
    if not c["prompt"]:
        return []
    n = min(c["portions"], c["prompt"])
    weights = [3 * k + 2 for k in range(n)]
    parts = [max(1, c["prompt"] * w // sum(weights)) for w in weights]
    parts[-1] += c["prompt"] - sum(parts)
    return parts


def _history(c, seed, name, n, dtype):
    """Random keys and values [layers, K|V, heads, n, 128] of n cached tokens."""
    z = DENSE[c["model"]]
    return _random(name, seed, (z["num_hidden_layers"], 2, z["num_key_value_heads"], n, 128), "unit", dtype)


def _cached(runner, c, seed, name, n):
    """A request that holds ``n`` tokens."""
    rc = runner.open(name)
    if not n:
        return rc
    if c["model"] in DENSE:
        runner.cache.ensure(rc, n + 1)
        runner.cache.commit(rc, n)
        pages = -(-n // PAGE)
        h = _history(c, seed, name, pages * PAGE, runner.dtype)
        h = h.view(h.shape[0], 2, h.shape[2], pages, PAGE, 128).permute(0, 3, 1, 2, 4, 5)
        runner.cache.kv[0][:, torch.tensor(rc.tables[0].pages[:pages], device=DEVICE)] = h
    else:                                  # a state comes from the tokens themselves
        runner.step([StepEntry(rc, _tokens(c, seed, n, name), [])])
    return rc


class State:
    pass


def prepare(case, seed):
    c = case
    dtype = torch.float32 if c["dtype"] == "float32" else torch.bfloat16
    config = config_from_dict(_config(c))
    model = build_model(describe_model(config))
    shapes = _shapes(c)
    load_into(model, TensorSource(lambda n: _random(n, seed, *shapes[n], dtype), {n: s for n, (s, _) in shapes.items()}),
              dtype, DEVICE)
    contexts, portions = _contexts(c), _portions(c)
    pages = sum((n + 1 + PAGE - 1) // PAGE for n in contexts) + sum((c["history"] + n + PAGE - 1) // PAGE for n in portions)
    most = max(contexts + [c["history"] + n for n in portions]) + 1
    s = State()
    s.runner = ModelRunner(model, config, num_pages=pages, page_size=PAGE, max_requests=len(contexts) + len(portions),
                           max_positions=most)
    s.case = c
    s.decoding = [_cached(s.runner, c, seed, f"d{i}", n) for i, n in enumerate(contexts)]
    s.single = _tokens(c, seed, max(1, len(contexts)), "single")
    s.prompts = [_tokens(c, seed, n, f"prompt{i}") for i, n in enumerate(portions)]
    s.started = [_cached(s.runner, c, seed, f"p{i}", c["history"]) for i in range(len(portions))] if c["history"] else None
    n = len(contexts) + len(portions)
    s.sampling = None
    if c["sampled"]:                       # every other request greedy, the others from the 40 likeliest tokens
        s.sampling = ([0.8 * (i % 2) for i in range(n)], [40] * n, [(0.37 + 0.61 * i) % 1.0 for i in range(n)])
    return s


def run(state):
    s = state
    runner = s.runner
    prompts = s.started or [runner.open(f"p{i}") for i in range(len(s.prompts))]
    entries = [StepEntry(rc, t, [len(t) - 1]) for rc, t in zip(prompts, s.prompts)]
    entries += [StepEntry(rc, [t], [0]) for rc, t in zip(s.decoding, s.single)]
    out = runner.step(entries, sampling=s.sampling)
    if s.started is None:                  # the prompt is served; its pages go to the next one
        for rc in prompts:
            runner.close(rc)
    else:                                  # the requests stay where they were: the next pass is the same step
        for rc, t in zip(prompts, s.prompts):
            rc.num_tokens -= len(t)
    for rc in s.decoding:
        rc.num_tokens -= 1
    logits, tokens = out if s.sampling is not None else (out, None)
    # the last page and the last slot belong to no request
    got = {"logits": logits, "cache": [kv[:, :-1] for kv in runner.cache.kv], "state": [st[:-1] for st in runner.cache.states]}
    if tokens is not None:
        got["tokens"] = tokens
    return got


# ---- what a step cannot do without --------------------------------------------------------------------------------

def work(case):
    c = case
    size = 4 if c["dtype"] == "float32" else 2
    shapes = _shapes(c)
    matrices = sum(math.prod(s) for n, (s, _) in shapes.items() if len(s) == 2 and "embed" not in n and n not in ("head", "lm_head.weight"))
    vectors = sum(s[0] for s, _ in shapes.values() if len(s) == 1)
    contexts, portions = _contexts(c), _portions(c)
    tokens, rows = len(contexts) + sum(portions), len(contexts) + len(portions)
    if c["model"] in DENSE:
        z = DENSE[c["model"]]
        V, D, L, H, G = z["vocab_size"], z["hidden_size"], z["num_hidden_layers"], z["num_attention_heads"], z["num_key_value_heads"]
        read = sum(contexts) + len(portions) * c["history"]
        pairs = sum(n + 1 for n in contexts) + sum(n * c["history"] + n * (n + 1) // 2 for n in portions)
        state = 0
        scan = 0
    else:
        V, D, L, H, G = VOCAB, WIDTH, LAYERS // 2, HEADS, KV_HEADS
        read = sum(n % BLOCK for n in contexts)
        pairs = read + len(contexts) + sum((n // BLOCK) * (BLOCK * (BLOCK + 1) // 2) + (n % BLOCK) * (n % BLOCK + 1) // 2 for n in portions)
        per_request = L * 4 * (32 * 64 * 64 + 32 * 128 * 128)
        state = (2 * len(contexts) + len(portions)) * per_request
        scan = tokens * L * (4 * 32 * 64 * 64 + 6 * 32 * 128 * 128)
    nbytes = (matrices + V * D + tokens * D) * size + vectors * size + (read + tokens) * L * 2 * G * 128 * size + rows * V * 4 + state
    flops = 2 * tokens * matrices + 2 * rows * V * D + 4 * pairs * L * H * 128 + scan
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    # two forms of the same step (every product through another kernel) differ by this over four, measured over the ranges
    if case["dtype"] == "float32":
        return {"rel": 2e-5, "max": 2e-4, "differ": 0.0}
    return {"rel": 0.025, "max": 0.25}


# ---- the same in 64 bits, from the formulas -----------------------------------------------------------------------

def _turn(x, positions, dims, base, factor=1.0):
    """x [T, heads, d]: pairs (i, i + dims / 2) turn by position * base^(-2 i / dims) / factor."""
    half = dims // 2
    rate = base ** (-2.0 * torch.arange(half, dtype=torch.float64, device=x.device) / dims) / factor
    a = positions.to(torch.float64)[:, None, None] * rate
    u, v = x[..., :half], x[..., half:]
    return torch.cat([u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()], dim=-1)


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def exact(case, seed):
    c = case
    dtype = torch.float32 if c["dtype"] == "float32" else torch.bfloat16
    shapes = _shapes(c)
    w = lambda n: _random(n, seed, *shapes[n], dtype).double()
    with torch.no_grad():
        logits = _exact_dense(c, seed, w, dtype) if c["model"] in DENSE else _exact_mixed(c, seed, w)
    got = {"logits": logits, "cache": None, "state": None}
    if c["sampled"]:
        got["tokens"] = None
    return got


def _exact_dense(c, seed, w, dtype):
    z = DENSE[c["model"]]
    L, H, G = z["num_hidden_layers"], z["num_attention_heads"], z["num_key_value_heads"]
    single = _tokens(c, seed, max(1, c["decode"]), "single")
    requests = [(f"p{i}", c["history"], _tokens(c, seed, n, f"prompt{i}")) for i, n in enumerate(_portions(c))]
    requests += [(f"d{i}", n, [single[i]]) for i, n in enumerate(_contexts(c))]
    past = [_history(c, seed, name, -(-n // PAGE) * PAGE, dtype)[:, :, :, :n] if n else None for name, n, _ in requests]
    at, ends, n = [], [], 0
    for _, start, t in requests:
        at.append(torch.arange(start, start + len(t), device=DEVICE))
        n += len(t)
        ends.append(n)
    at = torch.cat(at)
    x = w("model.embed_tokens.weight")[torch.tensor(sum((t for _, _, t in requests), []), device=DEVICE)]
    for i in range(L):
        p = f"model.layers.{i}."
        h = _rms(x, EPS) * w(p + "input_layernorm.weight")
        q, k, v = ((h @ w(f"{p}self_attn.{m}_proj.weight").T + w(f"{p}self_attn.{m}_proj.bias")).view(n, -1, 128) for m in "qkv")
        q, k = _turn(q, at, 128, THETA), _turn(k, at, 128, THETA)
        o = torch.empty_like(q)
        for (_, start, t), end, old in zip(requests, ends, past):
            own = slice(end - len(t), end)
            K, U = k[own].transpose(0, 1), v[own].transpose(0, 1)
            if old is not None:
                K, U = torch.cat([old[i, 0].double(), K], dim=1), torch.cat([old[i, 1].double(), U], dim=1)
            s = q[own].view(len(t), G, H // G, 128).permute(1, 2, 0, 3) @ K[:, None].transpose(-1, -2) * 128 ** -0.5
            late = torch.arange(start + len(t), device=DEVICE)[None, :] > at[own][:, None]
            o[own] = (s.masked_fill(late, float("-inf")).softmax(dim=-1) @ U[:, None]).permute(2, 0, 1, 3).reshape(len(t), H, 128)
        x = x + o.view(n, -1) @ w(p + "self_attn.o_proj.weight").T
        h = _rms(x, EPS) * w(p + "post_attention_layernorm.weight")
        h = _silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)
        x = x + h @ w(p + "mlp.down_proj.weight").T
    h = _rms(x[torch.tensor(ends, device=DEVICE) - 1], EPS) * w("model.norm.weight")
    return h @ w("model.embed_tokens.weight" if z["tie_word_embeddings"] else "lm_head.weight").T


def _exact_mixed(c, seed, w):
    single = _tokens(c, seed, max(1, c["decode"]), "single")
    sequences = [_tokens(c, seed, n, f"prompt{i}") for i, n in enumerate(_portions(c))]
    sequences += [_tokens(c, seed, n, f"d{i}") + [single[i]] for i, n in enumerate(_contexts(c))]
    norm = lambda x, name: _rms(x.unflatten(-1, (GROUPS, -1)), MIXED_EPS).flatten(-2) * w(name)
    B, T = len(sequences), max(len(s) for s in sequences)
    ids = torch.zeros((B, T), dtype=torch.long)            # shorter ones are followed by tokens that nothing before them sees
    for b, s in enumerate(sequences):
        ids[b, :len(s)] = torch.tensor(s)
    at = torch.arange(T, device=DEVICE)
    x = w("embed")[ids.to(DEVICE)]
    turn = lambda y, *a: torch.stack([_turn(r, at, *a) for r in y])
    seen = (at[None, :] <= at[:, None]) & (at[None, :] // BLOCK == at[:, None] // BLOCK)
    for i in range(LAYERS):
        p = f"l{i}."
        m = p + "mix."
        h = norm(x, p + "norm1")
        lin = lambda name, y=h: y @ w(name).T
        if i % 2 == 0:
            q, k = (turn(lin(m + "left." + n).unflatten(-1, (-1, DIM)), DIM, 200000.0, 4.0) for n in "qk")
            v = lin(m + "left.v").unflatten(-1, (KV_HEADS, DIM))
            rep = HEADS // KV_HEADS
            o = torch.empty_like(q)
            for j in range(HEADS):
                s = (q[:, :, j] @ k[:, :, j // rep].transpose(1, 2) * DIM ** -0.5).masked_fill(~seen, float("-inf"))
                top = s.amax(dim=-1, keepdim=True).clamp(min=0.0)
                e = torch.exp(s - top)
                o[:, :, j] = e / (torch.exp(-top) + e.sum(dim=-1, keepdim=True)) @ v[:, :, j // rep]
            left = (o.flatten(-2) * torch.sigmoid(lin(m + "left.g"))) @ w(m + "left.o").T
            q, k = (turn(lin(m + "right." + n).unflatten(-1, (32, 64)), 64, 10000.0) for n in "qk")
            v, k = lin(m + "right.v").unflatten(-1, (32, 64)), k * 64 ** -0.5
            decay = torch.tensor(DECAY, dtype=torch.float64, device=DEVICE)[:, None, None]
            S, o = torch.zeros((B, 32, 64, 64), dtype=torch.float64, device=DEVICE), torch.empty_like(v)
            for t in range(T):
                S = decay * S + k[:, t, :, :, None] * v[:, t, :, None, :]
                o[:, t] = (S.transpose(-1, -2) @ q[:, t, :, :, None])[..., 0]
            right = (_rms(o, MIXED_EPS).flatten(-2) * _silu(lin(m + "right.g"))) @ w(m + "right.o").T
            a = 0.8 * left + 1.25 * right
        else:
            def conv(name):
                u, taps = lin(m + name), w(m + name + ".conv")
                u = torch.cat([u.new_zeros((B, 3, u.shape[-1])), u], dim=1)
                return _silu(sum(u[:, j:j + T] * taps[:, j] for j in range(4)))
            q, k = (conv(n).unflatten(-1, (16, 128)) for n in "qk")
            q, k = (y / torch.sqrt((y * y).sum(dim=-1, keepdim=True) + 1e-6) for y in (q, k))
            q, k = (torch.repeat_interleave(y, 2, dim=2) for y in (q * 128 ** -0.5, k))
            v, beta = conv("v").unflatten(-1, (32, 128)), torch.sigmoid(lin(m + "b"))
            g = torch.exp(-torch.exp(w(m + "A_log")) * torch.nn.functional.softplus(lin(m + "a") + w(m + "dt_bias")))
            S, o = torch.zeros((B, 32, 128, 128), dtype=torch.float64, device=DEVICE), torch.empty_like(v)
            for t in range(T):
                S = g[:, t, :, None, None] * S
                u = beta[:, t, :, None] * (v[:, t] - (S.transpose(-1, -2) @ k[:, t, :, :, None])[..., 0])
                S = S + k[:, t, :, :, None] * u[:, :, None, :]
                o[:, t] = (S.transpose(-1, -2) @ q[:, t, :, :, None])[..., 0]
            o = _rms(o, MIXED_EPS) * w(m + "norm")
            a = (o.flatten(-2) * _silu(lin(m + "g"))) @ w(m + "o").T
        x = x + norm(a, p + "norm1b")
        h = norm(x, p + "norm2")
        f = _silu(h @ w(p + "mlp.gate").T + w(p + "mlp.gate.b")) * (h @ w(p + "mlp.up").T + w(p + "mlp.up.b"))
        x = x + norm(f @ w(p + "mlp.down").T + w(p + "mlp.down.b"), p + "norm2b")
    last = torch.stack([x[b, len(s) - 1] for b, s in enumerate(sequences)])
    return norm(last, "final.norm") @ w("head").T
