"""What is timed: steps of the engine's step function on LFM2 models, at the sizes that the engine is built for.

A case is ONE step: ``ModelRunner.step`` over a batch of segments, each the next tokens of one request, with the logits of
every segment's last token.  That call is what the scheduler, the trace replay and a user's own loop make, and everything
between token ids and logits happens inside it: the host's batch, the embedding, the mixers over the paged cache and the
state slots, the feed-forwards with their routers and experts, the head.  The models are the three that the benchmark is
quoted on (8B-A1B with routed experts, dense 1.2B, dense 2.6B), at full depth and width.

``segments`` says what a step holds: "2048@0" is a fresh request's prompt of 2,048 tokens (the request is admitted before
the step and freed after it), "1@8192" one decoded token of a request that holds 8,192 positions, "2048@30720" a portion of
a longer prompt; "*8" repeats a segment.  A held request goes back to its length after the step, so that each pass does
the same work.

Weights are drawn so that activations behave as in a trained model: unit embedding rows, matrices N(0, 0.02), gains around 1
and head gains around 1.5 (attention looks at some of the keys and not evenly at all of them), logits of a few units.  The
projections into the stream are scaled down by the square root of twice the depth, so that no layer replaces the stream.  The
routers know a token by a few strong features of its embedding, other experts in each layer, all experts equally often: like
trained ones they are sure of their picks, and rounding seldom turns one.  Held requests hold random keys, values and conv
rows.
"""
import math
import zlib

import torch

from snowllm_b200.cache import CacheManager
from snowllm_b200.engine import ModelRunner, StepEntry
from snowllm_b200.loader import build_model
from snowllm_b200.weights.loader import load_tensors

PAGE = 64


def _config(layers, attention, **more):
    return dict({"vocab_size": 65536, "hidden_size": 2048, "num_hidden_layers": layers,
                 "layer_types": ["full_attention" if i in attention else "conv" for i in range(layers)],
                 "num_attention_heads": 32, "num_key_value_heads": 8, "conv_L_cache": 3, "conv_bias": False,
                 "rope_theta": 1000000.0, "norm_eps": 1e-5, "tie_word_embeddings": True,
                 "max_position_embeddings": 128000}, **more)


MODELS = {
    "8b-a1b": _config(24, (2, 6, 10, 14, 18, 21), architectures=["Lfm2MoeForCausalLM"], num_dense_layers=2,
                      intermediate_size=7168, num_experts=32, num_experts_per_tok=4, moe_intermediate_size=1792,
                      norm_topk_prob=True, use_expert_bias=True, routed_scaling_factor=1.0),
    "dense-1.2b": _config(16, (2, 5, 8, 10, 12, 14), architectures=["Lfm2ForCausalLM"], intermediate_size=8192),
    "dense-2.6b": _config(30, (2, 6, 10, 14, 18, 22, 25, 28), architectures=["Lfm2ForCausalLM"], intermediate_size=10752),
}
DTYPES = {"bfloat16": torch.bfloat16, "float32": torch.float32}


# --- the cases ----------------------------------------------------------------------------------------------

def listed():
    def case(name, model, segments, dtype="bfloat16"):
        return {"name": name, "model": model, "dtype": dtype, "segments": segments}
    return [
        # one user chatting with the small model: the smallest step there is, all launches and latency
        case("dense1.2b-decode-1", "dense-1.2b", "1@513"),
        # one user, a long conversation with the model with experts (4 of 32 experts read in a layer)
        case("moe-decode-1", "8b-a1b", "1@8192"),
        # a few users at the benchmark's context: most experts of a layer are read
        case("moe-decode-8", "8b-a1b", "1@8192*8"),
        # a busy server: requests at whatever length they have got to
        case("moe-decode-64", "8b-a1b", " ".join(f"1@{127 + 131 * i}" for i in range(64))),
        # long documents open in 64 sessions: the cache is most of what a step reads
        case("dense1.2b-decode-64-32k", "dense-1.2b", "1@32700*64"),
        # one prompt in one step
        case("moe-prefill-2048", "8b-a1b", "2048@0"),
        # short questions that arrived together
        case("moe-prefill-short", "8b-a1b", "5@0 23@0 40@0 77@0 131@0"),
        # a full step budget of prompts of unequal length
        case("dense1.2b-prefill-8192", "dense-1.2b", "2047@0 128@0 1023@0 1601@0 511@0 1300@0 777@0 805@0"),
        # the last portion of a 32,768-token document
        case("dense2.6b-portion-32k", "dense-2.6b", "2048@30720"),
        # a portion of a document beside requests that go on decoding
        case("dense2.6b-mixed", "dense-2.6b", "2040@16384 1@8192*8"),
        # the 32-bit path: one user decoding, and a prompt, where results have to be reproduced exactly
        case("f32-moe-decode-4", "8b-a1b", "1@2048*4", "float32"),
        case("f32-dense1.2b-prefill-512", "dense-1.2b", "509@0", "float32"),
    ]


def draw(rng):
    most = max(_seconds(c) for c in listed())
    while True:
        case = _draw(rng)
        if _seconds(case) <= most:
            return case


def _seconds(case):
    """About what a step costs at the rates of the memory and of the units that its type runs on."""
    w = work(case)
    return max(w["bytes"] / 6e12, w["flops"] / (5e13 if case["dtype"] == "float32" else 1e15))


def _draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(sorted(MODELS))
    if rng.random() < 0.15:                        # the 32-bit path
        if rng.random() < 0.5:
            segments = " ".join(f"1@{log(16, 8192)}" for _ in range(log(1, 4)))
            return {"model": model, "dtype": "float32", "segments": segments}
        return {"model": model, "dtype": "float32", "segments": f"{log(17, 512)}@0"}
    kind = rng.choice(["decode", "decode", "prompts", "portion", "mixed"])
    if kind == "decode":                           # 1 to 64 requests, at lengths around one that is drawn too
        n, at = log(1, 64), log(64, 32000)
        return {"model": model, "dtype": "bfloat16",
                "segments": " ".join(f"1@{min(32700, max(1, round(at * rng.uniform(0.3, 1.7))))}" for _ in range(n))}
    if kind == "prompts":                          # 1 to 8 prompts in one step
        n = rng.randint(1, 8)
        return {"model": model, "dtype": "bfloat16", "segments": " ".join(f"{log(5, 1024)}@0" for _ in range(n))}
    n, at = log(64, 1536), log(256, 30720)
    more = "".join(f" 1@{log(64, 8192)}" for _ in range(log(1, 16))) if kind == "mixed" else ""
    return {"model": model, "dtype": "bfloat16", "segments": f"{n}@{at}" + more}


def _segments(case):
    """[(tokens, positions held before them)] of the step."""
    out = []
    for word in case["segments"].split():
        what, _, times = word.partition("*")
        n, start = what.split("@")
        out += [(int(n), int(start))] * int(times or 1)
    return out


# --- inputs, from the seed alone ----------------------------------------------------------------------------

def _generator(seed, *what):
    return torch.Generator(device="cuda").manual_seed(zlib.crc32(repr((seed,) + what).encode()))


def _weights(case, seed):
    """Checkpoint tensors by name."""
    c, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
    H, hd = c["hidden_size"], c["hidden_size"] // c["num_attention_heads"]
    kv, L = c["num_key_value_heads"] * hd, c["num_hidden_layers"]
    out_std = 0.02 / math.sqrt(2 * L)
    gen = _generator(seed, "weights")
    w = {}

    def normal(name, *shape, std=0.02, mean=0.0, keep=dtype):
        w[name] = torch.empty(shape, dtype=keep, device="cuda").normal_(mean, std, generator=gen)

    normal("model.embed_tokens.weight", c["vocab_size"], H, std=1.0)
    if "num_experts" in c:       # among the first features a token has those that the routers know it by
        E = c["num_experts"]
        known = torch.rand(c["vocab_size"], E, device="cuda", generator=gen).topk(c["num_experts_per_tok"], -1).indices
        w["model.embed_tokens.weight"].scatter_(1, known, 12.0)
    normal("model.embedding_norm.weight", H, std=0.005, mean=0.05)
    for i, kind in enumerate(c["layer_types"]):
        p = f"model.layers.{i}."
        normal(p + "operator_norm.weight", H, std=0.1, mean=1.0)
        normal(p + "ffn_norm.weight", H, std=0.1, mean=1.0)
        if kind == "conv":
            normal(p + "conv.in_proj.weight", 3 * H, H)
            normal(p + "conv.conv.weight", H, 1, c["conv_L_cache"], std=0.3)
            normal(p + "conv.out_proj.weight", H, H, std=out_std)
        else:
            a = p + "self_attn."
            normal(a + "q_proj.weight", H, H)
            normal(a + "k_proj.weight", kv, H)
            normal(a + "v_proj.weight", kv, H)
            normal(a + "out_proj.weight", H, H, std=out_std)
            normal(a + "q_layernorm.weight", hd, std=0.1, mean=1.5)
            normal(a + "k_layernorm.weight", hd, std=0.1, mean=1.5)
        f = p + "feed_forward."
        if i < c.get("num_dense_layers", L):
            normal(f + "w1.weight", c["intermediate_size"], H)
            normal(f + "w3.weight", c["intermediate_size"], H)
            normal(f + "w2.weight", H, c["intermediate_size"], std=out_std)
        else:
            E, F = c["num_experts"], c["moe_intermediate_size"]
            normal(f + "gate.weight", E, H)
            w[f + "gate.weight"][torch.randperm(E, device="cuda", generator=gen), torch.arange(E, device="cuda")] += 0.5
            normal(f + "expert_bias", E, std=0.01, keep=torch.float32)
            normal(f + "experts.gate_up_proj", E, 2 * F, H)
            normal(f + "experts.down_proj", E, H, F, std=out_std)
    return w


def _tokens(case, seed):
    gen = torch.Generator().manual_seed(zlib.crc32(repr((seed, "tokens")).encode()))
    V = MODELS[case["model"]]["vocab_size"]
    return [torch.randint(0, V, (n,), generator=gen).tolist() for n, _ in _segments(case)]


def _held(case, seed, layer, b, start):
    """What request ``b`` holds in a layer: keys and values [2, kv heads, start, head dim], or conv rows [taps - 1, H]."""
    c, dtype = MODELS[case["model"]], DTYPES[case["dtype"]]
    gen = _generator(seed, "held", layer, b)
    if c["layer_types"][layer] == "conv":
        return torch.empty(c["conv_L_cache"] - 1, c["hidden_size"], dtype=dtype, device="cuda").normal_(0, 0.8, generator=gen)
    hd = c["hidden_size"] // c["num_attention_heads"]
    t = torch.empty(2, c["num_key_value_heads"], start, hd, dtype=dtype, device="cuda").normal_(generator=gen)
    t[0].mul_(1.5)
    return t


def prepare(case, seed):
    c, segments = MODELS[case["model"]], _segments(case)
    model = build_model(c, case["dtype"])
    load_tensors(model, _weights(case, seed), "cuda")
    pages = [-(-(n + start) // PAGE) for n, start in segments]
    cache = CacheManager(model.cache_specs(), PAGE, sum(pages), len(segments), model.dtype, "cuda")
    state = {"model": model, "cache": cache, "runner": ModelRunner(model, cache, "cuda", use_graphs=True),
             "tokens": _tokens(case, seed), "segments": segments, "held": {},
             "conv": [t[:len(segments)] for t in cache.state_tensors()]}      # without the slot that no request owns
    for b, (n, start) in enumerate(segments):
        if start:
            rc = cache.admit()
            cache.ensure(rc, start + n)
            cache.commit(rc, start)
            state["held"][b] = rc
    if state["held"]:
        run(state)               # requests that decode have decoded before: the step's capture is there
    conv, paged = iter(cache.state_tensors()), iter(cache.paged_tensors())
    for i, kind in enumerate(c["layer_types"]):
        t = next(conv if kind == "conv" else paged)
        for b, rc in state["held"].items():
            held = _held(case, seed, i, b, segments[b][1])
            if kind == "conv":
                t[rc.slot] = held
                continue
            (table,) = rc.tables.values()
            full = held.shape[2] // PAGE
            if full:
                t[torch.tensor(table[:full], device="cuda")] = \
                    held[:, :, :full * PAGE].unflatten(2, (full, PAGE)).permute(2, 0, 1, 3, 4)
            if held.shape[2] % PAGE:
                t[table[full], :, :, :held.shape[2] % PAGE] = held[:, :, full * PAGE:]
    return state


def run(state):
    """One step; the logits [segments, vocab] and the states that it wrote (of fresh requests the keys and values too)."""
    cache, fresh, entries = state["cache"], [], []
    for b, ((n, start), tokens) in enumerate(zip(state["segments"], state["tokens"])):
        rc = state["held"].get(b)
        if rc is None:
            rc = cache.admit()
            cache.ensure(rc, n)
            fresh.append(rc)
        else:
            rc.num_tokens = start
        entries.append(StepEntry(rc, tokens, [n - 1]))
    out = {"logits": state["runner"].step(entries), "conv": state["conv"]}
    if len(fresh) == len(entries):
        out["kv"] = cache.paged_tensors()
    for rc in reversed(fresh):
        cache.free(rc)
    return out


# --- what a pass cannot do without --------------------------------------------------------------------------

def work(case):
    c, segments = MODELS[case["model"]], _segments(case)
    size = 4 if case["dtype"] == "float32" else 2
    H, V, L = c["hidden_size"], c["vocab_size"], c["num_hidden_layers"]
    kv = c["num_key_value_heads"] * (H // c["num_attention_heads"])
    M, B = sum(n for n, _ in segments), len(segments)
    # (query, key) pairs under the causal mask; positions read (the held ones) and written (the step's)
    pairs = sum(n * start + n * (n + 1) // 2 for n, start in segments)
    held = sum(start for _, start in segments)
    weights = V * H * size                                     # the head; the embedding's rows come on top
    nbytes = M * H * size + 4 * B * V
    flops = 2.0 * B * V * H
    for i, kind in enumerate(c["layer_types"]):
        if kind == "conv":
            weights += 4 * H * H * size
            flops += 2.0 * M * 4 * H * H
            nbytes += 2 * B * (c["conv_L_cache"] - 1) * H * size
        else:
            weights += (2 * H * H + 2 * H * kv) * size
            flops += 2.0 * M * (2 * H * H + 2 * H * kv) + 4.0 * H * pairs
            nbytes += 2 * kv * (held + M) * size
        if i < c.get("num_dense_layers", L):
            weights += 3 * H * c["intermediate_size"] * size
            flops += 2.0 * M * 3 * H * c["intermediate_size"]
        else:
            E, k, F = c["num_experts"], c["num_experts_per_tok"], c["moe_intermediate_size"]
            read = E * (1 - (1 - k / E) ** M)                  # experts that a token has picked, on average
            weights += (3 * H * F * read + E * H) * size
            flops += 2.0 * M * (k * 3 * H * F + E * H)
    return {"bytes": weights + nbytes, "flops": flops}


def tolerance(case):
    """Four times what was measured against 64 bits, over the outputs of a case: 5e-3 (and 0.026 at a single value) for
    bfloat16 without experts; with experts as much, where no pick turns, and 2e-2 (0.2) for a row where one does; 2.1e-6
    (8.6e-5) for float32."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 4e-4}
    return {"rel": 0.03, "max": 0.8} if "num_experts" in MODELS[case["model"]] else {"rel": 0.02, "max": 0.1}


# --- the same step in 64 bits -------------------------------------------------------------------------------

def _rms(x, weight, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight.double()


def _rotate(x, positions, theta):
    half = x.shape[-1] // 2
    f = theta ** (-torch.arange(half, dtype=torch.float64, device=x.device) / half)
    a = (positions.double()[:, None] * f)[:, None, :]
    lo, hi = x[..., :half], x[..., half:]
    return torch.cat((lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()), -1)


def _attend(q, k, v, start):
    """q [n, heads, hd] at positions from ``start`` on; k, v [kv heads, start + n, hd]; causal."""
    n, heads, hd = q.shape
    group = heads // k.shape[0]
    out = torch.empty_like(q)
    rows = max(1, (1 << 27) // (heads * k.shape[1]))
    for lo in range(0, n, rows):
        hi = min(n, lo + rows)
        part = q[lo:hi].view(hi - lo, k.shape[0], group, hd).permute(1, 2, 0, 3).reshape(k.shape[0], -1, hd)
        s = (part @ k.transpose(1, 2)) * hd ** -0.5
        s = s.view(k.shape[0], group, hi - lo, -1)
        at = start + torch.arange(lo, hi, device=q.device)
        s = s.masked_fill(torch.arange(k.shape[1], device=q.device)[None, :] > at[:, None], float("-inf"))
        o = s.softmax(-1).view(k.shape[0], group * (hi - lo), -1) @ v
        out[lo:hi] = o.view(k.shape[0], group, hi - lo, hd).permute(2, 0, 1, 3).reshape(hi - lo, heads, hd)
    return out


def _swiglu(x, gate, up, down):
    g = x @ gate.double().T
    return (torch.nn.functional.silu(g) * (x @ up.double().T)) @ down.double().T


def _experts(x, w, f, c):
    score = (x @ w[f + "gate.weight"].double().T).sigmoid()
    ids = (score + w[f + "expert_bias"].double()).topk(c["num_experts_per_tok"], -1).indices
    weight = score.gather(1, ids)
    weight = weight / (weight.sum(-1, keepdim=True) + 1e-6) * c["routed_scaling_factor"]
    out = torch.zeros_like(x)
    for e in range(c["num_experts"]):
        row, pick = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            gate, up = w[f + "experts.gate_up_proj"][e].chunk(2)
            out.index_add_(0, row, weight[row, pick, None] * _swiglu(x[row], gate, up, w[f + "experts.down_proj"][e]))
    return out


def exact(case, seed):
    c, segments, w = MODELS[case["model"]], _segments(case), _weights(case, seed)
    H, heads, eps, taps = c["hidden_size"], c["num_attention_heads"], c["norm_eps"], c["conv_L_cache"]
    nkv, hd = c["num_key_value_heads"], c["hidden_size"] // c["num_attention_heads"]
    cuts = [0]
    for n, _ in segments:
        cuts.append(cuts[-1] + n)
    spans = [(b, cuts[b], cuts[b + 1], start) for b, (_, start) in enumerate(segments)]
    fresh = all(start == 0 for _, start in segments)
    ids = torch.tensor([t for ts in _tokens(case, seed) for t in ts], device="cuda")
    x = w["model.embed_tokens.weight"][ids].double()
    out = {"logits": None, "conv": []}
    if fresh:
        out["kv"] = []
    for i, kind in enumerate(c["layer_types"]):
        p = f"model.layers.{i}."
        u = _rms(x, w[p + "operator_norm.weight"], eps)
        if kind == "conv":
            gate, c_gate, v = (u @ w[p + "conv.in_proj.weight"].double().T).chunk(3, -1)
            g, y = gate * v, torch.empty_like(v)
            states = []
            kernel = w[p + "conv.conv.weight"].double().reshape(H, taps)
            for b, lo, hi, start in spans:
                before = _held(case, seed, i, b, start).double() if start else g.new_zeros(taps - 1, H)
                rows = torch.cat((before, g[lo:hi]))
                y[lo:hi] = c_gate[lo:hi] * sum(rows[t:t + hi - lo] * kernel[:, t] for t in range(taps))
                states.append(rows[rows.shape[0] - taps + 1:])
            out["conv"].append(torch.stack(states))
            x = x + y @ w[p + "conv.out_proj.weight"].double().T
        else:
            a = p + "self_attn."
            heads_of = lambda name, n: (u @ w[a + name].double().T).view(-1, n, hd)
            at = torch.cat([torch.arange(start, start + hi - lo, device="cuda") for _, lo, hi, start in spans])
            q = _rotate(_rms(heads_of("q_proj.weight", heads), w[a + "q_layernorm.weight"], eps), at, c["rope_theta"])
            k = _rotate(_rms(heads_of("k_proj.weight", nkv), w[a + "k_layernorm.weight"], eps), at, c["rope_theta"])
            v = heads_of("v_proj.weight", nkv)
            o, pages = torch.empty_like(q), []
            for b, lo, hi, start in spans:
                new = torch.stack((k[lo:hi], v[lo:hi])).transpose(1, 2)
                if start:
                    new = torch.cat((_held(case, seed, i, b, start).double(), new), 2)
                o[lo:hi] = _attend(q[lo:hi], new[0], new[1], start)
                if fresh:
                    room = -(-(hi - lo) // PAGE)
                    new = torch.nn.functional.pad(new, (0, 0, 0, room * PAGE - (hi - lo)))
                    pages.append(new.unflatten(2, (room, PAGE)).permute(2, 0, 1, 3, 4))
            if fresh:
                out["kv"].append(torch.cat(pages))
            x = x + o.reshape(-1, H) @ w[a + "out_proj.weight"].double().T
        f = p + "feed_forward."
        u = _rms(x, w[p + "ffn_norm.weight"], eps)
        if i < c.get("num_dense_layers", c["num_hidden_layers"]):
            x = x + _swiglu(u, w[f + "w1.weight"], w[f + "w3.weight"], w[f + "w2.weight"])
        else:
            x = x + _experts(u, w, f, c)
    last = torch.tensor([hi - 1 for _, _, hi, _ in spans], device="cuda")
    h = _rms(x[last], w["model.embedding_norm.weight"], eps)
    out["logits"] = torch.cat([h @ part.double().T for part in w["model.embed_tokens.weight"].split(8192)], 1)
    return out
