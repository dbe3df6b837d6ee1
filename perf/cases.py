"""What the engine is asked to do in use, as a list of measurable cases.

Two kinds are whole calls of ``ModelRunner.step`` on the GQA model: a decode step of a batch over a long cache, and prompts.
The others are single layers of the registered architectures, called the way a model's block calls them: a part built from
its own constructor, its weights loaded by tensor name, its cache plane and state from the cache manager, its step laid
out by ``build_step``.  Layers of few rows (``captured``) run from a CUDA graph, as the engine runs its decode steps.

Sizes are those of the 0.9B and 3B members of the GQA family and of the other architectures laid out with the same layer
sizes, page size 16, prompts up to 2048 tokens a step and contexts up to 4096.

A case is a dict:

* ``kind``  ``decode_step`` | ``prompt`` | ``gqa_attention`` | ``window_attention`` | ``latent_attention`` |
  ``diff_attention`` | ``recurrence`` | ``swiglu`` | ``experts``
* ``size``  ``0.9b`` | ``3b`` (layer sizes);  ``dtype``  ``bf16`` | ``f32``
* ``requests``, ``history``, ``tokens``: that many requests, which already hold ``history`` tokens, feed ``tokens`` tokens in
  the step altogether, in shares of unequal length
* ``rule`` (recurrence): ``channel_delta`` | ``head_delta`` | ``decay`` | ``gated``
"""
import math

import torch

from tiny_inference_server_b200.cache.manager import CacheManager
from tiny_inference_server_b200.config import EngineConfig
from tiny_inference_server_b200.engine import ModelRunner, StepEntry, build_step
from tiny_inference_server_b200.parts.attention import GqaAttention
from tiny_inference_server_b200.parts.base import BuildContext, LayerBinding
from tiny_inference_server_b200.parts.delta_rule import ChannelDeltaRule, HeadDecayDeltaRule
from tiny_inference_server_b200.parts.diff_attention import DifferentialAttention
from tiny_inference_server_b200.parts.feed_forward import RoutedExperts, SwiGLU
from tiny_inference_server_b200.parts.gated_linear_attention import GatedLinearAttention
from tiny_inference_server_b200.parts.latent_attention import LatentAttention
from tiny_inference_server_b200.parts.linear_attention import DecayLinearAttention
from tiny_inference_server_b200.parts.positions import RotaryHalf, RotaryRescaled
from tiny_inference_server_b200.parts.window_attention import BiasedWindowAttention
from tiny_inference_server_b200.registry import build_model, config_from_dict

PAGE = 16
CONTEXT = 4096
SIZES = {"0.9b": {"width": 1536, "heads": 12, "kv_heads": 3, "ffn": 4096},
         "3b": {"width": 3072, "heads": 24, "kv_heads": 8, "ffn": 8192}}
DIM = 128                 # of every head, key and value
VOCAB = 49152
LAYERS = 8                # of the whole calls
WINDOW = 1024
RANK, ROT = 128, 64       # compressed keys and values: elements a token, rotated elements beside them
EXPERTS, TOP = 16, 3
DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
STD = 0.02                # of the random weights


def _case(name, kind, requests, tokens, history=0, size="0.9b", dtype="bf16", **more):
    c = {"kind": kind, "size": size, "dtype": dtype, "requests": requests, "history": history, "tokens": tokens}
    c.update(more)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a server with eight live chats, each some 4000 tokens long: one token for each of them
        _case("decode step 8 chats", "decode_step", 8, 8, CONTEXT - 8),
        # a document of 2048 tokens arrives: a step at the engine's token budget
        _case("prompt of 2048", "prompt", 1, 2048),
        # the same for its layers: two prompts that share a step
        _case("attention 2 prompts", "gqa_attention", 2, 2048),
        _case("feed-forward 2048 rows", "swiglu", 1, 2048),
        # a prompt through the windowed attention with a distance bias, in a step of its own
        _case("windowed attention prompt", "window_attention", 1, 2048),
        # the second half of a long document: compressed keys and values of the first half are in the cache
        _case("latent attention prompt", "latent_attention", 1, 1024, 1024),
        # eight chats through differential attention
        _case("diff attention 8 chats", "diff_attention", 8, 8, CONTEXT - 8),
        # a prompt through the delta rule
        _case("delta rule prompt", "recurrence", 1, 2048, rule="channel_delta"),
        # four prompts that share a step, in a larger model with gated linear attention
        _case("gated recurrence 4 prompts", "recurrence", 4, 2048, size="3b", rule="gated"),
        # an odd pair of short prompts in the 32-bit mode that checks and small experiments use
        _case("decay recurrence 32-bit", "recurrence", 2, 777, dtype="f32", rule="decay"),
        # routed experts behind a full prompt step and behind a decode step
        _case("experts 2048 rows", "experts", 1, 2048),
        _case("experts 8 rows", "experts", 8, 8),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode_step", "prompt", "gqa_attention", "window_attention", "latent_attention", "diff_attention",
                       "recurrence", "recurrence", "swiglu", "experts"])
    size = rng.choice(["0.9b", "0.9b", "3b"])
    if kind == "decode_step":
        n = _log_int(rng, 1, 32)
        return _case(None, kind, n, n, _log_int(rng, 200, CONTEXT - 8))
    if kind == "prompt":
        tokens = _log_int(rng, 65, 2048)
        return _case(None, kind, rng.randint(1, min(4, tokens // 64)), tokens)
    if kind == "recurrence":
        tokens = _log_int(rng, 65, 2048)
        return _case(None, kind, rng.randint(1, min(6, tokens // 16)), tokens, size=size,
                     dtype=rng.choice(["bf16", "bf16", "bf16", "f32"]),
                     rule=rng.choice(["channel_delta", "head_delta", "decay", "gated"]))
    if kind in ("swiglu", "experts"):
        return _case(None, kind, 1, _log_int(rng, 1, 2048), size="0.9b")
    if rng.random() < 0.3:
        n = _log_int(rng, 1, 32)
        return _case(None, kind, n, n, _log_int(rng, 200, CONTEXT - 8), size=size)
    tokens = _log_int(rng, 65, 2048)
    n = rng.randint(1, min(4, tokens // 16))
    return _case(None, kind, n, tokens, rng.choice([0, 0, _log_int(rng, 100, 2048)]), size=size)


# ---- inputs --------------------------------------------------------------------------------------------------------

def _shares(case):
    """Tokens of every request in the step: unequal where they are many, one each in a decode step."""
    n, total = case["requests"], case["tokens"]
    weights = [2 + (3 * i + 2) % 5 for i in range(n)]
    shares = [max(1, total * w // sum(weights)) for w in weights]
    shares[0] += total - sum(shares)
    return shares


def _wanted(tokens):
    """The places of a prompt whose logits are asked for: every sixteenth token (a prompt that is scored) and the last."""
    return sorted(set(range(15, tokens, 16)) | {tokens - 1})


def _captured(case):
    return case["tokens"] <= 64


def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _tensors(specs, gen, dtype):
    """Random weights by tensor name, as ``weights.random_init`` draws them, made on the device."""
    out = {}
    for name, s in specs.items():
        if s.init == "uniform":
            t = torch.rand(s.shape, generator=gen, device="cuda") * (s.hi - s.lo) + s.lo
        else:
            t = torch.randn(s.shape, generator=gen, device="cuda") * STD
            if s.init == "ones_normal":
                t = t + 1.0
        out[name] = t.to(s.dtype or dtype)
    return out


def _part(case):
    s, kind = SIZES[case["size"]], case["kind"]
    width, heads, kv = s["width"], s["heads"], s["kv_heads"]
    if kind == "gqa_attention":
        return GqaAttention(width, heads, kv, DIM, RotaryHalf(DIM, 10000.0, 2 * CONTEXT))
    if kind == "window_attention":
        return BiasedWindowAttention(width, heads, kv, DIM, DIM, DIM ** -0.5, WINDOW, 1e-6, conv_taps=4)
    if kind == "latent_attention":
        rot = RotaryRescaled(ROT, 1e6, 2 * CONTEXT, scaling={"factor": 8.0, "original": 2048, "fast": 32.0, "slow": 1.0})
        return LatentAttention(width, heads, 64, ROT, DIM, RANK, (64 + ROT) ** -0.5, 1e-6, rot)
    if kind == "diff_attention":
        return DifferentialAttention(width, heads, kv, 64, DIM, 64 ** -0.5, 0.25, 1e-6, q_temp=(0.2, 128))
    if kind == "swiglu":
        return SwiGLU(width, s["ffn"])
    if kind == "experts":
        hidden = s["ffn"] // (TOP + 1) // 32 * 32
        return RoutedExperts(width, hidden, EXPERTS, TOP, groups=4, keep=2, shared_hidden=hidden)
    rule = case["rule"]
    if rule == "channel_delta":
        return ChannelDeltaRule(width, heads, kv, DIM, DIM, 4, 1e-6, 64, 64)
    if rule == "head_delta":
        return HeadDecayDeltaRule(width, heads, kv, DIM, DIM, 4, 1e-6)
    if rule == "decay":
        return DecayLinearAttention(width, heads, DIM, DIM, [1.0 - 2.0 ** -(5 + i % 4) for i in range(heads)], 1e-6)
    return GatedLinearAttention(width, heads, DIM, DIM, 8.0, 64, 1e-6)


def _weights(part, gen, dtype):
    specs = {}
    for p in part.walk():
        specs.update(p.expected_tensors())
    return _tensors(specs, gen, dtype)


def _layer_inputs(case, seed):
    """(part, weights, inputs of the history, inputs of the step): rows of a normalised stream, one tensor a request."""
    gen, dtype = _generator(seed), DTYPES[case["dtype"]]
    part = _part(case)
    tensors = _weights(part, gen, dtype)
    width = SIZES[case["size"]]["width"]
    make = lambda n: torch.randn((n, width), generator=gen, device="cuda").to(dtype)  # noqa: E731
    shares = _shares(case)
    past = [make(case["history"]) for _ in shares]
    return part, tensors, past, [make(n) for n in shares]


def _model_config():
    s = SIZES["0.9b"]
    return dict(architecture="gqa_mtp_transformer", vocab_size=VOCAB, hidden_size=s["width"], num_layers=LAYERS,
                num_heads=s["heads"], num_kv_heads=s["kv_heads"], head_dim=DIM, ffn_hidden=s["ffn"], rms_norm_eps=2e-8,
                rope_theta=10000.0, max_context=CONTEXT, tie_word_embeddings=True, num_mtp_heads=0)


def _model_inputs(case, seed):
    gen = _generator(seed)
    cfg = config_from_dict(_model_config())
    tensors = _tensors(build_model(cfg).expected_tensors(), gen, DTYPES[case["dtype"]])
    shares = _shares(case)
    ids = [torch.randint(0, VOCAB, (case["history"] + n,), generator=gen, device="cuda") for n in shares]
    return cfg, tensors, ids, shares


def _prepare_model(case, seed):
    cfg, tensors, ids, shares = _model_inputs(case, seed)
    pages = sum(-(-len(t) // PAGE) + 1 for t in ids) + 8
    runner = ModelRunner(cfg, tensors, EngineConfig(page_size=PAGE, num_pages=pages, max_batch=max(8, len(ids)),
                                                    max_tokens_per_step=2048))
    del tensors
    ids = [t.tolist() for t in ids]
    state = {"kind": case["kind"], "runner": runner, "history": case["history"]}
    if case["kind"] == "prompt":
        state["prompts"] = [(t, _wanted(len(t))) for t in ids]
        return state
    slots = [runner.add_request() for _ in ids]
    for slot, t in zip(slots, ids):
        for a in range(0, case["history"], 2048):
            runner.step([StepEntry(slot, t[a:min(a + 2048, case["history"])])])
    runner.step_graphs.graphs.clear()
    state["slots"] = slots
    state["entries"] = [StepEntry(slot, t[case["history"]:], [0]) for slot, t in zip(slots, ids)]
    return state


def _layer_step(part, cache, slots, counts, fault):
    starts = [cache.extend(s, n) for s, n in zip(slots, counts)]
    cache.sync_tables()
    planners = part.step_planners() if hasattr(part, "step_planners") else ()
    step, _, _ = build_step([StepEntry(s, [0] * n) for s, n in zip(slots, counts)], starts, [0],
                            [g.table_dev for g in cache.groups], [PAGE] * len(cache.groups), fault, torch.device("cuda"), 1,
                            planners=planners)
    return step


def prepare(case, seed):
    if case["kind"] in ("decode_step", "prompt"):
        return _prepare_model(case, seed)
    part, tensors, past, new = _layer_inputs(case, seed)
    dtype = DTYPES[case["dtype"]]
    ctx = BuildContext(torch.device("cuda"), dtype)
    for p in part.walk():
        p.load(tensors, ctx)
    x = torch.cat(new)
    state = {"kind": case["kind"], "part": part, "x": x, "graph": None}
    if case["kind"] in ("swiglu", "experts"):
        call = lambda: part.forward(x)  # noqa: E731
    else:
        total = case["history"] + max(len(t) for t in new)
        kv, fixed = part.kv_spec(), part.state_spec()
        cache = CacheManager([kv], {"state": fixed} if fixed is not None else {}, page_size=PAGE,
                             num_pages=len(new) * (-(-total // PAGE) + 1), max_slots=len(new), max_positions=total + PAGE,
                             dtype=dtype, device=torch.device("cuda"))
        binding = LayerBinding(state=cache.states.get("state"))
        if cache.groups:
            grp, ref = cache.groups[0], cache.plane_refs[0]
            binding.kv_plane, binding.kv_group = grp.plane(ref.index), ref.group
            binding.k_pages, binding.v_pages = grp.key_pages(ref.index), grp.value_pages(ref.index)
        fault = torch.zeros(4, dtype=torch.int32, device="cuda")
        slots = [cache.admit() for _ in new]
        if case["history"]:
            for slot, t in zip(slots, past):
                part.forward(t, _layer_step(part, cache, [slot], [len(t)], fault), binding)
        step = _layer_step(part, cache, slots, [len(t) for t in new], fault)
        past_state = None if binding.state is None else binding.state.clone()
        state.update(binding=binding, step=step, cache=cache, past_state=past_state)
        call = lambda: part.forward(x, step, binding)  # noqa: E731
    if _captured(case):
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            call()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            state["out"] = call()
        state["graph"] = graph
    return state


def run(state):
    kind = state["kind"]
    if kind == "decode_step":
        runner = state["runner"]
        out = runner.step(state["entries"])
        for slot in state["slots"]:
            runner.cache.truncate(slot, state["history"])       # so that the same step can be taken again
        return out.main
    if kind == "prompt":
        runner = state["runner"]
        slots = [runner.add_request() for _ in state["prompts"]]
        out = runner.step([StepEntry(s, t, want) for s, (t, want) in zip(slots, state["prompts"])])
        for slot in slots:
            runner.release(slot)
        return out.main
    if state.get("past_state") is not None:
        state["binding"].state.copy_(state["past_state"])       # what the requests' state was before the step
    if state["graph"] is not None:
        state["graph"].replay()
        return state["out"]
    part, x = state["part"], state["x"]
    if kind in ("swiglu", "experts"):
        return part.forward(x)
    out = part.forward(x, state["step"], state["binding"])
    return (out, state["binding"].state) if kind == "recurrence" else out


# ---- what a pass cannot do without ---------------------------------------------------------------------------------

def _visible(case, window=None):
    """Pairs of a query row and a key it sees, and keys that any row of the step sees."""
    pairs = keys = 0
    for n in _shares(case):
        h = case["history"]
        for p in range(h, h + n):
            pairs += p + 1 if window is None else min(p + 1, window)
        keys += h + n if window is None else min(h + n, window + n)
    return pairs, keys


def work(case):
    s, kind = SIZES[case["size"]], case["kind"]
    e = 2 if case["dtype"] == "bf16" else 4
    width, heads, kv, ffn = s["width"], s["heads"], s["kv_heads"], s["ffn"]
    n = case["tokens"]
    rows = n * width * e * 2                                    # input and output
    if kind in ("decode_step", "prompt"):
        pairs, keys = _visible(case)
        per_layer = width * (heads + 2 * kv) * DIM + heads * DIM * width + 3 * width * ffn
        wanted = n if kind == "decode_step" else sum(len(_wanted(m)) for m in _shares(case))
        # every layer's weights, the output matrix, the cache (read what earlier steps left, write what is new), the logits
        cache = LAYERS * 2 * kv * DIM * (keys - n + n) * e
        return {"bytes": (LAYERS * per_layer + VOCAB * width) * e + cache + n * width * e + wanted * VOCAB * 4,
                "flops": 2.0 * n * LAYERS * per_layer + 4.0 * LAYERS * heads * DIM * pairs + 2.0 * wanted * VOCAB * width}
    if kind == "swiglu":
        return {"bytes": 3 * width * ffn * e + rows, "flops": 6.0 * n * width * ffn}
    if kind == "experts":
        hidden = ffn // (TOP + 1) // 32 * 32
        met = EXPERTS * (1.0 - (1.0 - TOP / EXPERTS) ** n)       # experts that some row meets
        return {"bytes": (3 * width * hidden * (met + 1) + EXPERTS * width) * e + rows,
                "flops": 6.0 * n * width * hidden * (TOP + 1) + 2.0 * n * width * EXPERTS}
    if kind == "recurrence":
        qk = kv if case["rule"] in ("channel_delta", "head_delta") else heads
        proj = width * (2 * qk + 2 * heads) * DIM + heads * DIM * width
        if case["rule"] == "channel_delta":
            proj = width * (2 * qk + heads) * DIM + heads * DIM * width + 128 * width + 64 * 2 * heads * DIM
        if case["rule"] == "gated":
            proj += 64 * width + 64 * heads * DIM
        steps = (3 if "delta" in case["rule"] else 2) * 2.0 * n * heads * DIM * DIM
        return {"bytes": proj * e + rows + case["requests"] * heads * DIM * DIM * 4, "flops": 2.0 * n * proj + steps}
    if kind == "gqa_attention":
        pairs, keys = _visible(case)
        proj = width * (heads + 2 * kv) * DIM + heads * DIM * width
        return {"bytes": proj * e + rows + 2 * kv * DIM * keys * e, "flops": 2.0 * n * proj + 4.0 * heads * DIM * pairs}
    if kind == "window_attention":
        pairs, keys = _visible(case, WINDOW)
        proj = width * (2 * heads + 2 * kv) * DIM + heads * DIM * width
        return {"bytes": proj * e + rows + 2 * kv * DIM * keys * e, "flops": 2.0 * n * proj + 4.0 * heads * DIM * pairs}
    if kind == "diff_attention":
        pairs, keys = _visible(case)
        proj = width * (heads + 2 * kv) * DIM + heads * DIM * width
        return {"bytes": proj * e + rows + 2 * kv * DIM * keys * e,
                "flops": 2.0 * n * proj + 2.0 * heads * (DIM + 2 * DIM) * pairs}
    pairs, keys = _visible(case)                                # latent attention
    proj = width * (heads * DIM + RANK + ROT) + heads * RANK * (64 + DIM) + heads * DIM * width
    return {"bytes": proj * e + rows + (RANK + ROT) * keys * e,
            "flops": 2.0 * n * proj + 2.0 * heads * (RANK + ROT + RANK) * pairs}


def tolerance(case):
    # about four times what the present kernels are off the same in 64 bits: 32-bit 9e-7 (sums of up to 1536 terms), layers in
    # bfloat16 0.0023 to 0.0048, differential attention (a difference of two maps, normed) 0.008, eight layers 0.011
    if case["dtype"] == "f32":
        return {"rel": 4e-6}
    return {"rel": {"decode_step": 4e-2, "prompt": 4e-2, "diff_attention": 3e-2}.get(case["kind"], 1.5e-2)}


# ---- the same in 64 bits, whole sequences, plain torch -------------------------------------------------------------

def _rope(x, positions, freqs, magnitude=1.0):
    """x (n, heads, 2 * len(freqs)): pairs (i, i + half)."""
    ang = torch.outer(positions.double(), freqs)
    c, s = (torch.cos(ang) * magnitude)[:, None], (torch.sin(ang) * magnitude)[:, None]
    a, b = x.chunk(2, -1)
    return torch.cat([a * c - b * s, b * c + a * s], -1)


def _softmax_attention(q, k, v, first, scale, window=None, bias=None, sink=None):
    """q (n, H, d) at positions first.., k (m, G, d), v (m, G, e) -> (n, H, e)."""
    n, H, _ = q.shape
    group = H // k.shape[1]
    out = torch.empty((n, H, v.shape[2]), dtype=q.dtype, device=q.device)
    kp = torch.arange(k.shape[0], device=q.device)
    qp = torch.arange(first, first + n, device=q.device)
    dist = qp[:, None] - kp[None]
    hidden = dist < 0 if window is None else (dist < 0) | (dist >= window)
    for h in range(H):
        s = q[:, h] @ k[:, h // group].t() * scale
        if bias is not None:
            s = s - bias[0][h] * torch.log1p(bias[1][h] * dist.clamp(min=0))
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(n, 1)], 1)
        p = torch.softmax(s, -1)
        out[:, h] = p[:, :k.shape[0]] @ v[:, h // group]
    return out


def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _conv(x, w, silu):
    """A causal convolution over time: x (n, C), w (C, taps)."""
    taps = w.shape[1]
    padded = torch.cat([x.new_zeros(taps - 1, x.shape[1]), x])
    y = sum(padded[j:j + x.shape[0]] * w[:, j] for j in range(taps))
    tail = padded[x.shape[0]:]
    return (torch.nn.functional.silu(y) if silu else y), tail


def _exact_gqa(part, w, x, first):
    H, G, d = part.num_heads, part.kv_heads, part.head_dim
    q, kv = x @ w["q_proj.weight"], x @ w["kv_proj.weight"]
    pos = torch.arange(len(x), device=x.device)
    freqs = 10000.0 ** (-2.0 * torch.arange(d // 2, dtype=torch.float64, device=x.device) / d)
    q = _rope(q.view(-1, H, d)[first:], pos[first:], freqs)
    k = _rope(kv[:, :G * d].reshape(-1, G, d), pos, freqs)
    o = _softmax_attention(q, k, kv[:, G * d:].reshape(-1, G, d), first, d ** -0.5)
    return o.flatten(1) @ w["linear_proj.weight"]


def _exact_window(part, w, x, first):
    H, G, d = part.num_heads, part.kv_heads, DIM
    q, k, v = (_conv(x @ w[n].t(), w[n + ".conv"], False)[0] for n in "qkv")
    q, k = _rms(q, part.eps) * w["q.norm"], _rms(k, part.eps) * w["k.norm"]
    o = _softmax_attention(q.view(-1, H, d)[first:], k.view(-1, G, d), v.view(-1, G, d), first, part.scale, part.window,
                           bias=(w["r1"], w["r2"]))
    return (o.flatten(1) * torch.sigmoid(x[first:] @ w["g"].t())) @ w["o"].t()


def _exact_latent(part, w, x, first):
    H, flat = part.num_heads, part.flat_dim
    freqs, magnitude = part.position.frequencies()
    freqs, pos = freqs.to(x.device), torch.arange(len(x), device=x.device)
    c = x @ w["dkv"].t()
    rot = _rope(c[:, None, RANK:], pos, freqs, magnitude)
    c = _rms(c[:, :RANK], part.eps) * w["dkv.norm"]
    q = (x[first:] @ w["q"].t()).view(-1, H, part.q_dim)
    q = torch.cat([q[..., :flat], _rope(q[..., flat:], pos[first:], freqs, magnitude)], -1)
    k = torch.cat([(c @ w["uk"].t()).view(-1, H, flat), rot.expand(-1, H, -1)], -1)
    o = _softmax_attention(q, k, (c @ w["uv"].t()).view(-1, H, part.v_dim), first, part.scale, sink=w["sink"])
    return o.flatten(1) @ w["o"].t()


def _exact_diff(part, w, x, first):
    H, G, d = part.num_heads, part.kv_heads, part.dim
    q = _rms((x[first:] @ w["q"].t() + w["q.b"]).view(-1, H, 2, d), part.eps) * w["q.norm"]
    k = _rms((x @ w["k"].t() + w["k.b"]).view(-1, G, 2, d), part.eps) * w["k.norm"]
    v = (x @ w["v"].t() + w["v.b"]).view(-1, G, part.v_dim)
    pos = torch.arange(first, len(x), device=x.device).double()
    temp = 1.0 + part.temp_coef * torch.log(torch.floor((pos + 1) / part.temp_every) + 1.0)
    q = q * temp[:, None, None, None]
    a = [_softmax_attention(q[:, :, m], k[:, :, m], v, first, part.scale) for m in (0, 1)]
    lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + part.diff
    return (_rms(a[0] - lam * a[1], part.eps) * (1.0 - part.diff)).flatten(1) @ w["o"].t()


def _exact_recurrence(part, rule, w, x):
    """(output rows, state of the request as the part keeps it)."""
    n, H, kd, vd = len(x), part.num_heads, part.k_dim, part.v_dim
    delta = rule in ("channel_delta", "head_delta")
    q, k, v = x @ w["q"].t(), x @ w["k"].t(), x @ w["v"].t()
    tails = []
    if delta:
        (q, tq), (k, tk), (v, tv) = (_conv(t, w[m + ".conv"], True) for t, m in ((q, "q"), (k, "k"), (v, "v")))
        tails = [torch.cat([tq, tk, tv], 1).flatten()]
        group = H // part.qk_heads
        q, k = (t.view(n, -1, kd) for t in (q, k))
        q, k = (t / torch.sqrt((t * t).sum(-1, keepdim=True) + part.UNIT_EPS) for t in (q, k))
        q, k = (q * kd ** -0.5).repeat_interleave(group, 1), k.repeat_interleave(group, 1)
        beta = torch.sigmoid(x @ w["b"].t())
        if rule == "channel_delta":
            a = ((x @ w["a1"].t()) @ w["a2"].t() + w["dt_bias"]).view(n, H, kd)
            gate = torch.sigmoid((x @ w["g1"].t()) @ w["g2"].t())
        else:
            a = (x @ w["a"].t() + w["dt_bias"])[..., None].expand(n, H, kd)
            gate = torch.nn.functional.silu(x @ w["g"].t())
        g = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a))
    else:
        q, k = q.view(n, H, kd), k.view(n, H, kd)
        if rule == "decay":
            q, k, v = (torch.nn.functional.silu(t) for t in (q, k, v))
            g = torch.tensor(part.decay_values, dtype=x.dtype, device=x.device)[None, :, None].expand(n, H, kd)
            gate = torch.sigmoid(x @ w["g"].t())
        else:
            q = q * kd ** -0.5
            z = ((x @ w["a1"].t()) @ w["a2"].t() + w["a2.b"]).view(n, H, kd)
            g = torch.exp(-torch.nn.functional.softplus(-z) / part.tau)
            gate = torch.nn.functional.silu(x @ w["g"].t())
    v = v.view(n, H, vd)
    S = x.new_zeros(H, kd, vd)
    o = x.new_empty(n, H, vd)
    for t in range(n):
        S = S * g[t][..., None]
        u = v[t]
        if delta:
            u = beta[t][:, None] * (u - torch.bmm(k[t][:, None], S)[:, 0])
        S = torch.baddbmm(S, k[t][..., None], u[:, None])
        o[t] = torch.bmm(q[t][:, None], S)[:, 0]
    if rule == "decay":
        y = _rms(o.flatten(1), part.eps) * w["norm"]
    else:
        y = (_rms(o, part.eps) * w["norm"]).flatten(1)
    return (y * gate) @ w["o"].t(), torch.cat([S.flatten()] + tails)


def _exact_experts(part, w, x):
    s = torch.sigmoid(x @ w["router"].t())
    pick = s + w["correction"]
    n, per = len(x), part.experts // part.groups
    strength = pick.view(n, part.groups, per).topk(2, -1).values.sum(-1)
    kept = torch.zeros_like(strength).scatter(1, strength.topk(part.keep, -1).indices, 1.0).bool()
    pick = pick.masked_fill(~kept.repeat_interleave(per, 1), -math.inf)
    chosen = torch.zeros_like(pick).scatter(1, pick.topk(part.top, -1).indices, 1.0)
    weight = s * chosen
    weight = weight / weight.sum(-1, keepdim=True)
    silu = torch.nn.functional.silu
    y = torch.sigmoid(x @ w["shared.sg"].t()) * ((silu(x @ w["shared.gate"].t()) * (x @ w["shared.up"].t())) @ w["shared.down"].t())
    for e in range(part.experts):
        y = y + weight[:, e:e + 1] * ((silu(x @ w[f"e{e}.gate"].t()) * (x @ w[f"e{e}.up"].t())) @ w[f"e{e}.down"].t())
    return y


def _exact_model(case, seed):
    cfg, tensors, ids, shares = _model_inputs(case, seed)
    w = {k: v.double() for k, v in tensors.items()}
    part = GqaAttention(cfg.hidden_size, cfg.num_heads, cfg.num_kv_heads, DIM, None)
    norm = lambda x, scale: x * math.sqrt(cfg.hidden_size) / (x.norm(dim=-1, keepdim=True) + cfg.rms_norm_eps) * scale  # noqa: E731
    out = []
    for t, n in zip(ids, shares):
        x = w["embedding.weight"][t]
        for i in range(LAYERS):
            p = f"transformer_block_list.{i}."
            block = {k[len(p):]: v for k, v in w.items() if k.startswith(p)}
            attention = {k[len("att."):]: v for k, v in block.items() if k.startswith("att.")}
            x = x + _exact_gqa(part, attention, norm(x, block["att.rms_norm_att.scale"]), 0)
            h = norm(x, block["rms_norm_ffn.scale"])
            gated = torch.nn.functional.silu(h @ block["ffn.swig.linear1.weight"]) * (h @ block["ffn.swig.linear2.weight"])
            x = x + gated @ block["ffn.fc.weight"]
        rows = [len(t) - n] if case["kind"] == "decode_step" else _wanted(n)
        out.append(norm(x[rows], w["rms_out.scale"]) @ w["embedding.weight"].t())
    return torch.cat(out)


def exact(case, seed):
    if case["kind"] in ("decode_step", "prompt"):
        if case["requests"] * (case["history"] + 1) > 40000:
            return None
        return _exact_model(case, seed)
    part, tensors, past, new = _layer_inputs(case, seed)
    w = {k: v.double() for k, v in tensors.items()}
    if case["kind"] == "swiglu":
        x = torch.cat(new).double()
        gated = torch.nn.functional.silu(x @ w["swig.linear1.weight"]) * (x @ w["swig.linear2.weight"])
        return gated @ w["fc.weight"]
    if case["kind"] == "experts":
        return _exact_experts(part, w, torch.cat(new).double())
    if case["kind"] == "recurrence":
        got = [_exact_recurrence(part, case["rule"], w, t.double()) for t in new]
        return torch.cat([y for y, _ in got]), torch.stack([s for _, s in got])
    layer = {"gqa_attention": _exact_gqa, "window_attention": _exact_window, "latent_attention": _exact_latent,
             "diff_attention": _exact_diff}[case["kind"]]
    return torch.cat([layer(part, w, torch.cat([a, b]).double(), len(a)) for a, b in zip(past, new)])
