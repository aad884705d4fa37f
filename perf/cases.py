"""The steps that the engine's speed is measured on: sizes, inputs, one pass, what a pass has to move and compute, and the
same results in 64 bits.

A case is one step of ``StepFunction``, which is what the engine, the scheduler and the replay program all run: ``rows``
requests that decode one token each behind contexts spread from ``low`` to ``high`` cached tokens (through the captured
graph, sampled and read back, as ``Engine.step`` runs them), ``prompts`` prompt portions of ``tokens`` tokens in all
(the first of them continues a prompt of which ``resume`` tokens are cached; a lone prompt longer than the engine's
default budget of 8192 tokens goes in portions of that size), or both in one mixed step.  Weights are seeded random
numbers, the contents of the cache and the token ids too; nothing is shared between two seeds.
"""
import math
import random

import torch

from llmserver_b200.cache import CacheManager
from llmserver_b200.cli import harness
from llmserver_b200.config import Qwen3Config
from llmserver_b200.config.registry import ARCHITECTURES
from llmserver_b200.engine.step import StepFunction
from llmserver_b200.models.decoder import DecoderModel
from llmserver_b200.parts import Runtime
from llmserver_b200.sampling import SamplingRow
from llmserver_b200.weights import RandomSource

DEVICE = "cuda:0"
PAGE = 16
BUDGET = 8192
MAX_CONTEXT = 4096      # what decode graphs are captured for
WINDOW = 1024           # of the differential-attention layers below
F = torch.float64

# a tiny float32 model: every option of the dense decoder away from its usual value
TINY = dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", vocab_size=509, hidden_size=96, intermediate_size=224,
            num_hidden_layers=3, num_attention_heads=6, num_key_value_heads=1, head_dim=32, rope_theta=1000000.0,
            rms_norm_eps=1e-5, tie_word_embeddings=False, max_position_embeddings=4096, hidden_act="silu",
            attention_bias=False, use_sliding_window=False)


def _case(name, model, rows=0, low=0, high=0, prompts=0, tokens=0, resume=0):
    return {"name": name, "model": model, "rows": rows, "low": low, "high": high, "prompts": prompts, "tokens": tokens, "resume": resume}


def listed():
    return [
        # one chat user: latency of a token
        _case("qwen3-8b decode 1", "qwen3-8b", rows=1, low=3072, high=3072),
        # the headline workload: 2048-token prompts decoded to 4096
        _case("qwen3-8b decode 8", "qwen3-8b", rows=8, low=3072, high=3072),
        # a busy server: many requests of any age, not a full bucket
        _case("qwen3-8b decode 61", "qwen3-8b", rows=61, low=301, high=4077),
        # first token of a short question, of the headline prompt, and of a document
        _case("qwen3-8b prompt 119", "qwen3-8b", prompts=1, tokens=119),
        _case("qwen3-8b prompt 2048", "qwen3-8b", prompts=1, tokens=2048),
        _case("qwen3-8b prompt 16384", "qwen3-8b", prompts=1, tokens=16384),
        # continuous batching: running requests decode while ragged prompts fill the token budget
        _case("qwen3-14b mixed 8192", "qwen3-14b", rows=21, low=140, high=2300, prompts=7, tokens=8171, resume=700),
        # the 32-bit path on a model that weighs nothing: launches and latency
        _case("tiny float32 decode 4", "tiny", rows=4, low=20, high=150),
        # routed experts, attention sinks
        _case("gefarax decode 24", "gefarax", rows=24, low=517, high=4003),
        _case("gefarax prompt 2048", "gefarax", prompts=1, tokens=2048),
        # differential attention over a window, linear attention, latent attention
        _case("dikusun decode 64", "dikusun", rows=64, low=900, high=4001),
        _case("dikusun prompt 2048", "dikusun", prompts=1, tokens=2048),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    base = rng.choice(listed())
    rows, low, high, prompts, tokens, resume = 0, 0, 0, 0, 0, 0
    if base["rows"]:
        most = {"qwen3-14b": 32, "tiny": 16}.get(base["model"], 64)
        longest = 200 if base["model"] == "tiny" else 4080
        rows = _spread(rng, 1, most)
        low, high = sorted(_spread(rng, 16, longest) for _ in range(2))
    if base["prompts"]:
        many = base["prompts"] > 1
        tokens = _spread(rng, 512 if many else 17, {"qwen3-8b": 16384, "qwen3-14b": BUDGET - rows}.get(base["model"], 4096))
        prompts, resume = (rng.randint(1, 9), rng.randrange(2049)) if many else (1, 0)
    return {key: value for key, value in _case("", base["model"], rows, low, high, prompts, tokens, resume).items() if key != "name"}


# ------------------------------------------------------------------------------------------------------ what is run
def _config(case):
    model = case["model"]
    if model == "gefarax":
        return harness.gefarax_config(harness.GEFARAX_SIZES["w4096-h128"], 4)
    if model == "dikusun":
        return harness.dikusun_config(harness.DIKUSUN_SIZES["w4096-mixed"])
    return Qwen3Config.from_dict(TINY if model == "tiny" else harness.SHAPES[model[6:]])


def _dtype(case):
    return torch.float32 if case["model"] == "tiny" else torch.bfloat16


def _shares(case):
    """(tokens cached, new tokens) of every request of the step: decoding requests, then prompt portions."""
    shares = []
    for row in range(case["rows"]):
        context = case["low"] + (case["high"] - case["low"]) * row // max(1, case["rows"] - 1)
        # a pass is repeated at the same place: stay off the token with which a window gives a page back
        shares.append((context + (context - WINDOW) % PAGE // (PAGE - 2) % 2, 1))
    left, weights = case["tokens"], list(range(3, 3 + case["prompts"]))
    for portion, weight in enumerate(weights):
        count = left if portion == len(weights) - 1 else max(1, case["tokens"] * weight // sum(weights))
        left -= count
        shares.append((case["resume"] if portion == 0 else 0, count))
    return shares


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(seed)


class _Weights(RandomSource):
    """Seeded random weights, of such sizes that the stream is made as a trained model's is: the embedded tokens are not small beside
    what the layers add, and deep dense models add a little per layer (their output projections shrink with the depth).  In models
    with routed experts the tokens fall into as many classes as there are experts, and a class's tokens clearly prefer its
    neighbouring experts: as trained routers have it, a choice does not hang on the last bit."""

    def get(self, name):
        tensor = super().get(name)
        if name.endswith(("o_proj.weight", "down_proj.weight")):
            outputs = sum(other.endswith(("o_proj.weight", "down_proj.weight")) for other in self.wanted)
            return (tensor.float() * outputs ** -0.5).to(tensor.dtype)
        if name not in ("model.embed_tokens.weight", "embed") and not name.endswith("mlp.router"):
            return tensor
        routers = [other for other in self.wanted if other.endswith("mlp.router")]
        if not routers:
            return (tensor.float() * 50.0).to(tensor.dtype)
        experts, width = self.wanted[routers[0]].shape
        classes = torch.randn((experts, width), generator=_generator(self.seed), device=self.device)
        if name == "embed":
            return (tensor.float() * 125.0 + 2.5 * classes[torch.arange(tensor.shape[0], device=self.device) % experts]).to(tensor.dtype)
        router = tensor * 0.2 + 5.0 / width * sum(classes.roll(shift, 0) for shift in range(6))
        return router.to(torch.bfloat16).to(torch.float32)      # what a bfloat16 checkpoint holds


def _source(case, seed):
    config = _config(case)
    spec = ARCHITECTURES[config.architecture].build_spec(config)
    return spec, _Weights(spec, seed, _dtype(case), torch.device(DEVICE))


def prepare(case, seed):
    spec, source = _source(case, seed)
    model = DecoderModel(spec, source, Runtime(_dtype(case), torch.device(DEVICE)))
    shares = _shares(case)
    pages = sum(-(-(start + count) // PAGE) for start, count in shares) + 9
    cache = CacheManager(model.cache_needs(), PAGE, pages, num_slots=len(shares), prefix_sharing=False)
    cache.materialize(model.runtime.device, model.runtime.dtype)
    step = StepFunction(model, cache)
    rng = random.Random(seed)
    fresh = [[rng.randrange(spec.vocab_size) for _ in range(count)] for _, count in shares]
    state = {"step": step, "shares": shares, "graph": None, "sampling": None,
             "entries": [(row, tokens, [len(tokens) - 1]) for row, tokens in enumerate(fresh)]}
    if not case["rows"]:
        return state
    for row, (start, count) in enumerate(shares):
        step.admit(row)
        cache.ensure(row, start + count)
        cache.advance(row, start)
        step.computed[row] = start
    if not case["prompts"]:
        step.enable_graphs(MAX_CONTEXT, 64)
        hot = case["model"] == "tiny"
        state["sampling"] = [SamplingRow(0.8 if hot else 0.0, seed + row, start) for row, (start, _) in enumerate(shares)]
        while not step.graph_steps:      # an engine that has been warmed up has its graphs
            _decode(state)
        state["graph"] = step.graphs.graphs[step.graphs.bucket_for(len(shares))]
    generator = _generator(seed + 1)
    for group in cache.groups:
        for tensor in (group.key_storage, group.value_storage):
            tensor.normal_(0.0, 1.0, generator=generator)
    for tensor in cache.slots.storage.values():
        tensor.normal_(0.0, 1.0, generator=generator)
    return state


def _decode(state):
    step = state["step"]
    step.run_and_sample(state["entries"], state["sampling"])
    for row, (start, _) in enumerate(state["shares"]):
        step.computed[row] = start       # the same step again the next time


def run(state):
    """Logits of the step; the recurrent states of its requests; where prompts ran, the pages that they filled."""
    step, shares = state["step"], state["shares"]
    cache = step.cache
    states = [tensor[:len(shares)] for tensor in cache.slots.storage.values()]
    if state["graph"] is not None:
        _decode(state)
        return {"logits": state["graph"].logits[:len(shares)], "states": states}
    if len(shares) > 1:
        logits = step.run(state["entries"])
        for row, (start, _) in enumerate(shares):
            step.computed[row] = start
    else:
        (_, tokens, _), = state["entries"]
        step.admit(0)
        for begin in range(0, len(tokens), BUDGET):
            part = tokens[begin:begin + BUDGET]
            logits = step.run([(0, part, [len(part) - 1] if begin + BUDGET >= len(tokens) else [])])
        step.release(0)
    return {"logits": logits, "states": states,
            "pages": [tensor for group in cache.groups for tensor in (group.key_storage, group.value_storage)]}


# ------------------------------------------------------------------------------------------------------ what it costs
def work(case):
    """Every weight of the step once (of routed experts those that its tokens are expected to choose), the cached keys, values
    and states that it reads and writes, its logits; the products of its tokens, attention over its (query, key) pairs."""
    config, shares = _config(case), _shares(case)
    new = sum(count for _, count in shares)
    held = sum(start + count for start, count in shares)
    pairs = sum(count * start + count * (count + 1) / 2 for start, count in shares)
    if case["model"] == "gefarax":
        moved, flops = harness.gefarax_step_cost(harness.GEFARAX_SIZES["w4096-h128"], 4, new, held, pairs)
    elif case["model"] == "dikusun":
        costs = [harness.dikusun_step_cost(harness.DIKUSUN_SIZES["w4096-mixed"], 4, count, 1, start) for start, count in shares]
        weights = harness.dikusun_step_cost(harness.DIKUSUN_SIZES["w4096-mixed"], 4, 0, 1, 0)[0]
        states = 2 * 4 * 32 * 64 * 128      # the linear-attention layer's state of a request, which ``weights`` counts too
        moved, flops = sum(cost[0] - weights + states for cost in costs) + weights - states, sum(cost[1] for cost in costs)
    else:
        layers = config.num_hidden_layers
        moved = harness.weight_bytes(config, layers) + harness.cache_bytes_per_token(config, layers) * held
        moved *= 2 if case["model"] == "tiny" else 1
        flops = harness.linear_flops_per_token(config, layers) * new + harness.attention_flops(config, layers, pairs)
    return {"bytes": moved + 4 * len(shares) * config.vocab_size, "flops": flops + 2 * len(shares) * config.vocab_size * config.hidden_size}


def tolerance(case):
    """About four times what the framework's own variants of its kernels (other splits, separate instead of fused kernels, the
    library's products) differ by on one set of inputs: 0.009 over 36 and 40 layers, 0.004 over Gefarax's 4, 0.007 over Dikusun's
    4 (0.06, 0.02 and 0.034 at the worst value); 32-bit results are 2e-7 to 8e-7 off their 64-bit values."""
    return {"tiny": {"rel": 4e-6}, "gefarax": {"rel": 0.016, "max": 0.1}, "dikusun": {"rel": 0.028, "max": 0.15}}.get(
        case["model"], {"rel": 0.03, "max": 0.25})


# ------------------------------------------------------------------------------------------------------ in 64 bits
def _norm(x, weight, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if weight is None else y * weight


def _turn(x, positions, frequencies, magnitude=1.0):
    """x [T, ..., dim]: element i turns with element i + dim / 2."""
    half = x.shape[-1] // 2
    angle = (positions.to(F)[:, None] * frequencies).view([-1] + [1] * (x.dim() - 2) + [half])
    cos, sin = torch.cos(angle) * magnitude, torch.sin(angle) * magnitude
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)


def _frequencies(base, dims):
    return base ** (-torch.arange(0, dims, 2, dtype=F, device=DEVICE) / dims)


def _stretched(base, dims, factor, original, fast, slow):
    """The stretched frequencies of long contexts, and the factor on the turned values."""
    def pair(turns):
        return dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))

    low, high = max(math.floor(pair(fast)), 0), min(math.ceil(pair(slow)), dims - 1)
    plain = _frequencies(base, dims)
    ramp = ((torch.arange(dims // 2, dtype=F, device=DEVICE) - low) / max(high - low, 0.001)).clamp(0.0, 1.0)
    return plain / factor * ramp + plain * (1.0 - ramp), 0.1 * math.log(factor) + 1.0


def _attend(q, k, v, start, scale, window=None, sink=None, cap=None):
    """q [n, heads, dim] at positions start .. start + n - 1 against k [t, groups, dim], v [t, groups, vdim]."""
    n, heads, _ = q.shape
    t, groups, vdim = v.shape
    out = torch.empty((n, heads, vdim), dtype=F, device=q.device)
    per = heads // groups
    keys = torch.arange(t, device=q.device)
    rows = max(1, (1 << 26) // (t * per))
    for group in range(groups):
        mine = slice(group * per, (group + 1) * per)
        for first in range(0, n, rows):
            last = min(n, first + rows)
            seen = min(t, start + last)
            scores = torch.einsum("nhd,td->hnt", q[first:last, mine], k[:seen, group]) * scale
            if cap:
                scores = cap * torch.tanh(scores / cap)
            distance = torch.arange(start + first, start + last, device=q.device)[:, None] - keys[None, :seen]
            hidden = distance < 0
            if window:
                hidden |= distance >= window
            scores.masked_fill_(hidden, -math.inf)
            if sink is not None:
                scores = torch.cat([scores, sink[mine][:, None, None].expand(per, last - first, 1)], dim=2)
            weights = torch.softmax(scores, dim=-1)[..., :seen]
            out[first:last, mine] = torch.einsum("hnt,td->nhd", weights, v[:seen, group])
    return out


class _Past:
    """What each request's cache held before the step."""

    def __init__(self, state):
        self.cache, self.shares = state["step"].cache, state["shares"]

    def rows(self, layer, row):
        """The cached keys and values of a layer, [start, heads, dim] each; None where nothing is cached."""
        start = self.shares[row][0]
        if not start:
            return None
        keys, values, group = self.cache.pages_of_entry(layer)
        table = torch.tensor(self.cache.table(row, group)[:-(-start // PAGE)], device=DEVICE).clamp(min=0)
        return [t[table].transpose(1, 2).flatten(0, 1)[:start].to(F) for t in (keys, values)]

    def with_new(self, layer, row, k, v):
        past = self.rows(layer, row)
        return (k, v) if past is None else (torch.cat([past[0], k]), torch.cat([past[1], v]))

    def state(self, layer, row):
        return self.cache.state_of_entry(layer)[row].to(F)


def exact(case, seed):
    state = prepare(case, seed)
    spec, source = _source(case, seed)
    shares, past, config = state["shares"], _Past(state), _config(case)
    if not case["rows"]:
        past.cache.admit(0)              # a new request's state is zero
    pieces, positions, first = [], [], 0
    for start, count in shares:
        pieces.append(slice(first, first + count))
        positions.append(torch.arange(start, start + count, device=DEVICE))
        first += count

    def weight(name):
        return source.get(name).to(F)

    tokens = torch.tensor([token for _, mine, _ in state["entries"] for token in mine], device=DEVICE)
    x = source.get(spec.embedding_name)[tokens].to(F)
    layer_of = {"Qwen3ForCausalLM": _qwen3_layer, "Gefarax": _gefarax_layer, "Dikusun": _dikusun_layer}[config.architecture]
    states = []
    for layer in range(len(spec.layers)):
        x = layer_of(x, layer, config, weight, past, pieces, positions, states)
    x = x[[piece.stop - 1 for piece in pieces]]
    eps = config.rms_norm_eps if hasattr(config, "rms_norm_eps") else config.norm_eps
    logits = _norm(x, weight("final.norm" if spec.embedding_name == "embed" else "model.norm.weight"), eps) @ weight(spec.head_name).T
    answer = {"logits": logits, "states": states}
    if state["graph"] is None:
        # where a page comes to lie is not a computed number
        answer["pages"] = [None for group in past.cache.groups for _ in range(2)]
    return answer


def _qwen3_layer(x, layer, config, weight, past, pieces, positions, states):
    name, eps, dim = f"model.layers.{layer}.", config.rms_norm_eps, config.head_dim
    h = _norm(x, weight(name + "input_layernorm.weight"), eps)
    q, k, v = ((h @ weight(f"{name}self_attn.{part}_proj.weight").T).view(len(h), -1, dim) for part in "qkv")
    q, k = (_norm(part, weight(f"{name}self_attn.{role}_norm.weight"), eps) for part, role in ((q, "q"), (k, "k")))
    frequencies = _frequencies(config.rope_theta, dim)
    out = []
    for row, (piece, places) in enumerate(zip(pieces, positions)):
        keys, values = past.with_new(layer, row, _turn(k[piece], places, frequencies), v[piece])
        out.append(_attend(_turn(q[piece], places, frequencies), keys, values, int(places[0]), dim ** -0.5).flatten(1))
    x = x + torch.cat(out) @ weight(name + "self_attn.o_proj.weight").T
    h = _norm(x, weight(name + "post_attention_layernorm.weight"), eps)
    gate = h @ weight(name + "mlp.gate_proj.weight").T
    return x + (gate * torch.sigmoid(gate) * (h @ weight(name + "mlp.up_proj.weight").T)) @ weight(name + "mlp.down_proj.weight").T


def _clamped(h, weight, prefix, limit):
    gate = (h @ weight(prefix + "gate").T).clamp(max=limit)
    up = (h @ weight(prefix + "up").T).clamp(-limit, limit)
    return (gate * torch.sigmoid(1.702 * gate) * (up + 1.0)) @ weight(prefix + "down").T


def _gefarax_layer(x, layer, config, weight, past, pieces, positions, states):
    name, eps, mixer, mlp = f"l{layer}.", config.norm_eps, config.layers[layer].mixer, config.layers[layer].mlp
    h = _norm(x, weight(name + "norm1"), eps)
    q, k, v = ((h @ weight(name + "mix." + part).T).view(len(h), -1, mixer["dim"] if part in "qk" else mixer["vdim"]) for part in "qkv")
    rot = mixer["rot"]
    turn = _stretched(rot["base"], rot["dims"], **rot["scaling"])
    out = []
    for row, (piece, places) in enumerate(zip(pieces, positions)):
        keys, values = past.with_new(layer, row, _turn(k[piece], places, *turn), v[piece])
        out.append(_attend(_turn(q[piece], places, *turn), keys, values, int(places[0]), mixer["scale"], sink=weight(name + "mix.sink")).flatten(1))
    x = x + _norm(torch.cat(out) @ weight(name + "mix.o").T, weight(name + "norm1b"), eps)
    h = _norm(x, weight(name + "norm2"), eps)
    scores = torch.sigmoid(h @ weight(name + "mlp.router").T)
    chosen = torch.topk(scores + weight(name + "mlp.correction"), mlp["router"]["top"], dim=-1).indices
    y = _clamped(h, weight, name + "mlp.shared.", mlp["shared"]["limit"])
    for expert in range(mlp["router"]["experts"]):
        rows = (chosen == expert).any(-1).nonzero()[:, 0]
        if len(rows):
            y[rows] += _clamped(h[rows], weight, f"{name}mlp.e{expert}.", mlp["expert"]["limit"]) * (scores[rows, expert] * mlp["router"]["scale"])[:, None]
    return x + _norm(y, weight(name + "norm2b"), eps)


def _dikusun_layer(x, layer, config, weight, past, pieces, positions, states):
    entry = config.layers[layer]
    name, eps, mixer = f"l{layer}.", config.norm_eps, entry.mixer
    mixed = {"attention": _differential, "latent_attention": _latent, "gla": _linear_attention}[entry.type](
        x, layer, mixer, eps, lambda part: weight(f"{name}mix.{part}"), past, pieces, positions, states)
    x = x + _norm(mixed, weight(name + "norm1"), eps)
    return x + _norm(_clamped(x, weight, name + "mlp.", entry.mlp["limit"]), weight(name + "norm2"), eps)


def _differential(h, layer, mixer, eps, weight, past, pieces, positions, states):
    dim, vdim, diff = mixer["dim"], mixer["vdim"], mixer["diff"]
    q, k, v = (h @ weight(part).T + weight(part + ".b") for part in "qkv")
    frequencies = _frequencies(mixer["rot"]["base"], dim)
    lam = torch.exp((weight("lq1") * weight("lk1")).sum()) - torch.exp((weight("lq2") * weight("lk2")).sum()) + diff
    q, k = (_norm(part.view(len(h), -1, 2, dim), weight(role), eps) for part, role in ((q, "q.norm"), (k, "k.norm")))
    out = []
    for row, (piece, places) in enumerate(zip(pieces, positions)):
        turned = _turn(q[piece], places, frequencies)
        keys, values = past.with_new(layer, row, _turn(k[piece], places, frequencies).flatten(2), v[piece].view(len(places), -1, vdim))
        maps = [_attend(turned[:, :, m], keys[..., m * dim:(m + 1) * dim], values, int(places[0]), mixer["scale"], mixer["mask"]["size"],
                        cap=mixer["softcap"]) for m in range(2)]
        out.append(_norm(maps[0] - lam * maps[1], None, eps) * (1.0 - diff))
    gated = torch.cat(out) * torch.sigmoid(h @ weight("g").T)[:, :, None]
    return gated.flatten(1) @ weight("o").T + weight("o.b")


def _latent(h, layer, mixer, eps, weight, past, pieces, positions, states):
    heads = mixer["heads"]
    q = (_norm(h @ weight("dq").T, weight("dq.norm"), eps) @ weight("uq").T).view(len(h), heads, -1)
    latent = _norm(h @ weight("dkv").T, weight("dkv.norm"), eps)[:, None]
    out = []
    for row, (piece, places) in enumerate(zip(pieces, positions)):
        cached = past.with_new(layer, row, latent[piece], latent[piece])[0][:, 0]
        keys, values = ((cached @ weight(part).T).view(len(cached), heads, -1) for part in ("uk", "uv"))
        out.append(_attend(q[piece], keys, values, int(places[0]), mixer["scale"]).flatten(1))
    return torch.cat(out) @ weight("o").T


def _linear_attention(h, layer, mixer, eps, weight, past, pieces, positions, states):
    heads, dim, vdim = mixer["heads"], mixer["dim"], mixer["vdim"]
    q, k, v = ((h @ weight(part).T).view(len(h), heads, -1) for part in "qkv")
    decay = torch.sigmoid((h @ weight("a1").T) @ weight("a2").T + weight("a2.b")).pow(1.0 / mixer["tau"]).view(-1, heads, dim)
    out, after = torch.empty((len(h), heads, vdim), dtype=F, device=h.device), []
    for row, piece in enumerate(pieces):
        held = past.state(layer, row)
        for t in range(piece.start, piece.stop):
            held = decay[t][:, :, None] * held + k[t][:, :, None] * v[t][:, None, :]
            out[t] = torch.einsum("hdv,hd->hv", held, q[t] * dim ** -0.5)
        after.append(held)
    states.append(torch.stack(after))
    gate = h @ weight("g").T
    return (_norm(out, weight("norm"), eps).flatten(1) * gate * torch.sigmoid(gate)) @ weight("o").T
