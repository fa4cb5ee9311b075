"""The work that a user of this engine has it do, as cases that can be timed and checked one by one.

Two kinds of case. ``model``: a Qwen3 decoder served through ``ModelRunner.step``, prompts in one step and then single
tokens. All others: one part of a decoder (a mixer with the cache it keeps, or a routed feed-forward) on one step's rows,
called through ``forward`` as the blocks call it, which is how a program puts the parts into a model of its own. Steps of
single tokens are captured once and replayed, as the engine's step function does with them; prompts are launched every time.

Layer sizes are those of ``bench.py`` (``--shape``, ``--compare``); page size 16 is the engine's default. Weights are random
with the spread of a trained layer's (rows of unit variance stay so), step sizes and decays of the recurrences are drawn
as those designs initialise them. A step's rows are those of a normed residual stream: unit variance.
"""

import math
import zlib

import torch

from llm_pipeline_b200.cache import CacheManager
from llm_pipeline_b200.config import resolve_config
from llm_pipeline_b200.engine import ModelRunner, StepEntry
from llm_pipeline_b200.engine.context import StepContext
from llm_pipeline_b200.models import build_model
from llm_pipeline_b200.ops import build_library
from llm_pipeline_b200.parts import LayerCache, lookup
from llm_pipeline_b200.weights.source import DictSource

PAGE = 16
EPS = 1e-5
THETA = 10000.0
DEVICE = "cuda:0"

# kind -> size -> the part's constructor arguments (``bench.py``: QWEN3 shapes, ZUPILORN, NUFOLIX, TUPIDRA, ZASUDRA, ZAVIZEN sizes)
SIZES = {
    "attention": {"1k": dict(hidden_size=1024, num_heads=16, num_kv_heads=8, head_dim=128),
                  "4k": dict(hidden_size=4096, num_heads=32, num_kv_heads=8, head_dim=128)},
    "latent": {"1k": dict(hidden_size=1024, num_heads=8, dim=64, rot_dim=32, vdim=64, kv_rank=256),
               "2k": dict(hidden_size=2048, num_heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=512)},
    "scan": {"1k": dict(hidden_size=1024, inner=2048, state=16, dt_rank=64, conv=4),
             "2k": dict(hidden_size=2048, inner=4096, state=16, dt_rank=128, conv=4)},
    "delta": {"1k": dict(hidden_size=1024, heads=8, qk_heads=8, dim=64, vdim=128, conv=4, decay_rank=64, gate_rank=64),
              "2k": dict(hidden_size=2048, heads=16, qk_heads=16, dim=128, vdim=128, conv=4, decay_rank=128, gate_rank=128)},
    "sigmoid": {"1k": dict(hidden_size=1024, num_heads=8, num_kv_heads=4, dim=128, vdim=128, softcap=30.0, rotary_dim=64),
                "2k": dict(hidden_size=2048, num_heads=16, num_kv_heads=4, dim=128, vdim=128, softcap=30.0, rotary_dim=64)},
    "window": {"1k": dict(hidden_size=1024, num_heads=8, num_kv_heads=4, dim=128, vdim=128, softcap=30.0, window=1024, keep_first=8),
               "2k": dict(hidden_size=2048, num_heads=16, num_kv_heads=4, dim=128, vdim=128, softcap=30.0, window=1024, keep_first=8)},
    "experts": {"1k": dict(hidden_size=1024, intermediate_size=1024, num_experts=16, top=4),
                "2k": dict(hidden_size=2048, intermediate_size=1408, num_experts=32, top=4)},
    "model": {"small": dict(hidden=1024, heads=16, kv=8, ff=3072, layers=4, vocab=32000),
              "large": dict(hidden=4096, heads=32, kv=8, ff=12288, layers=2, vocab=32000)},
}
PART = {"attention": "attention", "latent": "latent_attention", "scan": "selective_scan", "delta": "gated_delta_rule",
        "sigmoid": "sigmoid_attention", "window": "capped_attention", "experts": "routed_experts"}
RECURRENT = ("scan", "delta")


def _case(name, kind, size, requests, new, context=0, ragged=False, dtype="bfloat16", decode=0):
    return {"name": name, "kind": kind, "size": size, "requests": requests, "new": new, "context": context, "ragged": ragged,
            "dtype": dtype, "decode": decode}


def listed():
    return [
        # a few short chats at once on a small dense model: the smallest steps, where launches and latency count
        _case("dense chat, 4 short requests", "model", "small", 4, 40, ragged=True, decode=8),
        # several users' prompts of different lengths in one step of the large dense model
        _case("dense prompts, ragged", "model", "large", 3, 1500, ragged=True),
        # a serving step: eight requests at 2,048 tokens of context take one token each
        _case("dense attention, decode 8", "attention", "4k", 8, 1, context=2047),
        # a long document read by a layer that caches latent rows
        _case("latent attention, prompt", "latent", "2k", 1, 2048),
        # the same layer while it answers, at uneven contexts
        _case("latent attention, decode 8", "latent", "2k", 8, 1, context=2047, ragged=True),
        # a document through a selective scan: a chain over the tokens
        _case("selective scan, prompt", "scan", "2k", 1, 2048),
        # the exact path (float32 throughout) on a short question of odd length
        _case("selective scan, float32", "scan", "1k", 1, 203, dtype="float32"),
        # a document through the gated delta rule
        _case("delta rule, prompt", "delta", "2k", 1, 2048),
        # a few prompts of odd lengths together through the smaller delta rule layer
        _case("delta rule, ragged", "delta", "1k", 3, 613, ragged=True),
        # a document through sigmoid attention with mixed heads
        _case("sigmoid attention, prompt", "sigmoid", "2k", 1, 2048),
        # sixteen requests past the window of a windowed layer take one token each
        _case("window attention, decode 16", "window", "2k", 16, 1, context=1900, ragged=True),
        # a prompt through routed experts
        _case("experts, prompt", "experts", "2k", 1, 2048),
    ]


def draw(rng):
    """One more case of the same ranges: every kind and size, prompts of 16 to 2,048 tokens in up to four requests, single
    tokens of 1 to 16 requests over 64 to 4,096 keys, float32 for the shorter scans."""
    kind = rng.choice(["model", "attention", "latent", "latent", "scan", "scan", "delta", "delta", "sigmoid", "window", "experts"])
    size = rng.choice(sorted(SIZES[kind]))
    requests = rng.choice([1, 1, 2, 3, 4])
    tokens = int(round(math.exp(rng.uniform(math.log(16), math.log(2048)))))
    case = {"kind": kind, "size": size, "requests": requests, "new": max(1, tokens // requests), "context": 0,
            "ragged": rng.random() < 0.5, "dtype": "bfloat16", "decode": 0}
    if kind == "model":
        case["decode"] = rng.choice([0, 3, 6])
    elif kind == "scan" and rng.random() < 0.3:
        case.update(dtype="float32", size="1k", requests=1, new=min(tokens, 400))
    elif kind != "experts" and rng.random() < 0.45:
        case.update(requests=rng.randint(1, 16), new=1)
        top = 1200 if kind in RECURRENT else 4096
        case["context"] = min(int(round(math.exp(rng.uniform(math.log(64), math.log(top))))), 20000 // case["requests"])
    elif kind in ("latent", "window", "attention") and rng.random() < 0.4:
        case["context"] = rng.randint(1, 1500)
    elif kind == "experts" and rng.random() < 0.3:
        case.update(requests=1, new=rng.randint(1, 64))
    return case


# ---- sizes of a case ---------------------------------------------------------------------------------------------------

def _lengths(case):
    """(new tokens, cached tokens) of every request. Ragged batches: the first request is the longest, the last a fraction of it."""
    R, new, context = case["requests"], case["new"], case["context"]
    if not case["ragged"]:
        return [new] * R, [context] * R
    lens = [max(1, new * (R - i) // R - 3 * (i % 3)) for i in range(R)]
    starts = [max(1, context * (i + 1) // R - 5 * (i % 4)) if context else 0 for i in range(R)]
    return ([1] * R if new == 1 else lens), starts


def _dtype(case):
    return torch.float32 if case["dtype"] == "float32" else torch.bfloat16


def _args(case):
    args = dict(SIZES[case["kind"]][case["size"]])
    kind = case["kind"]
    if kind == "attention":
        args.update(scale=args["head_dim"] ** -0.5, qk_norm_eps=1e-6, position="rope")
    elif kind == "latent":
        args.update(scale=(args["dim"] + args["rot_dim"]) ** -0.5, norm_eps=EPS, position="rope", rot_dims=args["rot_dim"])
    elif kind == "delta":
        args.update(eps=EPS)
    elif kind == "sigmoid":
        args.update(scale=args["dim"] ** -0.5, bias=True, position="rope")
    elif kind == "window":
        args.update(scale=args["dim"] ** -0.5, distance_bias=True, sink=0.0, value_norm_eps=EPS, gate=True, bias=True)
    elif kind == "experts":
        args.update(score="chosen_softmax", form="relu_squared", router_bias=True)
    return args


def _rotated(case):
    a = SIZES[case["kind"]][case["size"]]
    return {"attention": a.get("head_dim", 0), "latent": a.get("rot_dim", 0), "sigmoid": a.get("rotary_dim", 0)}.get(case["kind"], 0)


# ---- weights -----------------------------------------------------------------------------------------------------------

def _tensors(case):
    """name -> (shape, how it is drawn) of the case's weights."""
    a, kind = SIZES[case["kind"]][case["size"]], case["kind"]
    if kind == "model":
        H, q, kv, I = a["hidden"], a["heads"] * 128, a["kv"] * 128, a["ff"]
        out = {"model.embed_tokens.weight": ((a["vocab"], H), "embedding"), "model.norm.weight": ((H,), "norm"),
               "lm_head.weight": ((a["vocab"], H), "matrix")}
        for i in range(a["layers"]):
            p = f"model.layers.{i}"
            out.update({f"{p}.input_layernorm.weight": ((H,), "norm"), f"{p}.post_attention_layernorm.weight": ((H,), "norm"),
                        f"{p}.mlp.gate_proj.weight": ((I, H), "matrix"), f"{p}.mlp.up_proj.weight": ((I, H), "matrix"),
                        f"{p}.mlp.down_proj.weight": ((H, I), "matrix")})
            out.update({f"{p}.self_attn.{n}": s for n, s in _attention_tensors(H, q, kv).items()})
        return out
    D = a["hidden_size"]
    if kind == "attention":
        return _attention_tensors(D, a["num_heads"] * 128, a["num_kv_heads"] * 128)
    if kind == "latent":
        H, C, R = a["num_heads"], a["kv_rank"], a["rot_dim"]
        return {"q": ((H * (a["dim"] + R), D), "matrix"), "dkv": ((C + R, D), "matrix"), "dkv.norm": ((C,), "norm"),
                "uk": ((H * a["dim"], C), "matrix"), "uv": ((H * a["vdim"], C), "matrix"), "o": ((D, H * a["vdim"]), "matrix")}
    if kind == "scan":
        I, N, R = a["inner"], a["state"], a["dt_rank"]
        return {"in": ((2 * I, D), "matrix"), "conv": ((I, a["conv"]), "taps"), "conv.b": ((I,), "small"), "x": ((R + 2 * N, I), "matrix"),
                "dt": ((I, R), "matrix"), "dt.b": ((I,), "step"), "A_log": ((I, N), "rates"), "D": ((I,), "norm"), "o": ((D, I), "matrix")}
    if kind == "delta":
        H, Q, V, d = a["heads"], a["qk_heads"] * a["dim"], a["heads"] * a["vdim"], a["dim"]
        return {"q": ((Q, D), "matrix"), "k": ((Q, D), "matrix"), "v": ((V, D), "matrix"), "q.conv": ((Q, a["conv"]), "taps"),
                "k.conv": ((Q, a["conv"]), "taps"), "v.conv": ((V, a["conv"]), "taps"), "b": ((H, D), "matrix"), "A_log": ((H,), "rate"),
                "dt_bias": ((H * d,), "step"), "a1": ((a["decay_rank"], D), "matrix"), "a2": ((H * d, a["decay_rank"]), "matrix"),
                "g1": ((a["gate_rank"], D), "matrix"), "g2": ((V, a["gate_rank"]), "matrix"), "norm": ((a["vdim"],), "norm"),
                "o": ((D, V), "matrix")}
    if kind in ("sigmoid", "window"):
        H, G, d, dv = a["num_heads"], a["num_kv_heads"], a["dim"], a["vdim"]
        out = {"q": ((H * d, D), "matrix"), "k": ((G * d, D), "matrix"), "v": ((G * dv, D), "matrix"), "o": ((D, H * dv), "matrix"),
               "q.b": ((H * d,), "small"), "k.b": ((G * d,), "small"), "v.b": ((G * dv,), "small")}
        if kind == "sigmoid":
            out.update({"talk": ((H, H), "mix"), "pb": ((H,), "bias")})
        else:
            out.update({"g": ((H * dv, D), "matrix"), "o.b": ((D,), "small")})
        return out
    E, I = a["num_experts"], a["intermediate_size"]
    out = {"router": ((E, D), "matrix"), "router.b": ((E,), "small")}
    for e in range(E):
        out.update({f"e{e}.up": ((I, D), "matrix"), f"e{e}.down": ((D, I), "matrix")})
    return out


def _attention_tensors(hidden, q, kv):
    return {"q_proj.weight": ((q, hidden), "matrix"), "k_proj.weight": ((kv, hidden), "matrix"), "v_proj.weight": ((kv, hidden), "matrix"),
            "o_proj.weight": ((hidden, q), "matrix"), "q_norm.weight": ((128,), "norm"), "k_norm.weight": ((128,), "norm")}


def _generator(seed, name):
    return torch.Generator(device=DEVICE).manual_seed((int(seed) << 20) ^ zlib.crc32(name.encode()))


def _weights(case, seed):
    """name -> tensor: matrices in the case's type, vectors in float32."""
    out = {}
    for name, (shape, how) in _tensors(case).items():
        g = _generator(seed, name)
        normal = lambda: torch.randn(shape, generator=g, device=DEVICE)   # noqa: E731
        uniform = lambda: torch.rand(shape, generator=g, device=DEVICE)   # noqa: E731
        if how == "matrix":
            out[name] = (normal() * shape[-1] ** -0.5).to(_dtype(case))
        elif how == "embedding":
            out[name] = normal().to(_dtype(case))
        elif how == "norm":
            out[name] = 1.0 + 0.1 * normal()
        elif how == "small":
            out[name] = 0.1 * normal()
        elif how == "taps":                     # a convolution's: uniform within 1 / sqrt(taps)
            out[name] = (2.0 * uniform() - 1.0) * shape[-1] ** -0.5
        elif how == "step":                     # softplus of it is a step size from 0.001 to 0.1, spread over its logarithm
            dt = torch.exp(uniform() * math.log(100.0) + math.log(0.001))
            out[name] = dt + torch.log(-torch.expm1(-dt))
        elif how == "rates":                    # decay rates 1 .. n of a channel's state entries
            out[name] = torch.log(torch.arange(1, shape[-1] + 1, dtype=torch.float32, device=DEVICE)).expand(shape).contiguous() + 0.05 * normal()
        elif how == "rate":                     # decay rates from 1 to 16 of the heads
            out[name] = torch.log(1.0 + 15.0 * uniform())
        elif how == "mix":                      # near the identity
            out[name] = torch.eye(shape[0], device=DEVICE) + 0.2 * shape[0] ** -0.5 * normal()
        else:                                   # "bias": a sigmoid's weights start small, so that a row's sum stays of order one
            out[name] = -6.0 + 0.5 * normal()
    return out


def _rows(case, seed):
    """The rows of every request, cached ones first, in the case's type."""
    lens, starts = _lengths(case)
    D = SIZES[case["kind"]][case["size"]]["hidden_size"]
    return [torch.randn((s + n, D), generator=_generator(seed, f"rows{r}"), device=DEVICE).to(_dtype(case))
            for r, (n, s) in enumerate(zip(lens, starts))]


def _ids(case, seed):
    """The tokens of every request: its prompt and, after it, the tokens it goes on with."""
    lens, _ = _lengths(case)
    vocab = SIZES["model"][case["size"]]["vocab"]
    return [torch.randint(0, vocab, (n + case["decode"],), generator=_generator(seed, f"ids{r}"), device=DEVICE) for r, n in enumerate(lens)]


# ---- what a program has in hand ----------------------------------------------------------------------------------------

def _context(cache, reqs, lens, starts, dtype):
    """The step's facts for the parts: ``lens`` new tokens behind ``starts`` cached ones."""
    device = torch.device(DEVICE)
    ctx = StepContext(device, dtype)
    tensor = lambda values: torch.tensor(values, dtype=torch.int32, device=device)   # noqa: E731
    R, N = len(reqs), sum(lens)
    ctx.num_tokens, ctx.num_requests, ctx.req_ids, ctx.starts, ctx.q_lens = N, R, list(reqs), list(starts), list(lens)
    keys = [s + n for s, n in zip(starts, lens)]
    ctx.max_q_len, ctx.max_ctx_len, ctx.total_ctx = max(lens), max(keys), sum(keys)
    ctx.table_width = max(1, -(-ctx.max_ctx_len // PAGE))
    ctx.token_ids = tensor([0] * N)
    ctx.positions = tensor([s + i for n, s in zip(lens, starts) for i in range(n)])
    ctx.position_ids = ctx.positions.view(1, N)
    ctx.token_request = tensor([r for r, n in enumerate(lens) for _ in range(n)])
    ctx.q_start = tensor([sum(lens[:r]) for r in range(R + 1)])
    ctx.ctx_len, ctx.slots = tensor(keys), tensor([cache.slot_of(q) for q in reqs])
    for g in range(len(cache.groups)):
        tables = [cache.block_table(q, g) for q in reqs]
        ctx.block_tables.append(tensor([(t + [-1] * ctx.table_width)[:ctx.table_width] for t in tables]))
        ctx.slot_mapping.append(tensor([cache.token_slot(q, g, s + i) for q, n, s in zip(reqs, lens, starts) for i in range(n)]))
    return ctx


def _prepare_model(case, seed):
    a = SIZES["model"][case["size"]]
    config = resolve_config({"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "vocab_size": a["vocab"], "hidden_size": a["hidden"],
                             "num_hidden_layers": a["layers"], "num_attention_heads": a["heads"], "num_key_value_heads": a["kv"], "head_dim": 128,
                             "intermediate_size": a["ff"], "rms_norm_eps": 1e-6, "rope_theta": 1000000.0, "tie_word_embeddings": False,
                             "max_position_embeddings": 4096})
    model = build_model(config)
    model.load(DictSource(_weights(case, seed)), torch.device(DEVICE), _dtype(case))
    ids = [row.tolist() for row in _ids(case, seed)]
    longest = max(len(row) for row in ids)
    pages = sum(-(-len(row) // PAGE) for row in ids)
    cache = CacheManager(model.cache_specs(), PAGE, pages, len(ids), -(-longest // PAGE) * PAGE, torch.device(DEVICE), _dtype(case))
    return {"case": case, "runner": ModelRunner(model, cache), "ids": ids}


def prepare(case, seed):
    build_library()
    if case["kind"] == "model":
        return _prepare_model(case, seed)
    dtype, kind = _dtype(case), case["kind"]
    lens, starts = _lengths(case)
    weights, rows = _weights(case, seed), _rows(case, seed)
    x = torch.cat([row[s:] for row, s in zip(rows, starts)])
    if kind == "experts":
        part = lookup("feed_forward", PART[kind])("p", **_args(case))
        part.load(lambda name, role: weights[name[2:]])
        ctx = StepContext(torch.device(DEVICE), dtype)
        ctx.num_tokens = x.shape[0]
        return {"case": case, "part": part, "x": x, "ctx": ctx, "cache": None, "graph": None}
    part = lookup("mixer", PART[kind])("p", **_args(case))
    part.load(lambda name, role: weights[name[2:]])
    reqs = list(range(len(lens)))
    longest = max(s + n for s, n in zip(starts, lens))
    pages = sum(-(-(s + n) // PAGE) for s, n in zip(starts, lens))
    room = -(-longest // PAGE) * PAGE
    cache = CacheManager([(part.cache_spec(), part.state_spec())], PAGE, pages, len(reqs), room, torch.device(DEVICE), dtype)
    view = LayerCache(pages=cache.pages_tensor(0) if cache.groups else None, group=0 if cache.groups else None, state=cache.state_tensor(0))
    rotary = lookup("position", "rotary")("rope", rotary_dim=_rotated(case), theta=THETA) if _rotated(case) else None

    def step(counts, done):
        for q, n, s in zip(reqs, counts, done):
            if not cache.reserve(q, s + n):
                raise RuntimeError("the cache has no pages left")
        ctx = _context(cache, reqs, counts, done, dtype)
        if rotary is not None:
            ctx.position_tables = {"rope": rotary.tables(ctx)}
        return ctx

    for q in reqs:
        cache.admit(q)
    with torch.no_grad():
        if case["context"]:
            # what the requests hold already: their earlier tokens through the same layer
            part.forward(torch.cat([row[:s] for row, s in zip(rows, starts)]), step(starts, [0] * len(reqs)), view)
            for q, s in zip(reqs, starts):
                cache.commit(q, s)
        ctx = step(lens, starts)
        state = {"case": case, "part": part, "x": x, "ctx": ctx, "cache": view, "graph": None}
        if case["new"] == 1:
            _width, ctx.decode_ctx_bound = ModelRunner.decode_graph_shape(longest, PAGE, room, part.captured_context_limit())
            part.forward(x, ctx, view)
            ctx.memo = {}
            torch.cuda.synchronize()
            state["graph"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(state["graph"]):
                state["out"] = part.forward(x, ctx, view)
    return state


# ---- one pass ------------------------------------------------------------------------------------------------------------

def _run_model(state):
    runner, ids, count = state["runner"], state["ids"], state["case"]["decode"]
    prompts = [row[:len(row) - count] for row in ids]
    logits = [runner.step([StepEntry(r, row, [0, len(row) - 1]) for r, row in enumerate(prompts)])]
    for k in range(count):
        # the buffer of a replayed step is the next step's too
        logits.append(runner.step([StepEntry(r, [row[len(row) - count + k]], [0]) for r, row in enumerate(ids)]).clone())
    for r in range(len(ids)):
        runner.release(r)
    return torch.cat(logits)


@torch.no_grad()
def run(state):
    """The rows (and bias, if any) that a layer leaves for the residual stream, and the state that a recurrence carries on;
    for a model the logits of every request's first and last prompt token and of every token it goes on with."""
    case = state["case"]
    if case["kind"] == "model":
        return {"logits": _run_model(state)}
    if state["graph"] is not None:
        state["graph"].replay()
        out, bias = state["out"]
    elif case["kind"] == "experts":
        out, bias = state["part"].forward(state["x"], state["ctx"])
    else:
        if state["cache"].state is not None:
            state["cache"].state.zero_()          # new requests: the cache manager hands their slots out so
        out, bias = state["part"].forward(state["x"], state["ctx"], state["cache"])
    result = {"rows": out}
    if bias is not None:
        result["bias"] = bias
    if case["kind"] in RECURRENT:
        result["state"] = state["cache"].state
    return result


# ---- what a pass cannot do without ---------------------------------------------------------------------------------------

def _pairs(case):
    """(query, key) pairs of all requests, and keys that have to be read."""
    lens, starts = _lengths(case)
    window, keep = (1024, 8) if case["kind"] == "window" else (1 << 40, 0)
    pairs = keys = 0
    for n, s in zip(lens, starts):
        pairs += sum(min(p + 1, window + min(keep, max(0, p + 1 - window))) for p in range(s, s + n))
        first = max(0, s - window + 1)
        keys += s + n - first + min(keep, first)
    return pairs, keys


def work(case):
    a, kind = SIZES[case["kind"]][case["size"]], case["kind"]
    size = 4 if case["dtype"] == "float32" else 2
    lens, starts = _lengths(case)
    R, N = case["requests"], sum(lens)
    if kind == "model":
        H, q, kv, I = a["hidden"], a["heads"] * 128, a["kv"] * 128, a["ff"]
        layer = H * (q + 2 * kv) + q * H + 3 * H * I
        steps, tokens = 1 + case["decode"], N + R * case["decode"]
        rows = 2 * R + R * case["decode"]
        pairs = sum((n + case["decode"]) * (n + case["decode"] + 1) // 2 for n in lens)
        keys = sum(n for n in lens) + sum(n + k + 1 for n in lens for k in range(case["decode"]))
        return {"bytes": steps * 2 * (a["layers"] * layer + H * a["vocab"]) + tokens * H * 2 + rows * a["vocab"] * 4 + a["layers"] * keys * 4 * kv,
                "flops": 2.0 * (a["layers"] * (tokens * layer + 2 * pairs * q) + rows * H * a["vocab"])}
    matrices = sum(math.prod(shape) for shape, how in _tensors(case).values() if how == "matrix")
    D = a["hidden_size"]
    traffic, flops = N * D * (size + 4), 2.0 * N * matrices
    if kind == "experts":
        E, used = a["num_experts"], a["top"] * N
        expert = 2 * a["intermediate_size"] * D
        touched = min(E, used)
        return {"bytes": traffic + E * D * size + touched * expert * size, "flops": 2.0 * (N * E * D + used * expert)}
    traffic += matrices * size
    if kind in RECURRENT:
        entries = a["inner"] * a["state"] if kind == "scan" else a["heads"] * a["dim"] * a["vdim"]
        traffic += R * entries * 4 * (2 if case["context"] else 1)
        flops += (6.0 if kind == "scan" else 8.0) * N * entries
        return {"bytes": traffic, "flops": flops}
    pairs, keys = _pairs(case)
    if kind == "latent":
        H, C, rot = a["num_heads"], a["kv_rank"], a["rot_dim"]
        # the cheaper of the two orders: heads over the cached rows, or keys and values of the heads formed first
        absorbed = 2.0 * pairs * H * (2 * C + rot)
        formed = 2.0 * (pairs * H * (a["dim"] + rot + a["vdim"]) + (keys - N) * H * (a["dim"] + a["vdim"]) * C)
        return {"bytes": traffic + keys * (C + rot) * size, "flops": flops + min(absorbed, formed)}
    d, dv = (128, 128) if kind == "attention" else (a["dim"], a["vdim"])
    return {"bytes": traffic + keys * a["num_kv_heads"] * (d + dv) * size, "flops": flops + 2.0 * pairs * a["num_heads"] * (d + dv)}


def tolerance(case):
    """About four times what the engine's results were measured to lie from 64 bits: 0.0053 for the small model's logits,
    0.0046 for softmax attention and 0.003 with a window, 0.0022 for sigmoid attention, 0.0018 for the recurrences and
    experts (roundings of a layer's intermediate rows to bfloat16); 1.2e-6 in float32, where about 1e-5 is what another
    order of the sums may give."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": {"model": 0.02, "attention": 0.018, "latent": 0.018, "window": 0.012, "sigmoid": 0.009}.get(case["kind"], 0.0075), "max": 0.3}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------------

def _rms(x, eps):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)


def _rotate(x, positions, dims, theta):
    """The first ``dims`` entries of the last axis, entry i with i + dims / 2; x: [tokens, heads, entries]."""
    half = dims // 2
    frequency = (1.0 / theta ** (torch.arange(0, dims, 2, dtype=torch.int64, device=x.device).float() / dims)).double()
    angle = positions.double()[:, None, None] * frequency
    lo, hi = x[..., :half], x[..., half:dims]
    return torch.cat([lo * angle.cos() - hi * angle.sin(), hi * angle.cos() + lo * angle.sin(), x[..., dims:]], dim=-1)


def _attend(q, k, v, start, weights_of):
    """Rows of q [n, H, d] at positions start.. over k [T, G, d], v [T, G, dv]; ``weights_of(scores, i, j)`` makes the weights
    [H, n, T] of the products. In parts of rows, to bound the memory."""
    n, H, _ = q.shape
    T, G, _ = k.shape
    k, v = k.repeat_interleave(H // G, dim=1).transpose(0, 1), v.repeat_interleave(H // G, dim=1).transpose(0, 1)
    j, out = torch.arange(T, device=q.device)[None, :], []
    for at in range(0, n, 256):
        part = q[at:at + 256].transpose(0, 1)
        i = start + at + torch.arange(part.shape[1], device=q.device)[:, None]
        out.append((weights_of(part @ k.transpose(1, 2), i, j) @ v).transpose(0, 1))
    return torch.cat(out)


def _softmax(scale):
    return lambda s, i, j: torch.softmax((s * scale).masked_fill(j > i, -math.inf), dim=-1)


def _exact_attention(w, x, start, heads, kv, theta):
    T = x.shape[0]
    at = torch.arange(T, device=x.device)
    q = (x[start:] @ w["q_proj.weight"].T).view(T - start, heads, 128)
    k, v = ((x @ w[n].T).view(T, kv, 128) for n in ("k_proj.weight", "v_proj.weight"))
    q = _rotate(_rms(q, 1e-6) * w["q_norm.weight"], at[start:], 128, theta)
    k = _rotate(_rms(k, 1e-6) * w["k_norm.weight"], at, 128, theta)
    return _attend(q, k, v, start, _softmax(128 ** -0.5)).reshape(T - start, heads * 128) @ w["o_proj.weight"].T


def _exact_latent(a, w, x, start):
    T, H, C = x.shape[0], a["num_heads"], a["kv_rank"]
    at = torch.arange(T, device=x.device)
    q = (x[start:] @ w["q"].T).view(T - start, H, a["dim"] + a["rot_dim"])
    q_rot = _rotate(q[..., a["dim"]:], at[start:], a["rot_dim"], THETA)
    rows = x @ w["dkv"].T
    c = _rms(rows[:, :C], EPS) * w["dkv.norm"]
    k_rot = _rotate(rows[:, None, C:], at, a["rot_dim"], THETA)
    k = torch.cat([(c @ w["uk"].T).view(T, H, a["dim"]), k_rot.expand(T, H, a["rot_dim"])], dim=-1)
    v = (c @ w["uv"].T).view(T, H, a["vdim"])
    o = _attend(torch.cat([q[..., :a["dim"]], q_rot], dim=-1), k, v, start, _softmax((a["dim"] + a["rot_dim"]) ** -0.5))
    return o.reshape(T - start, H * a["vdim"]) @ w["o"].T


def _conv(x, taps, bias=0.0):
    K = taps.shape[1]
    padded = torch.cat([x.new_zeros((K - 1, x.shape[1])), x])
    return torch.nn.functional.silu(sum(padded[j:j + x.shape[0]] * taps[:, j] for j in range(K)) + bias)


def _exact_scan(a, w, x, start):
    T, I, N, R = x.shape[0], a["inner"], a["state"], a["dt_rank"]
    xz = x @ w["in"].T
    xc = _conv(xz[:, :I], w["conv"], w["conv.b"])
    dbc = xc @ w["x"].T
    dt = torch.nn.functional.softplus(dbc[:, :R] @ w["dt"].T + w["dt.b"])
    rate, S, y = -torch.exp(w["A_log"]), x.new_zeros((I, N)), torch.empty_like(xc)
    for t in range(T):
        S = S * torch.exp(dt[t, :, None] * rate) + (dt[t] * xc[t])[:, None] * dbc[t, None, R:R + N]
        y[t] = S @ dbc[t, R + N:]
    y = (y + w["D"] * xc) * torch.nn.functional.silu(xz[:, I:])
    return y[start:] @ w["o"].T


def _exact_delta(a, w, x, start):
    T, H, G, d, dv = x.shape[0], a["heads"], a["qk_heads"], a["dim"], a["vdim"]
    q, k, v = (_conv(x @ w[n].T, w[n + ".conv"]) for n in ("q", "k", "v"))
    unit = lambda y: y * torch.rsqrt(y.square().sum(-1, keepdim=True) + 1e-6)   # noqa: E731
    q, k = (unit(y.view(T, G, d)).repeat_interleave(H // G, dim=1) for y in (q, k))
    q, v = q * d ** -0.5, v.view(T, H, dv)
    beta = torch.sigmoid(x @ w["b"].T)
    g = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(((x @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(T, H, d)))
    S, o = x.new_zeros((H, d, dv)), torch.empty_like(v)
    for t in range(T):
        S = S * g[t, :, :, None]
        u = beta[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
        S = S + k[t, :, :, None] * u[:, None, :]
        o[t] = torch.einsum("hdv,hd->hv", S, q[t])
    o = _rms(o, EPS) * w["norm"] * torch.sigmoid(((x @ w["g1"].T) @ w["g2"].T).view(T, H, dv))
    return o.reshape(T, H * dv)[start:] @ w["o"].T


def _exact_grouped(case, a, w, x, start):
    """The sigmoid and the windowed attention: the same projections, other weights."""
    T, H, G, d, dv = x.shape[0], a["num_heads"], a["num_kv_heads"], a["dim"], a["vdim"]
    at = torch.arange(T, device=x.device)
    q = (x[start:] @ w["q"].T + w["q.b"]).view(T - start, H, d)
    k = (x @ w["k"].T + w["k.b"]).view(T, G, d)
    v = (x @ w["v"].T + w["v.b"]).view(T, G, dv)
    capped = lambda s: a["softcap"] * torch.tanh(s * d ** -0.5 / a["softcap"])   # noqa: E731
    if case["kind"] == "sigmoid":
        q, k = _rotate(q, at[start:], a["rotary_dim"], THETA), _rotate(k, at, a["rotary_dim"], THETA)

        def weights_of(s, i, j):
            p = torch.sigmoid(capped(s) + w["pb"][:, None, None]).masked_fill(j > i, 0.0)
            return torch.einsum("hg,gij->hij", w["talk"], p)

        return _attend(q, k, v, start, weights_of).reshape(T - start, H * dv) @ w["o"].T
    v = _rms(v, EPS)
    slopes = 2.0 ** (-8.0 * torch.arange(1, H + 1, dtype=torch.float64, device=x.device) / H)

    def weights_of(s, i, j):
        seen = (j <= i) & ((i - j < a["window"]) | (j < a["keep_first"]))
        s = (capped(s) - slopes[:, None, None] * (i - j)).masked_fill(~seen, -math.inf)
        top = s.amax(-1, keepdim=True).clamp_min(0.0)
        e = torch.exp(s - top)
        return e / (torch.exp(-top) + e.sum(-1, keepdim=True))

    o = _attend(q, k, v, start, weights_of).reshape(T - start, H * dv) * torch.sigmoid(x[start:] @ w["g"].T)
    return o @ w["o"].T


def _exact_experts(a, w, x):
    z = x @ w["router"].T + w["router.b"]
    top, chosen = z.topk(a["top"], dim=-1)
    weight, out = torch.softmax(top, dim=-1), torch.zeros_like(x)
    for e in range(a["num_experts"]):
        rows, place = (chosen == e).nonzero(as_tuple=True)
        if rows.numel():
            y = torch.relu(x[rows] @ w[f"e{e}.up"].T).square() @ w[f"e{e}.down"].T
            out.index_add_(0, rows, y * weight[rows, place, None])
    return out


def _exact_model(case, w, ids):
    a, out = SIZES["model"][case["size"]], []
    hidden = []
    for row in ids:
        x = w["model.embed_tokens.weight"][row]
        for i in range(a["layers"]):
            p = f"model.layers.{i}."
            own = {n[len(p) + 10:]: t for n, t in w.items() if n.startswith(p + "self_attn.")}
            x = x + _exact_attention(own, _rms(x, 1e-6) * w[p + "input_layernorm.weight"], 0, a["heads"], a["kv"], 1000000.0)
            h = _rms(x, 1e-6) * w[p + "post_attention_layernorm.weight"]
            x = x + (torch.nn.functional.silu(h @ w[p + "mlp.gate_proj.weight"].T) * (h @ w[p + "mlp.up_proj.weight"].T)) @ w[p + "mlp.down_proj.weight"].T
        hidden.append(_rms(x, 1e-6) * w["model.norm.weight"])
    head, count = w["lm_head.weight"].T, case["decode"]
    for row in hidden:
        out.append(row[[0, row.shape[0] - count - 1]] @ head)
    for k in range(count):
        out.append(torch.stack([row[row.shape[0] - count + k] for row in hidden]) @ head)
    return torch.cat(out)


@torch.no_grad()
def exact(case, seed):
    w = {name: t.double() for name, t in _weights(case, seed).items()}
    if case["kind"] == "model":
        return {"logits": _exact_model(case, w, _ids(case, seed))}
    a, kind = SIZES[case["kind"]][case["size"]], case["kind"]
    _lens, starts = _lengths(case)
    rows = []
    for x, start in zip(_rows(case, seed), starts):
        x = x.double()
        if kind == "attention":
            rows.append(_exact_attention(w, x, start, a["num_heads"], a["num_kv_heads"], THETA))
        elif kind == "experts":
            rows.append(_exact_experts(a, w, x))
        elif kind in ("sigmoid", "window"):
            rows.append(_exact_grouped(case, a, w, x, start))
        else:
            rows.append({"latent": _exact_latent, "scan": _exact_scan, "delta": _exact_delta}[kind](a, w, x, start))
    result = {"rows": torch.cat(rows)}
    if kind == "window":
        result["bias"] = w["o.b"]
    if kind in RECURRENT:
        result["state"] = None                    # its layout is the engine's own
    return result
