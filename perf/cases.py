"""What is timed when this framework's speed is looked at: whole steps of the dense decoder through ``Engine.step`` and single
layers' parts (mixers, routed feed-forwards) as a step runs them, at the widths of ``bench.py``'s shapes.

A case is a dict of plain values.  ``kind`` says which path it takes:

  dense      a Qwen3-style decoder: a prompt in one step (``steps`` 0) or ``steps`` single-token steps behind cached prompts
  scan       the selective scan                      ssd      the state-space-duality recurrence
  delta      the gated delta rule                    linear   linear attention with a decay per head
  latent     attention over a cached latent, rotated part, window and sinks (``rot``) or a gate per element and no window
  experts    routed experts with a shared one, plain in groups (``gated`` False) or gated

``tokens`` of ``requests`` requests make one step; as many tokens as requests is a decode step, otherwise the requests bring
portions of uneven lengths.  ``context`` is how many tokens a request's cache holds before the step (the mean, uneven too).
"""
import math

import torch

from aien_sovereign_core_mv_b200 import Engine, EngineConfig
from aien_sovereign_core_mv_b200 import kernels as K
from aien_sovereign_core_mv_b200.models.decoder import Decoder
from aien_sovereign_core_mv_b200.models.loading import model_spec_for
from aien_sovereign_core_mv_b200.parts import GroupView, RunBinding, StepContext, StepLimits, Workspace
from aien_sovereign_core_mv_b200.registry import make_part

PAGE = 16
VOCAB = 32768
EPS = 1e-6


def listed():
    return [
        # one user chatting: a short model, one token at a time, every launch waits for the one before
        dict(name="dense_decode_1", kind="dense", width=2048, layers=4, tokens=1, requests=1, context=480, steps=4),
        # a serving batch that is no power of two, uneven contexts
        dict(name="dense_decode_24", kind="dense", width=4096, layers=4, tokens=24, requests=24, context=1600, steps=4),
        # prompts of three users in one step
        dict(name="dense_prefill", kind="dense", width=4096, layers=4, tokens=3000, requests=3, context=0, steps=0),
        # a prompt through one layer of each recurrence; two of them as portions of several users
        dict(name="scan_prefill", kind="scan", width=2048, tokens=2048, requests=1, context=0),
        dict(name="ssd_prefill", kind="ssd", width=2048, tokens=2000, requests=3, context=0),
        dict(name="delta_prefill", kind="delta", width=2048, tokens=2048, requests=1, context=0),
        dict(name="linear_prefill", kind="linear", width=2048, tokens=1900, requests=2, context=0),
        # the generating half of a recurrence: what counts is the state it reads and writes
        dict(name="ssd_decode_64", kind="ssd", width=2048, tokens=64, requests=64, context=1024),
        # a long prompt through windowed attention over a latent; many users generating over one without a window
        dict(name="latent_prefill", kind="latent", width=2048, tokens=2048, requests=1, context=0, rot=True),
        dict(name="latent_decode_64", kind="latent", width=2048, tokens=64, requests=64, context=1500, rot=False),
        # routed experts: a prompt reaches all of them, a few generating users a handful each
        dict(name="experts_prefill", kind="experts", width=2048, tokens=2048, requests=1, context=0, gated=False),
        dict(name="experts_decode_9", kind="experts", width=2048, tokens=9, requests=9, context=0, gated=True),
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("dense", "scan", "ssd", "delta", "linear", "latent", "experts"))
    width = rng.choice((1024, 2048, 2048, 4096))
    decode = rng.random() < 0.4
    if decode:
        requests = _spread(rng, 1, 64)
        case = dict(kind=kind, width=width, tokens=requests, requests=requests, context=_spread(rng, 64, 2000))
    else:
        tokens = _spread(rng, 64, 2048)
        case = dict(kind=kind, width=width, tokens=tokens, requests=rng.randint(1, max(1, min(6, tokens // 32))), context=rng.choice((0, 0, 0, _spread(rng, 64, 1500))))
    if kind == "dense":
        case.update(layers=rng.choice((2, 4)), steps=4 if decode else 0)
    elif kind == "latent":
        case.update(rot=rng.random() < 0.5)
    elif kind == "experts":
        case.update(gated=rng.random() < 0.5, context=0)
    return case


# ------------------------------------------------------------------ sizes
def _uneven(total, parts, least):
    """``total`` cut into ``parts`` uneven numbers of at least ``least``."""
    weight = [1.0 + ((5 * i + 2) % 7) / 3.0 for i in range(parts)]
    room = total - parts * least
    out = [least + int(room * w / sum(weight)) for w in weight]
    out[0] += total - sum(out)
    return out


def _step(case):
    """(tokens each request brings, tokens each request's cache holds before)."""
    S, T = case["requests"], case["tokens"]
    bring = [1] * S if T == S else _uneven(T, S, 2)
    # cached prompts end on a page boundary, as prompts shared by page do
    held = [max(PAGE, c // PAGE * PAGE) for c in _uneven(case["context"] * S, S, case["context"] // 2)] if case["context"] else [0] * S
    return bring, held


def _dense_config(case):
    w = case["width"]
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=case["layers"], hidden_size=w, num_attention_heads=w // 128,
                num_key_value_heads=w // 512, head_dim=128, intermediate_size=3 * w, vocab_size=VOCAB, rope_theta=1000000.0, rms_norm_eps=EPS,
                tie_word_embeddings=True, max_position_embeddings=8192, hidden_act="silu", attention_bias=False, eos_token_id=0)


def _heads(case):
    """(heads, size of a head) of the recurrences and the latent attention at this width."""
    return (16, 64) if case["width"] == 1024 else (case["width"] // 128, 128)


def _part(case):
    """(family, kind, parameters) of the part that the case runs."""
    w, kind = case["width"], case["kind"]
    n, d = _heads(case)
    if kind == "scan":
        return "mixer", "selective_scan", dict(hidden_size=w, inner=2 * w, state=16, dt_rank=w // 16, taps=4)
    if kind == "ssd":
        return "mixer", "state_space_duality", dict(hidden_size=w, num_heads=w // 64, value_dim=64, state=128, groups=1, norm_groups=1, taps=4, norm_eps=EPS)
    if kind == "delta":
        return "mixer", "gated_delta_rule", dict(hidden_size=w, num_heads=n, num_qk_heads=n // 2, head_dim=d, value_dim=d, taps=4, norm_eps=EPS)
    if kind == "linear":
        return "mixer", "decay_linear_attention", dict(hidden_size=w, num_heads=n, head_dim=d, value_dim=d, norm_eps=EPS,
                                                       decay=[1.0 - 2.0 ** (-5.0 - 3.0 * i / (n - 1)) for i in range(n)])
    if kind == "latent":
        p = dict(hidden_size=w, num_heads=n, head_dim=d, value_dim=d, kv_rank=4 * d, norm_eps=EPS)
        if case["rot"]:
            return "mixer", "latent_attention", dict(p, rot_dim=d // 2, q_rank=12 * d, window=8 * d, sink=True)
        return "mixer", "latent_attention", dict(p, rot_dim=0, q_rank=0, out_gate=True)
    experts, top, ff, shared = (16, 4, w // 2, w // 2) if case["gated"] else (64 if w == 2048 else 32, 6 if w == 2048 else 4, 3 * w // 8, 3 * w // 4)
    p = dict(hidden_size=w, expert_ff=ff, num_experts=experts, top=top, shared_ff=shared, combined=True)
    if case["gated"]:
        return "feed_forward", "routed_experts", dict(p, act="swiglu", score="sigmoid", weight_on_input=True, shared_gate=True)
    return "feed_forward", "routed_experts", dict(p, act="gelu", group_count=8, group_keep=4)


# ------------------------------------------------------------------ inputs
def _numbers(g, shape, kind):
    """A stored tensor of a trained model's size: matrices keep a vector's length, scales lie around one."""
    r = lambda: torch.randn(shape, generator=g, device="cuda")
    u = lambda lo, hi: torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo
    t = {"matrix": lambda: r() / math.sqrt(shape[-1]), "embedding": r, "norm": lambda: u(0.8, 1.2), "vector": r, "small": lambda: 0.1 * r(),
         "log_rate": lambda: u(-4.0, 1.0), "rate_bias": lambda: u(-4.5, -1.0)}[kind]()
    return t.to(torch.bfloat16)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _tensors(g, shapes):
    return {name: _numbers(g, tuple(shape), kind) for name, (shape, kind) in shapes.items()}


def _inputs(case, seed):
    """The part, its tensors, the step's rows and what its cache or state holds."""
    g = _generator(seed)
    family, kind, params = _part(case)
    rot = params.get("rot_dim", 0)
    position = make_part("position", "rotary", head_dim=rot, theta=10000.0, pairing="interleaved") if rot else make_part("position", "none")
    part = make_part(family, kind, **params, **({"position": position} if family == "mixer" else {}))
    tensors = _tensors(g, part.param_shapes())
    h = torch.randn(case["tokens"], case["width"], generator=g, device="cuda").to(torch.bfloat16)        # a normed stream
    bring, held = _step(case)
    S = case["requests"]
    need = part.cache_need() if family == "mixer" else None
    cache = blocks = None
    if need is not None and need.kind == "state":
        shape = tuple(need.state_shape)
        cache = 0.3 * torch.randn((1, S + 1) + shape, generator=g, device="cuda")
        if not case["context"]:
            cache.zero_()
        blocks = torch.randperm(S, generator=g, device="cuda").to(torch.int32)                          # the slot of every request
    elif need is not None:
        pages = [(a + b + PAGE - 1) // PAGE for a, b in zip(bring, held)]
        order = torch.randperm(sum(pages), generator=g, device="cuda").to(torch.int32)
        blocks = torch.full((S, max(pages)), -1, dtype=torch.int32, device="cuda")
        at = 0
        for s, n in enumerate(pages):
            blocks[s, :n] = order[at:at + n]
            at += n
        cache = torch.zeros((1, sum(pages) * PAGE) + tuple(need.planes[0][1]), dtype=torch.bfloat16, device="cuda")
        for s, n in enumerate(held):
            if n:
                cache[0, _slots(blocks[s], 0, n)] = torch.randn((n,) + tuple(need.planes[0][1]), generator=g, device="cuda").to(torch.bfloat16)
    return part, position, params, tensors, h, bring, held, need, cache, blocks


def _slots(blocks, lo, hi):
    """The cache rows of positions lo .. hi of a request with these pages."""
    p = torch.arange(lo, hi, device="cuda")
    return (blocks[p // PAGE].long() * PAGE + p % PAGE)


def _prepare_part(case, seed):
    part, position, params, tensors, h, bring, held, need, cache, blocks = _inputs(case, seed)
    part.bind(tensors)
    S, T = case["requests"], case["tokens"]
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    starts = [sum(bring[:i]) for i in range(S + 1)]
    decode = T == S
    limits = StepLimits(max_tokens=T, max_seqs=S, max_context=max(a + b for a, b in zip(bring, held)), itemsize=2)
    step_bytes = position.step_workspace_bytes(T) if params.get("rot_dim") else 0
    tiles = [(s, q) for s in range(S) for q in range(0, bring[s], K.PREFILL_TILE)]
    groups = []
    if need is not None and need.kind == "state":
        groups = [GroupView("state", PAGE, 0, 0, None, blocks, {"state": cache})]
    elif need is not None:
        slot_map = torch.cat([_slots(blocks[s], held[s], held[s] + bring[s]) for s in range(S)]).to(torch.int32)
        groups = [GroupView(need.kind, PAGE, need.window, blocks.shape[1], blocks, slot_map, {need.planes[0][0]: cache})]
    fixed = dict(dtype=torch.bfloat16, num_tokens=T, num_seqs=S, token_ids=i32([0] * T), positions=i32([held[s] + i for s in range(S) for i in range(bring[s])]),
                 seq_of_token=i32([s for s in range(S) for _ in range(bring[s])]), q_start=i32(starts), ctx_len=i32([a + b for a, b in zip(bring, held)]),
                 groups=groups, workspace=Workspace(step_bytes + 4096, part.workspace_bytes(limits) + (1 << 16), torch.device("cuda")),
                 max_q_len=max(bring), max_ctx_len=limits.max_context, decode_only=decode)
    if not decode:
        fixed.update(prefill_tiles=(i32([s for s, _ in tiles]), i32([q for _, q in tiles]), len(tiles)), single_tokens=(i32([0]), 0))
    return dict(part=part, h=h, step=fixed, cache=cache, run=RunBinding(0, 0, True) if need is not None else None)


def _run_part(state):
    step = state["step"]
    step["workspace"].reset()
    step["workspace"].begin_layer()
    ctx = StepContext(**step)
    with K.stream_scope():
        y = state["part"].forward(ctx, state["h"], state["run"]) if state["run"] is not None else state["part"].forward(ctx, state["h"])
    if y.dim() == 3:                                     # partial products, which the next norm would add
        y = y.sum(0)
    return [y] if state["cache"] is None else [y, state["cache"]]


def _prepare_dense(case, seed):
    g = _generator(seed)
    raw = _dense_config(case)
    cfg, spec = model_spec_for(raw)
    model = Decoder(spec)
    model.bind(_tensors(g, model.catalog()).items())
    bring, held = _step(case)
    S = case["requests"]
    pool = sum((c + PAGE) // PAGE + 2 for c in held) * PAGE + sum(bring) + (2 + S) * PAGE * 2
    engine = Engine(model, cfg, EngineConfig(dtype="bfloat16", page_size=PAGE, max_cache_tokens=pool, max_requests=2 * S + 2,
                                             max_batch_tokens=max(2048, case["tokens"]), max_context=8192))
    words = lambda n: torch.randint(0, VOCAB, (n,), generator=g, device="cuda").tolist()
    state = dict(engine=engine, requests=S, steps=case["steps"], held=[words(n) for n in held])
    for s, toks in enumerate(state["held"]):             # the prompts that the caches hold
        for at in range(0, len(toks), 2048):
            engine.step([(s, toks[at:at + 2048], [])])
    if case["steps"]:
        state["tokens"] = [[[t] for t in words(S)] for _ in range(case["steps"])]
        state["logits"] = [torch.empty(S, VOCAB, device="cuda") for _ in range(case["steps"])]
    else:
        state["tokens"] = [words(n) for n in bring]
        state["logits"] = [torch.empty(S, VOCAB, device="cuda")]
    _run_dense(state)                                    # a server has seen steps of this size before
    return state


def _run_dense(state):
    """Portions of prompts in one step, or tokens generated one by one behind the cached prompts; a second set of
    requests that share the prompts' pages, so that the prompts are there for the next ones."""
    engine, S = state["engine"], state["requests"]
    ids = range(1000, 1000 + S)
    for s, toks in enumerate(state["held"]):
        if toks:
            engine.fork(s, 1000 + s)
    if state["steps"]:
        for toks, logits in zip(state["tokens"], state["logits"]):
            engine.step([(i, t, (0,)) for i, t in zip(ids, toks)], logits)
    else:
        engine.step([(i, t, (len(t) - 1,)) for i, t in zip(ids, state["tokens"])], state["logits"][0])
    for i in ids:
        engine.end_request(i)
    return state["logits"]


def prepare(case, seed):
    return _prepare_dense(case, seed) if case["kind"] == "dense" else _prepare_part(case, seed)


def run(state):
    return _run_dense(state) if "engine" in state else _run_part(state)


# ------------------------------------------------------------------ what a pass cannot do without
def work(case):
    T, S, w, kind = case["tokens"], case["requests"], case["width"], case["kind"]
    bring, held = _step(case)
    # keys every token sees, summed over the step's tokens
    sees = lambda window: sum(sum(min(c + i + 1, window) for i in range(b)) for b, c in zip(bring, held))
    if kind == "dense":
        n, kv, ff, steps = w // 128, w // 512, 3 * w, max(1, case["steps"])
        layer = w * (n + 2 * kv) * 128 + n * 128 * w + 3 * w * ff
        keys = sees(1 << 30) + (steps - 1) / 2.0 * S
        read = sum(a + b for a, b in zip(bring, held)) + (steps - 1) / 2.0 * S
        per_layer = 2 * layer + read * 2 * kv * 128 * 2
        return dict(bytes=steps * (case["layers"] * per_layer + VOCAB * w * 2 + S * VOCAB * 4 + T * w * 2),
                    flops=steps * (case["layers"] * (2 * T * layer + 4 * keys * n * 128) + 2 * S * VOCAB * w))
    _, _, p = _part(case)
    n, d = _heads(case)
    rows = 2 * T * w + 4 * T * w                         # the stream read in 16 bits, the branch written in 32
    if kind == "scan":
        i, r = p["inner"], p["dt_rank"]
        m = 2 * i * w + (r + 32) * i + i * r + w * i
        return dict(bytes=2 * m + rows + 2 * S * (3 + 16) * i * 4, flops=2 * T * m + T * i * 16 * 6)
    if kind == "ssd":
        i, h = w, p["num_heads"]
        m = (2 * i + 256 + h) * w + w * i
        return dict(bytes=2 * m + rows + 2 * S * (3 * (i + 256) + i * 128) * 4, flops=2 * T * m + T * i * 128 * 5)
    if kind == "delta":
        m = (3 * n * d + 2 * n) * w + w * n * d          # q and k have half the heads each
        return dict(bytes=2 * m + rows + 2 * S * (6 * n * d + n * d * d) * 4, flops=2 * T * m + T * n * d * d * 7)
    if kind == "linear":
        m = 4 * n * d * w + w * n * d
        return dict(bytes=2 * m + rows + 2 * S * n * d * d * 4, flops=2 * T * m + T * n * d * d * 5)
    if kind == "latent":
        r, rot, q = p["kv_rank"], p["rot_dim"], p["q_rank"]
        m = (q * w + n * (d + rot) * q if q else n * d * w) + (r + rot) * w + 2 * n * d * r + w * n * d + (0 if q else n * d * w)
        keys = sees(p.get("window") or 1 << 30)
        read = sum(min(b + c, (p.get("window") or 1 << 30) + b) for b, c in zip(bring, held))
        return dict(bytes=2 * m + rows + read * (r + rot) * 2, flops=2 * T * m + 2 * keys * n * (2 * d + rot))
    e, top, ff, mats = p["num_experts"], p["top"], p["expert_ff"], 3 if case["gated"] else 2
    reached = e * (1.0 - (1.0 - top / e) ** T)           # experts that T tokens choose between them, on the average
    return dict(bytes=2 * (reached * mats * ff * w + mats * p["shared_ff"] * w + e * w) + rows, flops=2 * T * w * (mats * (top * ff + p["shared_ff"]) + e))


def tolerance(case):
    # 16-bit operands of float32 sums: about 2^-9 a rounding, a few of them on the way; a whole decoder adds up its layers'
    return {"rel": 0.02, "max": 0.4} if case["kind"] == "dense" else {"rel": 0.012, "max": 0.2}


# ------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    with torch.no_grad():
        return _exact_dense(case, seed) if case["kind"] == "dense" else _exact_part(case, seed)


def _norm(x, weight, eps=EPS):
    return x / torch.sqrt(x.square().mean(-1, keepdim=True) + eps) * weight


def _silu(x):
    return x * torch.sigmoid(x)


def _softplus(x):
    return torch.nn.functional.softplus(x, threshold=40.0)


def _pairs(x, pos, base):
    """Neighbouring numbers turned by pos * base^(-2i/n)."""
    n = x.shape[-1]
    a = pos.double()[:, None] * base ** (-torch.arange(0, n, 2, device="cuda").double() / n)
    a = a.view((a.shape[0],) + (1,) * (x.dim() - 2) + (n // 2,))
    re, im = x[..., 0::2], x[..., 1::2]
    return torch.stack([re * a.cos() - im * a.sin(), re * a.sin() + im * a.cos()], dim=-1).flatten(-2)


def _halves(x, pos, base):
    n = x.shape[-1]
    a = (pos.double()[:, None] * base ** (-torch.arange(0, n, 2, device="cuda").double() / n))[:, None]
    lo, hi = x[..., :n // 2], x[..., n // 2:]
    return torch.cat([lo * a.cos() - hi * a.sin(), hi * a.cos() + lo * a.sin()], dim=-1)


def _attend(q, k, v, scale, first, window=1 << 30, sink=None):
    """q [t, n, a], k [m, n, a], v [m, n, b]: query i stands at position first + i."""
    out = []
    for at in range(0, q.shape[0], 256):
        z = torch.einsum("tna,mna->ntm", q[at:at + 256], k) * scale
        i = first + at + torch.arange(z.shape[1], device="cuda")[:, None]
        j = torch.arange(k.shape[0], device="cuda")[None]
        z = z.masked_fill((j > i) | (j <= i - window), -math.inf)
        if sink is not None:
            z = torch.cat([z, sink.double()[:, None, None].expand(-1, z.shape[1], 1)], dim=-1)
        out.append(torch.einsum("ntm,mnb->tnb", z.softmax(-1)[..., :k.shape[0]], v))
    return torch.cat(out)


def _conv(u, w, b, before):
    """Causal convolution over time per channel and silu; ``before``: the rows ahead of the portion; the new rows to keep."""
    rows = torch.cat([before, u])
    taps = w.shape[1]
    y = sum(rows[j:j + u.shape[0]] * w[:, j] for j in range(taps))
    return _silu(y + b if b is not None else y), rows[-(taps - 1):]


def _exact_dense(case, seed):
    g = _generator(seed)
    raw = _dense_config(case)
    t = {k: v.double() for k, v in _tensors(g, Decoder(model_spec_for(raw)[1]).catalog()).items()}
    bring, held = _step(case)
    words = lambda n: torch.randint(0, VOCAB, (n,), generator=g, device="cuda").tolist()
    rows = [words(n) for n in held]
    more = [words(len(bring)) for _ in range(case["steps"])] if case["steps"] else [words(n) for n in bring]
    n, kv, out = raw["num_attention_heads"], raw["num_key_value_heads"], []
    for s in range(case["requests"]):
        seq = rows[s] + ([m[s] for m in more] if case["steps"] else more[s])
        x = t["model.embed_tokens.weight"][torch.tensor(seq, device="cuda")]
        pos = torch.arange(len(seq), device="cuda")
        for i in range(case["layers"]):
            at = lambda name: t["model.layers.%d.%s.weight" % (i, name)]
            h = _norm(x, at("input_layernorm"))
            split = lambda name, m: (h @ at("self_attn." + name).T).view(len(seq), m, 128)
            q = _halves(_norm(split("q_proj", n), at("self_attn.q_norm")), pos, 1000000.0)
            k = _halves(_norm(split("k_proj", kv), at("self_attn.k_norm")), pos, 1000000.0)
            k, v = (z.repeat_interleave(n // kv, dim=1) for z in (k, split("v_proj", kv)))
            x = x + _attend(q, k, v, 128 ** -0.5, 0).flatten(1) @ at("self_attn.o_proj").T
            h = _norm(x, at("post_attention_layernorm"))
            x = x + (_silu(h @ at("mlp.gate_proj").T) * (h @ at("mlp.up_proj").T)) @ at("mlp.down_proj").T
        last = max(1, case["steps"])
        out.append(_norm(x[-last:], t["model.norm.weight"]) @ t["model.embed_tokens.weight"].T)
    return [torch.stack([o[i] for o in out]) for i in range(max(1, case["steps"]))]


def _exact_part(case, seed):
    part, _, p, stored, h, bring, held, need, cache, blocks = _inputs(case, seed)
    t = {k: v.double() for k, v in stored.items()}
    h = h.double()
    if need is None:
        return [_exact_experts(case, p, t, h)]
    after = cache.double().clone()
    out, at = [], 0
    for s in range(case["requests"]):
        rows = h[at:at + bring[s]]
        at += bring[s]
        if need.kind == "state":
            old = after[0, int(blocks[s])]
            y, new = {"scan": _exact_scan, "ssd": _exact_ssd, "delta": _exact_delta, "linear": _exact_linear}[case["kind"]](p, t, rows, old.clone())
            after[0, int(blocks[s])] = new.reshape(old.shape)
        else:
            y = _exact_latent(p, t, rows, after, blocks[s], held[s])
        out.append(y)
    return [torch.cat(out), after]


def _exact_scan(p, t, h, state):
    i, n, r, k = p["inner"], p["state"], p["dt_rank"], p["taps"] - 1
    x, z = (h @ t["in_proj"].T).split(i, dim=-1)
    x, keep = _conv(x, t["conv"], t["conv_bias"], state[:k * i].view(k, i))
    dt, b, c = (x @ t["x_proj"].T).split((r, n, n), dim=-1)
    dt = _softplus(dt @ t["dt_proj"].T + t["dt_bias"])
    a, m, ys = -t["A_log"].exp(), state[k * i:].view(i, n), []
    for j in range(h.shape[0]):
        m = (dt[j, :, None] * a).exp() * m + (dt[j] * x[j])[:, None] * b[j]
        ys.append(m @ c[j])
    y = (torch.stack(ys) + t["D"] * x) * _silu(z)
    return y @ t["o_proj"].T, torch.cat([keep.flatten(), m.flatten()])


def _exact_ssd(p, t, h, state):
    n, v, m, k = p["num_heads"], p["value_dim"], p["state"], p["taps"] - 1
    i = n * v
    z, u, dt = (h @ t["in_proj"].T).split((i, i + 2 * m, n), dim=-1)
    u, keep = _conv(u, t["conv"], t["conv_bias"], state[:k * (i + 2 * m)].view(k, -1))
    x, b, c = u.split((i, m, m), dim=-1)
    x, dt = x.view(-1, n, v), _softplus(dt + t["dt_bias"])
    e, S, ys = (-t["A_log"].exp() * dt).exp(), state[k * (i + 2 * m):].view(n, v, m), []
    for j in range(h.shape[0]):
        S = e[j, :, None, None] * S + (dt[j, :, None] * x[j])[..., None] * b[j]
        ys.append(S @ c[j])
    y = (torch.stack(ys) + t["D"][:, None] * x).flatten(1) * _silu(z)
    return _norm(y, t["norm"]) @ t["o_proj"].T, torch.cat([keep.flatten(), S.flatten()])


def _exact_delta(p, t, h, state):
    n, nk, d, k = p["num_heads"], p["num_qk_heads"], p["head_dim"], p["taps"] - 1
    u = torch.cat([h @ t[c + "_proj"].T for c in "qkv"], dim=-1)
    u, keep = _conv(u, torch.cat([t[c + "_conv"] for c in "qkv"]), None, state[:k * u.shape[1]].view(k, -1))
    q, kk, v = u.split((nk * d, nk * d, n * d), dim=-1)
    unit = lambda a: (lambda b: b / torch.sqrt(b.square().sum(-1, keepdim=True) + 1e-6))(a.view(-1, nk, d)).repeat_interleave(n // nk, dim=1)
    q, kk, v = unit(q) * d ** -0.5, unit(kk), v.view(-1, n, d)
    beta = torch.sigmoid(h @ t["b_proj"].T)
    g = (-t["A_log"].exp() * _softplus(h @ t["a_proj"].T + t["dt_bias"])).exp()
    S, os = state[k * u.shape[1]:].view(n, d, d), []
    for j in range(h.shape[0]):
        S = g[j, :, None, None] * S
        S = S + kk[j][..., None] * (beta[j, :, None] * (v[j] - (S * kk[j][..., None]).sum(1)))[:, None]
        os.append((S * q[j][..., None]).sum(1))
    o = _norm(torch.stack(os), t["norm"]).flatten(1) * _silu(h @ t["g_proj"].T)
    return o @ t["o_proj"].T, torch.cat([keep.flatten(), S.flatten()])


def _exact_linear(p, t, h, state):
    n, d = p["num_heads"], p["head_dim"]
    q, k, v = (_silu(h @ t[c + "_proj"].T).view(-1, n, d) for c in "qkv")
    decay, S, os = torch.tensor(p["decay"], device="cuda").float().double()[:, None, None], state.view(n, d, d), []
    for j in range(h.shape[0]):
        S = decay * S + k[j][..., None] * v[j][:, None]
        os.append((S * q[j][..., None]).sum(1))
    o = _norm(torch.stack(os).flatten(1), t["norm"]) * torch.sigmoid(h @ t["g_proj"].T)
    return o @ t["o_proj"].T, S


def _exact_latent(p, t, h, cache, blocks, held):
    n, d, r, rot = p["num_heads"], p["head_dim"], p["kv_rank"], p["rot_dim"]
    pos = held + torch.arange(h.shape[0], device="cuda")
    q = (_norm(h @ t["dq_proj"].T, t["dq_norm"]) @ t["uq_proj"].T if p["q_rank"] else h @ t["q_proj"].T).view(-1, n, d + rot)
    down = h @ t["dkv_proj"].T
    c = _norm(down[:, :r], t["dkv_norm"])
    if rot:
        c = torch.cat([c, _pairs(down[:, r:], pos, 10000.0)], dim=-1)
        q = torch.cat([q[..., :d], _pairs(q[..., d:], pos, 10000.0)], dim=-1)
    cache[0, _slots(blocks, held, held + h.shape[0])] = c
    lat = cache[0, _slots(blocks, 0, held + h.shape[0])]
    k = (lat[:, :r] @ t["uk_proj"].T).view(-1, n, d)
    if rot:
        k = torch.cat([k, lat[:, None, r:].expand(-1, n, -1)], dim=-1)
    o = _attend(q, k, (lat[:, :r] @ t["uv_proj"].T).view(-1, n, d), (d + rot) ** -0.5, held, p.get("window") or 1 << 30, t.get("sink"))
    o = o.flatten(1)
    if p.get("out_gate"):
        o = o * torch.sigmoid(h @ t["g_proj"].T)
    return o @ t["o_proj"].T


def _exact_experts(case, p, t, h):
    gated, e, top = case["gated"], p["num_experts"], p["top"]
    z = h @ t["router"].T
    s = torch.sigmoid(z) if gated else z.softmax(-1)
    open_ = s
    if not gated:
        best = s.view(-1, 8, e // 8).amax(-1)
        kept = torch.zeros_like(best).scatter_(1, best.topk(4, dim=-1).indices, 1.0)
        open_ = s.masked_fill(kept.repeat_interleave(e // 8, dim=1) == 0, -1.0)
    ids = open_.topk(top, dim=-1).indices
    wts = s.gather(1, ids)
    gelu = torch.nn.functional.gelu
    y = torch.zeros_like(h)
    for j in range(e):
        tok, which = (ids == j).nonzero(as_tuple=True)
        a, w = h[tok], wts[tok, which][:, None]
        up, down = t["experts.%d.up" % j], t["experts.%d.down" % j]
        if gated:
            b = (_silu(a * w @ t["experts.%d.gate" % j].T) * (a * w @ up.T)) @ down.T
        else:
            b = w * (gelu(a @ up.T) @ down.T)
        y.index_add_(0, tok, b)
    if gated:
        shared = (_silu(h @ t["shared.gate_proj"].T) * (h @ t["shared.up"].T)) @ t["shared.down"].T
        return y + shared * torch.sigmoid(h @ t["shared.gate"].T)
    return y + gelu(h @ t["shared.up"].T) @ t["shared.down"].T
