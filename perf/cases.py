"""The work that performance is followed on: what users of this library have it do, at sizes of real models' layers.

Three kinds of path:

  decode   a decode step of a whole model through `LanguageModel.step`: every sequence brings one token behind its
           cached ones, logits of all of them come back.  The step is taken again and again at the same positions, as
           a program does that scores several candidates for the next token.
  block    one layer over the tokens of a step that brings prompts or portions of prompts: embedding, the layer's
           block and the final norm, through the parts' own `step`; the normed stream of every token comes back.
  feed     a feed-forward part alone on given rows.

Weights, token ids and rows come from the seed alone.  `exact` restates the same arithmetic in 64 bits with plain
torch.
"""
import math
import zlib

import numpy as np
import torch

from garlic_inference_b200.config.base import LayerSpec, ModelPlan, PartSpec, ScheduleEntry
from garlic_inference_b200.engine import DecoderModel, LanguageModel, StepEntry
from garlic_inference_b200.parts import Runtime, StepContext, StepShape, part_class

DEV = "cuda"
EPS = 1e-6
VOCAB = {"decode": 32000, "block": 4096}

# widths, heads and feed-forwards of dense models' layers (the last three are the benchmark's and its studies')
SIZES = {
    "small": dict(hidden=1024, heads=16, kv_heads=8, inter=3072),
    "1b": dict(hidden=2048, heads=16, kv_heads=4, inter=5632),
    "8b": dict(hidden=4096, heads=32, kv_heads=8, inter=12288),
    "14b": dict(hidden=5120, heads=40, kv_heads=8, inter=17408),
}


def _case(name, path, size, *, mixer="gqa", ff="swiglu", dtype="bfloat16", sequences=1, tokens=1, past=0, ragged=False,
          layers=1, head_dim=128):
    c = dict(path=path, size=size, mixer=mixer, ff=ff, dtype=dtype, sequences=sequences, tokens=tokens, past=past,
             ragged=ragged, layers=layers, head_dim=head_dim)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one user waiting for the next token: the smallest call, all latency and launches
        _case("decode_one", "decode", "8b", past=2048, layers=4),
        # the benchmark's batch: eight conversations of 2,048 tokens
        _case("decode_eight", "decode", "8b", sequences=8, past=2048, layers=4),
        # a busy server: many conversations of all lengths, a wider model with five query heads to a key/value head
        _case("decode_ragged_48", "decode", "14b", sequences=48, past=4000, ragged=True, layers=2),
        # a busy server of a latent-attention model
        _case("decode_latent_20", "decode", "8b", mixer="latent", sequences=20, past=4000, ragged=True, layers=2),
        # a whole prompt of the benchmark's length
        _case("prompt_2048", "block", "8b", tokens=2048),
        # what a server's scheduler puts together: several portions of prompts, some behind cached tokens, heads of 64
        _case("prompt_ragged_heads_64", "block", "1b", sequences=7, tokens=700, past=2500, ragged=True, head_dim=64),
        # the exact 32-bit engine that results are checked on
        _case("prompt_float32", "block", "1b", dtype="float32", sequences=2, tokens=300, ragged=True),
        # differential attention behind short filters: two softmax maps of 64 over values of 128
        _case("prompt_differential", "block", "8b", mixer="differential", ff="none", tokens=2048),
        # the gated delta rule with a decay per channel
        _case("prompt_delta_rule", "block", "8b", mixer="delta", ff="none", tokens=2048),
        # the real-gated linear recurrent unit over several prompts
        _case("prompt_rglru_ragged", "block", "8b", mixer="rglru", ff="none", sequences=4, tokens=900, ragged=True),
        # attention over a low-rank latent with a rotated part
        _case("prompt_latent", "block", "8b", mixer="latent", ff="none", tokens=2048),
        # the routed feed-forward of a decode step of 64 sequences
        _case("experts_64", "feed", "8b", mixer="none", ff="experts", tokens=64),
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["decode", "decode", "block", "block", "block", "feed"])
    if path == "decode":
        mixer = rng.choice(["gqa", "gqa", "latent"])
        size = rng.choice(["small", "1b", "8b", "14b"] if mixer == "gqa" else ["1b", "8b"])
        n = _spread(rng, 1, 64 if mixer == "gqa" else 32)
        return _case(None, path, size, mixer=mixer, sequences=n, past=_spread(rng, 20, min(6000, 190000 // n)), ragged=n > 1, layers=2,
                     head_dim=rng.choice([64, 128, 128]) if mixer == "gqa" else 128)
    if path == "feed":
        return _case(None, path, rng.choice(["1b", "8b"]), mixer="none", ff=rng.choice(["experts", "swiglu"]),
                     tokens=_spread(rng, 1, 1500))
    if rng.random() < 0.2:
        n = rng.randint(1, 4)
        return _case(None, path, rng.choice(["small", "1b"]), dtype="float32", sequences=n, tokens=_spread(rng, 10, 400) // n + 1,
                     past=rng.choice([0, rng.randint(1, 300)]), ragged=True, head_dim=rng.choice([64, 128]))
    n = _spread(rng, 1, 8)
    mixer = rng.choice(["gqa", "gqa", "differential", "distance", "delta", "rglru", "latent"])
    tokens = max(2, min(_spread(rng, 40, 2048), 2048 // n))
    return _case(None, path, rng.choice(["small", "1b", "8b"] if mixer == "gqa" else ["1b", "8b"]), mixer=mixer,
                 ff="swiglu" if mixer == "gqa" else "none", sequences=n, tokens=tokens, ragged=n > 1,
                 past=rng.choice([0, _spread(rng, 10, 3000)]) if mixer in ("gqa", "distance", "latent") else 0,
                 head_dim=rng.choice([64, 128]) if mixer == "gqa" else 128)


# ---- shapes ---------------------------------------------------------------------------------------------------------
def _lengths(case):
    """(new tokens, cached tokens) of each sequence: the longest first, the others spread evenly by the golden ratio."""
    n = case["sequences"]
    if case["path"] == "feed":
        return [case["tokens"]], [0]
    part = lambda i, a: 1.0 if i == 0 or not case["ragged"] else 0.05 + 0.95 * ((i * 0.6180339887 + a) % 1.0)
    lens = [max(1, int(case["tokens"] * part(i, 0.0))) for i in range(n)]
    past = [int(case["past"] * part(i, 0.0 if case["path"] == "decode" else 0.37)) for i in range(n)]
    if case["path"] == "block" and case["ragged"] and n > 2:
        past[n // 2] = 0                             # one of them only begins
    return lens, past


def _mixer(case):
    """(kind, params, position part's params or None, names of its tensors)"""
    s = SIZES[case["size"]]
    hid, H, G, d = s["hidden"], s["heads"], s["kv_heads"], case["head_dim"]
    m = case["mixer"]
    if m == "gqa":
        return ("gqa_attention", dict(hidden_size=hid, n_heads=H * 128 // d, n_kv_heads=G * 128 // d, head_dim=d, qk_norm=True,
                                      qk_norm_eps=EPS, window=None, softmax_scale=d ** -0.5),
                dict(head_dim=d, rotary_dim=d, theta=1e6, max_positions=8192))
    if m == "latent":
        return ("latent_attention", dict(hidden_size=hid, n_heads=H, plain_dim=128, rot_dim=64, value_dim=128, kv_rank=512,
                                         q_rank=3 * hid // 8, softmax_scale=192 ** -0.5, eps=EPS, head_gate=True, own_kv=True),
                dict(head_dim=64, rotary_dim=64, theta=1e4, max_positions=8192, layout="half", tables=False))
    if m == "differential":
        return ("masked_attention", dict(hidden_size=hid, n_heads=H // 2, n_kv_heads=max(1, H // 8), key_dim=64, value_dim=128,
                                         softmax_scale=64 ** -0.5, mask={"kind": "chunk", "size": 2048}, maps=2, diff=0.6,
                                         sub_norm_eps=EPS, out_mul=0.4, conv_taps=4, head_gate=True), None)
    if m == "distance":
        return ("masked_attention", dict(hidden_size=hid, n_heads=H, n_kv_heads=max(1, H // 4), key_dim=128, value_dim=64,
                                         softmax_scale=128 ** -0.5, mask={"kind": "causal"}, projection_norm_eps=EPS,
                                         distance_bias={"rows": 64, "max_distance": 2048},
                                         query_temperature={"coef": 0.1, "every": 512}), None)
    if m == "delta":
        rank = max(8, hid // 16)
        return ("gated_delta_rule", dict(hidden_size=hid, n_heads=H // 2, n_kv_heads=max(1, H // 4), key_dim=128, value_dim=128,
                                         conv_taps=4, eps=EPS, unit_eps=1e-6, decay_per="channel", decay_rank=rank,
                                         gate_rank=rank, out_gate="sigmoid"), None)
    if m == "rglru":
        return ("rglru", dict(hidden_size=hid, width=hid * 5 // 4, blocks=hid // 256, conv_taps=4, decay_scale=8.0), None)
    raise ValueError(m)


def _feed(case):
    s = SIZES[case["size"]]
    if case["ff"] == "swiglu":
        return "swiglu_mlp", dict(hidden_size=s["hidden"], intermediate_size=s["inter"])
    if case["ff"] == "experts":
        ff, unit = s["inter"] * 3 // 4, dict(activation="swish", swish_alpha=1.702, gate_max=7.0, up_limit=7.0, up_shift=1.0)
        return "routed_experts", dict(hidden_size=s["hidden"], expert_size=ff, n_experts=16, top=2, expert="glu", **unit,
                                      scores="sigmoid", correction=True, groups=4, groups_kept=2, group_score="top2_sum",
                                      normalize=True, weight_scale=2.5, shared=dict(size=ff // 2, **unit))
    return None


def _spec(kind, params, prefix):
    return PartSpec(kind, params, {n: prefix + n for n in part_class(kind).wanted(params)})


def _plan(case):
    hid, vocab = SIZES[case["size"]]["hidden"], VOCAB[case["path"]]
    kind, params, rot = _mixer(case)
    feed = _feed(case)
    norm = lambda name: PartSpec("rms_norm", dict(size=hid, eps=EPS), dict(weight=name))
    layers = []
    for i in range(case["layers"]):
        p = f"l{i}."
        norms = {"input": norm(p + "in.norm"), **({"post_mixer": norm(p + "post.norm")} if feed else {})}
        layers.append(LayerSpec("pre_norm_residual", _spec(kind, params, p + "mix."),
                                _spec(*feed, p + "ff.") if feed else None, norms, "rot" if rot else None))
    return ModelPlan("cases", hid, vocab, 8192, PartSpec("token_embedding", dict(vocab_size=vocab, hidden_size=hid), dict(weight="embed")),
                     {"rot": PartSpec("rotary", rot)} if rot else {}, tuple(layers),
                     tuple(ScheduleEntry(i, i) for i in range(case["layers"])), norm("final.norm"),
                     PartSpec("linear_head", dict(hidden_size=hid, vocab_size=vocab), dict(weight="head")))


# ---- weights and inputs ---------------------------------------------------------------------------------------------
class _Weights:
    """Random tensors by name: the spreads that trained layers have, so that attention, gates, decays and routers work
    where they work in earnest.  Stored as the engine keeps them: bfloat16, or float32 for the 32-bit engine."""

    def __init__(self, case, seed):
        self.seed = seed
        self.dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
        self.shapes = {}

    def want(self, spec):
        for local, w in part_class(spec.kind).wanted(spec.params).items():
            self.shapes[spec.weights[local]] = tuple(w.shape)

    def stored_dtype(self, name):
        return self.dtype

    def tensor(self, name):
        shape = self.shapes[name]
        g = torch.Generator(device=DEV).manual_seed((zlib.crc32(name.encode()) << 20) + self.seed)
        z = lambda: torch.randn(shape, generator=g, device=DEV)
        u = lambda lo, hi: torch.rand(shape, generator=g, device=DEV) * (hi - lo) + lo
        last = name.rsplit(".", 1)[-1]
        if last == "norm" or last in ("q_norm", "k_norm"):
            t = 1.0 + 0.1 * z()
        elif last == "A_log":
            t = torch.log(u(1.0, 16.0))
        elif last == "dt_bias":
            t = torch.log(torch.expm1(torch.exp(u(math.log(1e-3), math.log(0.1)))))
        elif last == "lam":
            t = torch.log(torch.expm1(-torch.log(u(0.9, 0.999)) / 8.0))
        elif last == "embed":
            t = z()
        elif last == "conv":
            t = 0.5 * z()
        elif last in ("lq1", "lk1", "lq2", "lk2"):
            t = 0.1 * z()
        elif last == "rel":
            t = 0.5 * z()
        elif last in ("b", "correction") and len(shape) < 2 or name.endswith((".ra.b", ".ri.b")):
            t = 0.05 * z()
        else:
            t = z() * shape[-1] ** -0.5
        return t.to(self.dtype)


def _weights(case, seed):
    w = _Weights(case, seed)
    if case["path"] == "feed":
        w.want(_spec(*_feed(case), "ff."))
        return w
    plan = _plan(case)
    for s in (plan.embedding, plan.final_norm, plan.head):
        w.want(s)
    for layer in plan.layers:
        for s in (layer.mixer, layer.feed_forward, *layer.norms.values()):
            if s is not None:
                w.want(s)
    return w


def _tokens(case, seed):
    """Token ids of each sequence, cached ones first."""
    lens, past = _lengths(case)
    r = np.random.default_rng([seed & 0x7fffffff, 7])
    return [r.integers(0, VOCAB[case["path"]], size=p + n) for n, p in zip(lens, past)]


def _rows(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed + 11)
    return torch.randn((case["tokens"], SIZES[case["size"]]["hidden"]), generator=g, device=DEV).to(
        torch.float32 if case["dtype"] == "float32" else torch.bfloat16)


class _Loader:
    """Hands a part its tensors by their local names."""

    def __init__(self, spec, weights):
        self.spec, self.weights = spec, weights

    def dtype(self, *names):
        return self.weights.dtype

    def __call__(self, local, out=None):
        t = self.weights.tensor(self.spec.weights[local])
        return t if out is None else out.copy_(t)


def prepare(case, seed):
    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    rt = Runtime(dtype, dev)
    weights = _weights(case, seed)
    lens, past = _lengths(case)
    if case["path"] == "feed":
        spec = _spec(*_feed(case), "ff.")
        part = part_class(spec.kind)(spec.params, _Loader(spec, weights), rt)
        n = case["tokens"]
        ctx = StepContext(n, torch.zeros(n, dtype=torch.int32, device=dev), torch.arange(n, dtype=torch.int32, device=dev),
                          torch.zeros(n, dtype=torch.int32, device=dev), [0], [0], [n], [0], n == 1, n)
        return dict(path="feed", part=part, x=_rows(case, seed), ctx=ctx)
    room = sum((p + n) // 64 * 64 + 128 for p, n in zip(past, lens))
    lm = LanguageModel(None, DecoderModel(_plan(case), weights, rt), max_tokens=room, max_slots=case["sequences"])
    ids = _tokens(case, seed)
    slots = [lm.alloc_slot() for _ in ids]
    for s, t, p in zip(slots, ids, past):             # the cached tokens, a portion at a time
        for a in range(0, p, 2048):
            lm.step([(s, t[a:min(p, a + 2048)].tolist(), [])])
    if case["path"] == "decode":
        state = dict(path="decode", lm=lm, slots=np.asarray(slots), past=np.asarray(past),
                     entries=[StepEntry(s, [int(t[-1])], [0]) for s, t in zip(slots, ids)])
        run(state)                                    # the first step of a batch size records it
        return state
    model, cache = lm.model, lm.engine.cache
    cache.prepare(slots, lens)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    i32 = lambda parts: torch.from_numpy(np.concatenate(parts).astype(np.int32)).to(dev)
    shape = StepShape(slots, starts, lens, past, all(n == 1 for n in lens))
    ctx = StepContext(sum(lens), i32([t[p:] for t, p in zip(ids, past)]),
                      i32([np.arange(p, p + n) for n, p in zip(lens, past)]), i32([np.full(n, s) for n, s in zip(lens, slots)]),
                      slots, starts, lens, past, shape.all_single, max(p + n for n, p in zip(lens, past)),
                      arrays={k: torch.from_numpy(a).to(dev) for k, a in model.step_arrays(shape, cache).items()},
                      status=cache.status)
    return dict(path="block", model=model, ctx=ctx, view=cache.view(0), lm=lm)


def run(state):
    if state["path"] == "feed":
        return state["part"].step(state["x"], state["ctx"])
    if state["path"] == "decode":
        state["lm"].engine.cache.lengths[state["slots"]] = state["past"]      # the candidate before is taken back
        return state["lm"].step(state["entries"])
    model, ctx, view = state["model"], state["ctx"], state["view"]
    if view.state is not None:
        view.state.zero_()                            # every sequence begins
    residual = model.embedding.step(ctx)
    delta = model.blocks[0].step(None, residual, ctx, view, True)
    return model.final_norm.add_norm(delta, residual)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------
def work(case):
    lens, past = _lengths(case)
    n = sum(lens)
    size = 4 if case["dtype"] == "float32" else 2
    hid = SIZES[case["size"]]["hidden"]
    nbytes = flops = 0.0

    def matrices(spec):
        return sum(math.prod(s) for name, s in _shapes(spec).items())

    def _shapes(spec):
        return {k: tuple(w.shape) for k, w in part_class(spec[0]).wanted(spec[1]).items()}

    feed = _feed(case)
    if feed and case["ff"] == "swiglu":
        nbytes, flops = matrices(feed) * size, 2.0 * n * matrices(feed)
    elif feed:
        p = feed[1]
        one, shared = 3 * hid * p["expert_size"], 3 * hid * p["shared"]["size"]
        seen = p["n_experts"] * (1.0 - (1.0 - p["top"] / p["n_experts"]) ** n)     # experts that some row chooses
        nbytes = (seen * one + shared + p["n_experts"] * hid) * size
        flops = 2.0 * n * (p["top"] * one + shared + p["n_experts"] * hid)
    if case["path"] == "feed":
        return {"bytes": nbytes + 2.0 * n * hid * size, "flops": flops}
    kind, p, _ = _mixer(case)
    w = matrices((kind, p))
    pairs = sum(sum(range(q + 1, q + t + 1)) for t, q in zip(lens, past))          # (query, key) pairs seen
    cached = sum(t + q for t, q in zip(lens, past))
    nbytes, flops = nbytes + w * size, flops + 2.0 * n * w
    m = case["mixer"]
    if m == "gqa":
        nbytes += cached * 2 * p["n_kv_heads"] * p["head_dim"] * size
        flops += 4.0 * pairs * p["n_heads"] * p["head_dim"]
    elif m == "latent":
        r, H, d, dv, dr = p["kv_rank"], p["n_heads"], p["plain_dim"], p["value_dim"], p["rot_dim"]
        nbytes += cached * (r + dr) * size
        # the cheaper of attention over the latent rows and attention over expanded keys and values, whose expansion of
        # the cached ones is work too (that of the new ones is in the matrices' share)
        over_rows = 2.0 * pairs * H * (2 * r + dr)
        expanded = 2.0 * pairs * H * (d + dr + dv) + 2.0 * (cached - n) * r * H * (d + dv)
        flops += min(over_rows, expanded)
    elif kind == "masked_attention":
        nbytes += cached * p["n_kv_heads"] * (p.get("maps", 1) * p["key_dim"] + p["value_dim"]) * size
        flops += 2.0 * pairs * p["n_heads"] * p.get("maps", 1) * (p["key_dim"] + p["value_dim"])
    elif m == "delta":
        flops += 8.0 * n * p["n_heads"] * p["key_dim"] * p["value_dim"]
        nbytes += 2.0 * len(lens) * p["n_heads"] * p["key_dim"] * p["value_dim"] * 4
    if case["path"] == "decode":
        return {"bytes": case["layers"] * nbytes + VOCAB["decode"] * (hid * size + n * 4.0),
                "flops": case["layers"] * flops + 2.0 * n * hid * VOCAB["decode"]}
    return {"bytes": nbytes + 2.0 * n * hid * size, "flops": flops}


def tolerance(case):
    """About four times the distance from `exact` that was measured: 1.0e-6 for the 32-bit engine, 2e-3 to 3.6e-3 for a
    block or feed-forward in bfloat16 and up to 4.7e-3 for whole decode steps, whose roundings travel through several
    layers."""
    if case["dtype"] == "float32":
        return {"rel": 5e-6}
    return {"rel": 2e-2 if case["path"] == "decode" else 1.2e-2}


# ---- the same arithmetic in 64 bits -------------------------------------------------------------------------------------
def _rms(x, w, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(z):
    return z * torch.sigmoid(z)


def _turn_halves(x, base):
    """Dimensions i and i + n/2 of the token at position p turn by p * base^(-2i/n); x [T, heads, n]."""
    n = x.shape[-1]
    f = base ** (-2.0 * torch.arange(n // 2, dtype=torch.float64, device=x.device) / n)
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None] * f
    c, s = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., :n // 2], x[..., n // 2:]
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def _attend(q, k, v, scale, bias=None):
    """q [T, H, d], k [T, G, d], v [T, G, dv], causal; a block of queries at a time.  `bias` [H, T] by distance."""
    T, H, _ = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    j = torch.arange(T, device=q.device)
    for h in range(H):
        kk, vv = k[:, h // (H // G)], v[:, h // (H // G)]
        for a in range(0, T, 4096):
            i = j[a:a + 4096, None]
            s = q[a:a + 4096, h] @ kk.T * scale
            if bias is not None:
                s = s + bias[h][(i - j).clamp(min=0)]
            out[a:a + 4096, h] = torch.softmax(s.masked_fill(j > i, -math.inf), -1) @ vv
    return out


def _conv(x, taps):
    K = taps.shape[1]
    pad = torch.cat([torch.zeros(K - 1, x.shape[1], dtype=x.dtype, device=x.device), x])
    return sum(pad[i:i + x.shape[0]] * taps[:, i] for i in range(K))


def _mix_exact(case, w, xs):
    """The mixer over each whole sequence of xs."""
    kind, p, rot = _mixer(case)
    m = case["mixer"]
    if m in ("delta", "rglru"):
        return _recur_exact(m, p, w, xs)
    out = []
    for x in xs:
        T = x.shape[0]
        if m == "gqa":
            H, G, d = p["n_heads"], p["n_kv_heads"], p["head_dim"]
            q = _turn_halves(_rms((x @ w["q_proj"].T).view(T, H, d), w["q_norm"]), rot["theta"])
            k = _turn_halves(_rms((x @ w["k_proj"].T).view(T, G, d), w["k_norm"]), rot["theta"])
            o, wo = _attend(q, k, (x @ w["v_proj"].T).view(T, G, d), p["softmax_scale"]), w["o_proj"]
        elif m == "latent":
            H, d, dr, dv, r = (p[n] for n in ("n_heads", "plain_dim", "rot_dim", "value_dim", "kv_rank"))
            q = (_rms(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(T, H, d + dr)
            c = x @ w["dkv"].T
            kr = _turn_halves(c[:, None, r:], rot["theta"]).expand(T, H, dr)
            c = _rms(c[:, :r], w["dkv.norm"])
            k = torch.cat([(c @ w["uk"].T).view(T, H, d), kr], -1)
            q = torch.cat([q[..., :d], _turn_halves(q[..., d:], rot["theta"])], -1)
            o = _attend(q, k, (c @ w["uv"].T).view(T, H, dv), p["softmax_scale"]) * torch.sigmoid(x @ w["g"].T)[:, :, None]
            wo = w["o"]
        elif m == "differential":
            H, G, d, dv = p["n_heads"], p["n_kv_heads"], p["key_dim"], p["value_dim"]
            q = _conv(x @ w["q"].T, w["q.conv"]).view(T, H, 2, d)
            k = _conv(x @ w["k"].T, w["k.conv"]).view(T, G, 2, d)
            v = _conv(x @ w["v"].T, w["v.conv"]).view(T, G, dv)
            assert T <= p["mask"]["size"]
            lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + p["diff"]
            o = _attend(q[:, :, 0], k[:, :, 0], v, p["softmax_scale"]) - lam * _attend(q[:, :, 1], k[:, :, 1], v, p["softmax_scale"])
            o, wo = _rms(o, 1.0) * p["out_mul"] * torch.sigmoid(x @ w["g"].T)[:, :, None], w["o"]
        else:
            H, G, d, dv = p["n_heads"], p["n_kv_heads"], p["key_dim"], p["value_dim"]
            rows, far = p["distance_bias"]["rows"], p["distance_bias"]["max_distance"]
            t = p["query_temperature"]
            at = torch.arange(T, dtype=torch.float64, device=x.device)
            q = _rms(x @ w["q"].T, w["q.norm"]) * (1.0 + t["coef"] * torch.log(torch.floor((at + 1.0) / t["every"]) + 1.0))[:, None]
            k = _rms(x @ w["k"].T, w["k.norm"])
            n = at.clamp(min=1.0)
            b = rows // 2 + torch.floor(torch.log(n / (rows // 2)) / math.log(far / (rows // 2)) * (rows - rows // 2))
            b = torch.where(at < rows // 2, at, b.clamp(max=rows - 1)).long()
            o = _attend(q.view(T, H, d), k.view(T, G, d), (x @ w["v"].T).view(T, G, dv), p["softmax_scale"], w["rel"][b].T)
            wo = w["o"]
        out.append(o.reshape(T, -1) @ wo.T)
    return out


def _recur_exact(m, p, w, xs):
    """Both recurrences token by token, all sequences side by side (short ones padded behind their end)."""
    T, B = max(x.shape[0] for x in xs), len(xs)
    x = torch.stack([torch.cat([x, torch.zeros(T - x.shape[0], x.shape[1], dtype=x.dtype, device=x.device)]) for x in xs])
    conv = lambda z, taps: torch.stack([_conv(s, taps) for s in z])
    if m == "rglru":
        W, nb = p["width"], p["blocks"]
        y = torch.nn.functional.gelu(x @ w["y"].T + w["y.b"], approximate="tanh")
        # in front of a sequence the filter sees zeros, not the bias
        u = conv(x @ w["x"].T + w["x.b"], w["conv"]) + w["conv.b"]
        ub = u.view(B, T, nb, W // nb)
        r = torch.sigmoid(torch.einsum("stbi,boi->stbo", ub, w["ra"]) + w["ra.b"]).reshape(B, T, W)
        i = torch.sigmoid(torch.einsum("stbi,boi->stbo", ub, w["ri"]) + w["ri.b"]).reshape(B, T, W)
        a = torch.exp(-p["decay_scale"] * r * torch.nn.functional.softplus(w["lam"]))
        b = torch.sqrt((1.0 - a * a).clamp(min=0.0)) * i * u
        S, o = torch.zeros(B, W, dtype=x.dtype, device=x.device), torch.empty_like(b)
        for t in range(T):
            S = a[:, t] * S + b[:, t]
            o[:, t] = S
        out = (o * y) @ w["o"].T
        return [out[s, :len(xs[s])] for s in range(B)]
    H, Hk, d, dv = p["n_heads"], p["n_kv_heads"], p["key_dim"], p["value_dim"]
    unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + p["unit_eps"])
    q = unit(_silu(conv(x @ w["q"].T, w["q.conv"])).view(B, T, Hk, d)).repeat_interleave(H // Hk, 2) * d ** -0.5
    k = unit(_silu(conv(x @ w["k"].T, w["k.conv"])).view(B, T, Hk, d)).repeat_interleave(H // Hk, 2)
    v = _silu(conv(x @ w["v"].T, w["v.conv"])).view(B, T, H, dv)
    beta = torch.sigmoid(x @ w["b"].T)
    a = (x @ w["a1"].T @ w["a2"].T + w["dt_bias"]).view(B, T, H, d)
    g = torch.exp(-torch.exp(w["A_log"])[:, None] * torch.nn.functional.softplus(a))
    S, o = torch.zeros(B, H, d, dv, dtype=x.dtype, device=x.device), torch.empty_like(v)
    for t in range(T):
        S = g[:, t, :, :, None] * S
        e = beta[:, t, :, None] * (v[:, t] - (k[:, t, :, None] @ S)[:, :, 0])
        S = S + k[:, t, :, :, None] * e[:, :, None]
        o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
    o = _rms(o, w["norm"]) * torch.sigmoid(x @ w["g1"].T @ w["g2"].T).view(B, T, H, dv)
    out = o.reshape(B, T, -1) @ w["o"].T
    return [out[s, :len(xs[s])] for s in range(B)]


def _unit(p, g, u):
    g, u = g.clamp(max=p["gate_max"]), u.clamp(-p["up_limit"], p["up_limit"])
    return g * torch.sigmoid(p["swish_alpha"] * g) * (u + p["up_shift"])


def _feed_exact(case, w, x):
    if case["ff"] == "swiglu":
        return (_silu(x @ w["gate_proj"].T) * (x @ w["up_proj"].T)) @ w["down_proj"].T
    p = _feed(case)[1]
    n, E, groups = x.shape[0], p["n_experts"], p["groups"]
    s = torch.sigmoid(x @ w["router"].T)
    choice = (s + w["correction"]).view(n, groups, E // groups)
    kept = choice.topk(2, -1).values.sum(-1).topk(p["groups_kept"], -1).indices
    stays = torch.zeros(n, groups, dtype=torch.bool, device=x.device).scatter_(1, kept, True)
    idx = choice.masked_fill(~stays[:, :, None], -math.inf).view(n, E).topk(p["top"], -1).indices
    wt = s.gather(1, idx)
    wt = wt / (wt.sum(-1, keepdim=True) + 1e-20) * p["weight_scale"]
    out = _unit(p["shared"], x @ w["shared.gate"].T, x @ w["shared.up"].T) @ w["shared.down"].T
    for e in range(E):
        row, c = (idx == e).nonzero(as_tuple=True)
        if len(row):
            z = _unit(p, x[row] @ w[f"e{e}.gate"].T, x[row] @ w[f"e{e}.up"].T) @ w[f"e{e}.down"].T
            out.index_add_(0, row, z * wt[row, c, None])
    return out


def exact(case, seed):
    weights = _weights(case, seed)

    class Local:                                      # a part's tensors, widened one at a time
        def __init__(self, prefix):
            self.prefix = prefix

        def __getitem__(self, n):
            return weights.tensor(self.prefix + n).double()

    if case["path"] == "feed":
        return _feed_exact(case, Local("ff."), _rows(case, seed).double())
    lens, past = _lengths(case)
    embed = Local("")["embed"]
    hs = [embed[torch.from_numpy(t).to(DEV)] for t in _tokens(case, seed)]
    for i in range(case["layers"]):
        p = f"l{i}."
        norm, mix = Local(p)["in.norm"], Local(p + "mix.")
        hs = [h + y for h, y in zip(hs, _mix_exact(case, _Held(mix), [_rms(h, norm) for h in hs]))]
        if _feed(case):
            norm, ff = Local(p)["post.norm"], _Held(Local(p + "ff."))
            hs = [h + _feed_exact(case, ff, _rms(h, norm)) for h in hs]
    out = _rms(torch.cat([h[q:] for h, q in zip(hs, past)]), Local("")["final.norm"])
    return out @ Local("")["head"].T if case["path"] == "decode" else out


class _Held:
    """Tensors that several sequences use, widened once."""

    def __init__(self, local):
        self.local, self.held = local, {}

    def __getitem__(self, n):
        if n not in self.held:
            self.held[n] = self.local[n]
        return self.held[n]
