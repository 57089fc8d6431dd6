"""The work whose speed this repository watches, as cases that can be timed and compared.

A case is a dict of plain values; ``prepare`` builds what a program has in hand before the call
(a model of seeded weights, its cache with earlier tokens in it, the step's inputs), ``run`` makes
one pass through the package's public entry points, ``exact`` says in 64 bits, in plain torch,
what the pass computes.  Sizes are those of ``bench.py``: the Qwen3 shapes, and the other families
at the widths of those shapes.

Three kinds of pass:

* ``step``: ``ModelRunner.step`` on a Qwen3 decoder of the shape's layer sizes and vocabulary (a
  few of its layers): decode steps from CUDA graphs, and a serving step of prompt portions beside
  decoded tokens.  Logits come back.
* ``layer``: one Qwen3 layer (``PreNormBlock.forward`` on a residual stream).
* the other families' characteristic sublayers, through ``Mixer.forward`` or
  ``FeedForward.forward``: ``memory`` (matrix memory), ``beside`` (convolved window attention
  beside retention), ``delta`` (gated delta rule), ``latent`` (latent attention), ``state_space``
  (Mamba-2), ``experts`` (mixture of experts with a shared one), ``differential``
  (differential attention).

A step's batch is ``portions`` prompt portions, the longest of ``tokens`` tokens behind ``before``
cached ones, and ``rows`` single tokens behind about ``context`` cached ones.
"""
import math
import zlib

import torch

from binfer_b200.config import (FikotarConfig, FolivikConfig, GukidraConfig, KetopelConfig,
                                PabelixConfig, Qwen3Config)
from binfer_b200.engine import StepItem, make_env, make_runner
from binfer_b200.parts import ResidualStream, build_model, param_specs_for
from binfer_b200.weights import TensorSource

F64 = torch.float64
DEVICE = "cuda:0"
PAGE = 16

# width -> (attention heads, kv heads, head size, feed-forward): the Qwen3 1.7B and 8B shapes
SHAPES = {2048: (16, 8, 128, 6144), 4096: (32, 8, 128, 12288)}
STATEFUL = ("memory", "beside", "delta", "state_space")


# --------------------------------------------------------------------------------- cases
def listed():
    step = dict(kind="step", dtype="bfloat16", portions=0, tokens=0, before=0)
    sub = dict(dtype="bfloat16", layers=1, vocab=64)
    return [
        # one user's decode step in a short conversation: latency and launches
        dict(step, name="decode_one", width=4096, layers=4, vocab=151936, rows=1, context=519),
        # the headline: eight requests with 4k tokens of context each
        dict(step, name="decode_eight", width=4096, layers=3, vocab=151936, rows=8, context=4096),
        # continuous batching under load: two prompt portions (one of them behind an earlier
        # portion) beside thirty decoded tokens
        dict(step, name="serving_step", width=2048, layers=4, vocab=151936, portions=2,
             tokens=1013, before=700, rows=30, context=900),
        # a prompt of 2,048 tokens through one layer of the 8B shape
        dict(sub, name="prompt_layer", kind="layer", width=4096, portions=1, tokens=2048,
             before=0, rows=0, context=0),
        # the engine's 32-bit path, which people check a checkpoint or a port against
        dict(sub, name="prompt_layer_float32", kind="layer", dtype="float32", width=2048,
             portions=1, tokens=333, before=0, rows=0, context=0),
        # a long prompt through a matrix memory layer
        dict(sub, name="memory_prompt", kind="memory", width=4096, portions=1, tokens=2048,
             before=0, rows=0, context=0),
        # prompts of several users, and users that already decode, in one step of window
        # attention beside retention
        dict(sub, name="beside_mixed", kind="beside", width=2048, portions=2, tokens=1300,
             before=0, rows=6, context=90),
        # two prompts of odd lengths through a delta rule layer
        dict(sub, name="delta_prompts", kind="delta", width=2048, portions=2, tokens=1111,
             before=0, rows=0, context=0),
        # the second portion of a prompt through latent attention
        dict(sub, name="latent_portion", kind="latent", width=2048, portions=1, tokens=1800,
             before=500, rows=0, context=0),
        # a prompt through a state space layer beside users that decode
        dict(sub, name="state_space_mixed", kind="state_space", width=2048, portions=1,
             tokens=2000, before=0, rows=8, context=60),
        # a full step of tokens through a mixture of experts
        dict(sub, name="experts_prompt", kind="experts", width=2048, portions=1, tokens=2048,
             before=0, rows=0, context=0),
        # a long prompt through differential attention
        dict(sub, name="differential_prompt", kind="differential", width=4096, portions=1,
             tokens=1999, before=0, rows=0, context=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Decode steps of 1 to 48 requests behind 60 to 4,000 tokens, serving steps, layers of
    prompt portions of 130 to 2,048 tokens with up to a dozen single tokens beside them."""
    kind = rng.choice(["step", "step", "layer", "memory", "beside", "delta", "latent",
                       "state_space", "experts", "differential"])
    width = rng.choice([2048, 4096])
    if kind == "step":
        mixed = rng.random() < 0.4
        rows = _log(rng, 1, 48)
        return dict(kind=kind, dtype="bfloat16", width=width, layers=rng.choice([2, 3]),
                    vocab=rng.choice([32000, 151936]), portions=rng.randint(1, 2) if mixed else 0,
                    tokens=_log(rng, 130, 1100) if mixed else 0,
                    before=rng.choice([0, rng.randint(1, 900)]) if mixed else 0, rows=rows,
                    context=_log(rng, 60, min(4000, 32000 // rows)))
    f32 = kind == "layer" and rng.random() < 0.4
    tokens = _log(rng, 130, 400 if f32 else 2048)
    portions = rng.choice([1, 1, 2, 3]) if tokens < 1200 else 1
    rows = rng.choice([0, 0, rng.randint(1, 12)])
    attends = kind in ("layer", "latent", "differential")
    return dict(kind=kind, dtype="float32" if f32 else "bfloat16", width=2048 if f32 else width,
                layers=1, vocab=64, portions=portions, tokens=tokens,
                before=rng.choice([0, rng.randint(1, 800)]) if attends and not f32 else 0,
                rows=rows, context=rng.randint(20, 500 if attends else 90))


def _requests(c):
    """(cached tokens, tokens of this step) of every request: the portions get shorter from one to
    the next, single tokens have contexts of different lengths."""
    out = [(c["before"] if i == 0 else 0, max(2, c["tokens"] * (8 - 3 * i) // 8))
           for i in range(c["portions"])]
    return out + [(max(1, c["context"] - (c["context"] // 64 + 1) * i), 1)
                  for i in range(c["rows"])]


# ----------------------------------------------------------------------- models and weights
def _config(c):
    w, kind = c["width"], c["kind"]
    heads, kv, d, ff = SHAPES[w]
    if kind in ("step", "layer"):
        return Qwen3Config.from_dict(dict(
            architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=c["layers"],
            hidden_size=w, num_attention_heads=heads, num_key_value_heads=kv, head_dim=d,
            intermediate_size=ff, vocab_size=c["vocab"], rope_theta=1e6, rms_norm_eps=1e-6,
            tie_word_embeddings=True, max_position_embeddings=40960, hidden_act="silu",
            attention_bias=False, use_sliding_window=False))
    raw = {"vocab": c["vocab"], "width": w, "norm": {"eps": 1e-5}}
    layer = {"mixer": _mixer(c), "mlp": None}
    if kind == "memory":
        return GukidraConfig.from_dict(dict(raw, embedding={"scale": 8.0},
                                            layers=[dict(layer, type="mlstm")]))
    if kind in ("beside", "experts"):
        mlp = {"kind": "moe", "router": {"experts": 8, "top": 2}, "expert": {"ff": ff // 4},
               "shared": {"ff": ff // 2}}
        return FikotarConfig.from_dict(dict(raw, logit_scale=1.0, layers=[
            dict(layer, type="parallel", mlp=mlp if kind == "experts" else None)]))
    if kind == "delta":
        return KetopelConfig.from_dict(dict(raw, embedding={"scale": 1.0},
                                            layers=[dict(layer, type="delta")]))
    if kind == "differential":
        return PabelixConfig.from_dict(dict(raw, layers=[dict(layer, type="attention")]))
    return FolivikConfig.from_dict(dict(raw, layers=[dict(
        layer, type="mamba2" if kind == "state_space" else "latent_attention")]))


def _mixer(c):
    """The mixer's sizes in the family's own words."""
    w, kind = c["width"], c["kind"]
    heads, kv, d, _ = SHAPES[w]
    if kind == "memory":
        return {"heads": w // 512, "dim": 256, "vdim": 512, "gate_cap": 15.0}
    if kind in ("beside", "experts"):
        rh = w // 256
        return {"left": {"heads": heads, "kv_heads": kv, "dim": d, "vdim": d, "conv": 3,
                         "scale": d ** -0.5, "mask": {"size": 1024, "keep_first": 4},
                         "rot": {"base": 1e6, "dims": d // 2}},
                "right": {"heads": rh, "dim": 128, "vdim": 256, "rot": {"base": 1e6, "dims": 128},
                          "decay": [1.0 - 2.0 ** (-5 - 4.0 * i / (rh - 1)) for i in range(rh)]},
                "left_scale": 1.0, "right_scale": 1.0}
    if kind == "delta":
        return {"heads": w // 128, "kv_heads": w // 256, "dim": 128, "vdim": 128, "conv": 4}
    if kind == "differential":
        return {"heads": heads, "kv_heads": kv, "dim": d // 2, "vdim": d,
                "scale": (d // 2) ** -0.5, "diff": 0.5, "q_temp": {"coef": 0.1, "every": 1024}}
    if kind == "state_space":
        return {"heads": 2 * w // 64, "vdim": 64, "state": 128, "groups": 8, "conv": 4,
                "norm_groups": 8}
    return {"heads": heads, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512,
            "q_rank": 3 * w // 8, "scale": 192 ** -0.5, "rot": {"base": 1e4, "dims": 64}}


def _generator(seed, name):
    g = torch.Generator(DEVICE)
    g.manual_seed((int(seed) * 1_000_003 + zlib.crc32(name.encode())) & 0x7FFF_FFFF_FFFF)
    return g


def _weight(c, seed, name, shape):
    """A checkpoint's tensor: matrices keep the size of what they multiply, norms lie about one,
    gates and decays where trained models have them; matrices in the engine's precision."""
    x = torch.empty(shape, dtype=torch.float32, device=DEVICE)
    x.normal_(generator=_generator(seed, name))
    leaf = name.split(".")[-1]
    if name.endswith("f.b"):
        return x.add_(4.0)                        # forget gates that remember
    if leaf == "dt_bias":
        return x.sub_(3.0)                        # steps of about 0.05
    if leaf == "A_log":
        return x.mul_(0.5).add_(1.0)
    if leaf == "conv":
        return x.mul_(0.5)
    if leaf in ("router", "sg"):
        return x.mul_(2.0 * shape[-1] ** -0.5)
    if leaf in ("b", "sink", "lq1", "lk1", "lq2", "lk2") and len(shape) == 1:
        return x.mul_(0.1)
    if len(shape) <= 1:                           # norms, and the skip of a state space layer
        return x.mul_(0.1).add_(0.0 if c["kind"] == "differential" else 1.0)
    if leaf != "embed" and "embed_tokens" not in name:
        x.mul_(shape[-1] ** -0.5)
    else:
        x.mul_(0.05)
    return x.to(torch.bfloat16) if c["dtype"] == "bfloat16" else x


def _inputs(c, seed):
    """Per request, what its cached and new tokens bring: token ids of a step, else rows."""
    out = []
    for i, (before, new) in enumerate(_requests(c)):
        g = _generator(seed, "inputs of request %d" % i)
        if c["kind"] == "step":
            out.append(torch.randint(0, c["vocab"], (before + new,), generator=g, device=DEVICE))
            continue
        x = torch.randn((before + new, c["width"]), generator=g, device=DEVICE)
        out.append(x if c["kind"] == "layer" or c["dtype"] == "float32" else x.to(torch.bfloat16))
    return out


# --------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    c = case
    env = make_env(c["dtype"], DEVICE)
    spec = _config(c).to_spec()
    shapes = {s.name: tuple(s.shape) for s in param_specs_for(spec)}
    model = build_model(spec, env, TensorSource(
        lambda name: _weight(c, seed, name, shapes[name]), shapes, where="(seeded)"))
    reqs, inputs = _requests(c), _inputs(c, seed)
    pages = sum(-(-(b + n + 1) // PAGE) + 1 for b, n in reqs) + 8
    runner = make_runner(model, env, page_size=PAGE, num_pages=pages, max_requests=len(reqs))
    for i in range(len(reqs)):
        runner.add_request(i)
    if c["kind"] == "step":
        return _prepare_step(c, runner, reqs, inputs)
    block = model.blocks[0]
    part = block if c["kind"] == "layer" else block.ffn if c["kind"] == "experts" else block.mixer
    s = {"case": c, "runner": runner, "view": runner.views[0], "part": part}
    for i, (before, _) in enumerate(reqs):        # the cached tokens, in portions
        for a in range(0, before if c["kind"] != "experts" else 0, 2048):
            b = min(before, a + 2048)
            items = [StepItem(i, [0] * (b - a))]
            runner.reserve(items)
            s["ctx"], s["x"] = runner.build_context(items), inputs[i][a:b].contiguous()
            _pass(s)
            runner.cache.commit(i, b)
    items = [StepItem(i, [0] * n) for i, (_, n) in enumerate(reqs)]
    runner.reserve(items)
    s["ctx"] = runner.build_context(items)
    s["x"] = torch.cat([x[b:] for x, (b, _) in zip(inputs, reqs)]).contiguous()
    s["slots"] = [runner.cache.get(i).slot for i in range(len(reqs))]
    s["saved"] = s["view"].state.clone() if c["kind"] in STATEFUL else None
    return s


def _prepare_step(c, runner, reqs, inputs):
    ids = [x.tolist() for x in inputs]
    for i, (before, _) in enumerate(reqs):
        for a in range(0, before, 2048):
            runner.step([StepItem(i, ids[i][a:min(before, a + 2048)])])
    items = [StepItem(i, ids[i][b:], [n - 1]) for i, (b, n) in enumerate(reqs)]
    s = {"case": c, "runner": runner, "items": items, "lengths": [b for b, _ in reqs]}
    if not c["portions"]:
        runner.enable_decode_graphs(max_batch=64, max_seq_len=4224)
        run(s)                                    # captures the graph, as a server does at its start
    return s


def _pass(s):
    if s["case"]["kind"] == "experts":
        return s["part"].forward(s["x"], s["ctx"])
    if s["case"]["kind"] != "layer":
        return s["part"].forward(s["x"], s["ctx"], s["view"])
    stream = ResidualStream(s["x"].clone())
    s["part"].forward(stream, s["ctx"], s["view"])
    stream.flush()
    return stream.x


def run(state):
    s = state
    if s["case"]["kind"] == "step":
        logits = s["runner"].step(s["items"])
        for i, n in enumerate(s["lengths"]):      # taken back, like a draft that is rejected
            s["runner"].cache.get(i).length = n
        return logits
    if s["saved"] is None:
        return _pass(s)
    s["view"].state.copy_(s["saved"])             # from the same earlier tokens every time
    y = _pass(s)
    return [y] + [s["view"].state[slot] for slot in s["slots"]]


# -------------------------------------------------------------------------------- work
def _attended(c, window=None):
    """Pairs of a new token and a key that it sees."""
    total = 0
    for before, new in _requests(c):
        if window is None or before + new <= window:
            total += new * before + new * (new + 1) // 2
        else:
            total += sum(min(window, p + 1) for p in range(before, before + new))
    return total


def work(case):
    c, w, kind = case, case["width"], case["kind"]
    heads, kv, d, ff = SHAPES[w]
    reqs = _requests(c)
    T, cached, size = sum(n for _, n in reqs), sum(b for b, _ in reqs), 4 if c["dtype"] == "float32" else 2
    if kind in ("step", "layer"):
        layer = w * (heads + 2 * kv) * d + heads * d * w + 3 * w * ff
        rows = len(reqs) if kind == "step" else 0
        flops = c["layers"] * (2.0 * T * layer + 4.0 * heads * d * _attended(c)) + 2.0 * rows * w * c["vocab"]
        head = c["vocab"] * w if kind == "step" else 0
        moved = (c["layers"] * (layer + 2 * kv * d * (cached + T)) + head) * size
        moved += rows * c["vocab"] * 4 + (0 if kind == "step" else 2 * T * w * 4)
        return {"bytes": moved, "flops": flops}
    mx = _mixer(c)
    state = core = cache = 0.0
    if kind == "memory":
        H, dk, dv = mx["heads"], mx["dim"], mx["vdim"]
        params = w * (2 * H * dk + 2 * H * dv + 2 * H) + H * dv * w
        state, core = H * dk * dv, 4.0 * T * H * dk * dv
    elif kind == "beside":
        r = mx["right"]
        H, dk, dv = r["heads"], r["dim"], r["vdim"]
        params = w * ((heads + 2 * kv) * d + 2 * H * (dk + dv)) + (heads * d + H * dv) * w
        state, core = H * dk * dv, 4.0 * T * H * dk * dv + 4.0 * heads * d * _attended(c, 1024)
        cache = 2 * kv * d
    elif kind == "delta":
        H, G, dk, dv = mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"]
        params = w * (2 * G * dk + 2 * H * dv + 2 * H) + H * dv * w
        state, core = H * dk * dv, 6.0 * T * H * dk * dv
    elif kind == "state_space":
        H, P, N, G = mx["heads"], mx["vdim"], mx["state"], mx["groups"]
        params = w * (2 * H * P + 2 * G * N + H) + H * P * w
        state, core = H * P * N, 4.0 * T * H * P * N
    elif kind == "latent":
        r, qr = mx["kv_rank"], mx["q_rank"]
        params = w * (qr + r + 64 + heads) + qr * heads * 192 + 2 * r * heads * 128 + heads * 128 * w
        core, cache = 2.0 * heads * (192 + 128) * _attended(c), r + 64
    elif kind == "experts":
        # every weight is read by some token; a token needs two experts and the shared one
        params = 3 * w * (8 * (ff // 4) + ff // 2)
        active = 3 * w * (2 * (ff // 4) + ff // 2)
        return {"bytes": 2.0 * params + 2.0 * T * 2 * w + 9 * w * 4, "flops": 2.0 * T * (active + 9 * w)}
    else:
        params = w * (2 * heads * d + 2 * kv * d) + heads * d * w
        core, cache = 2.0 * heads * 2 * (d // 2 + d) * _attended(c), 2 * kv * d
    return {"bytes": 2.0 * params + 2.0 * T * 2 * w + 8.0 * state * len(reqs) + 2.0 * cache * (T + cached),
            "flops": 2.0 * T * params + core}


# Four times the relative error that the cases show against exact(): 2^-9 roundings of products and
# activations in bfloat16 (a step's travel through all layers), the order of sums in float32.
_REL = {"step": 0.03, "layer": 0.008, "memory": 0.016, "beside": 0.017, "delta": 0.016,
        "latent": 0.022, "state_space": 0.016, "experts": 0.01, "differential": 0.018}


def tolerance(case):
    if case["dtype"] == "float32":
        return {"rel": 2e-6, "max": 1e-4}
    return {"rel": _REL[case["kind"]], "max": 0.5}


# -------------------------------------------------------------------------------- exact
def _rms(x, weight, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * weight


def _silu(z):
    return z * torch.sigmoid(z)


def _softplus(z):
    return torch.logaddexp(z, torch.zeros_like(z))


def _turn(x, base, dims, interleaved=False):
    """``x [T, heads, d]`` from position 0 on, the first ``dims`` sizes turned; the angles are a
    float's, which is how these models define them."""
    T, half = x.shape[0], dims // 2
    f = (base ** (-2.0 * torch.arange(half, dtype=F64, device=x.device) / dims)).float()
    ang = (torch.arange(T, device=x.device).float()[:, None] * f[None]).double()[:, None, :]
    c, s = torch.cos(ang), torch.sin(ang)
    out = x.clone()
    one, two = ((slice(0, dims, 2), slice(1, dims, 2)) if interleaved
                else (slice(0, half), slice(half, dims)))
    a, b = x[..., one], x[..., two]
    out[..., one], out[..., two] = a * c - b * s, b * c + a * s
    return out


def _conv(u, w, bias=None):
    taps = w.shape[1]
    y = torch.zeros_like(u) if bias is None else bias.expand_as(u).clone()
    for j in range(taps):
        back = taps - 1 - j
        if back < u.shape[0]:
            y[back:] += w[:, j] * u[:u.shape[0] - back]
    return y


def _attend(q, k, v, scale, first, window=None, keep=0, sink=None):
    """Causal attention of the queries from position ``first`` on, ``[T - first, H, dv]``."""
    T, H, G = q.shape[0], q.shape[1], k.shape[1]
    j = torch.arange(T, device=q.device)
    dist = j[first:, None] - j[None, :]
    seen = dist >= 0
    if window is not None:
        seen = seen & ((dist < window) | (j[None, :] < keep))
    out = torch.empty(T - first, H, v.shape[2], dtype=F64, device=q.device)
    for h in range(H):
        g = h // (H // G)
        s = (q[first:, h] @ k[:, g].T).mul_(scale).masked_fill_(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(T - first, 1)], dim=1)
        p = torch.softmax(s, dim=-1)
        out[:, h] = p[:, :T] @ v[:, g]
    return out


def exact(case, seed):
    c, kind = case, case["kind"]
    spec = {s.name: tuple(s.shape) for s in param_specs_for(_config(c).to_spec())}
    held = {}

    def w(name):
        if name not in held:
            held[name] = _weight(c, seed, name, spec[name]).double()
        return held[name]

    reqs, inputs = _requests(c), _inputs(c, seed)
    if kind == "step":
        return torch.cat([_decoder(c, w, ids, b + n - 1) for ids, (b, n) in zip(inputs, reqs)])
    if kind == "layer":
        return torch.cat([_qwen_layer(c, w, "model.layers.0.", x.double(), b)
                          for x, (b, _) in zip(inputs, reqs)])
    if kind == "experts":
        return torch.cat([_experts(c, w, x[b:].double()) for x, (b, _) in zip(inputs, reqs)])
    if kind in ("latent", "differential"):
        f = _latent if kind == "latent" else _differential
        return torch.cat([f(c, w, x.double(), b) for x, (b, _) in zip(inputs, reqs)])
    f = {"memory": _memory, "beside": _beside, "delta": _delta, "state_space": _state_space}[kind]
    got = [f(c, w, x.double(), b) for x, (b, _) in zip(inputs, reqs)]
    return [torch.cat([y for y, _ in got])] + [state for _, state in got]


def _qwen_layer(c, w, p, x, first):
    """The rows from position ``first`` on of the stream behind the layer."""
    heads, kv, d, _ = SHAPES[c["width"]]
    T = x.shape[0]
    h = _rms(x, w(p + "input_layernorm.weight"), 1e-6)
    q = (h @ w(p + "self_attn.q_proj.weight").T).view(T, heads, d)
    k = (h @ w(p + "self_attn.k_proj.weight").T).view(T, kv, d)
    v = (h @ w(p + "self_attn.v_proj.weight").T).view(T, kv, d)
    q = _turn(_rms(q, w(p + "self_attn.q_norm.weight"), 1e-6), 1e6, d)
    k = _turn(_rms(k, w(p + "self_attn.k_norm.weight"), 1e-6), 1e6, d)
    o = _attend(q, k, v, d ** -0.5, first).reshape(T - first, heads * d)
    x = x[first:] + o @ w(p + "self_attn.o_proj.weight").T
    h = _rms(x, w(p + "post_attention_layernorm.weight"), 1e-6)
    h = _silu(h @ w(p + "mlp.gate_proj.weight").T) * (h @ w(p + "mlp.up_proj.weight").T)
    return x + h @ w(p + "mlp.down_proj.weight").T


def _decoder(c, w, ids, row):
    x = w("model.embed_tokens.weight")[ids]
    for i in range(c["layers"]):
        x = _qwen_layer(c, w, "model.layers.%d." % i, x, row if i == c["layers"] - 1 else 0)
    return _rms(x, w("model.norm.weight"), 1e-6) @ w("model.embed_tokens.weight").T


def _memory(c, w, h, first):
    mx, p = _mixer(c), "l0.mix."
    T, H, dk, dv, cap = h.shape[0], mx["heads"], mx["dim"], mx["vdim"], mx["gate_cap"]
    q = (h @ w(p + "q").T).view(T, H, dk) * dk ** -0.5
    k, v = (h @ w(p + "k").T).view(T, H, dk), (h @ w(p + "v").T).view(T, H, dv)
    ig = cap * torch.tanh((h @ w(p + "i").T + w(p + "i.b")) / cap)
    fg = -_softplus(-cap * torch.tanh((h @ w(p + "f").T + w(p + "f.b")) / cap))
    S, n = h.new_zeros(H, dk, dv), h.new_zeros(H, dk)
    m, o = h.new_zeros(H), h.new_zeros(T, H, dv)
    for t in range(T):
        m_new = torch.maximum(fg[t] + m, ig[t])
        a, b = torch.exp(fg[t] + m - m_new), torch.exp(ig[t] - m_new)
        S = S * a[:, None, None] + (k[t] * b[:, None])[:, :, None] * v[t][:, None, :]
        n = a[:, None] * n + b[:, None] * k[t]
        m = m_new
        den = torch.maximum((n * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        o[t] = (q[t][:, None, :] @ S)[:, 0] / den[:, None]
    o = _rms(o, 1.0, 1e-5).reshape(T, H * dv)[first:] * w(p + "norm")
    y = (o * torch.sigmoid(h[first:] @ w(p + "g").T)) @ w(p + "o").T
    pad = h.new_zeros(H, 3)
    return y, torch.cat([S.reshape(H, -1), n, m[:, None], pad], dim=1)


def _beside(c, w, h, first):
    mx, T = _mixer(c), h.shape[0]
    a, p = mx["left"], "l0.mix.left."
    H, G, d = a["heads"], a["kv_heads"], a["dim"]
    raw = [h @ w(p + n).T for n in "qkv"]
    q, k, v = (_conv(u, w(p + n + ".conv")) for u, n in zip(raw, "qkv"))
    q = _rms(_turn(q.view(T, H, d), 1e6, d // 2), 1.0, 1e-5)
    k = _rms(_turn(k.view(T, G, d), 1e6, d // 2), 1.0, 1e-5)
    o = _attend(q, k, v.view(T, G, d), a["scale"], first, 1024, 4, w(p + "sink"))
    y = o.reshape(T - first, H * d) @ w(p + "o").T
    raw = torch.cat(raw, dim=1)
    tail = torch.cat([raw.new_zeros(2, raw.shape[1]), raw])[-2:]       # the convolution's reach

    r, p = mx["right"], "l0.mix.right."
    H, d, dv = r["heads"], r["dim"], r["vdim"]
    q = _turn((h @ w(p + "q").T).view(T, H, d), 1e6, d)
    k = _turn((h @ w(p + "k").T).view(T, H, d), 1e6, d) * d ** -0.5
    v = (h @ w(p + "v").T).view(T, H, dv)
    # the engine holds a decay as a float
    decay = torch.tensor(r["decay"], dtype=F64).float().double().to(h.device)
    o, S = _linear_scan(q, k, v, decay.expand(T, H))
    o = _rms(o, 1.0, 1e-5).reshape(T, H * dv)[first:]
    y = y + (o * _silu(h[first:] @ w(p + "g").T)) @ w(p + "o").T
    return y, torch.cat([tail.reshape(-1), S.transpose(1, 2).reshape(-1)])


def _linear_scan(q, k, v, decay):
    """``S <- decay S + k v^T, o = S^T q`` per head; ``(o, S)``."""
    T, H = v.shape[:2]
    S, o = v.new_zeros(H, k.shape[2], v.shape[2]), torch.empty_like(v)
    for t in range(T):
        S = S * decay[t][:, None, None] + k[t][:, :, None] * v[t][:, None, :]
        o[t] = (q[t][:, None, :] @ S)[:, 0]
    return o, S


def _delta(c, w, h, first):
    mx, p = _mixer(c), "l0.mix."
    T, H, G, d, dv = h.shape[0], mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"]
    raw = [h @ w(p + n).T for n in "qkv"]
    q, k, v = (_silu(_conv(u, w(p + n + ".conv"))) for u, n in zip(raw, "qkv"))
    q, k, v = q.view(T, G, d), k.view(T, G, d), v.view(T, H, dv)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * d ** -0.5
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q, k = q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1)
    beta = torch.sigmoid(h @ w(p + "b").T)
    decay = torch.exp(-torch.exp(w(p + "A_log")) * _softplus(h @ w(p + "a").T + w(p + "dt_bias")))
    S, o = h.new_zeros(H, d, dv), h.new_zeros(T, H, dv)
    for t in range(T):
        S = S * decay[t][:, None, None]
        u = beta[t][:, None] * (v[t] - (k[t][:, None, :] @ S)[:, 0])
        S = S + k[t][:, :, None] * u[:, None, :]
        o[t] = (q[t][:, None, :] @ S)[:, 0]
    o = _rms(o, w(p + "norm"), 1e-5).reshape(T, H * dv)[first:]
    y = (o * _silu(h[first:] @ w(p + "g").T)) @ w(p + "o").T
    raw = torch.cat(raw, dim=1)
    tail = torch.cat([raw.new_zeros(3, raw.shape[1]), raw])[-3:]
    return y, torch.cat([S.transpose(1, 2).reshape(-1), tail.reshape(-1)])


def _state_space(c, w, h, first):
    mx, p = _mixer(c), "l0.mix."
    T, H, P, N, G = h.shape[0], mx["heads"], mx["vdim"], mx["state"], mx["groups"]
    inner, parts = H * P, mx["norm_groups"]
    u = h @ w(p + "in").T
    z, raw, dt = u[:, :inner], u[:, inner:2 * inner + 2 * G * N], u[:, 2 * inner + 2 * G * N:]
    xbc = _silu(_conv(raw, w(p + "conv"), w(p + "conv.b")))
    x = xbc[:, :inner].view(T, H, P)
    B = xbc[:, inner:inner + G * N].view(T, G, N).repeat_interleave(H // G, 1)
    C = xbc[:, inner + G * N:].view(T, G, N).repeat_interleave(H // G, 1)
    dt = _softplus(dt + w(p + "dt_bias"))
    o, S = _linear_scan(C, B, x * dt[:, :, None], torch.exp(-torch.exp(w(p + "A_log")) * dt))
    y = (o + w(p + "D")[:, None] * x).reshape(T, inner) * _silu(z)
    y = _rms(y.view(T, parts, inner // parts), 1.0, 1e-5).reshape(T, inner) * w(p + "norm")
    tail = torch.cat([raw.new_zeros(3, raw.shape[1]), raw])[-3:]
    return y[first:] @ w(p + "o").T, torch.cat([S.transpose(1, 2).reshape(-1), tail.reshape(-1)])


def _latent(c, w, h, first):
    mx, p = _mixer(c), "l0.mix."
    T, H, d, dr, dv, rank = h.shape[0], mx["heads"], 128, 64, 128, 512
    q = (_rms(h @ w(p + "dq").T, w(p + "dq.norm"), 1e-5) @ w(p + "uq").T).view(T, H, d + dr)
    down = h @ w(p + "dkv").T
    lat = _rms(down[:, :rank], w(p + "dkv.norm"), 1e-5)
    k_rot = _turn(down[:, rank:].view(T, 1, dr), 1e4, dr, True)
    q = torch.cat([q[..., :d], _turn(q[..., d:], 1e4, dr, True)], dim=-1)
    k = torch.cat([(lat @ w(p + "uk").T).view(T, H, d), k_rot.expand(T, H, dr)], dim=-1)
    o = _attend(q, k, (lat @ w(p + "uv").T).view(T, H, dv), mx["scale"], first)
    o = o * torch.sigmoid(h[first:] @ w(p + "g").T)[:, :, None]
    return o.reshape(T - first, H * dv) @ w(p + "o").T


def _experts(c, w, h):
    p, act = "l0.mlp.", _silu
    vals, ids = torch.sort(h @ w(p + "router").T, dim=-1, descending=True)
    wts = torch.zeros(h.shape[0], 8, dtype=F64, device=h.device)
    wts.scatter_(1, ids[:, :2], torch.softmax(vals[:, :2], dim=-1))

    def one(e):
        return (act(h @ w(p + e + "gate").T) * (h @ w(p + e + "up").T)) @ w(p + e + "down").T

    out = torch.sigmoid(h @ w(p + "shared.sg").T) * one("shared.")
    for e in range(8):
        out = out + wts[:, e:e + 1] * one("e%d." % e)
    return out


def _differential(c, w, h, first):
    mx, p = _mixer(c), "l0.mix."
    T, H, G, d, dv = h.shape[0], mx["heads"], mx["kv_heads"], mx["dim"], mx["vdim"]
    steps = (torch.arange(T, device=h.device) + 1).div(mx["q_temp"]["every"], rounding_mode="floor")
    temp = 1.0 + mx["q_temp"]["coef"] * torch.log(steps.double() + 1.0)
    q = (h @ w(p + "q").T).view(T, H, 2, d) * temp[:, None, None, None]
    k, v = (h @ w(p + "k").T).view(T, G, 2, d), (h @ w(p + "v").T).view(T, G, dv)
    lam = (torch.exp((w(p + "lq1") * w(p + "lk1")).sum())
           - torch.exp((w(p + "lq2") * w(p + "lk2")).sum()) + mx["diff"])
    one, two = (_attend(q[:, :, i], k[:, :, i], v, mx["scale"], first) for i in (0, 1))
    o = _rms(one - lam * two, 1.0, 1e-5) * (1.0 - mx["diff"])
    o = o.reshape(T - first, H * dv) * torch.sigmoid(h[first:] @ w(p + "g").T)
    return o @ w(p + "o").T
