"""What the engine is measured on: passes through its public entry points as a serving program
makes them, each with its inputs, the work it cannot do without, and its result in 64 bits.

Five kinds of pass, over the layer sizes the benchmark names (GPT-2 small, medium and XL, and the
Zuretar design of GPT-2 small's sizes):

  decode    `steps` steps of one token for each of `batch` requests that hold `context` tokens
            (from `context` down to `spread` times that, so that lengths are ragged), ids given
            by the caller; every step's logits are kept.  After a pass the requests are rewound.
  prompt    one step with `prompts` prompts of up to `length` tokens; the logits of each one's last
            `want` tokens.
  mixed     one step of a busy server: a token for each of `batch` requests, and a portion of
            `length` tokens of one more prompt.
  generate  whole requests through the native engine's scheduler: greedy, ids and
            log-probabilities out.
  serve     a model with recurrent state, from fresh requests: the prompts in one step, `steps`
            steps of single tokens behind it, every step's logits (a state cannot be rewound).

The weights are random, made on the GPU from a fixed seed (a model's are the same for every case),
the ids and lengths from the case's own.  A program loads its model once and serves many requests, so
the last model loaded is kept between calls of prepare().
"""
import itertools
import json
import math
import os
import tempfile
import weakref
import zlib

import numpy as np
import torch

from sglang_c_b200.config import resolve_architecture
from sglang_c_b200.engine import Engine, StepEntry, sched_new
from sglang_c_b200.sampling import SamplingParams
from sglang_c_b200.weights.loader import required_tensors
from sglang_c_b200.weights.safetensors_io import write_safetensors

PAGE = 16
STEP_TOKENS = 2048
VOCAB = 50257
POSITIONS = 1024


def _gpt2(n_layer, n_embd, n_head):
    return dict(architectures=["GPT2LMHeadModel"], model_type="gpt2", n_layer=n_layer, n_embd=n_embd, n_head=n_head,
                n_inner=4 * n_embd, vocab_size=VOCAB, n_positions=POSITIONS, layer_norm_epsilon=1e-5,
                activation_function="gelu_new")


def _zuretar(width, n_layer, heads):
    """Layers in fours: delta rule with a dense feed-forward, delta rule with experts, attention in
    chunks beside a linear attention with experts, the first one's weights again.  (Every expert is
    chosen, in its own weight: where a few are, random weights leave near ties, and a token whose
    choice turns on the last bit of a score has another result altogether.)"""
    dense = {"kind": "dense", "ff": width * 8 // 3}
    moe = {"kind": "moe", "expert": {"ff": width * 4 // 3},
           "router": {"experts": 8, "top": 8}}
    delta = {"heads": heads, "kv_heads": heads // 2, "dim": 64, "vdim": 64, "conv": 4}
    few = heads // 4
    side = {"left": {"heads": heads, "kv_heads": few, "dim": 64, "vdim": 64, "scale": 0.125, "mask": {"size": 256},
                     "rot": {"base": 10000.0, "dims": 64,
                             "scaling": {"factor": 8.0, "original": 256, "fast": 16.0, "slow": 2.0}}},
            "right": {"heads": few, "dim": 64, "vdim": 64, "decay": [1.0 - 2.0 ** -(3 + i % 6) for i in range(few)]}}
    kinds = [{"type": "delta", "mixer": delta, "mlp": dense}, {"type": "delta", "mixer": delta, "mlp": moe},
             {"type": "parallel", "mixer": side, "mlp": moe}, {"type": "delta", "mixer": delta, "mlp": dense}]
    layers = [dict(kinds[i % 4], weights_of=i - 3) if i % 4 == 3 else kinds[i % 4] for i in range(n_layer)]
    return {"architecture": "Zuretar", "vocab": VOCAB, "width": width, "norm": {"eps": 1e-5}, "layers": layers,
            "max_positions": POSITIONS}


MODELS = {"small": _gpt2(12, 768, 12), "medium": _gpt2(24, 1024, 16), "xl": _gpt2(48, 1600, 25),
          "zuretar": _zuretar(768, 12, 12)}
#: Tokens a state's requests may hold together; the engine's pool has room for four states.
HELD = {"small": 65536, "medium": 24576, "xl": 8192, "zuretar": 16384}


def listed():
    return [
        # one user's chat: the smallest step, where every launch and every wait counts
        dict(name="chat", kind="decode", model="small", dtype="bfloat16", batch=1, context=512, spread=1.0, steps=8),
        # the headline workload: eight requests at a context of 512
        dict(name="decode_8", kind="decode", model="small", dtype="bfloat16", batch=8, context=512, spread=1.0, steps=8),
        # a full server: 64 requests, short and long ones side by side
        dict(name="decode_64_ragged", kind="decode", model="small", dtype="bfloat16", batch=64, context=960, spread=0.07,
             steps=8),
        # the next size of model, an odd number of requests of unequal lengths
        dict(name="decode_medium_13", kind="decode", model="medium", dtype="bfloat16", batch=13, context=700, spread=0.5,
             steps=8),
        # a chat message: time to the first token of a short prompt
        dict(name="prompt_short", kind="prompt", model="small", dtype="bfloat16", prompts=1, length=45, spread=1.0, want=1),
        # a full step of prompts: the benchmark's prefill
        dict(name="prompt_2x1024", kind="prompt", model="small", dtype="bfloat16", prompts=2, length=1024, spread=1.0,
             want=1),
        # the same on the largest model
        dict(name="prompt_xl_2x1024", kind="prompt", model="xl", dtype="bfloat16", prompts=2, length=1024, spread=1.0,
             want=1),
        # continuous batching: running requests beside a portion of a new prompt
        dict(name="mixed_31_and_481", kind="mixed", model="small", dtype="bfloat16", batch=31, context=640, spread=0.3,
             length=481),
        # the precise mode, prompts to last token through the native engine: requests of unequal lengths
        dict(name="generate_fp32", kind="generate", model="small", dtype="float32", prompts=8, length=120, spread=0.4,
             steps=24),
        # the precise mode on long documents: three prompts, scored at their ends
        dict(name="prompt_fp32", kind="prompt", model="small", dtype="float32", prompts=3, length=780, spread=0.6, want=4),
        # a hybrid model reading two long documents, and scoring their last words
        dict(name="hybrid_2x1024", kind="serve", model="zuretar", dtype="bfloat16", prompts=2, length=1024, spread=1.0,
             want=16, steps=0),
        # the same model serving eight requests from their prompts on
        dict(name="hybrid_serve_8", kind="serve", model="zuretar", dtype="bfloat16", prompts=8, length=100, spread=0.5,
             want=1, steps=16),
    ]


def _size(rng, lo, hi):
    """A whole number between lo and hi, spread over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "prompt", "prompt", "mixed", "generate", "prompt32", "serve"])
    spread = round(rng.uniform(0.05, 1.0), 2)
    if kind == "decode":
        model = rng.choice(["small", "small", "medium"])
        batch = _size(rng, 1, 64 if model == "small" else 24)
        return dict(kind=kind, model=model, dtype="bfloat16", batch=batch, context=_size(rng, 16, 1000), spread=spread,
                    steps=rng.randint(6, 10))
    if kind == "prompt":
        model = rng.choice(["small", "small", "medium", "xl"])
        prompts = _size(rng, 1, 8)
        return dict(kind=kind, model=model, dtype="bfloat16", prompts=prompts,
                    length=_size(rng, 8, min(1024, 2048 // prompts)), spread=spread, want=1)
    if kind == "mixed":
        return dict(kind=kind, model=rng.choice(["small", "medium"]), dtype="bfloat16", batch=_size(rng, 2, 24),
                    context=_size(rng, 32, 1000), spread=spread, length=_size(rng, 16, 1000))
    if kind == "generate":
        return dict(kind=kind, model="small", dtype="float32", prompts=_size(rng, 1, 16), length=_size(rng, 8, 128),
                    spread=spread, steps=rng.randint(10, 20))
    if kind == "prompt32":
        prompts = _size(rng, 1, 4)
        return dict(kind="prompt", model="small", dtype="float32", prompts=prompts,
                    length=_size(rng, 8, min(1024, 2048 // prompts)), spread=spread, want=rng.randint(1, 4))
    prompts = _size(rng, 1, 12)
    return dict(kind="serve", model="zuretar", dtype="bfloat16", prompts=prompts,
                length=_size(rng, 24, min(1000, 2000 // prompts)), spread=spread, want=rng.randint(8, 16),
                steps=rng.randint(0, 12))


# -- a model's weights ---------------------------------------------------------------------------
def _plan(name):
    d = MODELS[name]
    arch = resolve_architecture(d)
    cfg = arch.config_class.from_dict(d)
    return cfg, arch.build_plan(cfg)


def _weight(model, name, decl, dtype):
    """One tensor, made on the GPU: matrices in the model's precision, vectors in 32 bits."""
    g = torch.Generator(device="cuda")
    g.manual_seed(zlib.crc32(("%s %s" % (model, name)).encode()))
    x = torch.randn(tuple(decl.shape), generator=g, device="cuda", dtype=torch.float32)
    scale = 0.4 if decl.init == "conv_taps" else 0.1 if decl.init == "norm_gain" else 0.02
    if name.endswith("c_attn.weight"):
        scale = 0.04            # scores that tell keys apart, as a trained model's do
    x *= scale
    if decl.init == "norm_gain":
        x += 1.0
    if name.endswith("dt_bias"):
        x = x * 50.0 - 3.0      # states that remember a few to some hundred tokens
    return x.to(torch.bfloat16) if dtype == "bfloat16" and len(decl.shape) >= 2 else x


def _weights(model, dtype):
    _, plan = _plan(model)
    return {n: _weight(model, n, d, dtype) for n, d in required_tensors(plan).items()}


_kept = {}                       # the one model that is loaded: {(model, dtype, native): engine}
_number = itertools.count()


def _load(model, dtype, native):
    key = (model, dtype, native)
    if key not in _kept:
        for old in _kept.values():
            if hasattr(old, "close"):
                old.close()
        _kept.clear()
        torch.cuda.empty_cache()
        cfg, _ = _plan(model)
        with tempfile.TemporaryDirectory() as d:
            with open(os.path.join(d, "config.json"), "w") as f:
                json.dump(cfg.to_dict(), f)
            write_safetensors(os.path.join(d, "model.safetensors"), {n: t.cpu() for n, t in _weights(model, dtype).items()})
            size = dict(page_size=PAGE, max_step_tokens=STEP_TOKENS, dtype=dtype)
            if native:
                _kept[key] = sched_new(d, native=True, max_tokens=16384, max_requests=16, prefill_chunk=512,
                                       want_logprobs=True, **size)
            else:
                _kept[key] = Engine.from_dir(d, max_tokens=4 * HELD[model], max_requests=256, **size)
    return _kept[key]


# -- inputs ----------------------------------------------------------------------------------------
def _inputs(case, seed):
    """The case's requests as whole numbers: for each, the ids it holds or brings at once, and the ids
    that follow one by one."""
    r = np.random.default_rng(int(seed) * 7919 + zlib.crc32(json.dumps(
        {k: v for k, v in sorted(case.items()) if k != "name"}).encode()))
    kind = case["kind"]
    n = case["batch"] if kind in ("decode", "mixed") else case["prompts"]
    longest = case["context"] if kind in ("decode", "mixed") else case["length"]
    lens = np.rint(longest * np.linspace(1.0, case["spread"], n)).astype(int).clip(1, None)
    if kind in ("decode", "mixed"):
        lens = lens.clip(1, POSITIONS - case.get("steps", 1))
        if n * longest > HELD[case["model"]]:
            lens = lens.clip(1, HELD[case["model"]] // n)
    r.shuffle(lens)
    held = [r.integers(0, VOCAB, size=int(k)).astype(np.int32) for k in lens]
    after = r.integers(0, VOCAB, size=(n, case.get("steps", 1))).astype(np.int32)
    more = r.integers(0, VOCAB, size=case["length"]).astype(np.int32) if kind == "mixed" else None
    return held, after, more


class _State:
    pass


def _end(engine, ids):
    for q in ids:
        if engine.has_request(q):
            engine.end_request(q)


def prepare(case, seed):
    s = _State()
    s.case = case
    held, after, more = _inputs(case, seed)
    s.engine = eng = _load(case["model"], case["dtype"], case["kind"] == "generate")
    if case["kind"] == "generate":
        s.prompts = [p.tolist() for p in held]
        return s
    me = next(_number)
    s.ids = ["%d.%d" % (me, i) for i in range(len(held) + (1 if more is not None else 0))]
    s.after, s.lens, s.held = after.tolist(), [len(p) for p in held], held
    if case["kind"] in ("decode", "mixed"):
        for q in s.ids:
            eng.add_request(q)
        weakref.finalize(s, _end, eng, s.ids)
        todo = [(q, p, 0) for q, p in zip(s.ids, held)]
        while todo:                                          # the contexts, in steps of as many tokens as fit
            room, entries, rest = STEP_TOKENS, [], []
            for q, p, at in todo:
                n = min(len(p) - at, room)
                if n > 0:
                    entries.append(StepEntry(q, p[at:at + n], []))
                    room -= n
                if at + n < len(p):
                    rest.append((q, p, at + n))
            eng.step(entries)
            todo = rest
    s.more = more
    rows = {"decode": len(held) * case.get("steps", 0), "serve": len(held) * case.get("steps", 0)}.get(case["kind"], 0)
    s.out = torch.empty((max(rows, 1), VOCAB), device="cuda") if rows else None
    return s


# -- one pass ------------------------------------------------------------------------------------
def _singles(s, eng, ids):
    """The steps of single tokens, every step's logits kept."""
    n = len(ids)
    for k in range(s.case["steps"]):
        logits = eng.step([StepEntry(q, [s.after[i][k]], [0]) for i, q in enumerate(ids)])
        s.out[k * n:(k + 1) * n].copy_(logits)
    return s.out


def run(s):
    case, eng = s.case, s.engine
    kind = case["kind"]
    if kind == "generate":
        sp = SamplingParams(temperature=0.0, ignore_eos=True)
        ids = [eng.submit_ids(p, case["steps"], sp) for p in s.prompts]
        eng.run_until_done()
        done = {}
        while (got := eng.poll()) is not None:
            done[got[0]] = (got[1], eng.last_logprobs)
        return {"ids": np.array([done[i][0] for i in ids], dtype=np.int64),
                "logprobs": np.array([done[i][1] for i in ids], dtype=np.float32)}
    if kind == "decode":
        for q, n in zip(s.ids, s.lens):
            eng.truncate(q, n)
        return _singles(s, eng, s.ids)
    if kind == "mixed":
        for q, n in zip(s.ids, s.lens + [0]):
            eng.truncate(q, n)
        entries = [StepEntry(q, [t[0]], [0]) for q, t in zip(s.ids, s.after)]
        entries.append(StepEntry(s.ids[-1], s.more, [len(s.more) - 1]))
        return eng.step(entries)
    # fresh requests, as a server meets them
    for q in s.ids:
        eng.add_request(q)
    entries = [StepEntry(q, p, list(range(max(0, len(p) - case["want"]), len(p)))) for q, p in zip(s.ids, s.held)]
    logits = eng.step(entries)
    if case.get("steps"):
        logits = {"prompts": logits.clone(), "steps": _singles(s, eng, s.ids)}
    for q in s.ids:
        eng.end_request(q)
    return logits


# -- what a pass cannot do without -----------------------------------------------------------------
def _counts(model):
    """(numbers of the matrices a token passes through, of the head, of all matrices, of cached numbers a
    position, of state numbers a request)."""
    d = MODELS[model]
    if model != "zuretar":
        E, L = d["n_embd"], d["n_layer"]
        body = 12 * E * E * L
        return body, VOCAB * E, body + VOCAB * E, 2 * E * L, 0
    E, used, held, cached, state, seen = d["width"], 0, 0, 0, 0, set()
    for i, l in enumerate(d["layers"]):
        m, f = l["mixer"], l["mlp"]
        if l["type"] == "delta":
            a = E * (2 * m["kv_heads"] * m["dim"] + 3 * m["heads"] * m["vdim"] + 2 * m["heads"])
            state += m["heads"] * m["dim"] * m["vdim"]
        else:
            le, ri = m["left"], m["right"]
            a = E * (2 * le["heads"] * le["dim"] + 2 * le["kv_heads"] * le["dim"]) + 5 * E * ri["heads"] * ri["dim"]
            cached += 2 * le["kv_heads"] * le["dim"]
            state += ri["heads"] * ri["dim"] * ri["vdim"]
        ff = f["ff"] if f["kind"] == "dense" else f["expert"]["ff"]
        each = 3 * E * ff
        used += a + each * (1 if f["kind"] == "dense" else f["router"]["top"])
        if l.get("weights_of") is None:
            held += a + each * (1 if f["kind"] == "dense" else f["router"]["experts"])
    return used, VOCAB * E, held + VOCAB * E, cached, state


def work(case):
    held, after, more = _inputs(case, 0)
    used, head, matrices, cached, state = _counts(case["model"])
    lens = [len(p) for p in held]
    e = 2 if case["dtype"] == "bfloat16" else 4
    n, kind, steps = len(lens), case["kind"], case.get("steps", 1)
    nbytes = flops = 0.0
    attend = 2.0 * cached                                    # a query and a position: scores and sums

    def prompt(q, wanted):
        """Whole prompts from position 0: all matrices read, keys and values written, logits out."""
        t = float(sum(q))
        pairs = sum(k * (k + 1) / 2.0 for k in q)
        return (matrices * e + t * cached * e + 2 * 4.0 * state * len(q) + 4.0 * wanted * VOCAB,
                2.0 * used * t + 2.0 * head * wanted + attend * pairs)

    def single(at):
        """One token for requests that hold `at` tokens each."""
        return (matrices * e + sum(at) * cached * e + 2 * 4.0 * state * len(at) + 4.0 * len(at) * VOCAB,
                2.0 * (used + head) * len(at) + attend * sum(at))

    if kind in ("prompt", "serve", "generate"):
        b, f = prompt(lens, sum(min(k, case.get("want", 1)) for k in lens))
        nbytes, flops = nbytes + b, flops + f
        lens = [k + 1 for k in lens]
        steps = steps - 1 if kind == "generate" else case.get("steps", 0)
    if kind in ("decode", "serve", "generate"):
        for k in range(steps):
            b, f = single([x + k for x in lens])
            nbytes, flops = nbytes + b, flops + f
    if kind == "mixed":
        b, f = single(lens)
        c, g = prompt([len(more)], 1)
        nbytes, flops = b + c - matrices * e, f + g
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what two ways of rounding differ by: the results lie 1.3e-6 (32-bit), 0.003 to 0.007
    (bfloat16) and 0.015 (the hybrid, whose norms of every part's result bring small parts' rounding up)
    from the 64-bit ones."""
    if case["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4, "differ": 0.005}
    return {"rel": 0.03, "max": 0.4} if case["model"] == "zuretar" else {"rel": 0.02, "max": 0.15}


# -- the same in 64 bits ---------------------------------------------------------------------------
def _norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w + b


def _gpt2_stream(d, w, ids, rows):
    """The final norm's rows of one sequence in 64 bits, at the last `rows` places."""
    E, H, n = d["n_embd"], d["n_head"], len(ids)
    x = w["wte.weight"][ids] + w["wpe.weight"][:n]
    above = torch.ones((n, n), dtype=torch.bool, device="cuda").triu(1)
    for i in range(d["n_layer"]):
        p = "h.%d." % i
        h = _norm(x, w[p + "ln_1.weight"], w[p + "ln_1.bias"], d["layer_norm_epsilon"])
        qkv = h @ w[p + "attn.c_attn.weight"] + w[p + "attn.c_attn.bias"]
        q, k, v = (t.reshape(n, H, E // H).transpose(0, 1) for t in qkv.split(E, -1))
        a = (q @ k.transpose(1, 2) / math.sqrt(E // H)).masked_fill(above, -math.inf).softmax(-1)
        x = x + (a @ v).transpose(0, 1).reshape(n, E) @ w[p + "attn.c_proj.weight"] + w[p + "attn.c_proj.bias"]
        h = _norm(x, w[p + "ln_2.weight"], w[p + "ln_2.bias"], d["layer_norm_epsilon"])
        u = h @ w[p + "mlp.c_fc.weight"] + w[p + "mlp.c_fc.bias"]
        u = 0.5 * u * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (u + 0.044715 * u ** 3)))
        x = x + u @ w[p + "mlp.c_proj.weight"] + w[p + "mlp.c_proj.bias"]
    return _norm(x[n - rows:], w["ln_f.weight"], w["ln_f.bias"], d["layer_norm_epsilon"]) @ w["wte.weight"].T


def _rms(x, w, eps):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)
    return y if w is None else y * w


def _turn(x, rot):
    """Rotary positions with YaRN's blend of frequencies: [n, heads, dim], entry i with i + dims/2."""
    half, sc = rot["dims"] // 2, rot["scaling"]
    i = torch.arange(half, dtype=torch.float64, device="cuda")
    f = rot["base"] ** (-2.0 * i / rot["dims"])

    def at(turns):
        return rot["dims"] * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))

    lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), rot["dims"] - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    a = torch.arange(len(x), dtype=torch.float64, device="cuda")[:, None] * (f / sc["factor"] * ramp + f * (1 - ramp))
    m = 0.1 * math.log(sc["factor"]) + 1.0
    c, s = (a.cos() * m)[:, None], (a.sin() * m)[:, None]
    u, v = x[..., :half], x[..., half:2 * half]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., 2 * half:]], -1)


def _conv(x, taps):
    K = taps.shape[1]
    pad = torch.cat([x.new_zeros(K - 1, x.shape[1]), x])
    return sum(pad[j:j + len(x)] * taps[:, j] for j in range(K))


def _recur(q, k, v, decay, beta):
    """S <- decay S + k u^T with u = v, or beta (v - S^T k) for the delta rule; o = S^T q.  [n, H, D]."""
    n, H, D = q.shape
    S, out = q.new_zeros(H, v.shape[-1], D), torch.empty_like(v)
    for t in range(n):
        S = S * decay[t][:, None, None]
        u = v[t] if beta is None else beta[t][:, None] * (v[t] - torch.bmm(S, k[t][..., None])[..., 0])
        S = torch.baddbmm(S, u[..., None], k[t][:, None])
        out[t] = torch.bmm(S, q[t][..., None])[..., 0]
    return out


def _delta(h, w, p, m, eps):
    n, H, G, D, V, silu = len(h), m["heads"], m["kv_heads"], m["dim"], m["vdim"], torch.nn.functional.silu
    q, k, v = (silu(_conv(h @ w[p + c].T, w[p + c + ".conv"])) for c in "qkv")
    q, k, v = q.reshape(n, G, D), k.reshape(n, G, D), v.reshape(n, H, V)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) / math.sqrt(D)
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    decay = torch.exp(-torch.exp(w[p + "A_log"]) * torch.nn.functional.softplus(h @ w[p + "a"].T + w[p + "dt_bias"]))
    o = _recur(q.repeat_interleave(H // G, 1), k.repeat_interleave(H // G, 1), v, decay, torch.sigmoid(h @ w[p + "b"].T))
    return (_rms(o, w[p + "norm"], eps) * silu(h @ w[p + "g"].T).reshape(n, H, V)).reshape(n, H * V) @ w[p + "o"].T


def _side(h, w, p, m, eps):
    le, ri, n, silu = m["left"], m["right"], len(h), torch.nn.functional.silu
    H, G, D = le["heads"], le["kv_heads"], le["dim"]
    q, k, v = ((h @ w[p + "left." + c].T).reshape(n, -1, D) for c in "qkv")
    q, k = _rms(_turn(q, le["rot"]), None, eps), _rms(_turn(k, le["rot"]), None, eps)
    k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
    at = torch.arange(n, device="cuda")
    off = (at[None, :] > at[:, None]) | (at[None, :] // le["mask"]["size"] != at[:, None] // le["mask"]["size"])
    a = (torch.einsum("nhd,mhd->hnm", q, k) * le["scale"]).masked_fill(off, -math.inf)
    a = torch.cat([a, w[p + "left.sink"][:, None, None].expand(H, n, 1)], -1).softmax(-1)[..., :-1]
    left = torch.einsum("hnm,mhd->nhd", a, v).reshape(n, H * D) @ w[p + "left.o"].T
    q, k, v = (silu(h @ w[p + "right." + c].T).reshape(n, ri["heads"], -1) for c in "qkv")
    decay = torch.tensor(ri["decay"], dtype=torch.float64, device="cuda").expand(n, -1)
    o = _rms(_recur(q, k, v, decay, None).reshape(n, -1), w[p + "right.norm"], eps)
    right = (o * torch.sigmoid(h @ w[p + "right.g"].T)) @ w[p + "right.o"].T
    return 0.5 * (_rms(left, w[p + "left.out"], eps) + _rms(right, w[p + "right.out"], eps))


def _experts(h, w, p, mlp):
    r, silu = mlp["router"], torch.nn.functional.silu
    s = torch.sigmoid(h @ w[p + "router"].T)
    part = torch.zeros_like(s).scatter_(1, (s + w[p + "correction"]).topk(r["top"], -1).indices, 1.0) * s
    return sum(part[:, e:e + 1] * ((silu(h @ w["%se%d.gate" % (p, e)].T) * (h @ w["%se%d.up" % (p, e)].T))
                                   @ w["%se%d.down" % (p, e)].T) for e in range(r["experts"]))


def _zuretar_stream(d, w, ids, rows):
    x, eps, silu = w["embed"][ids], d["norm"]["eps"], torch.nn.functional.silu
    for i, l in enumerate(d["layers"]):
        p = "l%d." % l.get("weights_of", i)
        h = _rms(x, w[p + "norm1"], eps)
        y = (_delta if l["type"] == "delta" else _side)(h, w, p + "mix.", l["mixer"], eps)
        m = p + "mlp."
        if l["mlp"]["kind"] == "moe":
            y = y + _experts(h, w, m, l["mlp"])
        else:
            y = y + (silu(h @ w[m + "gate"].T + w[m + "gate.b"]) * (h @ w[m + "up"].T + w[m + "up.b"])) @ w[m + "down"].T \
                + w[m + "down.b"]
        x = x + y
    return _rms(x[len(x) - rows:], w["final.norm"], eps) @ w["head"].T


def exact(case, seed):
    held, after, more = _inputs(case, seed)
    d, kind = MODELS[case["model"]], case["kind"]
    w = {n: t.double() for n, t in _weights(case["model"], case["dtype"]).items()}

    def last(ids, rows):
        ids = torch.from_numpy(np.asarray(ids, dtype=np.int64)).cuda()
        return (_zuretar_stream if case["model"] == "zuretar" else _gpt2_stream)(d, w, ids, rows)

    if kind == "generate":
        found, probs = [], []
        for p in held:
            ids, lp = p.tolist(), []
            for _ in range(case["steps"]):
                row = last(ids, 1)[0].log_softmax(-1)
                ids.append(int(row.argmax()))
                lp.append(float(row[ids[-1]]))
            found.append(ids[len(p):])
            probs.append(lp)
        return {"ids": np.array(found, dtype=np.int64), "logprobs": np.array(probs)}
    if kind == "prompt":
        return torch.cat([last(p, min(len(p), case["want"])) for p in held])
    if kind == "mixed":
        return torch.cat([last(np.append(p, t), 1) for p, t in zip(held, after)] + [last(more, 1)])
    steps = case["steps"]
    rows = [last(np.append(p, t), steps + (min(len(p), case["want"]) if kind == "serve" else 0)) for p, t in zip(held, after)]
    singles = torch.stack([r[len(r) - steps:] for r in rows], 1).reshape(-1, VOCAB) if steps else None
    if kind == "decode":
        return singles
    prompts = torch.cat([r[:len(r) - steps] for r in rows])
    return {"prompts": prompts, "steps": singles} if steps else prompts
