"""What a user of this framework has it do, as cases that can be timed and compared.

A case is one pass through the engine's step function, `ModelRunner.step` (or, for the tiny model, a whole generation
with it and the sampler): `decoding` requests bring one token each on a context they already hold, `prompts` new
requests bring their first tokens, and the pass returns the float32 logits that those steps hand out.  Sizes are this
repository's own: the Qwen3-8B layer sizes and a tiny Qwen3 configuration, and the benchmark's "2k" sizes of two of the
other decoders, which between them have what the others are made of (latent attention, capped attention, recurrent
mixers, routed experts with and without a shared one).  Eight layers, as the benchmark runs the other decoders: bfloat16
rounding through more layers of random weights would hide what the comparison is to show.  Weights are the framework's
seeded random ones, prompts seeded uniform token ids; caches and states hold what real prompts leave.
"""
import math

import torch

from vllm_lite_b200.config import plan_from_config_json
from vllm_lite_b200.engine import ModelRunner, StepEntry, random_model
from vllm_lite_b200.parts.model import declare_model
from vllm_lite_b200.sampling import SamplingParams
from vllm_lite_b200.sampling.sampler import Sampler

DEVICE = "cuda:0"
PAGE = 64
STEP_TOKENS = 4096                 # the scheduler's default limit on a step
F = torch.float64


# ---------------------------------------------------------------------------------------------- models
def _qwen3(layers, hidden, heads, kv_heads, head_dim, ff, vocab, theta, eps):
    return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", hidden_size=hidden, num_hidden_layers=layers,
                num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=ff,
                vocab_size=vocab, rope_theta=theta, rms_norm_eps=eps, tie_word_embeddings=False, max_position_embeddings=40960)


def _layers(kinds, n):
    return [dict(type=kinds[i % 4][0], mixer=kinds[i % 4][1], mlp=kinds[i % 4][2]) for i in range(n)]


def _puturax(layers):
    lat = dict(heads=16, dim=128, rot_dim=64, vdim=128, q_rank=768, kv_rank=64, scale=192 ** -0.5, rot=dict(dims=64, base=500000.0))
    par = dict(left=dict(heads=16, kv_heads=4, dim=128, vdim=128, scale=0.2, softcap=30.0, q_temp=dict(coef=0.1, every=1024)),
               right=dict(heads=32, dim=64, decay_rank=64), left_scale=0.7, right_scale=0.6)
    moe = dict(kind="moe", expert=dict(ff=1024), router=dict(experts=32, top=4, groups=dict(count=4, keep=2)), shared=dict(ff=1024))
    kinds = [("latent_attention", lat, dict(kind="dense", ff=8192)), ("parallel", par, moe), ("parallel", par, moe), ("parallel", par, moe)]
    return dict(architecture="Puturax", vocab=65536, width=2048, norm=dict(eps=1e-6), embedding=dict(scale=2048 ** 0.5),
                max_position_embeddings=16384, layers=_layers(kinds, layers))


def _vekusun(layers):
    delta = dict(heads=16, kv_heads=8, dim=128, vdim=128, conv=4)
    one = dict(heads=16, dim=128, vdim=128, q_rank=768, kv_rank=256, scale=128 ** -0.5)
    two = dict(heads=16, dim=128, rot_dim=64, vdim=128, kv_rank=192, scale=192 ** -0.5,
               rot=dict(dims=64, base=500000.0, scaling=dict(factor=4.0, original=4096, fast=32.0, slow=1.0)))
    dense = dict(kind="dense", ff=8192)
    moe = dict(kind="moe", expert=dict(ff=1024), router=dict(experts=32, top=4))
    kinds = [("delta", delta, dense), ("latent_attention", one, moe), ("latent_attention_2", two, dense), ("delta", delta, moe)]
    return dict(architecture="Vekusun", vocab=65536, width=2048, norm=dict(eps=1e-6), logit_softcap=30.0, residual_mult=0.5,
                loop=dict(start=1, stop=3, times=2), max_position_embeddings=16384, layers=_layers(kinds, layers))


def _config(case):
    n = case["layers"]
    if case["model"] == "qwen3-8b":
        return _qwen3(n, 4096, 32, 8, 128, 12288, 151936, 1e6, 1e-6)
    if case["model"] == "qwen3-tiny":
        return _qwen3(n, 96, 8, 2, 32, 160, 333, 1e6, 1e-5)
    return {"puturax-2k": _puturax, "vekusun-2k": _vekusun}[case["model"]](n)


def _model(case, seed):
    dtype = getattr(torch, case["dtype"])
    config = _config(case)
    std = 0.05 if case["model"] == "qwen3-tiny" else None
    _, plan, weights = random_model(config, seed=seed, dtype=dtype, device=DEVICE, std=std,
                                    store_dtype=torch.float32 if dtype == torch.float32 else torch.bfloat16)
    for name in weights:
        if name.endswith(".correction"):                 # smaller than the scores: the tokens spread over the experts
            weights[name] = weights[name] * 0.01
        elif case["model"] == "puturax-2k" and (name == "final.norm" or name.split(".")[-1] in ("norm1", "norm1b", "norm2", "norm2b")):
            weights[name] = weights[name] - 1            # this decoder stores a norm's weight around zero
    return config, plan, weights


# ---------------------------------------------------------------------------------------------- the cases
def _case(name, model, layers, decoding=0, context=(0, 0), limit=4096, prompts=0, prompt=(0, 0), generate=0, dtype="bfloat16"):
    return dict(name=name, model=model, layers=layers, dtype=dtype, decoding=decoding, context_low=context[0],
                context_high=context[1], limit=limit, prompts=prompts, prompt_low=prompt[0], prompt_high=prompt[1], generate=generate)


def listed():
    return [
        # a test or a first trial: a tiny float32 model, a few short prompts, sixteen tokens each
        _case("tiny-generate-f32", "qwen3-tiny", 3, prompts=5, prompt=(1, 100), generate=16, limit=512, dtype="float32"),
        # one user's chat: a token at a time on a long context; latency is all
        _case("qwen3-decode-1", "qwen3-8b", 8, decoding=1, context=(2600, 3000)),
        # the benchmark's headline: eight requests decoding
        _case("qwen3-decode-8", "qwen3-8b", 8, decoding=8, context=(2200, 3300)),
        # a loaded server: many requests of middling length
        _case("qwen3-decode-64", "qwen3-8b", 8, decoding=64, context=(400, 1500), limit=2048),
        # time to the first token of a long prompt
        _case("qwen3-prompt-2048", "qwen3-8b", 8, prompts=1, prompt=(2048, 2048)),
        # a short question, an odd number of tokens
        _case("qwen3-prompt-short", "qwen3-8b", 8, prompts=1, prompt=(173, 173)),
        # continuous batching: decoding requests beside a portion of a new prompt (the scheduler's default 512)
        _case("qwen3-mixed", "qwen3-8b", 8, decoding=24, context=(300, 1500), limit=2048, prompts=1, prompt=(512, 512)),
        # latent attention, capped attention beside a time mixing, grouped experts with a shared one
        _case("puturax-prompt-2048", "puturax-2k", 8, prompts=1, prompt=(2048, 2048)),
        _case("puturax-decode-32", "puturax-2k", 8, decoding=32, context=(200, 1000), limit=2048),
        # latent attentions, delta rule with one decay a head, layers that run twice: prompts of ragged length, few and many decoding
        _case("vekusun-prompts", "vekusun-2k", 8, prompts=3, prompt=(500, 1500)),
        _case("vekusun-decode-8", "vekusun-2k", 8, decoding=8, context=(600, 2500)),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    model = rng.choice(["qwen3-tiny", "qwen3-8b", "qwen3-8b", "puturax-2k", "vekusun-2k"])
    if model == "qwen3-tiny":
        low = log_int(1, 100)
        return _without_name(_case("", model, 3, prompts=rng.randint(1, 8), prompt=(low, rng.randint(low, 120)),
                                   generate=rng.randint(4, 20), limit=512, dtype="float32"))
    layers, kind = 8, rng.choice(["prompt", "decode", "mixed"])
    decoding, prompts = 0, 0
    context, prompt, limit = (0, 0), (0, 0), 4096
    if kind != "prompt":
        decoding = log_int(1, 64 if kind == "decode" else 32)
        most = min(3000, 40000 // decoding)              # so that a preparation stays short
        low = log_int(16, most)
        context = (low, rng.randint(low, most))
        limit = 4096 if context[1] > 1500 else 2048
    if kind != "decode":
        prompts = rng.randint(1, 4) if kind == "prompt" else 1
        most = 2048 // prompts if kind == "prompt" else 512
        low = log_int(20, most)
        prompt = (low, rng.randint(low, most))
    return _without_name(_case("", model, layers, decoding=decoding, context=context, limit=limit, prompts=prompts, prompt=prompt))


def _without_name(case):
    return {k: v for k, v in case.items() if k != "name"}


def _lengths(low, high, n):
    """`n` lengths over [low, high], ragged (steps of the golden ratio), the same for every seed."""
    return [low + int((high - low + 1) * (((i + 0.5) * 0.6180339887498949) % 1.0)) for i in range(n)]


def _tokens(case, seed):
    """(token ids of every decoding request: its context and what it is fed afterwards, token ids of every new prompt)."""
    vocab = _config(case).get("vocab_size") or _config(case)["vocab"]
    gen = torch.Generator().manual_seed(1000003 * seed + 17)
    ids = lambda n: torch.randint(0, vocab, (n,), generator=gen).tolist()
    decoding = [ids(case["limit"]) for _ in range(case["decoding"])]
    return decoding, [ids(n) for n in _lengths(case["prompt_low"], case["prompt_high"], case["prompts"])]


# ---------------------------------------------------------------------------------------------- a pass
class _Serving:
    """An engine that has been serving: weights bound, graphs recorded, contexts in the cache."""

    def __init__(self, case, seed):
        _, plan, weights = _model(case, seed)
        self.case = case
        self.ids, self.prompts = _tokens(case, seed)
        self.contexts = _lengths(case["context_low"], case["context_high"], case["decoding"])
        pages = case["decoding"] * -(-case["limit"] // PAGE) + sum(-(-(len(p) + case["generate"]) // PAGE) for p in self.prompts)
        self.runner = ModelRunner(plan, weights, dtype=getattr(torch, case["dtype"]), device=DEVICE, page_size=PAGE,
                                  num_pages=pages, max_requests=case["decoding"] + case["prompts"], max_context=case["limit"],
                                  own_weights=True)
        self.sampler = Sampler(DEVICE)
        self.fed = []
        self.fill()

    def fill(self):
        """The contexts run through the model, several requests to a step."""
        for i in range(len(self.fed)):
            self.runner.release(f"d{i}")
        self.fed = list(self.contexts)
        entries, room = [], STEP_TOKENS
        for i, n in enumerate(self.contexts):
            at = 0
            while at < n:
                take = min(room, n - at)
                entries.append(StepEntry(f"d{i}", self.ids[i][at:at + take], []))
                at, room = at + take, room - take
                if room == 0:
                    self.runner.step(entries)
                    entries, room = [], STEP_TOKENS
        if entries:
            self.runner.step(entries)

    def step(self):
        if self.fed and max(self.fed) >= self.case["limit"]:
            self.fill()
        entries = [StepEntry(f"d{i}", [self.ids[i][n]], [0]) for i, n in enumerate(self.fed)]
        entries += [StepEntry(f"p{i}", p, [len(p) - 1]) for i, p in enumerate(self.prompts)]
        logits = self.runner.step(entries)
        self.fed = [n + 1 for n in self.fed]
        for i in range(len(self.prompts)):
            self.runner.release(f"p{i}")
        return {"logits": logits}

    def generate(self):
        greedy = [SamplingParams()] * len(self.prompts)
        entries = [StepEntry(f"p{i}", p, [len(p) - 1]) for i, p in enumerate(self.prompts)]
        logits, tokens = [], []
        for _ in range(self.case["generate"]):
            out = self.runner.step(entries)
            logits.append(out.clone())                   # the next step writes the buffer again
            tokens.append(self.sampler.sample(out, greedy, [()] * len(greedy))[0].tolist())
            entries = [StepEntry(f"p{i}", [t], [0]) for i, t in enumerate(tokens[-1])]
        for i in range(len(self.prompts)):
            self.runner.release(f"p{i}")
        return {"logits": torch.stack(logits), "tokens": torch.tensor(tokens)}


def prepare(case, seed):
    state = _Serving(case, seed)
    run(state)                                           # an engine's first step records its graphs
    return state


def run(state):
    return state.generate() if state.case["generate"] else state.step()


# ---------------------------------------------------------------------------------------------- work and tolerance
def _mixer_costs(case, config):
    """Per layer run: (cached bytes a token, flops a (query, key) pair, window, state bytes a request, state flops a token)."""
    size = 4 if case["dtype"] == "float32" else 2
    if "architectures" in config:
        h, kv, d = config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"]
        return [(2 * kv * d * size, 4 * h * d, None, 0, 0)] * config["num_hidden_layers"]
    costs = []
    for layer in config["layers"]:
        m, t = layer["mixer"], layer["type"]
        if t == "parallel":
            a, r = m["left"], m["right"]
            d, p = (r["state"], r["vdim"]) if "state" in r else (r["dim"], r["dim"])
            costs.append((a["kv_heads"] * (a["dim"] + a["vdim"]) * size, 2 * a["heads"] * (a["dim"] + a["vdim"]),
                          a.get("mask", {}).get("size"), 4 * r["heads"] * d * p, 6 * r["heads"] * d * p))
        elif t.startswith("latent_attention"):
            row = m["kv_rank"] + m.get("rot_dim", 0)
            costs.append((row * size, 2 * m["heads"] * (row + m["kv_rank"]), None, 0, 0))
        else:
            state = m["heads"] * m["dim"] * m["vdim"]
            costs.append((0, 0, None, 4 * state, 8 * state))
    loop = config.get("loop")
    if loop:
        lo, hi = loop["start"], loop["stop"]
        costs = costs[:lo] + costs[lo:hi] * loop["times"] + costs[hi:]
    return costs


def work(case):
    config = _config(case)
    size = 4 if case["dtype"] == "float32" else 2
    _, plan = plan_from_config_json(config)
    moe = next((l["mlp"]["router"] for l in config.get("layers", []) if l["mlp"]["kind"] == "moe"), None)
    loop = config.get("loop") or dict(start=0, stop=0, times=1)
    body = head = experts = 0                            # matrix elements: met by every token (loop runs counted), by a wanted row
    read = 0                                             # of them, read once
    for name, decl in declare_model(plan).items():
        if len(decl.shape) < 2:
            continue
        n = math.prod(decl.shape)
        if name in ("embed", "model.embed_tokens.weight"):
            head += n if plan.tie_word_embeddings else 0
        elif name in ("head", "lm_head.weight"):
            head += n
        else:
            layer = int(name[1:name.index(".")]) if name.startswith("l") and name[1].isdigit() else -1
            times = loop["times"] if loop["start"] <= layer < loop["stop"] else 1
            if ".mlp.e" in name:
                experts += n
                body += times * n * moe["top"] / moe["experts"]
            else:
                body += times * n
                read += n

    def one_step(spans):                                 # [(first position, tokens)] of the step's requests
        tokens = sum(n for _, n in spans)
        reached = 1 - (1 - moe["top"] / moe["experts"]) ** tokens if moe else 0
        by = size * (read + experts * reached + head)
        fl = 2 * body * tokens + 2 * head * len(spans)
        for row, pair, window, state, step in _mixer_costs(case, config):
            for at, n in spans:
                met = [min(p + 1, window or p + 1) for p in (at, at + n - 1)]
                pairs = sum(met) / 2 * n if window is None or at + n <= window else sum(min(p + 1, window) for p in range(at, at + n))
                by += row * (met[1] + n if at else n) + (2 if at else 1) * state
                fl += pair * pairs + step * n
        return by, fl

    new = _lengths(case["prompt_low"], case["prompt_high"], case["prompts"])
    spans = [(c, 1) for c in _lengths(case["context_low"], case["context_high"], case["decoding"])] + [(0, n) for n in new]
    steps = [spans] + [[(n + k, 1) for n in new] for k in range(case["generate"] - 1)]
    done = [one_step(s) for s in steps]
    return {"bytes": float(sum(b for b, _ in done)), "flops": float(sum(f for _, f in done))}


def tolerance(case):
    # float32: sums in another order.  bfloat16: every activation is rounded to 8 bits many times over; where a router's two
    # candidates lie close, rounding decides which expert a token meets.
    # Against 64 bits: float32 6e-7, Qwen3 0.02 (eight layers, few keys to a row's softmax that stand out), the others 0.002 to 0.01.
    if case["dtype"] == "float32":
        return {"rel": 3e-6, "max": 1e-3}
    return {"rel": 0.01 if case["model"] == "puturax-2k" else 0.03, "max": 0.5}


# ---------------------------------------------------------------------------------------------- the same in 64 bits
# Plain functions on padded batches of sequences: x [B, T, W], every sequence from its first token; all operations are
# causal, so what stands behind a sequence's end is never seen by it.
def _lin(w, x, b=None):
    y = x @ w.to(F).t()
    return y if b is None else y + b.to(F)


def _unit_rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _sub(w, prefix):
    return {k[len(prefix):]: t for k, t in w.items() if k.startswith(prefix)}


def _conv(x, taps, bias=None):
    n = taps.shape[1]
    pad = torch.cat([x.new_zeros(x.shape[0], n - 1, x.shape[2]), x], 1)
    y = sum(pad[:, j:j + x.shape[1]] * taps[:, j].to(F) for j in range(n))
    return y if bias is None else y + bias.to(F)


def _turn(x, freqs, halves, amplitude=1.0):
    """x [B, T, heads, n]: pairs (i, i + half) or (2i, 2i + 1) of the first 2 * len(freqs) features turned by position * frequency."""
    half = len(freqs)
    angle = torch.arange(x.shape[1], device=x.device, dtype=F)[:, None] * torch.tensor(freqs, device=x.device, dtype=F)
    c, s = (amplitude * torch.cos(angle))[None, :, None], (amplitude * torch.sin(angle))[None, :, None]
    a, b = (slice(0, half), slice(half, 2 * half)) if halves else (slice(0, 2 * half, 2), slice(1, 2 * half, 2))
    out = x.clone()
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _freqs(dims, base, scaling=None):
    plain = [float(base) ** (-2.0 * i / dims) for i in range(dims // 2)]
    if scaling is None:
        return plain
    at = lambda turns: dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(at(scaling["fast"])), 0), min(math.ceil(at(scaling["slow"])), dims - 1)
    ramp = [min(max((i - lo) / max(hi - lo, 0.001), 0.0), 1.0) for i in range(dims // 2)]
    return [f * (1 - r) + f / scaling["factor"] * r for f, r in zip(plain, ramp)]


def _attend(q, k, v, scale, window=None, shape=None, sink=None):
    """q [B, T, H, D], k and v [B, T, G, ...]; `shape(scores, head)` bends the scaled scores, `sink[head]` joins the denominator."""
    B, T, H, _ = q.shape
    G = k.shape[2]
    back = torch.arange(T, device=q.device)[:, None] - torch.arange(T, device=q.device)[None]
    hidden = (back < 0) | (back >= window) if window else back < 0
    out = q.new_empty(B, T, H, v.shape[3])
    for b in range(B):
        for h in range(H):
            s = (q[b, :, h] @ k[b, :, h * G // H].t()) * scale
            if shape is not None:
                s = shape(s, h)
            s = s.masked_fill_(hidden, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = torch.clamp(top, min=float(sink[h]))
            e = torch.exp_(s - top)
            den = e.sum(-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(float(sink[h]) - top)
            out[b, :, h] = (e @ v[b, :, h * G // H]) / den
    return out


def _experts(h, w, ids, weights):
    """h [N, W], ids and weights [N, top]."""
    out = torch.zeros_like(h)
    for e in range(sum(1 for k in w if k.endswith(".down") and k[0] == "e")):
        row, col = (ids == e).nonzero(as_tuple=True)
        if row.numel():
            x = h[row]
            y = _lin(w[f"e{e}.down"], _silu(_lin(w[f"e{e}.gate"], x)) * _lin(w[f"e{e}.up"], x))
            out.index_add_(0, row, y * weights[row, col, None])
    return out


def _of_groups(choice, router, top):
    """Choice values outside the best groups (by the sum of a group's `top` best) set to minus infinity."""
    groups = router.get("groups")
    if not groups:
        return choice
    parts = choice.view(choice.shape[0], groups["count"], -1)
    kept = parts.topk(top, -1).values.sum(-1).topk(groups["keep"], -1).indices
    mask = torch.ones_like(parts, dtype=torch.bool).scatter_(1, kept[:, :, None].expand(-1, -1, parts.shape[2]), False)
    return parts.masked_fill(mask, -math.inf).view_as(choice)


def _exact_qwen3(config, w, x, last):
    eps, H, G, D = config["rms_norm_eps"], config["num_attention_heads"], config["num_key_value_heads"], config["head_dim"]
    norm = lambda v, name: _unit_rms(v, eps) * w[name].to(F)
    freqs = _freqs(D, config["rope_theta"])
    for i in range(config["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = norm(x, p + "input_layernorm.weight")
        q, k, v = (_lin(w[p + f"self_attn.{n}_proj.weight"], h).unflatten(-1, (-1, D)) for n in "qkv")
        q = _turn(norm(q, p + "self_attn.q_norm.weight"), freqs, True)
        k = _turn(norm(k, p + "self_attn.k_norm.weight"), freqs, True)
        x = x + _lin(w[p + "self_attn.o_proj.weight"], _attend(q, k, v, D ** -0.5).flatten(2))
        h = norm(x, p + "post_attention_layernorm.weight")
        x = x + _lin(w[p + "mlp.down_proj.weight"], _silu(_lin(w[p + "mlp.gate_proj.weight"], h)) * _lin(w[p + "mlp.up_proj.weight"], h))
    return _lin(w["lm_head.weight"], norm(last(x), "model.norm.weight"))


def _delta_steps(q, k, v, beta, decay):
    """decay [B, T, H]: decay, correct, write, then read."""
    decay = decay[..., None, None]
    state, out = q.new_zeros(*q.shape[:1], *q.shape[2:], v.shape[3]), torch.empty_like(v)
    for t in range(q.shape[1]):
        state = decay[:, t] * state
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdp,bhd->bhp", state, k[:, t]))
        state = state + k[:, t, :, :, None] * u[:, :, None]
        out[:, t] = torch.einsum("bhdp,bhd->bhp", state, q[:, t])
    return out


def _exact_puturax(config, w, x, last):
    eps = config["norm"]["eps"]
    norm = lambda v, name: _unit_rms(v, eps) * (1 + w[name].to(F))

    def latent(h, p, m):
        H, D, R, K = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        freqs = _freqs(m["rot"]["dims"], m["rot"]["base"])
        q = _lin(p["uq"], _unit_rms(_lin(p["dq"], h), eps) * p["dq.norm"].to(F)).unflatten(-1, (H, D + R))
        low = _lin(p["dkv"], h)
        c = _unit_rms(low[..., :K], eps) * p["dkv.norm"].to(F)
        turned = _turn(low[..., None, K:], freqs, True).expand(-1, -1, H, -1)
        q = torch.cat([q[..., :D], _turn(q[..., D:], freqs, True)], -1)
        k = torch.cat([_lin(p["uk"], c).unflatten(-1, (H, D)), turned], -1)
        out = _attend(q, k, _lin(p["uv"], c).unflatten(-1, (H, -1)), m["scale"]).flatten(2)
        return _lin(p["o"], out * torch.sigmoid(_lin(p["g"], h)))

    def attention(h, p, m):
        q, k, v = (_unit_rms(_lin(p[n], h).unflatten(-1, (-1, m["dim"])), eps) for n in "qkv")
        T = h.shape[1]
        at = torch.arange(T, device=h.device)
        q = q * (1 + m["q_temp"]["coef"] * torch.log(((at + 1) // m["q_temp"]["every"] + 1).to(F)))[:, None, None]
        back = (at[:, None] - at[None]).clamp(min=0).to(F)
        bend = lambda s, i: m["softcap"] * torch.tanh(s / m["softcap"]) - p["r1"].to(F)[i] * torch.log1p(p["r2"].to(F)[i] * back)
        out = _attend(q, k, v, m["scale"], shape=bend, sink=[0.0] * m["heads"]).flatten(2)
        return _lin(p["o"], out * torch.sigmoid(_lin(p["g"], h)))

    def time_mix(h, p, m):
        H = m["heads"]
        before = torch.cat([torch.zeros_like(h[:, :1]), h[:, :-1]], 1)
        mix = {n: h + (before - h) * p["mu." + n].to(F) for n in "rkvgw"}
        r, k, v = (_lin(p[n], mix[n]).unflatten(-1, (H, -1)) for n in "rkv")
        decay = torch.exp(-torch.exp(_lin(p["w2"], torch.tanh(_lin(p["w1"], mix["w"]))) + p["w0"].to(F))).unflatten(-1, (H, -1))
        u = p["u"].to(F).reshape(H, -1)
        state, out = h.new_zeros(h.shape[0], H, k.shape[3], v.shape[3]), torch.empty_like(v)
        for t in range(h.shape[1]):
            kv = k[:, t, :, :, None] * v[:, t, :, None]
            out[:, t] = torch.einsum("bhdp,bhd->bhp", state + u[..., None] * kv, r[:, t])
            state = decay[:, t, :, :, None] * state + kv
        return _lin(p["o"], _unit_rms(out, eps).flatten(2) * p["norm"].to(F) * _silu(_lin(p["g"], mix["g"])))

    def mixer(h, p, layer):
        m = layer["mixer"]
        if layer["type"] == "parallel":
            return m["left_scale"] * attention(h, _sub(p, "left."), m["left"]) + m["right_scale"] * time_mix(h, _sub(p, "right."), m["right"])
        return latent(h, p, m)

    def ff(h, p, m):
        if m["kind"] == "dense":
            return _lin(p["down"], torch.relu(_lin(p["up"], h)) ** 2)
        flat = h.flatten(0, 1)
        s = torch.sigmoid(_lin(p["router"], flat))
        ids = _of_groups(s + p["correction"].to(F), m["router"], 2).topk(m["router"]["top"], -1).indices
        weights = s.gather(1, ids)
        y = _experts(flat, p, ids, weights / (weights.sum(-1, keepdim=True) + 1e-20)).view_as(h)
        return y + _lin(p["shared.down"], _silu(_lin(p["shared.gate"], h)) * _lin(p["shared.up"], h))

    x = x * config["embedding"]["scale"]
    for i, layer in enumerate(config["layers"]):
        p = f"l{i}."
        x = x + norm(mixer(norm(x, p + "norm1"), _sub(w, p + "mix."), layer), p + "norm1b")
        x = x + norm(ff(norm(x, p + "norm2"), _sub(w, p + "mlp."), layer["mlp"]), p + "norm2b")
    return _lin(w["embed"], norm(last(x), "final.norm"))


def _exact_vekusun(config, w, x, last):
    eps = config["norm"]["eps"]
    norm = lambda v, g: _unit_rms(v, eps) * g.to(F)

    def latent(h, p, m):
        q = _lin(p["uq"], norm(_lin(p["dq"], h), p["dq.norm"])).unflatten(-1, (m["heads"], -1))
        c = norm(_lin(p["dkv"], h), p["dkv.norm"])
        k, v = (_lin(p[n], c).unflatten(-1, (m["heads"], -1)) for n in ("uk", "uv"))
        return _lin(p["o"], _attend(q, k, v, m["scale"], sink=p["sink"].tolist()).flatten(2))

    def rotated(h, p, m):
        H, D, K, rot = m["heads"], m["dim"], m["kv_rank"], m["rot"]
        freqs, amp = _freqs(rot["dims"], rot["base"], rot["scaling"]), 0.1 * math.log(rot["scaling"]["factor"]) + 1
        q, low = _lin(p["q"], h).unflatten(-1, (H, -1)), _lin(p["dkv"], h)
        c = norm(low[..., :K], p["dkv.norm"])
        k, v = (_lin(p[n], c).unflatten(-1, (H, -1)) for n in ("uk", "uv"))
        q = torch.cat([q[..., :D], _turn(q[..., D:], freqs, False, amp)], -1)
        k = torch.cat([k, _turn(low[..., None, K:], freqs, False, amp).expand(-1, -1, H, -1)], -1)
        return _lin(p["o"], (_attend(q, k, v, m["scale"]) * torch.sigmoid(_lin(p["g"], h))[..., None]).flatten(2))

    def delta(h, p, m):
        H, G = m["heads"], m["kv_heads"]
        q, k, v = (_silu(_conv(_lin(p[n], h), p[n + ".conv"])) for n in "qkv")
        q, k = (t.unflatten(-1, (G, -1)) for t in (q, k))
        q, k = ((t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(H // G, 2) for t in (q, k))
        decay = torch.exp(-torch.exp(p["A_log"].to(F)) * torch.nn.functional.softplus(_lin(p["a"], h) + p["dt_bias"].to(F)))
        o = _delta_steps(q * m["dim"] ** -0.5, k, v.unflatten(-1, (H, -1)), torch.sigmoid(_lin(p["b"], h)), decay)
        return _lin(p["o"], (norm(o, p["norm"]) * _silu(_lin(p["g"], h)).unflatten(-1, (H, -1))).flatten(2))

    def ff(h, p, m):
        if m["kind"] == "dense":
            return _lin(p["down"], torch.nn.functional.gelu(_lin(p["up"], h)))
        flat = h.flatten(0, 1)
        s = torch.softmax(_lin(p["router"], flat), -1)
        ids = (s + p["correction"].to(F)).topk(m["router"]["top"], -1).indices
        return _experts(flat, p, ids, s.gather(1, ids)).view_as(h)

    mixers = {"latent_attention": latent, "latent_attention_2": rotated, "delta": delta}
    n, (lo, hi, times) = len(config["layers"]), (config["loop"][k] for k in ("start", "stop", "times"))
    order = [(i, None) for i in range(lo)] + [(i, t) for t in range(times) for i in range(lo, hi)] + [(i, None) for i in range(hi, n)]
    first = x
    for i, turn in order:
        if turn is not None and i == lo:
            x = x + (first if turn else 0) + w["loop.step"].to(F)[turn]
        layer, p = config["layers"][i], _sub(w, f"l{i}.")
        h = norm(x, p["norm1"])
        y = p["ls1"].to(F) * mixers[layer["type"]](h, _sub(p, "mix."), layer["mixer"]) + p["ls2"].to(F) * ff(h, _sub(p, "mlp."), layer["mlp"])
        x = x + config["residual_mult"] * y
    cap = config["logit_softcap"]
    return cap * torch.tanh(_lin(w["head"], norm(last(x), w["final.norm"])) / cap)


def _exact_logits(case, config, weights, sequences):
    """Logits [len(sequences), vocab] at the last token of every sequence."""
    name = case["model"].split("-")[0]
    rows = []
    table = weights["model.embed_tokens.weight" if name == "qwen3" else "embed"]
    group = max(1, 16384 // max(len(s) for s in sequences))
    for at in range(0, len(sequences), group):
        part = sequences[at:at + group]
        ids = torch.zeros(len(part), max(len(s) for s in part), dtype=torch.long)
        for i, s in enumerate(part):
            ids[i, :len(s)] = torch.tensor(s)
        ends = torch.tensor([len(s) - 1 for s in part], device=DEVICE)
        last = lambda x, ends=ends: x[torch.arange(len(ends), device=DEVICE), ends]
        x = table[ids.to(DEVICE)].to(F)
        rows.append(globals()["_exact_" + name](config, weights, x, last))
    return torch.cat(rows)


def exact(case, seed):
    # the pass after the one that `prepare` makes: every decoding request has been fed one token and is fed the next
    decoding, prompts = _tokens(case, seed)
    ends = [n + 2 for n in _lengths(case["context_low"], case["context_high"], case["decoding"])]
    sequences = [ids[:n] for ids, n in zip(decoding, ends)] + prompts
    padded = len(sequences) * max(len(s) for s in sequences)
    if padded > 12000 and case["model"] == "qwen3-8b" or padded > 32000:
        return None                                      # minutes in 64 bits
    config, _, weights = _model(case, seed)
    with torch.no_grad():
        if not case["generate"]:
            return {"logits": _exact_logits(case, config, weights, sequences)}
        logits, tokens = [], []
        for _ in range(case["generate"]):
            logits.append(_exact_logits(case, config, weights, sequences))
            tokens.append(logits[-1].argmax(-1).tolist())
            sequences = [s + [t] for s, t in zip(sequences, tokens[-1])]
        return {"logits": torch.stack(logits), "tokens": torch.tensor(tokens)}
