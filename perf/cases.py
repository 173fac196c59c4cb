"""The work this framework is measured by: whole calls of `LLM.generate`, from token ids to token ids.

A case is a model, a compute dtype, a number of requests, the lengths of their prompts (spread evenly, in logarithm, over
`lo` .. `hi`; the order shuffled by a fixed rule), how many tokens each generates, and the temperature. Every pass is what a
serving program does with new prompts on a loaded engine: scheduling, prefill in portions, decode steps, token picks. The
result is every generated token and, for at most eight of the requests, the logits behind their last one.

Models: the Llama decoder at the sizes bench.py measures (1B, 3B, 8B) in bfloat16, the 1B sizes in float32 (the reference's
only dtype), and the Lomopel decoder (attention with a sink beside windowed attention and a gated delta rule) at bench.py's
sizes. Weights are random: projections N(0, 0.02), those that write the residual scaled down with the depth, and
an output head that prefers one token by several deviations, as a trained model does: the token that follows is then the
same in any correct implementation, whatever its rounding, and the logits of the last step can be compared.
"""
import math

import numpy as np
import torch

VOCAB = 128256
NEW_MOST = 64

# width, layers, attention heads, kv heads, head size, feed-forward, rope factor, tied head (bench.py's SIZES)
LLAMA = {
    "llama-1b": dict(width=2048, layers=16, heads=32, kv=8, hd=64, ff=8192, rope=32.0, tied=True),
    "llama-3b": dict(width=3072, layers=28, heads=24, kv=8, hd=128, ff=8192, rope=32.0, tied=True),
    "llama-8b": dict(width=4096, layers=32, heads=32, kv=8, hd=128, ff=14336, rope=8.0, tied=False),
}
# bench.py's LOMOPEL_SIZES["1b"], eight layers: twice [attention, parallel, parallel, attention]
LOMOPEL = {
    "lomopel-1b": dict(width=2048, kinds=("attention", "parallel", "parallel", "attention") * 2, heads=32, kv=8, hd=64, ff=8192,
                       window=1024, rot=32, rot_base=1e4, q_temp=(0.1, 1024), d_heads=16, d_kv=8, d_dim=128, conv=4, rank=64),
}
# what an engine of the model may hold: (requests at once, longest request, pages of 16 tokens)
LIMITS = {
    ("llama-1b", "bfloat16"): (64, 16384, 8192), ("llama-3b", "bfloat16"): (16, 8192, 4096),
    ("llama-8b", "bfloat16"): (16, 8192, 2048), ("llama-1b", "float32"): (16, 4096, 2048),
    ("lomopel-1b", "bfloat16"): (16, 4096, 2048),
}


def listed():
    def c(name, model, dtype, requests, lo, hi, new, temperature=0.0):
        return dict(name=name, model=model, dtype=dtype, requests=requests, lo=lo, hi=hi, new=new, temperature=temperature)
    return [
        # a short question, a few tokens back: the smallest call, all latency
        c("1b short", "llama-1b", "bfloat16", 1, 24, 24, 8),
        # one user, an answer of ordinary length
        c("1b answer", "llama-1b", "bfloat16", 1, 517, 517, 64),
        # a handful of chats at once, sampled; prompts of very different lengths
        c("1b chats", "llama-1b", "bfloat16", 8, 61, 1000, 48, 0.7),
        # a full batch of short requests: decode steps of 64 rows
        c("1b batch", "llama-1b", "bfloat16", 64, 17, 260, 32),
        # time to the first token of one full portion
        c("1b first token", "llama-1b", "bfloat16", 1, 2048, 2048, 1),
        # a few short prompts whose next token is all that is wanted (scoring, classification)
        c("1b scoring", "llama-1b", "bfloat16", 4, 33, 150, 1),
        # a long document, several portions over a growing cache, then decode far behind it
        c("1b document", "llama-1b", "bfloat16", 1, 11777, 11777, 16),
        # a serving mix at 3B: portions of prompts beside decoded tokens
        c("3b serving", "llama-3b", "bfloat16", 12, 130, 3000, 24),
        # a few requests at 8B
        c("8b chats", "llama-8b", "bfloat16", 4, 300, 1500, 16),
        # the 32-bit engine: one request, as a trace is checked token by token
        c("f32 answer", "llama-1b", "float32", 1, 100, 100, 16),
        # the 32-bit engine: several prompts at once
        c("f32 prompts", "llama-1b", "float32", 5, 50, 700, 4),
        # the recurrent design: portions through the gated delta rule and the window, then decode
        c("lomopel chats", "lomopel-1b", "bfloat16", 4, 200, 1500, 32),
    ]


def lengths(case):
    """The prompts' lengths: evenly spread in logarithm, in an order that is no order."""
    n, lo, hi = case["requests"], case["lo"], case["hi"]
    if n == 1:
        return [hi]
    got = [int(round(lo * (hi / lo) ** (i / (n - 1)))) for i in range(n)]
    step = next(s for s in (7, 5, 3, 2, 1) if math.gcd(s, n) == 1)
    return [got[(i * step + n // 2) % n] for i in range(n)]


def _cost(case):
    """A rough time of a pass, to keep drawn cases within the largest listed one."""
    w = work(case)
    return w["bytes"] / 4e12 + w["flops"] / (3e13 if case["dtype"] == "float32" else 8e14) + \
        (1.2e-6 * sum(lengths(case)) if case["model"] in LOMOPEL else 0.0)


def draw(rng):
    most = max(_cost(c) for c in listed())

    def spread(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))
    while True:
        model, dtype = rng.choice([("llama-1b", "bfloat16")] * 5 + [("llama-1b", "float32")] * 2 + [("lomopel-1b", "bfloat16")] * 2
                                  + [("llama-3b", "bfloat16"), ("llama-8b", "bfloat16")])
        seqs, longest, pages = LIMITS[(model, dtype)]
        n, new = spread(1, seqs), spread(1, NEW_MOST)
        a, b = sorted((spread(17, min(longest, 12000) - new), spread(17, min(longest, 12000) - new)))
        if n == 1:
            a = b
        case = dict(model=model, dtype=dtype, requests=n, lo=a, hi=b, new=new, temperature=rng.choice((0.0, 0.0, 0.7)))
        if sum(-(-(x + new) // 16) for x in lengths(case)) <= pages and _cost(case) <= most:
            return case


# ------------------------------------------------------------------------------------------------ weights
def _shapes(model):
    """(name, shape, kind) of every tensor. Kinds: in / out (projections from / to the residual), embed, head, final,
    and the small ones of the designs."""
    if model in LLAMA:
        m = LLAMA[model]
        h, q, kv, ff = m["width"], m["heads"] * m["hd"], m["kv"] * m["hd"], m["ff"]
        got = [("model.embed_tokens.weight", (VOCAB, h), "embed")]
        for i in range(m["layers"]):
            p = f"model.layers.{i}."
            got += [(p + "input_layernorm.weight", (h,), "norm"), (p + "self_attn.q_proj.weight", (q, h), "in"),
                    (p + "self_attn.k_proj.weight", (kv, h), "in"), (p + "self_attn.v_proj.weight", (kv, h), "in"),
                    (p + "self_attn.o_proj.weight", (h, q), "out"), (p + "post_attention_layernorm.weight", (h,), "norm"),
                    (p + "mlp.gate_proj.weight", (ff, h), "in"), (p + "mlp.up_proj.weight", (ff, h), "in"),
                    (p + "mlp.down_proj.weight", (h, ff), "out")]
        got.append(("model.norm.weight", (h,), "final"))
        return got + ([] if m["tied"] else [("lm_head.weight", (VOCAB, h), "head")])
    m = LOMOPEL[model]
    w, q, kv, ff = m["width"], m["heads"] * m["hd"], m["kv"] * m["hd"], m["ff"]
    dk, dq, r = m["d_kv"] * m["d_dim"], m["d_heads"] * m["d_dim"], m["rank"]
    got = [("embed", (VOCAB, w), "embed")]
    for i, kind in enumerate(m["kinds"]):
        p, x = f"l{i}.", f"l{i}.mix."
        got += [(p + "norm1", (w,), "small"), (p + "ls1", (w,), "norm")]
        if kind == "attention":
            got += [(x + "q", (q, w), "in"), (x + "q.b", (q,), "small"), (x + "k", (kv, w), "in"), (x + "k.b", (kv,), "small"),
                    (x + "v", (kv, w), "in"), (x + "v.b", (kv,), "small"), (x + "sink", (m["heads"],), "small"),
                    (x + "o", (w, q), "out"), (x + "o.b", (w,), "small"), (x + "vmix", (), "vmix")]
        else:
            y = x + "left."
            got += [(y + "q", (q, w), "in"), (y + "k", (kv, w), "in"), (y + "v", (kv, w), "in"), (y + "g", (q, w), "in"),
                    (y + "o", (w, q), "out")]
            y = x + "right."
            got += [(y + "q", (dk, w), "in"), (y + "q.conv", (dk, m["conv"]), "conv"), (y + "k", (dk, w), "in"),
                    (y + "k.conv", (dk, m["conv"]), "conv"), (y + "v", (dq, w), "in"), (y + "v.conv", (dq, m["conv"]), "conv"),
                    (y + "b", (m["d_heads"], w), "in"), (y + "A_log", (m["d_heads"],), "A_log"), (y + "norm", (m["d_dim"],), "norm"),
                    (y + "a1", (r, w), "in"), (y + "a2", (dq, r), "in"), (y + "dt_bias", (dq,), "dt_bias"), (y + "g1", (r, w), "in"),
                    (y + "g2", (dq, r), "in"), (y + "o", (w, dq), "out")]
        got += [(p + "norm2", (w,), "small"), (p + "ls2", (w,), "norm"), (p + "mlp.gate", (ff, w), "in"), (p + "mlp.up", (ff, w), "in"),
                (p + "mlp.down", (w, ff), "out")]
    return got + [("final.norm", (w,), "small"), ("head", (VOCAB, w), "head")]


HEAD_SCALE = 0.05                       # logits of a deviation of about two
FOLLOW, FOLLOW_STEP = 77761, 12345      # an untied head prefers token (t * FOLLOW + FOLLOW_STEP) mod VOCAB behind token t


def _layers(model):
    return LLAMA[model]["layers"] if model in LLAMA else len(LOMOPEL[model]["kinds"])


def _weights(model, dtype):
    """Every tensor on the GPU, the same at every call."""
    g = torch.Generator(device="cuda").manual_seed(20240613)
    dt = getattr(torch, dtype)
    out_std = 0.02 / math.sqrt(2 * _layers(model)) * 2.0
    got = {}

    def normal(shape, std, mean=0.0):
        return (torch.randn(shape, generator=g, device="cuda", dtype=torch.float32) * std + mean).to(dt)
    for name, shape, kind in _shapes(model):
        if kind == "embed":
            t = normal(shape, 1.0)
        elif kind == "head":
            embed = got["model.embed_tokens.weight" if model in LLAMA else "embed"]
            t = torch.empty_like(embed)
            t[(torch.arange(VOCAB, device="cuda") * FOLLOW + FOLLOW_STEP) % VOCAB] = embed * HEAD_SCALE
        elif kind == "final":
            t = normal(shape, 0.002, HEAD_SCALE if LLAMA[model]["tied"] else 1.0)
        elif kind == "A_log":
            t = (torch.rand(shape, generator=g, device="cuda") * 15 + 1).log().to(dt)
        elif kind == "dt_bias":         # the inverse softplus of steps spread over 0.001 .. 0.1
            t = torch.exp(torch.rand(shape, generator=g, device="cuda") * math.log(100.0) + math.log(0.001)).expm1().log().to(dt)
        elif kind == "vmix":
            t = torch.full(shape, 0.5, device="cuda", dtype=dt)
        else:
            std, mean = {"in": (0.02, 0.0), "out": (out_std, 0.0), "norm": (0.1, 1.0), "small": (0.1, 0.0), "conv": (0.3, 0.0)}[kind]
            t = normal(shape, std, mean)
        got[name] = t
    return got


def _prompts(case, seed):
    g = torch.Generator().manual_seed(int(seed))
    return [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in lengths(case)]


def _asked(case):
    """The requests whose last logits are wanted: at most eight, spread over the batch."""
    n = case["requests"]
    return list(range(0, n, -(-n // 8)))


# ------------------------------------------------------------------------------------------------ the framework's side
_engine = {}        # the engine of the model last asked for: a serving program loads its model once


def _llm(model, dtype):
    key = (model, dtype)
    if key not in _engine:
        _engine.clear()
        torch.cuda.empty_cache()
        from vllm_oxide_b200 import config as C
        from vllm_oxide_b200 import models  # noqa: F401  (registers the architectures)
        from vllm_oxide_b200.engine import LLM, ModelRunner
        if model in LLAMA:
            m = LLAMA[model]
            cfg = C.LlamaConfig(hidden_size=m["width"], intermediate_size=m["ff"], num_hidden_layers=m["layers"],
                                num_attention_heads=m["heads"], num_key_value_heads=m["kv"], head_dim=m["hd"], vocab_size=VOCAB,
                                max_position_embeddings=131072, rms_norm_eps=1e-5, rope_theta=500000.0,
                                rope_scaling=C.RopeScaling(m["rope"], 1.0, 4.0, 8192), tie_word_embeddings=m["tied"],
                                bos_token_id=128000, eos_token_ids=(128001,))
        else:
            m = LOMOPEL[model]
            heads = dict(heads=m["heads"], kv_heads=m["kv"], dim=m["hd"], vdim=m["hd"])
            full = C.SoftmaxMixerConfig(scale=m["hd"] ** -0.5, q_temp=m["q_temp"], v_mix=True, **heads)
            left = C.SoftmaxMixerConfig(scale=1.0 / 8, window=m["window"], rot_dims=m["rot"], rot_base=m["rot_base"], **heads)
            right = C.GatedDeltaConfig(heads=m["d_heads"], kv_heads=m["d_kv"], dim=m["d_dim"], vdim=m["d_dim"], conv=m["conv"],
                                       decay_rank=m["rank"], gate_rank=m["rank"])
            kinds = {"attention": C.LomopelLayer("attention", attention=full, ff=m["ff"]),
                     "parallel": C.LomopelLayer("parallel", left=left, right=right, left_scale=1.0, right_scale=1.0, ff=m["ff"])}
            cfg = C.LomopelConfig(vocab=VOCAB, width=m["width"], layers=tuple(kinds[k] for k in m["kinds"]), norm_eps=1e-5,
                                  embedding_scale=1.0)
        seqs, longest, pages = LIMITS[key]
        _engine[key] = LLM(ModelRunner(cfg, _weights(model, dtype), C.EngineConfig(
            max_batch_tokens=2048, max_seqs=seqs, max_model_len=longest, block_size=16, num_pages=pages, dtype=dtype)))
        torch.cuda.empty_cache()
    return _engine[key]


def prepare(case, seed):
    from vllm_oxide_b200.sampling import SamplingParams
    llm, asked = _llm(case["model"], case["dtype"]), set(_asked(case))
    params = [SamplingParams(max_new_tokens=case["new"], temperature=case["temperature"], seed=1000 * (int(seed) % 1000000) + i,
                             stop_token_ids=(), capture_logits=(case["new"] - 1,) if i in asked else ())
              for i in range(case["requests"])]
    return {"llm": llm, "prompts": _prompts(case, seed), "params": params, "asked": sorted(asked), "last": case["new"] - 1}


def run(state):
    outs = state["llm"].generate(state["prompts"], state["params"])
    return {"tokens": torch.tensor([o.token_ids for o in outs]), "logits": [outs[i].logits[state["last"]] for i in state["asked"]]}


# ------------------------------------------------------------------------------------------------ what a pass needs
def work(case):
    """A pass reads the weights once for the prompts and once for every further token (each depends on the one in front, and
    no model here fits the cache), the keys and values of every decoded token's context, and writes what was asked for."""
    model, new, n = case["model"], case["new"], lengths(case)
    es = 4 if case["dtype"] == "float32" else 2
    table = next(math.prod(s) for _, s, k in _shapes(model) if k == "embed")
    proj = sum(math.prod(s) for _, s, k in _shapes(model) if k not in ("embed", "head"))
    m = LLAMA.get(model) or LOMOPEL[model]
    tokens = sum(n) + len(n) * (new - 1)
    flops = 2.0 * proj * tokens + 2.0 * table * len(n) * new
    read = 0.0
    state = 0.0
    for i in range(_layers(model)):
        window = 1 << 40
        if model in LOMOPEL and m["kinds"][i] == "parallel":
            window = m["window"]
            flops += 8.0 * m["d_heads"] * m["d_dim"] ** 2 * tokens
            state += 2.0 * 4 * m["d_heads"] * m["d_dim"] ** 2 * len(n) * new
        for length in n:
            total = length + new - 1
            t = min(total, window)
            flops += 4.0 * m["heads"] * m["hd"] * (t * (t + 1) / 2 + (total - t) * window)
            read += 2.0 * m["kv"] * m["hd"] * es * sum(min(x, window) for x in range(length + 1, total + 1))
    written = 4.0 * VOCAB * len(_asked(case)) + 8.0 * len(n) * new
    return {"bytes": (proj + table) * es * float(new) + read + state + written, "flops": flops}


def tolerance(case):
    """Four times the largest error seen against `exact`: 0.006 (1B, 3B) to 0.010 (8B) in bfloat16, 2.6e-6 in float32. Tokens
    are the same: an output head that prefers one by several deviations leaves nothing to rounding."""
    return {"rel": 1e-5, "max": 1e-4} if case["dtype"] == "float32" else {"rel": 0.03, "max": 0.2}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x, eps=1e-5):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, scale, window=0, sink=None):
    """Causal attention of one sequence: q [T, H, d], k and v [T, G, d]; query head a reads key head a // (H / G)."""
    T, H, d = q.shape
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    q = q.reshape(T, G, H // G, d)
    for a in range(0, T, 512):
        b = min(T, a + 512)
        first = max(0, a + 1 - window) if window else 0
        s = torch.einsum("tgrd,sgd->grts", q[a:b], k[first:b]) * scale
        at = torch.arange(a, b, device=q.device)[:, None] - torch.arange(first, b, device=q.device)[None, :]
        s.masked_fill_((at < 0) | (at >= window) if window else at < 0, -math.inf)
        top = s.amax(-1, keepdim=True)
        if sink is not None:
            top = torch.maximum(top, sink.reshape(G, H // G, 1, 1))
        e = torch.exp(s - top)
        den = e.sum(-1, keepdim=True)
        if sink is not None:
            den = den + torch.exp(sink.reshape(G, H // G, 1, 1) - top)
        out[a:b] = torch.einsum("grts,sgd->tgrd", e / den, v[first:b]).reshape(b - a, H, -1)
    return out.reshape(T, -1)


def _turn(x, angles):
    """Rotary positions, pairs half of the rotated features apart: x [T, heads, d], angles [T, half] in 64 bits."""
    half = angles.shape[1]
    c, s = torch.cos(angles)[:, None], torch.sin(angles)[:, None]
    a, b = x[..., :half], x[..., half:2 * half]
    return torch.cat([a * c - b * s, b * c + a * s, x[..., 2 * half:]], dim=-1)


def _llama_angles(m, T):
    """float32(position) * frequency, as the reference forms it; frequencies with the llama3 rule."""
    half = m["hd"] // 2
    f = (1.0 / np.power(500000.0, np.arange(half) * 2.0 / m["hd"])).astype(np.float32)
    wave = 2 * np.pi / f.astype(np.float64)
    smooth = np.clip((8192 / wave - 1.0) / 3.0, 0.0, 1.0)
    f = ((1 - smooth) * f / m["rope"] + smooth * f).astype(np.float32)
    at = torch.arange(T, dtype=torch.float32)[:, None] * torch.from_numpy(f)
    return at.double().cuda()


def _gated_delta(h, t, m):
    """The gated delta rule of one sequence, token by token."""
    T, H, G, d = h.shape[0], m["d_heads"], m["d_kv"], m["d_dim"]

    def conv(name):
        x, w = h @ t(name).T, t(name + ".conv")
        x = torch.cat([x.new_zeros(m["conv"] - 1, x.shape[1]), x])
        y = sum(x[j:j + T] * w[:, j] for j in range(m["conv"]))
        return y * torch.sigmoid(y)

    def unit(x):
        return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
    q = (unit(conv("q").reshape(T, G, d)) * d ** -0.5).repeat_interleave(H // G, dim=1)
    k = unit(conv("k").reshape(T, G, d)).repeat_interleave(H // G, dim=1)
    v = conv("v").reshape(T, H, d)
    beta = torch.sigmoid(h @ t("b").T)[..., None]
    step = torch.nn.functional.softplus(h @ t("a1").T @ t("a2").T + t("dt_bias")).reshape(T, H, d)
    decay = torch.exp(-torch.exp(t("A_log"))[:, None] * step)
    S = h.new_zeros(H, d, d)
    o = h.new_empty(T, H, d)
    for i in range(T):
        S = S * decay[i][:, :, None]
        u = beta[i] * (v[i] - torch.bmm(k[i][:, None], S)[:, 0])
        S = torch.baddbmm(S, k[i][:, :, None], u[:, None])
        o[i] = torch.bmm(q[i][:, None], S)[:, 0]
    gate = torch.sigmoid(h @ t("g1").T @ t("g2").T).reshape(T, H, d)
    return (_rms(o) * t("norm") * gate).reshape(T, H * d) @ t("o").T


def exact(case, seed):
    """The prompts with the tokens that follow them through plain torch in 64 bits: the tokens of the largest logits, and the
    logits of the last step. Sampled tokens come from the framework's own random numbers: nothing in 64 bits says which."""
    model, new, n = case["model"], case["new"], lengths(case)
    if case["temperature"] > 0 or sum(n) * sum(math.prod(s) for _, s, k in _shapes(model) if k in ("in", "out")) > 1.0e14:
        return None
    w = _weights(model, case["dtype"])
    llama = model in LLAMA
    m = LLAMA.get(model) or LOMOPEL[model]
    seqs = []
    for p in _prompts(case, seed):
        while len(p) < n[len(seqs)] + new - 1:
            p.append(p[-1] if llama and m["tied"] else (p[-1] * FOLLOW + FOLLOW_STEP) % VOCAB)
        seqs.append(p)
    at = np.cumsum([0] + [len(p) for p in seqs])
    spans = [slice(int(a), int(b)) for a, b in zip(at[:-1], at[1:])]
    x = w["model.embed_tokens.weight" if llama else "embed"][torch.tensor([t for p in seqs for t in p], device="cuda")].double()
    heads = lambda z, c: z.reshape(len(z), c, m["hd"])  # noqa: E731
    if llama:
        angles = _llama_angles(m, max(len(p) for p in seqs))
        for i in range(m["layers"]):
            t = lambda name: w[f"model.layers.{i}.{name}.weight"].double()  # noqa: E731
            h = _rms(x) * t("input_layernorm")
            q, k, v = h @ t("self_attn.q_proj").T, h @ t("self_attn.k_proj").T, h @ t("self_attn.v_proj").T
            a = torch.cat([_attend(_turn(heads(q[s], m["heads"]), angles[:s.stop - s.start]), _turn(heads(k[s], m["kv"]), angles[:s.stop - s.start]),
                                   heads(v[s], m["kv"]), m["hd"] ** -0.5) for s in spans])
            x = x + a @ t("self_attn.o_proj").T
            h = _rms(x) * t("post_attention_layernorm")
            x = x + (torch.nn.functional.silu(h @ t("mlp.gate_proj").T) * (h @ t("mlp.up_proj").T)) @ t("mlp.down_proj").T
        final, head = w["model.norm.weight"].double(), w["model.embed_tokens.weight" if m["tied"] else "lm_head.weight"]
    else:
        v_first = None
        freq = m["rot_base"] ** (-2.0 * torch.arange(m["rot"] // 2, dtype=torch.float64, device="cuda") / m["rot"])
        for i, kind in enumerate(m["kinds"]):
            t = lambda name: w[f"l{i}.{name}"].double()  # noqa: E731
            h = _rms(x) * (1 + t("norm1"))
            if kind == "attention":
                q, k, v = (h @ t("mix." + c).T + t(f"mix.{c}.b") for c in "qkv")
                if v_first is None:
                    v_first = v
                else:
                    v = (1 - t("mix.vmix")) * v + t("mix.vmix") * v_first
                ys = []
                for s in spans:
                    pos = torch.arange(s.stop - s.start, device="cuda")
                    coef, every = m["q_temp"]
                    factor = 1 + coef * torch.log(((pos + 1) // every + 1).double())
                    ys.append(_attend(heads(q[s], m["heads"]) * factor[:, None, None], heads(k[s], m["kv"]), heads(v[s], m["kv"]),
                                      m["hd"] ** -0.5, sink=t("mix.sink")))
                y = torch.cat(ys) @ t("mix.o").T + t("mix.o.b")
            else:
                q, k, v = (h @ t("mix.left." + c).T for c in "qkv")
                ys = []
                for s in spans:
                    ang = torch.arange(s.stop - s.start, device="cuda").double()[:, None] * freq
                    ys.append(_attend(_rms(_turn(heads(q[s], m["heads"]), ang)), _rms(_turn(heads(k[s], m["kv"]), ang)),
                                      heads(v[s], m["kv"]), 1.0 / 8, window=m["window"]))
                y = (torch.cat(ys) * torch.sigmoid(h @ t("mix.left.g").T)) @ t("mix.left.o").T
                y = y + torch.cat([_gated_delta(h[s], lambda name: t("mix.right." + name), m) for s in spans])
            x = x + y * t("ls1")
            h = _rms(x) * (1 + t("norm2"))
            x = x + ((torch.nn.functional.gelu(h @ t("mlp.gate").T, approximate="tanh") * (h @ t("mlp.up").T)) @ t("mlp.down").T) * t("ls2")
        final, head = 1 + w["final.norm"].double(), w["head"]
    x = _rms(x) * final
    rows = torch.cat([x[s.stop - new:s.stop] for s in spans])
    logits = torch.cat([rows @ head[a:a + 8192].double().T for a in range(0, VOCAB, 8192)], dim=1).reshape(len(n), new, VOCAB)
    return {"tokens": logits.argmax(-1).cpu(), "logits": [logits[i, -1].cpu() for i in _asked(case)]}
