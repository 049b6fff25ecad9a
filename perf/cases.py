"""The work that a user has this library do, as measurable cases.

A case is one pass through the public entry points on a model with seeded random weights: a decode step of a batch, the
prompts of a batch, a conversation's next turn, whole requests from prompt to last token, scoring of a text, or sampling
from a batch's logits.  Three of the architectures stand for the kinds of model the library runs: Qwen3 (dense, attention
over a paged cache), Sokirax (routed experts, attention in a window, a state per sequence) and Gigopel (latent attention,
parallel blocks).  Layer sizes are those of `bench.py` ("2k", "4k", "8b"), a small generic one ("1k") and one whose sizes
are no powers of two ("odd"); depths are cut so that a model with its inputs fits a card several times.

Every function is a plain function of a case (a dict of plain values) and a seed; `exact` is the same computation in
64 bits in plain torch.
"""
import math

import numpy as np
import torch

import gogguf_b200 as gg
from gogguf_b200.config import config_from_dict
from gogguf_b200.engine import Model

PAGE = 64

# hidden, query heads, key/value heads, head size, inner width, vocabulary, tied head
QWEN = {
    "1k": dict(hidden=1024, heads=16, kv=8, dim=64, inter=3072, vocab=32000, tied=True),
    "2k": dict(hidden=2048, heads=16, kv=8, dim=128, inter=5376, vocab=65536, tied=True),
    "odd": dict(hidden=1800, heads=15, kv=5, dim=120, inter=4744, vocab=50021, tied=False),
    "8b": dict(hidden=4096, heads=32, kv=8, dim=128, inter=12288, vocab=151936, tied=False),
}
SOKIRAX = {"2k": dict(width=2048, heads=16, kv=8, window=1024, ret=8, experts=16, top=2, ff=1024, shared=1024, vocab=65536)}
GIGOPEL = {"2k": dict(width=2048, heads=16, dim=64, rot=32, vdim=64, rank=256, window=1024, ff=8192, vocab=65536)}


def listed():
    return [
        # the smallest call: one person's short chat with a small model, a token at a time; latency and launches
        dict(name="decode_b1_1k", model="qwen3", shape="1k", layers=4, dtype="bfloat16", do="decode", batch=1, ctx=23, new=1),
        # the headline: a batch of eight goes on by one token from 2,048-token contexts
        dict(name="decode_b8_8b", model="qwen3", shape="8b", layers=8, dtype="bfloat16", do="decode", batch=8, ctx=2048, new=1),
        # a busy server: many requests of unequal lengths
        dict(name="decode_b61_2k", model="qwen3", shape="2k", layers=8, dtype="bfloat16", do="decode", batch=61, ctx=700, new=1),
        # one long prompt
        dict(name="prompt_2048_8b", model="qwen3", shape="8b", layers=8, dtype="bfloat16", do="prompt", batch=1, ctx=0, new=2048),
        # a batch of short prompts of unequal lengths, run together
        dict(name="prompt_ragged_2k", model="qwen3", shape="2k", layers=8, dtype="bfloat16", do="prompt", batch=6, ctx=0, new=90),
        # a conversation's next turn: a few hundred new tokens over a long history
        dict(name="turn_8b", model="qwen3", shape="8b", layers=4, dtype="bfloat16", do="decode", batch=1, ctx=6100, new=333),
        # the 32-bit path: prompts (layer-by-layer comparisons, reference runs) ...
        dict(name="f32_prompt_2k", model="qwen3", shape="2k", layers=4, dtype="float32", do="prompt", batch=3, ctx=0, new=150),
        # ... and decode steps
        dict(name="f32_decode_2k", model="qwen3", shape="2k", layers=8, dtype="float32", do="decode", batch=4, ctx=600, new=1),
        # routed experts: a long prompt
        dict(name="experts_prompt_2k", model="sokirax", shape="2k", layers=4, dtype="bfloat16", do="prompt", batch=1, ctx=0, new=2048),
        # routed experts: whole short requests, from prompt to last token
        dict(name="experts_requests_2k", model="sokirax", shape="2k", layers=4, dtype="bfloat16", do="requests", batch=8, ctx=0, new=60),
        # latent attention: whole requests with longer prompts
        dict(name="latent_requests_2k", model="gigopel", shape="2k", layers=4, dtype="bfloat16", do="requests", batch=4, ctx=0, new=350),
        # choosing the next tokens of a batch: temperature, top-k and top-p
        dict(name="sample_b64", model="sampler", vocab=151936, do="sample", batch=64, temp=0.6, top_k=20, top_p=0.95),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["decode", "decode", "prompt", "prompt", "turn", "score", "f32_prompt", "f32_decode", "experts", "experts",
                       "latent", "sample"])
    if kind == "sample":
        top_k = rng.choice([0, 20, 50, 400])
        return dict(model="sampler", vocab=log(30000, 152000), do="sample", batch=log(1, 64), temp=rng.choice([0.6, 1.0]),
                    top_k=top_k, top_p=rng.choice([0.9, 0.95]) if top_k == 0 else rng.choice([0.8, 0.95, 1.0]))
    if kind == "experts":
        do = rng.choice(["prompt", "requests"])
        batch = log(1, 8)
        return dict(model="sokirax", shape="2k", layers=rng.choice([2, 4]), dtype="bfloat16", do=do, batch=batch, ctx=0,
                    new=log(40, 2048) // batch + 3 if do == "prompt" else log(5, 120))
    if kind == "latent":
        do = rng.choice(["prompt", "requests"])
        batch = log(1, 8)
        return dict(model="gigopel", shape="2k", layers=rng.choice([2, 4]), dtype="bfloat16", do=do, batch=batch, ctx=0,
                    new=log(40, 2048) // batch + 3)
    if kind in ("f32_prompt", "f32_decode"):
        batch = log(1, 8)
        c = dict(model="qwen3", shape=rng.choice(["1k", "2k", "odd"]), layers=rng.choice([2, 4]), dtype="float32", batch=batch)
        if kind == "f32_prompt":
            return dict(c, do="prompt", ctx=0, new=log(10, 600) // batch + 1)
        return dict(c, do="decode", ctx=log(16, 900), new=1)
    shape = rng.choice(["1k", "2k", "odd", "8b"])
    c = dict(model="qwen3", shape=shape, layers=rng.choice([2, 4, 8]) if shape != "8b" else rng.choice([2, 4]), dtype="bfloat16")
    if kind == "decode":
        batch = log(1, 64)
        return dict(c, do="decode", batch=batch, ctx=log(16, min(3000, 60000 // batch)), new=1)
    if kind == "prompt":
        batch = log(1, 8)
        return dict(c, do="prompt", batch=batch, ctx=0, new=log(8, 2048) // batch + 1)
    if kind == "turn":
        return dict(c, do="decode", batch=rng.choice([1, 1, 2]), ctx=log(500, 6000), new=log(2, 400))
    return dict(c, do="score", batch=1, ctx=0, new=log(5, 300))


# ------------------------------------------------------------------------------------------------------------ sizes
def _lengths(case, mean):
    """Unequal lengths around `mean`, one per sequence (0.4 to 1.6 times it); one sequence has exactly `mean`."""
    b = case["batch"]
    if b == 1 or mean <= 1 or (mean & (mean - 1)) == 0:      # a power of two: equal lengths
        return [mean] * b
    return [max(1, int(mean * (0.4 + 1.2 * ((i * 0.61803398875 + 0.5) % 1.0)))) for i in range(b)]


def _new_tokens(case):
    return _lengths(case, case["new"])


REQUEST_STEPS = 4        # decode steps of a "requests" pass


def _config(case):
    if case["model"] == "qwen3":
        z = QWEN[case["shape"]]
        return dict(architectures=["Qwen3ForCausalLM"], model_type="qwen3", num_hidden_layers=case["layers"], hidden_size=z["hidden"],
                    num_attention_heads=z["heads"], num_key_value_heads=z["kv"], head_dim=z["dim"], intermediate_size=z["inter"],
                    vocab_size=z["vocab"], rope_theta=1000000.0, rms_norm_eps=1e-6, tie_word_embeddings=z["tied"],
                    max_position_embeddings=8192)
    if case["model"] == "sokirax":
        z = SOKIRAX[case["shape"]]
        H, G, R = z["heads"], z["kv"], z["ret"]
        att = dict(heads=H, kv_heads=G, dim=128, vdim=128, scale=128 ** -0.5, mask=dict(size=z["window"]),
                   rot=dict(base=500000.0, dims=64))
        left = dict(heads=H, kv_heads=G, dim=64, vdim=64, scale=0.125, mask=dict(size=z["window"]), rot=dict(base=100000.0, dims=32))
        right = dict(heads=R, dim=128, vdim=128, rot=dict(base=500000.0, dims=32),
                     decay=[1.0 - 2.0 ** (-5.0 - 7.0 * i / max(R - 1, 1)) for i in range(R)])
        par = dict(left=left, right=right, left_scale=1.0, right_scale=0.9)
        mlp = dict(kind="moe", expert=dict(ff=z["ff"]), router=dict(experts=z["experts"], top=z["top"]), shared=dict(ff=z["shared"]))
        return dict(architecture="Sokirax", vocab=z["vocab"], width=z["width"], norm=dict(eps=1e-6),
                    layers=[dict(type="attention", mixer=att, mlp=mlp) if i % 2 == 0 else dict(type="parallel", mixer=par, mlp=mlp)
                            for i in range(case["layers"])])
    z = GIGOPEL[case["shape"]]
    mixer = dict(heads=z["heads"], dim=z["dim"], rot_dim=z["rot"], vdim=z["vdim"], kv_rank=z["rank"],
                 scale=(z["dim"] + z["rot"]) ** -0.5, rot=dict(base=500000.0, dims=z["rot"]), mask=dict(size=z["window"]))
    return dict(architecture="Gigopel", vocab=z["vocab"], width=z["width"], residual_mult=0.5, norm=dict(eps=1e-6),
                layers=[dict(type="latent_attention", mixer=mixer, mlp=dict(kind="dense", ff=z["ff"])) for _ in range(case["layers"])])


# ----------------------------------------------------------------------------------------------------------- weights
class _Draw:
    def __init__(self, case, seed):
        self.g = torch.Generator(device="cuda").manual_seed(seed * 7919 + 17)
        self.dtype = torch.float32 if case["dtype"] == "float32" else torch.bfloat16

    def matrix(self, *shape, std=0.02):
        return (torch.randn(shape, generator=self.g, device="cuda", dtype=self.dtype) * std).to(self.dtype)

    def vector(self, n, mean=1.0, std=0.05):
        return (mean + std * torch.randn(n, generator=self.g, device="cuda")).to(self.dtype)


def _weights(case, seed):
    """The model's tensors by checkpoint name."""
    d, t = _Draw(case, seed), {}
    L = case["layers"]
    if case["model"] == "qwen3":
        z = QWEN[case["shape"]]
        W, D, I = z["hidden"], z["dim"], z["inter"]
        t["model.embed_tokens.weight"] = d.matrix(z["vocab"], W)
        for i in range(L):
            p = f"model.layers.{i}."
            for name, n, k in (("self_attn.q_proj", z["heads"] * D, W), ("self_attn.k_proj", z["kv"] * D, W),
                               ("self_attn.v_proj", z["kv"] * D, W), ("self_attn.o_proj", W, z["heads"] * D),
                               ("mlp.gate_proj", I, W), ("mlp.up_proj", I, W), ("mlp.down_proj", W, I)):
                t[p + name + ".weight"] = d.matrix(n, k)
            for name, n in (("self_attn.q_norm", D), ("self_attn.k_norm", D), ("input_layernorm", W), ("post_attention_layernorm", W)):
                t[p + name + ".weight"] = d.vector(n)
        t["model.norm.weight"] = d.vector(W)
        if not z["tied"]:
            t["lm_head.weight"] = d.matrix(z["vocab"], W)
    elif case["model"] == "sokirax":
        z = SOKIRAX[case["shape"]]
        W, H, G, R, E, F = z["width"], z["heads"], z["kv"], z["ret"], z["experts"], z["ff"]
        routers = []
        for i in range(L):
            p = f"l{i}."
            for name in ("norm1", "norm2"):
                t[p + name] = d.vector(W)
            for name in ("norm1b", "norm2b"):         # what a part adds is small next to the stream, as after training
                t[p + name] = d.vector(W, mean=0.25, std=0.02)

            def attn(q, dim, whole):
                t[q + "q"], t[q + "k"] = d.matrix(H * dim, W), d.matrix(G * dim, W)
                t[q + "v"], t[q + "o"] = d.matrix(G * dim, W), d.matrix(W, H * dim)
                t[q + "q.norm"], t[q + "k.norm"] = (d.vector(H * dim), d.vector(G * dim)) if whole else (d.vector(dim), d.vector(dim))

            if i % 2 == 0:
                attn(p + "mix.", 128, False)
            else:
                attn(p + "mix.left.", 64, True)
                t[p + "mix.left.sink"] = d.vector(H, mean=0.0, std=0.5)
                for name in ("q", "k", "v", "g"):
                    t[p + "mix.right." + name] = d.matrix(R * 128, W)
                t[p + "mix.right.o"] = d.matrix(W, R * 128)
            m = p + "mlp."
            t[m + "router"] = d.matrix(E, W)
            routers.append(t[m + "router"])
            for e in list(range(E)):
                t[f"{m}e{e}.gate"], t[f"{m}e{e}.up"], t[f"{m}e{e}.down"] = d.matrix(F, W), d.matrix(F, W), d.matrix(W, F)
            S = z["shared"]
            t[m + "shared.gate"], t[m + "shared.up"], t[m + "shared.down"] = d.matrix(S, W), d.matrix(S, W), d.matrix(W, S)
        # a token leans towards two experts of every layer, as routers that were trained see it: their choice is no toss-up
        x = torch.randn((z["vocab"], W), generator=d.g, device="cuda")
        for r in routers:
            first = torch.randint(0, E, (z["vocab"],), generator=d.g, device="cuda")
            second = (first + torch.randint(1, E, (z["vocab"],), generator=d.g, device="cuda")) % E
            x += 10.0 * r.float()[first] + 8.0 * r.float()[second]
        t["embed"] = x.to(d.dtype)
        t["final.norm"] = d.vector(W)
        t["head"] = d.matrix(z["vocab"], W)
    else:
        z = GIGOPEL[case["shape"]]
        W, H = z["width"], z["heads"]
        t["embed"] = d.matrix(z["vocab"], W)
        for i in range(L):
            p = f"l{i}."
            t[p + "norm1"] = d.vector(W, mean=0.0)
            m = p + "mix."
            t[m + "q"], t[m + "dkv"] = d.matrix(H * (z["dim"] + z["rot"]), W), d.matrix(z["rank"] + z["rot"], W)
            t[m + "dkv.norm"] = d.vector(z["rank"])
            t[m + "uk"], t[m + "uv"] = d.matrix(H * z["dim"], z["rank"], std=0.05), d.matrix(H * z["vdim"], z["rank"], std=0.05)
            t[m + "o"] = d.matrix(W, H * z["vdim"])
            t[p + "mlp.up"], t[p + "mlp.down"] = d.matrix(z["ff"], W), d.matrix(W, z["ff"], std=0.01)
            t[p + "mlp.act"] = torch.tensor([0.3, 0.2], device="cuda").to(d.dtype)
        t["final.norm"] = d.vector(W, mean=0.0)
    return t


def _tokens(case, seed):
    """Token ids: a history of `ctx` tokens per sequence, the new tokens, and the tokens of the decode steps after them."""
    r = np.random.RandomState(seed % (1 << 31))
    vocab = _vocab(case)
    ctx = _lengths(case, case["ctx"]) if case["ctx"] else [0] * case["batch"]
    return ([r.randint(0, vocab, n).tolist() for n in ctx], [r.randint(0, vocab, n).tolist() for n in _new_tokens(case)],
            [r.randint(0, vocab, case["batch"]).tolist() for _ in range(REQUEST_STEPS)])


def _vocab(case):
    return case.get("vocab") or {"qwen3": QWEN, "sokirax": SOKIRAX, "gigopel": GIGOPEL}[case["model"]][case["shape"]]["vocab"]


# ------------------------------------------------------------------------------------------------------------- a pass
class State:
    """What a user's program holds: an engine with its weights, a context, open sequences, the next tokens."""


def prepare(case, seed):
    s = State()
    s.case = case
    if case["do"] == "sample":
        g = torch.Generator(device="cuda").manual_seed(seed + 5)
        s.logits = torch.randn((case["batch"], case["vocab"]), generator=g, device="cuda") * 2.0
        likely = torch.randint(0, case["vocab"], (case["batch"], 64), generator=g, device="cuda")   # a few ids stand out
        s.logits.scatter_(1, likely, 12.0 + 2.0 * torch.randn(likely.shape, generator=g, device="cuda"))
        s.sampler = gg.new_sampler(gg.SamplerConfig(temp=case["temp"], top_k=case["top_k"], top_p=case["top_p"], seed=seed))
        s.streams, s.steps = list(range(case["batch"])), [7 + 3 * i for i in range(case["batch"])]
        return s
    s.history, s.new, s.after = _tokens(case, seed)
    model = Model(config_from_dict(_config(case)).to_spec(), _weights(case, seed), dtype=case["dtype"], consume=True)
    room = sum(-(-(len(h) + len(n) + REQUEST_STEPS) // PAGE) * PAGE for h, n in zip(s.history, s.new))
    s.ctx = gg.Engine(model, gg.LoadOptions(dtype=case["dtype"], max_tokens=room + PAGE)).new_context()
    s.slots = []
    if case["do"] == "decode":
        s.slots = [s.ctx.cache.open() for _ in s.history]
        at = 0
        while at < len(s.slots):                       # the histories, a few thousand tokens a step
            upto = at + 1
            while upto < len(s.slots) and sum(len(h) for h in s.history[at:upto + 1]) <= 8192:
                upto += 1
            s.ctx.stepper.step([gg.StepEntry(q, h) for q, h in zip(s.slots[at:upto], s.history[at:upto])])
            at = upto
    return s


def run(s):
    do = s.case["do"]
    if do == "sample":
        return torch.tensor(s.sampler.sample(s.logits, s.streams, s.steps))
    cache, stepper = s.ctx.cache, s.ctx.stepper
    if do == "score":
        return s.ctx.forward_token_ids(s.new[0])
    if do == "decode":
        logits = stepper.step([gg.StepEntry(q, n, want=[len(n) - 1]) for q, n in zip(s.slots, s.new)])
        for q, h in zip(s.slots, s.history):           # back to the history, as when an answer is asked for again
            cache.truncate(q, len(h))
        return logits
    slots = [cache.open() for _ in s.new]
    logits = stepper.step([gg.StepEntry(q, n, want=[len(n) - 1]) for q, n in zip(slots, s.new)])
    if do == "requests":
        out = [logits.clone()]                         # a step's logits live until the next step
        for ids in s.after:
            out.append(stepper.step([gg.StepEntry(q, [i], want=[0]) for q, i in zip(slots, ids)]).clone())
        logits = out
    for q in slots:
        cache.close(q)
    return logits


# --------------------------------------------------------------------------------------------------------------- work
def work(case):
    """Every weight that the pass uses and every cached row that it reads, once; the logits written."""
    if case["do"] == "sample":
        n = case["batch"] * case["vocab"]
        return {"bytes": 4.0 * n, "flops": 2.0 * n}
    item = 4 if case["dtype"] == "float32" else 2
    ctx = _lengths(case, case["ctx"]) if case["ctx"] else [0] * case["batch"]
    passes = [list(zip(ctx, _new_tokens(case)))]
    if case["do"] == "requests":
        for k in range(REQUEST_STEPS):
            passes.append([(n + k, 1) for _, n in passes[0]])
    total_b = total_f = 0.0
    for seqs in passes:
        T = sum(n for _, n in seqs)
        keys = lambda win: sum(sum(min(c + i + 1, win) for i in range(n)) for c, n in seqs)          # noqa: E731
        rows = lambda win: sum(min(c, win) + n for c, n in seqs)                                      # noqa: E731
        mats, extra_w, attn, cache = 0, 0, 0.0, 0.0
        L = case["layers"]
        if case["model"] == "qwen3":
            z = QWEN[case["shape"]]
            W, q, kv = z["hidden"], z["heads"] * z["dim"], z["kv"] * z["dim"]
            mats = L * (2 * q * W + 2 * kv * W + 3 * W * z["inter"])
            attn = L * 4.0 * q * keys(1 << 30)
            cache = L * 2.0 * kv * rows(1 << 30) * item
        elif case["model"] == "sokirax":
            z = SOKIRAX[case["shape"]]
            W, H, G, win = z["width"], z["heads"], z["kv"], z["window"]
            a, b = (L + 1) // 2, L // 2
            mats = a * 128 * W * (2 * H + 2 * G) + b * (64 * W * (2 * H + 2 * G) + 5 * z["ret"] * 128 * W)
            one = 3 * W * z["ff"]
            mats += L * (z["top"] * one + 3 * W * z["shared"] + z["experts"] * W)
            extra_w = L * one * (min(z["experts"], T * z["top"]) - z["top"])
            attn = a * 4.0 * H * 128 * keys(win) + b * (4.0 * H * 64 * keys(win) + 4.0 * T * z["ret"] * 128 * 128)
            cache = 2.0 * G * rows(win) * (a * 128 + b * 64) * item + b * 2 * len(seqs) * z["ret"] * 128 * 128 * 4.0
        else:
            z = GIGOPEL[case["shape"]]
            W, H, R = z["width"], z["heads"], z["rank"]
            mats = L * (H * (z["dim"] + z["rot"]) * W + (R + z["rot"]) * W + H * (z["dim"] + z["vdim"]) * R + W * H * z["vdim"]
                        + 2 * W * z["ff"])
            attn = L * 2.0 * H * (z["dim"] + z["rot"] + z["vdim"]) * keys(z["window"])
            cache = L * (R + z["rot"]) * rows(z["window"]) * float(item)
        want = T if case["do"] == "score" else len(seqs)
        V = _vocab(case)
        total_f += 2.0 * T * mats + attn + 2.0 * want * V * W
        total_b += (mats + extra_w + V * W + T * W) * item + cache + 4.0 * want * V
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    if case["do"] == "sample":
        return "exact"
    # about four times what the passes are off `exact` (measured: 32-bit 6e-6, Sokirax 0.003, Gigopel 0.006, Qwen3 0.007 to 0.018)
    if case["dtype"] == "float32":
        return {"rel": 2.5e-5}
    return {"rel": {"sokirax": 0.012, "gigopel": 0.024, "qwen3": 0.03}[case["model"]], "max": 0.5}


# ------------------------------------------------------------------------------------------------- the same in 64 bits
def _unit(x, eps=1e-6):
    return x / torch.sqrt((x * x).mean(dim=-1, keepdim=True) + eps)


def _angles(n, dims, base):
    f = torch.tensor([base ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device="cuda")
    a = torch.arange(n, dtype=torch.float64, device="cuda")[:, None] * f
    return torch.cos(a)[:, None, :], torch.sin(a)[:, None, :]


def _turn_halves(v, dims, base):
    """Element i of the first `dims` turns with element i + dims/2."""
    c, s = _angles(v.shape[0], dims, base)
    h = dims // 2
    u, w = v[..., :h], v[..., h:dims]
    return torch.cat([u * c - w * s, w * c + u * s, v[..., dims:]], dim=-1)


def _turn_neighbours(v, dims, base):
    """Element 2i turns with element 2i + 1."""
    c, s = _angles(v.shape[0], dims, base)
    u, w = v[..., 0:dims:2], v[..., 1:dims:2]
    return torch.cat([torch.stack([u * c - w * s, w * c + u * s], dim=-1).flatten(-2), v[..., dims:]], dim=-1)


def _softmax_attention(q, k, v, scale, window=1 << 30, sink=None):
    """q [n, H, d], k [n, G, d], v [n, G, dv]: causal inside a window; the sink joins the denominator."""
    n, H, G = q.shape[0], q.shape[1], k.shape[1]
    out = torch.empty(n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    block = max(1, (1 << 27) // max(n, 1))
    for a in range(0, n, block):
        i = torch.arange(a, min(n, a + block), device=q.device)[:, None]
        j = torch.arange(n, device=q.device)[None, :]
        hide = (j > i) | (i - j >= window)
        for h in range(H):
            g = h // (H // G)
            s = ((q[a:a + block, h] @ k[:, g].T) * scale).masked_fill_(hide, float("-inf"))
            m = s.amax(dim=-1, keepdim=True)
            if sink is not None:
                m = torch.clamp(m, min=float(sink[h]))
            s = torch.exp(s - m)
            den = s.sum(dim=-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(sink[h] - m)
            out[a:a + block, h] = (s @ v[:, g]) / den
    return out


def _silu(x):
    return x * torch.sigmoid(x)


def _exact_qwen3(case, t, seqs):
    """The rows before the head, [tokens, hidden], of whole sequences."""
    z = QWEN[case["shape"]]
    W = lambda name: t[name].double()                                                                # noqa: E731
    D = z["dim"]
    ids = torch.tensor([i for s in seqs for i in s], device="cuda")
    x = t["model.embed_tokens.weight"][ids].double()
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        h = _unit(x) * W(p + "input_layernorm.weight")
        q = _unit((h @ W(p + "self_attn.q_proj.weight").T).view(-1, z["heads"], D)) * W(p + "self_attn.q_norm.weight")
        k = _unit((h @ W(p + "self_attn.k_proj.weight").T).view(-1, z["kv"], D)) * W(p + "self_attn.k_norm.weight")
        v = (h @ W(p + "self_attn.v_proj.weight").T).view(-1, z["kv"], D)
        o, at = [], 0
        for s in seqs:
            r = slice(at, at + len(s))
            o.append(_softmax_attention(_turn_halves(q[r], D, 1e6), _turn_halves(k[r], D, 1e6), v[r], D ** -0.5))
            at += len(s)
        x = x + torch.cat(o).flatten(1) @ W(p + "self_attn.o_proj.weight").T
        h = _unit(x) * W(p + "post_attention_layernorm.weight")
        x = x + (_silu(h @ W(p + "mlp.gate_proj.weight").T) * (h @ W(p + "mlp.up_proj.weight").T)) @ W(p + "mlp.down_proj.weight").T
    return _unit(x) * W("model.norm.weight"), t["model.embed_tokens.weight"] if z["tied"] else t["lm_head.weight"]


def _exact_sokirax(case, t, seqs):
    z, cfg = SOKIRAX[case["shape"]], _config(case)
    H, G, R = z["heads"], z["kv"], z["ret"]
    W = lambda name: t[name].double()                                                                # noqa: E731
    x = W("embed")[torch.tensor([i for s in seqs for i in s], device="cuda")]

    def split(f):
        out, at = [], 0
        for s in seqs:
            out.append(f(slice(at, at + len(s))))
            at += len(s)
        return torch.cat(out).flatten(1)

    def attention(h, p, m, whole, sink):
        d, dims, base = m["dim"], m["rot"]["dims"], m["rot"]["base"]
        q, k, v = h @ W(p + "q").T, h @ W(p + "k").T, (h @ W(p + "v").T).view(-1, G, d)
        if whole:
            q, k = (_unit(q) * W(p + "q.norm")).view(-1, H, d), (_unit(k) * W(p + "k.norm")).view(-1, G, d)
        else:
            q, k = _unit(q.view(-1, H, d)) * W(p + "q.norm"), _unit(k.view(-1, G, d)) * W(p + "k.norm")
        o = split(lambda r: _softmax_attention(_turn_halves(q[r], dims, base), _turn_halves(k[r], dims, base), v[r], m["scale"],
                                               m["mask"]["size"], W(p + "sink") if sink else None))
        return o @ W(p + "o").T

    def retention(h, p, m):
        dims, base = m["rot"]["dims"], m["rot"]["base"]
        q, k, v = ((h @ W(p + name).T).view(-1, R, 128) for name in ("q", "k", "v"))

        def one(r):
            n = r.stop - r.start
            a, b = _turn_halves(q[r], dims, base), _turn_halves(k[r], dims, base) * 128 ** -0.5
            gap = (torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None, :]).double()
            o = torch.empty(n, R, 128, dtype=torch.float64, device="cuda")
            for i in range(R):
                s = (a[:, i] @ b[:, i].T) * torch.where(gap >= 0, m["decay"][i] ** gap.clamp(min=0), 0.0)
                o[:, i] = s @ v[r][:, i]
            return _unit(o)

        return (split(one) * _silu(h @ W(p + "g").T)) @ W(p + "o").T

    def unit(h, p):
        return (_silu(h @ W(p + "gate").T) * (h @ W(p + "up").T)) @ W(p + "down").T

    for i, ld in enumerate(cfg["layers"]):
        p, m = f"l{i}.", ld["mixer"]
        h = _unit(x) * W(p + "norm1")
        if ld["type"] == "attention":
            y = attention(h, p + "mix.", m, False, False)
        else:
            y = m["left_scale"] * attention(h, p + "mix.left.", m["left"], True, True) \
                + m["right_scale"] * retention(h, p + "mix.right.", m["right"])
        x = x + _unit(y) * W(p + "norm1b")
        h = _unit(x) * W(p + "norm2")
        best = torch.topk(h @ W(p + "mlp.router").T, z["top"], dim=-1)
        share = torch.softmax(best.values, dim=-1)
        y = unit(h, p + "mlp.shared.")
        for e in range(z["experts"]):
            row, col = torch.nonzero(best.indices == e, as_tuple=True)
            if row.numel():
                y.index_add_(0, row, share[row, col][:, None] * unit(h[row], f"{p}mlp.e{e}."))
        x = x + _unit(y) * W(p + "norm2b")
    return _unit(x) * W("final.norm"), t["head"]


def _exact_gigopel(case, t, seqs):
    z = GIGOPEL[case["shape"]]
    H, d, r, dv, R = z["heads"], z["dim"], z["rot"], z["vdim"], z["rank"]
    W = lambda name: t[name].double()                                                                # noqa: E731
    x = t["embed"][torch.tensor([i for s in seqs for i in s], device="cuda")].double()
    for i in range(case["layers"]):
        p = f"l{i}."
        m = p + "mix."
        h = _unit(x) * (1.0 + W(p + "norm1"))
        q, kv = (h @ W(m + "q").T).view(-1, H, d + r), h @ W(m + "dkv").T
        c = _unit(kv[:, :R]) * W(m + "dkv.norm")
        k, v = (c @ W(m + "uk").T).view(-1, H, d), (c @ W(m + "uv").T).view(-1, H, dv)
        o, at = [], 0
        for s in seqs:
            n = slice(at, at + len(s))
            kr = _turn_neighbours(kv[n, None, R:], r, 500000.0).expand(-1, H, -1)
            qa = torch.cat([q[n][..., :d], _turn_neighbours(q[n][..., d:], r, 500000.0)], dim=-1)
            o.append(_softmax_attention(qa, torch.cat([k[n], kr], dim=-1), v[n], (d + r) ** -0.5, z["window"]))
            at += len(s)
        y = torch.cat(o).flatten(1) @ W(m + "o").T
        a = W(p + "mlp.act")
        ap, aq = torch.log1p(torch.exp(a[0])), 0.5 + torch.log1p(torch.exp(a[1]))
        u = h @ W(p + "mlp.up").T
        u = torch.where(u > 0, ap * u * u + 0.5 * u, aq * (torch.expm1(u) - u) + 0.5 * u)
        x = x + 0.5 * (y + u @ W(p + "mlp.down").T)
    return _unit(x) * (1.0 + W("final.norm")), t["embed"]


def exact(case, seed):
    if case["do"] == "sample":
        return None
    t = _weights(case, seed)
    history, new, after = _tokens(case, seed)
    if case["do"] == "requests":
        seqs = [n + [ids[b] for ids in after] for b, n in enumerate(new)]
    else:
        seqs = [h + n for h, n in zip(history, new)]
    rows, head = {"qwen3": _exact_qwen3, "sokirax": _exact_sokirax, "gigopel": _exact_gigopel}[case["model"]](case, t, seqs)
    ends = np.cumsum([len(s) for s in seqs]) - 1
    if case["do"] == "score":
        return rows @ head.double().T
    if case["do"] != "requests":
        return rows[torch.as_tensor(ends, device="cuda")] @ head.double().T
    return [rows[torch.as_tensor(ends - REQUEST_STEPS + k, device="cuda")] @ head.double().T for k in range(REQUEST_STEPS + 1)]
