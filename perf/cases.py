"""What a user of this library waits for, as cases that can be timed and checked.

Every case is one or several steps of an ``Engine`` over a model with random weights, through the calls that a
session, the trace replay and the benchmark make: slots, ``step`` with prompts, ``step`` with one token per sequence.
A case says how many sequences there are, how much of each the cache holds already (``held``), how many tokens each
brings in a first step (``new``) and how many decode steps follow (``decode``).  Token ids come from the host every
step, the float32 logits of every step are the outputs (a copy of each, as a caller that samples later keeps them).

The models are the benchmark's: Qwen3 layers of three widths, and three of the other designs (recurrent layers, latent
attention, routed experts), with the benchmark's layer sizes and layer orders, eight layer runs each.  Weights have the
scales of an initialised model (matrices N(0, 0.02), those that write into the residual stream smaller by the root of
twice the depth, token vectors N(0, 1)).  Routers tell the tokens' experts apart as clearly as trained ones do: a
token's vector leans towards two experts of every routed layer, so that a choice does not hang on the last bit.

``exact`` states the same models in float64 torch, whole sequences at once, without this library.
"""
from __future__ import annotations

import math
import zlib

import torch

# Layer sizes by width, as in the benchmark (Qwen3-8B is the width of 4096, Qwen3-14B the one of 5120).
SIZES = {
    2048: dict(heads=16, kv=4, inter=6144, vocab=32768, gla_heads=8, rank=32, rec=16, q_rank=768),
    4096: dict(heads=32, kv=8, inter=12288, vocab=65536, gla_heads=16, rank=64, rec=32, q_rank=1536),
    5120: dict(heads=40, kv=8, inter=17408, vocab=65536),
}
DIM = 128               # lanes of an attention head, of a recurrent head's keys, and of a latent layer's values
GLA_VDIM = 256
TAPS = 4                # of the delta rule's short convolutions
EXPERTS, TOP = 16, 2
LAYERS = 8              # layer runs of every model
EPS = 1e-6
LEAN = 8.0              # how far a token's vector leans towards its experts, in standard deviations of a router logit
STEP_TOKENS = 8192      # the most tokens a preparing step brings


def listed():
    return [
        # a chat message of a few words after a short conversation with a small model: launches and latency
        dict(name="turn-24", design="qwen3", width=2048, dtype="bfloat16", seqs=1, held=700, new=24, decode=0),
        # a pasted paragraph, or a tool's answer, in a conversation with an 8B-sized model
        dict(name="turn-200", design="qwen3", width=4096, dtype="bfloat16", seqs=1, held=1500, new=200, decode=0),
        # a reply to one user, token by token
        dict(name="decode-1", design="qwen3", width=4096, dtype="bfloat16", seqs=1, held=2500, new=0, decode=8),
        # the benchmark's headline: eight sequences decoded together in the middle of a 4 096-token context
        dict(name="decode-8", design="qwen3", width=4096, dtype="bfloat16", seqs=8, held=3072, new=0, decode=8),
        # a full server: many shorter conversations at once
        dict(name="decode-64", design="qwen3", width=4096, dtype="bfloat16", seqs=64, held=1000, new=0, decode=4),
        # the benchmark's prompt
        dict(name="prompt-2048", design="qwen3", width=4096, dtype="bfloat16", seqs=1, held=0, new=2048, decode=0),
        # a batch of documents of unequal lengths with 14B-sized layers, one step for all
        dict(name="prompts-16", design="qwen3", width=5120, dtype="bfloat16", seqs=16, held=0, new=1090, decode=0),
        # a request in true 32-bit, the precision that results are checked in: its prompt, and its reply
        dict(name="float32-prompt", design="qwen3", width=2048, dtype="float32", seqs=1, held=0, new=300, decode=0),
        dict(name="float32-decode", design="qwen3", width=2048, dtype="float32", seqs=2, held=600, new=0, decode=4),
        # whole requests of the other designs: recurrent layers with windowed attention beside them,
        dict(name="romepel-request", design="romepel", width=2048, dtype="bfloat16", seqs=1, held=0, new=2048, decode=16),
        # the delta rule with latent attention,
        dict(name="pikalorn-requests", design="pikalorn", width=4096, dtype="bfloat16", seqs=4, held=0, new=700, decode=8),
        # and routed experts in a loop of layers
        dict(name="zevivik-requests", design="zevivik", width=2048, dtype="bfloat16", seqs=8, held=0, new=250, decode=8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["turn", "turn", "decode", "decode", "decode", "prompt", "prompt", "float32", "float32",
                       "romepel", "pikalorn", "zevivik"])
    c = dict(design="qwen3", width=rng.choice([2048, 4096]), dtype="bfloat16", seqs=1, held=0, new=0, decode=0)
    if kind == "turn":
        c.update(held=_log(rng, 50, 4000), new=_log(rng, 2, 256))
    elif kind == "decode":
        c.update(width=rng.choice([2048, 4096, 5120]), seqs=_log(rng, 1, 64), decode=rng.randint(3, 8))
        c.update(held=_log(rng, 50, min(8000, 64000 // c["seqs"])))
    elif kind == "prompt":
        c.update(width=rng.choice([2048, 4096, 5120]), seqs=_log(rng, 1, 16))
        c.update(new=_log(rng, 60, min(8192, 16000 // c["seqs"])))
    elif kind == "float32":
        c.update(width=2048, dtype="float32")
        if rng.random() < 0.5:
            c.update(new=_log(rng, 8, 600))
        else:
            c.update(seqs=_log(rng, 1, 16), held=_log(rng, 50, 1000), decode=rng.randint(2, 5))
    else:
        c.update(design=kind, seqs=_log(rng, 1, 8), decode=rng.randint(4, 16))
        c.update(new=_log(rng, 60, min(2048, 4000 // c["seqs"])))
    return c


def lengths(total, seqs):
    """Lengths of ``seqs`` sequences around ``total``: unequal (from an eighth to fifteen eighths of it), in a mixed
    order; a single sequence has exactly ``total``."""
    if total == 0 or seqs == 1:
        return [total] * seqs
    spread = [total / 8 + (total * 14 / 8) * i / (seqs - 1) for i in range(seqs)]
    step = next(s for s in (7, 5, 3, 1) if math.gcd(s, seqs) == 1)
    return [max(1, int(spread[i * step % seqs])) for i in range(seqs)]


# -- the models: configuration and weights -----------------------------------------------------------------------

def configuration(case):
    z, w, name = SIZES[case["width"]], case["width"], case["design"]
    att = dict(heads=z["heads"], kv_heads=z["kv"], dim=DIM, vdim=DIM, scale=DIM ** -0.5)
    rot = dict(base=1000000.0, dims=DIM)
    dense = dict(kind="dense", ff=z["inter"])
    if name == "qwen3":
        return dict(architectures=["Qwen3ForCausalLM"], num_hidden_layers=LAYERS, hidden_size=w, num_attention_heads=z["heads"],
                    num_key_value_heads=z["kv"], head_dim=DIM, intermediate_size=z["inter"], vocab_size=z["vocab"],
                    rope_theta=1000000.0, rms_norm_eps=EPS, tie_word_embeddings=False, attention_bias=False,
                    max_position_embeddings=40960)
    if name == "romepel":
        ff = dict(kind="dense", ff=z["inter"] * 3 // 2)
        attn = dict(type="attention", mlp=ff, mixer=dict(att, mask=dict(size=w // 4), q_temp=dict(coef=0.25, every=256)))
        gla = dict(type="gla", mlp=ff, mixer=dict(heads=z["gla_heads"], dim=DIM, vdim=GLA_VDIM, tau=8.0, rank=z["rank"]))
        return dict(architecture="Romepel", vocab=z["vocab"], width=w, max_positions=4096, norm=dict(eps=EPS), logit_softcap=30.0,
                    layers=[gla if i % 3 == 0 else attn for i in range(LAYERS)])
    if name == "pikalorn":
        lrot = dict(base=10000.0, dims=64, scaling=dict(factor=8.0, original=1024, fast=32.0, slow=1.0))
        lat = dict(heads=z["heads"], dim=64, rot_dim=64, vdim=DIM, kv_rank=64, q_rank=z["q_rank"], scale=128 ** -0.5, rot=lrot)
        delta = dict(heads=z["rec"], kv_heads=z["rec"] // 2, dim=DIM, vdim=DIM, conv=TAPS)
        layers = []
        for i in range(0, LAYERS, 4):
            layers += [dict(type="attention", mlp=dense, mixer=dict(att, rot=rot)),
                       dict(type="latent_attention", mlp=dense, mixer=lat),
                       dict(type="delta", mlp=dense, mixer=delta),
                       dict(type="latent_attention", mlp=dense, mixer=dict(lat, kv_from=i + 1))]
        return dict(architecture="Pikalorn", vocab=z["vocab"], width=w, norm=dict(eps=EPS), embedding=dict(scale=1.0), layers=layers)
    if name == "zevivik":
        moe = dict(kind="moe", expert=dict(ff=z["inter"] // 4, limit=7.0), router=dict(experts=EXPERTS, top=TOP),
                   shared=dict(ff=z["inter"] // 2, limit=7.0))
        block = dict(att, mask=dict(size=1024), rot=rot)
        lat = dict(heads=16, dim=DIM, vdim=w // 16, kv_rank=DIM, scale=DIM ** -0.5)

        def layer(kind, mixer, mlp):
            return dict(type=kind, mixer=mixer, mlp=mlp)
        return dict(architecture="Zevivik", vocab=z["vocab"], width=w, norm=dict(eps=EPS), embedding=dict(scale=1.0),
                    loop=dict(start=1, stop=3, times=2),
                    layers=[layer("attention", block, dense), layer("attention", block, moe), layer("latent_attention", lat, moe),
                            layer("attention", block, moe), layer("latent_attention", lat, dense), layer("attention", block, dense)])
    raise ValueError(name)


def shapes(case):
    """name -> (shape, mean, standard deviation) of every tensor."""
    cfg, w, out = configuration(case), case["width"], {}
    into_stream = 0.02 / math.sqrt(2 * LAYERS)

    def matrix(name, rows, cols, std=0.02):
        out[name] = ((rows, cols), 0.0, std)

    def vector(name, n, mean=0.0, std=0.1):
        out[name] = ((n,), mean, std)

    if case["design"] == "qwen3":
        v, inter = cfg["vocab_size"], cfg["intermediate_size"]
        q, kv = cfg["num_attention_heads"] * DIM, cfg["num_key_value_heads"] * DIM
        matrix("model.embed_tokens.weight", v, w, 1.0)
        for i in range(LAYERS):
            p = f"model.layers.{i}."
            vector(p + "input_layernorm.weight", w, 1.0)
            vector(p + "post_attention_layernorm.weight", w, 1.0)
            vector(p + "self_attn.q_norm.weight", DIM, 1.0)
            vector(p + "self_attn.k_norm.weight", DIM, 1.0)
            matrix(p + "self_attn.q_proj.weight", q, w)
            matrix(p + "self_attn.k_proj.weight", kv, w)
            matrix(p + "self_attn.v_proj.weight", kv, w)
            matrix(p + "self_attn.o_proj.weight", w, q, into_stream)
            matrix(p + "mlp.gate_proj.weight", inter, w)
            matrix(p + "mlp.up_proj.weight", inter, w)
            matrix(p + "mlp.down_proj.weight", w, inter, into_stream)
        vector("model.norm.weight", w, 1.0)
        matrix("lm_head.weight", v, w)
        return out
    norm_mean = 0.0 if case["design"] == "romepel" else 1.0        # its norms' weights are stored around zero
    matrix("embed", cfg["vocab"], w, 1.0)
    if case["design"] == "romepel":
        matrix("pos", cfg["max_positions"], w, 0.1)
    if "loop" in cfg:
        matrix("loop.step", cfg["loop"]["times"], w, 0.1)

    def gated(p, ff):
        matrix(p + ".gate", ff, w)
        matrix(p + ".up", ff, w)
        matrix(p + ".down", w, ff, into_stream)

    for i, layer in enumerate(cfg["layers"]):
        m, mlp, p = layer["mixer"], layer["mlp"], f"l{i}.mix"
        vector(f"l{i}.norm1", w, norm_mean)
        if case["design"] == "romepel":
            for n in ("norm1b", "norm2", "norm2b"):
                vector(f"l{i}.{n}", w, 0.0)
        elif case["design"] == "zevivik":
            vector(f"l{i}.norm2", w, 1.0)
        H = m["heads"]
        if layer["type"] == "attention":
            q, kv = H * DIM, m["kv_heads"] * DIM
            for n, rows in (("q", q), ("k", kv)) + ((("v", kv),) if case["design"] != "pikalorn" else ()):
                matrix(f"{p}.{n}", rows, w)
                if case["design"] != "zevivik":
                    vector(f"{p}.{n}.b", rows, 0.0, 0.02)
            matrix(f"{p}.o", w, q, into_stream)
            if case["design"] == "pikalorn":
                vector(f"{p}.o.b", w, 0.0, 0.02)
                vector(f"{p}.q.norm", DIM, 1.0)
                vector(f"{p}.k.norm", DIM, 1.0)
                vector(f"{p}.sink", H, 0.0, 1.0)
                matrix(f"{p}.g", q, w)
        elif layer["type"] == "latent_attention":
            q = H * (m["dim"] + m.get("rot_dim", 0))
            if "q_rank" in m:
                matrix(f"{p}.dq", m["q_rank"], w)
                vector(f"{p}.dq.norm", m["q_rank"], 1.0)
                matrix(f"{p}.uq", q, m["q_rank"], 0.05)
                vector(f"{p}.sink", H, 0.0, 1.0)
            else:
                matrix(f"{p}.q", q, w)
                matrix(f"{p}.g", H, w, 0.05)
            if "kv_from" not in m:
                matrix(f"{p}.dkv", m["kv_rank"] + m.get("rot_dim", 0), w)
                vector(f"{p}.dkv.norm", m["kv_rank"], 1.0)
            matrix(f"{p}.uk", H * m["dim"], m["kv_rank"], 0.05)
            matrix(f"{p}.uv", H * m["vdim"], m["kv_rank"], 0.05)
            matrix(f"{p}.o", w, H * m["vdim"], into_stream)
        elif layer["type"] == "gla":
            for n, rows in (("q", H * DIM), ("k", H * DIM), ("v", H * GLA_VDIM), ("g", H * GLA_VDIM)):
                matrix(f"{p}.{n}", rows, w)
            matrix(f"{p}.o", w, H * GLA_VDIM, into_stream)
            vector(f"{p}.norm", GLA_VDIM, 1.0)
            matrix(f"{p}.a1", m["rank"], w)
            matrix(f"{p}.a2", H * DIM, m["rank"], 0.2)
            vector(f"{p}.a2.b", H * DIM, 0.0, 1.0)
        else:
            qk = m["kv_heads"] * DIM
            for n, rows in (("q", qk), ("k", qk), ("v", H * DIM)):
                matrix(f"{p}.{n}", rows, w)
                matrix(f"{p}.{n}.conv", rows, TAPS, 0.5)
            matrix(f"{p}.b", H, w)
            matrix(f"{p}.a", H, w)
            vector(f"{p}.A_log", H, 0.0, 0.5)
            vector(f"{p}.dt_bias", H, 0.0, 0.5)
            matrix(f"{p}.g", H * DIM, w)
            vector(f"{p}.norm", DIM, 1.0)
            matrix(f"{p}.o", w, H * DIM, into_stream)
        p = f"l{i}.mlp"
        if case["design"] == "romepel":
            matrix(f"{p}.up", mlp["ff"], w)
            vector(f"{p}.up.b", mlp["ff"], 0.0, 0.02)
            matrix(f"{p}.down", w, mlp["ff"], into_stream)
            vector(f"{p}.down.b", w, 0.0, 0.02)
            vector(f"{p}.act", 2, 0.0, 0.5)
        elif mlp["kind"] == "dense":
            gated(p, mlp["ff"])
        else:
            matrix(f"{p}.router", EXPERTS, w)
            vector(f"{p}.router.b", EXPERTS, 0.0, 0.1)
            for e in range(EXPERTS):
                gated(f"{p}.e{e}", mlp["expert"]["ff"])
            gated(f"{p}.shared", mlp["shared"]["ff"])
    vector("final.norm", w, norm_mean)
    matrix("head", cfg["vocab"], w)
    return out


def weights(case, seed):
    """The model's tensors on the GPU, in the case's element type, from the seed alone."""
    dt = torch.float32 if case["dtype"] == "float32" else torch.bfloat16
    gen, out = torch.Generator(device="cuda"), {}
    for name, (shape, mean, std) in shapes(case).items():
        gen.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
        out[name] = torch.empty(shape, dtype=dt, device="cuda").normal_(mean, std, generator=gen)
    routers = [n for n in out if n.endswith(".router")]
    if routers:
        token = torch.arange(out["embed"].shape[0], device="cuda")
        for i, name in enumerate(routers):
            r = out[name].float()
            r = r / r.norm(dim=1, keepdim=True)
            first = (token * 40503 + i * 7919 >> 4) % EXPERTS
            second = (first + 1 + (token * 2971 + i * 104729 >> 3) % (EXPERTS - 1)) % EXPERTS
            out["embed"] += (LEAN * (r[first] + r[second])).to(dt)
    return out


# -- inputs, the pass, its outputs ----------------------------------------------------------------------------------

def tokens(case, seed):
    """Per sequence: the tokens held, the first step's, and the decode steps'."""
    vocab, gen = SIZES[case["width"]]["vocab"], torch.Generator().manual_seed(seed)

    def ids(n):
        return torch.randint(0, vocab, (n,), generator=gen).tolist()
    held, new = lengths(case["held"], case["seqs"]), lengths(case["new"], case["seqs"])
    return [(ids(h), ids(n), ids(case["decode"])) for h, n in zip(held, new)]


def prepare(case, seed):
    from nncpu_b200 import Engine, Model
    from nncpu_b200.config import config_from_dict
    from nncpu_b200.parts import Runtime
    toks = tokens(case, seed)
    longest = max(len(h) + len(n) + len(d) for h, n, d in toks)
    room = sum((len(h) + len(n) + len(d) + 63) // 64 * 64 for h, n, d in toks)
    runtime = Runtime("cuda:0", torch.float32 if case["dtype"] == "float32" else torch.bfloat16)
    model = Model(config_from_dict(configuration(case)), weights(case, seed), runtime)
    engine = Engine(model, max_tokens=room, n_slots=case["seqs"], max_seq_len=longest,
                    max_step_tokens=min(room, max(STEP_TOKENS, sum(len(n) for _, n, _ in toks))))
    state = dict(engine=engine, case=case, prompts=[n for _, n, _ in toks],
                 steps=[[[d[i]] for _, _, d in toks] for i in range(case["decode"])], slots=None,
                 held=[len(h) for h, _, _ in toks])
    if case["held"]:
        state["slots"] = [engine.alloc_slot() for _ in toks]
        waiting = [(s, h[at:at + STEP_TOKENS]) for s, (h, _, _) in zip(state["slots"], toks)
                   for at in range(0, len(h), STEP_TOKENS)]
        while waiting:          # as many sequences in a step as its tokens allow, a sequence's portions in order
            part, count = [], 0
            while waiting and count + len(waiting[0][1]) <= STEP_TOKENS and waiting[0][0] not in [s for s, _ in part]:
                part.append(waiting.pop(0))
                count += len(part[-1][1])
            engine.step([s for s, _ in part], [t for _, t in part])
    run(state)                  # the engine has served a batch of this size before: its steps are captured
    return state


def run(state):
    engine, case = state["engine"], state["case"]
    if state["slots"] is None:
        slots = [engine.alloc_slot() for _ in range(case["seqs"])]
    else:
        slots = state["slots"]
        for s, n in zip(slots, state["held"]):
            engine.cache.truncate(s, n)
    out = {}
    if case["new"]:
        out["prompt"] = engine.step(slots, state["prompts"]).clone()
    if case["decode"]:
        rows = torch.empty((case["decode"], case["seqs"], engine.vocab_size), dtype=torch.float32, device="cuda")
        for i, step in enumerate(state["steps"]):
            rows[i].copy_(engine.step(slots, step))
        out["decode"] = rows
    if state["slots"] is None:
        for s in slots:
            engine.free_slot(s)
    return out


def work(case):
    size = 4 if case["dtype"] == "float32" else 2
    cfg, z, sh = configuration(case), SIZES[case["width"]], shapes(case)
    layers = cfg.get("layers")
    runs = [layers[i] for i in (0, 1, 2, 1, 2, 3, 4, 5)] if "loop" in cfg else layers
    times = {i: (2 if "loop" in cfg and 1 <= i < 3 else 1) for i in range(LAYERS)}
    # weights by the number of times a step runs them: always read, and per expert
    fixed = expert = head = 0
    for name, (shape, _, _) in sh.items():
        n = math.prod(shape)
        if name in ("head", "lm_head.weight"):
            head = n
        elif name not in ("embed", "pos", "model.embed_tokens.weight"):
            layer = int(name.split(".")[0][1:]) if layers and name.startswith("l") and name[1].isdigit() else None
            times_run = times[layer] if layer is not None else 1
            if ".mlp.e" in name:
                expert += n * times_run
            else:
                fixed += n * times_run
    # numbers kept per token (keys, values, latents), multiply-adds per key that a token sees, and recurrent states
    kept = mac = state = 0
    for layer in runs or [dict(type="attention", mixer=dict(heads=z["heads"], kv_heads=z["kv"]))] * LAYERS:
        m, kind = layer["mixer"], layer["type"]
        if kind == "attention":
            kept += 2 * m["kv_heads"] * DIM
            mac += 2 * m["heads"] * DIM
        elif kind == "latent_attention":
            kept += 0 if "kv_from" in m else m["kv_rank"] + m.get("rot_dim", 0)
            mac += m["heads"] * (m["dim"] + m.get("rot_dim", 0) + m["vdim"])
        else:
            state += m["heads"] * DIM * (GLA_VDIM if kind == "gla" else DIM)
    window = {"romepel": case["width"] // 4, "zevivik": 1024}.get(case["design"])

    def seen(p):
        return min(p + 1, window) if window else p + 1

    held, new = lengths(case["held"], case["seqs"]), lengths(case["new"], case["seqs"])
    nbytes = flops = 0.0

    def step(starts, counts):
        nonlocal nbytes, flops
        n = sum(counts)
        touched = EXPERTS * (1 - (1 - TOP / EXPERTS) ** n)
        nbytes += size * (fixed + head + expert / EXPERTS * touched)
        nbytes += size * kept * (sum(min(s, window) if window else s for s in starts) + n)      # keys read, keys written
        nbytes += 8 * state * len(starts) + 4 * n + 4 * len(starts) * z["vocab"]
        flops += 2.0 * n * (fixed + expert / EXPERTS * TOP) + 2.0 * len(starts) * head
        flops += 2.0 * mac * sum(sum(seen(s + i) for i in range(c)) for s, c in zip(starts, counts)) + 6.0 * state * n

    if case["new"]:
        step(held, new)
    for i in range(case["decode"]):
        step([h + n + i for h, n in zip(held, new)], [1] * case["seqs"])
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    return {"rel": 1e-5, "max": 1e-4} if case["dtype"] == "float32" else {"rel": 0.02, "max": 0.3}


# -- the same in float64 -----------------------------------------------------------------------------------------------

def _mm(x, w):
    return x @ w.double().T


def _rms(x, w, offset=0.0):
    x = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    return x if w is None else x * (w.double() + offset)


def _rotate(x, pos, base, dims, scaling=None, neighbours=False):
    """x [T, heads, lanes]: the first ``dims`` lanes turn, pairs (i, i + dims / 2) or neighbouring lanes."""
    i = torch.arange(dims // 2, dtype=torch.float64, device=x.device)
    f, stretch = base ** (-2.0 * i / dims), 1.0
    if scaling is not None:
        def lane(turns):
            return dims * math.log(scaling["original"] / (2 * math.pi * turns)) / (2 * math.log(base))
        lo, hi = max(math.floor(lane(scaling["fast"])), 0), min(math.ceil(lane(scaling["slow"])), dims - 1)
        ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
        f = f / scaling["factor"] * ramp + f * (1 - ramp)
        stretch = 0.1 * math.log(scaling["factor"]) + 1.0
    a = pos.double()[:, None, None] * f
    c, s = a.cos() * stretch, a.sin() * stretch
    out = x.clone()
    u, v = (x[..., 0:dims:2], x[..., 1:dims:2]) if neighbours else (x[..., :dims // 2], x[..., dims // 2:dims])
    if neighbours:
        out[..., 0:dims:2], out[..., 1:dims:2] = u * c - v * s, v * c + u * s
    else:
        out[..., :dims // 2], out[..., dims // 2:dims] = u * c - v * s, v * c + u * s
    return out


def _attend(q, k, v, scale, window=0, block=0, slopes=None, sink=None):
    """Causal attention of one sequence, q [T, H, d] over k [T, G, d], v [T, G, e]; [T, H * e]."""
    T, H, _ = q.shape
    G, out = k.shape[1], torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    t = torch.arange(T, device=q.device)
    away = t[:, None] - t[None, :]
    unseen = away < 0
    if window:
        unseen |= away >= window
    if block:
        unseen |= (t[:, None] // block) != (t[None, :] // block)
    for h in range(H):
        g = h // (H // G)
        s = (q[:, h] @ k[:, g].T) * scale
        if slopes is not None:
            s -= slopes[h] * away
        s.masked_fill_(unseen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].double().expand(T, 1)], dim=1)
        p = s.softmax(-1)
        out[:, h] = p[:, :T] @ v[:, g]
    return out.reshape(T, -1)


def _gla(q, k, v, alpha):
    T, H, d = q.shape
    S = torch.zeros(H, d, v.shape[2], dtype=torch.float64, device=q.device)
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    for t in range(T):
        S = S * alpha[t][:, :, None] + k[t][:, :, None] * v[t][:, None, :]
        out[t] = torch.einsum("hde,hd->he", S, q[t])
    return out


def _delta(q, k, v, g, b):
    T, H, d = q.shape
    S = torch.zeros(H, d, v.shape[2], dtype=torch.float64, device=q.device)
    out = torch.empty(T, H, v.shape[2], dtype=torch.float64, device=q.device)
    for t in range(T):
        S = S * g[t][:, None, None]
        u = b[t][:, None] * (v[t] - torch.einsum("hde,hd->he", S, k[t]))
        S = S + k[t][:, :, None] * u[:, None, :]
        out[t] = torch.einsum("hde,hd->he", S, q[t])
    return out


def _conv(x, taps):
    taps = taps.double()
    pad = torch.cat([x.new_zeros(TAPS - 1, x.shape[1]), x])
    return torch.nn.functional.silu(sum(pad[j:j + x.shape[0]] * taps[:, j] for j in range(TAPS)))


def _swish_clamp(g, u, limit):
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(1.702 * g) * (u + 1.0)


def _gated(h, w, p, act):
    return _mm(act(_mm(h, w[p + "gate"]), _mm(h, w[p + "up"])), w[p + "down"])


def _silu_gate(g, u):
    return torch.nn.functional.silu(g) * u


def _gelu_gate(g, u):
    return torch.nn.functional.gelu(g, approximate="tanh") * u


def _experts(h, w, p, mlp):
    def act(g, u):
        return _swish_clamp(g, u, mlp["expert"]["limit"])
    z, ids = (_mm(h, w[p + "router"]) + w[p + "router.b"].double()).topk(TOP, dim=-1)
    share, out = z.softmax(-1), _gated(h, w, p + "shared.", act)
    for e in range(EXPERTS):
        rows, slot = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            out[rows] += share[rows, slot][:, None] * _gated(h[rows], w, f"{p}e{e}.", act)
    return out


def _mixer(design, layer, h, w, p, pos, kept, i):
    """One sequence's rows through a mixer."""
    m, T = layer["mixer"], h.shape[0]
    H = m["heads"]
    if layer["type"] == "gla":
        z = _mm(_mm(h, w[p + "a1"]), w[p + "a2"]) + w[p + "a2.b"].double()
        alpha = (torch.nn.functional.logsigmoid(z) / m["tau"]).exp().view(T, H, DIM)
        o = _gla(_mm(h, w[p + "q"]).view(T, H, DIM) * DIM ** -0.5, _mm(h, w[p + "k"]).view(T, H, DIM),
                 _mm(h, w[p + "v"]).view(T, H, GLA_VDIM), alpha)
        o = _rms(o, w[p + "norm"]).reshape(T, -1) * torch.nn.functional.silu(_mm(h, w[p + "g"]))
        return _mm(o, w[p + "o"])
    if layer["type"] == "delta":
        G = m["kv_heads"]
        q, k = (_conv(_mm(h, w[p + n]), w[p + n + ".conv"]).view(T, G, DIM) for n in "qk")
        q, k = (x * torch.rsqrt(x.pow(2).sum(-1, keepdim=True) + 1e-6) for x in (q, k))
        q, k = (x.repeat_interleave(H // G, dim=1) for x in (q * DIM ** -0.5, k))
        v = _conv(_mm(h, w[p + "v"]), w[p + "v.conv"]).view(T, H, DIM)
        g = torch.exp(-w[p + "A_log"].double().exp() * torch.nn.functional.softplus(_mm(h, w[p + "a"]) + w[p + "dt_bias"].double()))
        o = _rms(_delta(q, k, v, g, torch.sigmoid(_mm(h, w[p + "b"]))), w[p + "norm"])
        o = o * torch.nn.functional.silu(_mm(h, w[p + "g"])).view(T, H, DIM)
        return _mm(o.reshape(T, -1), w[p + "o"])
    if layer["type"] == "latent_attention":
        d, R, e, rot = m["dim"], m.get("rot_dim", 0), m["vdim"], m.get("rot")
        if "kv_from" not in m:
            z = _mm(h, w[p + "dkv"])
            kr = _rotate(z[:, None, -R:], pos, rot["base"], R, rot["scaling"], True) if R else None
            kept[i] = (_rms(z[:, :m["kv_rank"]], w[p + "dkv.norm"]), kr)
        c, kr = kept[m.get("kv_from", i)]
        q = (_mm(_rms(_mm(h, w[p + "dq"]), w[p + "dq.norm"]), w[p + "uq"]) if "q_rank" in m else _mm(h, w[p + "q"])).view(T, H, d + R)
        k, v = _mm(c, w[p + "uk"]).view(T, H, d), _mm(c, w[p + "uv"]).view(T, H, e)
        if R:
            q = torch.cat([q[..., :d], _rotate(q[..., d:], pos, rot["base"], R, rot["scaling"], True)], dim=-1)
            k = torch.cat([k, kr.expand(T, H, R)], dim=-1)
        o = _attend(q, k, v, m["scale"], sink=w.get(p + "sink"))
        if "q_rank" not in m:
            o = (o.view(T, H, e) * torch.sigmoid(_mm(h, w[p + "g"]))[:, :, None]).reshape(T, -1)
        return _mm(o, w[p + "o"])
    G = m["kv_heads"]
    q, k = _mm(h, w[p + "q"]).view(T, H, DIM), _mm(h, w[p + "k"]).view(T, G, DIM)
    if design == "romepel":
        q, k = q + w[p + "q.b"].double().view(H, DIM), k + w[p + "k.b"].double().view(G, DIM)
        v = (_mm(h, w[p + "v"]) + w[p + "v.b"].double()).view(T, G, DIM)
        t = m["q_temp"]
        q = q * (1 + t["coef"] * torch.log(torch.floor((pos.double() + 1) / t["every"]) + 1))[:, None, None]
        slopes = [2.0 ** (-8.0 * (a + 1) / H) for a in range(H)]
        return _mm(_attend(q, k, v, m["scale"], window=m["mask"]["size"], slopes=slopes), w[p + "o"])
    rot = m["rot"]
    if design == "pikalorn":
        q, k = q + w[p + "q.b"].double().view(H, DIM), k + w[p + "k.b"].double().view(G, DIM)
        v, q, k = k, _rms(q, w[p + "q.norm"]), _rms(k, w[p + "k.norm"])
    else:
        v = _mm(h, w[p + "v"]).view(T, G, DIM)
    q, k = _rotate(q, pos, rot["base"], DIM), _rotate(k, pos, rot["base"], DIM)
    o = _attend(q, k, v, m["scale"], block=(m.get("mask") or {}).get("size", 0), sink=w.get(p + "sink"))
    if design == "pikalorn":
        return _mm(o * torch.sigmoid(_mm(h, w[p + "g"])), w[p + "o"]) + w[p + "o.b"].double()
    return _mm(o, w[p + "o"])


def _by_sequence(f, h, cuts):
    return torch.cat([f(h[a:b], torch.arange(b - a, device=h.device)) for a, b in cuts])


def _forward_qwen3(cfg, w, ids, cuts):
    H, G = cfg["num_attention_heads"], cfg["num_key_value_heads"]
    x = w["model.embed_tokens.weight"][ids].double()
    for i in range(LAYERS):
        p = f"model.layers.{i}."
        h = _rms(x, w[p + "input_layernorm.weight"])
        qkv = [_mm(h, w[p + f"self_attn.{n}_proj.weight"]) for n in "qkv"]

        def mix(rows, pos):
            q, k, v = (y.view(-1, n, DIM) for y, n in zip(rows.split([H * DIM, G * DIM, G * DIM], dim=1), (H, G, G)))
            q = _rotate(_rms(q, w[p + "self_attn.q_norm.weight"]), pos, cfg["rope_theta"], DIM)
            k = _rotate(_rms(k, w[p + "self_attn.k_norm.weight"]), pos, cfg["rope_theta"], DIM)
            return _attend(q, k, v, DIM ** -0.5)
        x = x + _mm(_by_sequence(mix, torch.cat(qkv, dim=1), cuts), w[p + "self_attn.o_proj.weight"])
        h = _rms(x, w[p + "post_attention_layernorm.weight"])
        x = x + _mm(_silu_gate(_mm(h, w[p + "mlp.gate_proj.weight"]), _mm(h, w[p + "mlp.up_proj.weight"])),
                    w[p + "mlp.down_proj.weight"])
    return x


def _forward_design(design, cfg, w, ids, cuts):
    offset = 1.0 if design == "romepel" else 0.0
    x0 = w["embed"][ids].double()
    if design == "romepel":
        x0 = x0 + torch.cat([w["pos"][:b - a] for a, b in cuts]).double()
    x, kept = x0, [dict() for _ in cuts]
    order = [(i, None) for i in range(len(cfg["layers"]))]
    if "loop" in cfg:
        order = [(0, None), (1, 0), (2, None), (1, 1), (2, None), (3, None), (4, None), (5, None)]
    for i, turn in order:
        layer = cfg["layers"][i]
        if turn is not None:
            x = x + (x0 if turn else 0.0) + w["loop.step"][turn].double()
        h = _rms(x, w[f"l{i}.norm1"], offset)
        y = torch.cat([_mixer(design, layer, h[a:b], w, f"l{i}.mix.", torch.arange(b - a, device=x.device), kept[s], i)
                       for s, (a, b) in enumerate(cuts)])
        p, mlp = f"l{i}.mlp.", layer["mlp"]
        if design == "romepel":
            x = x + _rms(y, w[f"l{i}.norm1b"], 1.0)
            z = _mm(_rms(x, w[f"l{i}.norm2"], 1.0), w[p + "up"]) + w[p + "up.b"].double()
            a, b = torch.nn.functional.softplus(w[p + "act"].double())
            z = torch.where(z > 0, a * z * z + 0.5 * z, (0.5 + b) * (torch.expm1(z.clamp(max=0)) - z) + 0.5 * z)
            x = x + _rms(_mm(z, w[p + "down"]) + w[p + "down.b"].double(), w[f"l{i}.norm2b"], 1.0)
        elif design == "pikalorn":
            x = x + y + _gated(h, w, p, _silu_gate)
        else:
            h = _rms(x, w[f"l{i}.norm2"])
            x = x + y + (_gated(h, w, p, _gelu_gate) if mlp["kind"] == "dense" else _experts(h, w, p, mlp))
    return x


@torch.no_grad()
def exact(case, seed):
    toks, w, cfg = tokens(case, seed), weights(case, seed), configuration(case)
    whole = [h + n + d for h, n, d in toks]
    ends, cuts = [], []
    for s in whole:
        cuts.append((ends[-1] if ends else 0, (ends[-1] if ends else 0) + len(s)))
        ends.append(cuts[-1][1])
    ids = torch.tensor([t for s in whole for t in s], device="cuda")
    design = case["design"]
    x = _forward_qwen3(cfg, w, ids, cuts) if design == "qwen3" else _forward_design(design, cfg, w, ids, cuts)
    norm, head = (w["model.norm.weight"], w["lm_head.weight"]) if design == "qwen3" else (w["final.norm"], w["head"])

    def logits(rows):
        y = _mm(_rms(x[rows], norm, 1.0 if design == "romepel" else 0.0), head)
        return 30.0 * torch.tanh(y / 30.0) if design == "romepel" else y
    out = {}
    if case["new"]:
        out["prompt"] = logits([b - case["decode"] - 1 for _, b in cuts])
    if case["decode"]:
        out["decode"] = torch.stack([logits([b - case["decode"] + i for _, b in cuts]) for i in range(case["decode"])])
    return out
