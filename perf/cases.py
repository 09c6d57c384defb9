"""The work that is timed: the framework's layers at the sizes of its designs, and a whole model.

A case names a layer, a phase and sizes.  "prompt": the rows of one or several new sequences go
through the layer in one step, eagerly, as the engine runs prompts.  "step": one row a sequence
after `context` earlier ones, replayed from a CUDA graph, as the engine runs decode steps.  Layers
are registered parts, built from their specs, bound to seeded weights and given a cache; the
widths are those of bench.py's designs and of the Qwen3 family (heads of 128, a quarter as many
key/value heads, and so on: `_sizes`).  "model" is a whole Qwen3 model through `Engine`: prompts
together, then decode steps, with the logits of all of them.
"""

import math

import torch

from reflex_b200.cache.store import Cache
from reflex_b200.config.spec import FeedForwardSpec, MixerSpec, NormSpec, PositionSpec
from reflex_b200.engine import Engine
from reflex_b200.engine.batch import make_batch
from reflex_b200.engine.model import RunContext
from reflex_b200.ops import workspace
from reflex_b200.parts.registry import FEED_FORWARDS, MIXERS
from reflex_b200.weights import random_model_on_device

DEVICE = "cuda:0"
EPS = 1e-6
WIDTHS = (1024, 1536, 2048, 2560, 3072, 4096)
VOCAB = 32768
STATE_ROWS = 16  # rows a sequence with fixed-size state has seen before a "step"


def listed():
    def case(name, layer, phase, width, seqs, rows, context=0, dtype="bf16", layers=1, steps=1):
        return dict(name=name, layer=layer, phase=phase, width=width, seqs=seqs, rows=rows, context=context,
                    dtype=dtype, layers=layers, steps=steps)

    return [
        # serving: eight requests of unequal length are prefilled together and decoded together
        case("generate", "model", "generate", 2048, 8, 4000, layers=4, steps=16),
        # one prompt of the benchmark's length through the attention layer of Qwen3-8B
        case("attention_prompt", "attention", "prompt", 4096, 1, 2048),
        # a full batch deep in its context: the step is the keys and values it reads
        case("attention_step_b64", "attention", "step", 4096, 64, 64, context=2048),
        # the feed-forward of Qwen3-8B at the headline's batch: weights streamed for eight rows
        case("swiglu_step_b8", "swiglu", "step", 4096, 8, 8),
        # the true 32-bit path on a few unequal prompts
        case("attention_prompts_f32", "attention", "prompt", 1024, 3, 701, dtype="f32"),
        # Kegasun's matrix memory over a prompt
        case("mlstm_prompt", "mlstm", "prompt", 2048, 1, 2048),
        # Zelinex's pair (sigmoid-weight attention beside a state-space recurrence) over a prompt
        case("pair_prompt", "pair", "prompt", 2048, 1, 2048),
        # Zelinex's delta rule over unequal prompts
        case("delta_prompts", "delta", "prompt", 2048, 4, 1999),
        # Zivulix's gated delta rule over a long prompt
        case("gated_delta_prompt", "gated_delta", "prompt", 2048, 1, 4096),
        # a single sequence decoding through Purusun's selective scan: the smallest call
        case("scan_step_b1", "scan", "step", 1024, 1, 1),
        # Pidodra's routed experts for a batch that decodes
        case("moe_step_b8", "moe", "step", 2048, 8, 8),
        # Pidodra's latent attention for a batch that decodes
        case("latent_step_b8", "latent", "step", 2048, 8, 8, context=4000),
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    layer = rng.choice(("model", "attention", "attention", "swiglu", "mlstm", "pair", "delta", "gated_delta", "scan",
                        "moe", "latent"))
    width = rng.choice(WIDTHS)
    dtype = "f32" if layer in ("attention", "swiglu") and rng.random() < 0.35 else "bf16"
    if layer == "model":
        seqs = spread(1, 12)
        return dict(layer=layer, phase="generate", width=rng.choice(WIDTHS[:3]), seqs=seqs,
                    rows=seqs * spread(16, 512) + rng.randrange(seqs), context=0, dtype="bf16",
                    layers=rng.randint(2, 4), steps=rng.randint(2, 16))
    if rng.random() < 0.6:
        rows = spread(17, 1024 if dtype == "f32" else 4096)
        return dict(layer=layer, phase="prompt", width=width, seqs=min(rows // 8, rng.choice((1, 1, 2, 3, 5, 8))),
                    rows=rows, context=0, dtype=dtype, layers=1, steps=1)
    seqs = spread(1, 64)
    context = spread(24, 4096) if layer in ("attention", "pair", "latent") else 0
    if dtype == "f32":
        seqs, context = min(seqs, 16), min(context, 1024)
    if context:
        context = min(context, 131072 // seqs)
    return dict(layer=layer, phase="step", width=width, seqs=seqs, rows=seqs, context=context, dtype=dtype, layers=1,
                steps=1)


# ---- sizes, specs and weights ---------------------------------------------------------------
def _sizes(c):
    W = c["width"]
    return dict(W=W, H=W // 128, KV=max(1, W // 512), d=128, ff=4 * W if W < 4096 else 3 * W, q_rank=3 * W // 8,
                kv_rank=256 if W > 1024 else 128, rot=64, mh=W // 256, mdv=256, sh=W // 64, N=128, G=2, taps=4,
                dh=W // 64, dd=64, rank=max(8, W // 16), gh=W // 64, gk=W // 128, gd=128, C=2 * W, NS=16, R=W // 16,
                E=16, top=4, eff=2048, window=1024)


def _spec(c):
    z = _sizes(c)
    W, d = z["W"], z["d"]
    layer = c["layer"]
    norm = NormSpec("rmsnorm", d, EPS)
    if layer == "attention":
        return MixerSpec("gqa_attention", W, z["H"], z["KV"], d, d ** -0.5, qk_norm=norm,
                         position=PositionSpec("rope_neox", d, d, 1e6))
    if layer == "latent":
        rd = z["rot"]
        return MixerSpec("latent_attention", W, z["H"], 1, d, (d + rd) ** -0.5, v_head_dim=d,
                         position=PositionSpec("rope_neox", rd, rd, 500000.0, params=(("pairing", "consecutive"),)),
                         params=(("q_rank", z["q_rank"]), ("kv_rank", z["kv_rank"]), ("rot_dim", rd), ("eps", EPS),
                                 ("sink", True), ("gate", "element")))
    if layer == "mlstm":
        return MixerSpec("mlstm", W, z["mh"], 0, d, d ** -0.5, v_head_dim=z["mdv"],
                         params=(("gate_cap", 15.0), ("eps", EPS)))
    if layer == "pair":
        left = MixerSpec("sigmoid_attention", W, z["H"], z["KV"], d, d ** -0.5, window=z["window"], v_head_dim=d,
                         position=PositionSpec("rope_neox", d, d // 2, 500000.0))
        right = MixerSpec("ssd", W, params=(("heads", z["sh"]), ("vdim", 64), ("state", z["N"]), ("groups", z["G"]),
                                            ("taps", z["taps"]), ("norm_groups", 2), ("eps", EPS)))
        return MixerSpec("pair", W, params=(("left", left), ("right", right), ("combine", "scaled_sum"),
                                            ("left_scale", 0.75), ("right_scale", 0.55)))
    if layer == "delta":
        return MixerSpec("delta_rule", W, z["dh"], 0, z["dd"],
                         params=(("rate", math.exp(-0.5)), ("unit_eps", 1e-6), ("eps", EPS)))
    if layer == "gated_delta":
        return MixerSpec("gated_delta", W, z["gh"], z["gk"], z["gd"], z["gd"] ** -0.5, v_head_dim=z["gd"],
                         params=(("taps", z["taps"]), ("unit_eps", 1e-6), ("eps", EPS)))
    if layer == "scan":
        return MixerSpec("selective_scan", W, params=(("inner", z["C"]), ("state", z["NS"]), ("dt_rank", z["R"]),
                                                      ("taps", z["taps"])))
    if layer == "swiglu":
        return FeedForwardSpec("swiglu", W, z["ff"])
    if layer == "moe":
        return FeedForwardSpec("moe", W, z["eff"], params=(
            ("experts", z["E"]), ("top", z["top"]), ("activation", "swiglu"), ("scores", "softmax"),
            ("score_scale", 1.5), ("groups", (4, 2))))
    raise ValueError(layer)


def _shapes(c):
    """role -> (shape, how it is drawn) of a layer's weights."""
    z = _sizes(c)
    W, H, KV, d = z["W"], z["H"], z["KV"], z["d"]
    m, n, b, f = "matrix", "norm", "bias", "filter"
    layer = c["layer"]
    if layer == "attention":
        return {"q_proj": ((H * d, W), m), "k_proj": ((KV * d, W), m), "v_proj": ((KV * d, W), m),
                "o_proj": ((W, H * d), m), "q_norm": ((d,), n), "k_norm": ((d,), n)}
    if layer == "latent":
        qr, kr, r = z["q_rank"], z["kv_rank"], z["rot"]
        return {"q_down": ((qr, W), m), "q_norm": ((qr,), n), "q_up": ((H * (d + r), qr), m),
                "kv_down": ((kr + r, W), m), "kv_norm": ((kr,), n), "k_up": ((H * d, kr), m), "v_up": ((H * d, kr), m),
                "o_proj": ((W, H * d), m), "sink": ((H,), b), "gate": ((H * d, W), m)}
    if layer == "mlstm":
        h, dv = z["mh"], z["mdv"]
        return {"q_proj": ((h * d, W), m), "k_proj": ((h * d, W), m), "v_proj": ((h * dv, W), m),
                "gate": ((h * dv, W), m), "o_proj": ((W, h * dv), m), "norm": ((h * dv,), n), "i_proj": ((h, W), m),
                "i_bias": ((h,), b), "f_proj": ((h, W), m), "f_bias": ((h,), b)}
    if layer == "pair":
        h, N, G, inner = z["sh"], z["N"], z["G"], z["sh"] * 64
        cc = inner + 2 * G * N
        return {"left/q_proj": ((H * d, W), m), "left/k_proj": ((KV * d, W), m), "left/v_proj": ((KV * d, W), m),
                "left/score_bias": ((H,), b), "left/o_proj": ((W, H * d), m),
                "right/in_proj": ((inner + cc + h, W), m), "right/conv": ((cc, z["taps"]), f),
                "right/conv_bias": ((cc,), b), "right/dt_bias": ((h,), b), "right/A_log": ((h,), b),
                "right/D": ((h,), b), "right/norm": ((inner,), n), "right/o_proj": ((W, inner), m)}
    if layer == "delta":
        hd = z["dh"] * z["dd"]
        out = {r: ((hd, W), m) for r in ("r_proj", "k_proj", "v_proj", "g_proj", "a_proj")}
        out.update({"a_bias": ((hd,), b), "w1_proj": ((z["rank"], W), m), "w2_proj": ((hd, z["rank"]), m),
                    "w0": ((hd,), b), "norm": ((hd,), n), "o_proj": ((W, hd), m)})
        return out
    if layer == "gated_delta":
        h, g, gd, t = z["gh"], z["gk"], z["gd"], z["taps"]
        return {"q_proj": ((g * gd, W), m), "k_proj": ((g * gd, W), m), "v_proj": ((h * gd, W), m),
                "g_proj": ((h * gd, W), m), "b_proj": ((h, W), m), "a_proj": ((h, W), m), "q_conv": ((g * gd, t), f),
                "k_conv": ((g * gd, t), f), "v_conv": ((h * gd, t), f), "A_log": ((h,), b), "dt_bias": ((h,), b),
                "norm": ((gd,), n), "o_proj": ((W, h * gd), m)}
    if layer == "scan":
        C, N, R = z["C"], z["NS"], z["R"]
        return {"in_proj": ((2 * C, W), m), "conv": ((C, z["taps"]), f), "conv_bias": ((C,), b),
                "x_proj": ((R + 2 * N, C), m), "dt_proj": ((C, R), m), "dt_bias": ((C,), b), "A_log": ((C, N), b),
                "D": ((C,), b), "o_proj": ((W, C), m)}
    if layer == "swiglu":
        return {"gate_proj": ((z["ff"], W), m), "up_proj": ((z["ff"], W), m), "down_proj": ((W, z["ff"]), m)}
    if layer == "moe":
        out = {"router": ((z["E"], W), m)}
        for e in range(z["E"]):
            out.update({f"expert_gate#{e}": ((z["eff"], W), m), f"expert_up#{e}": ((z["eff"], W), m),
                        f"expert_down#{e}": ((W, z["eff"]), m)})
        return out
    raise ValueError(layer)


def _dtype(c):
    return torch.float32 if c["dtype"] == "f32" else torch.bfloat16


def _weights(c, seed):
    """Seeded weights, distributed as the framework's random models are."""
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 1)
    out = {}
    for role, (shape, how) in _shapes(c).items():
        if how == "matrix":
            out[role] = torch.randn(shape, generator=g, device=DEVICE).mul_(0.02).to(_dtype(c))
        else:
            u = torch.rand(shape, generator=g, device=DEVICE)
            out[role] = {"norm": lambda: 0.9 + 0.2 * u, "bias": lambda: u - 0.5,
                         "filter": lambda: 1.2 * u - 0.6}[how]()
    return out


def _lengths(c):
    """(new rows, earlier rows) of each sequence: unequal, as requests are."""
    S = c["seqs"]
    if c["phase"] == "step":
        ctx = c["context"] or (0 if c["layer"] in ("swiglu", "moe") else STATE_ROWS)
        return [1] * S, [ctx - (i * 37) % (ctx // 2 + 1) if c["context"] else ctx for i in range(S)]
    share = [2 + (i * 5) % 3 for i in range(S)]
    new = [max(1, c["rows"] * s // sum(share)) for s in share]
    new[0] += c["rows"] - sum(new)
    return new, [0] * S


def _inputs(c, seed):
    """The rows that enter the layer (normed rows are about N(0, 1)), those of the state's earlier
    rows first for each sequence, and what the cache holds of earlier positions."""
    g = torch.Generator(device=DEVICE).manual_seed(seed * 7919 + 2)
    z, (new, old) = _sizes(c), _lengths(c)
    dt = _dtype(c)
    x = torch.randn((sum(new), z["W"]), generator=g, device=DEVICE).to(dt)
    past, cached = None, None
    if c["phase"] == "step" and c["layer"] not in ("swiglu", "moe"):
        past = torch.randn((c["seqs"], STATE_ROWS, z["W"]), generator=g, device=DEVICE).to(dt)
        if c["context"]:
            heads, width = (1, z["kv_rank"] + z["rot"]) if c["layer"] == "latent" else (z["KV"], z["d"])
            n = max(old)
            k = torch.randn((c["seqs"], n, heads, width), generator=g, device=DEVICE).to(dt)
            v = torch.randn((c["seqs"], n, heads, width), generator=g, device=DEVICE).to(dt)
            cached = (k, v)
    return x, past, cached


# ---- prepare and run ------------------------------------------------------------------------
class _Layer:
    """A layer with its weights, its cache and one step's descriptors."""

    def __init__(self, c, seed):
        self.prompt = c["phase"] == "prompt"
        spec = _spec(c)
        registry = FEED_FORWARDS if c["layer"] in ("swiglu", "moe") else MIXERS
        self.mixer = registry is MIXERS
        self.part = registry.get(spec.kind)(spec, _dtype(c), DEVICE)
        self.part.bind(_weights(c, seed))
        self.x, past, cached = _inputs(c, seed)
        self.workspace = workspace.Workspace(DEVICE)
        self.ctx, self.states, self.out = None, [], None
        if self.mixer:
            new, old = _lengths(c)
            total = sum(-(-(a + b) // 64) * 64 for a, b in zip(new, old))
            self.cache = Cache({0: self.part.cache_spec()}, total + 64, 32768, _dtype(c), DEVICE, max_slots=c["seqs"])
            slots = [self.cache.take_slot() for _ in new]
            self.states = [g.data[0] for g in self.cache.state_groups]
            self.cache.reserve([(s, a + b) for s, a, b in zip(slots, new, old)])
            if self.states and past is not None:  # the state after some earlier rows of each sequence
                self.ctx = self._context(slots, [0] * len(slots), [STATE_ROWS] * len(slots))
                self.part.forward(past.reshape(-1, past.shape[-1]), self.ctx)
            if cached is not None:
                self._fill(slots, old, cached)
            self.ctx = self._context(slots, old, new)
        if not self.prompt:
            kept = [s.clone() for s in self.states]
            self.forward()  # sizes what is made lazily
            torch.cuda.synchronize()
            self.graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(self.graph):
                self.out = self.forward()
            for s, k in zip(self.states, kept):
                s.copy_(k)

    def _context(self, slots, old, new):
        batch = make_batch([[0] * n for n in new], slots, old, [[] for _ in new], DEVICE)
        ctx = RunContext(batch=batch, writes_cache=True, entry=0)
        kind = self.cache.has(0)
        views = self.cache.views(0) if kind == "parts" else [self.cache.kv(0) if kind == "kv" else self.cache.state(0)]
        ctx.parts = views if kind == "parts" else None
        ctx.kv = next((v for v in views if not isinstance(v, torch.Tensor)), None)
        ctx.state = next((v for v in views if isinstance(v, torch.Tensor)), None)
        return ctx

    def _fill(self, slots, old, cached):
        """Earlier positions' keys and values (or latents) into the sequences' pages."""
        view = self.cache.kv_groups[0].view(self.cache.kv_groups[0].entries[0])
        tables = view.page_table.long()
        for i, (s, n) in enumerate(zip(slots, old)):
            at = torch.arange(n, device=DEVICE)
            pages, rows = tables[s][at // 64], at % 64
            width = cached[0].shape[-1]
            if view.v_pages.data_ptr() == view.k_pages.data_ptr():
                view.k_pages[pages, :, rows] = 0.0
            else:
                view.v_pages[pages, :, rows, :width] = cached[1][i, :n]
            view.k_pages[pages, :, rows, :width] = cached[0][i, :n]

    def forward(self):
        return self.part.forward(self.x, self.ctx) if self.mixer else self.part.forward(self.x)

    def run(self):
        if self.prompt:
            for s in self.states:
                s.zero_()  # a sequence's start
            with workspace.use(self.workspace):
                self.out = self.forward()
            self.workspace.settle()
        else:
            self.graph.replay()
        return {"out": self.out, "state": list(self.states)}


def _qwen3(c):
    z = _sizes(c)
    return {"architectures": ["Qwen3ForCausalLM"], "model_type": "qwen3", "num_hidden_layers": c["layers"],
            "hidden_size": z["W"], "num_attention_heads": z["H"], "num_key_value_heads": z["KV"], "head_dim": z["d"],
            "intermediate_size": z["ff"], "vocab_size": VOCAB, "rope_theta": 1000000.0, "rms_norm_eps": EPS,
            "tie_word_embeddings": False, "max_position_embeddings": 40960, "hidden_act": "silu"}


class _Model:
    """A model with its engine; prompts, and the tokens that follow them, given."""

    def __init__(self, c, seed):
        self.lm = random_model_on_device(_qwen3(c), seed, torch.bfloat16, DEVICE)
        self.steps = c["steps"]
        self.prompts, self.later = _tokens(c, seed)
        self.fed = torch.tensor(self.later, dtype=torch.int32, device=DEVICE)
        total = sum(-(-(len(p) + c["steps"] + 1) // 64) * 64 for p in self.prompts)
        self.engine = Engine(self.lm, max_tokens=total + 64, max_slots=c["seqs"])

    def run(self):
        e = self.engine
        seqs = [e.open() for _ in self.prompts]
        logits = [e.step([(s, p, [len(p) - 1]) for s, p in zip(seqs, self.prompts)])]
        for i in range(self.steps):
            logits.append(e.step_decode(seqs, self.fed[i]))
        for s in seqs:
            e.close(s)
        return {"logits": logits}


def _tokens(c, seed):
    g = torch.Generator().manual_seed(seed * 7919 + 3)
    new, _ = _lengths(c)
    prompts = [torch.randint(0, VOCAB, (n,), generator=g).tolist() for n in new]
    return prompts, torch.randint(0, VOCAB, (c["steps"], c["seqs"]), generator=g).tolist()


def prepare(case, seed):
    return _Model(case, seed) if case["layer"] == "model" else _Layer(case, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without -------------------------------------------------------------
def work(case):
    c = case
    z = _sizes(c)
    size = 4 if c["dtype"] == "f32" else 2
    new, old = _lengths(c)
    R = sum(new)
    if c["layer"] == "model":
        W, d = z["W"], z["d"]
        per = W * (z["H"] + 2 * z["KV"]) * d + z["H"] * d * W + 3 * W * z["ff"]
        weights = 2.0 * (c["layers"] * per + VOCAB * W)
        kv = 2.0 * 2 * z["KV"] * d * c["layers"]
        S = c["seqs"]
        rows = R + S * c["steps"]
        pairs = sum(n * n / 2.0 + c["steps"] * n for n in new)
        flops = 2.0 * rows * c["layers"] * per + 2.0 * S * (c["steps"] + 1) * VOCAB * W + 4.0 * c["layers"] * z["H"] * d * pairs
        data = (1 + c["steps"]) * weights + kv * (R + sum(c["steps"] * n for n in new)) + 4.0 * S * (c["steps"] + 1) * VOCAB
        return {"bytes": data, "flops": flops}
    mats = {k: s for k, (s, how) in _shapes(c).items() if how == "matrix"}
    params = sum(s[0] * s[1] for s in mats.values())
    rest = sum(math.prod(s) for s, how in _shapes(c).values() if how != "matrix")
    data, flops = 4.0 * rest + R * z["W"] * (size + 4.0), 2.0 * R * params
    keys = sum(n * (n + 1) / 2 + n * o for n, o in zip(new, old))  # (query, key) pairs
    layer, d = c["layer"], z["d"]
    state = 0
    if layer == "moe":
        one = 3 * z["W"] * z["eff"]
        hit = z["E"] * (1 - (1 - z["top"] / z["E"]) ** R)  # experts that some row chooses, on average
        data += size * (hit * one + z["E"] * z["W"])
        flops = 2.0 * R * (z["top"] * one + z["E"] * z["W"])
    else:
        data += size * params
    if layer == "attention":
        flops += 4.0 * z["H"] * d * keys
        data += size * 2 * z["KV"] * d * (R + sum(old))
    elif layer == "latent":
        flops += 2.0 * z["H"] * (2 * d + z["rot"]) * keys
        data += size * (z["kv_rank"] + z["rot"]) * (R + sum(old))
    elif layer == "pair":
        w = z["window"]
        keys = sum(sum(min(w, o + i + 1) for i in range(n)) for n, o in zip(new, old))
        flops += 4.0 * z["H"] * d * keys + 6.0 * R * z["sh"] * 64 * z["N"]
        data += size * 2 * z["KV"] * d * (R + sum(min(w, o) for o in old))
        state = z["sh"] * 64 * z["N"] + 3 * (z["sh"] * 64 + 2 * z["G"] * z["N"])
    elif layer == "mlstm":
        flops += 6.0 * R * z["mh"] * d * z["mdv"]
        state = z["mh"] * (d * z["mdv"] + d)
    elif layer == "delta":
        flops += 8.0 * R * z["dh"] * z["dd"] ** 2
        state = z["dh"] * z["dd"] ** 2
    elif layer == "gated_delta":
        flops += 8.0 * R * z["gh"] * z["gd"] ** 2
        state = z["gh"] * z["gd"] ** 2 + 3 * (z["gh"] + 2 * z["gk"]) * z["gd"]
    elif layer == "scan":
        flops += 7.0 * R * z["C"] * z["NS"]
        state = z["C"] * (z["NS"] + 3)
    return {"bytes": data + 4.0 * c["seqs"] * state * (1 if c["phase"] == "prompt" else 2), "flops": flops}


def tolerance(case):
    # measured against 64 bits: whole model 1.3e-2, 32-bit layer 1.1e-6, bfloat16 layers 1.6e-3 to 4e-3
    if case["layer"] == "model":
        return {"rel": 2.5e-2, "max": 0.2}
    if case["dtype"] == "f32":
        return {"rel": 1e-5, "max": 4e-4}
    return {"rel": 1e-2, "max": 0.2}


# ---- the same in 64 bits ---------------------------------------------------------------------------
def exact(case, seed):
    if case["layer"] == "model":
        return _model_exact(case, seed)
    w = {k: t.double() for k, t in _weights(case, seed).items()}
    x, past, cached = _inputs(case, seed)
    x = x.double()
    if case["layer"] == "swiglu":
        g = x @ w["gate_proj"].T
        return {"out": (g * torch.sigmoid(g) * (x @ w["up_proj"].T)) @ w["down_proj"].T, "state": []}
    if case["layer"] == "moe":
        return {"out": _moe(case, w, x), "state": []}
    new, old = _lengths(case)
    fn = {"attention": _attention, "latent": _latent, "mlstm": _mlstm, "pair": _pair, "delta": _delta,
          "gated_delta": _gated_delta, "scan": _scan}[case["layer"]]
    outs, states, r0 = [], [], 0
    for i, (n, o) in enumerate(zip(new, old)):
        xi = x[r0:r0 + n]
        r0 += n
        before = None if past is None else past[i].double()
        kv = None if cached is None else tuple(t[i, :o].double() for t in cached)
        y, s = fn(case, w, xi, o, before, kv)
        outs.append(y)
        states.append(s)
    groups = [torch.stack([s[k] for s in states]) for k in range(len(states[0]))]
    return {"out": torch.cat(outs), "state": groups}


def _rms(x, weight=None):
    y = x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
    return y if weight is None else y * weight


def _rotate(x, start, base, rd, pairs="half"):
    """x [rows, heads, d]: the first rd elements turn by position / base^(2 i / rd)."""
    i = torch.arange(rd // 2, device=x.device, dtype=torch.float64)
    pos = start + torch.arange(x.shape[0], device=x.device, dtype=torch.float64)
    a = (pos[:, None] / base ** (2 * i / rd))[:, None, :]
    y = x.clone()
    lo, hi = (slice(0, rd // 2), slice(rd // 2, rd)) if pairs == "half" else (slice(0, rd, 2), slice(1, rd, 2))
    u, v = x[..., lo], x[..., hi]
    y[..., lo], y[..., hi] = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
    return y


def _heads(q, k, v, start, scale, weigh):
    """q [n, H, d], k and v [m, KV, *] of positions 0..m-1, queries from `start` on."""
    out = []
    rep = q.shape[1] // k.shape[1]
    dist = (start + torch.arange(q.shape[0], device=q.device))[:, None] - torch.arange(k.shape[0], device=q.device)
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // rep].T * scale
        out.append(weigh(s, dist, h) @ v[:, h // rep])
    return torch.stack(out, 1)


def _attention_heads(z, p, x, start, kv):
    """Qwen3's attention layer up to its heads; p(role) gives a weight."""
    H, KV, d = z["H"], z["KV"], z["d"]
    q = _rotate(_rms((x @ p("q_proj").T).view(-1, H, d), p("q_norm")), start, 1e6, d)
    k = _rotate(_rms((x @ p("k_proj").T).view(-1, KV, d), p("k_norm")), start, 1e6, d)
    v = (x @ p("v_proj").T).view(-1, KV, d)
    if kv is not None:
        k, v = torch.cat([kv[0], k]), torch.cat([kv[1], v])
    o = _heads(q, k, v, start, d ** -0.5, lambda s, dist, h: torch.softmax(s.masked_fill(dist < 0, -math.inf), -1))
    return o.flatten(1) @ p("o_proj").T, k, v


def _attention(c, w, x, start, before, kv):
    return _attention_heads(_sizes(c), w.__getitem__, x, start, kv)[0], []


def _latent(c, w, x, start, before, kv):
    z = _sizes(c)
    H, d, r, kr = z["H"], z["d"], z["rot"], z["kv_rank"]
    q = (_rms(x @ w["q_down"].T, w["q_norm"]) @ w["q_up"].T).view(-1, H, d + r)
    # pairs of neighbours turn; their order among the rotated elements changes no score, but the
    # cached part holds all first elements of the pairs, then all second ones
    order = torch.cat([torch.arange(0, r, 2), torch.arange(1, r, 2)]).to(x.device)
    q_rot = _rotate(q[..., d:], start, 500000.0, r, "consecutive")[..., order]
    low = x @ w["kv_down"].T
    lat = _rms(low[:, :kr], w["kv_norm"])
    k_rot = _rotate(low[:, None, kr:], start, 500000.0, r, "consecutive")[:, 0][:, order]
    if kv is not None:
        lat = torch.cat([kv[0][:, 0, :kr], lat])
        k_rot = torch.cat([kv[0][:, 0, kr:], k_rot])
    k = torch.cat([(lat @ w["k_up"].T).view(-1, H, d), k_rot[:, None].expand(-1, H, -1)], -1)
    v = (lat @ w["v_up"].T).view(-1, H, d)

    def weigh(s, dist, h):
        s = torch.cat([s.masked_fill(dist < 0, -math.inf), w["sink"][h].expand(s.shape[0], 1)], 1)
        return torch.softmax(s, -1)[:, :-1]

    o = _heads(torch.cat([q[..., :d], q_rot], -1), k, v, start, (d + r) ** -0.5, weigh).flatten(1)
    return (torch.sigmoid(x @ w["gate"].T) * o) @ w["o_proj"].T, []


def _with_past(x, before):
    return (x, 0) if before is None else (torch.cat([before, x]), before.shape[0])


def _conv(x, filters, bias=None):
    """silu of a causal filter a channel: x [n, C], filters [C, taps], the last tap on the row itself."""
    taps = filters.shape[1]
    pad = torch.cat([x.new_zeros((taps - 1, x.shape[1])), x])
    y = sum(pad[t:t + x.shape[0]] * filters[:, t] for t in range(taps))
    y = y if bias is None else y + bias
    return y * torch.sigmoid(y), pad[x.shape[0]:]


def _mlstm(c, w, x, start, before, kv):
    z = _sizes(c)
    H, d, dv = z["mh"], z["d"], z["mdv"]
    x, skip = _with_past(x, before)
    n = x.shape[0]
    q, k = ((x @ w[r].T).view(n, H, d) for r in ("q_proj", "k_proj"))
    v = (x @ w["v_proj"].T).view(n, H, dv)
    cap = lambda t: 15.0 * torch.tanh(t / 15.0)  # noqa: E731
    i = cap(x @ w["i_proj"].T + w["i_bias"])
    f = torch.nn.functional.logsigmoid(cap(x @ w["f_proj"].T + w["f_bias"]))
    S, nn, m, outs = x.new_zeros((H, d, dv)), x.new_zeros((H, d)), x.new_zeros(H), []
    q = q * d ** -0.5
    for t in range(n):
        m2 = torch.maximum(f[t] + m, i[t])
        a, b = torch.exp(f[t] + m - m2), torch.exp(i[t] - m2)
        S = a[:, None, None] * S + (b[:, None] * k[t])[:, :, None] * v[t][:, None, :]
        nn = a[:, None] * nn + b[:, None] * k[t]
        m = m2
        den = torch.maximum((nn * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
        outs.append((S * q[t][:, :, None]).sum(1) / den[:, None])
    o = _rms(torch.stack(outs)).flatten(1) * w["norm"] * torch.sigmoid(x @ w["gate"].T)
    state = torch.cat([S.flatten(1), nn, m[:, None].expand(-1, dv // 64)], 1)
    return o[skip:] @ w["o_proj"].T, [state]


def _pair(c, w, x, start, before, kv):
    z = _sizes(c)
    H, KV, d, h, N, G = z["H"], z["KV"], z["d"], z["sh"], z["N"], z["G"]
    left = {k[5:]: t for k, t in w.items() if k.startswith("left/")}
    right = {k[6:]: t for k, t in w.items() if k.startswith("right/")}
    q = _rotate((x @ left["q_proj"].T).view(-1, H, d), start, 500000.0, d // 2)
    k = _rotate((x @ left["k_proj"].T).view(-1, KV, d), start, 500000.0, d // 2)
    v = (x @ left["v_proj"].T).view(-1, KV, d)
    if kv is not None:
        k, v = torch.cat([kv[0], k]), torch.cat([kv[1], v])
    o = _heads(q, k, v, start, d ** -0.5, lambda s, dist, hh: torch.sigmoid(s + left["score_bias"][hh])
               * ((dist >= 0) & (dist < z["window"])))
    a = o.flatten(1) @ left["o_proj"].T
    x, skip = _with_past(x, before)
    n, inner = x.shape[0], h * 64
    proj = x @ right["in_proj"].T
    gate, xbc, dt = proj[:, :inner], proj[:, inner:-h], proj[:, -h:]
    xbc, tail = _conv(xbc, right["conv"], right["conv_bias"])
    xs = xbc[:, :inner].view(n, h, 64)
    B = xbc[:, inner:inner + G * N].view(n, G, N).repeat_interleave(h // G, 1)
    C = xbc[:, inner + G * N:].view(n, G, N).repeat_interleave(h // G, 1)
    dt = torch.nn.functional.softplus(dt + right["dt_bias"], threshold=1e9)
    decay = torch.exp(-torch.exp(right["A_log"]) * dt)
    S, ys = x.new_zeros((h, 64, N)), []
    for t in range(n):
        S = decay[t][:, None, None] * S + (dt[t][:, None] * xs[t])[:, :, None] * B[t][:, None, :]
        ys.append((S * C[t][:, None, :]).sum(-1))
    y = (torch.stack(ys) + right["D"][:, None] * xs).flatten(1) * (gate * torch.sigmoid(gate))
    y = _rms(y.view(n, 2, -1)).flatten(1) * right["norm"]
    return 0.75 * a + 0.55 * (y[skip:] @ right["o_proj"].T), [torch.cat([tail.flatten(), S.flatten()])]


def _delta(c, w, x, start, before, kv):
    z = _sizes(c)
    H, d = z["dh"], z["dd"]
    x, skip = _with_past(x, before)
    n = x.shape[0]
    r, k, v = ((x @ w[p].T).view(n, H, d) for p in ("r_proj", "k_proj", "v_proj"))
    decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(torch.tanh(x @ w["w1_proj"].T) @ w["w2_proj"].T + w["w0"]))
    decay = decay.view(n, H, d)
    a = torch.sigmoid(x @ w["a_proj"].T + w["a_bias"]).view(n, H, d)
    u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    au = a * u
    S, outs = x.new_zeros((H, d, d)), []  # [value, key]
    for t in range(n):
        seen = (S * u[t][:, None, :]).sum(-1)
        S = S * decay[t][:, None, :] - seen[:, :, None] * au[t][:, None, :] + v[t][:, :, None] * k[t][:, None, :]
        outs.append((S * r[t][:, None, :]).sum(-1))
    o = _rms(torch.stack(outs)).flatten(1) * w["norm"] * torch.sigmoid(x @ w["g_proj"].T)
    return o[skip:] @ w["o_proj"].T, [S.flatten()]


def _gated_delta(c, w, x, start, before, kv):
    z = _sizes(c)
    H, G, d = z["gh"], z["gk"], z["gd"]
    x, skip = _with_past(x, before)
    n = x.shape[0]
    q, k, v, tails = None, None, None, []
    made = []
    for p in ("q", "k", "v"):
        y, tail = _conv(x @ w[p + "_proj"].T, w[p + "_conv"])
        made.append(y)
        tails.append(tail)
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)  # noqa: E731
    q = (unit(made[0].view(n, G, d)) * d ** -0.5).repeat_interleave(H // G, 1)
    k = unit(made[1].view(n, G, d)).repeat_interleave(H // G, 1)
    v = made[2].view(n, H, d)
    beta = torch.sigmoid(x @ w["b_proj"].T)
    g = torch.exp(-torch.exp(w["A_log"]) * torch.nn.functional.softplus(x @ w["a_proj"].T + w["dt_bias"], threshold=1e9))
    S, outs = x.new_zeros((H, d, d)), []  # [value, key]
    for t in range(n):
        S = S * g[t][:, None, None]
        u = beta[t][:, None] * (v[t] - (S * k[t][:, None, :]).sum(-1))
        S = S + u[:, :, None] * k[t][:, None, :]
        outs.append((S * q[t][:, None, :]).sum(-1))
    gate = (x @ w["g_proj"].T).view(n, H, d)
    o = (_rms(torch.stack(outs)) * w["norm"] * gate * torch.sigmoid(gate)).flatten(1)
    return o[skip:] @ w["o_proj"].T, [torch.cat([torch.cat(tails, 1).flatten(), S.flatten()])]


def _scan(c, w, x, start, before, kv):
    z = _sizes(c)
    C, N, R = z["C"], z["NS"], z["R"]
    x, skip = _with_past(x, before)
    n = x.shape[0]
    xz = x @ w["in_proj"].T
    u, tail = _conv(xz[:, :C], w["conv"], w["conv_bias"])
    gate = xz[:, C:]
    low = u @ w["x_proj"].T
    dt = torch.nn.functional.softplus(low[:, :R] @ w["dt_proj"].T + w["dt_bias"], threshold=1e9)
    B, Cc = low[:, R:R + N], low[:, R + N:]
    A = -torch.exp(w["A_log"])
    S, ys = x.new_zeros((C, N)), []
    for t in range(n):
        S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * B[t]
        ys.append(S @ Cc[t])
    y = (torch.stack(ys) + w["D"] * u) * (gate * torch.sigmoid(gate))
    return y[skip:] @ w["o_proj"].T, [torch.cat([tail.flatten(), S.flatten()])]


def _moe(c, w, x):
    z = _sizes(c)
    logits = x @ w["router"].T
    groups = logits.view(-1, 4, z["E"] // 4)
    keep = groups.max(-1).values.topk(2, -1).indices
    mask = torch.full_like(groups, -math.inf).scatter_(1, keep[:, :, None].expand(-1, -1, z["E"] // 4), 0.0)
    ids = (groups + mask).flatten(1).topk(z["top"], -1).indices
    wts = 1.5 * torch.softmax(logits, -1).gather(1, ids)
    out = torch.zeros_like(x)
    for e in range(z["E"]):
        r, k = (ids == e).nonzero(as_tuple=True)
        g = x[r] @ w[f"expert_gate#{e}"].T
        y = (g * torch.sigmoid(g) * (x[r] @ w[f"expert_up#{e}"].T)) @ w[f"expert_down#{e}"].T
        out.index_add_(0, r, wts[r, k][:, None] * y)
    return out


def _model_exact(c, seed):
    """The model's own weights (drawn by name, as a checkpoint holds them) in 64-bit formulas."""
    lm = random_model_on_device(_qwen3(c), seed, torch.bfloat16, DEVICE)
    z = _sizes(c)
    H, KV, d, ff, W = z["H"], z["KV"], z["d"], z["ff"], z["W"]
    prompts, later = _tokens(c, seed)
    rows = [[] for _ in range(c["steps"] + 1)]
    emb, head = lm.embedding, lm.head.double()
    for i, p in enumerate(prompts):
        ids = torch.tensor(p + [later[t][i] for t in range(c["steps"])], device=DEVICE)
        x = emb[ids].double()
        for layer in lm.layers:
            m, f = layer.mixer, layer.feed_forward
            cut = {"q_proj": m.qkv[:H * d], "k_proj": m.qkv[H * d:(H + KV) * d], "v_proj": m.qkv[(H + KV) * d:],
                   "o_proj": m.o, "q_norm": m.q_norm, "k_norm": m.k_norm}
            y, _, _ = _attention_heads(z, lambda r: cut[r].double(), _rms(x, layer.mixer_norm.weight.double()), 0, None)
            x = x + y
            h = _rms(x, layer.feed_forward_norm.weight.double())
            pairs = f.gate_up.view(ff, 2, W)
            g = h @ pairs[:, 0].double().T
            x = x + (g * torch.sigmoid(g) * (h @ pairs[:, 1].double().T)) @ f.down.double().T
        logits = _rms(x[len(p) - 1:], lm.final_norm.weight.double()) @ head.T
        for t in range(c["steps"] + 1):
            rows[t].append(logits[t])
    return {"logits": [torch.stack(r) for r in rows]}
