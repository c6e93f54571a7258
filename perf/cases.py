"""The work that is measured when this framework is made faster: its layers, each through an entry point that a program calls, and one
whole serving call. Sizes are those of bench.py's model configurations and of the tests; `draw` spreads them over the range.

Kinds of case:

- `block`: one transformer layer of the encoder / decoder models (attention, feed-forward, norms): training (forward and backward of an
  encoder layer under right-padding), a prompt or one token per sequence of a cached decoder layer, a forward pass.
- `attention`, `recurrence`: one sequence mixer of the packed-step decoders with the projection that feeds it, on whole prompts
  (`prompt`) or on one token per sequence behind `length` cached positions (`token`).
- `experts`: a mixture of experts with a shared expert and identity experts.
- `requests`: a batch of requests through the batching engine: prompts, then given tokens one step at a time, logits of every step.
"""
import contextlib
import io
import math

import torch

from vyomai_b200 import HybridBatchEngine, HybridCacheManager, KifetarConfig, KifetarForCausalLM, StaticCacheOne
from vyomai_b200.functional import MaskSpec, RopeTables
from vyomai_b200.layers.mixers import (BiasedAttention, GatedDeltaMixer, HeadDecayDeltaMixer, LatentAttention, LightningMixer, MoEFeedForward,
                                       Projection, SigmoidAttention, StateSpaceMixer, TalkingHeadsAttention, WindowSinkAttention, pack_biases,
                                       pack_rows)
from vyomai_b200.layers.positional_embeddings import RotaryEmbedding
from vyomai_b200.models.decoder import DecoderLayer
from vyomai_b200.models.encoder import EncoderLayer
from vyomai_b200.ops import PackedBatch
from vyomai_b200.paged import LayerCacheView

PAGE = 16
EPS = 1e-6
DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}


def listed():
    return [
        # one captioner / encoder training layer at the batch of the headline benchmark: bf16, right-padded text
        {"name": "block_train_64x128", "kind": "block", "mode": "train", "dtype": "bf16", "seqs": 64, "length": 128, "width": 768, "kv_heads": 4},
        # an image encoder's layer in single precision (197 = 14 x 14 patches and the class token)
        {"name": "block_forward_fp32_8x197", "kind": "block", "mode": "forward", "dtype": "fp32", "seqs": 8, "length": 197, "width": 768, "kv_heads": 12},
        # prompts of a cached decoder layer
        {"name": "block_prompt_8x512", "kind": "block", "mode": "prompt", "dtype": "bf16", "seqs": 8, "length": 512, "width": 768, "kv_heads": 4},
        # the smallest call: the next token of one sequence
        {"name": "block_token_1x300", "kind": "block", "mode": "token", "dtype": "bf16", "seqs": 1, "length": 300, "width": 768, "kv_heads": 4},
        # windowed attention with kept tokens and a sink while 32 sequences decode
        {"name": "sink_token_32x2048", "kind": "attention", "form": "sink", "mode": "token", "dtype": "bf16", "seqs": 32, "length": 2048, "width": 1024,
         "window": 512},
        # capped, distance-biased windowed attention over long prompts of unequal length
        {"name": "biased_prompt_4x2048", "kind": "attention", "form": "biased", "mode": "prompt", "dtype": "bf16", "seqs": 4, "length": 2048, "width": 1024,
         "window": 512},
        # latent attention over the whole context
        {"name": "latent_prompt_4x2048", "kind": "attention", "form": "latent", "mode": "prompt", "dtype": "bf16", "seqs": 4, "length": 2048, "width": 1024,
         "window": 0},
        # heads that exchange scores, an odd prompt length
        {"name": "talking_prompt_2x1437", "kind": "attention", "form": "talking", "mode": "prompt", "dtype": "bf16", "seqs": 2, "length": 1437, "width": 1024,
         "window": 0},
        # gated delta rule with a decay per channel
        {"name": "delta_prompt_4x2048", "kind": "recurrence", "form": "delta", "mode": "prompt", "dtype": "bf16", "seqs": 4, "length": 2048, "width": 1024},
        # state-space recurrence
        {"name": "ssm_prompt_4x2048", "kind": "recurrence", "form": "ssm", "mode": "prompt", "dtype": "bf16", "seqs": 4, "length": 2048, "width": 1024},
        # mixture of experts on prompt-sized rows
        {"name": "experts_4096", "kind": "experts", "mode": "prompt", "dtype": "bf16", "seqs": 2, "length": 2048, "width": 1024},
        # serving: 8 requests of 128 tokens and 16 more each, sigmoid attention and head-decay delta layers in turn
        {"name": "requests_8x128", "kind": "requests", "mode": "serve", "dtype": "bf16", "seqs": 8, "length": 128, "steps": 16, "width": 1024, "window": 512},
    ]


def draw(rng):
    """Another case of the same ranges: every kind and form alike, lengths and batches over their logarithm, odd ones among them."""
    spread = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    kind, form = rng.choice([("block", None)] * 4 + [("attention", f) for f in ("sink", "biased", "latent", "talking", "sigmoid")]
                            + [("recurrence", f) for f in ("lightning", "delta", "head_delta", "ssm")] + [("experts", None), ("requests", None)])
    dtype = "fp32" if rng.random() < 0.2 else "bf16"
    if kind == "block":
        mode = rng.choice(["train", "forward", "prompt", "token"])
        c = {"kind": kind, "mode": mode, "dtype": dtype, "seqs": spread(1, 64), "length": spread(8, 512 if mode != "token" else 500),
             "width": rng.choice([768, 768, 1024]), "kv_heads": 4}
        if mode in ("train", "forward"):
            c["kv_heads"] = rng.choice([4, c["width"] // 64])
        while mode != "token" and c["seqs"] * c["length"] > 8192:
            c["seqs"] = (c["seqs"] + 1) // 2
        return c
    if kind == "requests":
        return {"kind": kind, "mode": "serve", "dtype": "bf16", "seqs": spread(1, 12), "length": spread(16, 300), "steps": rng.randint(4, 16), "width": 1024,
                "window": rng.choice([64, 512])}
    c = {"kind": kind, "mode": "prompt" if kind == "experts" or rng.random() < 0.6 else "token", "dtype": dtype}
    if form:
        c["form"] = form
    c["width"] = rng.choice([512, 1024, 1024, 2048])
    c["seqs"] = spread(1, 32 if c["mode"] == "token" else 8)
    c["length"] = spread(16, 2048)
    # fp32 products and wide models are the dear ones
    most = (8192 if c["width"] < 2048 else 3000) if dtype == "bf16" else 2000 if c["width"] < 2048 else 700
    while c["mode"] == "prompt" and c["seqs"] * c["length"] > most:
        if c["seqs"] > 1:
            c["seqs"] = (c["seqs"] + 1) // 2
        else:
            c["length"] = most - rng.randint(0, 40)
    if kind == "attention":
        c["window"] = rng.choice([0, 512, 512, 100]) if form in ("latent", "talking") else rng.choice([512, 512, 100])
    return c


# ---- seeded inputs, on the GPU ----
class Rand:
    def __init__(self, seed):
        self.g = torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)

    def normal(self, *shape, std=1.0, mean=0.0, dtype=torch.float32):
        return (torch.randn(shape, generator=self.g, device="cuda") * std + mean).to(dtype)

    def uniform(self, lo, hi, *shape, dtype=torch.float32):
        return (torch.rand(shape, generator=self.g, device="cuda") * (hi - lo) + lo).to(dtype)

    def ids(self, hi, *shape):
        return torch.randint(0, hi, shape, generator=self.g, device="cuda")


def lengths_of(case):
    """Prompts of unequal length, the first the longest; a token case has one new row per sequence."""
    L = case["length"]
    return [1] * case["seqs"] if case["mode"] == "token" else [L - (i * 37) % (L // 2 + 1) for i in range(case["seqs"])]


def starts_of(case):
    """Positions already cached: none for prompts, unequal ones up to `length` for token cases."""
    L = case["length"]
    return [L - (i * 53) % (L // 2 + 1) for i in range(case["seqs"])] if case["mode"] == "token" else [0] * case["seqs"]


def packed_batch(case):
    new, old = lengths_of(case), starts_of(case)
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")  # noqa: E731
    cu = [0]
    for n in new:
        cu.append(cu[-1] + n)
    pages = [(a + b + PAGE - 1) // PAGE for a, b in zip(old, new)]
    table, at = torch.zeros((len(new), max(pages)), dtype=torch.int32), 0
    for i, n in enumerate(pages):
        table[i, :n] = torch.arange(at, at + n, dtype=torch.int32)
        at += n
    return PackedBatch(ints(cu), ints(old), ints(list(range(len(new)))), max(new), table.cuda(), PAGE, all_start=case["mode"] != "token"), at


# ---- the mixers of the packed-step decoders: configuration and weights, as bench.py's models have them ----
def mixer_config(case):
    W, f = case["width"], case["form"]
    H, Hn = W // 128, W // 64
    if f in ("sink", "biased", "sigmoid"):
        m = {"heads": H, "kv_heads": max(H // 4, 1), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": case["window"]}}
        if f == "sink":
            m["mask"]["keep_first"] = 4
        elif f == "biased":
            m.update(softcap=30.0, q_temp={"coef": 0.1, "every": 512})
        else:
            m["rot"] = {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 1024}}
        return m
    if f == "talking":
        return {"heads": Hn, "kv_heads": max(Hn // 4, 1), "dim": 64, "vdim": 64, "scale": 0.125, "softcap": 30.0, "rot": {"base": 10000.0, "dims": 64},
                **({"mask": {"size": case["window"]}} if case["window"] else {})}
    if f == "latent":
        return {"heads": Hn, "dim": 64, "rot_dim": 32, "vdim": 64, "kv_rank": 192, "q_rank": W // 2, "scale": 96 ** -0.5, "rot": {"base": 10000.0, "dims": 32},
                **({"mask": {"size": case["window"]}} if case["window"] else {})}
    if f == "lightning":
        return {"heads": H, "dim": 128, "vdim": 128, "decay": [1.0 - 2.0 ** -(3 + 5 * i / max(H - 1, 1)) for i in range(H)]}
    if f in ("delta", "head_delta"):
        return {"heads": H, "kv_heads": max(H // 2, 1), "dim": 128, "vdim": 128, "conv": 4}
    Hs = 2 * W // 64
    return {"heads": Hs, "vdim": 64, "state": 128, "groups": max(Hs // 8, 1), "conv": 4, "norm_groups": max(Hs // 8, 1)}


MIXERS = {"sink": WindowSinkAttention, "biased": BiasedAttention, "sigmoid": SigmoidAttention, "talking": TalkingHeadsAttention, "latent": LatentAttention,
          "lightning": LightningMixer, "delta": GatedDeltaMixer, "head_delta": HeadDecayDeltaMixer, "ssm": StateSpaceMixer}


def mixer_weights(case, m, r):
    W, f, dt = case["width"], case["form"], DTYPES[case["dtype"]]
    lin = lambda o, i: r.normal(o, i, std=i ** -0.5, dtype=dt)  # noqa: E731
    vec = lambda n, std=0.1, mean=0.0: r.normal(n, std=std, mean=mean, dtype=dt)  # noqa: E731
    H = m["heads"]
    w = {}
    if f in ("sink", "biased", "sigmoid", "talking"):
        G, d, dv = m["kv_heads"], m["dim"], m["vdim"]
        w.update(q=lin(H * d, W), k=lin(G * d, W), o=lin(W, H * dv))
        if f != "sigmoid":
            w["v"] = lin(G * dv, W)
        if f != "sink":
            w.update({"q.b": vec(H * d), "k.b": vec(G * d)})
            if f != "sigmoid":
                w["v.b"] = vec(G * dv)
        if f == "sink":
            w.update({"q.norm": vec(H * d, mean=1.0), "k.norm": vec(G * d, mean=1.0), "sink": vec(H, std=1.0), "g": lin(H, W)})
        elif f == "biased":
            w["sink"] = vec(H, std=1.0)
        elif f == "sigmoid":
            w.update({"q.norm": vec(d, mean=1.0), "k.norm": vec(d, mean=1.0), "temp": vec(H, std=0.5, mean=2.0), "pb": vec(H, std=0.5, mean=-2.0), "g": lin(H, W)})
        else:
            talk = torch.eye(H, device="cuda") + 0.3 * r.normal(H, H) / H ** 0.5
            w.update({"talk": talk.to(dt), "g": lin(H * dv, W), "o.b": vec(W)})
    elif f == "latent":
        dn, dr, dv, R, Q = m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
        w.update({"dq": lin(Q, W), "dq.norm": vec(Q, mean=1.0), "uq": lin(H * (dn + dr), Q), "dkv": lin(R + dr, W), "dkv.norm": vec(R, mean=1.0),
                  "uk": lin(H * dn, R), "uv": lin(H * dv, R), "o": lin(W, H * dv)})
    elif f == "lightning":
        d, dv = m["dim"], m["vdim"]
        w.update(q=lin(H * d, W), k=lin(H * d, W), v=lin(H * dv, W), g=lin(H * dv, W), o=lin(W, H * dv), norm=vec(H * dv, mean=1.0))
    elif f in ("delta", "head_delta"):
        G, d, dv, t = m["kv_heads"], m["dim"], m["vdim"], m["conv"]
        w.update({"q": lin(G * d, W), "k": lin(G * d, W), "v": lin(H * dv, W), "o": lin(W, H * dv), "b": lin(H, W), "norm": vec(dv, mean=1.0),
                  "q.conv": r.normal(G * d, t, std=0.5, dtype=dt), "k.conv": r.normal(G * d, t, std=0.5, dtype=dt), "v.conv": r.normal(H * dv, t, std=0.5, dtype=dt),
                  "A_log": r.uniform(-2.0, 0.0, H, dtype=dt)})
        if f == "delta":
            w.update(a1=lin(16, W), a2=lin(H * d, 16), g1=lin(16, W), g2=lin(H * dv, 16), dt_bias=r.uniform(-3.0, -1.0, H * d, dtype=dt))
        else:
            w.update(a=lin(H, W), g=lin(H * dv, W), dt_bias=r.uniform(-3.0, -1.0, H, dtype=dt))
    else:
        N, dv, gn = m["state"], m["vdim"], m["groups"] * m["state"]
        inner = H * dv
        w.update({"in": lin(2 * inner + 2 * gn + H, W), "conv": r.normal(inner + 2 * gn, m["conv"], std=0.5, dtype=dt), "conv.b": vec(inner + 2 * gn),
                  "dt_bias": r.uniform(-2.0, 0.0, H, dtype=dt), "A_log": r.uniform(-1.0, 1.0, H, dtype=dt), "D": vec(H, std=0.5, mean=0.5), "norm": vec(inner, mean=1.0),
                  "o": lin(W, inner)})
    return w


def mixer_state(case, spec, pages, r):
    """What the cache holds before the pass: nothing that counts before a prompt, the sequences' past before a token."""
    past = case["mode"] == "token"
    view = LayerCacheView()
    if spec["pages"]:
        g, dk, dv = spec["pages"]
        make = (lambda *s: r.normal(*s)) if past else (lambda *s: torch.zeros(s, device="cuda"))
        view.k_pool = make(pages, PAGE, g, dk)
        view.v_pool = make(pages, PAGE, g, dv) if dv else None
    for name, shape in spec["states"].items():
        dt = spec.get("state_dtypes", {}).get(name, torch.float32)
        shape = (case["seqs"],) + tuple(shape)
        view.states[name] = r.normal(*shape, std=0.3 if name == "S" else 1.0) if past and dt == torch.float32 else torch.zeros(shape, device="cuda", dtype=dt)
    return view


def mixer_inputs(case, seed):
    r = Rand(seed)
    m = mixer_config(case)
    w = mixer_weights(case, m, r)
    batch, pages = packed_batch(case)
    h = r.normal(sum(lengths_of(case)), case["width"], dtype=DTYPES[case["dtype"]])   # the layer's normed input
    return m, w, batch, pages, h, r


def prepare_mixer(case, seed):
    m, w, batch, pages, h, r = mixer_inputs(case, seed)
    kw = {"sink": "zero"} if case["form"] == "talking" else {}
    mixer = MIXERS[case["form"]](m, w, EPS, DTYPES[case["dtype"]], True, **kw)
    packed, spans = pack_rows(mixer.input_weights())
    return {"mixer": mixer, "inp": Projection(packed, True), "spans": spans, "bias": pack_biases(spans, packed.shape[0], mixer.input_biases(), packed),
            "batch": batch, "cache": mixer_state(case, mixer.cache_spec(), pages, r), "h": h}


def run_mixer(s):
    with torch.no_grad():
        p = s["inp"](s["h"], bias=s["bias"])
        y = s["mixer"].forward([p[:, o:o + n] for o, n in s["spans"]], s["batch"], s["cache"])
    c = s["cache"]
    out = {"y": y, "state": {k: v for k, v in c.states.items() if k != "done"}}
    if c.k_pool is not None:
        out["k"] = c.k_pool
    if c.v_pool is not None:
        out["v"] = c.v_pool
    return out


# ---- experts ----
EXPERTS, IDENTITY, TOP = 28, 4, 4


def expert_inputs(case, seed):
    r, W, dt = Rand(seed), case["width"], DTYPES[case["dtype"]]
    lin = lambda o, i, s=1.0: r.normal(o, i, std=s * i ** -0.5, dtype=dt)  # noqa: E731
    w = {"router": lin(EXPERTS + IDENTITY, W, 2.0), "correction": r.normal(EXPERTS + IDENTITY, std=0.02, dtype=dt), "shared.sg": lin(1, W)}
    for pre, ff in [(f"e{e}.", W // 4) for e in range(EXPERTS)] + [("shared.", W // 2)]:
        w.update({pre + "gate": lin(ff, W), pre + "up": lin(ff, W), pre + "down": lin(W, ff)})
    return w, r.normal(sum(lengths_of(case)), W, dtype=dt)


def prepare_experts(case, seed):
    w, h = expert_inputs(case, seed)
    moe = MoEFeedForward(w, EXPERTS, TOP, 1.0, DTYPES[case["dtype"]], True, shared=True, router="softmax", normalize=False, form="swiglu", identity=IDENTITY)
    return {"moe": moe, "h": h, "batch": packed_batch(case)[0]}


def run_experts(s):
    with torch.no_grad():
        y, identity = s["moe"].forward_parts(s["h"], s["batch"])
    return {"y": y, "identity": identity}


# ---- transformer layers ----
class BlockConfig:
    num_hidden_layers = 1
    max_position_embeddings = 514
    hidden_dropout_prob = 0.0
    layer_norm_eps = 1e-5
    hidden_act = "gelu"

    def __init__(self, case):
        self.hidden_size, self.num_attention_heads, self.num_key_value_heads = case["width"], case["width"] // 64, case["kv_heads"]


def block_inputs(case, seed):
    """The layer's parameters (by shape: matrices ~ N(0, 1 / in)), its input rows, key padding (train / forward), the output's gradient."""
    cfg, r, dt = BlockConfig(case), Rand(seed), DTYPES[case["dtype"]]
    cls = EncoderLayer if case["mode"] in ("train", "forward") else DecoderLayer
    gqa = "gqa" if cfg.num_key_value_heads != cfg.num_attention_heads else None
    with contextlib.redirect_stdout(io.StringIO()), torch.device("cuda"):
        layer = cls(cfg, 0, gqa).to(dt)
    with torch.no_grad():
        for name, p in layer.named_parameters():
            std = p.shape[1] ** -0.5 if p.dim() == 2 else 0.1
            p.copy_(r.normal(*p.shape, std=std, mean=1.0 if "layernorm.weight" in name else 0.0))
    B, S = case["seqs"], 1 if case["mode"] == "token" else case["length"]
    x = r.normal(B, S, cfg.hidden_size, dtype=dt)
    valid = torch.tensor([S - (i * 29) % (S // 2 + 1) for i in range(B)], device="cuda")
    mask = (torch.arange(S, device="cuda")[None] < valid[:, None]).long() if case["mode"] in ("train", "forward") else torch.ones((B, S), device="cuda", dtype=torch.long)
    grad = r.normal(B, S, cfg.hidden_size, dtype=dt) if case["mode"] == "train" else None
    past = None
    if case["mode"] in ("prompt", "token"):
        shape = (B, cfg.num_key_value_heads, case["length"] + (1 if case["mode"] == "token" else 0), 64)
        make = (lambda: r.normal(*shape, dtype=dt)) if case["mode"] == "token" else (lambda: torch.zeros(shape, device="cuda", dtype=dt))
        past = (make(), make())
    return cfg, layer, x, mask, grad, past


def prepare_block(case, seed):
    cfg, layer, x, mask, grad, past = block_inputs(case, seed)
    s = {"mode": case["mode"], "layer": layer, "x": x, "grad": grad, "rope": RopeTables(RotaryEmbedding(cfg)(cfg.max_position_embeddings))}
    if past is None:
        s["mask"] = MaskSpec.from_attention_mask(mask, causal=False)
    else:
        s["mask"] = MaskSpec.from_attention_mask(mask, causal=True) if case["mode"] == "prompt" else None
        s["start"] = 0 if case["mode"] == "prompt" else case["length"]
        s["cache"] = StaticCacheOne(cfg, max_cache_len=past[0].shape[2], batch_size=case["seqs"], dtype=x.dtype, is_gqa=True)
        s["cache"].key_cache[0].copy_(past[0])
        s["cache"].value_cache[0].copy_(past[1])
    if case["mode"] == "train":
        x.requires_grad_()
        s["params"] = list(layer.named_parameters())
    else:
        layer.eval()
    return s


def run_block(s):
    if s["mode"] == "train":
        y = s["layer"](s["x"], s["mask"], s["rope"])
        g = torch.autograd.grad(y, [s["x"]] + [p for _, p in s["params"]], s["grad"])
        return {"y": y, "dx": g[0], "grads": {n: t for (n, _), t in zip(s["params"], g[1:])}}
    with torch.no_grad():
        if s["mode"] == "forward":
            return {"y": s["layer"](s["x"], s["mask"], s["rope"])}
        y, cache = s["layer"](s["x"], s["mask"], freqs=s["rope"], use_cache=True, kv_cache=s["cache"], start_pos=s["start"])
    return {"y": y, "k": cache.key_cache[0], "v": cache.value_cache[0]}


# ---- requests through the engine ----
VOCAB = 8192


def request_inputs(case, seed):
    W, r = case["width"], Rand(seed)
    H = W // 128
    dl = {"type": "delta", "mixer": {"heads": H, "kv_heads": max(H // 2, 1), "dim": 128, "vdim": 128, "conv": 4}}
    at = {"type": "attention", "mixer": {"heads": H, "kv_heads": max(H // 4, 1), "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "mask": {"size": case["window"]},
                                         "rot": {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 1024}}}}
    cfg = {"architecture": "Kifetar", "vocab": VOCAB, "width": W, "norm": {"eps": EPS},
           "layers": [{**(dl if i % 2 == 0 else at), "mlp": {"kind": "dense", "ff": 8 * W // 3 // 128 * 128}} for i in range(4)]}
    w = {}
    for name, shape in KifetarConfig(cfg).tensor_shapes().items():
        leaf = name.split(".")[-1]
        if leaf == "A_log":
            w[name] = r.uniform(-2.0, 0.0, *shape, dtype=torch.bfloat16)
        elif leaf == "dt_bias":
            w[name] = r.uniform(-3.0, -1.0, *shape, dtype=torch.bfloat16)
        else:
            std, mean = (1.0, 0.0) if leaf == "embed" else (0.5, 0.0) if leaf == "conv" else (0.5, 2.0) if leaf == "temp" else (0.5, -2.0) if leaf == "pb" else \
                (shape[1] ** -0.5, 0.0) if len(shape) == 2 else (0.1, 0.0) if leaf == "b" else (0.1, 1.0)
            w[name] = r.normal(*shape, std=std, mean=mean, dtype=torch.bfloat16)
    return cfg, w, r.ids(VOCAB, case["seqs"], case["length"] + case["steps"])


def prepare_requests(case, seed):
    cfg, w, ids = request_inputs(case, seed)
    model = KifetarForCausalLM(KifetarConfig(cfg), w, dtype=torch.bfloat16)
    n = case["seqs"]
    mgr = HybridCacheManager(model, max_tokens=n * (case["length"] + case["steps"] + PAGE), block_size=PAGE, max_seqs=n)
    return {"engine": HybridBatchEngine(model, mgr), "ids": ids.tolist(), "prompt": case["length"], "steps": case["steps"]}


def run_requests(s):
    e, P = s["engine"], s["prompt"]
    out = [e.feed([(i, t[:P], [P - 1]) for i, t in enumerate(s["ids"])])]
    for k in range(P, P + s["steps"]):
        out.append(e.feed([(i, [t[k]], [0]) for i, t in enumerate(s["ids"])]))
    e.release(range(len(s["ids"])))
    return out


KINDS = {"block": (prepare_block, run_block), "attention": (prepare_mixer, run_mixer), "recurrence": (prepare_mixer, run_mixer),
         "experts": (prepare_experts, run_experts), "requests": (prepare_requests, run_requests)}


def prepare(case, seed):
    state = KINDS[case["kind"]][0](case, seed)
    state["run"] = KINDS[case["kind"]][1]
    return state


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without ----
def visible_pairs(new, old, window):
    """(query, key) pairs under the causal mask; a window sees the last `window` positions."""
    total = 0
    for n, o in zip(new, old):
        for p in range(o, o + n):
            total += min(p + 1, window) if window else p + 1
    return total


def work(case):
    W, es = case["width"], 2 if case["dtype"] == "bf16" else 4
    if case["kind"] == "block":
        B, S = case["seqs"], 1 if case["mode"] == "token" else case["length"]
        rows, kv = B * S, case["kv_heads"] * 64
        weights = W * (W + 2 * kv) + W * W + 8 * W * W
        keys = case["length"] + 1 if case["mode"] == "token" else S
        pairs = B * (S * keys if case["mode"] != "prompt" else S * (S + 1) // 2)
        flops = 2.0 * rows * weights + 4.0 * pairs * W
        byts = weights * es + 2 * rows * W * es
        if case["mode"] == "train":
            flops, byts = 3.0 * flops, 2 * weights * es + 4 * rows * W * es
        elif case["mode"] != "forward":
            byts += 2 * B * keys * kv * es
        return {"bytes": byts, "flops": flops}
    if case["kind"] == "requests":
        H, ff, n = W // 128, 8 * W // 3 // 128 * 128, case["seqs"]
        qk = 2 * max(H // 2, 1) * 128
        weights = 2 * (W * (qk + 2 * W + 2 * H) + W * W) + 2 * (W * (W + max(H // 4, 1) * 128 + H) + W * W) + 4 * 3 * W * ff
        rows, calls = n * (case["length"] + case["steps"]), 1 + case["steps"]
        pairs = visible_pairs([case["length"] + case["steps"]] * n, [0] * n, case["window"])
        flops = 2.0 * rows * weights + 2.0 * n * calls * W * VOCAB + 2 * 4.0 * pairs * W + 2 * 6.0 * rows * W * 128
        return {"bytes": calls * (weights + W * VOCAB) * 2 + calls * n * VOCAB * 4 + 2 * n * case["steps"] * 2 * W * 128 * 4, "flops": flops}
    rows = sum(lengths_of(case))
    if case["kind"] == "experts":
        per, shared = 3 * W * (W // 4), 3 * W * (W // 2)
        return {"bytes": (EXPERTS * per + shared + W * (EXPERTS + IDENTITY)) * es + rows * W * (es + 4) + rows * 4,
                "flops": 2.0 * rows * (TOP * EXPERTS / (EXPERTS + IDENTITY) * per + shared + W * (EXPERTS + IDENTITY))}
    m, f, n = mixer_config(case), case["form"], case["seqs"]
    H = m["heads"]
    if case["kind"] == "attention":
        new, old = lengths_of(case), starts_of(case)
        pairs = visible_pairs(new, old, case["window"])
        if f == "latent":
            dn, dr, dv, R, Q = m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"], m["q_rank"]
            weights, row, per_pair = W * (Q + R + dr) + Q * H * (dn + dr) + W * H * dv, R + dr, 2 * H * (dn + dr + dv)
            extra = 2.0 * rows * H * (dn + dv) * R
        else:
            G, d, dv = m["kv_heads"], m["dim"], m["vdim"]
            weights, row, per_pair = W * (H * d + G * d) + W * H * dv, G * (d + dv), 2 * H * (d + dv)
            weights += 0 if f == "sigmoid" else W * G * dv
            weights += W * H * dv if f == "talking" else W * H if f in ("sink", "sigmoid") else 0
            extra = 2.0 * pairs * H * H if f == "talking" else 0.0
        seen = sum(min(o + k, case["window"] + k) if case["window"] else o + k for o, k in zip(old, new))   # cached rows a sequence reads
        return {"bytes": weights * es + rows * W * (es + 4) + (rows + (seen if case["mode"] == "token" else 0)) * row * 4,
                "flops": 2.0 * rows * weights + extra + float(pairs) * per_pair}
    if f == "ssm":
        inner, gn = H * m["vdim"], m["groups"] * m["state"]
        weights, state = W * (2 * inner + 2 * gn + H) + W * inner, H * m["state"] * m["vdim"]
    else:
        d, dv, G = m["dim"], m["vdim"], m.get("kv_heads", H)
        weights, state = W * (2 * G * d + H * dv) + 2 * W * H * dv, H * d * dv
        if f == "delta":
            weights += -W * H * dv + W * (H + 32) + 16 * H * (d + dv)
        elif f == "head_delta":
            weights += 2 * W * H
    return {"bytes": weights * es + rows * W * (es + 4) + n * state * 4 * (2 if case["mode"] == "token" else 1),
            "flops": 2.0 * rows * weights + (6.0 if "delta" in f else 4.0) * rows * state}


def tolerance(case):
    """bf16 products round their inputs (2^-9 each, several in a chain); fp32 layers of the packed decoders are fp32 throughout, fp32
    transformer layers run their products in tf32 with bf16 attention operands."""
    if case["kind"] == "requests":
        return {"rel": 0.025, "max": 0.5}
    if case["kind"] == "block":
        return {"rel": 0.025, "max": 0.5} if case["dtype"] == "bf16" else {"rel": 0.015, "max": 0.3}
    if case["kind"] == "experts":   # a near tie between two experts may go either way and then moves a whole row
        return {"rel": 0.02, "max": 1.0 - 1e-6}
    return {"rel": 0.012, "max": 0.25} if case["dtype"] == "bf16" else {"rel": 2e-5, "max": 1e-3}


# ---- the same in 64 bits, from the equations ----
def f64(t):
    return t.detach().to(torch.float64)


def rms(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def unit(x):
    return x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)


def silu(x):
    return x * torch.sigmoid(x)


def softplus(x):
    return torch.clamp(x, min=0.0) + torch.log1p(torch.exp(-x.abs()))


def frequencies(rot):
    """base^(-2i / dims); with scaling, long waves are divided by the factor, short ones stay, those between are blended."""
    dims, out, sc = rot["dims"], [], rot.get("scaling")
    for i in range(dims // 2):
        f = rot["base"] ** (-2.0 * i / dims)
        if sc:
            wave = 2.0 * math.pi / f
            if wave > sc["original"] / sc["low"]:
                f /= sc["factor"]
            elif wave >= sc["original"] / sc["high"]:
                u = (sc["original"] / wave - sc["low"]) / (sc["high"] - sc["low"])
                f = (1.0 - u) * f / sc["factor"] + u * f
        out.append(f)
    # the frequencies are fp32 constants of the layer, as its positions are whole numbers
    return torch.tensor(out, dtype=torch.float64).to(torch.float32).double().cuda()


def rotate(x, rot, pos, layout):
    """x [T, n, d] at positions pos [T]: the first rot["dims"] entries turn, paired i with i + dims / 2 ("half") or 2i with 2i + 1."""
    half = rot["dims"] // 2
    a = (pos.double()[:, None] * frequencies(rot))[:, None, :]
    c, s, y = torch.cos(a), torch.sin(a), x.clone()
    u, v = (x[..., :half], x[..., half:2 * half]) if layout == "half" else (x[..., 0:2 * half:2], x[..., 1:2 * half:2])
    if layout == "half":
        y[..., :half], y[..., half:2 * half] = u * c - v * s, v * c + u * s
    else:
        y[..., 0:2 * half:2], y[..., 1:2 * half:2] = u * c - v * s, v * c + u * s
    return y


def attend(q, k, v, pos, *, scale, window=0, keep=0, cap=0.0, slopes=None, sink=None, zero_sink=False, talk=None, sigmoid=None):
    """q [T, H, d] at positions pos, k [N, G, d] and v [N, G, dv] at positions 0 .. N - 1 -> [T, H, dv]."""
    H, G = q.shape[1], k.shape[1]
    k, v = k.repeat_interleave(H // G, 1), v.repeat_interleave(H // G, 1)
    s = torch.einsum("thd,jhd->htj", q, k) * scale
    if sigmoid is not None:
        s = s * sigmoid[0][:, None, None] + sigmoid[1][:, None, None]
    if cap:
        s = cap * torch.tanh(s / cap)
    if talk is not None:
        s = torch.einsum("ab,bij->aij", talk, s)
    i, j = pos[:, None], torch.arange(k.shape[0], device="cuda")[None, :]
    if slopes is not None:
        s = s - slopes[:, None, None] * (i - j)
    seen = j <= i
    if window:
        seen = seen & ((i - j < window) | (j < keep))
    if sigmoid is not None:
        return torch.einsum("htj,jhd->thd", torch.where(seen, torch.sigmoid(s), torch.zeros_like(s)), v)
    s = s.masked_fill(~seen, -math.inf)
    end = torch.zeros(H, dtype=torch.float64, device="cuda") if zero_sink else sink
    top = s.max(-1, keepdim=True).values
    if end is not None:
        top = torch.maximum(top, end[:, None, None])
    e = torch.exp(s - top)
    den = e.sum(-1, keepdim=True) + (torch.exp(end[:, None, None] - top) if end is not None else 0.0)
    return torch.einsum("htj,jhd->thd", e / den, v)


def exact_attention(case, seed):
    m, w, batch, pages, h, r = mixer_inputs(case, seed)
    f = case["form"]
    spec = {"pages": (1, m["kv_rank"] + m["rot_dim"], 0) if f == "latent" else (m["kv_heads"], m["dim"], m.get("vdim", m["dim"])), "states": {}}
    view = mixer_state(case, spec, pages, r)
    kp, vp = f64(view.k_pool), None if view.v_pool is None else f64(view.v_pool)
    w, h, H, W = {k: f64(t) for k, t in w.items()}, f64(h), m["heads"], case["width"]
    window, ys, at, page = (m.get("mask") or {}).get("size", 0), [], 0, 0
    slopes = torch.tensor([2.0 ** (-8.0 * (a + 1) / H) for a in range(H)], dtype=torch.float64, device="cuda")
    for n, old in zip(lengths_of(case), starts_of(case)):
        x, pos = h[at:at + n], torch.arange(old, old + n, device="cuda")
        at += n
        count = (old + n + PAGE - 1) // PAGE
        kr, vr = kp[page:page + count].view(-1, *kp.shape[2:]), None if vp is None else vp[page:page + count].view(-1, *vp.shape[2:])
        page += count
        if f == "latent":
            dn, R, dv = m["dim"], m["kv_rank"], m["vdim"]
            d = x @ w["dkv"].T
            kr[old:old + n, 0] = torch.cat([rms(d[:, :R]) * w["dkv.norm"], rotate(d[:, None, R:], m["rot"], pos, "pairs")[:, 0]], 1)
            row = kr[:old + n, 0]
            q = ((rms(x @ w["dq"].T) * w["dq.norm"]) @ w["uq"].T).view(n, H, -1)
            q = torch.cat([q[..., :dn], rotate(q[..., dn:], m["rot"], pos, "pairs")], -1)
            k = torch.cat([(row[:, :R] @ w["uk"].T).view(-1, H, dn), row[:, None, R:].expand(-1, H, -1)], -1)
            o = attend(q, k, (row[:, :R] @ w["uv"].T).view(-1, H, dv), pos, scale=m["scale"], window=window)
            ys.append(o.reshape(n, -1) @ w["o"].T)
            continue
        G, d, bias = m["kv_heads"], m["dim"], lambda name: w.get(name, 0.0)
        q, k = x @ w["q"].T + bias("q.b"), x @ w["k"].T + bias("k.b")
        v = k if f == "sigmoid" else x @ w["v"].T + bias("v.b")
        kw = {}
        if f == "sink":
            q, k = rms(q) * w["q.norm"], rms(k) * w["k.norm"]
            kw = dict(sink=w["sink"], keep=m["mask"]["keep_first"])
        q, k, v = q.view(n, H, d), k.view(n, G, d), v.view(n, G, -1)
        if f == "biased":
            c, every = m["q_temp"]["coef"], m["q_temp"]["every"]
            q, k = rms(q) * (1.0 + c * torch.log(torch.div(pos + 1, every, rounding_mode="floor") + 1.0))[:, None, None], rms(k)
            kw = dict(sink=w["sink"], cap=m["softcap"], slopes=slopes)
        elif f == "sigmoid":
            q, k = rotate(rms(q) * w["q.norm"], m["rot"], pos, "half"), rotate(rms(k) * w["k.norm"], m["rot"], pos, "half")
            kw = dict(sigmoid=(w["temp"], w["pb"]))
        elif f == "talking":
            q, k = rotate(q, m["rot"], pos, "pairs"), rotate(k, m["rot"], pos, "pairs")
            kw = dict(cap=m["softcap"], talk=w["talk"], zero_sink=True)
        kr[old:old + n], vr[old:old + n] = k, v
        o = attend(q, kr[:old + n], vr[:old + n], pos, scale=m["scale"], window=window, **kw)
        if f in ("sink", "sigmoid"):
            o = o * torch.sigmoid(x @ w["g"].T)[:, :, None]
        o = o.reshape(n, -1)
        if f == "talking":
            o = o * torch.sigmoid(x @ w["g"].T)
        ys.append(o @ w["o"].T + bias("o.b"))
    out = {"y": torch.cat(ys), "state": {}, "k": kp}
    if vp is not None:
        out["v"] = vp
    return out


def convolve(x, w, before):
    """Causal depthwise convolution of x [T, C] with w [C, taps] (last column: the token itself); before [taps - 1, C]: the inputs before."""
    taps = w.shape[1]
    xs = torch.cat([before, x])
    return sum(w[:, d] * xs[d:d + x.shape[0]] for d in range(taps))


def scan(q, k, v, g, beta, S, lens, skip=None):
    """S <- g S (+ k u^T with u = beta (v - S^T k), or k v^T without beta), o = S^T q, for n sequences at a time, padded to one length:
    q, k [n, T, H, dk], v [n, T, H, dv], g [n, T, H, dk or 1], beta [n, T, H] or None. Returns (o, S at each sequence's end)."""
    n, T = q.shape[:2]
    out, ends = torch.zeros_like(v), S.clone()
    lens = torch.tensor(lens, device="cuda")
    for t in range(T):
        S = g[:, t, :, :, None] * S
        u = v[:, t]
        if beta is not None:
            u = beta[:, t, :, None] * (u - torch.einsum("nhkv,nhk->nhv", S, k[:, t]))
        S = S + k[:, t, :, :, None] * u[:, :, None, :]
        out[:, t] = torch.einsum("nhkv,nhk->nhv", S, q[:, t])
        ends = torch.where((lens == t + 1)[:, None, None, None], S, ends)
    return out, ends


def pad(parts):
    T = max(p.shape[0] for p in parts)
    return torch.stack([torch.nn.functional.pad(p, [0, 0] * (p.dim() - 1) + [0, T - p.shape[0]]) for p in parts])


def mixed_rows(x, w, m, f, states, i, pos0):
    """The recurrence's inputs of one sequence: (q, k, v, g, beta, what the read-out still needs), its convolutions' states updated."""
    H, n = m["heads"], x.shape[0]
    if f == "lightning":
        q, k, v = (silu(x @ w[a].T).view(n, H, -1) for a in "qkv")
        return q, k, v, torch.tensor(m["decay"], dtype=torch.float32, device="cuda").double()[None, :, None].expand(n, H, 1), None
    taps = m["conv"]

    def ring(xs, rows):
        """Inputs before the portion, oldest first, from a ring by position; the portion's own last inputs enter it."""
        before = torch.stack([rows[(pos0 - d) % taps] if pos0 - d >= 0 else torch.zeros_like(rows[0]) for d in range(taps - 1, 0, -1)])
        for t in range(max(0, n - taps), n):
            rows[(pos0 + t) % taps] = xs[t]
        return before

    if f == "ssm":
        N, dv, G = m["state"], m["vdim"], m["groups"]
        inner = H * dv
        p = x @ w["in"].T
        z, xbc, dt = p[:, :inner], p[:, inner:-H], softplus(p[:, -H:] + w["dt_bias"])
        xbc = silu(convolve(xbc, w["conv"], ring(xbc, states["conv"][i])) + w["conv.b"])
        xs, B, C = xbc[:, :inner].reshape(n, H, dv), xbc[:, inner:inner + G * N].reshape(n, G, N), xbc[:, inner + G * N:].reshape(n, G, N)
        B, C = B.repeat_interleave(H // G, 1), C.repeat_interleave(H // G, 1)
        g = torch.exp(-torch.exp(w["A_log"]) * dt)[:, :, None]
        return C, B * dt[:, :, None], xs, g, None, z
    G, d, dv = m["kv_heads"], m["dim"], m["vdim"]
    raw = [x @ w[a].T for a in "qkv"]
    if f == "head_delta":
        before = ring(torch.cat(raw, 1), states["conv"][i]).split([t.shape[1] for t in raw], 1)
    else:
        before = []
        for a, t in zip("qkv", raw):
            rows = states["conv_" + a][i]   # [channels, taps - 1], oldest first
            before.append(rows.T.clone() if pos0 > 0 else torch.zeros_like(rows.T))
            rows.copy_(torch.cat([before[-1], t])[-(taps - 1):].T)
    q, k, v = (silu(convolve(t, w[a + ".conv"], b)) for a, t, b in zip("qkv", raw, before))
    q, k = unit(q.view(n, G, d)).repeat_interleave(H // G, 1) * d ** -0.5, unit(k.view(n, G, d)).repeat_interleave(H // G, 1)
    beta, A = torch.sigmoid(x @ w["b"].T), torch.exp(w["A_log"])[:, None]
    if f == "head_delta":
        g = torch.exp(-A * softplus(x @ w["a"].T + w["dt_bias"])[:, :, None])
    else:
        g = torch.exp(-A * softplus((x @ w["a1"].T) @ w["a2"].T + w["dt_bias"]).view(n, H, d))
    return q, k, v.view(n, H, dv), g, beta


def read_out(o, x, w, m, f, v=None, z=None):
    """The recurrence's read-outs o [T, H, dv] of one sequence, normed, gated and projected."""
    n = o.shape[0]
    if f == "lightning":
        return (rms(o.reshape(n, -1)) * w["norm"] * torch.sigmoid(x @ w["g"].T)) @ w["o"].T
    if f == "ssm":
        y = (o + w["D"][:, None] * v).reshape(n, -1) * silu(z)
        return (rms(y.view(n, m["norm_groups"], -1)).reshape(n, -1) * w["norm"]) @ w["o"].T
    o = (rms(o) * w["norm"]).reshape(n, -1)
    return (o * (torch.sigmoid((x @ w["g1"].T) @ w["g2"].T) if f == "delta" else silu(x @ w["g"].T))) @ w["o"].T


def recur(parts, S, lens):
    q, k, v, g = (pad([p[a] for p in parts]) for a in range(4))
    return scan(q, k, v, g, None if parts[0][4] is None else pad([p[4] for p in parts]), S, lens)


def exact_recurrence(case, seed):
    m, w, batch, pages, h, r = mixer_inputs(case, seed)
    f = case["form"]
    view = mixer_state(case, MIXERS[f](m, w, EPS, DTYPES[case["dtype"]], True).cache_spec(), pages, r)
    w, h, lens, xs, at = {k: f64(t) for k, t in w.items()}, f64(h), lengths_of(case), [], 0
    states = {k: f64(t) for k, t in view.states.items() if k != "done"}
    for n in lens:
        xs.append(h[at:at + n])
        at += n
    parts = [mixed_rows(x, w, m, f, states, i, p) for i, (x, p) in enumerate(zip(xs, starts_of(case)))]
    S = states["S"] if case["mode"] == "token" else torch.zeros_like(states["S"])
    o, states["S"] = recur(parts, S, lens)
    ys = [read_out(o[i, :n], xs[i], w, m, f, *((parts[i][2], parts[i][5]) if f == "ssm" else ())) for i, n in enumerate(lens)]
    return {"y": torch.cat(ys), "state": states}


def exact_experts(case, seed):
    w, h = expert_inputs(case, seed)
    w, h = {k: f64(t) for k, t in w.items()}, f64(h)
    mlp = lambda x, pre: (silu(x @ w[pre + "gate"].T) * (x @ w[pre + "up"].T)) @ w[pre + "down"].T  # noqa: E731
    s = torch.softmax(h @ w["router"].T, -1)
    idx = (s + w["correction"]).topk(TOP, -1).indices
    wt = torch.zeros_like(s).scatter(1, idx, s.gather(1, idx))
    y = torch.sigmoid(h @ w["shared.sg"].T) * mlp(h, "shared.")
    for e in range(EXPERTS):
        rows = wt[:, e].nonzero()[:, 0]
        y[rows] += wt[rows, e:e + 1] * mlp(h[rows], f"e{e}.")
    return {"y": y, "identity": wt[:, EXPERTS:].sum(1)}


def layer_norm(x, w, b, eps):
    m = x.mean(-1, keepdim=True)
    d = x - m
    return d / torch.sqrt((d * d).mean(-1, keepdim=True) + eps) * w + b


def exact_block(case, seed):
    cfg, layer, x, mask, grad, past = block_inputs(case, seed)
    dt, H, G = x.dtype, cfg.num_attention_heads, cfg.num_key_value_heads
    p = {n: f64(t).requires_grad_(case["mode"] == "train") for n, t in layer.named_parameters()}
    x = f64(x).requires_grad_(case["mode"] == "train")
    B, S, W = x.shape
    start = case["length"] if case["mode"] == "token" else 0
    f = 10000.0 ** (-torch.arange(0, 64, 2, dtype=torch.float64, device="cuda") / 64)
    a = torch.arange(start, start + S, device="cuda").double()[:, None] * f
    cos, sin = a.cos().to(dt).double(), a.sin().to(dt).double()   # the tables are kept in the layer's type

    def turn(t):
        u, v = t[..., :32], t[..., 32:]
        return torch.cat([u * cos - v * sin, v * cos + u * sin], -1)

    lin = lambda t, n: t @ p[n + ".weight"].T + p[n + ".bias"]  # noqa: E731
    heads = lambda t, n: t.view(B, S, n, 64).transpose(1, 2)  # noqa: E731
    q, k, v = turn(heads(lin(x, "attention.query"), H)), turn(heads(lin(x, "attention.key"), G)), heads(lin(x, "attention.value"), G)
    out = {}
    if past is not None:
        kc, vc = f64(past[0]), f64(past[1])
        kc[:, :, start:start + S], vc[:, :, start:start + S] = k, v
        out, k, v = {"k": kc, "v": vc}, kc, vc
    s = q @ k.repeat_interleave(H // G, 1).transpose(2, 3) / 8.0
    if case["mode"] in ("train", "forward"):
        s = s.masked_fill(mask[:, None, None, :] == 0, -math.inf)
    elif case["mode"] == "prompt":
        s = s.masked_fill(torch.ones(S, S, device="cuda").triu(1).bool(), -math.inf)
    o = (torch.softmax(s, -1) @ v.repeat_interleave(H // G, 1)).transpose(1, 2).reshape(B, S, W)
    ln = lambda t, n: layer_norm(t, p[n + ".weight"], p[n + ".bias"], cfg.layer_norm_eps)  # noqa: E731
    y = ln(lin(o, "attention.out.dense") + x, "attention.out.layernorm")
    y = ln(lin(torch.nn.functional.gelu(lin(y, "feed_forward.intermediate")), "feed_forward.out") + x, "feed_forward.layernorm")
    out["y"] = y
    if case["mode"] == "train":
        g = torch.autograd.grad(y, [x] + list(p.values()), f64(grad))
        out["dx"], out["grads"] = g[0], dict(zip(p, g[1:]))
    return out


def exact_requests(case, seed):
    cfg, w, ids = request_inputs(case, seed)
    w = {k: f64(t) for k, t in w.items()}
    ln = lambda x, n: layer_norm(x, w[n], w[n + ".b"], EPS)  # noqa: E731
    n, T = ids.shape
    x = w["embed"][ids]
    pos = torch.arange(T, device="cuda")
    for i, L in enumerate(cfg["layers"]):
        q, m = f"l{i}.mix.", L["mixer"]
        mw = {k[len(q):]: t for k, t in w.items() if k.startswith(q)}
        h, H = ln(x, f"l{i}.norm1"), m["heads"]
        if L["type"] == "delta":
            taps, ch = m["conv"], 2 * m["kv_heads"] * m["dim"] + H * m["vdim"]
            conv = {"conv": torch.zeros((n, taps, ch), dtype=torch.float64, device="cuda")}
            parts = [mixed_rows(h[b], mw, m, "head_delta", conv, b, 0) for b in range(n)]
            o, _ = recur(parts, torch.zeros((n, H, m["dim"], m["vdim"]), dtype=torch.float64, device="cuda"), [T] * n)
            y = torch.stack([read_out(o[b], h[b], mw, m, "head_delta") for b in range(n)])
        else:
            ys = []
            for b in range(n):
                qq, k = (h[b] @ mw["q"].T + mw["q.b"]).view(T, H, -1), (h[b] @ mw["k"].T + mw["k.b"]).view(T, m["kv_heads"], -1)
                turn = lambda t, a: rotate(rms(t) * mw[a], m["rot"], pos, "half")  # noqa: E731
                o = attend(turn(qq, "q.norm"), turn(k, "k.norm"), k, pos, scale=m["scale"], window=m["mask"]["size"], sigmoid=(mw["temp"], mw["pb"]))
                ys.append((o * torch.sigmoid(h[b] @ mw["g"].T)[:, :, None]).reshape(T, -1) @ mw["o"].T)
            y = torch.stack(ys)
        x = x + ln(y, f"l{i}.norm1b")
        h = ln(x, f"l{i}.norm2")
        y = (silu(h @ w[f"l{i}.mlp.gate"].T) * (h @ w[f"l{i}.mlp.up"].T)) @ w[f"l{i}.mlp.down"].T
        x = x + ln(y, f"l{i}.norm2b")
    logits = ln(x[:, case["length"] - 1:], "final.norm") @ w["embed"].T
    return [logits[:, t] for t in range(case["steps"] + 1)]


def exact(case, seed):
    fn = {"block": exact_block, "attention": exact_attention, "recurrence": exact_recurrence, "experts": exact_experts, "requests": exact_requests}[case["kind"]]
    if case["kind"] == "block" and case["mode"] == "train":
        return fn(case, seed)
    with torch.no_grad():
        return fn(case, seed)
