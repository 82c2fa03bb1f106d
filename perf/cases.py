"""Timed cases: the work that programs built on this library ask of it, through its public entry points.

Most cases are steps of the Llama decoder at the layer sizes of the library's own configurations: prompts of a few to
some thousand tokens (``Engine.step`` on freshly acquired slots, the call that a server makes for new requests), decode
steps of 1 to 64 sequences (``Model.forward`` on one token per sequence, captured in a CUDA graph as ``Engine`` itself
does), both storage types. Beside them stand the sampler, a Duzinex decoder with one layer of each of its mixers, and
a layer of routed experts as Gozatar, Kugirax and Luvavik have them.

Weights are N(0, 0.02) with norm weights around 1, token ids uniform over the vocabulary, both from the seed alone.
``exact`` states the same models in plain 64-bit tensor arithmetic.
"""
from __future__ import annotations

import math
import random

import torch

from spissa_b200 import Engine, LlamaConfig, Sampler, SamplingParams
from spissa_b200.config import DuzinexConfig, PartSpec
from spissa_b200.engine import pack_step
from spissa_b200.parts import Runtime, build_part

DEV = "cuda:0"
F64 = torch.float64

LLAMA_1B = dict(hidden_size=2048, num_attention_heads=32, num_key_value_heads=8, head_dim=64, intermediate_size=8192,
                tie_word_embeddings=True, factor=32.0)
LLAMA_8B = dict(hidden_size=4096, num_attention_heads=32, num_key_value_heads=8, head_dim=128, intermediate_size=14336,
                tie_word_embeddings=False, factor=8.0)
SHAPES = {"1b": LLAMA_1B, "8b": LLAMA_8B}
VOCAB = 128256

DUZINEX = dict(width=2048, ff=8192, vocab=32000, eps=1e-6, heads=16, kv_heads=4, dim=64, vdim=128, window=1024, keep_first=4,
               cap=30.0, diff=0.5, ret_heads=8, ret_dim=128, ret_vdim=256)
EXPERTS = dict(width=2048, ff=2048, experts=32, top=4, groups=4, keep=2, limit=7.0, slope=1.702)


# ---------------------------------------------------------------------------------------------------------- the cases
def prompt(name, shape, layers, tokens, seqs, dtype="bfloat16"):
    return dict(name=name, kind="prompt", shape=shape, layers=layers, tokens=tokens, seqs=seqs, dtype=dtype)


def decode(name, shape, layers, batch, context, dtype="bfloat16"):
    return dict(name=name, kind="decode", shape=shape, layers=layers, batch=batch, context=context, dtype=dtype)


def listed():
    return [
        # a chat turn: a few dozen new tokens of one user, where the time to the first token is all latency
        prompt("prompt_40", "1b", 16, 40, 1),
        # three requests of unequal length that arrive together, some hundred tokens in all
        prompt("prompt_ragged_301", "1b", 16, 301, 3),
        # one document-sized prompt: the headline prompt workload
        prompt("prompt_2048", "1b", 16, 2048, 1),
        # a long document through layers of the 8B shape (heads of 128)
        prompt("prompt_8b_6000", "8b", 4, 6000, 1),
        # one user's decode step behind a prompt of 2,048 tokens: the smallest call a server makes
        decode("decode_1", "1b", 16, 1, 2048),
        # the headline decode workload
        decode("decode_8", "1b", 16, 8, 2048),
        # a full server
        decode("decode_64", "1b", 8, 64, 2048),
        # the true 32-bit mode, in which traces are replayed and compared: a prompt, and decode steps
        prompt("prompt_fp32_500", "1b", 4, 500, 1, "float32"),
        decode("decode_fp32_4", "1b", 4, 4, 500, "float32"),
        # the draw of every generated token that is not greedy: temperature and nucleus over the whole vocabulary
        dict(name="sample_8", kind="sample", rows=8, vocab=VOCAB),
        # another architecture's prompt: one layer each of retention, gated recurrence and differential attention
        dict(name="duzinex_prompt_2000", kind="duzinex", tokens=2000, dtype="bfloat16"),
        # routed experts of a prompt: 4 of 32 experts a token and a shared one
        dict(name="experts_2048", kind="experts", tokens=2048, dtype="bfloat16"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choice(["prompt", "prompt", "prompt", "prompt_8b", "decode", "decode", "decode", "prompt32", "decode32", "sample",
                       "duzinex", "experts"])
    if kind == "prompt":
        tokens = _log(rng, 2, 2048)
        c = prompt("", "1b", 16, tokens, rng.randint(1, min(8, tokens)))
    elif kind == "prompt_8b":
        c = prompt("", "8b", 4, _log(rng, 300, 6000), rng.randint(1, 3))
    elif kind == "decode":
        c = decode("", "1b", 8, _log(rng, 1, 64), _log(rng, 100, 2048))
    elif kind == "prompt32":
        c = prompt("", "1b", 4, _log(rng, 20, 500), rng.randint(1, 3), "float32")
    elif kind == "decode32":
        c = decode("", "1b", 4, rng.randint(1, 8), _log(rng, 50, 600), "float32")
    elif kind == "sample":
        c = dict(kind="sample", rows=_log(rng, 1, 64), vocab=rng.choice([VOCAB, 32000, 50257]))
    elif kind == "duzinex":
        c = dict(kind="duzinex", tokens=_log(rng, 100, 2048), dtype="bfloat16")
    else:
        c = dict(kind="experts", tokens=_log(rng, 1, 2048), dtype="bfloat16")
    c.pop("name", None)
    return c


# ------------------------------------------------------------------------------------------------------------- inputs
class Source:
    """Random tensors and token ids from one seed."""

    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV)
        self.gen.manual_seed(1000003 * int(seed) + 17)
        self.host = random.Random(1000003 * int(seed) + 29)

    def normal(self, *shape, std=0.02, mean=0.0, dtype=torch.bfloat16):
        t = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(mean, std, generator=self.gen)
        return t.to(dtype)

    def ids(self, n, vocab):
        return [self.host.randrange(vocab) for _ in range(n)]


def torch_dtype(case):
    return getattr(torch, case["dtype"])


def llama_config(case):
    s = SHAPES[case["shape"]]
    return LlamaConfig.from_dict(dict(
        architectures=["LlamaForCausalLM"], model_type="llama", num_hidden_layers=case["layers"], vocab_size=VOCAB,
        rope_theta=500000.0, rms_norm_eps=1e-5, max_position_embeddings=131072,
        rope_scaling=dict(rope_type="llama3", factor=s["factor"], low_freq_factor=1.0, high_freq_factor=4.0,
                          original_max_position_embeddings=8192),
        **{k: v for k, v in s.items() if k != "factor"}))


def llama_tensors(case, src):
    s, dt = SHAPES[case["shape"]], torch_dtype(case)
    H, I, hd = s["hidden_size"], s["intermediate_size"], s["head_dim"]
    nh, nkv = s["num_attention_heads"], s["num_key_value_heads"]
    t = {"model.embed_tokens.weight": src.normal(VOCAB, H, dtype=dt)}
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        for name, shape in (("self_attn.q_proj", (nh * hd, H)), ("self_attn.k_proj", (nkv * hd, H)),
                            ("self_attn.v_proj", (nkv * hd, H)), ("self_attn.o_proj", (H, nh * hd)),
                            ("mlp.gate_proj", (I, H)), ("mlp.up_proj", (I, H)), ("mlp.down_proj", (H, I))):
            t[p + name + ".weight"] = src.normal(*shape, dtype=dt)
        for name in ("input_layernorm", "post_attention_layernorm"):
            t[p + name + ".weight"] = src.normal(H, std=0.1, mean=1.0, dtype=dt)
    t["model.norm.weight"] = src.normal(H, std=0.1, mean=1.0, dtype=dt)
    if not s["tie_word_embeddings"]:
        t["lm_head.weight"] = src.normal(VOCAB, H, dtype=dt)
    return t


def lengths_of(total, seqs):
    """``total`` tokens over ``seqs`` sequences of unequal length, each at least one."""
    r = random.Random(total * 131 + seqs)
    w = [r.uniform(0.3, 1.0) for _ in range(seqs)]
    out = [max(1, int(total * x / sum(w))) for x in w]
    out[-1] += total - sum(out)
    if out[-1] < 1:
        out[out.index(max(out))] += out[-1] - 1
        out[-1] = 1
    return out


def contexts_of(case):
    """The cached length of each sequence of a decode step: around ``context``."""
    r = random.Random(case["context"] * 131 + case["batch"])
    return [max(1, int(case["context"] * r.uniform(0.8, 1.1))) for _ in range(case["batch"])] if case["batch"] > 1 else [case["context"]]


def llama_inputs(case, seed):
    """(weights, token ids of each sequence)"""
    src = Source(seed)
    tensors = llama_tensors(case, src)
    if case["kind"] == "prompt":
        counts = lengths_of(case["tokens"], case["seqs"])
    else:
        counts = [n + 1 for n in contexts_of(case)]                 # the cached ones and the step's own
    return tensors, [src.ids(n, VOCAB) for n in counts]


def duzinex_config():
    z = DUZINEX
    att = dict(type="attention", mixer=dict(heads=z["heads"], kv_heads=z["kv_heads"], dim=z["dim"], vdim=z["vdim"], diff=z["diff"],
                                            scale=z["dim"] ** -0.5, softcap=z["cap"],
                                            mask=dict(size=z["window"], keep_first=z["keep_first"]),
                                            rot=dict(dims=z["dim"], base=10000.0)))
    ret = dict(type="retention", mixer=dict(heads=z["ret_heads"], dim=z["ret_dim"], vdim=z["ret_vdim"],
                                            decay=[1.0 - 2.0 ** (-5 - i % 4) for i in range(z["ret_heads"])]))
    gru = dict(type="mingru", mixer=dict(width=z["width"]))
    mlp = dict(kind="dense", ff=z["ff"])
    return dict(architecture="Duzinex", vocab=z["vocab"], width=z["width"], embedding=dict(scale=z["width"] ** 0.5),
                norm=dict(eps=z["eps"]), layers=[dict(layer, mlp=mlp) for layer in (ret, gru, att)])


def duzinex_inputs(case, seed):
    src, z, dt = Source(seed), DUZINEX, torch_dtype(case)
    W, ff = z["width"], z["ff"]
    t = {"embed": src.normal(z["vocab"], W, dtype=dt)}

    def norm(name):
        t[name] = src.normal(W, std=0.1, mean=1.0, dtype=dt)
        t[name + ".b"] = src.normal(W, dtype=dt)
        t[name + ".alpha"] = torch.full((), 0.5, dtype=dt, device=DEV)

    rh, rd, rv, h, g, d, vd = (z[k] for k in ("ret_heads", "ret_dim", "ret_vdim", "heads", "kv_heads", "dim", "vdim"))
    mixers = [dict(q=(rh * rd, W), k=(rh * rd, W), v=(rh * rv, W), g=(rh * rv, W), o=(W, rh * rv)),
              dict(z=(W, W), x=(W, W), g=(W, W), o=(W, W)),
              dict(q=(h * 2 * d, W), k=(g * 2 * d, W), v=(g * vd, W), o=(W, h * vd))]
    biases = [(), ("z", "x"), ("q", "k", "v", "o")]
    for i, (shapes, with_bias) in enumerate(zip(mixers, biases)):
        p = f"l{i}."
        norm(p + "norm1")
        norm(p + "norm2")
        t[p + "shift"] = src.normal(W, std=0.2, mean=0.3, dtype=dt)
        for k, shape in shapes.items():
            t[p + "mix." + k] = src.normal(*shape, dtype=dt)
            if k in with_bias:
                t[p + "mix." + k + ".b"] = src.normal(shape[0], dtype=dt)
        t[p + "mlp.up"], t[p + "mlp.down"] = src.normal(ff, W, dtype=dt), src.normal(W, ff, dtype=dt)
        t[p + "mlp.act"] = src.normal(4, std=0.1, mean=0.5, dtype=dt)
    for k in ("lq1", "lk1", "lq2", "lk2"):
        t["l2.mix." + k] = src.normal(d, std=0.1, dtype=dt)
    norm("final.norm")
    return t, src.ids(case["tokens"], z["vocab"])


def experts_inputs(case, seed):
    src, z, dt = Source(seed), EXPERTS, torch_dtype(case)
    W, ff = z["width"], z["ff"]
    t = {"router": src.normal(z["experts"], W, dtype=dt), "correction": src.normal(z["experts"], dtype=dt)}
    for p in [f"e{i}." for i in range(z["experts"])] + ["shared."]:
        t[p + "gate"], t[p + "up"] = src.normal(ff, W, dtype=dt), src.normal(ff, W, dtype=dt)
        t[p + "down"] = src.normal(W, ff, dtype=dt)
    return t, src.normal(case["tokens"], W, std=1.0, dtype=dt)


def sample_inputs(case, seed):
    """Logits as a language model leaves them: a wide floor and some dozens of likely tokens in each row."""
    src = Source(seed)
    logits = src.normal(case["rows"], case["vocab"], std=1.5, dtype=torch.float32)
    for r in range(case["rows"]):
        at = torch.tensor(src.ids(40, case["vocab"]), device=DEV)
        logits[r, at] += torch.linspace(2.0 + 8.0 * src.host.random(), 0.0, 40, device=DEV)
    return logits


# ------------------------------------------------------------------------------------------------------------ running
def prepare(case, seed):
    if case["kind"] == "sample":
        return dict(case=case, logits=sample_inputs(case, seed), sampler=Sampler(DEV),
                    params=SamplingParams(temperature=0.8, top_p=0.95, seed=seed), step=0)
    if case["kind"] == "experts":
        tensors, x = experts_inputs(case, seed)
        z = EXPERTS
        shared = PartSpec("clamped_glu", dict(hidden_size=z["width"], intermediate_size=z["ff"], limit=z["limit"], slope=z["slope"]),
                          prefix="shared.")
        part = build_part("ffn", PartSpec("routed_experts", dict(
            hidden_size=z["width"], intermediate_size=z["ff"], experts=z["experts"], top=z["top"], limit=z["limit"],
            slope=z["slope"], groups=z["groups"], keep_groups=z["keep"], shared=shared)))
        part.bind_all(tensors, Runtime(torch.device(DEV), torch_dtype(case)))
        return dict(case=case, part=part, x=x)
    if case["kind"] == "duzinex":
        tensors, ids = duzinex_inputs(case, seed)
        engine = Engine(DuzinexConfig.from_dict(duzinex_config()), tensors, case["dtype"], case["tokens"] + 64, 2, DEV)
        return dict(case=case, engine=engine, prompts=[ids])
    tensors, seqs = llama_inputs(case, seed)
    room = sum(-(-(len(s) + 1) // 64) * 64 for s in seqs)
    engine = Engine(llama_config(case), tensors, case["dtype"], room, len(seqs), DEV)
    del tensors
    if case["kind"] == "prompt":
        return dict(case=case, engine=engine, prompts=seqs)
    # a decode step: the sequences' earlier tokens go into the cache, then the step is captured as ``Engine`` does it
    slots = [engine.acquire() for _ in seqs]
    for at in range(0, len(slots), 4):
        engine.step([(slot, s[:-1], []) for slot, s in zip(slots[at:at + 4], seqs[at:at + 4])])
    cached = [engine.length(slot) for slot in slots]
    pages = engine.cache.reserve([(slot, 1) for slot in slots])
    batch = pack_step([(slot, s[-1:], [0]) for slot, s in zip(slots, seqs)], cached, pages.tables, torch.device(DEV))
    engine.model.forward(batch, engine.cache)                        # plans are made and kernels loaded outside the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        logits = engine.model.forward(batch, engine.cache)
    return dict(case=case, engine=engine, batch=batch, graph=graph, logits=logits, pages=pages)


def run(state):
    kind = state["case"]["kind"]
    if kind == "decode":
        state["graph"].replay()
        return state["logits"]
    if kind == "sample":
        rows = state["logits"].shape[0]
        return state["sampler"].sample(state["logits"], state["params"], list(range(rows)), state["step"])
    if kind == "experts":
        x = state["x"]
        y = torch.zeros(x.shape, dtype=torch.float32, device=x.device)
        state["part"].forward(x, None, y)
        return y
    engine = state["engine"]
    slots = [engine.acquire() for _ in state["prompts"]]
    logits = engine.step([(slot, ids, [len(ids) - 1]) for slot, ids in zip(slots, state["prompts"])])
    for slot in slots:
        engine.release(slot)
    return logits


# --------------------------------------------------------------------------------------------- the least work of a pass
def work(case):
    if case["kind"] == "sample":
        n = case["rows"] * case["vocab"]
        return dict(bytes=4 * n + 4 * case["rows"], flops=4 * n)     # every logit once: scaled, exponentiated, summed
    eb = 2 if case["dtype"] == "bfloat16" else 4
    if case["kind"] == "experts":
        z, T = EXPERTS, case["tokens"]
        one = 3 * z["width"] * z["ff"]
        touched = z["experts"] * (1.0 - (1.0 - z["top"] / z["experts"]) ** T)         # experts that some token chose
        return dict(bytes=eb * (one * (touched + 1) + z["width"] * (z["experts"] + T)) + 4 * z["width"] * T,
                    flops=2.0 * T * (one * (z["top"] + 1) + z["width"] * z["experts"]))
    if case["kind"] == "duzinex":
        z, T = DUZINEX, case["tokens"]
        W, C = z["width"], 1
        ret = 2 * W * z["ret_heads"] * (z["ret_dim"] + z["ret_vdim"]) + W * z["ret_heads"] * z["ret_vdim"]
        gru = 4 * W * W
        att = W * (z["heads"] * (2 * z["dim"] + z["vdim"]) + z["kv_heads"] * (2 * z["dim"] + z["vdim"]))
        params = ret + gru + att + 3 * 2 * W * z["ff"]
        seen = sum(min(t + 1, z["window"] + z["keep_first"]) for t in range(T))
        flops = 2.0 * T * params + seen * z["heads"] * 2.0 * (2 * z["dim"] + 2 * z["vdim"]) \
            + 4.0 * T * z["ret_heads"] * z["ret_dim"] * z["ret_vdim"] + 2.0 * C * W * z["vocab"]
        state = 4 * (z["ret_heads"] * z["ret_dim"] * z["ret_vdim"] + 4 * W)
        cache = eb * T * z["kv_heads"] * (2 * z["dim"] + z["vdim"])
        return dict(bytes=eb * (params + W * (z["vocab"] + T)) + cache + state + 4 * z["vocab"], flops=flops)
    s = SHAPES[case["shape"]]
    H, hd, nh, nkv, L = s["hidden_size"], s["head_dim"], s["num_attention_heads"], s["num_key_value_heads"], case["layers"]
    layer = 2 * H * nh * hd + 2 * H * nkv * hd + 3 * H * s["intermediate_size"]
    if case["kind"] == "prompt":
        counts = lengths_of(case["tokens"], case["seqs"])
        new, pairs, wanted, read = sum(counts), sum(n * (n + 1) / 2 for n in counts), len(counts), 0
    else:
        counts = contexts_of(case)
        new, pairs, wanted, read = len(counts), sum(n + 1 for n in counts), len(counts), sum(counts)
    row = 2 * nkv * hd * L * eb                                      # a position's keys and values in all layers
    return dict(bytes=eb * (layer * L + H * (VOCAB + new)) + row * (new + read) + 4 * VOCAB * wanted,
                flops=2.0 * new * layer * L + 4.0 * pairs * nh * hd * L + 2.0 * wanted * H * VOCAB)


# ----------------------------------------------------------------------------------------------------------- tolerance
def tolerance(case):
    if case["kind"] == "sample":
        return "exact"                                               # token ids
    if case["kind"] == "experts":
        return dict(rel=7e-3, max=0.1)                               # one layer: 1.7e-3 from the exact result
    if case["kind"] == "duzinex":
        return dict(rel=1.8e-2, max=0.2)                             # three layers: 4.4e-3
    if case["dtype"] == "float32":
        return dict(rel=3e-5, max=6e-4)                              # 4e-6 to 7e-6, the rotation's angles included
    return dict(rel=3e-2, max=0.4)                                   # 4 to 16 layers in 16 bits: 9e-3 to 1.8e-2


# --------------------------------------------------------------------------- the same in 64 bits, plain tensor arithmetic
def rms(v, eps):
    return v / torch.sqrt((v * v).mean(dim=-1, keepdim=True) + eps)


def silu(v):
    return v * torch.sigmoid(v)


def rope_frequencies(case):
    s = SHAPES[case["shape"]]
    hd, n0, low, high = s["head_dim"], 8192.0, 1.0, 4.0
    freq = 1.0 / torch.pow(torch.tensor(500000.0), torch.arange(0, hd, 2, dtype=torch.float32) / hd)     # a 32-bit table
    lam = 2.0 * math.pi / freq
    smooth = (n0 / lam - low) / (high - low)
    mid = (1.0 - smooth) * freq / s["factor"] + smooth * freq
    out = torch.where(lam > n0 / low, freq / s["factor"], freq)
    return torch.where((lam <= n0 / low) & (lam >= n0 / high), mid, out).to(DEV, F64)


def rotate_halves(v, angle):
    """v [T, heads, d]: dim i turns with dim i + d/2."""
    c, s = torch.cos(angle)[:, None, :], torch.sin(angle)[:, None, :]
    a, b = v.chunk(2, dim=-1)
    return torch.cat([a * c - b * s, b * c + a * s], dim=-1)


def llama_exact(case, tensors, ids):
    """Logits of the last token."""
    s = SHAPES[case["shape"]]
    hd, nh, nkv, eps = s["head_dim"], s["num_attention_heads"], s["num_key_value_heads"], 1e-5
    w = lambda name: tensors[name + ".weight"].to(F64)               # noqa: E731
    T = len(ids)
    x = tensors["model.embed_tokens.weight"][torch.tensor(ids, device=DEV)].to(F64)
    angle = torch.arange(T, dtype=F64, device=DEV)[:, None] * rope_frequencies(case)[None, :]
    hidden = torch.ones(T, T, dtype=torch.bool, device=DEV).triu(1)
    for i in range(case["layers"]):
        p = f"model.layers.{i}."
        a = rms(x, eps) * w(p + "input_layernorm")
        q = rotate_halves((a @ w(p + "self_attn.q_proj").T).view(T, nh, hd), angle)
        k = rotate_halves((a @ w(p + "self_attn.k_proj").T).view(T, nkv, hd), angle)
        v = (a @ w(p + "self_attn.v_proj").T).view(T, nkv, hd)
        o = torch.empty(T, nh, hd, dtype=F64, device=DEV)
        for h in range(nh):
            g = h // (nh // nkv)
            sc = ((q[:, h] @ k[:, g].T) / math.sqrt(hd)).masked_fill_(hidden, float("-inf"))
            o[:, h] = torch.softmax(sc, dim=-1) @ v[:, g]
        x = x + o.view(T, nh * hd) @ w(p + "self_attn.o_proj").T
        a = rms(x, eps) * w(p + "post_attention_layernorm")
        x = x + (silu(a @ w(p + "mlp.gate_proj").T) * (a @ w(p + "mlp.up_proj").T)) @ w(p + "mlp.down_proj").T
    last = rms(x[-1:], eps) * w("model.norm")
    return last @ w("model.embed_tokens" if s["tie_word_embeddings"] else "lm_head").T


def duzinex_exact(case, tensors, ids):
    z, T = DUZINEX, len(ids)
    eps = z["eps"]
    w = {k: v.to(F64) for k, v in tensors.items() if k != "embed"}
    embed = tensors["embed"].to(F64)
    x = embed[torch.tensor(ids, device=DEV)] * z["width"] ** 0.5
    i = torch.arange(T, device=DEV)

    def norm(v, name):
        return torch.tanh(w[name + ".alpha"] * v) * w[name] + w[name + ".b"]

    def retention(a, p):
        H, d, vd = z["ret_heads"], z["ret_dim"], z["ret_vdim"]
        q, k = (a @ w[p + "q"].T).view(T, H, d), (a @ w[p + "k"].T).view(T, H, d) / math.sqrt(d)
        v = (a @ w[p + "v"].T).view(T, H, vd)
        dist = (i[:, None] - i[None, :]).to(F64)
        out = []
        for h in range(H):
            g = 1.0 - 2.0 ** (-5 - h % 4)
            keep = torch.where(dist >= 0, torch.pow(torch.tensor(g, dtype=F64, device=DEV), dist.clamp(min=0)), torch.zeros_like(dist))
            out.append(rms(((q[:, h] @ k[:, h].T) * keep) @ v[:, h], eps))
        return (torch.cat(out, dim=-1) * silu(a @ w[p + "g"].T)) @ w[p + "o"].T

    def mingru(a, p):
        gate = torch.sigmoid(a @ w[p + "z"].T + w[p + "z.b"])
        u = a @ w[p + "x"].T + w[p + "x.b"]
        cand = torch.where(u >= 0, u + 0.5, torch.sigmoid(u))
        s, rows = torch.zeros_like(cand[0]), torch.empty_like(cand)
        for t in range(T):
            s = (1.0 - gate[t]) * s + gate[t] * cand[t]
            rows[t] = s
        return (rows * silu(a @ w[p + "g"].T)) @ w[p + "o"].T

    def attention(a, p):
        H, G, d, vd = z["heads"], z["kv_heads"], z["dim"], z["vdim"]
        freq = 10000.0 ** (-2.0 * torch.arange(d // 2, dtype=F64, device=DEV) / d)
        c, s = (f(i.to(F64)[:, None] * freq)[:, None, None, :] for f in (torch.cos, torch.sin))

        def turn(v):                                                 # neighbouring dims turn together
            even, odd = v[..., 0::2], v[..., 1::2]
            return torch.stack([even * c - odd * s, odd * c + even * s], dim=-1).flatten(-2)

        q = turn((a @ w[p + "q"].T + w[p + "q.b"]).view(T, H, 2, d))
        k = turn((a @ w[p + "k"].T + w[p + "k.b"]).view(T, G, 2, d))
        v = (a @ w[p + "v"].T + w[p + "v.b"]).view(T, G, vd)
        see = (i[None, :] <= i[:, None]) & ((i[:, None] - i[None, :] < z["window"]) | (i[None, :] < z["keep_first"]))
        lam = torch.exp((w[p + "lq1"] * w[p + "lk1"]).sum()) - torch.exp((w[p + "lq2"] * w[p + "lk2"]).sum()) + z["diff"]
        heads = []
        for h in range(H):
            g, maps = h // (H // G), []
            for m in range(2):
                sc = z["cap"] * torch.tanh((q[:, h, m] @ k[:, g, m].T) * d ** -0.5 / z["cap"])
                maps.append(torch.softmax(sc.masked_fill(~see, float("-inf")), dim=-1) @ v[:, g])
            heads.append(rms(maps[0] - lam * maps[1], eps) * (1.0 - z["diff"]))
        return torch.cat(heads, dim=-1) @ w[p + "o"].T + w[p + "o.b"]

    for layer, mixer in enumerate((retention, mingru, attention)):
        p = f"l{layer}."
        a = norm(x, p + "norm1")
        before = torch.cat([torch.zeros_like(a[:1]), a[:-1]], dim=0)
        x = x + mixer(a + (before - a) * w[p + "shift"], p + "mix.")
        u = norm(x, p + "norm2") @ w[p + "mlp.up"].T
        c = w[p + "mlp.act"]
        x = x + (c[0] * rms(u, eps) + c[1] * rms(u * u, eps) + c[2] * rms(u * u * u, eps) + c[3]) @ w[p + "mlp.down"].T
    return norm(x[-1:], "final.norm") @ embed.T


def experts_exact(case, tensors, x):
    z = EXPERTS
    w = lambda name: tensors[name].to(F64)                           # noqa: E731
    x = x.to(F64)
    T, E = x.shape[0], z["experts"]

    def unit(p, v):
        g = (v @ w(p + "gate").T).clamp(max=z["limit"])
        u = (v @ w(p + "up").T).clamp(-z["limit"], z["limit"])
        return (g * torch.sigmoid(z["slope"] * g) * (u + 1.0)) @ w(p + "down").T

    score = torch.sigmoid(x @ w("router").T)
    choice = score + w("correction")
    groups = choice.view(T, z["groups"], E // z["groups"])
    best = groups.topk(2, dim=-1).values.sum(dim=-1).topk(z["keep"], dim=-1).indices
    allowed = torch.zeros(T, z["groups"], dtype=torch.bool, device=DEV).scatter_(1, best, True)
    allowed = allowed[:, :, None].expand_as(groups).reshape(T, E)
    ids = choice.masked_fill(~allowed, float("-inf")).topk(z["top"], dim=-1).indices
    weight = score.gather(1, ids)
    weight = weight / (weight.sum(dim=-1, keepdim=True) + 1e-20)
    y = unit("shared.", x)
    for e in range(E):
        rows, place = (ids == e).nonzero(as_tuple=True)
        if rows.numel():
            y[rows] += weight[rows, place][:, None] * unit(f"e{e}.", x[rows])
    return y


def exact(case, seed):
    if case["kind"] == "sample":
        return None                                                  # tokens, no computed numbers
    with torch.no_grad():
        if case["kind"] == "experts":
            return experts_exact(case, *experts_inputs(case, seed))
        if case["kind"] == "duzinex":
            tensors, ids = duzinex_inputs(case, seed)
            return duzinex_exact(case, tensors, ids)
        tensors, seqs = llama_inputs(case, seed)
        return torch.cat([llama_exact(case, tensors, ids) for ids in seqs])
