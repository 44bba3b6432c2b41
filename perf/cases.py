"""What the framework is timed on: prompts going through `DecodeEngine.feed` and decode steps
through `DecodeEngine.step`, for the three decoders it serves.

A case is a model (family and size; the layers are those of a real size, their number is cut and
the vocabulary is small), its type and page layout, and a batch of sequences:

  phase "prefill"  every sequence is opened, its prompt is fed in portions of at most `portion`
                   tokens, its last logits come back to the host, and it is finished: what a
                   server does until a request's first token
  phase "decode"   one step of a running batch whose contexts are in the cache: host arrays,
                   their copy, the CUDA graph, the token ids back on the host

Weights are random, of the size that keeps activations near one.  The head is a scaled copy of the
embedding, so a sequence goes on repeating its last token with a wide margin: greedy tokens do not
hang on rounding, and the batch keeps as many different tokens as it has sequences.
"""
from __future__ import annotations

import math
import random

import torch

from fastkernels_b200.candidate.L4.llama import LlamaConfig
from fastkernels_b200.engine import DecodeEngine
from fastkernels_b200.models.mixers import Yarn
from fastkernels_b200.models.pinuvik import PinuvikConfig, PinuvikLayer
from fastkernels_b200.models.rivilix import (Bigram, DenseConfig, ExpertsConfig, LatentConfig,
                                             MatrixMemoryConfig, RivilixConfig, RivilixLayer)
from fastkernels_b200.models.weights import DictSource

VOCAB = 32768
EPS = 1e-6
THETA = 1e6
SOFTCAP = 30.0
DEVICE = "cuda"
# decode steps after which a sequence is done and the next request takes its place
REPLY = 48

# the sizes of the models' own benchmark; "layers" is the cut
SIZES = {
    "1b": dict(layers=8, width=2048, ff=6144, heads=16, kv=4, dim=128, chunk=1024,
               delta=(32, 64), rank=64),
    "3b": dict(layers=6, width=3072, ff=8192, heads=48, kv=12, dim=64, chunk=2048,
               delta=(24, 128), rank=64),
    "8b": dict(layers=4, width=4096, ff=12288, heads=32, kv=8, dim=128, chunk=2048,
               delta=(64, 64), rank=96),
}
# latent: heads, unrotated, rotated, value channels, rank; memory: heads, dim, vdim;
# experts: number, chosen, ff, shared ff
RIVILIX = {
    "1b": dict(layers=8, width=2048, ff=6144, latent=(16, 96, 32, 128, 512),
               memory=(8, 128, 256), experts=(32, 4, 1024, 2048)),
    "3b": dict(layers=8, width=2560, ff=6400, latent=(40, 64, 32, 64, 256),
               memory=(10, 128, 256), experts=(16, 2, 1600, 1600)),
    "8b": dict(layers=4, width=4096, ff=12288, latent=(32, 96, 32, 128, 512),
               memory=(16, 128, 256), experts=(64, 6, 1408, 2816)),
}


def case(name, family, size, phase, sequences, shortest, longest, portion=8192, dtype="bfloat16",
         layout="NHD", page=64):
    c = dict(family=family, size=size, phase=phase, sequences=sequences, shortest=shortest,
             longest=longest, portion=portion, dtype=dtype, layout=layout, page=page)
    return dict(c, name=name) if name else c


def listed():
    return [
        # first token of one short prompt: nothing but launches and weights
        case("llama-1b prompt 1x61", "llama", "1b", "prefill", 1, 61, 61),
        # one user's reply: latency of a step that streams the weights once
        case("llama-1b step 1", "llama", "1b", "decode", 1, 777, 777),
        # a full serving batch with long, mixed contexts: the KV cache is most of the bytes
        case("llama-8b step 64 long", "llama", "8b", "decode", 64, 1024, 8192, page=256),
        # a half-full batch on the 16-token head-major pages of the serving engine's default
        case("llama-8b step 23 HND", "llama", "8b", "decode", 23, 300, 3000, layout="HND",
             page=16),
        # a long document
        case("llama-8b prompt 1x8192", "llama", "8b", "prefill", 1, 8192, 8192),
        # a burst of chat prompts of every length, portions as a server cuts them
        case("llama-1b prompts 24 mixed", "llama", "1b", "prefill", 24, 17, 1500, portion=4096),
        # the second decoder: steps of a small batch, then prompts longer than its chunks
        case("pinuvik-1b step 16", "pinuvik", "1b", "decode", 16, 900, 1900),
        case("pinuvik-8b prompts 5", "pinuvik", "8b", "prefill", 5, 700, 2500),
        # the third decoder: a small batch, a full batch that visits every expert, prompts
        case("rivilix-1b step 9", "rivilix", "1b", "decode", 9, 200, 1500),
        case("rivilix-8b step 64", "rivilix", "8b", "decode", 64, 500, 2000),
        case("rivilix-8b prompts 8", "rivilix", "8b", "prefill", 8, 600, 1500),
        # true fp32, the type in which given traces are replayed for comparison
        case("rivilix-1b prompts 3 fp32", "rivilix", "1b", "prefill", 3, 40, 333,
             dtype="float32"),
    ]


def draw(rng):
    """Families, sizes, phases, types and page layouts of the list; lengths and numbers of
    sequences over their logarithm."""
    def between(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    family = rng.choice(["llama", "llama", "pinuvik", "rivilix"])
    size = rng.choice(sorted(SIZES))
    phase = rng.choice(["prefill", "decode"])
    dtype = "float32" if family != "llama" and phase == "prefill" and rng.random() < 0.2 \
        else "bfloat16"
    layout, page = ("NHD", 64) if family != "llama" else \
        rng.choice([("NHD", 64), ("NHD", 256), ("HND", 16)])
    # tokens: at most what the largest prefill and decode of the list have
    if dtype == "float32":
        n = between(1, 4)
        longest = between(17, 1000 // n)
    elif phase == "prefill":
        n = between(1, 32)
        longest = between(16, 7800 // n)
    else:
        n = between(1 if family == "llama" else 4, 64)
        longest = between(100, 6000 if family == "llama" else 2500)
    portion = rng.choice([1024, 4096, 8192])
    return case(None, family, size, phase, n, max(1, int(longest * rng.uniform(0.2, 1.0))),
                longest, portion, dtype, layout, page)


def lengths(c):
    """Context or prompt lengths: the longest, and others down to the shortest."""
    r = random.Random(1000 * c["longest"] + c["sequences"])
    return [c["longest"]] + [r.randint(c["shortest"], c["longest"])
                             for _ in range(c["sequences"] - 1)]


# ------------------------------------------------------------------------------ models
def rivilix_layers(z):
    """Every fourth layer is a memory; half of them hold experts."""
    kinds = [("memory", "ff"), ("latent", "experts"), ("latent", "ff"), ("latent", "experts")]
    return [kinds[i % 4] for i in range(z["layers"])]


def config(c):
    longest = max(lengths(c)) + REPLY + 2
    dtype = getattr(torch, c["dtype"])
    z = (RIVILIX if c["family"] == "rivilix" else SIZES)[c["size"]]
    if c["family"] == "llama":
        scale = 128 // z["dim"]             # this decoder has heads of 128 channels
        return LlamaConfig(
            hidden_size=z["width"], intermediate_size=z["ff"], num_hidden_layers=z["layers"],
            num_attention_heads=z["heads"] // scale, num_key_value_heads=z["kv"] // scale,
            head_dim=128, vocab_size=VOCAB, max_position_embeddings=longest, rms_norm_eps=EPS,
            rope_theta=THETA, qk_norm=True, kv_block_size=c["page"], kv_layout=c["layout"],
            dtype=dtype)
    if c["family"] == "pinuvik":
        return PinuvikConfig(
            vocab_size=VOCAB, hidden_size=z["width"], eps=EPS, dtype=dtype,
            kv_block_size=c["page"],
            layers=[PinuvikLayer(z["heads"], z["kv"], z["dim"], z["dim"] ** -0.5, z["chunk"],
                                 z["dim"], THETA, *z["delta"], z["rank"], z["ff"])
                    for _ in range(z["layers"])])
    h, dim, rot, vdim, rank = z["latent"]
    mixers = {"memory": MatrixMemoryConfig(*z["memory"], 15.0),
              "latent": LatentConfig(h, dim, rot, vdim, rank, (dim + rot) ** -0.5, THETA,
                                     Yarn(8.0, 4096, 32.0, 1.0))}
    ffs = {"ff": DenseConfig(z["ff"]), "experts": ExpertsConfig(*z["experts"])}
    return RivilixConfig(vocab_size=VOCAB, hidden_size=z["width"], eps=EPS, dtype=dtype,
                         kv_block_size=c["page"],
                         layers=[RivilixLayer(mixers[m], ffs[f]) for m, f in rivilix_layers(z)],
                         bigram=Bigram(8192, 40503, 9973), softcap=SOFTCAP)


def weights(c, seed):
    """Weights by name, all of them bf16 numbers."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    z = (RIVILIX if c["family"] == "rivilix" else SIZES)[c["size"]]
    wd, w = z["width"], {}

    def mat(name, n, k, gain=1.0):
        t = torch.empty((n, k), dtype=torch.bfloat16, device=DEVICE)
        w[name] = t.normal_(0.0, gain / math.sqrt(k), generator=gen)

    def vec(name, shape, lo, hi):
        t = torch.empty(shape, dtype=torch.bfloat16, device=DEVICE)
        w[name] = t.uniform_(lo, hi, generator=gen)

    def ff(p, n, gain=0.5):
        mat(p + "gate", n, wd, 1.5)
        mat(p + "up", n, wd)
        mat(p + "down", wd, n, gain)

    embed, head, final = ("model.embed_tokens.weight", "lm_head.weight", "model.norm.weight") \
        if c["family"] == "llama" else ("embed", "head", "final.norm")
    mat(embed, VOCAB, wd, math.sqrt(wd))
    w[head] = w[embed] * (2.0 / math.sqrt(wd))
    if c["family"] == "llama":
        vec(final, (wd,), 0.8, 1.2)
        cfg = config(c)
        for i in range(z["layers"]):
            p = f"model.layers.{i}."
            a = p + "self_attn."
            for n in ("input_layernorm", "post_attention_layernorm"):
                vec(f"{p}{n}.weight", (wd,), 0.6, 1.4)
            for n in "qk":
                vec(f"{a}{n}_norm.weight", (128,), 0.8, 1.6)
            mat(a + "q_proj.weight", cfg.num_attention_heads * 128, wd)
            for n in "kv":
                mat(f"{a}{n}_proj.weight", cfg.num_key_value_heads * 128, wd)
            mat(a + "o_proj.weight", wd, cfg.num_attention_heads * 128, 0.7)
            mat(p + "mlp.gate_proj.weight", z["ff"], wd, 1.5)
            mat(p + "mlp.up_proj.weight", z["ff"], wd)
            mat(p + "mlp.down_proj.weight", wd, z["ff"], 0.5)
    elif c["family"] == "pinuvik":
        vec(final, (), 0.9, 1.1)
        for i in range(z["layers"]):
            p, left, right = f"l{i}.", f"l{i}.mix.left.", f"l{i}.mix.right."
            hd = z["delta"][0] * z["delta"][1]
            for n in ("norm1", "norm2"):
                vec(p + n, (), 0.8, 1.2)
            for n in ("norm1b", "norm2b"):
                vec(p + n, (), 0.3, 0.6)
            vec(p + "shift", (wd,), 0.1, 0.8)
            mat(left + "q", z["heads"] * z["dim"], wd)
            mat(left + "k", z["kv"] * z["dim"], wd)
            mat(left + "o", wd, z["heads"] * z["dim"])
            for n in "rkvga":
                mat(right + n, hd, wd)
            vec(right + "a.b", (hd,), -1.0, 1.0)
            vec(right + "w0", (hd,), -4.0, 1.0)
            mat(right + "w1", z["rank"], wd)
            mat(right + "w2", hd, z["rank"])
            vec(right + "norm", (hd,), 0.5, 1.5)
            mat(right + "o", wd, hd)
            for n in (left, right):
                vec(n + "out", (wd,), 0.5, 1.5)
            ff(p + "mlp.", z["ff"])
    else:
        heads, dim, rot, vdim, rank = z["latent"]
        mh, md, mv = z["memory"]
        n_exp, _, ff_exp, ff_shared = z["experts"]

        def norm(name):
            vec(name, (wd,), 0.6, 1.4)
            vec(name + ".b", (wd,), -0.2, 0.2)
        norm(final)
        mat("bigram", 8192 + 1, wd, 0.5 * math.sqrt(wd))
        for i, (mixer, kind) in enumerate(rivilix_layers(z)):
            p, m = f"l{i}.", f"l{i}.mix."
            norm(p + "norm1")
            norm(p + "norm2")
            if mixer == "memory":
                for n, k in (("q", mh * md), ("k", mh * md), ("v", mh * mv), ("g", mh * mv)):
                    mat(m + n, k, wd)
                mat(m + "i", mh, wd, 1.5)
                mat(m + "f", mh, wd, 0.5)
                vec(m + "i.b", (mh,), -2.0, 1.0)
                vec(m + "f.b", (mh,), 3.0, 6.0)
                vec(m + "norm", (mh * mv,), 0.5, 1.5)
                mat(m + "o", wd, mh * mv, 0.5)
            else:
                mat(m + "q", heads * (dim + rot), wd)
                mat(m + "dkv", rank + rot, wd)
                vec(m + "dkv.norm", (rank,), 0.5, 1.5)
                mat(m + "uk", heads * dim, rank)
                mat(m + "uv", heads * vdim, rank)
                mat(m + "o", wd, heads * vdim, 0.7)
            q = p + "mlp."
            if kind == "ff":
                ff(q, z["ff"])
                for n, k in (("gate.b", z["ff"]), ("up.b", z["ff"]), ("down.b", wd)):
                    vec(q + n, (k,), -0.2, 0.2)
                continue
            # experts have a part in common: where a choice hangs on the last bits of a row,
            # the row still comes out alike
            mat(q + "router", n_exp, wd, 2.0)
            vec(q + "router.b", (n_exp,), -0.5, 0.5)
            ff(q + "e0.", ff_exp)
            for e in range(n_exp - 1, -1, -1):
                ff(f"{q}own.", ff_exp)
                for leaf in ("gate", "up", "down"):
                    w[f"{q}e{e}.{leaf}"] = (w[f"{q}e0.{leaf}"] + 0.25 * w[f"{q}own.{leaf}"]) \
                        .to(torch.bfloat16)
            for leaf in ("gate", "up", "down"):
                del w[f"{q}own.{leaf}"]
            ff(q + "shared.", ff_shared)
    return w


def prompts(c, seed):
    r = random.Random(seed)
    return [[r.randrange(VOCAB) for _ in range(n)] for n in lengths(c)]


# --------------------------------------------------------------------------- one pass
def graph_size(n):
    """The batch sizes that a server captures: 1, 2, 4, 8 and multiples of 16."""
    return next(b for b in (1, 2, 4, 8) if b >= n) if n <= 8 else -(-n // 16) * 16


def prepare(c, seed):
    """An engine with its weights; for decode steps the contexts are in the cache and the
    graph is captured."""
    cfg, tokens = config(c), prompts(c, seed)
    n, longest = len(tokens), max(map(len, tokens)) + REPLY + 1
    rows = graph_size(n)
    with torch.no_grad():
        eng = DecodeEngine(
            cfg, max_num_seqs=rows, max_model_len=longest, init_scale=None,
            num_kv_blocks=DecodeEngine.pages_for(cfg, sum(map(len, tokens)) + n * (REPLY + 1),
                                                 rows))
        eng.load_weights(DictSource(weights(c, seed)))
    state = dict(case=c, engine=eng, prompts=tokens, steps=0)
    if c["phase"] == "decode":
        eng.prefill(tokens, chunk_tokens=16384)
        eng.capture_cudagraph([rows])
    torch.cuda.empty_cache()
    return state


def run(state):
    eng, tokens = state["engine"], state["prompts"]
    if state["case"]["phase"] == "decode":
        if state["steps"] == REPLY:     # the replies are done: the next requests' turn
            for s in reversed(list(eng.seqs)):
                eng.finish(s)
            eng.add_sequences([len(t) + 1 for t in tokens], [t[-1] for t in tokens])
            state["steps"] = 0
        ids = eng.step()
        state["steps"] += 1
        return {"tokens": ids, "logits": eng.graph_vars["lm_logits"][:len(ids)]}
    seqs = [eng.open_sequence() for _ in tokens]
    left = [list(t) for t in tokens]
    logits = [None] * len(seqs)
    while any(left):
        room, which, part, want = state["case"]["portion"], [], [], []
        for i, t in enumerate(left):
            if t and room > 0:
                which.append(i)
                part.append((seqs[i], t[:room]))
                want.append([len(t) - 1] if len(t) <= room else [])
                left[i], room = t[room:], room - len(t)
        for i, w, out in zip(which, want, eng.feed(part, want)):
            if w:
                logits[i] = out
    for s in reversed(seqs):
        eng.finish(s)
    return {"logits": torch.cat(logits)}


# ------------------------------------------------------------------- what a pass needs
def work(c):
    z = (RIVILIX if c["family"] == "rivilix" else SIZES)[c["size"]]
    wd, lens, decode = z["width"], lengths(c), c["phase"] == "decode"
    e = 2 if c["dtype"] == "bfloat16" else 4
    n, rows = len(lens), len(lens) if decode else sum(lens)
    # bytes, and multiply-adds, of the head, the embedding rows in and the logits out
    nbytes, macs = e * (VOCAB * wd + rows * wd) + (2 if decode else 4) * n * VOCAB, n * VOCAB * wd

    def product(out, k, times=1.0):
        nonlocal nbytes, macs
        nbytes, macs = nbytes + e * out * k, macs + out * k * rows * times

    def keys(chunk=None):
        """(keys that are read from or written to the cache, query-key pairs)"""
        total, pairs = 0, 0
        for t in lens:
            if decode:
                seen = t + 1 if chunk is None else t % chunk + 1
                total, pairs = total + seen, pairs + seen
            else:
                total += t
                for a in range(0, t, chunk or t):
                    m = min(t - a, chunk or t)
                    pairs += m * (m + 1) // 2
        return total, pairs
    for i in range(z["layers"]):
        if c["family"] == "rivilix":
            mixer, kind = rivilix_layers(z)[i]
            if mixer == "memory":
                h, d, v = z["memory"]
                product(2 * h * d + 2 * h * v + 2 * h, wd)
                product(wd, h * v)
                nbytes += n * h * d * (v + 1) * 4 * (2 if decode else 1)
                macs += 2 * rows * h * d * v
            else:
                h, d, r, v, rank = z["latent"]
                total, pairs = keys()
                product(h * (d + r) + rank + r, wd)
                product(wd, h * v)
                product(h * (d + v), rank)
                nbytes += total * (rank + r) * e
                macs += pairs * h * (2 * rank + r if decode else d + r + v)
            if kind == "ff":
                product(3 * z["ff"], wd)
            else:
                number, top, ff, shared = z["experts"]
                product(number + 3 * shared, wd)
                used = number * (1 - (1 - top / number) ** rows)
                nbytes += used * 3 * ff * wd * e
                macs += rows * top * 3 * ff * wd
            continue
        scale = 128 // z["dim"] if c["family"] == "llama" else 1
        h, kv, d = z["heads"] // scale, z["kv"] // scale, z["dim"] * scale
        total, pairs = keys(None if c["family"] == "llama" else z["chunk"])
        product((h + (2 * kv if c["family"] == "llama" else kv)) * d, wd)
        product(wd, h * d)
        product(3 * z["ff"], wd)
        nbytes += 2 * total * kv * d * e
        macs += 2 * pairs * h * d
        if c["family"] == "pinuvik":
            dh, dd = z["delta"]
            product(5 * dh * dd + z["rank"], wd)
            product(dh * dd, z["rank"])
            product(wd, dh * dd)
            nbytes += n * dh * dd * dd * 4 * (2 if decode else 1)
            macs += 4 * rows * dh * dd * dd
    return {"bytes": float(nbytes), "flops": 2.0 * macs}


def tolerance(c):
    """Logits against `exact`: 1.1e-2 off (2-norm) for the bf16 residual of the first decoder,
    4 to 7e-3 for the fp32 residual of the other two, 2.5e-6 in fp32; two implementations that
    round at different places are off by up to twice that from one another."""
    if c["dtype"] == "float32":
        return {"rel": 1e-5, "max": 2e-4}
    return {"rel": 0.03, "max": 0.3} if c["family"] == "llama" else {"rel": 0.02, "max": 0.2}


# ----------------------------------------------------- the same in plain torch, 64 bits
def rms(x):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)


def layer_norm(x, w, name):
    x = x - x.mean(-1, keepdim=True)
    return rms(x) * w[name].double() + w[name + ".b"].double()


def causal(q, k, v, scale):
    """q [T, H, d], k [T, G, d], v [T, G, e]."""
    t, heads, _ = q.shape
    per = heads // k.shape[1]
    mask = torch.ones((t, t), dtype=torch.bool, device=q.device).triu(1)
    out = q.new_empty((t, heads, v.shape[2]))
    for h in range(heads):
        s = (q[:, h] @ k[:, h // per].T * scale).masked_fill_(mask, -math.inf)
        out[:, h] = torch.softmax(s, -1) @ v[:, h // per]
    return out


def turn(x, freqs, paired, size=1.0):
    """Rotation of x [T, H, d]: channels (2i, 2i + 1) if paired, else (i, i + d / 2)."""
    a = torch.arange(x.shape[0], dtype=torch.float64, device=x.device)[:, None, None] * freqs
    c, s = a.cos() * size, a.sin() * size
    if paired:
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    u, v = x.chunk(2, -1)
    return torch.cat([u * c - v * s, v * c + u * s], -1)


def frequencies(dims, base, yarn=None):
    i = torch.arange(dims // 2, dtype=torch.float64, device=DEVICE)
    f = base ** (-2.0 * i / dims)
    if yarn is None:
        return f
    factor, original, fast, slow = yarn

    def pair(turns):
        return dims * math.log(original / (2 * math.pi * turns)) / (2 * math.log(base))
    lo, hi = max(math.floor(pair(fast)), 0), min(math.ceil(pair(slow)), dims - 1)
    ramp = ((i - lo) / max(hi - lo, 0.001)).clamp(0, 1)
    return f / factor * ramp + f * (1 - ramp)


def padded(x, lens):
    """[tokens, ...] -> [sequences, longest, ...]"""
    return torch.nn.utils.rnn.pad_sequence(list(x.split(lens)), batch_first=True)


def unpadded(x, lens):
    return torch.cat([x[i, :n] for i, n in enumerate(lens)])


def delta_rule(r, k, v, decay, rate):
    """[sequences, T, heads, d]: S <- diag(w) S - (a u)(u^T S) + k v^T, o = S^T r."""
    u = k * torch.rsqrt(k.square().sum(-1, keepdim=True) + 1e-6)
    s = k.new_zeros((*k[:, 0].shape, k.shape[-1]))
    o, au = torch.empty_like(v), rate * u
    for t in range(k.shape[1]):
        seen = u[:, t, :, None] @ s
        s = decay[:, t, ..., None] * s
        s -= au[:, t, ..., None] * seen
        s += k[:, t, ..., None] * v[:, t, :, None]
        o[:, t] = (r[:, t, :, None] @ s)[:, :, 0]
    return o


def matrix_memory(q, k, v, i, f):
    """[sequences, T, heads, ...]: S <- e^f S + e^i k v^T with a running maximum."""
    s = k.new_zeros((*k[:, 0].shape, v.shape[-1]))
    n, m, o = torch.zeros_like(k[:, 0]), torch.zeros_like(i[:, 0]), torch.empty_like(v)
    for t in range(k.shape[1]):
        m1 = torch.maximum(f[:, t] + m, i[:, t])
        keep, add, m = (f[:, t] + m - m1).exp(), (i[:, t] - m1).exp(), m1
        ka = k[:, t] * add[..., None]
        n = n * keep[..., None] + ka
        s = s * keep[..., None, None]
        s += ka[..., None] * v[:, t, :, None]
        low = torch.maximum((n * q[:, t]).sum(-1).abs(), (-m).exp()) + 1e-6
        o[:, t] = (q[:, t, :, None] @ s)[:, :, 0] / low[..., None]
    return o


@torch.no_grad()
def exact(c, seed):
    if work(dict(c, phase="prefill"))["flops"] > 1.5e14:
        return None
    z = (RIVILIX if c["family"] == "rivilix" else SIZES)[c["size"]]
    w, tokens = weights(c, seed), prompts(c, seed)
    if c["phase"] == "decode":                  # a token predicts itself
        tokens = [t + t[-1:] for t in tokens]
    lens, ids = [len(t) for t in tokens], torch.tensor(sum(tokens, []), device=DEVICE)
    last = torch.tensor(lens, device=DEVICE).cumsum(0) - 1
    heads, kv, dim = z.get("heads"), z.get("kv"), z.get("dim")

    def mul(x, name):
        return x @ w[name].double().T

    def gated(h, p, act, bias=False, suffix=""):
        g, u = mul(h, p + "gate" + suffix), mul(h, p + "up" + suffix)
        if bias:
            g, u = g + w[p + "gate.b"].double(), u + w[p + "up.b"].double()
        return mul(act(g).mul_(u), p + "down" + suffix) + \
            (w[p + "down.b"].double() if bias else 0.0)

    def each(f, *rows):
        return torch.cat([f(*x) for x in zip(*(r.split(lens) for r in rows))])
    silu = torch.nn.functional.silu
    if c["family"] == "llama":
        heads, kv, dim = heads * dim // 128, kv * dim // 128, 128
        freqs = frequencies(dim, THETA)
        x = w["model.embed_tokens.weight"][ids].double()
        for i in range(z["layers"]):
            p = f"model.layers.{i}."
            a = p + "self_attn."
            h = rms(x) * w[p + "input_layernorm.weight"].double()
            q, k, v = (mul(h, f"{a}{n}_proj.weight").unflatten(-1, (-1, dim)) for n in "qkv")
            q, k = (rms(t) * w[f"{a}{n}_norm.weight"].double() for n, t in (("q", q), ("k", k)))
            o = each(lambda q, k, v: causal(turn(q, freqs, False), turn(k, freqs, False), v,
                                            dim ** -0.5), q, k, v)
            x = x + mul(o.flatten(1), a + "o_proj.weight")
            h = rms(x) * w[p + "post_attention_layernorm.weight"].double()
            x = x + gated(h, p + "mlp.", silu, suffix="_proj.weight")
        logits = mul(rms(x[last]) * w["model.norm.weight"].double(), "lm_head.weight")
    elif c["family"] == "pinuvik":
        freqs, chunk = frequencies(dim, THETA), z["chunk"]

        def attend(q, k):
            qn, kn = rms(turn(q, freqs, True)), rms(turn(k, freqs, True))
            return torch.cat([causal(*s, dim ** -0.5) for s in
                              zip(qn.split(chunk), kn.split(chunk), k.split(chunk))])
        x = w["embed"][ids].double()
        for i in range(z["layers"]):
            p, left, right = f"l{i}.", f"l{i}.mix.left.", f"l{i}.mix.right."
            h = rms(x) * w[p + "norm1"].double()
            before = each(lambda t: torch.cat([torch.zeros_like(t[:1]), t[:-1]]), h)
            h = h + (before - h) * w[p + "shift"].double()
            o = each(attend, mul(h, left + "q").unflatten(-1, (heads, dim)),
                     mul(h, left + "k").unflatten(-1, (kv, dim)))
            a = rms(mul(o.flatten(1), left + "o")) * w[left + "out"].double()
            r, k, v = (mul(h, right + n).unflatten(-1, z["delta"]) for n in "rkv")
            decay = torch.exp(-math.exp(-0.5) * torch.sigmoid(
                mul(mul(h, right + "w1").tanh(), right + "w2") + w[right + "w0"].double()))
            rate = torch.sigmoid(mul(h, right + "a") + w[right + "a.b"].double())
            o = unpadded(delta_rule(*(padded(t.view_as(k), lens)
                                      for t in (r, k, v, decay, rate))), lens)
            y = rms(o).flatten(1) * w[right + "norm"].double() * torch.sigmoid(mul(h, right + "g"))
            b = rms(mul(y, right + "o")) * w[right + "out"].double()
            x = x + rms(0.5 * (a + b)) * w[p + "norm1b"].double()
            h = rms(x) * w[p + "norm2"].double()
            y = gated(h, p + "mlp.", lambda g: torch.nn.functional.gelu(g, approximate="tanh"))
            x = x + rms(y) * w[p + "norm2b"].double()
        logits = mul(rms(x[last]) * w["final.norm"].double(), "head")
    else:
        heads, dim, rot, vdim, rank = z["latent"]
        mh, md, mv = z["memory"]
        number, top, _, _ = z["experts"]
        freqs, size = frequencies(rot, THETA, (8.0, 4096, 32.0, 1.0)), 0.1 * math.log(8.0) + 1
        pair = each(lambda t: torch.cat([t.new_full((1,), 8192),
                                         (t[:-1] * 40503 + t[1:] * 9973) % 8192]), ids)
        x = w["embed"][ids].double() + w["bigram"][pair].double()

        def latent(q, row, p):
            k = rms(row[:, :rank]) * w[p + "dkv.norm"].double()
            shared = turn(row[:, None, rank:], freqs, True, size).expand(-1, heads, -1)
            kk = torch.cat([mul(k, p + "uk").unflatten(-1, (heads, dim)), shared], -1)
            qq = torch.cat([q[..., :dim], turn(q[..., dim:], freqs, True, size)], -1)
            return causal(qq, kk, mul(k, p + "uv").unflatten(-1, (heads, vdim)),
                          (dim + rot) ** -0.5)

        def mixture(h, p):
            share, chosen = (mul(h, p + "router") + w[p + "router.b"].double()).topk(top)
            share, y = share.softmax(-1), gated(h, p + "shared.", silu)
            for e in range(number):
                row, place = (chosen == e).nonzero(as_tuple=True)
                if row.numel():
                    y.index_add_(0, row, share[row, place, None] *
                                 gated(h[row], f"{p}e{e}.", silu))
            return y
        for i, (mixer, kind) in enumerate(rivilix_layers(z)):
            p, m = f"l{i}.", f"l{i}.mix."
            h = layer_norm(x, w, p + "norm1")
            if mixer == "memory":
                q, k, v = (mul(h, m + n).unflatten(-1, (mh, -1)) for n in "qkv")
                gi, gf = (15.0 * torch.tanh((mul(h, m + n) + w[f"{m}{n}.b"].double()) / 15.0)
                          for n in "if")
                o = unpadded(matrix_memory(
                    *(padded(t, lens) for t in (q * md ** -0.5, k, v, gi,
                                                torch.nn.functional.logsigmoid(gf)))), lens)
                y = mul(rms(o).flatten(1) * w[m + "norm"].double()
                        * torch.sigmoid(mul(h, m + "g")), m + "o")
            else:
                y = mul(each(lambda q, row: latent(q, row, m),
                             mul(h, m + "q").unflatten(-1, (heads, dim + rot)),
                             mul(h, m + "dkv")).flatten(1), m + "o")
            h = layer_norm(x, w, p + "norm2")
            x = x + y + (gated(h, p + "mlp.", silu, bias=True) if kind == "ff"
                         else mixture(h, p + "mlp."))
        logits = mul(layer_norm(x[last], w, "final.norm"), "head")
        logits = SOFTCAP * torch.tanh(logits / SOFTCAP)
    if c["phase"] == "decode":
        return {"tokens": None, "logits": logits}
    return {"logits": logits.cpu()}
