"""Performance cases: what programs that serve language models with this package have it do, through its public classes.

A case is a model and one piece of work of its sessions:

  sessions  1, or the members of a session group (one pass over the weights for all of them)
  kept      tokens that the caches hold already (a conversation so far); the pass returns to this place first
  pushed    tokens of a prompt that are evaluated together, in steps of at most `step`
  decoded   tokens evaluated one after the other, each pushed and followed by the prediction of the next one

The tokens are given (not the predicted ones), so that two implementations that round differently still evaluate the same sequence.
A pass returns the logits after the last token, for every session.

The models have random weights: ggjt files of LLaMA geometry (q4_0 and q8_0 blocks), and model folders of the two hybrid designs
(bfloat16).  A program opens a model once and makes many sessions on it, so opened models are kept here as well, up to a limit of bytes.
The weights depend on the model alone, the tokens on the seed.
"""
import collections
import functools
import importlib.util
import json
import math
import os
import random
import shutil
import struct
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
VOCAB, HEAD = 32000, 128
OPEN_MODELS_BYTES = 40e9


def package():
    """The package directory has a hyphen in its name."""
    name = "llama_vulkan_b200"
    if name not in sys.modules:
        at = os.path.join(ROOT, "llama-vulkan_b200")
        spec = importlib.util.spec_from_file_location(name, os.path.join(at, "__init__.py"), submodule_search_locations=[at])
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


# ---- the cases -----------------------------------------------------------------------------

LLAMA_FF = {1024: 2048, 2048: 5632, 4096: 11008, 5120: 13824}
SONUZEN = {      # width: query heads, key/value heads, recurrent width, experts, expert width, experts of a token, layers
    1024: (8, 2, 1536, 16, 512, 4, 8),
    2048: (16, 4, 2560, 16, 1408, 4, 8),
    4096: (32, 8, 4096, 8, 5504, 2, 4),
}
NUFORAX = {      # width: attention heads, state-space heads, groups, feed-forward width, layers
    1024: (8, 32, 2, 3072, 8),
    2048: (16, 64, 4, 8448, 8),
    4096: (32, 128, 8, 16512, 4),
}


def case(name, model, width, layers, dtype, kept=0, pushed=0, decoded=0, step=64, sessions=1, sampled=False):
    c = dict(model=model, width=width, layers=layers, dtype=dtype, sessions=sessions, kept=kept, pushed=pushed, decoded=decoded, step=step,
             sampled=sampled)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one token of the two-layer 7B geometry: the smallest call, bound by latency
        case("token-2-layers", "llama", 4096, 2, "q4_0", kept=16, decoded=1),
        # a chat answer of LLaMA-7B with a short context, greedy
        case("chat-7b-q4", "llama", 4096, 32, "q4_0", kept=64, decoded=24),
        # a chat answer after a long conversation, drawn with the sampler (the reference's default); the 7B geometry in q8_0
        case("chat-7b-q8-long", "llama", 4096, 8, "q8_0", kept=1100, decoded=24, step=1, sampled=True),
        # a chat answer of the 13B geometry
        case("chat-13b-q4", "llama", 5120, 8, "q4_0", kept=200, decoded=24),
        # a document of 1024 tokens read by LLaMA-7B
        case("prompt-7b-q4", "llama", 4096, 32, "q4_0", pushed=1024),
        # a short question in a running conversation: 37 tokens in one step
        case("question-7b-q8", "llama", 4096, 8, "q8_0", kept=200, pushed=37),
        # a server with 16 and with 50 running sessions
        case("sessions-16-7b-q4", "llama", 4096, 8, "q4_0", kept=200, decoded=6, sessions=16),
        case("sessions-50-7b-q4", "llama", 4096, 8, "q4_0", kept=120, decoded=6, sessions=50),
        # the hybrid designs: prompts in the default steps of 512, and whole requests (a recurrent state cannot be taken back, so a
        # request begins with its prompt)
        case("prompt-sonuzen", "sonuzen", 2048, 8, "bf16", pushed=2048, step=512),
        case("request-sonuzen", "sonuzen", 2048, 8, "bf16", pushed=60, decoded=24, step=512),
        case("prompt-nuforax", "nuforax", 2048, 8, "bf16", pushed=1531, step=512),
        case("request-nuforax", "nuforax", 4096, 4, "bf16", pushed=1000, decoded=24, step=512),
    ]


def draw(rng):
    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["chat", "chat", "prompt", "prompt", "sessions", "prompt-hybrid", "request-hybrid", "request-hybrid"])
    if kind.endswith("hybrid"):
        model, width = rng.choice(["sonuzen", "nuforax"]), rng.choice([1024, 2048, 2048])
        layers = (SONUZEN if model == "sonuzen" else NUFORAX)[width][-1]
        if kind == "prompt-hybrid":
            return case(None, model, width, layers, "bf16", pushed=between(100, 2048), step=rng.choice([256, 512, 512, 2048]))
        return case(None, model, width, layers, "bf16", pushed=between(5, 1200), decoded=between(8, 40), step=512)
    width, dtype = rng.choice([2048, 4096, 4096, 5120]), rng.choice(["q4_0", "q4_0", "q8_0"])
    layers = rng.randint(2, 6)
    if kind == "chat":
        kept = between(10, 1900)
        return case(None, "llama", width, layers, dtype, kept=kept, decoded=between(1, 40), step=64 if kept < 200 else 1, sampled=rng.random() < 0.5)
    if kind == "prompt":
        step = rng.choice([32, 64, 64])
        if rng.random() < 0.5:
            return case(None, "llama", width, layers, dtype, kept=between(5, 120), pushed=between(6, 120), step=step)
        return case(None, "llama", width, layers, dtype, pushed=step * between(2, 1152 // step), step=step)
    return case(None, "llama", width, layers, dtype, kept=between(10, 600), decoded=between(2, 8), sessions=between(2, 64))


# ---- weights -------------------------------------------------------------------------------

BLOCKS, VALUES = 262139, 8388593          # primes: no two rows of a matrix begin at the same place of the repeated slab


@functools.lru_cache(None)
def blocks(dtype):
    """Quantised blocks of N(0, 0.02) values -> (bytes [BLOCKS][18 or 34], float64 values [BLOCKS][32])."""
    x = 0.02 * np.random.default_rng(11).standard_normal((BLOCKS, 32), dtype=np.float32)
    amax = np.abs(x).max(axis=1, keepdims=True)
    d = (amax / (8 if dtype == "q4_0" else 127)).astype(np.float16)
    q = np.rint(x / d.astype(np.float32))
    if dtype == "q4_0":
        q = np.clip(q, -8, 7)
        u = (q + 8).astype(np.uint8)
        body = u[:, :16] | (u[:, 16:] << 4)
    else:
        q = np.clip(q, -127, 127)
        body = q.astype(np.int8).view(np.uint8)
    return np.concatenate([d.view(np.uint8).reshape(-1, 2), body], axis=1), q.astype(np.float64) * d.astype(np.float64)


@functools.lru_cache(None)
def normals():
    return np.random.default_rng(12).standard_normal(VALUES, dtype=np.float32)


def bf16(x):
    u = np.ascontiguousarray(x, np.float32).view(np.uint32)
    return ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)


@functools.lru_cache(8)
def normals_bf16(gain):
    """bfloat16 bits of the slab times a power of two."""
    return bf16(normals() * gain)


def pieces(slab, at, n):
    """n items of the slab, repeated, from place `at` on."""
    while n:
        k = min(n, len(slab) - at)
        yield slab[at:at + k]
        n, at = n - k, 0


def place(name, size):
    return random.Random(name).randrange(size)


def key_of(c):
    return c["model"], c["width"], c["layers"], c["dtype"]


def llama_tensors(key):
    """name -> (rows, columns or None for a norm vector)."""
    _, dim, layers, _ = key
    ff = LLAMA_FF[dim]
    t = {"tok_embeddings": (VOCAB, dim), "norm": (dim, None), "output": (VOCAB, dim)}
    for i in range(layers):
        p = f"layers.{i}."
        for n in ("wq", "wk", "wv", "wo"):
            t[f"{p}attention.{n}"] = (dim, dim)
        t[p + "feed_forward.w1"], t[p + "feed_forward.w2"], t[p + "feed_forward.w3"] = (ff, dim), (dim, ff), (ff, dim)
        t[p + "attention_norm"] = t[p + "ffn_norm"] = (dim, None)
    return t


def llama_norm(name, n):
    a = place(name, VALUES - n)
    return (1 + 0.01 * normals()[a:a + n]).astype(np.float32)


def write_llama(path, key):
    _, dim, layers, dtype = key
    kind, slab = {"q4_0": 2, "q8_0": 8}[dtype], blocks(dtype)[0]
    with open(path, "wb") as f:
        f.write(struct.pack("<9I", 0x67676A74, 3, VOCAB, dim, 256, dim // HEAD, layers, HEAD, kind))
        for i in range(VOCAB):
            text = bytes([i - 3]) if 3 <= i < 259 else b"t%d" % i
            f.write(struct.pack("<i", len(text)) + text + struct.pack("<f", 0.0))
        for name, (rows, cols) in llama_tensors(key).items():
            full = (name + ".weight").encode()
            f.write(struct.pack("<3I", 1 if cols is None else 2, len(full), 0 if cols is None else kind))
            f.write(struct.pack("<I", rows) if cols is None else struct.pack("<2I", cols, rows))
            f.write(full)
            f.write(b"\0" * (-f.tell() % 32))
            if cols is None:
                f.write(llama_norm(name, rows).tobytes())
            else:
                for part in pieces(slab, place(name, BLOCKS), rows * cols // 32):
                    f.write(part.data)


def sonuzen_config(width):
    heads, kv, gru, experts, ff, top, layers = SONUZEN[width]
    mlp = {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": experts, "top": top}}
    attention = {"type": "attention", "mixer": {"heads": heads, "kv_heads": kv, "dim": HEAD, "vdim": HEAD, "scale": HEAD ** -0.5}, "mlp": mlp}
    recurrent = {"type": "mingru", "mixer": {"width": gru}, "mlp": mlp}
    return {"architecture": "Sonuzen", "width": width, "vocab": VOCAB, "layers": [recurrent if i % 4 == 1 else attention for i in range(layers)],
            "loop": None, "canon": {"taps": 4}, "norm": {"eps": 1e-5}, "residual_mult": 0.5, "logit_scale": 1.0}


ROT, RANK, WINDOW, SSM_DIM, SSM_STATE, BUCKETS = 64, 512, 1024, 64, 128, 20011


def nuforax_config(width):
    heads, ssm, groups, ff, layers = NUFORAX[width]
    out = []
    for i in range(layers):      # of four layers: attention, a state space, attention, attention over the third's cache
        if i % 4 == 1:
            out.append({"type": "mamba2", "mlp": {"kind": "dense", "ff": ff},
                        "mixer": {"heads": ssm, "vdim": SSM_DIM, "state": SSM_STATE, "groups": groups, "conv": 4, "norm_groups": groups}})
            continue
        m = {"heads": heads, "dim": HEAD, "rot_dim": ROT, "vdim": HEAD, "kv_rank": RANK, "mask": {"size": WINDOW}, "scale": (HEAD + ROT) ** -0.5,
             "rot": {"dims": ROT, "base": 10000.0, "scaling": {"factor": 4.0, "original": 4096, "fast": 32.0, "slow": 1.0}}}
        if i % 4 == 3:
            m["kv_from"] = i - 1
        out.append({"type": "latent_attention", "mlp": {"kind": "dense", "ff": ff}, "mixer": m})
    return {"architecture": "Nuforax", "width": width, "vocab": VOCAB, "layers": out, "norm": {"eps": 1e-5},
            "embedding": {"scale": width ** 0.5, "bigram": {"buckets": BUCKETS, "mul_prev": 41, "mul_cur": 13}}}


def config_of(key):
    return sonuzen_config(key[1]) if key[0] == "sonuzen" else nuforax_config(key[1])


def power(x):
    return 2.0 ** round(math.log2(x))


def folder_tensors(key):
    """name -> (shape, gain) of a matrix, (shape, mean, spread) of a vector, (shape, experts) of a routing table."""
    cfg, W = config_of(key), key[1]
    t = {}

    def matrix(name, rows, cols, gain=1.0):
        t[name] = ((rows, cols), power(gain * cols ** -0.5))

    def vector(name, *shape, mean=0.0, spread=0.1):
        t[name] = (shape, mean, spread)

    if key[0] == "sonuzen":
        heads, kv, gru, experts, ff, top, _ = SONUZEN[W]
        matrix("embed", VOCAB, W, W ** 0.5)
        matrix("head", VOCAB, W)
        for i, l in enumerate(cfg["layers"]):
            p = f"l{i}."
            for n in ("norm1", "norm1b", "norm2", "norm2b"):
                vector(p + n, W)
            vector(p + "canon1", W, 4, spread=0.3)
            vector(p + "canon2", W, 4, spread=0.3)
            if l["type"] == "attention":
                matrix(p + "mix.q", heads * HEAD, W)
                matrix(p + "mix.k", kv * HEAD, W)
                matrix(p + "mix.v", kv * HEAD, W)
                vector(p + "mix.q.norm", HEAD, mean=1.2)
                vector(p + "mix.k.norm", HEAD, mean=1.2)
                vector(p + "mix.r1", heads, mean=0.3, spread=0.05)
                vector(p + "mix.r2", heads, mean=0.5, spread=0.1)
                matrix(p + "mix.o", W, heads * HEAD)
            else:
                for n in "zxg":
                    matrix(p + "mix." + n, gru, W)
                vector(p + "mix.z.b", gru, mean=-1.5, spread=1.0)
                vector(p + "mix.x.b", gru, spread=0.5)
                matrix(p + "mix.o", W, gru)
            for e in range(experts):
                matrix(f"{p}mlp.e{e}.gate", ff, W)
                matrix(f"{p}mlp.e{e}.up", ff, W)
                matrix(f"{p}mlp.e{e}.down", W, ff)
            t[p + "mlp.table"] = ((VOCAB, top), experts)
        vector("final.norm", W)
        return t
    matrix("embed", VOCAB, W)
    matrix("bigram", BUCKETS + 1, W, 0.5 * W ** 0.5)
    for i, l in enumerate(cfg["layers"]):
        p, mix, m = f"l{i}.", f"l{i}.mix.", l["mixer"]
        H = m["heads"]
        vector(p + "norm1", W, mean=0.7)
        vector(p + "norm2", W, mean=0.7)
        if l["type"] == "latent_attention":
            matrix(mix + "q", H * (HEAD + ROT), W)
            if "kv_from" not in m:
                matrix(mix + "dkv", RANK + ROT, W)
                vector(mix + "dkv.norm", RANK, mean=1.0)
            matrix(mix + "uk", H * HEAD, RANK)
            matrix(mix + "uv", H * HEAD, RANK)
            vector(mix + "sink", H, mean=1.0, spread=0.5)
            matrix(mix + "o", W, H * HEAD)
        else:
            inner, bc = H * SSM_DIM, 2 * m["groups"] * SSM_STATE
            matrix(mix + "in", 2 * inner + bc + H, W)
            vector(mix + "conv", inner + bc, 4, spread=0.5)
            vector(mix + "conv.b", inner + bc, spread=0.2)
            vector(mix + "dt_bias", H, mean=-1.0, spread=1.0)
            vector(mix + "A_log", H, mean=-1.5, spread=1.0)
            vector(mix + "D", H, mean=0.5, spread=0.5)
            vector(mix + "norm", inner, mean=1.0)
            matrix(mix + "o", W, inner)
        matrix(p + "mlp.up", l["mlp"]["ff"], W)
        matrix(p + "mlp.down", W, l["mlp"]["ff"])
    vector("final.norm", W, mean=1.0)
    return t


def vector_of(name, spec):
    shape, mean, spread = spec
    n, a = math.prod(shape), place(name, VALUES // 2)
    return bf16(mean + spread * normals()[a:a + n]).reshape(shape)


@functools.lru_cache(None)
def table_of(name, top, experts):
    return np.random.default_rng(place(name, 1 << 30)).random((VOCAB, experts), dtype=np.float32).argsort(axis=1)[:, :top].astype(np.int32)


def write_folder(path, key):
    os.makedirs(path, exist_ok=True)
    with open(os.path.join(path, "config.json"), "w") as f:
        json.dump(config_of(key), f)
    head, at, tensors = {}, 0, folder_tensors(key)
    for name, spec in tensors.items():
        n = math.prod(spec[0]) * (4 if name.endswith("table") else 2)
        head[name] = {"dtype": "I32" if name.endswith("table") else "BF16", "shape": list(spec[0]), "data_offsets": [at, at + n]}
        at += n
    text = json.dumps(head).encode()
    with open(os.path.join(path, "model.safetensors"), "wb") as f:
        f.write(len(text).to_bytes(8, "little") + text)
        for name, spec in tensors.items():
            if name.endswith("table"):
                f.write(table_of(name, spec[0][1], spec[1]).tobytes())
            elif len(spec) == 3:
                f.write(vector_of(name, spec).tobytes())
            else:
                for part in pieces(normals_bf16(spec[1]), place(name, VALUES), math.prod(spec[0])):
                    f.write(part.data)


# ---- sessions ------------------------------------------------------------------------------

class Model:
    def __init__(self, key):
        folder = tempfile.mkdtemp(prefix="perf_cases_")
        try:
            path = os.path.join(folder, "model")
            (write_llama if key[0] == "llama" else write_folder)(path, key)
            self.context = package().HostContext(path, 0)
        finally:
            shutil.rmtree(folder, ignore_errors=True)          # the weights are on the GPU
        self.bytes = sum(weight_bytes(key).values())

    def __del__(self):
        if getattr(self, "context", None) is not None:
            self.context.close()


OPEN = collections.OrderedDict()


def open_model(key):
    if key not in OPEN:
        OPEN[key] = Model(key)
        while len(OPEN) > 1 and sum(m.bytes for m in OPEN.values()) > OPEN_MODELS_BYTES:
            OPEN.popitem(last=False)                           # closed when its last session is gone
    OPEN.move_to_end(key)
    return OPEN[key]


class State:
    def __init__(self, model):
        self.model, self.sessions, self.group = model, [], None

    def __del__(self):
        if self.group is not None:
            self.group.close()
        for s in self.sessions:
            s.close()


def tokens_of(c, seed):
    """[sessions][kept + pushed + decoded]; members of a group hold contexts of different lengths (see kept_of)."""
    n = c["kept"] + c["pushed"] + c["decoded"]
    return np.random.default_rng([seed, n, c["sessions"]]).integers(3, VOCAB, (c["sessions"], n))


def kept_of(c, member):
    if c["sessions"] == 1:
        return c["kept"]
    kept = c["kept"] - (member * 7) % (c["kept"] // 2 + 1)
    return kept if c["kept"] <= 240 else max(1, kept // c["step"]) * c["step"]


def prepare(c, seed):
    s = State(open_model(key_of(c)))
    s.kept, s.pushed, s.decoded = [], [], []
    for m, row in enumerate(tokens_of(c, seed).tolist()):
        session = s.model.context.session(0 if c["model"] == "llama" else max(2048, len(row) + 64))
        s.sessions.append(session)
        session.set_deterministic(not c["sampled"])
        session.set_seed(seed % 1000 + m)
        if not session.set_max_batch(c["step"]):
            raise RuntimeError("steps of %d are refused" % c["step"])
        kept = kept_of(c, m)
        s.kept.append(kept)
        for t in row[:kept]:
            session.push_token(t)
        if kept and session.predict_next_token() == 0xFFFFFFFF:
            raise RuntimeError("the context cannot be evaluated")
        s.pushed.append(row[kept:kept + c["pushed"]])
        s.decoded.append(row[kept + c["pushed"]:kept + c["pushed"] + c["decoded"]])
    if c["sessions"] > 1:
        s.group = package().SessionGroup(s.model.context, s.sessions)
    return s


def run(s):
    for session, kept in zip(s.sessions, s.kept):
        session.rewind(kept)
    if s.group is not None:
        for step in zip(*s.decoded):
            for session, token in zip(s.sessions, step):
                session.push_token(token)
            if s.group.step() is None:
                raise RuntimeError("the group cannot step")
        return [np.stack([s.group.logits(m, VOCAB) for m in range(len(s.sessions))])]
    session = s.sessions[0]
    if s.pushed[0]:
        for token in s.pushed[0]:
            session.push_token(token)
        if session.predict_next_token() == 0xFFFFFFFF:
            raise RuntimeError("the prompt cannot be evaluated")
    for token in s.decoded[0]:
        session.push_token(token)
        if session.predict_next_token() == 0xFFFFFFFF:
            raise RuntimeError("the token cannot be evaluated")
    return [session.logits(VOCAB)[None]]


# ---- what a pass cannot do without -----------------------------------------------------------

def weight_bytes(key):
    """Bytes of the weights by kind: `layers` read by every step, `head` read where logits are wanted, `rest` (embedding rows)."""
    if key[0] == "llama":
        t, per = llama_tensors(key), {"q4_0": 18 / 32, "q8_0": 34 / 32}[key[3]]
        size = {n: r * (k * per if k else 4) for n, (r, k) in t.items()}
        return {"layers": sum(v for n, v in size.items() if n.startswith("layers")), "head": size["output"] + size["norm"], "rest": size["tok_embeddings"]}
    size = {n: math.prod(s[0]) * (4 if n.endswith("table") else 2) for n, s in folder_tensors(key).items()}
    tied = "head" not in size
    layers = sum(v for n, v in size.items() if n[0] == "l" and not n.endswith("table"))
    return {"layers": layers, "head": size["embed"] if tied else size["head"], "rest": sum(size.values()) - layers - (size["embed"] if tied else size["head"])}


def step_work(key, n, pos, head=1):
    """(bytes, flops) of evaluating n tokens together from position pos on; head: rows that go through the output matrix."""
    w, W = weight_bytes(key), key[1]
    seen = n * pos + n * (n + 1) / 2                            # pairs of a token and a position that it sees
    if key[0] == "llama":
        L, active = key[2], 4 * W * W + 3 * LLAMA_FF[W] * W
        return w["layers"] + (w["head"] if head else 0) + L * (pos + n) * 4 * W, 2.0 * n * L * active + L * seen * 4 * W + 2.0 * head * VOCAB * W
    nbytes, flops = w["layers"] + (w["head"] if head else 0), 2.0 * head * VOCAB * W
    if key[0] == "sonuzen":
        heads, kv, gru, experts, ff, top, layers = SONUZEN[W]
        rec = sum(i % 4 == 1 for i in range(layers))
        nbytes -= layers * max(0, experts - n * top) * 6 * W * ff
        nbytes += (layers - rec) * (pos + n) * 4 * kv * HEAD + rec * gru * 8
        active = layers * 3 * top * W * ff + rec * 4 * W * gru + (layers - rec) * 2 * W * (heads + kv) * HEAD
        return nbytes, flops + 2.0 * n * active + (layers - rec) * seen * 4 * heads * HEAD
    heads, ssm, groups, ff, layers = NUFORAX[W]
    rec = sum(i % 4 == 1 for i in range(layers))
    own = layers - rec - sum(i % 4 == 3 for i in range(layers))
    inner, state = ssm * SSM_DIM, ssm * SSM_DIM * SSM_STATE
    seen = n * min(pos, WINDOW) + n * (n + 1) / 2 if pos + n <= WINDOW else n * WINDOW
    nbytes += (layers - rec) * min(pos + n, WINDOW) * 2 * (RANK + ROT) + rec * 8 * state
    active = layers * 2 * W * ff + rec * (3 * W * inner + 2 * W * groups * SSM_STATE) + own * W * (RANK + ROT)
    active += (layers - rec) * (heads * (HEAD + ROT) * W + W * heads * HEAD + 2 * heads * HEAD * RANK)
    return nbytes, flops + 2.0 * n * active + (layers - rec) * seen * 2 * heads * (2 * HEAD + ROT) + rec * n * 4.0 * state


def work(c):
    key, total = key_of(c), [0.0, 0.0]
    if c["sessions"] > 1:
        for j in range(c["decoded"]):
            each = [step_work(key, 1, kept_of(c, m) + j) for m in range(c["sessions"])]
            fixed = weight_bytes(key)
            fixed = fixed["layers"] + fixed["head"]
            total[0] += fixed + sum(b - fixed for b, _ in each)
            total[1] += sum(f for _, f in each)
    else:
        steps = [(c["pushed"], c["kept"])] if c["pushed"] else []
        steps += [(1, c["kept"] + c["pushed"] + j) for j in range(c["decoded"])]
        for n, pos in steps:
            b, f = step_work(key, n, pos)
            total[0] += b
            total[1] += f
    return {"bytes": total[0], "flops": total[1]}


def tolerance(c):
    # measured against exact(): 0.8e-3 for two layers to 3.3e-3 for 32 (16-bit caches, 11-bit weight tiles of batched steps); 4e-3 to 6e-3
    # for the bfloat16 models
    return {"rel": 1e-2 if c["model"] == "llama" else 2e-2}


# ---- the same in 64 bits -------------------------------------------------------------------

def exact(c, seed):
    key, rows = key_of(c), tokens_of(c, seed)
    n = c["pushed"] + c["decoded"]
    sequences = [torch.tensor(rows[m][:kept_of(c, m) + n]) for m in range(c["sessions"])]
    with torch.no_grad():
        f = {"llama": llama_exact, "sonuzen": sonuzen_exact, "nuforax": nuforax_exact}[key[0]]
        return [f(key, [s.cuda() for s in sequences])]


def normed(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def llama_exact(key, sequences):
    """Logits [sequences][VOCAB] after the last tokens; all sequences pass a layer together."""
    _, dim, layers, dtype = key
    slab = torch.tensor(blocks(dtype)[1], device="cuda")
    shapes = llama_tensors(key)
    heads, eps_free = dim // HEAD, 0.0

    def w(name):
        r, k = shapes[name]
        if k is None:
            return torch.tensor(llama_norm(name, r), device="cuda", dtype=torch.float64)
        at = (place(name, BLOCKS) + torch.arange(r * k // 32, device="cuda")) % BLOCKS
        return slab[at].reshape(r, k)

    def norm(x, weight):
        return x * weight / torch.sqrt(((x - x.mean(-1, keepdim=True)) ** 2).mean(-1, keepdim=True) + eps_free)

    theta = torch.tensor(np.power(10000.0, -np.arange(HEAD // 2, dtype=np.float32) / np.float32(HEAD // 2)).astype(np.float32).astype(np.float64), device="cuda")

    def turn(x):
        a = torch.arange(x.shape[0], device="cuda", dtype=torch.float64)[:, None, None] * theta
        u, v = x[..., 0::2], x[..., 1::2]
        return torch.stack([u * torch.cos(a) - v * torch.sin(a), u * torch.sin(a) + v * torch.cos(a)], -1).flatten(-2)

    lengths = [len(s) for s in sequences]
    x = w("tok_embeddings")[torch.cat(sequences)]
    for i in range(layers):
        p = f"layers.{i}."
        h = norm(x, w(p + "attention_norm"))
        q, k, v = (h @ w(f"{p}attention.{n}").T for n in ("wq", "wk", "wv"))
        out = []
        for a, b, d in zip(q.split(lengths), k.split(lengths), v.split(lengths)):
            T = len(a)
            a, b, d = turn(a.reshape(T, heads, HEAD)), turn(b.reshape(T, heads, HEAD)), d.reshape(T, heads, HEAD)
            later = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
            s = (torch.einsum("ihd,jhd->hij", a, b) * HEAD ** -0.5).masked_fill(later, -math.inf)
            out.append(torch.einsum("hij,jhd->ihd", s.softmax(-1), d).reshape(T, dim))
        x = x + torch.cat(out) @ w(p + "attention.wo").T
        h = norm(x, w(p + "ffn_norm"))
        gate = h @ w(p + "feed_forward.w1").T
        x = x + (gate * torch.sigmoid(gate) * (h @ w(p + "feed_forward.w3").T)) @ w(p + "feed_forward.w2").T
    last = torch.tensor(lengths, device="cuda").cumsum(0) - 1
    return norm(x[last], w("norm")) @ w("output").T


def folder_weights(key):
    tensors = folder_tensors(key)

    def value(bits):
        return torch.tensor((bits.astype(np.uint32) << 16).view(np.float32), device="cuda").double()

    def w(name):
        spec = tensors[name]
        if name.endswith("table"):
            return torch.tensor(table_of(name, spec[0][1], spec[1]), device="cuda", dtype=torch.long)
        if len(spec) == 3:
            return value(vector_of(name, spec))
        at = (place(name, VALUES) + torch.arange(math.prod(spec[0]), device="cuda")) % VALUES
        return value(normals_bf16(spec[1]))[at].reshape(spec[0])
    return w


def causal_taps(h, w):
    padded = torch.cat([h.new_zeros(w.shape[1] - 1, h.shape[1]), h])
    return sum(padded[j:j + len(h)] * w[:, j] for j in range(w.shape[1]))


def silu(x):
    return x * torch.sigmoid(x)


def sonuzen_exact(key, sequences):
    (tokens,), W, w = sequences, key[1], folder_weights(key)
    cfg, T = config_of(key), len(tokens)
    heads, kv, gru, experts, ff, top, _ = SONUZEN[W]
    eps, mult = cfg["norm"]["eps"], cfg["residual_mult"]
    x = w("embed")[tokens]
    i, j = torch.arange(T, device="cuda")[:, None], torch.arange(T, device="cuda")[None]
    for n, l in enumerate(cfg["layers"]):
        p = f"l{n}."
        h = normed(x, eps) * (1 + w(p + "norm1"))
        h = h + causal_taps(h, w(p + "canon1"))
        if l["type"] == "mingru":
            z = torch.sigmoid(h @ w(p + "mix.z").T + w(p + "mix.z.b"))
            u = h @ w(p + "mix.x").T + w(p + "mix.x.b")
            u = torch.where(u >= 0, u + 0.5, torch.sigmoid(u)) * z
            s, out = torch.zeros(gru, device="cuda", dtype=torch.float64), []
            for t in range(T):
                s = (1 - z[t]) * s + u[t]
                out.append(s)
            y = torch.stack(out) * silu(h @ w(p + "mix.g").T)
        else:
            q = normed((h @ w(p + "mix.q").T).reshape(T, heads, HEAD), eps) * w(p + "mix.q.norm")
            k = normed((h @ w(p + "mix.k").T).reshape(T, kv, HEAD), eps) * w(p + "mix.k.norm")
            v = (h @ w(p + "mix.v").T).reshape(T, kv, HEAD)
            r1, r2, out = w(p + "mix.r1"), w(p + "mix.r2"), []
            for a in range(heads):
                g = a // (heads // kv)
                s = q[:, a] @ k[:, g].T * HEAD ** -0.5 - r1[a] * torch.log1p(r2[a] * (i - j).clamp(min=0))
                s = s.masked_fill(j > i, -math.inf)
                m = s.amax(-1, keepdim=True).clamp(min=0)
                e = torch.exp(s - m)
                out.append(e @ v[:, g] / (torch.exp(-m) + e.sum(-1, keepdim=True)))
            y = torch.cat(out, -1)
        x = x + mult * normed(y @ w(p + "mix.o").T, eps) * (1 + w(p + "norm1b"))
        h = normed(x, eps) * (1 + w(p + "norm2"))
        h = h + causal_taps(h, w(p + "canon2"))
        chosen, y = w(p + "mlp.table")[tokens], torch.zeros_like(x)
        for e in range(experts):
            at = (chosen == e).any(-1).nonzero()[:, 0]
            a = h[at]
            y[at] += (silu(a @ w(f"{p}mlp.e{e}.gate").T) * (a @ w(f"{p}mlp.e{e}.up").T)) @ w(f"{p}mlp.e{e}.down").T / top
        x = x + mult * normed(y, eps) * (1 + w(p + "norm2b"))
    return (normed(x[-1:], eps) * (1 + w("final.norm"))) @ w("head").T


def nuforax_exact(key, sequences):
    (tokens,), W, w = sequences, key[1], folder_weights(key)
    cfg, T = config_of(key), len(tokens)
    eps, e = cfg["norm"]["eps"], cfg["embedding"]
    pair = torch.cat([tokens.new_tensor([BUCKETS]), (tokens[:-1] * e["bigram"]["mul_prev"] + tokens[1:] * e["bigram"]["mul_cur"]) % BUCKETS])
    x = w("embed")[tokens] * e["scale"] + w("bigram")[pair]
    r = cfg["layers"][0]["mixer"]["rot"]
    sc = r["scaling"]
    f = np.array([r["base"] ** (-2.0 * i / ROT) for i in range(ROT // 2)])

    def bend(t):
        return ROT * math.log(sc["original"] / (2 * math.pi * t)) / (2 * math.log(r["base"]))
    lo, hi = max(math.floor(bend(sc["fast"])), 0), min(math.ceil(bend(sc["slow"])), ROT - 1)
    ramp = np.clip((np.arange(ROT // 2) - lo) / max(hi - lo, 0.001), 0.0, 1.0)
    angles = torch.arange(T, device="cuda", dtype=torch.float64)[:, None] * torch.tensor(f / sc["factor"] * ramp + f * (1 - ramp), device="cuda")
    mult = 0.1 * math.log(sc["factor"]) + 1.0
    co, si = torch.cos(angles) * mult, torch.sin(angles) * mult

    def turn(a):
        c, s = (co, si) if a.dim() == 2 else (co[:, None], si[:, None])
        u, v = a[..., 0::2], a[..., 1::2]
        return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)

    d = torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]
    hidden = (d < 0) | (d >= WINDOW)
    kept = {}
    for n, l in enumerate(cfg["layers"]):
        p, mix, m = f"l{n}.", f"l{n}.mix.", l["mixer"]
        H = m["heads"]
        if l["type"] == "latent_attention":
            q = (x @ w(mix + "q").T).reshape(T, H, HEAD + ROT)
            q = torch.cat([q[..., :HEAD], turn(q[..., HEAD:])], -1)
            if "kv_from" not in m:
                a = x @ w(mix + "dkv").T
                kept[n] = normed(a[:, :RANK], eps) * w(mix + "dkv.norm"), turn(a[:, RANK:])
            c, k_rot = kept[m.get("kv_from", n)]
            k, v, sink, out = (c @ w(mix + "uk").T).reshape(T, H, HEAD), (c @ w(mix + "uv").T).reshape(T, H, HEAD), w(mix + "sink"), []
            for a in range(H):
                s = ((q[:, a, :HEAD] @ k[:, a].T + q[:, a, HEAD:] @ k_rot.T) * m["scale"]).masked_fill(hidden, -math.inf)
                top = s.amax(-1, keepdim=True).clamp(min=sink[a].item())
                b = torch.exp(s - top)
                out.append(b @ v[:, a] / (torch.exp(sink[a] - top) + b.sum(-1, keepdim=True)))
            y = torch.cat(out, -1) @ w(mix + "o").T
        else:
            inner, G = H * SSM_DIM, m["groups"]
            z, xbc, dt = (x @ w(mix + "in").T).split([inner, inner + 2 * G * SSM_STATE, H], -1)
            xbc = silu(causal_taps(xbc, w(mix + "conv")) + w(mix + "conv.b"))
            xs, B, C = xbc.split([inner, G * SSM_STATE, G * SSM_STATE], -1)
            xs = xs.reshape(T, H, SSM_DIM)
            B, C = (a.reshape(T, G, SSM_STATE).repeat_interleave(H // G, 1) for a in (B, C))
            dt = torch.logaddexp(dt + w(mix + "dt_bias"), torch.zeros((), device="cuda", dtype=torch.float64))
            decay = torch.exp(-torch.exp(w(mix + "A_log")) * dt)
            S, out, D = torch.zeros(H, SSM_STATE, SSM_DIM, device="cuda", dtype=torch.float64), [], w(mix + "D")
            for t in range(T):
                S = decay[t, :, None, None] * S + (dt[t, :, None] * B[t])[:, :, None] * xs[t][:, None]
                out.append((C[t][:, None] @ S)[:, 0])
            y = (torch.stack(out) + D[:, None] * xs).reshape(T, inner) * silu(z)
            y = normed(y.reshape(T, m["norm_groups"], -1), eps).reshape(T, inner) * w(mix + "norm")
            y = y @ w(mix + "o").T
        x = x + normed(y, eps) * w(p + "norm1")
        y = (x @ w(p + "mlp.up").T).clamp(min=0) ** 2 @ w(p + "mlp.down").T
        x = x + normed(y, eps) * w(p + "norm2")
    return (normed(x[-1:], eps) * w("final.norm")) @ w("embed").T
