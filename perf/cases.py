"""The work this library is used for, as cases that can be timed and compared: requests to language models (prompt, then greedy
generation, in one turn or several), the quantizer, and the matrix product behind both.

    listed()              the cases themselves
    draw(rng)             one more case of the same ranges
    prepare(case, seed)   inputs, weights and handles a program has before the call
    run(state)            one pass through the public entry points; returns its outputs
    work(case)            bytes and operations the pass cannot do without
    tolerance(case)       how far another correct implementation may be off
    exact(case, seed)     the same outputs in 64 bits, by plain torch

A request keeps its context: every pass clears it, feeds the prompt of a turn, generates `generate` tokens ("host": one
next_token call per token, as an interactive client does; "device": the chained loop on the GPU) and goes on with the next
turn's prompt behind them; the pass ends with the logits that follow the last token.  With generate = 0 it is the prompt alone
(time to the first token): its logits.

Weights are random with unit gain.  The output matrix also points from every token to one successor, so that the next token is
as clear as it usually is in a trained model and rounding does not decide it; routers read a few channels that only the
embedding writes, so that the choice of experts is clear for the same reason.
"""
import ctypes
import importlib.util
import json
import math
import os
import sys
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def library():
    if "llama_cu_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("llama_cu_b200", os.path.join(ROOT, "llama.cu_b200", "__init__.py"))
        module = importlib.util.module_from_spec(spec)
        sys.modules["llama_cu_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["llama_cu_b200"]


# ------------------------------------------------------------------ cases
def llama(name, dim, heads, layers, block, prompt, generate, loop="host", turns=1, vocab=32000, context=2048):
    return {"name": name, "kind": "llama", "dim": dim, "heads": heads, "layers": layers, "vocab": vocab, "block": block, "prompt": prompt,
            "generate": generate, "loop": loop, "turns": turns, "context": context}


def filulix(name, width, layers, prompt, generate, loop="host", turns=1, ff=None, dim=128, heads=None, wkv_dim=64, window=1024, pool=16, streams=4,
            passes=0, vocab=32000, context=4096):
    return {"name": name, "kind": "filulix", "width": width, "ff": ff or width * 11 // 4, "layers": layers, "heads": heads or width // 256, "dim": dim,
            "wkv_dim": wkv_dim, "window": window, "pool": pool, "streams": streams, "passes": passes, "vocab": vocab, "prompt": prompt,
            "generate": generate, "loop": loop, "turns": turns, "context": context}


def zibovik(name, width, layers, prompt, generate, loop="host", turns=1, ff=None, heads=None, dim=128, rot=64, rank=None, window=1024, experts=8, top=2,
            passes=0, vocab=32000, context=4096):
    return {"name": name, "kind": "zibovik", "width": width, "ff": ff or width * 11 // 8, "layers": layers, "heads": heads or width // 128, "dim": dim,
            "rot": rot, "rank": rank or min(512, width // 4), "window": window, "experts": experts, "top": top, "passes": passes, "vocab": vocab,
            "prompt": prompt, "generate": generate, "loop": loop, "turns": turns, "context": context}


def listed():
    return [
        # a short exchange with a small model: latency of every call, launches, host round trips
        llama("llama-1024 chat", 1024, 8, 8, 0, prompt=11, generate=16, turns=2),
        # the headline workload, interactive: 128 tokens in, answers token by token
        llama("llama-7b decode", 4096, 32, 32, 0, prompt=128, generate=32),
        # the same with 8-bit weights, two turns, generated on the device
        llama("llama-7b-u8 chat", 4096, 32, 32, 128, prompt=61, generate=20, loop="device", turns=2),
        # time to the first token of an ordinary prompt
        llama("llama-7b prompt 509", 4096, 32, 32, 0, prompt=509, generate=0),
        # a long document with 8-bit weights
        llama("llama-7b-u8 prompt 1999", 4096, 32, 32, 128, prompt=1999, generate=0),
        # the largest: a wide model behind a full context
        llama("llama-13b long", 5120, 40, 40, 0, prompt=2048, generate=16, loop="device", context=2304),
        # block models: long prompts, and answers token by token
        filulix("filulix-1024 prompt 2000", 1024, 8, prompt=2000, generate=0),
        filulix("filulix-2048 chat", 2048, 4, prompt=57, generate=24, turns=2),
        zibovik("zibovik-2048 prompt 2000", 2048, 4, prompt=2000, generate=0),
        zibovik("zibovik-1024 chat", 1024, 8, prompt=19, generate=32, loop="device"),
        # quantizing one large matrix (an embedding table) of a model
        {"name": "quantize 32000x4096", "kind": "quantize", "rows": 32000, "cols": 4096, "block": 128},
        # the operator by itself, on 8-bit weights that the caller owns
        {"name": "matmul u8 200 rows", "kind": "matmul", "m": 200, "k": 4096, "n": 11008, "block": 64},
    ]


def log_int(rng, lo, hi):
    """A whole number from lo to hi, spread evenly over its logarithm."""
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw_request(rng):
    generate = rng.choice([0, log_int(rng, 1, 32), log_int(rng, 1, 32)])
    prompt = log_int(rng, 1, 2000 if generate == 0 else 1000)
    return {"prompt": prompt, "generate": generate, "loop": rng.choice(["host", "device"]), "turns": rng.choice([1, 1, 2]) if prompt <= 500 else 1}


def draw(rng):
    kind = rng.choice(["llama", "llama", "llama", "llama", "filulix", "filulix", "zibovik", "zibovik", "quantize", "matmul"])
    if kind == "llama":
        dim = 256 * log_int(rng, 2, 16)
        c = llama(None, dim, dim // rng.choice([64, 128, 128]), log_int(rng, 2, 32), rng.choice([0, 0, 32, 64, 128, 128]), vocab=256 * log_int(rng, 8, 125),
                  context=rng.choice([2048, 2048, 2300, 4096]), **draw_request(rng))
    elif kind == "filulix":
        width = 8 * log_int(rng, 32, 256)
        c = filulix(None, width, rng.choice([2, 4, 6]), ff=8 * int(width * rng.uniform(0.25, 0.4)), dim=rng.choice([64, 96, 128, 128]),
                    heads=rng.choice([2, 4, 8]), wkv_dim=rng.choice([32, 64, 64]), window=log_int(rng, 64, 2048), pool=rng.choice([8, 16, 32]),
                    streams=rng.choice([2, 4, 4]), passes=rng.choice([0, 0, 2]), vocab=250 * log_int(rng, 8, 128), **draw_request(rng))
    elif kind == "zibovik":
        width = 8 * log_int(rng, 32, 256)
        c = zibovik(None, width, rng.choice([2, 3, 4]), ff=8 * int(width * rng.uniform(0.06, 0.17)), heads=max(2, width // 128),
                    dim=rng.choice([64, 128, 128]), rot=rng.choice([32, 64, 64]), rank=rng.choice([64, 128, 200, 256, 512]), window=log_int(rng, 64, 2048),
                    experts=rng.choice([4, 8, 8, 16]), top=rng.choice([1, 2, 2, 4]), passes=rng.choice([0, 0, 2]), vocab=250 * log_int(rng, 8, 128),
                    **draw_request(rng))
        c["ff"] = min(c["ff"], 11 * width // c["experts"])  # (all experts together: as many weights as in the listed cases)
    elif kind == "quantize":
        c = {"kind": kind, "rows": log_int(rng, 16, 32000), "cols": 128 * log_int(rng, 2, 64), "block": rng.choice([32, 64, 128])}
        c["rows"] = max(1, min(c["rows"], 32000 * 4096 // c["cols"]))
    else:
        c = {"kind": kind, "m": log_int(rng, 1, 600), "k": 256 * log_int(rng, 2, 43), "n": 32 * log_int(rng, 16, 344), "block": rng.choice([0, 0, 64, 128])}
    c.pop("name", None)
    return c


# ------------------------------------------------------------------ random values
class Values:
    """Random tensors on the GPU, made from the seed and their order alone."""

    def __init__(self, seed):
        self.seed, self.made = seed, 0

    def generator(self):
        self.made += 1
        return torch.Generator(device="cuda").manual_seed(self.seed * 100003 + self.made)

    def normal(self, *shape, std=1.0, dtype=torch.float32):
        return torch.randn(shape, generator=self.generator(), device="cuda").mul_(std).to(dtype)

    def matrix(self, rows, cols, gain=1.0, dtype=torch.float32):
        return self.normal(rows, cols, std=gain * cols ** -0.5, dtype=dtype)

    def between(self, lo, hi, *shape):
        return torch.rand(shape, generator=self.generator(), device="cuda").mul_(hi - lo).add_(lo)


def successor(token, vocab):
    return (token + vocab // 3 + 1) % vocab


def output_matrix(values, embedding):
    """Unit-gain noise, and for every token a step towards its successor."""
    vocab, width = embedding.shape
    return values.matrix(vocab, width) + torch.roll(embedding.float(), vocab // 3 + 1, 0) * (18.0 / width)


def prompts(case, seed):
    r = np.random.default_rng(seed)
    return [r.integers(3, case["vocab"], case["prompt"]).astype(np.int16) for _ in range(case["turns"])]


# ------------------------------------------------------------------ LLaMA family
def ffn_dim(dim):
    return (dim * 8 // 3 + 255) // 256 * 256


def blocks_of(w, bs):
    """8-bit values and fp16 scales of every block of bs along a row, value = (q - 127.5) * scale."""
    b = w.view(w.shape[0], -1, bs)
    scale = (b.abs().amax(2, keepdim=True) / 127.5).clamp_(min=1e-4).half()
    q = (b / scale.float()).add_(127.5).round_().clamp_(0, 255).to(torch.uint8)
    return q.view(w.shape), scale.view(w.shape[0], -1)


def llama_weights(case, seed):
    """(name, tensor or (8-bit values, scales)) in the order of the layers; the output matrix needs the embedding, so both come first."""
    v, d, f, bs = Values(seed), case["dim"], ffn_dim(case["dim"]), case["block"]

    def stored(w):
        return blocks_of(w, bs) if bs else w.half()

    embedding = stored(v.normal(case["vocab"], d))
    yield "tok_embeddings", embedding
    yield "output", stored(output_matrix(v, plain(embedding, torch.float32)))
    yield "norm", v.between(0.8, 1.2, d).half()
    out_gain = 0.7 / case["layers"] ** 0.5  # (the residual row keeps about the size of the embedding)
    for i in range(case["layers"]):
        p = "layers.%d." % i
        yield p + "attention_norm", v.between(0.8, 1.2, d).half()
        yield p + "ffn_norm", v.between(0.8, 1.2, d).half()
        for n in ("wq", "wk", "wv"):
            yield p + "attention." + n, stored(v.matrix(d, d, 1.2))
        yield p + "attention.wo", stored(v.matrix(d, d, 2 * out_gain))
        for n in ("w1", "w3"):
            yield p + "feed_forward." + n, stored(v.matrix(f, d))
        yield p + "feed_forward.w2", stored(v.matrix(d, f, 2 * out_gain))


def plain(t, dtype):
    if not isinstance(t, tuple):
        return t.to(dtype)
    q, scale = t
    return ((q.to(dtype) - 127.5).view(*scale.shape, -1) * scale.to(dtype)[..., None]).view(q.shape)


def llama_model(case, seed):
    lcu = library()
    handle = ctypes.c_void_p()
    lcu.check(lcu.lib.lcu_model_create(lcu.pack_params(case["dim"], 256, case["heads"], case["layers"], case["vocab"], 1e-5, case["block"]), None,
                                       ctypes.byref(handle)))
    model = lcu.Model(handle, case["vocab"], case["dim"])
    for name, t in llama_weights(case, seed):
        for which, part in enumerate(t if isinstance(t, tuple) else (t,)):
            ptr, size, _ = model.tensor(name, which)
            assert size == part.numel() * part.element_size(), (name, size)
            lcu.check(lcu.lib.lcu_memcpy_d2d(ptr, part.data_ptr(), size))
    torch.cuda.synchronize()
    return model


def llama_logits(case, seed, tokens, dtype=torch.float64):
    """Logits at every place of a sequence."""
    n, d, heads = len(tokens), case["dim"], case["heads"]
    hd = d // heads
    weights = llama_weights(case, seed)
    take = lambda: plain(next(weights)[1], dtype)  # noqa: E731
    x = take()[torch.from_numpy(tokens).long().cuda()]
    output, final = take(), take()
    angle = torch.arange(n, device="cuda", dtype=dtype)[:, None] * 10000.0 ** (-torch.arange(0, hd, 2, device="cuda", dtype=dtype) / hd)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def norm(x, w):
        return x / (x.square().mean(1, keepdim=True) + 1e-5).sqrt() * w

    def turn(a):
        a = a.view(n, heads, hd // 2, 2)
        u, w = a[..., 0], a[..., 1]
        return torch.stack((u * cos - w * sin, u * sin + w * cos), -1).view(n, heads, hd)

    hidden = torch.ones(n, n, dtype=torch.bool, device="cuda").triu_(1)
    for _ in range(case["layers"]):
        attn_norm, ffn_norm = take(), take()
        h = norm(x, attn_norm)
        q, k, v = turn(h @ take().T), turn(h @ take().T), (h @ take().T).view(n, heads, hd)
        s = torch.einsum("ihd,jhd->hij", q, k) * hd ** -0.5
        s = s.masked_fill_(hidden, -math.inf).softmax(2)
        x = x + torch.einsum("hij,jhd->ihd", s, v).reshape(n, d) @ take().T
        h = norm(x, ffn_norm)
        x = x + (torch.nn.functional.silu(h @ take().T) * (h @ take().T)) @ take().T
    return norm(x, final), output


# ------------------------------------------------------------------ block models (config.json + model.safetensors)
def run_order(case):
    """Layer of every layer run: with `passes`, the layers between the first and the last run that often."""
    n = case["layers"]
    return list(range(n)) if not case["passes"] else [0] + list(range(1, n - 1)) * case["passes"] + ([n - 1] if n > 1 else [])


def block_config(case):
    loop = {"start": 1, "stop": max(1, case["layers"] - 1), "times": case["passes"]} if case["passes"] else None
    c = {"vocab": case["vocab"], "width": case["width"], "norm": {"eps": 1e-6}}
    if case["kind"] == "filulix":
        h, dim = case["heads"], case["dim"]
        parallel = {"type": "parallel", "mlp": {"kind": "dense", "ff": case["ff"]},
                    "mixer": {"left": {"heads": h, "kv_heads": max(1, h // 4), "dim": dim, "vdim": dim, "scale": dim ** -0.5,
                                       "mask": {"size": case["window"], "pool": case["pool"]}}, "left_scale": 0.7,
                              "right": {"heads": h, "dim": dim, "vdim": dim, "decay": [1 - 2.0 ** (-5 - 7 * i / h) for i in range(h)],
                                        "rot": {"base": 10000.0, "dims": dim}}, "right_scale": 0.7}}
        wkv = {"type": "wkv", "mlp": {"kind": "dense", "ff": case["ff"]}, "mixer": {"heads": case["width"] // case["wkv_dim"], "dim": case["wkv_dim"]}}
        c.update(architecture="Filulix", streams=case["streams"], layers=[wkv if i % 2 else parallel for i in range(case["layers"])], loop=loop,
                 embedding={"scale": 1.0, "bigram": {"buckets": 4093, "mul_cur": 31, "mul_prev": 1009}})
    else:
        layer = {"type": "latent_attention",
                 "mixer": {"heads": case["heads"], "dim": case["dim"], "rot_dim": case["rot"], "vdim": case["dim"], "kv_rank": case["rank"],
                           "mask": {"size": case["window"]}, "rot": {"base": 10000.0, "dims": case["rot"]}, "scale": (case["dim"] + case["rot"]) ** -0.5},
                 "mlp": {"kind": "moe", "expert": {"ff": case["ff"]}, "router": {"experts": case["experts"], "top": case["top"]}}}
        c.update(architecture="Zibovik", layers=[layer] * case["layers"])
        if loop:
            c["loop"] = loop
    return c


def block_weights(case, seed):
    """{name: bfloat16 tensor} of a block model's file."""
    v, w, f, W = Values(seed), case["width"], case["ff"], {}
    out_gain = 1.0 / (2 * len(run_order(case))) ** 0.5

    def mat(name, rows, cols, gain=1.0):
        W[name] = v.matrix(rows, cols, gain)

    W["embed"] = v.normal(case["vocab"], w)
    if case["kind"] == "filulix":
        s, h, dim = case["streams"], case["heads"], case["dim"]
        W["bigram"] = v.normal(4094, w, std=0.3)
        for i in range(case["layers"]):
            p = "l%d." % i
            for q in "12":
                W[p + "norm" + q] = v.normal(w, std=0.1)
                W[p + "hc%s.in" % q] = v.between(0.7, 1.3, s) / s
                W[p + "hc%s.out" % q] = v.between(0.7, 1.3, s)
                W[p + "hc%s.mix" % q] = 0.9 * torch.eye(s, device="cuda") + v.between(0.05, 0.15, s, s) / s
            if i % 2 == 0:
                for n, rows in (("q", h * dim), ("k", max(1, h // 4) * dim), ("v", max(1, h // 4) * dim)):
                    mat(p + "mix.left." + n, rows, w)
                mat(p + "mix.left.o", w, h * dim, out_gain)
                for n in "qkvg":
                    mat(p + "mix.right." + n, h * dim, w)
                mat(p + "mix.right.o", w, h * dim, out_gain)
            else:
                d = case["wkv_dim"]
                n = w // d * d
                for x in "rkvgw":
                    W[p + "mix.mu." + x] = v.between(0, 1, w)
                for x in "rkvg":
                    mat(p + "mix." + x, n, w)
                mat(p + "mix.w1", 64, w)
                mat(p + "mix.w2", n, 64)
                W[p + "mix.w0"] = v.normal(n, std=1.5) - 3.0
                W[p + "mix.u"] = v.normal(n // d, d)
                W[p + "mix.norm"] = v.between(0.5, 1.5, n)
                mat(p + "mix.o", w, n, out_gain)
            mat(p + "mlp.gate", f, w)
            mat(p + "mlp.up", f, w)
            mat(p + "mlp.down", w, f, 2 * out_gain)
        W["final.norm"] = v.normal(w, std=0.1)
    else:
        h, dim, rot, rank, E = case["heads"], case["dim"], case["rot"], case["rank"], case["experts"]
        free = w - E  # the channels before it are what sublayers write
        W["embed"][:, free:] = torch.linspace(-2, 2, E, device="cuda")[torch.argsort(v.between(0, 1, case["vocab"], E), 1)]
        if case["passes"]:
            mat("loop.in", w, 2 * w)
            W["loop.in"][free:] = 0
            c = torch.arange(free, w, device="cuda")
            W["loop.in"][c, c], W["loop.in"][c, w + c] = 0.75, 0.25
        for i in range(case["layers"]):
            p = "l%d." % i
            for q in "12":
                W[p + "norm" + q] = v.between(0.8, 1.2, w)
                W[p + "norm%sb" % q] = v.between(0.8, 1.2, w)
                W[p + "ls" + q] = v.between(0.5, 1.5, w) * out_gain
            mat(p + "mix.q", h * (dim + rot), w)
            mat(p + "mix.dkv", rank + rot, w)
            W[p + "mix.dkv.norm"] = v.between(0.8, 1.2, rank)
            mat(p + "mix.uk", h * dim, rank)
            mat(p + "mix.uv", h * dim, rank)
            W[p + "mix.sink"] = v.normal(h)
            mat(p + "mix.g", h, w)
            mat(p + "mix.o", w, h * dim)
            W[p + "mix.o"][free:] = 0
            for e in range(E):
                mat(p + "mlp.e%d.gate" % e, f, w)
                mat(p + "mlp.e%d.up" % e, f, w)
                mat(p + "mlp.e%d.down" % e, w, f)
                W[p + "mlp.e%d.down" % e][free:] = 0
            W[p + "norm2"][free:] = 1
            W[p + "mlp.router"] = torch.zeros(E, w, device="cuda")
            W[p + "mlp.router"][torch.arange(E), free + torch.arange(E)] = 1
        W["final.norm"] = v.between(0.8, 1.2, w)
    W["head"] = output_matrix(v, W["embed"])
    return {k: t.bfloat16() for k, t in W.items()}


def block_model(case, seed):
    lcu = library()
    shm = "/dev/shm"
    roomy = os.path.isdir(shm) and os.statvfs(shm).f_bavail * os.statvfs(shm).f_frsize > 8 << 30
    with tempfile.TemporaryDirectory(dir=shm if roomy else None) as path:
        with open(os.path.join(path, "config.json"), "w") as f:
            json.dump(block_config(case), f)
        W, head, at = block_weights(case, seed), {}, 0
        for k, t in W.items():
            size = t.numel() * 2
            head[k] = {"dtype": "BF16", "shape": list(t.shape), "data_offsets": [at, at + size]}
            at += size
        h = json.dumps(head).encode()
        h += b" " * (-len(h) % 8)
        with open(os.path.join(path, "model.safetensors"), "wb") as f:
            f.write(len(h).to_bytes(8, "little") + h)
            for t in W.values():
                t.view(torch.int16).cpu().numpy().tofile(f)
        return lcu.Model.load(path, dtype="bfloat16")


def unit_rms(x):
    return x / (x.square().mean(-1, keepdim=True) + 1e-6).sqrt()


def filulix_logits(case, seed, tokens, dtype=torch.float64):
    W = {k: t.to(dtype) for k, t in block_weights(case, seed).items()}
    n, h, dim = len(tokens), case["heads"], case["dim"]
    ids = torch.from_numpy(tokens).long().cuda()
    pair = torch.cat((torch.tensor([4093], device="cuda"), (ids[:-1] * 1009 + ids[1:] * 31) % 4093))
    streams = (W["embed"][ids] + W["bigram"][pair]).expand(case["streams"], -1, -1)
    at = torch.arange(n, device="cuda")
    silu = torch.nn.functional.silu

    def attention(x, p):
        size, pool, g = case["window"], case["pool"], max(1, h // 4)
        q, k, v = ((x @ W[p + c].T).view(n, -1, dim) for c in "qkv")
        nb = n // pool
        k, v = (torch.cat((a, a[:nb * pool].view(nb, pool, g, dim).mean(1))).repeat_interleave(h // g, 1) for a in (k, v))
        s = torch.einsum("ihd,jhd->hij", q, k) * dim ** -0.5
        near = (at[None] <= at[:, None]) & (at[None] > at[:, None] - size)
        far = (torch.arange(nb, device="cuda") * pool + pool - 1)[None] <= at[:, None] - size
        s = s.masked_fill_(~torch.cat((near, far), 1), -math.inf).softmax(2)
        return torch.einsum("hij,jhd->ihd", s, v).reshape(n, -1) @ W[p + "o"].T

    def retention(x, p):
        q, k, v = ((x @ W[p + c].T).view(n, h, dim) for c in "qkv")
        angle = at[:, None] * 10000.0 ** (-2.0 * torch.arange(dim // 2, device="cuda", dtype=dtype) / dim)
        cos, sin = angle.cos()[:, None], angle.sin()[:, None]
        turn = lambda a: torch.cat((a[..., :dim // 2] * cos - a[..., dim // 2:] * sin, a[..., dim // 2:] * cos + a[..., :dim // 2] * sin), -1)  # noqa: E731
        s = torch.einsum("ihd,jhd->hij", turn(q), turn(k)) * dim ** -0.5
        decay = torch.tensor(np.float32([1 - 2.0 ** (-5 - 7 * i / h) for i in range(h)]), device="cuda").to(dtype)
        back = (at[:, None] - at[None]).to(dtype)
        s = s * torch.where(back >= 0, decay[:, None, None] ** back.clamp(min=0), 0.0)
        o = unit_rms(torch.einsum("hij,jhd->ihd", s, v)).reshape(n, -1)
        return (o * silu(x @ W[p + "g"].T)) @ W[p + "o"].T

    def wkv(x, p):
        d = case["wkv_dim"]
        back = torch.cat((torch.zeros_like(x[:1]), x[:-1]))
        mix = {c: x + (back - x) * W[p + "mu." + c] for c in "rkvgw"}
        r, k, v = ((mix[c] @ W[p + c].T).view(n, -1, d) for c in "rkv")
        w = (-(((mix["w"] @ W[p + "w1"].T).tanh() @ W[p + "w2"].T) + W[p + "w0"]).exp()).exp().view(n, -1, d, 1)
        u, S, o = W[p + "u"][:, :, None], torch.zeros(v.shape[1], d, d, dtype=dtype, device="cuda"), torch.empty_like(v)
        for t in range(n):
            kv = k[t, :, :, None] * v[t, :, None, :]
            o[t] = (r[t, :, None, :] @ (S + u * kv))[:, 0]
            S = w[t] * S + kv
        return (unit_rms(o).reshape(n, -1) * W[p + "norm"] * silu(mix["g"] @ W[p + "g"].T)) @ W[p + "o"].T

    def sublayer(streams, hc, norm, fn):
        y = fn(unit_rms(torch.einsum("s,std->td", W[hc + ".in"], streams)) * (1 + W[norm]))
        return torch.einsum("st,txd->sxd", W[hc + ".mix"].T, streams) + W[hc + ".out"][:, None, None] * y

    for i in run_order(case):
        p = "l%d." % i
        mixer = (lambda x: wkv(x, p + "mix.")) if i % 2 else (lambda x: 0.7 * (attention(x, p + "mix.left.") + retention(x, p + "mix.right.")))
        streams = sublayer(streams, p + "hc1", p + "norm1", mixer)
        streams = sublayer(streams, p + "hc2", p + "norm2", lambda x: (silu(x @ W[p + "mlp.gate"].T) * (x @ W[p + "mlp.up"].T)) @ W[p + "mlp.down"].T)
    return unit_rms(streams.sum(0)) * (1 + W["final.norm"]), W["head"]


def zibovik_logits(case, seed, tokens, dtype=torch.float64):
    W = {k: t.to(dtype) for k, t in block_weights(case, seed).items()}
    n, h, dim, rot, rank = len(tokens), case["heads"], case["dim"], case["rot"], case["rank"]
    x = start = W["embed"][torch.from_numpy(tokens).long().cuda()]
    at = torch.arange(n, device="cuda")
    angle = at[:, None] * 10000.0 ** (-2.0 * torch.arange(rot // 2, device="cuda", dtype=dtype) / rot)
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]
    unseen = (at[None] > at[:, None]) | (at[None] <= at[:, None] - case["window"])

    def turn(a):
        u, w = a[..., 0::2], a[..., 1::2]
        return torch.stack((u * cos - w * sin, w * cos + u * sin), -1).flatten(-2)

    def attention(x, p):
        q = (x @ W[p + "q"].T).view(n, h, dim + rot)
        down = x @ W[p + "dkv"].T
        c = unit_rms(down[:, :rank]) * W[p + "dkv.norm"]
        k = torch.cat(((c @ W[p + "uk"].T).view(n, h, dim), turn(down[:, None, rank:]).expand(n, h, rot)), 2)
        s = torch.einsum("ihd,jhd->hij", torch.cat((q[..., :dim], turn(q[..., dim:])), 2), k) * (dim + rot) ** -0.5
        s = torch.cat((s.masked_fill_(unseen, -math.inf), W[p + "sink"][:, None, None].expand(h, n, 1)), 2).softmax(2)[..., :n]
        o = torch.einsum("hij,jhd->ihd", s, (c @ W[p + "uv"].T).view(n, h, dim)) * (x @ W[p + "g"].T).sigmoid()[..., None]
        return o.reshape(n, -1) @ W[p + "o"].T

    def experts(x, p):
        score, pick = (x @ W[p + "router"].T).topk(case["top"], 1)
        out = torch.zeros_like(x)
        for e in range(case["experts"]):
            row, place = (pick == e).nonzero(as_tuple=True)
            r = x[row] * score[row, place].sigmoid()[:, None]
            w = p + "e%d." % e
            out.index_add_(0, row, (torch.nn.functional.silu(r @ W[w + "gate"].T) * (r @ W[w + "up"].T)) @ W[w + "down"].T)
        return out

    for i in run_order(case):
        p = "l%d." % i
        if case["passes"] and i == 1 < case["layers"] - 1:  # a pass over the looped layers begins
            x = torch.cat((x, start), 1) @ W["loop.in"].T
        for q, fn in (("1", lambda h: attention(h, p + "mix.")), ("2", lambda h: experts(h, p + "mlp."))):
            x = x + W[p + "ls" + q] * W[p + "norm%sb" % q] * unit_rms(fn(unit_rms(x) * W[p + "norm" + q]))
    return unit_rms(x) * W["final.norm"], W["head"]


# ------------------------------------------------------------------ states
class Session:
    """A model with a context, and the prompts of a request."""

    def __init__(self, case, seed):
        lcu = library()
        self.model = (llama_model if case["kind"] == "llama" else block_model)(case, seed)
        self.context = lcu.Context(self.model, context_len=case["context"], temperature=1.0)
        self.prompts, self.generate, self.chained = prompts(case, seed), case["generate"], case["loop"] == "device"

    def __del__(self):
        for part in ("context", "model"):
            if hasattr(self, part):
                getattr(self, part).close()


def prepare(case, seed):
    if case["kind"] in ("llama", "filulix", "zibovik"):
        return Session(case, seed)
    v = Values(seed)
    if case["kind"] == "quantize":
        w = v.normal(case["rows"], case["cols"], std=0.02, dtype=torch.float16)
        return {"kind": "quantize", "w": w, "q": torch.empty_like(w, dtype=torch.uint8), "block": case["block"],
                "scale": torch.empty(case["rows"], case["cols"] // case["block"], dtype=torch.float16, device="cuda")}
    s = {"kind": "matmul", "x": v.normal(case["m"], case["k"], dtype=torch.float16), "out": torch.empty(case["m"], case["n"], dtype=torch.float16, device="cuda"),
         "block": case["block"]}
    w = v.matrix(case["n"], case["k"])
    s["w"] = blocks_of(w, case["block"]) if case["block"] else w.half()
    return s


def answer(s):
    """The request of a session."""
    ctx, tokens = s.context, []
    ctx.clear_tokens()
    feed = None
    for prompt in s.prompts:
        feed = prompt if feed is None else np.concatenate((feed, prompt))
        if s.generate == 0:
            logits = ctx.step(feed, want=[len(feed) - 1])
            feed = None
            continue
        tokens.append(ctx.next_token(feed))
        if s.chained and s.generate > 1:
            tokens += ctx.decode_chained(tokens[-1], s.generate - 1)[0].tolist()
        else:
            for _ in range(s.generate - 1):
                tokens.append(ctx.next_token([tokens[-1]]))
        feed = np.int16([tokens[-1]])
    if s.generate:
        logits = ctx.step(feed, want=[0])
    return {"logits": logits, "tokens": np.array(tokens, np.int64)}


def run(state):
    if isinstance(state, Session):
        return answer(state)
    lcu, stream = library(), torch.cuda.current_stream().cuda_stream
    if state["kind"] == "quantize":
        w, q, scale = state["w"], state["q"], state["scale"]
        lcu.check(lcu.lib.lcu_quantize_absmax_uint8(q.data_ptr(), scale.data_ptr(), w.data_ptr(), w.shape[0], w.shape[1], state["block"], stream))
        return {"q": q, "scale": scale}
    x, w, out = state["x"], state["w"], state["out"]
    if state["block"]:
        lcu.check(lcu.lib.lcu_matmul_nt_fp16u8(out.data_ptr(), x.data_ptr(), w[0].data_ptr(), w[1].data_ptr(), x.shape[0], x.shape[1], out.shape[1],
                                               state["block"], 0.0, stream))
    else:
        lcu.check(lcu.lib.lcu_matmul_nt_f16(out.data_ptr(), x.data_ptr(), w.data_ptr(), x.shape[0], x.shape[1], out.shape[1], 0.0, stream))
    return {"out": out}


# ------------------------------------------------------------------ what a pass is and gives
def passes_of(case):
    """(rows, first position) of every pass over the model that a request takes."""
    out, pos = [], 0
    for t in range(case["turns"]):
        rows = case["prompt"] + (1 if t and case["generate"] else 0)
        out.append((rows, pos))
        pos += rows
        for _ in range(max(0, case["generate"] - 1)):
            out.append((1, pos))
            pos += 1
    if case["generate"]:
        out.append((1, pos))
    return out


def keys_seen(rows, pos, window=1 << 30):
    """Pairs of a row and a position that it sees, and the positions that any row sees."""
    return sum(min(pos + i + 1, window) for i in range(rows)), min(pos + rows, window - 1 + rows)


def work(case):
    kind = case["kind"]
    if kind == "quantize":
        n = case["rows"] * case["cols"]
        return {"bytes": 3 * n + 2 * n // case["block"], "flops": 3 * n}
    if kind == "matmul":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": 2 * m * (k + n) + n * k * (1 + 2 / case["block"] if case["block"] else 2), "flops": 2 * m * k * n}
    total, flops, vocab = 0.0, 0.0, case["vocab"]
    for rows, pos in passes_of(case):
        if kind == "llama":
            d, f = case["dim"], ffn_dim(case["dim"])
            per = 1 + 2 / case["block"] if case["block"] else 2
            pairs, keys = keys_seen(rows, pos)
            layer = 4 * d * d + 3 * d * f
            total += case["layers"] * (layer * per + 4 * keys * d) + vocab * d * per
            flops += case["layers"] * (2 * rows * layer + 4 * pairs * d) + 2 * vocab * d
            continue
        w, ff = case["width"], case["ff"]
        for i in run_order(case):
            if kind == "filulix":
                h, dim = case["heads"], case["dim"]
                g = max(1, h // 4)
                pairs, keys = keys_seen(rows, pos, case["window"])
                mats = 3 * w * ff + (w // case["wkv_dim"] * case["wkv_dim"] * 5 * w + 64 * 2 * w if i % 2 else w * dim * (7 * h + 2 * g))
                state = case["wkv_dim"] * w if i % 2 else h * dim * dim
                total += 2 * mats + 8 * state + (0 if i % 2 else 4 * keys * g * dim)
                flops += 2 * rows * mats + 6 * rows * state + (0 if i % 2 else 4 * pairs * h * dim)
            else:
                h, dim, rot, rank, top = case["heads"], case["dim"], case["rot"], case["rank"], case["top"]
                pairs, keys = keys_seen(rows, pos, case["window"])
                shared = w * (h * (dim + rot) + rank + rot + h * dim + h) + 2 * h * dim * rank
                total += 2 * (shared + 3 * w * ff * min(case["experts"], rows * top)) + 2 * keys * (rank + rot)
                flops += 2 * rows * (shared + 3 * w * ff * top) + 2 * pairs * h * (2 * dim + rot)
        total += 2 * vocab * w
        flops += 2 * vocab * w
    return {"bytes": total, "flops": flops}


def tolerance(case):
    if case["kind"] == "quantize":
        return "exact"
    if case["kind"] == "matmul":
        return {"rel": 1.2e-3}  # (half-precision results, and half-rounded weights behind 8-bit ones: 3e-4 off the 64-bit product)
    if case["kind"] == "llama":
        return {"rel": 1e-2}  # (half precision after every operator: 2.2e-3 off)
    return {"rel": 1.6e-2}  # (bfloat16 activations: 3.9e-3 off)


def sequence(case, seed):
    """Tokens a request feeds and the places among them that its tokens follow, the successors taken as given."""
    fed, places, tokens = [], [], []
    for prompt in prompts(case, seed):
        fed += prompt.tolist()
        for _ in range(case["generate"]):
            places.append(len(fed) - 1)
            tokens.append(successor(fed[-1], case["vocab"]))
            fed.append(tokens[-1])
    return np.array(fed, np.int64), places, np.array(tokens, np.int64)


def exact(case, seed):
    if case["kind"] == "quantize":
        w = prepare(case, seed)["w"].double().view(case["rows"], -1, case["block"])
        scale = (w.abs().amax(2) / 127.5).half().double()
        q = (w / scale[..., None] + 127.5).clamp(0, 255)
        return {"q": (q + 0.5).floor().to(torch.uint8).view(case["rows"], -1), "scale": scale}
    if case["kind"] == "matmul":
        s = prepare(case, seed)
        return {"out": s["x"].double() @ plain(s["w"], torch.float64).T}
    fed, places, tokens = sequence(case, seed)
    rows, output = {"llama": llama_logits, "filulix": filulix_logits, "zibovik": zibovik_logits}[case["kind"]](case, seed, fed)
    if places and not np.array_equal((rows[places] @ output.T).argmax(1).cpu().numpy(), tokens):
        return None  # (a next token that is not clear: the request took another way)
    return {"logits": rows[-1:] @ output.T, "tokens": tokens}
