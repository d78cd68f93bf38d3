"""Timed cases of this framework's work, through its public entry points.

Four kinds of case, each a dict of plain values:

  product    rows of activations times an int4 matrix (``cuda.gemv_q4``, ``cuda.gemv_q4p``, ``cuda.gemm_q4``)
  attention  one decoding step of attention over a ``cuda.kv_cache``
  decoder    the int4 ``Q4Decoder``: a prompt pass and/or single tokens behind ``ctx`` cached positions
  stack      a layer-stack model (``Zavilorn``, ``Daronex``): a new sequence, its prompt, then single tokens

``listed`` has the fixed cases, ``draw`` more of the same ranges.  ``exact`` restates every kind in plain torch
in 64 bits.  Weights and prompts are random; the distributions are those of the benchmark.
"""
import math
import zlib

import numpy as np
import torch

from cpp_tensorlib_b200 import cuda as tl
from cpp_tensorlib_b200 import daronex, zavilorn
from cpp_tensorlib_b200.decoder import Q4Decoder

GROUP = 32                                   # weights that share a scale
EPS = 1e-6


# ------------------------------------------------------------------------------------ the cases
def product(M, K, N, packed=False, name=None):
    return _named(name, kind="product", M=M, K=K, N=N, packed=packed)


def attention(n_q, n_kv, D, ctx, capacity, bf16, name=None):
    return _named(name, kind="attention", n_q=n_q, n_kv=n_kv, D=D, ctx=ctx, capacity=capacity, bf16=bf16)


def decoder(hidden, layers, n_q, n_kv, hd, ff, vocab, ctx, prompt, steps, bf16, name=None):
    """bf16: type of the caches.  `ctx` positions are cached before the pass."""
    return _named(name, kind="decoder", hidden=hidden, layers=layers, n_q=n_q, n_kv=n_kv, hd=hd, ff=ff, vocab=vocab,
                  ctx=ctx, prompt=prompt, steps=steps, bf16=bf16)


def stack(model, width, layers, vocab, window, prompt, steps, f32=False, name=None):
    return _named(name, kind="stack", model=model, width=width, layers=layers, vocab=vocab, window=window, prompt=prompt,
                  steps=steps, f32=f32)


def _named(name, **c):
    return dict(c, name=name) if name else c


def listed():
    big = dict(hidden=3584, layers=28, n_q=28, n_kv=4, hd=128, ff=18944, vocab=152064)
    small = dict(hidden=896, layers=24, n_q=14, n_kv=2, hd=64, ff=4864, vocab=151936)
    return [
        # one projection of a small decoder on the storage layout: the smallest call, latency counts
        product(1, 896, 4864, name="gemv_small"),
        # a few rows at once (short drafts, a small batch) against a large feed-forward matrix
        product(8, 3584, 18944, name="gemm_rows_8"),
        # every head with keys of its own, long context: the largest cache read
        attention(28, 28, 128, 32768, 32768, False, name="attend_heads_32k"),
        # grouped heads on a 16-bit cache, a ragged position in a larger cache
        attention(28, 4, 128, 12345, 16384, True, name="attend_grouped_bf16"),
        # the benchmark: single tokens of the 7B shape behind 4096 positions
        decoder(**big, ctx=4096, prompt=0, steps=4, bf16=False, name="decode_7b"),
        # the 0.5B shape with the command line's 16-bit caches: short launches
        decoder(**small, ctx=131, prompt=0, steps=16, bf16=True, name="decode_half_b"),
        # a prompt at both shapes, again as the command line runs it (of 7B the four layers of the benchmark's option)
        decoder(**dict(big, layers=4), ctx=0, prompt=1000, steps=0, bf16=True, name="prompt_7b"),
        decoder(**small, ctx=0, prompt=517, steps=0, bf16=True, name="prompt_half_b"),
        # a document read by each layer stack, at the benchmark's sizes
        stack("zavilorn", 2048, 8, 65536, 2048, 4096, 0, name="zavilorn_prompt"),
        stack("daronex", 2048, 8, 65536, 2048, 3001, 0, name="daronex_prompt"),
        # a short question and its answer, token by token
        stack("zavilorn", 2048, 8, 65536, 2048, 150, 48, name="zavilorn_answer"),
        stack("daronex", 2048, 8, 65536, 2048, 700, 48, name="daronex_answer"),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["product", "product", "attention", "decoder", "decoder", "stack", "stack"])
    if kind == "product":
        rows = rng.choice(["one", "few", "many"])
        if rows != "many":
            M = 1 if rows == "one" else _log(rng, 2, 8)
            return product(M, 32 * _log(rng, 16, 592), _log(rng, 256, 37888), M == 1 and rng.random() < 0.5)
        # a prompt's rows: the matrices of the two decoders and ragged neighbours of theirs
        K, N, most = rng.choice([(896, 9728, 1024), (896, 1152, 1024), (896, 896, 1024), (4864, 896, 512), (3584, 4608, 256),
                                 (3584, 3584, 256), (18944, 3584, 256)])
        return product(_log(rng, 33, most), K, N - rng.choice([0, 0, 1, 7, 64, 100]))
    if kind == "attention":
        n_kv, group = rng.choice([(28, 1), (14, 1), (8, 4), (8, 1), (4, 7), (4, 8), (2, 7), (2, 5), (2, 2), (1, 7)])
        ctx = _log(rng, 16, 32768)
        return attention(n_kv * group, n_kv, rng.choice([64, 128]), ctx, min(32768, ctx + rng.choice([0, 1, 17, 128, 4096])),
                         rng.random() < 0.5)
    if kind == "decoder":
        reads = rng.random() < 0.5
        n_kv, group, hd = rng.choice([(2, 7, 64), (2, 4, 64), (4, 4, 64), (1, 7, 128), (8, 1, 128)] if reads else
                                     [(2, 7, 64), (2, 6, 128), (4, 7, 128), (4, 4, 128), (8, 4, 64), (2, 8, 128), (12, 1, 64)])
        hidden = n_kv * group * hd
        ff, layers, bf16 = 128 * round(hidden * rng.uniform(2.6, 5.4) / 128), rng.randint(2, 12), reads or rng.random() < 0.5
        ctx, prompt, steps = (_log(rng, 1, 8192), 0, _log(rng, 1, 16))
        if reads:
            ctx, prompt, steps = rng.choice([(0, _log(rng, 33, 2048), 0), (0, _log(rng, 33, 512), 8), (ctx // 2, _log(rng, 33, 512), 0)])
        return decoder(hidden, layers, n_kv * group, n_kv, hd, ff, _log(rng, 4000, 152064), ctx, prompt, steps, bf16)
    f32 = rng.random() < 0.2
    prompt, steps = rng.choice([(_log(rng, 128, 256 if f32 else 4096), 0), (_log(rng, 1, 256 if f32 else 1024), rng.randint(8, 48))])
    return stack(rng.choice(["zavilorn", "daronex"]), 256 * rng.randint(2, 8), rng.choice([4, 8]), _log(rng, 4000, 65536),
                 rng.choice([256, 1000, 2048]), prompt, steps, f32)


# ------------------------------------------------------------------------------------ inputs
def _normal(seed, what, shape, std=1.0, mean=0.0):
    g = torch.Generator(device="cuda").manual_seed((seed * 1000003 + zlib.crc32(what.encode())) & 0x7FFFFFFF)
    return torch.randn(shape, generator=g, device="cuda").mul_(std).add_(mean)


def _ids(seed, vocab, n):
    return [int(t) for t in np.random.default_rng(seed).integers(0, vocab, n)]


def _linears(c):
    """Name -> (K, N) of a decoder layer's matrices."""
    heads = (c["n_q"] + 2 * c["n_kv"]) * c["hd"]
    return dict(wqkv=(c["hidden"], heads), wo=(c["n_q"] * c["hd"], c["hidden"]), wgu=(c["hidden"], 2 * c["ff"]),
                wd=(c["ff"], c["hidden"]))


def _layer_vectors(c):
    return dict(an=(c["hidden"], 1.0), fn=(c["hidden"], 1.0), bq=(c["n_q"] * c["hd"], 0.0), bk=(c["n_kv"] * c["hd"], 0.0),
                bv=(c["n_kv"] * c["hd"], 0.0))


def _cached(c, seed, layer):
    return [_normal(seed, f"{layer}{n}", (c["n_kv"], c["ctx"], c["hd"])) for n in ("cached k", "cached v")]


ROPE_BASE = 1e6


def _config(c):
    """A layer-stack configuration: the benchmark's proportions at `width`."""
    w, n = c["width"], c["width"] // 128
    if c["model"] == "zavilorn":
        kv = max(1, n // 4)
        par = dict(type="parallel", mlp=dict(kind="dense", ff=int(2.75 * w), limit=7.0), mixer=dict(
            left=dict(heads=kv * (n // kv), kv_heads=kv, dim=128, vdim=128, mask=dict(size=c["window"], keep_first=4),
                      rot=dict(base=1e5, dims=64), scale=128 ** -0.5),
            right=dict(heads=n, kv_heads=n // 2, dim=128, vdim=128, conv=4), left_scale=1.0, right_scale=0.5))
        mam = dict(type="mamba2", mlp=None, mixer=dict(heads=w // 32, groups=8, state=128, vdim=64, conv=4, norm_groups=8))
        return dict(architecture="Zavilorn", vocab=c["vocab"], width=w, embedding=dict(scale=1.0), norm=dict(eps=EPS),
                    layers=[par, mam, mam, mam] * (c["layers"] // 4))
    lat = dict(heads=n, dim=128, rot_dim=64, vdim=128, q_rank=w // 2, kv_rank=512, rot=dict(base=1e5, dims=64),
               scale=192 ** -0.5)
    mlp = dict(kind="dense", ff=4 * w)
    gla = dict(type="gla", mlp=mlp, mixer=dict(heads=w // 256, dim=128, vdim=256, tau=16.0))
    win = dict(type="latent_attention_2", mlp=mlp, mixer=dict(lat, mask=dict(size=c["window"])))
    layers = [dict(type="latent_attention", mlp=mlp, mixer=lat), gla, win, gla,
              dict(type="latent_attention", mlp=mlp, mixer=dict(lat, kv_from=0)), gla, win, gla]
    return dict(architecture="Daronex", vocab=c["vocab"], width=w, norm=dict(eps=EPS), logit_scale=1.0,
                layers=layers[:c["layers"]])


class Weights:
    """Random tensors of a layer stack, made on the GPU, with values that 16 bits hold: what a weight file has."""

    def __init__(self, case, seed):
        self.seed, self.model = seed, case["model"]
        self.shapes = {"zavilorn": zavilorn, "daronex": daronex}[self.model].tensor_shapes(_config(case))

    def device(self, name):
        shape = self.shapes[name]
        centre, std = 0.0, 1.0
        if name.endswith(("norm1", "norm2")) or name == "final.norm":
            centre, std = (0.0 if self.model == "daronex" else 1.0), 0.1
        elif name.endswith("norm"):
            centre, std = 1.0, 0.1
        elif name.endswith("A_log"):
            std = 0.3
        elif name.endswith("dt_bias"):
            centre, std = -3.0, 0.5
        elif name.endswith("a2.b"):
            centre = 3.0
        elif len(shape) == 2 and name != "embed":
            std = shape[1] ** -0.5
        return _normal(self.seed, name, shape, std, centre).to(torch.bfloat16)

    def raw(self, name):
        return self.device(name).view(torch.int16).cpu().numpy().view(np.uint16)

    def f32(self, name):
        return self.device(name).float().cpu().numpy()

    def shape(self, name):
        return self.shapes[name]

    def __contains__(self, name):
        return name in self.shapes


# ------------------------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_product(c, seed):
    wq = tl.to_q4(_normal(seed, "w", (c["K"], c["N"]), 0.02))
    x = _normal(seed, "x", (c["M"], c["K"]))
    if c["packed"]:
        return dict(run=_run_packed, x=x.reshape(-1), w=tl.Q4Packed(wq))
    if c["M"] == 1:
        return dict(run=_run_row, x=x.reshape(-1), w=wq)
    return dict(run=_run_rows, x=x, w=wq)


def _run_packed(s):
    return tl.gemv_q4p(s["x"], s["w"])


def _run_row(s):
    return tl.gemv_q4(s["x"], s["w"])


def _run_rows(s):
    return tl.gemm_q4(s["x"], s["w"])


def _prepare_attention(c, seed):
    cache = tl.kv_cache(c["n_kv"], c["capacity"], c["D"], dtype=torch.bfloat16 if c["bf16"] else torch.float32)
    cache.fill(*[_normal(seed, n, (c["n_kv"], c["ctx"], c["D"])) for n in "kv"])
    return dict(run=_run_attention, cache=cache, q=_normal(seed, "q", (c["n_q"], c["D"])), scale=c["D"] ** -0.5)


def _run_attention(s):
    return s["cache"].attn(s["q"], s["scale"])


def _prepare_decoder(c, seed):
    cfg = dict({k: c[k] for k in ("hidden", "layers", "n_q", "n_kv", "hd", "ff", "vocab")}, eps=EPS, rope_base=ROPE_BASE)
    d = Q4Decoder(cfg, c["ctx"] + c["prompt"] + c["steps"] + 1, kv_dtype="bf16" if c["bf16"] else "f32")
    d.set_vector_full(0, "embed", _normal(seed, "embed", (c["vocab"], c["hidden"]), 0.02))
    d.set_vector_full(0, "onorm", _normal(seed, "onorm", (c["hidden"],), 0.02, 1.0))
    d.set_linear_full(0, "lm_head", _normal(seed, "lm_head", (c["hidden"], c["vocab"]), 0.02))
    for l in range(c["layers"]):
        for n, shape in _linears(c).items():
            d.set_linear_full(l, n, _normal(seed, f"{l}{n}", shape, 0.02))
        for n, (size, centre) in _layer_vectors(c).items():
            d.set_vector_full(l, n, _normal(seed, f"{l}{n}", (size,), 0.02, centre))
        if c["ctx"]:
            d.fill_kv(l, *_cached(c, seed, l))
    d.capture()
    ids = _ids(seed, c["vocab"], c["prompt"] + c["steps"])
    return dict(run=_run_decoder, d=d, ctx=c["ctx"], prompt=ids[:c["prompt"]], tokens=ids[c["prompt"]:])


def _run_decoder(s):
    """Ids of the following tokens are left out: the best two logits can be closer than rounding."""
    d = s["d"]
    d.set_pos(s["ctx"])
    if s["prompt"]:
        d.prefill(s["prompt"])
    for t in s["tokens"]:
        d.step(t)
    return dict(logits=d.logits())


def _prepare_stack(c, seed):
    cls = {"zavilorn": zavilorn.Zavilorn, "daronex": daronex.Daronex}[c["model"]]
    d = cls.from_folder(_config(c), Weights(c, seed), "float32" if c["f32"] else "bfloat16", c["prompt"] + c["steps"] + 1)
    d.capture()
    ids = _ids(seed, c["vocab"], c["prompt"] + c["steps"])
    return dict(run=_run_stack, d=d, prompt=ids[:c["prompt"]], tokens=ids[c["prompt"]:])


def _run_stack(s):
    d = s["d"]
    d.set_pos(0)
    if len(s["prompt"]) > 1:
        d.prefill(s["prompt"])
    else:
        d.step(s["prompt"][0])
    for t in s["tokens"]:
        d.step(t)
    return dict(logits=d.host_logits())


# ------------------------------------------------------------------------------------ work and tolerance
def _attended(ctx, n, window=None, keep=0):
    """(pairs, rows in sight of any of them) of `n` queries behind `ctx` positions."""
    pairs = sum(min(p + 1, window + keep) if window else p + 1 for p in range(ctx, ctx + n))
    return pairs, ctx + n if not window else min(ctx + n, window + keep + n)


def work(case):
    return globals()["_work_" + case["kind"]](case)


def _q4_bytes(K, N):
    return N * K / 2 + N * (K // GROUP) * 4


def _work_product(c):
    M, K, N = c["M"], c["K"], c["N"]
    return {"bytes": _q4_bytes(K, N) + 4 * M * (K + N), "flops": 2 * M * N * K}


def _work_attention(c):
    rows = 2 * c["n_kv"] * c["ctx"] * c["D"]
    return {"bytes": rows * (2 if c["bf16"] else 4) + 8 * c["n_q"] * c["D"], "flops": 4 * c["n_q"] * c["ctx"] * c["D"]}


def _work_decoder(c):
    mats, head = c["layers"] * sum(K * N for K, N in _linears(c).values()), c["hidden"] * c["vocab"]
    row = 2 * c["n_kv"] * c["hd"] * (2 if c["bf16"] else 4) * c["layers"]
    nbytes = flops = 0
    runs = ([(c["ctx"], c["prompt"])] if c["prompt"] else []) + [(c["ctx"] + c["prompt"] + i, 1) for i in range(c["steps"])]
    for at, n in runs:
        pairs, seen = _attended(at, n)
        nbytes += (mats + head) * 0.625 + row * seen + 4 * (n * c["hidden"] + c["vocab"])
        flops += 2 * (mats * n + head) + 4 * c["n_q"] * c["hd"] * pairs * c["layers"]
    return {"bytes": nbytes, "flops": flops}


def _work_stack(c):
    cfg = _config(c)
    shapes = {"zavilorn": zavilorn, "daronex": daronex}[c["model"]].tensor_shapes(cfg)
    elt = 4 if c["f32"] else 2
    head = c["width"] * c["vocab"]
    mats = sum(s[0] * s[1] for n, s in shapes.items() if len(s) == 2 and n not in ("embed", "head") and not n.endswith("conv"))
    nbytes = flops = 0
    for at, n in [(0, c["prompt"])] + [(c["prompt"] + i, 1) for i in range(c["steps"])]:
        nbytes += elt * (mats + head + n * c["width"]) + 4 * c["vocab"]
        flops += 2 * (mats * n + head)
        for L in cfg["layers"]:
            m = L["mixer"]
            if L["type"] == "parallel":
                a, r = m["left"], m["right"]
                pairs, seen = _attended(at, n, a["mask"]["size"], a["mask"]["keep_first"])
                state = r["heads"] * r["dim"] * r["vdim"]
                nbytes += 2 * a["kv_heads"] * a["dim"] * elt * seen + 4 * state * (2 if at else 1)
                flops += 4 * a["heads"] * a["dim"] * pairs + 8 * state * n
            elif L["type"] in ("mamba2", "gla"):
                state = m["heads"] * m["vdim"] * m["state" if L["type"] == "mamba2" else "dim"]
                nbytes += 4 * state * (2 if at else 1)
                flops += 5 * state * n
            else:
                pairs, seen = _attended(at, n, m["mask"]["size"] if "mask" in m else None)
                nbytes += (m["kv_rank"] + m["rot_dim"]) * elt * seen
                flops += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]) * pairs
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    if case["kind"] == "product":
        return {"rel": 4e-6, "max": 1e-4}
    if case["kind"] == "attention":
        return {"rel": 2e-6, "max": 4e-5}
    if case["kind"] == "decoder":
        return {"rel": 8e-3, "max": 8e-2} if case["bf16"] else {"rel": 4e-5, "max": 4e-4}
    return {"rel": 2e-4, "max": 2e-3} if case["f32"] else {"rel": 3e-2, "max": 0.3}


# ------------------------------------------------------------------------------------ the same in 64 bits
def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _quantised(w):
    """[K, N] in 64 bits: groups of 32 along K over a seventh of their largest, rounded half away from zero."""
    K, N = w.shape
    out = torch.empty((K, N), dtype=torch.float64, device=w.device)
    for a in range(0, N, 8192):
        g = w[:, a:a + 8192].reshape(K // GROUP, GROUP, -1)
        s = g.abs().amax(1, keepdim=True).clamp_min(1e-8) / torch.full((), 7.0, device=w.device)   # a number would be inverted first
        q = (g / s).double()
        q = (q.sign() * (q.abs() + 0.5).floor()).clamp_(-8, 7)
        out[:, a:a + 8192] = (q * s.double()).reshape(K, -1)
    return out


def _exact_product(c, seed):
    y = _normal(seed, "x", (c["M"], c["K"])).double() @ _quantised(_normal(seed, "w", (c["K"], c["N"]), 0.02))
    return y[0] if c["M"] == 1 else y


def _attend(q, k, v, scale, at, window=None, keep=0):
    """q [H, T, D] at positions at.., k [G, n, D], v [G, n, E] of positions 0.. -> [H, T, E]."""
    H, T, D = q.shape
    G, n, E = v.shape
    out = torch.empty((H, T, E), dtype=q.dtype, device=q.device)
    for a in range(0, T, 512):
        b = min(a + 512, T)
        i = torch.arange(at + a, at + b, device=q.device)[:, None]
        j = torch.arange(n, device=q.device)[None]
        hidden = j > i
        if window is not None:
            hidden |= (i - j >= window) & (j >= keep)
        s = q[:, a:b].reshape(G, H // G, b - a, D) @ k[:, None].transpose(2, 3) * scale
        out[:, a:b] = (s.masked_fill_(hidden, -math.inf).softmax(-1) @ v[:, None]).reshape(H, b - a, E)
    return out


def _exact_attention(c, seed):
    k, v = [_normal(seed, n, (c["n_kv"], c["ctx"], c["D"])) for n in "kv"]
    if c["bf16"]:
        k, v = k.to(torch.bfloat16), v.to(torch.bfloat16)
    q = _normal(seed, "q", (c["n_q"], c["D"])).double()
    return _attend(q[:, None], k.double(), v.double(), c["D"] ** -0.5, c["ctx"] - 1)[:, 0]


def _norm(x, w, parts=1):
    s = x.reshape(x.shape[:-1] + (parts, -1))
    return (s / (s.square().mean(-1, keepdim=True) + EPS).sqrt()).reshape(x.shape) * w


def _angles(at, n, dims, base):
    f = base ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device="cuda") / dims)
    a = torch.arange(at, at + n, dtype=torch.float64, device="cuda")[:, None] * f
    return a.cos(), a.sin()


def _rotate(x, at, dims, base, half):
    """x [..., T, D]: pairs (2i, 2i + 1) of the first `dims`, or with `half` (i, i + dims / 2)."""
    c, s = _angles(at, x.shape[-2], dims, base)
    first, second = (slice(0, dims // 2), slice(dims // 2, dims)) if half else (slice(0, dims, 2), slice(1, dims, 2))
    out = x.clone()
    out[..., first] = x[..., first] * c - x[..., second] * s
    out[..., second] = x[..., second] * c + x[..., first] * s
    return out


def _silu(z):
    return z * z.sigmoid()


def _heads(x, h):
    return x.reshape(x.shape[0], h, -1).transpose(0, 1)


def _exact_decoder(c, seed):
    """A prompt and the single tokens behind it are one causal run.  Cached rows as the cache holds them, the run's
    own rows in 64 bits."""
    vec = lambda n, size, centre: _normal(seed, n, (size,), 0.02, centre).double()
    ids = torch.tensor(_ids(seed, c["vocab"], c["prompt"] + c["steps"]), device="cuda")
    x = _normal(seed, "embed", (c["vocab"], c["hidden"]), 0.02)[ids].double()
    n, nq, nk = len(ids), c["n_q"] * c["hd"], c["n_kv"] * c["hd"]
    for l in range(c["layers"]):
        W = {k: (lambda k=k, s=s: _quantised(_normal(seed, f"{l}{k}", s, 0.02))) for k, s in _linears(c).items()}
        V = {k: vec(f"{l}{k}", size, centre) for k, (size, centre) in _layer_vectors(c).items()}
        q, k, v = (_norm(x, V["an"]) @ W["wqkv"]()).split([nq, nk, nk], 1)
        q, k, v = _heads(q + V["bq"], c["n_q"]), _heads(k + V["bk"], c["n_kv"]), _heads(v + V["bv"], c["n_kv"])
        q, k = (_rotate(a, c["ctx"], c["hd"], ROPE_BASE, True) for a in (q, k))
        if c["ctx"]:
            kc, vc = (a.to(torch.bfloat16).double() if c["bf16"] else a.double() for a in _cached(c, seed, l))
            k, v = torch.cat([kc, k], 1), torch.cat([vc, v], 1)
        o = _attend(q, k, v, c["hd"] ** -0.5, c["ctx"])
        x = x + o.transpose(0, 1).reshape(n, nq) @ W["wo"]()
        gate, up = (_norm(x, V["fn"]) @ W["wgu"]()).chunk(2, 1)
        x = x + (_silu(gate) * up) @ W["wd"]()
    x = _norm(x[-1], vec("onorm", c["hidden"], 1.0))
    return dict(logits=x @ _quantised(_normal(seed, "lm_head", (c["hidden"], c["vocab"]), 0.02)))


def _conv(x, w, b=None):
    taps = w.shape[1]
    p = torch.cat([x.new_zeros((taps - 1, x.shape[1])), x])
    y = sum(p[a:a + len(x)] * w[:, a] for a in range(taps))
    return _silu(y if b is None else y + b)


def _scan(T, S, step):
    return torch.stack([step(S, t) for t in range(T)])


def _delta(h, W, p, c):
    T, H, G, D, E = len(h), c["heads"], c["kv_heads"], c["dim"], c["vdim"]
    q, k, v = (_conv(h @ W(p + n).T, W(p + n + ".conv")) for n in "qkv")
    unit = lambda a: a / (a.square().sum(-1, keepdim=True) + 1e-6).sqrt()
    q, k = (unit(a.reshape(T, G, D)).repeat_interleave(H // G, 1) for a in (q, k))
    q, v = q * D ** -0.5, v.reshape(T, H, E)
    beta = (h @ W(p + "b").T).sigmoid()
    decay = (-W(p + "A_log").exp() * torch.nn.functional.softplus(h @ W(p + "a").T + W(p + "dt_bias"))).exp()

    def step(S, t):
        S.mul_(decay[t, :, None, None])
        u = beta[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
        S.baddbmm_(k[t, :, :, None], u[:, None])
        return (q[t, :, None] @ S)[:, 0]
    o = _scan(T, h.new_zeros((H, D, E)), step)
    o = _norm(o, W(p + "norm")) * _silu(h @ W(p + "g").T).reshape(T, H, E)
    return o.reshape(T, H * E) @ W(p + "o").T


def _mamba2(h, W, p, c):
    T, H, E, N, G = len(h), c["heads"], c["vdim"], c["state"], c["groups"]
    inner = H * E
    z, xbc, dt = (h @ W(p + "in").T).split([inner, inner + 2 * G * N, H], 1)
    x, B, C = _conv(xbc, W(p + "conv"), W(p + "conv.b")).split([inner, G * N, G * N], 1)
    x = x.reshape(T, H, E)
    B, C = (a.reshape(T, G, N).repeat_interleave(H // G, 1) for a in (B, C))
    dt = torch.nn.functional.softplus(dt + W(p + "dt_bias"))
    decay, xs = (-W(p + "A_log").exp() * dt).exp(), x * dt[..., None]

    def step(S, t):
        S.mul_(decay[t, :, None, None]).baddbmm_(B[t, :, :, None], xs[t, :, None])
        return (C[t, :, None] @ S)[:, 0]
    y = _scan(T, h.new_zeros((H, N, E)), step) + W(p + "D")[:, None] * x
    return _norm(y.reshape(T, inner) * _silu(z), W(p + "norm"), c["norm_groups"]) @ W(p + "o").T


def _window(h, W, p, c):
    T, H, G = len(h), c["heads"], c["kv_heads"]
    q, k = (_norm(h @ W(p + n).T, W(p + n + ".norm")) for n in "qk")
    q, k, v = _heads(q, H), _heads(k, G), _heads(h @ W(p + "v").T, G)
    q, k = (_rotate(a, 0, c["rot"]["dims"], c["rot"]["base"], False) for a in (q, k))
    o = _attend(q, k, v, c["scale"], 0, c["mask"]["size"], c["mask"]["keep_first"])
    return (o.transpose(0, 1).reshape(T, -1) * (h @ W(p + "g").T).sigmoid()) @ W(p + "o").T


def _zavilorn(cfg, W, ids, last):
    x = W("embed")[ids]
    for i, L in enumerate(cfg["layers"]):
        p, c = f"l{i}.", L["mixer"]
        h = _norm(x, W(p + "norm1"))
        if L["type"] == "parallel":
            x = x + c["left_scale"] * _window(h, W, p + "mix.left.", c["left"]) + \
                c["right_scale"] * _delta(h, W, p + "mix.right.", c["right"])
        else:
            x = x + _mamba2(h, W, p + "mix.", c)
        if L.get("mlp"):
            h, lim = _norm(x, W(p + "norm2")), L["mlp"]["limit"]
            g, u = (h @ W(p + "mlp.gate").T).clamp(max=lim), (h @ W(p + "mlp.up").T).clamp(-lim, lim)
            x = x + (g * (1.702 * g).sigmoid() * (u + 1)) @ W(p + "mlp.down").T
    return _norm(x[last], W("final.norm")) @ W("embed").T


def _gla(h, W, p, c):
    T, H, D, E = len(h), c["heads"], c["dim"], c["vdim"]
    q, k, v = (h @ W(p + n).T for n in "qkv")
    q, k, v = q.reshape(T, H, D) * D ** -0.5, k.reshape(T, H, D), v.reshape(T, H, E)
    z = (h @ W(p + "a1").T) @ W(p + "a2").T + W(p + "a2.b")
    decay = (torch.nn.functional.logsigmoid(z) / c["tau"]).exp().reshape(T, H, D)

    def step(S, t):
        S.mul_(decay[t, :, :, None]).baddbmm_(k[t, :, :, None], v[t, :, None])
        return (q[t, :, None] @ S)[:, 0]
    o = _norm(_scan(T, h.new_zeros((H, D, E)), step), W(p + "norm"))
    return (o.reshape(T, H * E) * _silu(h @ W(p + "g").T)) @ W(p + "o").T


def _latent(h, W, p, c, half, kept):
    T, H, D, R = len(h), c["heads"], c["dim"], c["rot_dim"]
    lat, kr = kept
    q = _heads(_norm(h @ W(p + "dq").T, W(p + "dq.norm")) @ W(p + "uq").T, H)
    q = torch.cat([q[..., :D], _rotate(q[..., D:].contiguous(), 0, R, c["rot"]["base"], half)], -1)
    k = torch.cat([_heads(lat @ W(p + "uk").T, H), kr.expand(H, T, R)], -1)
    o = _attend(q, k, _heads(lat @ W(p + "uv").T, H), c["scale"], 0, c["mask"]["size"] if half else None)
    o = o.transpose(0, 1).reshape(T, -1)
    return (o * (h @ W(p + "g").T).sigmoid() if half else o) @ W(p + "o").T


def _daronex(cfg, W, ids, last):
    x, kept = W("embed")[ids], {}
    for i, L in enumerate(cfg["layers"]):
        p, c = f"l{i}.mix.", L["mixer"]
        if L["type"] == "gla":
            y = _gla(x, W, p, c)
        else:
            half, src = L["type"] == "latent_attention_2", c.get("kv_from")
            if src is None:
                src, t = i, x @ W(p + "dkv").T
                kept[i] = (_norm(t[:, :c["kv_rank"]], W(p + "dkv.norm")),
                           _rotate(t[:, c["kv_rank"]:].contiguous(), 0, c["rot_dim"], c["rot"]["base"], half))
            y = _latent(x, W, p, c, half, kept[src])
        x = x + _norm(y, 1 + W(f"l{i}.norm1"))
        if L.get("mlp"):
            y = (x @ W(f"l{i}.mlp.up").T).clamp(min=0).square() @ W(f"l{i}.mlp.down").T
            x = x + _norm(y, 1 + W(f"l{i}.norm2"))
    return _norm(x[last], 1 + W("final.norm")) @ W("head").T * cfg["logit_scale"]


def _exact_stack(c, seed):
    w = Weights(c, seed)
    ids = torch.tensor(_ids(seed, c["vocab"], c["prompt"] + c["steps"]), device="cuda")
    forward = {"zavilorn": _zavilorn, "daronex": _daronex}[c["model"]]
    return dict(logits=forward(_config(c), lambda n: w.device(n).double(), ids, -1).cpu().numpy())
