"""What a user of this framework has it do, as cases that can be timed and checked.

A case names its work and its sizes; `prepare` makes what a program holds before the call (weights on the device, a session,
host tokens), `run` makes one pass through the public entry points, `exact` states the same results in 64 bits from the
definition of the formats and of the models alone.

Weights look like a trained model's after quantization: bell-shaped codes, block scales that vary, a spread of about
1 / sqrt(columns), so that activations keep their size through the layers.  The output matrix is the embedding with its rows
in another order: a model then names the next token with the margin a trained one has, and greedy tokens do not hang on the
last bit of a logit."""
import math

import numpy as np
import torch

from llama_rust_b200 import DTYPES, DecoderSession, Executor, Session
from llama_rust_b200.executor import (GATE_ELEMENT, GATE_HEAD, MIXER_ATTENTION, MIXER_DELTA, MIXER_GATED_LINEAR, MIXER_LATENT, MIXER_RETENTION,
                                      NORM_INPUT, NORM_OUTPUT, UNIT_CLAMPED, UNIT_GELU)

FORMATS = ("Q4_K", "Q5_K", "Q6_K", "Q8_0", "Q4_0", "Q4_1", "Q5_0", "Q5_1", "F16", "BF16", "F32")
ROW_BYTES = {"Q4_K": (256, 144), "Q5_K": (256, 176), "Q6_K": (256, 210), "Q8_0": (32, 34), "Q4_0": (32, 18), "Q4_1": (32, 20), "Q5_0": (32, 22),
             "Q5_1": (32, 24), "F16": (1, 2), "BF16": (1, 2), "F32": (1, 4)}
LAYERED = ("attention", "latent", "mixed", "parallel", "delta", "gated", "recurrent")
BATCH_ROWS = 512  # most rows of one ragged batch of a Llama session


def listed():
    return [
        # the smallest call there is: one product of one host vector, as a program that keeps its own walk on the host makes it
        dict(name="call_q8_0", work="product", fmt="Q8_0", rows=4096, cols=4096, tokens=1, layers=1, host=True),
        # the rows of a few sequences that decode together, through the feed-forward of a few layers
        dict(name="rows_q4_k", work="product", fmt="Q4_K", rows=14336, cols=4096, tokens=6, layers=4, host=False),
        # a ragged prompt chunk of an attention projection in a five-bit format
        dict(name="chunk_q5_1_ragged", work="product", fmt="Q5_1", rows=4096, cols=4096, tokens=77, layers=6, host=False),
        # a prompt chunk through feed-forward matrices in the most common format
        dict(name="chunk_q4_k", work="product", fmt="Q4_K", rows=14336, cols=4096, tokens=256, layers=4, host=False),
        # all products of one decoded token, eight layers in one launch
        dict(name="token_program", work="program", fmt="Q4_K_M", width=4096, kv_width=1024, ff=14336, layers=8, tokens=1),
        # one routed feed-forward layer over the rows of a middle-sized batch, host rows in and out
        dict(name="experts", work="experts", fmt="Q4_K", width=4096, ff=14336, experts=8, used=2, tokens=64),
        # reading a prompt
        dict(name="llama_prompt", work="llama", does="prompt", fmt="Q4_K_M", width=4096, heads=32, kv_heads=8, dim=128, ff=14336, layers=4, vocab=32000,
             experts=0, prompt=512, gen=0, seqs=1),
        # answering it: the cached prompt is used again, then greedy tokens one by one
        dict(name="llama_answer", work="llama", does="answer", fmt="Q4_K_M", width=4096, heads=32, kv_heads=8, dim=128, ff=14336, layers=4, vocab=32000,
             experts=0, prompt=512, gen=24, seqs=1),
        # a server at work: the prompts of two dozen users in ragged batches, then their tokens step by step
        dict(name="llama_serve", work="llama", does="serve", fmt="Q4_K_M", width=4096, heads=32, kv_heads=8, dim=128, ff=14336, layers=4, vocab=32000,
             experts=0, prompt=40, gen=8, seqs=24),
        # a long prompt through windowed and latent attention
        dict(name="layered_prompt", work="layered", does="prompt", model="mixed", width=4096, heads=32, kv_heads=8, dim=128, ff=14336, rank=512, window=1024,
             layers=4, vocab=32000, prompt=2048, gen=0, seqs=1),
        # a prompt of an odd length through recurrent mixers
        dict(name="recurrent_prompt", work="layered", does="prompt", model="recurrent", width=2048, heads=16, kv_heads=8, dim=128, ff=8192, rank=512, window=1024,
             layers=4, vocab=32000, prompt=1001, gen=0, seqs=1),
        # the same on recurrent mixers
        dict(name="recurrent_serve", work="layered", does="serve", model="recurrent", width=2048, heads=16, kv_heads=8, dim=128, ff=8192, rank=512, window=1024,
             layers=4, vocab=32000, prompt=24, gen=8, seqs=32),
    ]


def draw(rng):
    def spread(lo, hi, step=1):  # even over the logarithm
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))

    def heads():
        dim = rng.choice((64, 128))
        n = rng.choice((8, 12, 16, 24, 32)) if dim == 128 else rng.choice((8, 12, 14, 16, 32))
        kv = rng.choice([g for g in (1, 2, 4, 8, 12, 16) if n % g == 0 and n // g <= 8])
        return n, kv, dim

    kind = rng.choice(("product",) * 6 + ("program", "experts") + ("llama",) * 5 + ("layered",) * 4)
    if kind == "product":
        while True:
            fmt = rng.choice(FORMATS)
            cols = spread(256, 14336, 256 if fmt.endswith("_K") or rng.random() < 0.7 else 32)
            c = dict(work="product", fmt=fmt, rows=spread(128, 14336), cols=cols, tokens=spread(1, 1024), layers=rng.randint(1, 4), host=rng.random() < 0.3)
            if c["rows"] * cols * c["tokens"] * c["layers"] < 6e10:
                return c
    if kind == "program":
        width = spread(1024, 4096, 1024)
        return dict(work="program", fmt=rng.choice(("Q4_K_M", "Q4_K", "Q8_0")), width=width, kv_width=width // rng.choice((1, 2, 4)), ff=spread(2048, 14336, 2048),
                    layers=rng.randint(2, 8), tokens=rng.randint(1, 8))
    if kind == "experts":
        experts = rng.choice((4, 8, 16))
        return dict(work="experts", fmt=rng.choice(("Q4_K", "Q5_K", "Q8_0")), width=spread(1024, 4096, 256), ff=spread(1024, 7168, 256), experts=experts,
                    used=rng.choice((1, 2, 4)), tokens=spread(1, 400))
    does = rng.choice(("prompt", "answer", "serve"))
    n, kv, dim = heads()
    c = dict(work=kind, does=does, width=n * dim if n * dim % 256 == 0 and rng.random() < 0.8 else spread(512, 4096, 256), heads=n, kv_heads=kv, dim=dim,
             layers=rng.randint(2, 4), vocab=spread(2000, 32000), prompt=spread(24, 1400) if does != "serve" else rng.randint(8, 60),
             gen=0 if does == "prompt" else rng.randint(2, 8) if does == "serve" else rng.randint(4, 24), seqs=rng.randint(2, 32) if does == "serve" else 1,
             ff=spread(1024, 12288, 256))
    if kind == "llama":
        experts = rng.choice((0, 0, 0, 4))
        return dict(c, fmt="Q4_K_M" if rng.random() < 0.4 else rng.choice(("Q4_K", "Q5_K", "Q8_0", "Q4_0", "Q5_1", "BF16", "F16")), experts=experts,
                    ff=min(c["ff"], 4096) if experts else c["ff"])
    return dict(c, model=rng.choice(LAYERED), rank=rng.choice((128, 256, 512)), window=rng.choice((96, 333, 1024)))


# ---- weights: the formats' fields, packed as a model file holds them, or as the numbers they stand for -----------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _normal(g, *shape):
    return torch.randn(shape, device="cuda", generator=g)


def _codes(g, n, per, top, spread):
    return (_normal(g, n, per) * spread + top / 2).round_().clamp_(0, top).to(torch.uint8)


def _scale(g, n, size):
    return ((torch.rand(n, device="cuda", generator=g) * 0.5 + 0.75) * size).to(torch.float16)


def _bytes(*parts):
    n = parts[0].shape[0]
    return torch.cat([p.contiguous().view(torch.uint8).reshape(n, -1) for p in parts], 1)


def _k_scales(sc, mn):
    lo = sc[:, :4] | (sc[:, 4:] >> 4 << 6)
    mid = mn[:, :4] | (mn[:, 4:] >> 4 << 6)
    return torch.cat([lo, mid, (sc[:, 4:] & 15) | ((mn[:, 4:] & 15) << 4)], 1)


def _bits(b):  # [n, 8 k] of 0 / 1 -> [n, k] bytes, lowest bit first
    return (b.view(b.shape[0], -1, 8) << torch.arange(8, device="cuda", dtype=torch.uint8)).sum(2, dtype=torch.uint8)


def _matrix(fmt, rows, cols, g, size=None, exact=False):
    """Seeded weights of spread `size`: packed bytes [rows, row bytes], or (exact) their float64 values [rows, cols]."""
    size = size or 1.0 / math.sqrt(cols)
    if fmt in ("F32", "F16", "BF16"):
        w = (_normal(g, rows, cols) * size).to({"F32": torch.float32, "F16": torch.float16, "BF16": torch.bfloat16}[fmt])
        return w.double() if exact else w.view(torch.uint8)
    per, _ = ROW_BYTES[fmt]
    n = rows * cols // per
    if fmt in ("Q4_K", "Q5_K"):
        top = 15 if fmt == "Q4_K" else 31
        q = _codes(g, n, 256, top, top * 0.18)
        sc = torch.randint(24, 64, (n, 8), device="cuda", generator=g, dtype=torch.uint8)
        mn = torch.randint(24, 64, (n, 8), device="cuda", generator=g, dtype=torch.uint8)
        d = _scale(g, n, size / (44 * top * 0.18))
        m = (d.float() * (top / 2)).to(torch.float16)
        mn = torch.where(torch.rand(n, 8, device="cuda", generator=g) < 0.9, sc, mn)
        if exact:
            w = d.double()[:, None, None] * sc.double()[:, :, None] * q.view(n, 8, 32) - (m.double()[:, None] * mn)[:, :, None]
            return w.view(rows, cols)
        s = q.view(n, 4, 2, 32)
        low = (s[:, :, 0] & 15) | ((s[:, :, 1] & 15) << 4)
        high = [_bits(((q >> 4).view(n, 8, 32)).transpose(1, 2).reshape(n, 256))] if fmt == "Q5_K" else []
        return _bytes(d, m, _k_scales(sc, mn), *high, low).view(rows, -1)
    if fmt == "Q6_K":
        q = _codes(g, n, 256, 63, 11.0)
        sc = torch.randint(24, 64, (n, 16), device="cuda", generator=g, dtype=torch.int8)
        sc = torch.where(torch.rand(n, 16, device="cuda", generator=g) < 0.5, -sc, sc)
        d = _scale(g, n, size / (44 * 11.0))
        if exact:
            return (d.double()[:, None, None] * sc.double()[:, :, None] * (q.view(n, 16, 16).double() - 32)).view(rows, cols)
        s = q.view(n, 2, 4, 32)  # halves of 128, four runs of 32 each
        low = torch.stack([(s[:, :, 0] & 15) | (s[:, :, 2] & 15) << 4, (s[:, :, 1] & 15) | (s[:, :, 3] & 15) << 4], 2)
        high = (s[:, :, 0] >> 4) | (s[:, :, 1] >> 4 << 2) | (s[:, :, 2] >> 4 << 4) | (s[:, :, 3] >> 4 << 6)
        return _bytes(low, high, sc, d).view(rows, -1)
    if fmt == "Q8_0":
        q = (_normal(g, n, 32) * 40).round_().clamp_(-127, 127).to(torch.int8)
        d = _scale(g, n, size / 40)
        return (d.double()[:, None] * q).view(rows, cols) if exact else _bytes(d, q).view(rows, -1)
    top = 15 if fmt.startswith("Q4") else 31
    q = _codes(g, n, 32, top, top * 0.18)
    d = _scale(g, n, size / (top * 0.18))
    m = (d.float() * (-top / 2) + _normal(g, n) * size * 0.1).to(torch.float16)
    if exact:
        return (d.double()[:, None] * q + m.double()[:, None] if fmt.endswith("_1") else d.double()[:, None] * (q.double() - (top + 1) // 2)).view(rows, cols)
    low = (q[:, :16] & 15) | (q[:, 16:] & 15) << 4
    return _bytes(d, *([m] if fmt.endswith("_1") else []), *([_bits(q >> 4)] if top == 31 else []), low).view(rows, -1)


_held = {}


def _executor():
    """The one executor of this thread, as a program keeps it."""
    if "executor" not in _held:
        _held["executor"] = Executor(0)
    return _held["executor"]


def _upload(fmt, rows, cols, packed):
    n = packed.numel()
    if "stage" not in _held or _held["stage"].numel() < n:
        _held["stage"] = torch.empty(n, dtype=torch.uint8).pin_memory()
    stage = _held["stage"][:n]
    stage.copy_(packed.reshape(-1))
    return _executor().upload(DTYPES[fmt], rows, cols, stage.numpy())


def _host(v):
    return None if v is None else v.float().cpu().numpy()


class _Maker:
    """Draws a model's tensors in a fixed order: resident matrices and host vectors, or float64 tensors (exact)."""

    def __init__(self, seed, exact):
        self.g, self.exact = _gen(seed), exact

    def matrix(self, fmt, rows, cols, size=None):
        w = _matrix(fmt, rows, cols, self.g, size, self.exact)
        return w if self.exact else _upload(fmt, rows, cols, w)

    def table(self, fmt, rows, cols):
        """The embedding and the output matrix: the same rows in another order."""
        w = _matrix(fmt, rows, cols, self.g, 1.0, self.exact)
        other = w[torch.randperm(rows, device="cuda", generator=self.g)]
        return (w, other) if self.exact else (_upload(fmt, rows, cols, w), _upload(fmt, rows, cols, other))

    def vector(self, *shape, mean=0.0, size=1.0):
        v = (_normal(self.g, *shape) * size + mean).float()
        return v.double() if self.exact else _host(v)


def _tokens(c, seed):
    rng = np.random.default_rng(seed + 77)
    if c["does"] != "serve":
        return [rng.integers(0, c["vocab"], c["prompt"]).astype(np.int32)]
    longest = min(2 * c["prompt"], BATCH_ROWS)  # ragged prompts around the size that the case names
    return [rng.integers(0, c["vocab"], int(n)).astype(np.int32) for n in rng.integers(2, longest, c["seqs"])]


# ---- products, programs, routed layers ----------------------------------------------------------------------------------------
def _mix(fmt):
    """Formats of q, k, v, o, gate, up, down and of the tables."""
    return ("Q4_K", "Q4_K", "Q6_K", "Q4_K", "Q4_K", "Q4_K", "Q6_K", "Q6_K") if fmt == "Q4_K_M" else (fmt,) * 8


def _sweep_shapes(c):
    E, K, F = c["width"], c["kv_width"], c["ff"]
    return ((E, E), (K, E), (K, E), (E, E), (F, E), (F, E), (E, F))


SWEEP_INPUT, SWEEP_PHASE = (-1, -1, -1, 0, 3, 3, 4), (0, 0, 0, 1, 2, 2, 3)  # which earlier result a product of the sweep reads


def _product(c, seed, exact):
    mk = _Maker(seed, exact)
    mats = [mk.matrix(c["fmt"], c["rows"], c["cols"]) for _ in range(c["layers"])]
    x = [_normal(mk.g, c["tokens"], c["cols"]) for _ in mats]
    return mats, x


def _program(c, seed, exact):
    mk = _Maker(seed, exact)
    mats = [[mk.matrix(f, *shape) for f, shape in zip(_mix(c["fmt"]), _sweep_shapes(c))] for _ in range(c["layers"])]
    return mats, _normal(mk.g, c["tokens"], c["width"])


def _experts(c, seed, exact):
    mk = _Maker(seed, exact)
    router = mk.matrix("F32", c["experts"], c["width"])
    parts = [[mk.matrix(c["fmt"], r, k) for _ in range(c["experts"])] for r, k in ((c["ff"], c["width"]), (c["ff"], c["width"]), (c["width"], c["ff"]))]
    return router, parts, _normal(mk.g, c["tokens"], c["width"])


# ---- the models -------------------------------------------------------------------------------------------------------------------
def _llama(c, seed, exact):
    mk, E, H, G, d, F = _Maker(seed, exact), c["width"], c["heads"], c["kv_heads"], c["dim"], c["ff"]
    names = ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
    shapes = ((H * d, E), (G * d, E), (G * d, E), (E, H * d), (F, E), (F, E), (E, F))
    fmts = _mix(c["fmt"])
    layers = []
    for _ in range(c["layers"]):
        L = dict(attn_norm=mk.vector(E, mean=1.0, size=0.2), ffn_norm=mk.vector(E, mean=1.0, size=0.2))
        for i, (n, s) in enumerate(zip(names, shapes)):
            if c["experts"] and n.startswith("ffn"):
                L[n + "_exps"] = [mk.matrix(fmts[i], *s) for _ in range(c["experts"])]
            else:
                L[n] = mk.matrix(fmts[i], *s)
        if c["experts"]:
            L.update(ffn_gate_inp=mk.matrix("F32", c["experts"], E), n_expert_used=2)
        layers.append(L)
    embd, out = mk.table(fmts[7], c["vocab"], E)
    return dict(embd=embd, out=out, norm=mk.vector(E, mean=1.0, size=0.2), layers=layers)


def _kinds(c):
    turn = dict(mixed=("latent", "attention", "attention", "shared"), recurrent=("delta", "parallel", "parallel", "gated")).get(c["model"], (c["model"],))
    return [turn[i % len(turn)] for i in range(c["layers"])]


def _eights(n):
    return -(-n // 8) * 8


def _layered(c, seed, exact):
    """Layers as the models of the registry describe them: windowed attention with a distance bias, latent attention, rotated
    attention beside a retention, the gated delta rule, the gated linear recurrence."""
    mk, W, H, G, d, R, F = _Maker(seed, exact), c["width"], c["heads"], c["kv_heads"], c["dim"], c["rank"], c["ff"]
    kinds = _kinds(c)
    inputs = c["model"] in ("parallel", "delta", "gated", "recurrent")  # norms on the sublayers' inputs
    freq = 5e5 ** (-2.0 * np.arange(d // 2) / d)
    bf = lambda rows, cols: mk.matrix("BF16", rows, cols)  # noqa: E731
    layers, source = [], -1
    for i, kind in enumerate(kinds):
        L = dict(mixer_norm=mk.vector(W, mean=1.0, size=0.2), mlp_norm=mk.vector(W, mean=1.0, size=0.2))
        L["mlp"] = dict(n_ff=F, gate_up=bf(2 * F, W), down=bf(W, F), **(dict(unit=UNIT_GELU) if inputs else dict(unit=UNIT_CLAMPED, limit=7.0, alpha=1.702, shift=1.0)))
        if kind == "attention":
            m = dict(kind=MIXER_ATTENTION, n_head=H, n_head_kv=G, dim=d, vdim=d, scale=d ** -0.5, window=c["window"], keep_first=4, gate=GATE_ELEMENT,
                     rel=mk.vector(32, H), bias_max=128, in_bias=mk.vector((H + 2 * G) * d, size=0.3), q_norm=mk.vector(H * d, mean=1.0, size=0.2),
                     k_norm=mk.vector(G * d, mean=1.0, size=0.2), out=bf(W, H * d))
            m["in"] = bf((2 * H + 2 * G) * d, W)
        elif kind in ("latent", "shared"):
            own = kind == "latent" or source < 0
            m = dict(kind=MIXER_LATENT, n_head=H, dim=d, vdim=d, kv_rank=R, scale=d ** -0.5, kv_from=-1 if own else source, window=c["window"], gate=GATE_HEAD,
                     up_k=bf(H * d, R), up_v=bf(H * d, R), kv_norm=mk.vector(R, mean=1.0, size=0.2) if own else None, out=bf(W, H * d))
            m["in"] = bf(H * d + (R if own else 0) + H, W)
            source = i if own else source
        elif kind == "parallel":
            m = dict(kind=MIXER_ATTENTION, n_head=H, n_head_kv=G, dim=d, vdim=d, scale=d ** -0.5, gate=GATE_HEAD, rot_freq=freq, sink=mk.vector(H, mean=3.0),
                     out=bf(W, (H + G) * d))
            m["in"] = bf(_eights((H + 2 * G) * d + H) + 4 * G * d, W)
            L.update(beside=dict(kind=MIXER_RETENTION, n_head=G, dim=d, vdim=d, scale=d ** -0.5, rot_freq=freq, decay=np.linspace(0.9, 0.9999, G)),
                     mixer_scale=0.7, beside_scale=1.3)
        elif kind == "gated":
            # the recurrence's width and blocks are the heads'
            N = H * d
            m = dict(kind=MIXER_GATED_LINEAR, width=N, blocks=H, taps=4, scale=8.0, in_bias=mk.vector(2 * N, size=0.3), conv=mk.vector(N, 4, size=0.5),
                     conv_bias=mk.vector(N, size=0.2), gates=bf(2 * N, d), gate_bias=mk.vector(2 * N, size=0.5), decay=mk.vector(N, mean=-4.0, size=1.5), out=bf(W, N))
            m["in"] = bf(2 * N, W)
        else:
            g, rank = max(1, H // 2), 128
            rows = (2 * g + H) * d
            m = dict(kind=MIXER_DELTA, n_head=H, n_head_kv=g, dim=d, vdim=d, scale=d ** -0.5, taps=4, unit_eps=1e-6, decay_rank=rank, gate_rank=rank,
                     decay_up=bf(H * d, rank), gate_up=bf(H * d, rank), conv=mk.vector(rows, 4, size=0.6), decay=mk.vector(H, mean=-1.0, size=0.5),
                     step_bias=mk.vector(H * d, mean=-3.0), head_norm=mk.vector(d, mean=1.0, size=0.2), out=bf(W, H * d))
            m["in"] = bf(_eights(rows + 2 * rank + H), W)
        layers.append(dict(L, mixer=m))
    embd, out = mk.table("BF16", c["vocab"], W)
    pos = None if inputs else mk.matrix("BF16", _positions(c), W, 0.3)
    return dict(embd=embd, out=out, norm=mk.vector(W, mean=1.0, size=0.2), pos=pos, layers=layers, inputs=inputs)


def _positions(c):
    return (2 * c["prompt"] if c["does"] == "serve" else c["prompt"]) + c["gen"] + 8


def _session(c, seed):
    if c["work"] == "llama":
        w = _llama(c, seed, False)
        cfg = dict(n_layer=c["layers"], n_embd=c["width"], n_head=c["heads"], n_head_kv=c["kv_heads"], head_dim=c["dim"], n_ff=c["ff"], n_vocab=c["vocab"],
                   n_ctx=_positions(c))
        return Session(_executor(), cfg, w["embd"], w["layers"], output=w["out"], output_norm=w["norm"], n_seq=c["seqs"])
    w = _layered(c, seed, False)
    cfg = dict(n_embd=c["width"], n_vocab=c["vocab"], n_ctx=_positions(c), norm_eps=1e-6, embd_scale=1.0, norm_place=NORM_INPUT if w["inputs"] else NORM_OUTPUT)
    return DecoderSession(_executor(), cfg, w["embd"], w["layers"], w["norm"], pos_embd=w["pos"], output=w["out"], n_seq=c["seqs"])


# ---- the interface -----------------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c, ex = case, _executor()
    if c["work"] == "product":
        mats, x = _product(c, seed, False)
        if c["host"]:
            return dict(c=c, mats=mats, x=[_host(v) for v in x], y=[np.empty((c["tokens"], c["rows"]), np.float32) for _ in mats])
        return dict(c=c, mats=mats, x=x, y=[torch.empty(c["tokens"], c["rows"], device="cuda") for _ in mats])
    if c["work"] == "program":
        mats, x = _program(c, seed, False)
        entries, ys, last = [], [], x
        for li, layer in enumerate(mats):
            y = [torch.empty(c["tokens"], m.rows, device="cuda") for m in layer]
            for m, src, phase, out in zip(layer, SWEEP_INPUT, SWEEP_PHASE, y):
                entries.append((m, (last if src < 0 else y[src]).data_ptr(), out.data_ptr(), c["tokens"], 4 * li + phase))
            ys += y
            last = y[-1]
        return dict(c=c, mats=mats, x=x, y=ys, program=ex.program(entries))
    if c["work"] == "experts":
        router, parts, x = _experts(c, seed, False)
        return dict(c=c, router=router, parts=parts, x=_host(x), out=np.empty((c["tokens"], c["width"]), np.float32))
    return dict(c=c, s=_session(c, seed), tokens=_tokens(c, seed))


def run(state):
    c = state["c"]
    if c["work"] == "product":
        ex = _executor()
        for m, x, y in zip(state["mats"], state["x"], state["y"]):
            if not c["host"]:
                ex.matmul_device(m, c["tokens"], x.data_ptr(), y.data_ptr())
            elif c["tokens"] == 1:
                ex.gemv_resident(m, x, y)
            else:
                ex.gemm_resident(m, c["tokens"], x, y)
        return state["y"]
    if c["work"] == "program":
        state["program"].run()
        return state["y"]
    if c["work"] == "experts":
        out, ids, weights = _executor().moe_ffn(state["router"], *state["parts"], min(c["used"], c["experts"]), True, state["x"], state["out"])
        return dict(out=out, ids=ids, weights=weights)
    s, tokens = state["s"], state["tokens"]
    if c["does"] == "prompt":
        s.reset()
        return dict(logits=s.prefill(tokens[0], want_logits=True))
    if c["does"] == "answer":
        first = s.prompt(tokens[0])
        ids, margin = s.decode(c["gen"])
        return dict(first=first, ids=ids, margin=margin, logits=s.logits())
    for q in range(c["seqs"]):
        s.seq_reset(q)
    got, left = [], list(enumerate(tokens))
    while left:  # as many whole prompts as a batch has room for
        batch, room = [], BATCH_ROWS
        while left and len(left[0][1]) <= room:
            room -= len(left[0][1])
            batch.append(left.pop(0))
        got.append(s.batch(batch)[0])
    ids, logits = [np.concatenate(got)], None
    for step in range(c["gen"]):
        nxt, logits = s.batch([(q, [int(t)]) for q, t in enumerate(ids[-1])], want_logits=step == c["gen"] - 1)
        ids.append(nxt)
    return dict(ids=np.stack(ids), logits=logits)


def _bytes_of(fmt, rows, cols):
    per, size = ROW_BYTES[fmt]
    return rows * cols // per * size


def work(case):
    c = case
    if c["work"] == "product":
        n = c["layers"]
        return dict(bytes=n * (_bytes_of(c["fmt"], c["rows"], c["cols"]) + 4 * c["tokens"] * (c["rows"] + c["cols"])), flops=2 * n * c["tokens"] * c["rows"] * c["cols"])
    if c["work"] == "program":
        shapes = _sweep_shapes(c)
        return dict(bytes=c["layers"] * sum(_bytes_of(f, *s) + 4 * c["tokens"] * sum(s) for f, s in zip(_mix(c["fmt"]), shapes)),
                    flops=2 * c["layers"] * c["tokens"] * sum(r * k for r, k in shapes))
    if c["work"] == "experts":
        used = min(c["used"], c["experts"])
        hit = min(c["experts"], c["tokens"] * used)  # experts that have rows
        each = 2 * _bytes_of(c["fmt"], c["ff"], c["width"]) + _bytes_of(c["fmt"], c["width"], c["ff"])
        return dict(bytes=hit * each + 8 * c["tokens"] * c["width"], flops=2 * c["tokens"] * used * 3 * c["width"] * c["ff"])
    # a model: its weights once per forward pass, its multiplications once per token, the cached rows once per pass
    E, H, G, d, F, V = (c[k] for k in ("width", "heads", "kv_heads", "dim", "ff", "vocab"))
    if c["work"] == "llama":
        fm, experts = _mix(c["fmt"]), c["experts"]
        attn = [(H * d, E), (G * d, E), (G * d, E), (E, H * d)]
        ffn = [(F, E), (F, E), (E, F)]
        dense = sum(_bytes_of(f, *s) for f, s in zip(fm, attn))
        one = sum(_bytes_of(f, *s) for f, s in zip(fm[4:], ffn))
        layer = lambda n: c["layers"] * (dense + one * (min(experts, 2 * n) if experts else 1))  # noqa: E731
        per_token = c["layers"] * (sum(r * k for r, k in attn) + (2 if experts else 1) * sum(r * k for r, k in ffn))
        head = _bytes_of(fm[7], V, E)
        seen, cache = (lambda n: c["layers"] * n), 2 * 4 * G * d
    else:
        R, win = c["rank"], c["window"]
        rows = dict(attention=(2 * H + 2 * G) * d + H * d, latent=H * d + R + H + H * d, shared=2 * H * d + H, parallel=(H + 2 * G) * d + H + 4 * G * d + (H + G) * d,
                    delta=(H + 2 * max(1, H // 2)) * d + 256 + H + H * d, gated=3 * H * d)
        inner = dict(attention=0, latent=2 * H * d * R, shared=2 * H * d * R, parallel=0, delta=2 * H * d * 128, gated=2 * H * d * d)
        kinds = _kinds(c)
        per_token = sum(rows[k] * E + inner[k] + 3 * F * E for k in kinds)
        layer, head = (lambda n: 2 * per_token), 2 * V * E
        spans = [min(win, 1 << 30) if k in ("attention", "latent", "shared") else 1 << 30 if k == "parallel" else d for k in kinds]
        seen, cache = (lambda n: sum(min(s, n) for s in spans)), 2 * 4 * G * d
    n, gen, S = c["prompt"], c["gen"], c["seqs"]
    look = 4 * H * d  # operations of one query row on one earlier position, all heads
    if c["does"] == "prompt":
        return dict(bytes=layer(n) + head + 4 * V, flops=2 * n * per_token + 2 * V * E + look * seen(n) * n / 2)
    if c["does"] == "answer":
        return dict(bytes=(gen + 1) * (layer(1) + head + cache * seen(n)), flops=(gen + 1) * (2 * per_token + 2 * V * E + look * seen(n)))
    rows = S * (n + gen)
    passes = -(-S * n // BATCH_ROWS)
    return dict(bytes=passes * layer(BATCH_ROWS) + gen * layer(S) + (passes + gen) * head + gen * S * cache * seen(n), flops=rows * 2 * per_token + (gen + 1) * S * 2 * V * E + rows * look * seen(n) / 2)


def tolerance(case):
    """About four times what the path is off its 64-bit statement: sums in 32 bits where few rows are multiplied; operands of 16
    bits in the matrix instructions from 64 rows on (binary16 for blocks, bfloat16 for BF16 weights) and in a prompt's attention,
    more so through several layers."""
    c = case
    if c["work"] == "program" or (c["work"] == "product" and (c["tokens"] < 64 or c["fmt"] in ("F16", "F32"))):
        return {"rel": 1e-5}
    if c["work"] == "product":
        return {"rel": 1e-2 if c["fmt"] == "BF16" else 4e-3}
    return {"rel": 6e-3 if c["work"] == "experts" else 1e-2 if c["work"] == "llama" and c["fmt"] != "BF16" else 2e-2}


# ---- 64-bit statements of the results -----------------------------------------------------------------------------------------------
def _rms(x, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _gelu(x):
    return 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))


def _softplus(x):
    return torch.logaddexp(x, torch.zeros_like(x))


def _seen(n, window=0, keep=0):
    i, j = torch.arange(n, device="cuda")[:, None], torch.arange(n, device="cuda")[None]
    return (j <= i) & ((i - j < window) | (j < keep)) if window else j <= i


def _attend(q, k, v, scale, seen, bias=None, sink=None):
    """q [n, H, d], k [n, G, d], v [n, G, dv] -> [n, H, dv]; query heads share key heads in runs, one head at a time."""
    out, rep = [], q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        s = q[:, h] @ k[:, h // rep].T * scale
        if bias is not None:
            s = s + bias[h]
        s = s.masked_fill(~seen, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(len(s), 1)], 1)
        p = torch.softmax(s, 1)[:, :len(k)]
        out.append(p @ v[:, h // rep])
    return torch.stack(out, 1)


def _route(x, router, used, norm):
    p = torch.softmax(x @ router.T, 1)
    w, ids = torch.sort(p, dim=1, descending=True, stable=True)
    w, ids = w[:, :used], ids[:, :used]
    return ids, w / w.sum(1, keepdim=True).clamp_min(2.0 ** -14) if norm else w


def _routed(x, router, gate, up, down, used, norm):
    ids, w = _route(x, router, used, norm)
    out = torch.zeros_like(x)
    for e in range(len(gate)):
        rows, slot = torch.where(ids == e)
        if len(rows):
            r = x[rows]
            out[rows] += (_silu(r @ gate[e].T) * (r @ up[e].T)) @ down[e].T * w[rows, slot][:, None]
    return out, ids, w


def _rotate_pairs(x, base=10000.0):
    n, _, d = x.shape
    a = torch.arange(n, device="cuda", dtype=torch.float64)[:, None] * base ** (-torch.arange(0, d, 2, device="cuda", dtype=torch.float64) / d)
    co, si = a.cos()[:, None], a.sin()[:, None]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * co - v * si, u * si + v * co], -1).flatten(-2)


def _rotate_halves(x, freq):
    a = torch.arange(len(x), device="cuda", dtype=torch.float64)[:, None] * torch.from_numpy(freq).cuda()
    co, si = a.cos()[:, None], a.sin()[:, None]
    u, v = x.chunk(2, -1)
    return torch.cat([u * co - v * si, v * co + u * si], -1)


def _llama_forward(c, w, tokens):
    H, G, d = c["heads"], c["kv_heads"], c["dim"]
    x = w["embd"][tokens]
    n = len(x)
    for L in w["layers"]:
        h = _rms(x, 1e-5) * L["attn_norm"]
        q, k = _rotate_pairs((h @ L["attn_q"].T).view(n, H, d)), _rotate_pairs((h @ L["attn_k"].T).view(n, G, d))
        x = x + _attend(q, k, (h @ L["attn_v"].T).view(n, G, d), d ** -0.5, _seen(n)).reshape(n, H * d) @ L["attn_output"].T
        h = _rms(x, 1e-5) * L["ffn_norm"]
        if c["experts"]:
            x = x + _routed(h, L["ffn_gate_inp"], L["ffn_gate_exps"], L["ffn_up_exps"], L["ffn_down_exps"], 2, True)[0]
        else:
            x = x + (_silu(h @ L["ffn_gate"].T) * (h @ L["ffn_up"].T)) @ L["ffn_down"].T
    return _rms(x[-1:], 1e-5) * w["norm"] @ w["out"].T


def _conv(x, taps):
    T = taps.shape[1]
    p = torch.cat([torch.zeros(T - 1, x.shape[1], dtype=x.dtype, device=x.device), x])
    return sum(p[j:j + len(x)] * taps[:, j] for j in range(T))


def _mixer(h, m, L, latents, i, W):
    n, z = len(h), h @ m["in"].T
    if m["kind"] == MIXER_GATED_LINEAR:
        N, B = m["width"], m["blocks"]
        z = z + m["in_bias"]
        u = _conv(z[:, N:], m["conv"]) + m["conv_bias"]
        gates = torch.einsum("boc,nbc->nbo", m["gates"].view(B, 2 * N // B, N // B), u.view(n, B, N // B)) + m["gate_bias"].view(B, 2 * N // B)
        r, inp = (torch.sigmoid(t).reshape(n, N) for t in gates.chunk(2, 2))
        log_a = -m["scale"] * r * _softplus(m["decay"])
        a, b, S, out = log_a.exp(), (-torch.expm1(2 * log_a)).sqrt() * inp * u, torch.zeros(N, dtype=h.dtype, device=h.device), []
        for t in range(n):
            S = a[t] * S + b[t]
            out.append(S)
        return (torch.stack(out) * _gelu(z[:, :N])) @ m["out"].T
    H, d, dv = m["n_head"], m["dim"], m["vdim"]
    if m["kind"] == MIXER_LATENT:
        R = m["kv_rank"]
        own = m["kv_from"] < 0
        q, g = z[:, :H * d].view(n, H, d), z[:, -H:]
        if own:
            latents[i] = _rms(z[:, H * d:H * d + R], 1e-6) * m["kv_norm"]
        lat = latents[i if own else m["kv_from"]]
        o = _attend(q, (lat @ m["up_k"].T).view(n, H, d), (lat @ m["up_v"].T).view(n, H, dv), m["scale"], _seen(n, m["window"]))
        return (o * torch.sigmoid(g)[:, :, None]).reshape(n, H * dv) @ m["out"].T
    G = m["n_head_kv"]
    if m["kind"] == MIXER_DELTA:
        qk, rows = G * d, 2 * G * d + H * dv
        y = _silu(_conv(z[:, :rows], m["conv"]))
        unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + m["unit_eps"])  # noqa: E731
        q, k = unit(y[:, :qk].view(n, G, d)) * m["scale"], unit(y[:, qk:2 * qk].view(n, G, d))
        q, k = (t.repeat_interleave(H // G, 1) for t in (q, k))
        v, rank = y[:, 2 * qk:].view(n, H, dv), m["decay_rank"]
        step = _softplus(z[:, rows:rows + rank] @ m["decay_up"].T + m["step_bias"]).view(n, H, d)
        g = torch.exp(-m["decay"].exp()[:, None] * step)
        gate = torch.sigmoid(z[:, rows + rank:rows + rank + m["gate_rank"]] @ m["gate_up"].T)
        beta = torch.sigmoid(z[:, rows + rank + m["gate_rank"]:][:, :H])
        S, out = torch.zeros(H, d, dv, dtype=h.dtype, device=h.device), []
        for t in range(n):
            S = g[t][:, :, None] * S
            S = S + k[t][:, :, None] * (beta[t][:, None] * (v[t] - (S * k[t][:, :, None]).sum(1)))[:, None]
            out.append((S * q[t][:, :, None]).sum(1))
        return ((_rms(torch.stack(out), 1e-6) * m["head_norm"]).reshape(n, H * dv) * gate) @ m["out"].T
    a, b = H * d, (H + G) * d
    q, k, v, g = z[:, :a], z[:, a:b], z[:, b:b + G * dv], z[:, b + G * dv:]
    if "in_bias" in m:  # normed queries and keys, a bias by distance, an element gate
        q, k, v = q + m["in_bias"][:a], k + m["in_bias"][a:b], v + m["in_bias"][b:]
        q, k = _rms(q, 1e-6) * m["q_norm"], _rms(k, 1e-6) * m["k_norm"]
        half, nb = len(m["rel"]) // 2, len(m["rel"])
        dist = np.arange(n)
        far = half + np.floor(np.log(np.maximum(dist, half) / half) / math.log(m["bias_max"] / half) * (nb - half) + 1e-9)
        bucket = torch.from_numpy(np.where(dist < half, dist, np.minimum(nb - 1, far)).astype(np.int64)).cuda()
        at = (torch.arange(n, device="cuda")[:, None] - torch.arange(n, device="cuda")[None]).clamp_min(0)
        bias = [m["rel"][bucket, hd][at] for hd in range(H)]
        o = _attend(q.view(n, H, d), k.view(n, G, d), v.reshape(n, G, dv), m["scale"], _seen(n, m["window"], m["keep_first"]), bias=bias)
        return (o.reshape(n, H * dv) * torch.sigmoid(g)) @ m["out"].T
    o = _attend(_rotate_halves(q.reshape(n, H, d), m["rot_freq"]), _rotate_halves(k.reshape(n, G, d), m["rot_freq"]), v.reshape(n, G, dv), m["scale"], _seen(n), sink=m["sink"])
    left = (o * torch.sigmoid(g[:, :H])[:, :, None]).reshape(n, H * dv) * L["mixer_scale"]
    r = L["beside"]
    N, at = r["n_head"], _eights(b + G * dv + H)
    q, k, v, g = z[:, at:at + 4 * N * d].chunk(4, 1)
    q, k = _rotate_halves(q.reshape(n, N, d), r["rot_freq"]), _rotate_halves(k.reshape(n, N, d), r["rot_freq"]) * r["scale"]
    v, S, out = v.reshape(n, N, d), torch.zeros(N, d, d, dtype=h.dtype, device=h.device), []
    decay = torch.from_numpy(r["decay"].astype(np.float32)).double().cuda()
    for t in range(n):
        S = decay[:, None, None] * S + k[t][:, :, None] * v[t][:, None]
        out.append((S * q[t][:, :, None]).sum(1))
    right = _rms(torch.stack(out), 1e-6).reshape(n, N * d) * _silu(g) * L["beside_scale"]
    return torch.cat([left, right], 1) @ m["out"].T


def _layered_forward(c, w, tokens):
    x, latents = w["embd"][tokens], {}
    if w["pos"] is not None:
        x = x + w["pos"][:len(x)]
    for i, L in enumerate(w["layers"]):
        f = L["mlp"]

        def mlp(h):
            g, u = (h @ f["gate_up"].T).chunk(2, 1)
            if w["inputs"]:
                return (_gelu(g) * u) @ f["down"].T
            g, u = g.clamp_max(7.0), u.clamp(-7.0, 7.0)
            return (g * torch.sigmoid(1.702 * g) * (u + 1.0)) @ f["down"].T
        for norm, sub in ((L["mixer_norm"], lambda h: _mixer(h, L["mixer"], L, latents, i, w)), (L["mlp_norm"], mlp)):
            x = x + (sub(_rms(x, 1e-6) * norm) if w["inputs"] else _rms(sub(x), 1e-6) * norm)
    return _rms(x[-1:], 1e-6) * w["norm"] @ w["out"].T


def exact(case, seed):
    c = case
    if c["work"] == "product":
        mats, x = _product(c, seed, True)
        return [v.double() @ m.T for m, v in zip(mats, x)]
    if c["work"] == "program":
        mats, x = _program(c, seed, True)
        ys, last = [], x.double()
        for layer in mats:
            y = []
            for m, src in zip(layer, SWEEP_INPUT):
                y.append((last if src < 0 else y[src]) @ m.T)
            ys += y
            last = y[-1]
        return ys
    if c["work"] == "experts":
        router, parts, x = _experts(c, seed, True)
        out, ids, w = _routed(x.double(), router, *parts, min(c["used"], c["experts"]), True)
        return dict(out=out, ids=ids.int(), weights=w)
    w = (_llama if c["work"] == "llama" else _layered)(c, seed, True)
    forward = _llama_forward if c["work"] == "llama" else _layered_forward
    seqs = [torch.from_numpy(t.astype(np.int64)).cuda() for t in _tokens(c, seed)]
    if c["does"] == "prompt":
        return dict(logits=forward(c, w, seqs[0])[0])
    rows, ids, margin = [], [], []
    for t in seqs:  # greedy, the whole sequence again for every token
        logits = [forward(c, w, t)[0]]
        mine = []
        for _ in range(c["gen"]):
            top = torch.topk(logits[-1], 2).values
            margin.append(top[0] - top[1])
            mine.append(logits[-1].argmax())
            t = torch.cat([t, mine[-1][None]])
            logits.append(forward(c, w, t)[0])
        rows.append(logits)
        ids.append(torch.stack(mine + [logits[-1].argmax()]).int())
    if c["does"] == "answer":
        return dict(first=rows[0][0], ids=ids[0][:-1], margin=torch.stack(margin), logits=rows[0][-1])
    return dict(ids=torch.stack(ids, 1), logits=torch.stack([r[-1] for r in rows]))
