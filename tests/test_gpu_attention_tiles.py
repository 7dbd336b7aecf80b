"""Prompt attention on the tensor cores at the edges of its tiles (128 pairs of row and query head, steps of 128 or 64 keys, chunks of
64 columns, parts of 256 value dimensions) against the plain float64 statement, with the tolerance of the path that serves."""
import numpy as np
import pytest

import nagolix_models as nm
import nagolix_plain as plain

pytestmark = pytest.mark.gpu

SHAPES = {
    "one head per key, a window of a step": nm.attention(3, 3, 64, 64, 128, 0, 30),
    "kept tokens fill more than a step": nm.attention(8, 2, 128, 128, 40, 140, 90),
    "kept tokens that meet the window": nm.attention(4, 1, 128, 72, 33, 200, 20),
    "heads that share no divisor with a tile": nm.attention(7, 1, 72, 40, 1000, 5, 300),
    "biases too long for shared memory": nm.attention(8, 1, 64, 64, 1000, 0, 600),
    "long keys, short values": nm.attention(2, 1, 136, 128, 150, 3, 40),
    "short keys, two parts of values": nm.attention(2, 1, 64, 264, 90, 2, 40),
    "long keys and values": nm.attention(2, 2, 256, 200, 129, 2, 40),
    "keys of nine chunks": nm.attention(2, 1, 520, 64, 127, 1, 40),
    "keys of thirteen chunks": nm.attention(2, 1, 776, 64, 127, 1, 40),
    "the longest keys of 16 bits": nm.attention(3, 1, 848, 32, 127, 1, 40),
    "long keys, values of three quarters of a part": nm.attention(2, 1, 800, 128, 127, 70, 40),
    "keys beyond the tile kernel": nm.attention(2, 1, 856, 32, 127, 1, 40),
    "latent of one chunk": nm.latent(5, 16, 24, 64, 65),
    "latent of two chunks": nm.latent(16, 16, 24, 128, 1000),
    "latent of an odd size": nm.latent(9, 16, 24, 200, 64),
    "latent of two parts": nm.latent(4, 16, 24, 320, 63),
    "latent of full width": nm.latent(32, 16, 24, 512, 200),
}


@pytest.mark.parametrize("name", list(SHAPES))
def test_tiles(tmp_path, name):
    from llama_rust_b200 import Executor, models
    cfg = nm.config(64, 90, [SHAPES[name]], 0)
    w = nm.weights(cfg, 17, 10, nm.SHARP[nm.AUTO])
    toks = nm.tokens(320, cfg, 23)
    want = plain.forward(cfg, w, toks)
    with Executor(0) as ex:
        s = models.load(ex, nm.write(tmp_path / "m", cfg, w), n_seq=3, block_tokens=7)
        for cut in ([320], [128, 129, 63], [16, 17, 255, 32]):
            s.seq_reset(1)
            at, got = 0, []
            for n in cut:
                got.append(s.forward([(1, toks[at:at + n])], [list(range(n))]))
                at += n
            assert nm.error(np.concatenate(got), want).max() <= nm.TOLERANCE[nm.AUTO], cut
        # groups of unequal sizes share the launches, a single row among them
        s.seq_reset(0), s.seq_reset(1), s.seq_reset(2)
        got = s.forward([(0, toks[:200]), (1, toks[:1]), (2, toks[:33])], [list(range(200)), [0], list(range(33))])
        assert nm.error(got, np.concatenate([want[:200], want[:1], want[:33]])).max() <= nm.TOLERANCE[nm.AUTO]
        s.free()


def _llama(ex, n_ctx, n_seq=1, heads=4, kv_heads=2, head_dim=64, vocab=300, edit=None, rms_eps=1e-5, **session):
    """A small Llama session with F32 weights: what differs between the paths is attention alone.  edit(weights) changes them by name."""
    import llama_walk as lw
    from helpers import ALL
    from llama_rust_b200 import Session
    cfg = dict(n_layer=2, n_embd=heads * head_dim, n_head=heads, n_head_kv=kv_heads, head_dim=head_dim, n_ff=256, n_vocab=vocab, rms_eps=rms_eps)
    rng = np.random.default_rng(72)
    w = {n: (rng.standard_normal((r, c)) / np.sqrt(c)).astype(np.float32) for n, _, r, c in lw.tensor_list(cfg)}
    w["embd"] = rng.standard_normal((vocab, cfg["n_embd"])).astype(np.float32)
    if edit:
        edit(w)
    up = {n: ex.upload(ALL["F32"], a.shape[0], a.shape[1], np.ascontiguousarray(a).view(np.uint8).ravel()) for n, a in w.items()}
    names = ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
    layers = [{n: up[f"blk.{i}.{n}.weight"] for n in names} for i in range(2)]
    return Session(ex, dict(cfg, n_ctx=n_ctx), up["embd"], layers, output=up["output.weight"], n_seq=n_seq, **session)


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_llama_rows_that_are_not_numbers(bad):
    """A token whose activations are not numbers makes its own row and every later one of its sequence not a number, and nothing else: not
    the rows before it, whose tiles hold its keys and values masked, nor the sequences that lie beside it in the gathered keys."""
    from llama_rust_b200 import Executor
    toks = [(7 * np.arange(n) + 3 * n) % 299 for n in (70, 150, 90)]  # never token 299
    toks[1][100] = 299

    def edit(w):
        w["embd"][299, 5] = bad
    with Executor(0) as ex:
        got = {}
        for path in (0, 3):
            ex.set_path(path)
            toks[1][100] = 299 if path == 0 else 298  # f32: another token's numbers there
            s = _llama(ex, 200, 3, edit=edit)
            got[path] = s.batch_rows([(q, t.tolist()) for q, t in enumerate(toks)], list(range(310)))
            s.free()
    finite = np.isfinite(got[0])
    clean = np.ones(310, bool)
    clean[70 + 100:70 + 150] = False
    assert finite[clean].all() and not finite[~clean].any()
    assert np.abs(got[0] - got[3])[clean].max() <= 1e-3 * np.abs(got[3]).max()


def test_llama_values_beyond_binary16_are_not_bounded():
    """Values of 1e6: the f32 path gives numbers, 16-bit operands infinities.  Anything else that is finite would be a wrong answer."""
    from llama_rust_b200 import Executor
    toks = (7 * np.arange(130)) % 299

    def edit(w):
        w["blk.0.attn_v.weight"] *= 1e6
    with Executor(0) as ex:
        s = _llama(ex, 200, edit=edit)
        ex.set_path(3)
        f32 = s.batch_rows([(0, toks.tolist())], [129])
        assert np.isfinite(f32).all()
        s.reset()
        ex.set_path(0)
        assert not np.isfinite(s.batch_rows([(0, toks.tolist())], [129])).any()
        s.free()


def test_layered_rows_that_are_not_numbers(tmp_path):
    """One layer with a window: the rows that see the broken token, no more and no less; the others have the numbers they have without it."""
    from llama_rust_b200 import Executor, models
    cfg = nm.config(64, 90, [nm.attention(4, 2, 72, 40, 40, 3, 24)], 0)
    w = nm.weights(cfg, 17, 10, nm.SHARP[nm.AUTO])
    toks = [t % 89 for t in nm.tokens(320, cfg, 23)]
    toks[200] = 89
    want = plain.forward(cfg, w, toks)
    w["embed"] = w["embed"].copy()
    w["embed"][89] = np.nan
    sees = (np.arange(320) >= 200) & (np.arange(320) < 240)
    with Executor(0) as ex:
        s = models.load(ex, nm.write(tmp_path / "m", cfg, w), n_seq=2)
        got = s.forward([(0, toks), (1, toks[:150])], [list(range(320)), list(range(150))])
        got, beside = got[:320], got[320:]
        # the embedding is the output matrix too: its broken row is one logit of every row
        got, beside, want = got[:, :89], beside[:, :89], want[:, :89]
        assert np.array_equal(~np.isfinite(got).any(1), sees), np.nonzero(~np.isfinite(got).any(1) != sees)[0]
        assert nm.error(got[~sees], want[~sees]).max() <= nm.TOLERANCE[nm.AUTO]
        assert nm.error(beside, want[:150]).max() <= nm.TOLERANCE[nm.AUTO]
        s.free()


# Heads beyond what 16-bit operands are for: more than 512 value dimensions, long keys beside long values.  Values of a million say which
# operands a prompt has: binary16 ends at 65504.
@pytest.mark.parametrize("dk,dv", [(64, 520), (64, 1024), (640, 512), (768, 192), (704, 264), (856, 32), (840, 64)])
def test_wide_heads_keep_32_bits(tmp_path, dk, dv):
    from llama_rust_b200 import Executor, models
    cfg = nm.config(64, 90, [nm.attention(2, 1, dk, dv, 90, 2, 40)], 0)
    w = nm.weights(cfg, 17, 10, nm.SHARP[nm.AUTO])
    w["l0.mix.v"], w["l0.mix.v.b"] = w["l0.mix.v"] * 2.0 ** 20, w["l0.mix.v.b"] * 2.0 ** 20
    toks = nm.tokens(140, cfg, 23)
    want = plain.forward(cfg, w, toks)
    with Executor(0) as ex:
        s = models.load(ex, nm.write(tmp_path / "m", cfg, w))
        assert nm.error(s.forward([(0, toks)], [list(range(140))]), want).max() <= nm.TOLERANCE[nm.AUTO]
        s.free()


# One key that outweighs all others together.  Where it appears after a reference has been taken, sums that lie in tensor memory are rescaled
# (steps of 128 keys: from key 256 on, each set of warps its own; of 64: from key 64 on), and rows on either side of a window's edge or of the
# kept tokens' end differ by all of it.
DOMINANT = {
    "two sets of warps": (nm.attention(2, 1, 64, 64, 1000, 0, 30), (0, 127, 255, 256, 257, 300, 400)),
    "a window of two steps": (nm.attention(6, 2, 128, 128, 256, 0, 30), (64, 130, 300)),
    "kept tokens beyond a step": (nm.attention(4, 2, 72, 128, 40, 140, 30), (127, 139, 140, 200)),
    "steps of 64 keys": (nm.attention(2, 1, 136, 264, 150, 70, 30), (63, 64, 69, 70, 130, 257)),
    "latent of 128": (nm.latent(8, 16, 24, 128, 300), (100, 130, 256, 390)),
    "latent of two parts": (nm.latent(4, 24, 24, 512, 200), (63, 64, 65, 130, 255)),
}


def _dominant(cfg, nats):
    """Weights of a one-layer model whose last token's key scores about `nats` above the others', which are spread by a third of a nat."""
    w = nm.weights(cfg, 17, 10, 0.3)
    L, W = cfg["layers"][0], cfg["width"]
    m, p, token = L["mixer"], "l0.mix.", cfg["vocab"] - 1
    H, d = m["heads"], m["dim"]
    w["embed"][:, :2] = 0  # input 0: this token; input 1: every row
    w["pos"][:, :2] = [0, 2]
    w["embed"][token, 0] = 4
    heads = np.arange(H) * d
    if L["type"] == "attention":
        G = m["kv_heads"]
        keys = np.arange(G) * d
        w[p + "rel"][:] = 0
        for t in ("q", "k", "v"):
            w[p + t][:, :2] = 0
        for t, at in (("q", heads), ("k", keys)):
            w[p + t][at], w[p + t + ".b"][at] = 0, 0
        w[p + "q.b"][heads] = 1
        w[p + "k"][keys, 0] = 1
        h = plain.embed(np.asarray([0, token]), w["embed"], w["pos"], cfg["embedding"]["scale"])
        q, k = (plain.rms(h @ w[p + t].T + w[p + t + ".b"], cfg["norm"]["eps"])[i] for t, i in (("q", 0), ("k", 1)))
        w[p + "q.norm"][heads] = 1
        w[p + "k.norm"][keys] = nm.plain.bf16_round(nats / (m["scale"] * q[0] * k[0]))
    else:
        for t in ("q", "dkv"):
            w[p + t][:, :2] = 0
        w[p + "q"] *= 0.5
        w[p + "q"][heads], w[p + "q"][heads, 1] = 0, 1
        w[p + "dkv"][0] = 0
        w[p + "dkv"][0, 0] = 1
        w[p + "dkv.norm"][0] = 1
        w[p + "uk"][:, 0] = 0
        w[p + "uk"][heads] = 0
        h = plain.embed(np.asarray([0, token]), w["embed"], w["pos"], cfg["embedding"]["scale"])
        c = plain.latent_of(h, w, p, cfg["norm"]["eps"])[1, 0]
        w[p + "uk"][heads, 0] = nm.plain.bf16_round(nats / (m["scale"] * (h @ w[p + "q"].T)[0, 0] * c))
    return w


@pytest.mark.parametrize("name", list(DOMINANT))
def test_one_dominant_key(tmp_path, name):
    from llama_rust_b200 import Executor, models
    layer, places = DOMINANT[name]
    cfg = nm.config(64, 90, [layer], 0)
    w = _dominant(cfg, 9.0)
    with Executor(0) as ex:
        s = models.load(ex, nm.write(tmp_path / "m", cfg, w))
        for at in places:
            toks = [t % 89 for t in nm.tokens(440, cfg, 23 + at)]
            toks[at] = 89
            want = plain.forward(cfg, w, toks)
            for cut in ([440], [130, 310], [16, 41, 383]):
                s.reset()
                done, got = 0, []
                for n in cut:
                    got.append(s.forward([(0, toks[done:done + n])], [list(range(n))]))
                    done += n
                assert nm.error(np.concatenate(got), want).max() <= nm.TOLERANCE[nm.AUTO], (at, cut)
        s.free()


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(4, 2, 64), (4, 1, 128)])
def test_one_dominant_key_of_a_llama_prompt(heads, kv_heads, head_dim):
    """The same through the Llama walk: the last pair of dimensions, which turns by a twentieth of a radian over the prompt, carries the key."""
    from llama_rust_b200 import Executor
    E, places, n = heads * head_dim, (127, 255, 256, 300, 400), 460

    def edit(w):
        embd, wq, wk = w["embd"], w["blk.0.attn_q.weight"], w["blk.0.attn_k.weight"]
        embd[:, :2] = [0, 1]
        embd[299, 0] = 4
        wq *= 0.2
        for m in (wq, wk):
            m[:, :2] = 0
            m[head_dim - 2::head_dim] = 0
            m[head_dim - 1::head_dim] = 0
        rows = embd / np.sqrt((embd ** 2).mean(1, keepdims=True))
        wq[head_dim - 2::head_dim, 1] = 1
        wk[head_dim - 2::head_dim, 0] = 9.0 * np.sqrt(head_dim) / (rows[0, 1] * rows[299, 0])
    with Executor(0) as ex:
        s = _llama(ex, 512, 2, heads, kv_heads, head_dim, edit=edit)
        for at in places:
            toks = (7 * np.arange(n) + at) % 299
            toks[at] = 299
            got = {}
            for path in (3, 0):
                ex.set_path(path)
                s.reset()
                got[path] = s.batch_rows([(1, toks.tolist())], list(range(n)))
            assert np.abs(got[0] - got[3]).max() <= 2e-3 * np.abs(got[3]).max(), at
        s.free()


@pytest.mark.parametrize("head_dim", [64, 128])
def test_weights_of_a_llama_prompt_are_not_rounded_to_binary16(head_dim):
    """Values of +-64 and scores within a few sixteenths of a nat: what 16-bit queries and keys cost is an eleventh-bit rounding of those
    (2^-11 / 16, twice), while weights rounded to eleven bits would be off by 2^-11 / sqrt(12) = 1.4e-4, and the results with them."""
    from llama_rust_b200 import Executor
    E, n = 2 * head_dim, 400

    def edit(w):
        w["embd"][:] = np.where(w["embd"] > 0, 1, -1)  # root mean square 1: the norm leaves them
        rng = np.random.default_rng(5)
        for t, size in (("q", 1 / 16), ("k", 1), ("v", 64)):
            m = w[f"blk.0.attn_{t}.weight"]
            m[:] = 0
            m[np.arange(len(m)), rng.permutation(E)[np.arange(len(m)) % E]] = size
        for name in ("blk.0.ffn_down.weight", "blk.1.attn_output.weight", "blk.1.ffn_down.weight"):
            w[name][:] = 0
    toks = np.random.default_rng(6).integers(0, 300, n).tolist()
    with Executor(0) as ex:
        s = _llama(ex, 512, 1, 2, 1, head_dim, edit=edit, rms_eps=0.0)
        got = {}
        for path in (3, 0):
            ex.set_path(path)
            s.reset()
            got[path] = s.batch_rows([(0, toks)], list(range(100, n))).astype(np.float64)
        assert np.linalg.norm(got[0] - got[3]) <= 4e-5 * np.linalg.norm(got[3])
        s.free()
