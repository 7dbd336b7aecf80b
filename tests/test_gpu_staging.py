"""Workspaces of staged activations: digit records up to 63 rows, 16-bit rows from 64 on.  Products of the same rows that follow each
other in a session (q, k, v and gate, up) share them; a wrong reuse multiplies other rows than the layer's."""
import numpy as np
import pytest

import llama_walk as lw
from helpers import F32, Q4_0, Q4_K, Q6_K, Q8_0

pytestmark = pytest.mark.gpu

NAMES = ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
VOCAB, WIDTH, FF = 512, 2048, 512


def _packed(kind, rows, cols, seed):
    from llama_rust_b200 import synth
    w = synth.packed_matrix(kind, rows, cols, seed)
    return lw.center_q4k(w) if kind == Q4_K else w


def _soft(packed):
    """Q8_0 under scales 2^-6 of the recipe's: query and key values of about 0.4, scores of about 2 (at the recipe's, thousands: the
    softmax then hangs on the last bits of a score)."""
    blocks = packed.reshape(-1, 34).copy()
    blocks[:, :2] = (blocks[:, :2].copy().view(np.float16) * np.float16(2.0 ** -6)).view(np.uint8)
    return blocks.reshape(-1)


def _out_of_half_range(packed):
    """A Q8_0 matrix whose first block is all zeros under a scale that binary16 operands cannot carry: bfloat16 is taken for it."""
    packed = packed.copy()
    packed[:34] = 0
    packed[:2] = np.array([60000.0], np.float16).view(np.uint8)
    return packed


def _session(ex, kinds, heads, kv_heads, n_seq, n_ctx, wide=()):
    from llama_rust_b200 import Session
    shapes = ((heads * 128, WIDTH), (kv_heads * 128, WIDTH), (kv_heads * 128, WIDTH), (WIDTH, heads * 128), (FF, WIDTH), (FF, WIDTH), (WIDTH, FF))
    layer = {}
    for i, (name, kind, (rows, cols)) in enumerate(zip(NAMES, kinds, shapes)):
        w = _packed(kind, rows, cols, 40 + i)
        if kind == Q8_0 and name in ("attn_q", "attn_k"):
            w = _soft(w)
        layer[name] = ex.upload(kind, rows, cols, _out_of_half_range(w) if name in wide else w)
    embd = ex.upload(F32, VOCAB, WIDTH, np.random.default_rng(3).standard_normal(VOCAB * WIDTH).astype(np.float32).view(np.uint8))
    out = ex.synth(Q6_K, VOCAB, WIDTH, 50)
    cfg = dict(n_layer=1, n_embd=WIDTH, n_head=heads, n_head_kv=kv_heads, head_dim=128, n_ff=FF, n_vocab=VOCAB, n_ctx=n_ctx)
    return Session(ex, cfg, embd, [layer], output=out, n_seq=n_seq)


def _residual(s, seq, ids):
    s.batch([(seq, ids)])
    return s.residual(len(ids))


def _same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


# (80, 10): q has so many rows that its product needs no room for unit sums, k needs more than q left: the buffer grows between them
@pytest.mark.parametrize("heads,kv_heads", [(16, 2), (80, 10)])
def test_digit_records_shared_by_products_of_the_same_rows(heads, kv_heads):
    """13 to 63 rows as one batch, on an executor whose workspace is still small, against the same rows eight at a time (the decode
    kernel, which stages nothing): the same bits, across Q4_K and Q6_K."""
    from llama_rust_b200 import Executor
    kinds = (Q4_K, Q4_K, Q6_K, Q4_K, Q4_K, Q6_K, Q4_K)
    with Executor(0) as ex:
        counts = (24, 13, 48, 25, 63)
        s = _session(ex, kinds, heads, kv_heads, len(counts), 64)
        for q, n in enumerate(counts):
            ids = lw.prompt_ids(n, VOCAB, 60 + n)
            got = _residual(s, q, ids)
            s.seq_reset(q)
            want = np.concatenate([_residual(s, q, ids[i:i + 8]) for i in range(0, n, 8)])
            assert _same_bits(got, want), n
        s.free()


def test_short_memory_between_products_of_the_same_rows(monkeypatch):
    """13 rows leave a workspace that the products of 24 rows outgrow.  Where it may not grow, the tall q falls back to the decode
    kernel, k and v fit what is there: they must not take the earlier rows' records in it for their own."""
    from llama_rust_b200 import Executor
    kinds = (Q4_K, Q4_K, Q6_K, Q4_K, Q4_K, Q4_K, Q4_K)
    got = {}
    for limit in ("", "1500000"):  # bytes; q at 24 rows: 1.78 million, at 13 rows 0.99, k at 24 rows 0.40
        if limit:
            monkeypatch.setenv("LLR_DIGITS_LIMIT", limit)
        with Executor(0) as ex:
            s = _session(ex, kinds, 16, 2, 2, 64)
            got[limit] = [_residual(s, 0, lw.prompt_ids(13, VOCAB, 7)), _residual(s, 1, lw.prompt_ids(24, VOCAB, 8))]
            s.free()
    for a, b in zip(got[""], got["1500000"]):
        assert _same_bits(a, b)


@pytest.mark.parametrize("n", [64, 77, 256])
def test_16_bit_rows_shared_by_products_of_the_same_rows(n):
    """64 rows and more: binary16 rows shared by all, and not shared where a matrix in between wants bfloat16 ones (k and up).
    Against f32 products: operands of eight bits are off by 2^-9 each, so a score of about 2 by 2^-7 at most and its softmax weight by as
    much; the sums over random signs that follow shrink that, and 2^-6 of a row's norm holds.  Rows of another format or another
    batch would miss it by the norm itself.  Where k and up convert for themselves the layer has three launches
    more (k, v and up)."""
    from llama_rust_b200 import Executor
    kinds = (Q8_0, Q8_0, Q4_0, Q8_0, Q8_0, Q8_0, Q8_0)
    launches = {}
    for wide in ((), ("attn_k", "ffn_up")):
        with Executor(0) as ex:
            s = _session(ex, kinds, 16, 2, 2, 256, wide)
            got = {}
            for path in (0, 3):
                ex.set_path(path)
                s.reset()
                s.batch([(1, lw.prompt_ids(n, VOCAB, 90))])  # other rows staged before
                before = ex.counters()["launches"]
                got[path] = _residual(s, 0, lw.prompt_ids(n, VOCAB, 91))
                if path == 0:
                    launches[wide] = ex.counters()["launches"] - before
            err = np.linalg.norm(got[0].astype(np.float64) - got[3], axis=1) / np.linalg.norm(got[3].astype(np.float64), axis=1)
            assert err.max() <= 2.0 ** -6, (wide, err.max())
            s.free()
    assert launches[("attn_k", "ffn_up")] - launches[()] == 3


def test_routed_layers_ask_for_the_workspaces_they_use(monkeypatch):
    """Experts of 13 to 63 rows each.  In one grouped launch (the automatic choice) they use no workspace of digits, and none is
    allocated: the device's free memory does not hang on LLR_DIGITS_LIMIT (8 MB for the gate matrices, were it grown).  On the
    f32-faithful path they use it, and the layer's bits are those without."""
    import torch
    from llama_rust_b200 import Executor
    width, ff, n = 2048, 8192, 40
    x = np.random.default_rng(5).standard_normal((n, width)).astype(np.float32)
    taken, out = {}, {}
    for turn, limit in enumerate(("0", "0", "1000000000")):  # the first loads the kernels
        monkeypatch.setenv("LLR_DIGITS_LIMIT", limit)
        with Executor(0) as ex:
            router = ex.synth(F32, 4, width, 70)
            parts = [[ex.synth(Q4_K, r, c, 71 + 4 * k + i) for i in range(4)] for k, (r, c) in enumerate(((ff, width), (ff, width), (width, ff)))]
            before = torch.cuda.mem_get_info()[0]
            _, ids, _ = ex.moe_ffn(router, *parts, 2, True, x)
            taken[turn] = before - torch.cuda.mem_get_info()[0]
            assert all(13 <= c <= 63 for c in np.bincount(ids.ravel(), minlength=4))
            ex.set_path(3)
            out[turn] = ex.moe_ffn(router, *parts, 2, True, x)[0]
    assert abs(taken[2] - taken[1]) < 4 << 20, taken
    assert _same_bits(out[1], out[2])
