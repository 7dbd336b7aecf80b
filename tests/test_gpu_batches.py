"""Batches of many rows and of many sequences: products of a few dozen activation rows, ragged batches whose groups share the
attention launches."""
import numpy as np
import pytest

import nagolix_models as nm
import nagolix_plain as plain
from helpers import ALL

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ex():
    from llama_rust_b200 import Executor
    with Executor(0) as e:
        yield e


def _product(ex, m, x):
    y = np.empty((len(x), m.rows), np.float32)
    ex.gemm_resident(m, len(x), x, y)
    return y


def _same_bits(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("rows,cols", [(1, 8), (31, 264), (65, 1032), (9500, 512)])  # ends of tiles, of column steps; four and two weight rows per warp
@pytest.mark.parametrize("name", ["F32", "F16", "BF16"])
def test_rows_of_unpacked_formats_alone_and_in_a_batch(ex, name, rows, cols):
    """Up to 32 activation rows a row's bits do not depend on the batch; above, every sum stays within the bound of a sum of
    `cols` products formed in any order."""
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL[name], rows, cols, 5)
    x = synth.activations(40 * cols, 6).reshape(40, cols)
    alone = np.concatenate([_product(ex, m, x[t:t + 1]) for t in range(32)])
    for n in (3, 4, 5, 8, 9, 16, 17, 32):
        assert _same_bits(_product(ex, m, x[:n]), alone[:n]), n
    w = ex.dequant_rows(m).astype(np.float64)
    exact, size = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    for n in (33, 40):
        assert np.all(np.abs(_product(ex, m, x[:n]) - exact[:n]) <= 2.0 ** -24 * (cols + 3) * size[:n]), n
    m.free()


@pytest.mark.parametrize("rows,cols", [(5, 128), (200, 256), (9500, 200), (31, 520), (130, 2056), (9500, 264)])
@pytest.mark.parametrize("name", ["F32", "F16"])
def test_more_than_32_rows_of_unpacked_formats(ex, name, rows, cols):
    """Passes of sixteen and of eight rows with remainders of both kinds.  Up to 256 columns a sum is one run and has the bits of the row
    alone; beyond, it stays within the bound of a sum of `cols` products formed in any order."""
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL[name], rows, cols, 17)
    x = synth.activations(58 * cols, 18).reshape(58, cols)
    w = ex.dequant_rows(m).astype(np.float64)
    exact, size = x.astype(np.float64) @ w.T, np.abs(x).astype(np.float64) @ np.abs(w).T
    alone = np.concatenate([_product(ex, m, x[t:t + 1]) for t in range(58)]) if cols <= 256 else None
    for n in (33, 41, 48, 58):
        y = _product(ex, m, x[:n])
        assert np.all(np.abs(y - exact[:n]) <= 2.0 ** -24 * (cols + 3) * size[:n]), n
        assert alone is None or _same_bits(y, alone[:n]), n
    m.free()


@pytest.mark.parametrize("cols", [264, 2304, 4096, 6144, 6152, 14336])
@pytest.mark.parametrize("name", ["F32", "BF16"])
def test_rounding_of_more_than_32_rows(ex, name, cols):
    """40 rows, values of one size and of very different sizes: the error against 64-bit sums is no larger than that of the staged
    kernel (path 2), which took such batches before; two hundredths for the chance of 20000 roundings that fall otherwise."""
    import torch
    from llama_rust_b200 import synth
    m = ex.synth(ALL[name], 500, cols, 19)
    w = torch.from_numpy(ex.dequant_rows(m)).cuda().double()
    x = synth.activations(40 * cols, 20).reshape(40, cols)
    for rows in (x, x * np.exp(3 * synth.activations(40 * cols, 21).reshape(40, cols)).astype(np.float32)):
        exact = torch.from_numpy(rows).cuda().double() @ w.T
        err = {}
        for path in (0, 2):
            ex.set_path(path)
            err[path] = float((torch.from_numpy(_product(ex, m, rows)).cuda().double() - exact).norm())
        assert err[0] <= 1.02 * err[2], err
    ex.set_path(0)
    m.free()


@pytest.mark.parametrize("rows,cols", [(1, 1024), (17, 1032), (33, 2048), (7, 2304), (40, 5000), (2368, 1096), (2369, 1096)])
@pytest.mark.parametrize("name", ["F32", "F16", "BF16"])
def test_few_weight_rows_in_tiles_of_many_columns(ex, name, rows, cols):
    """Three and four activation rows against up to a block per SM of weight rows (2368 of them on 148 SMs): whole tiles of 1024 columns,
    tiles that end in the middle of a step, one tile alone.  The bits of each row alone."""
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL[name], rows, cols, 15)
    x = synth.activations(4 * cols, 16).reshape(4, cols)
    alone = np.concatenate([_product(ex, m, x[t:t + 1]) for t in range(4)])
    for n in (3, 4):
        assert _same_bits(_product(ex, m, x[:n]), alone[:n]), n
    m.free()


# tiles of 256 activation rows: whole ones and not, with rows that are and are not stored as vectors
@pytest.mark.parametrize("rows,cols,tokens", [(16400, 264, 257), (16390, 128, 300), (16384, 192, 489), (16384, 64, 512)])
def test_wide_tiles_of_bf16_products(ex, rows, cols, tokens):
    """Products of bfloat16 values are exact in f32; every sum of `cols` of them, in whatever order, stays within cols ulps of the
    sum of their sizes (the tensor cores cut where f32 rounds, twice its unit)."""
    import torch
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL["BF16"], rows, cols, 5)
    x = synth.activations(tokens * cols, 6).reshape(tokens, cols)
    w = torch.from_numpy(ex.dequant_rows(m)).cuda().double()
    xb = torch.from_numpy(x).cuda().bfloat16().double()
    err = (torch.from_numpy(_product(ex, m, x)).cuda().double() - xb @ w.T).abs()
    assert bool((err <= 2.0 ** -23 * (cols + 3) * (xb.abs() @ w.abs().T)).all())
    m.free()


@pytest.mark.parametrize("rows", [10240, 12288, 14336, 16384])  # tiles of 160, 176, 208 and 224 weight rows: rings of eight, eight, six and six
def test_paired_tiles_give_the_same_bits_each_time(ex, rows):
    """Two tiles of activation rows, the second almost empty (257 rows: three of them; its copies arrive first), 64 column steps."""
    import torch
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL["BF16"], rows, 4096, 5)
    x = torch.from_numpy(synth.activations(300 * 4096, 6)).cuda()
    for tokens in (257, 300):
        want = torch.empty(tokens, rows, device="cuda")
        got = torch.empty_like(want)
        ex.matmul_device(m, tokens, x.data_ptr(), want.data_ptr())
        ex.synchronize()
        for _ in range(20):
            got.fill_(float("nan"))
            torch.cuda.synchronize()
            ex.matmul_device(m, tokens, x.data_ptr(), got.data_ptr())
            ex.synchronize()
            assert torch.equal(got, want), tokens
    m.free()


def test_wide_tiles_of_gated_units(ex, tmp_path):
    """A feed-forward layer whose gate | up product takes tiles of 256 activation rows, against the plain model."""
    from llama_rust_b200 import models
    cfg = nm.config(80, 120, [nm.attention(2, 1, 24, 24, 9, 2, 20)], 8200, limit=0.8)
    w = nm.weights(cfg, 23, 8, nm.SHARP[nm.AUTO])
    ex.set_path(nm.AUTO)
    s = models.load(ex, nm.write(tmp_path / "m", cfg, w), n_seq=1, n_ctx=300)
    t = nm.tokens(300, cfg, 24)
    got = s.forward([(0, t)], [list(range(300))])
    assert nm.error(got, plain.forward(cfg, w, t)).max() <= nm.TOLERANCE[nm.AUTO]
    s.free()


# one block; the last rows of a tile; parts of 4096 columns that end in single blocks, in pairs and singles; units spread over CTAs; many tiles
@pytest.mark.parametrize("name,rows,cols", [("Q4_K", 1, 256), ("Q4_K", 127, 2304), ("Q4_K", 130, 4096 + 256), ("Q4_K", 257, 2 * 4096 + 9 * 256),
                                            ("Q4_K", 9600, 768), ("Q5_K", 64, 256), ("Q5_K", 129, 6400), ("Q5_K", 5000, 1024),
                                            ("Q6_K", 3, 2048), ("Q6_K", 129, 4096), ("Q6_K", 260, 3 * 2048), ("Q6_K", 6000, 2048)])
def test_rows_of_k_quants_alone_and_in_a_batch(ex, name, rows, cols):
    """A row's bits do not depend on its batch: eight rows go through the decode kernel, more through the integer GEMM (whose sums are
    the same integers).  Rows of zeros, of tiny and of huge values, of one sign, and one with an infinity among them."""
    from llama_rust_b200 import synth
    m = ex.synth(ALL[name], rows, cols, 7)
    x = synth.activations(100 * cols, 8).reshape(100, cols).copy()
    x[1] = 0
    x[2] *= 1e-30
    x[3] *= 1e30
    x[4] = 1
    x[5, ::3] *= 1e4
    x[6] = np.abs(x[6])
    x[23, cols // 2] = np.inf
    ex.set_path(3)
    alone = np.concatenate([_product(ex, m, x[t:t + 8]) for t in range(0, 100, 8)])
    finite = np.arange(100) != 23
    assert np.isnan(alone[23]).all() and np.isfinite(alone[finite]).all()
    for path, counts in ((0, (5, 6, 12, 13, 16, 17, 24, 25, 32, 33, 48, 49, 63)), (3, (64, 100))):
        ex.set_path(path)
        for n in counts:
            y = _product(ex, m, x[:n])
            assert _same_bits(y[finite[:n]], alone[:n][finite[:n]]) and np.isnan(y[23:24]).all(), n
    ex.set_path(0)
    m.free()


def test_products_on_other_streams_keep_their_bits(ex):
    """The integer GEMM's workspace belongs to the executor's stream: on streams of the caller's, also while one is captured, the
    decode kernel makes the same products."""
    import torch
    from llama_rust_b200 import synth
    ex.set_path(0)
    m = ex.synth(ALL["Q4_K"], 640, 1024, 9)
    x = torch.from_numpy(synth.activations(20 * 1024, 10)).cuda()
    want = torch.empty(20 * 640, device="cuda")
    ex.matmul_device(m, 20, x.data_ptr(), want.data_ptr())
    ex.synchronize()
    side = torch.cuda.Stream()
    got = torch.empty_like(want)
    ex.matmul_device(m, 20, x.data_ptr(), got.data_ptr(), side.cuda_stream)
    side.synchronize()
    assert torch.equal(got, want)
    graph = torch.cuda.CUDAGraph()
    got.zero_()
    with torch.cuda.graph(graph, stream=side):
        ex.matmul_device(m, 20, x.data_ptr(), got.data_ptr(), torch.cuda.current_stream().cuda_stream)
    big = ex.synth(ALL["Q4_K"], 256, 4096, 9)
    _product(ex, big, np.ones((63, 4096), np.float32))  # a larger workspace between capture and replay
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    del graph
    m.free()
    big.free()


@pytest.mark.parametrize("lens", [[1 + i * 7 % 13 for i in range(70)],      # more runs of short groups than one list holds
                                  [15, 16, 17, 1, 64, 2, 16, 40, 31, 1, 3, 100]])
def test_many_groups_in_one_batch(ex, tmp_path, lens):
    """f32: the bits of every sequence alone; the serving path: the plain logits."""
    from llama_rust_b200 import models
    cfg, buckets = nm.MODELS["mix"]
    for path in (nm.F32, nm.AUTO):
        w = nm.weights(cfg, 21, buckets, nm.SHARP[path])
        ex.set_path(path)
        s = models.load(ex, nm.write(tmp_path / f"m{path}", cfg, w), n_seq=len(lens), n_ctx=160)
        toks = [nm.tokens(n, cfg, 100 + i) for i, n in enumerate(lens)]
        together = s.forward(list(enumerate(toks)), [list(range(n)) for n in lens])
        s.reset()
        at = 0
        for i, t in enumerate(toks):
            mine = together[at:at + len(t)]
            at += len(t)
            if path == nm.F32 and i % 5 == 0:
                assert _same_bits(mine, s.forward([(0, t)], [list(range(len(t)))])), i
                s.reset()
            elif path == nm.AUTO:
                assert nm.error(mine, plain.forward(cfg, w, t)).max() <= nm.TOLERANCE[path], i
        s.free()
    ex.set_path(0)


def test_groups_whose_keys_do_not_fit_one_launch(ex, tmp_path):
    """Twelve groups that each see hundreds of cached keys: the gathered keys of all exceed the scratch, which holds those of one
    group of the longest kind, so the groups go in several launches."""
    from llama_rust_b200 import models
    cfg, buckets = nm.MODELS["wide window"]
    w = nm.weights(cfg, 22, buckets, nm.SHARP[nm.AUTO])
    ex.set_path(nm.AUTO)
    s = models.load(ex, nm.write(tmp_path / "m", cfg, w), n_seq=12, n_ctx=400)
    toks = [nm.tokens(300 + 17 + q, cfg, 200 + q) for q in range(12)]
    s.forward([(q, t[:300]) for q, t in enumerate(toks)], [[] for _ in toks])
    got = s.forward([(q, t[300:]) for q, t in enumerate(toks)], [list(range(17 + q)) for q in range(12)])
    at = 0
    for q in (0, 5, 11):
        at = sum(17 + i for i in range(q))
        assert nm.error(got[at:at + 17 + q], plain.forward(cfg, w, toks[q])[300:]).max() <= nm.TOLERANCE[nm.AUTO], q
    s.free()


def test_llama_batch_of_every_kind_of_group(ex):
    """Groups for the three attention kernels of the Llama walk in one batch (a block per row, tiles of one sequence, binary16
    MMAs) with F32 weights: short groups have the bits they have alone, long ones agree with f32 attention."""
    import llama_walk as lw
    from llama_rust_b200 import Session
    cfg = dict(n_layer=2, n_embd=256, n_head=4, n_head_kv=2, head_dim=64, n_ff=256, n_vocab=300)
    rng = np.random.default_rng(72)
    tl = lw.tensor_list(cfg)
    mats = [ex.upload(ALL["F32"], r, c, (rng.standard_normal(r * c) / np.sqrt(c)).astype(np.float32).view(np.uint8)) for _, _, r, c in tl]
    embd = ex.upload(ALL["F32"], 300, 256, rng.standard_normal(300 * 256).astype(np.float32).view(np.uint8))
    names = ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
    layers = [dict(zip(names, mats[7 * i:7 * i + 7])) for i in range(2)]
    lens = [1, 1, 2, 3, 4, 15, 16, 17, 33, 63, 64, 65, 1, 130]
    toks = [lw.prompt_ids(n, 300, n + i) for i, n in enumerate(lens)]
    logits = {}
    for path in (3, 0):
        ex.set_path(path)
        s = Session(ex, dict(cfg, n_ctx=512), embd, layers, output=mats[14], n_seq=len(lens))
        logits[path] = s.batch(list(enumerate(toks)), want_logits=True)[1]
        if path == 3:
            s.reset()
            for q, t in enumerate(toks):
                assert _same_bits(s.batch([(q, t)], want_logits=True)[1][0], logits[3][q]), lens[q]
        s.free()
    ex.set_path(0)
    for q, n in enumerate(lens):
        err, size = np.abs(logits[0][q] - logits[3][q]).max(), np.abs(logits[3][q]).max()
        assert err <= 1e-3 * size if n >= 64 else err <= 1e-5 * size, n


def _llama(ex, n_ctx, n_seq, vocab=300, **session):
    import llama_walk as lw
    from llama_rust_b200 import Session
    cfg = dict(n_layer=2, n_embd=256, n_head=4, n_head_kv=2, head_dim=64, n_ff=256, n_vocab=vocab, n_ctx=n_ctx)
    rng = np.random.default_rng(72)
    tl = lw.tensor_list(cfg)
    mats = [ex.upload(ALL["F32"], r, c, (rng.standard_normal(r * c) / np.sqrt(c)).astype(np.float32).view(np.uint8)) for _, _, r, c in tl]
    embd = ex.upload(ALL["F32"], vocab, 256, rng.standard_normal(vocab * 256).astype(np.float32).view(np.uint8))
    names = ("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down")
    return Session(ex, cfg, embd, [dict(zip(names, mats[7 * i:7 * i + 7])) for i in range(2)], output=mats[14], n_seq=n_seq, **session)


def test_logits_to_pageable_memory(ex):
    """What goes through two pinned pieces of a megabyte in turn (from 256 KB on) has the bytes of a copy to pinned memory: less than a piece,
    a piece and a little, two whole pieces and a little, five; to addresses that are not a page's."""
    import torch
    from llama_rust_b200.executor import lib
    V, S = 16411, 64  # 65644 bytes a row
    s = _llama(ex, 16, S, vocab=V)
    for groups in (1, 3, 4, 16, 17, 32, 47, 64):
        seqs, counts, toks = np.arange(groups, dtype=np.uint32), np.ones(groups, np.uint32), np.arange(groups, dtype=np.int32) * 31
        pinned = torch.full((groups * V,), float("nan")).pin_memory()
        for shift in (0, 1, 1023):
            room = np.full(groups * V + shift + 1, 7, np.float32)
            for ptr in (pinned.data_ptr(), room[shift:].ctypes.data):
                s.reset()
                ex._check(lib().llr_session_batch(s._h, groups, seqs.ctypes.data, counts.ctypes.data, toks.ctypes.data, ptr, None))
            assert _same_bits(room[shift:-1], pinned.numpy()) and (room[:shift] == 7).all() and room[-1] == 7, (groups, shift)
    s.free()


def test_logits_to_device_memory(ex):
    """A device pointer is no host buffer: an error or the driver's own copy, never the host's; the session goes on."""
    import torch
    from llama_rust_b200.executor import lib
    V, S = 16411, 8
    s = _llama(ex, 16, S, vocab=V)
    seqs, counts, toks, want = np.arange(S, dtype=np.uint32), np.ones(S, np.uint32), np.arange(S, dtype=np.int32) * 31, np.arange(S, dtype=np.uint32)
    host = s.batch(list(enumerate(toks[:, None].tolist())), want_logits=True)[1]
    s.reset()
    there = torch.zeros(S, V, device="cuda")
    for call in (lambda p: lib().llr_session_batch(s._h, S, seqs.ctypes.data, counts.ctypes.data, toks.ctypes.data, p, None),
                 lambda p: lib().llr_session_batch_rows(s._h, S, seqs.ctypes.data, counts.ctypes.data, toks.ctypes.data, S, want.ctypes.data, p)):
        assert call(there.data_ptr()) != 0 or _same_bits(there.cpu().numpy(), host)
        s.reset()
        assert _same_bits(s.batch(list(enumerate(toks[:, None].tolist())), want_logits=True)[1], host)
        s.reset()
    s.free()


def test_a_batch_that_runs_out_of_blocks(ex):
    """A batch that fails in the middle of its reservations leaves the blocks of its first groups theirs: what follows finds them."""
    from llama_rust_b200.executor import NativeCudaError
    ex.set_path(0)
    toks = [[(5 * i + 11 * q) % 300 for i in range(60)] for q in range(3)]
    roomy, tight = _llama(ex, 64, 3), _llama(ex, 64, 3, kv_blocks=6)  # 16 positions a block
    first = [(0, toks[0][:20]), (1, toks[1][:40])]  # two blocks and three
    with pytest.raises(NativeCudaError):
        tight.batch(first + [(2, toks[2][:40])])
    assert [tight.seq_position(q) for q in range(3)] == [0, 0, 0]
    for groups in (first, [(0, toks[0][20:32]), (1, toks[1][40:48])], [(0, toks[0][32:33])]):
        assert _same_bits(tight.batch(groups, want_logits=True)[1], roomy.batch(groups, want_logits=True)[1])
    with pytest.raises(NativeCudaError):
        tight.batch([(1, toks[1][48:49])])
    tight.seq_reset(0), roomy.seq_reset(0)
    groups = [(2, toks[2][:33]), (1, toks[1][48:50])]
    with pytest.raises(NativeCudaError):
        tight.batch(groups + [(0, toks[0][:1])])
    for g in (groups[1:], [(2, toks[2][:16])]):
        assert _same_bits(tight.batch(g, want_logits=True)[1], roomy.batch(g, want_logits=True)[1])
    roomy.free()
    tight.free()


def test_pool_far_smaller_than_the_context(ex):
    """The attention scratch is sized for the positions that the pool holds: prompts that fill it, in one batch and in chunks, have the bits
    they have beside a full pool."""
    ex.set_path(0)
    toks = [[(5 * i + 11 * q) % 300 for i in range(320)] for q in range(2)]
    full, small = _llama(ex, 4096, 2), _llama(ex, 4096, 2, kv_blocks=20)
    for lens in ([(160, 160)], [(65, 80), (95, 80)], [(0, 100), (0, 100), (0, 119)], [(64, 0), (256, 0)]):
        got = {}
        for s in (full, small):
            s.reset()
            at, out = [0, 0], []
            for part in lens:
                groups = [(q, toks[q][at[q]:at[q] + n]) for q, n in enumerate(part) if n]
                out.append(s.batch_rows(groups, list(range(sum(part)))))
                at = [a + n for a, n in zip(at, part)]
            got[s] = np.concatenate(out)
        assert _same_bits(got[full], got[small]), lens
    full.reset(), small.reset()
    assert _same_bits(full.prefill(toks[0], want_logits=True), small.prefill(toks[0], want_logits=True))
    full.free()
    small.free()
