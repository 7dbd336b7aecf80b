"""The device-resident Llama walk (llr_session_*: embedding lookup, RMSNorm, RoPE, KV cache, grouped-query attention,
SwiGLU, residual adds and greedy argmax on the device) against the CPU walk of the oracle (the reference's host code,
langtax/src/decode.rs:2710-3097).  The two differ in the order of a few f32 sums, so tokens are compared up to the first
step the CPU walk itself decides narrowly, and logits within the reference's model-level tolerance of 1e-3 of their scale."""
import json
import os

import numpy as np
import pytest

import llama_walk as lw

pytestmark = pytest.mark.gpu
GOLDEN_CENTERED = os.path.join(os.path.dirname(__file__), "golden", "config3_centered_golden.json")


def _session(ex, cfg, n_ctx, mats, embd_mat, norms=None, **kw):
    from llama_rust_b200 import Session
    layers = []
    for li in range(cfg["n_layer"]):
        m = mats[7 * li:7 * li + 7]
        L = dict(zip(("attn_q", "attn_k", "attn_v", "attn_output", "ffn_gate", "ffn_up", "ffn_down"), m))
        if norms is not None:
            L["attn_norm"], L["ffn_norm"] = norms[li]
        layers.append(L)
    return Session(ex, dict(cfg, n_ctx=n_ctx), embd_mat, layers, output=mats[7 * cfg["n_layer"]], **kw)


def test_small_model_tokens_and_logits_match_the_cpu_walk(orc):
    from llama_rust_b200 import Executor
    cfg = dict(n_layer=3, n_embd=512, n_head=8, n_head_kv=2, head_dim=64, n_ff=2048, n_vocab=3000)
    n_prompt, n_gen, n_ctx = 24, 40, 64
    tl = lw.tensor_list(cfg)
    weights, embd = lw.centered_weights(cfg, 33)
    prompt = lw.prompt_ids(n_prompt, cfg["n_vocab"], 99)
    ids_cpu, margin, logits_cpu = lw.run_cpu(cfg, n_ctx, weights, embd, prompt, n_gen, want_logits=True)
    scale = float(np.abs(logits_cpu).max())
    ex = Executor(0)
    ex.set_path(3)  # f32-faithful products for every batch size
    mats = [ex.upload(dt, rows, cols, w) for (name, dt, rows, cols), w in zip(tl, weights)]
    embd_mat = ex.upload(lw.Q4_K, cfg["n_vocab"], cfg["n_embd"], embd)
    s = _session(ex, cfg, n_ctx, mats, embd_mat)
    first = s.prefill(prompt, want_logits=True)
    assert s.position == n_prompt and np.all(np.isfinite(first))
    ids, m_dev = s.decode(n_gen)
    assert s.position == n_prompt + n_gen
    n = lw.compared_prefix(ids_cpu, margin, scale)
    assert n >= n_gen // 2, (n, margin.min(), scale)
    assert np.array_equal(ids[:n], ids_cpu[:n]), (ids, ids_cpu, margin)
    if n == n_gen:  # the same sequence was fed back: the last logits and the margins are comparable
        assert np.abs(s.logits() - logits_cpu).max() <= 1e-3 * scale
        assert np.abs(m_dev - margin).max() <= 2e-3 * scale
    # a second sequence after a reset gives the same tokens (the cache and the position start over)
    s.reset()
    s.prefill(prompt)
    ids2, _ = s.decode(n_gen)
    assert np.array_equal(ids2, ids)
    # prefill in two parts equals prefill in one (positions and the cache carry over)
    s.reset()
    s.prefill(prompt[:10])
    s.prefill(prompt[10:])
    ids3, _ = s.decode(8)
    assert np.array_equal(ids3, ids[:8])
    s.free()
    ex.close()


@pytest.mark.parametrize("n_ctx", [128, 4096])  # slices of 32 positions; of 128, the longest the tiled kernel stages
def test_prompt_chunks_and_single_tokens_give_the_same_bits(orc, n_ctx):
    """A prompt forwarded as one chunk (rows share each slice's keys and values through a shared-memory tile), in ragged
    pieces, and token by token (one row per block, straight from the paged cache) leaves the same logits, bit for bit:
    both attention kernels run one per-row routine.  Context of 100 positions: several slices per row."""
    from llama_rust_b200 import Executor
    cfg = dict(n_layer=2, n_embd=512, n_head=8, n_head_kv=2, head_dim=64, n_ff=1024, n_vocab=1000)
    tl = lw.tensor_list(cfg)
    weights, embd = lw.centered_weights(cfg, 5)
    ex = Executor(0)
    ex.set_path(3)
    mats = [ex.upload(dt, rows, cols, w) for (name, dt, rows, cols), w in zip(tl, weights)]
    embd_mat = ex.upload(lw.Q4_K, cfg["n_vocab"], cfg["n_embd"], embd)
    n_prompt = 100 if n_ctx == 128 else 300  # 300: rows in the first, second and third slice of 128 positions
    prompt = lw.prompt_ids(n_prompt, cfg["n_vocab"], 3)
    s = _session(ex, cfg, n_ctx, mats, embd_mat, n_seq=1, kv_blocks=128, block_tokens=4)
    whole = s.prefill(prompt, want_logits=True)
    s.reset()
    for piece in (prompt[:3], prompt[3:40], prompt[40:41], prompt[41:n_prompt - 1]):
        s.prefill(piece)
    pieces = s.prefill(prompt[n_prompt - 1:], want_logits=True)
    s.reset()
    for t in prompt[:-1]:
        s.prefill([t])
    single = s.prefill(prompt[-1:], want_logits=True)
    assert np.array_equal(whole.view(np.uint32), pieces.view(np.uint32))
    assert np.array_equal(whole.view(np.uint32), single.view(np.uint32))
    s.free()
    ex.close()


@pytest.mark.parametrize("n_head,n_head_kv,head_dim,n_ctx", [(4, 2, 64, 1024), (4, 1, 128, 2048), (8, 1, 64, 2048), (2, 2, 128, 512),
                                                             (4, 2, 128, 4096)])  # 4096: the f32 kernels' slices are 128 positions long
def test_prompt_attention_on_tensor_cores_agrees_with_the_f32_kernels(orc, n_head, n_head_kv, head_dim, n_ctx):
    """Prompt chunks of 64 rows and more run their attention as binary16 MMAs with f32 accumulation on the automatic path.
    With F32 weights the products are the same f32 kernels on both paths, so the logits of the automatic path and of the
    f32-faithful path differ by the attention kernel alone: they must agree within the 16-bit tolerance (1e-3 of the
    logit scale; a misplaced fragment would change them by the scale itself), for one to eight query heads per kv head, contexts with
    f32 slices of 32, 64 and 128 positions beside them, prompts that are not a multiple of the row tile, a second chunk that starts in the
    middle of a step of 128 keys, and against the CPU walk.  (Prompts beyond two steps: test_gpu_attention_tiles.py.)"""
    from llama_rust_b200 import Executor
    from helpers import F32
    cfg = dict(n_layer=2, n_embd=n_head * head_dim, n_head=n_head, n_head_kv=n_head_kv, head_dim=head_dim, n_ff=256, n_vocab=300)
    rng = np.random.default_rng(n_head * 100 + head_dim + n_ctx)
    tl = lw.tensor_list(cfg)
    weights = [(rng.standard_normal(r * c) / np.sqrt(c)).astype(np.float32).view(np.uint8) for _, _, r, c in tl]
    embd = rng.standard_normal(cfg["n_vocab"] * cfg["n_embd"]).astype(np.float32).view(np.uint8)
    prompt = lw.prompt_ids(150, cfg["n_vocab"], 5)
    more = lw.prompt_ids(77, cfg["n_vocab"], 6)
    logits = {}
    ex = Executor(0)
    mats = [ex.upload(F32, r, c, w) for (_, _, r, c), w in zip(tl, weights)]
    embd_mat = ex.upload(F32, cfg["n_vocab"], cfg["n_embd"], embd)
    for path in (0, 3):
        ex.set_path(path)
        s = _session(ex, cfg, n_ctx, mats, embd_mat)
        a = s.prefill(prompt, want_logits=True)
        b = s.prefill(more, want_logits=True)  # positions 150..226: the chunk starts inside a step
        logits[path] = (a, b)
        s.free()
    cpu = lw.run_cpu(cfg, n_ctx, weights, embd, np.concatenate([prompt, more]), 0, want_logits=True, kinds=[F32] * len(tl), embd_kind=F32)[2]
    for i in range(2):
        scale = float(np.abs(logits[3][i]).max())
        assert np.all(np.isfinite(logits[0][i]))
        err = float(np.abs(logits[0][i] - logits[3][i]).max())
        assert 0.0 < err <= 1e-3 * scale, (i, err, scale)  # not zero either: the automatic path took the other kernel
    assert np.abs(logits[0][1] - cpu).max() <= 1e-3 * float(np.abs(cpu).max())
    assert np.abs(logits[3][1] - cpu).max() <= 1e-4 * float(np.abs(cpu).max())
    ex.close()


def test_ragged_batch_over_several_sequences_equals_running_them_one_by_one(orc):
    """Engine-style batches (engine.rs:1215-1274): ragged groups of prompt chunks and single decode tokens of three
    sequences flattened into one activation matrix per step, against the same sequences run alone in a one-sequence
    session.  With the f32-faithful products a row does not depend on its batch: logits must be the same bits.  The KV
    pool is paged (blocks of 4 positions, fewer blocks than three full contexts) and blocks return on reset."""
    from llama_rust_b200 import Executor, NativeCudaError
    cfg = dict(n_layer=2, n_embd=512, n_head=8, n_head_kv=2, head_dim=64, n_ff=1024, n_vocab=1000)
    n_ctx = 48
    tl = lw.tensor_list(cfg)
    weights, embd = lw.centered_weights(cfg, 21)
    ex = Executor(0)
    ex.set_path(3)
    mats = [ex.upload(dt, rows, cols, w) for (name, dt, rows, cols), w in zip(tl, weights)]
    embd_mat = ex.upload(lw.Q4_K, cfg["n_vocab"], cfg["n_embd"], embd)
    prompts = [lw.prompt_ids(n, cfg["n_vocab"], 50 + n) for n in (11, 5, 17)]
    # reference: each sequence alone, prompt in one piece, then greedy tokens one by one with their logits
    alone = _session(ex, cfg, n_ctx, mats, embd_mat)
    want = []
    for p in prompts:
        alone.reset()
        lg = [alone.prefill(p, want_logits=True)]
        toks = []
        for _ in range(3):
            t = int(np.argmax(lg[-1]))
            toks.append(t)
            lg.append(alone.prefill([t], want_logits=True))
        want.append((toks, lg))
    alone.free()
    s = _session(ex, cfg, n_ctx, mats, embd_mat, n_seq=3, kv_blocks=24, block_tokens=4)  # 24 blocks x 4 = 96 positions < 3 x 48
    # step 1: ragged prompt chunks (sequence 2's prompt arrives in two chunks; groups given out of order)
    nxt, lg = s.batch([(2, prompts[2][:9]), (0, prompts[0]), (1, prompts[1])], want_logits=True)
    assert np.array_equal(lg[1].view(np.uint32), want[0][1][0].view(np.uint32))
    assert np.array_equal(lg[2].view(np.uint32), want[1][1][0].view(np.uint32))
    assert nxt[1] == want[0][0][0] and nxt[2] == want[1][0][0]
    # step 2: sequences 0 and 1 decode one token each while sequence 2 takes the rest of its prompt
    nxt, lg = s.batch([(0, [want[0][0][0]]), (1, [want[1][0][0]]), (2, prompts[2][9:])], want_logits=True)
    assert np.array_equal(lg[0].view(np.uint32), want[0][1][1].view(np.uint32))
    assert np.array_equal(lg[1].view(np.uint32), want[1][1][1].view(np.uint32))
    assert np.array_equal(lg[2].view(np.uint32), want[2][1][0].view(np.uint32))
    assert [int(v) for v in nxt] == [want[0][0][1], want[1][0][1], want[2][0][0]]
    # step 3: all three decode
    nxt, lg = s.batch([(q, [want[q][0][1 if q < 2 else 0]]) for q in range(3)], want_logits=True)
    for q in range(3):
        assert np.array_equal(lg[q].view(np.uint32), want[q][1][2 if q < 2 else 1].view(np.uint32)), q
    assert [s.seq_position(q) for q in range(3)] == [13, 7, 18]
    # the pool is bounded: 13 + 7 + 18 positions hold 4 + 2 + 5 = 11 of the 24 blocks
    s.batch([(0, list(range(35)))])              # sequence 0 to its full context: 12 blocks, 5 left
    with pytest.raises(NativeCudaError) as err:
        s.batch([(1, list(range(41)))])          # sequence 1 would need 10 more
    assert err.value.code == 7 and s.seq_position(1) == 7
    s.seq_reset(0)                               # its 12 blocks return to the pool
    s.batch([(1, list(range(41)))])
    assert s.seq_position(1) == 48 and s.seq_position(0) == 0
    with pytest.raises(NativeCudaError):
        s.batch([(1, [1])])                      # beyond the context length
    with pytest.raises(NativeCudaError):
        s.batch([(0, [1]), (0, [2])])            # a sequence twice in one batch
    s.free()
    ex.close()


def test_ragged_batch_with_long_groups_takes_the_tensor_cores_per_group(orc):
    """On the automatic path every group of 64 rows and more of a ragged batch runs its attention on the tensor cores (one
    sequence at consecutive positions), the runs of shorter groups between them keep the f32 kernels.  F32 weights: the
    products are the same on both paths, so short groups must give the bits of the f32-faithful path and long groups
    must agree with it within the 16-bit tolerance (and differ from it: the other kernel did run)."""
    from llama_rust_b200 import Executor
    from helpers import F32
    cfg = dict(n_layer=2, n_embd=256, n_head=4, n_head_kv=2, head_dim=64, n_ff=256, n_vocab=300)
    rng = np.random.default_rng(71)
    tl = lw.tensor_list(cfg)
    weights = [(rng.standard_normal(r * c) / np.sqrt(c)).astype(np.float32).view(np.uint8) for _, _, r, c in tl]
    embd = rng.standard_normal(cfg["n_vocab"] * cfg["n_embd"]).astype(np.float32).view(np.uint8)
    ex = Executor(0)
    mats = [ex.upload(F32, r, c, w) for (_, _, r, c), w in zip(tl, weights)]
    embd_mat = ex.upload(F32, cfg["n_vocab"], cfg["n_embd"], embd)
    groups1 = [(0, lw.prompt_ids(3, 300, 1)), (1, lw.prompt_ids(100, 300, 2)), (2, lw.prompt_ids(5, 300, 3)), (3, lw.prompt_ids(1, 300, 4)),
               (4, lw.prompt_ids(70, 300, 5))]
    groups2 = [(1, lw.prompt_ids(90, 300, 6)), (0, lw.prompt_ids(2, 300, 7)), (4, lw.prompt_ids(64, 300, 8))]  # long groups start mid-slice
    got = {}
    for path in (0, 3):
        ex.set_path(path)
        s = _session(ex, cfg, 1024, mats, embd_mat, n_seq=5, kv_blocks=0, block_tokens=16)
        _, lg1 = s.batch(groups1, want_logits=True)
        _, lg2 = s.batch(groups2, want_logits=True)
        got[path] = (lg1, lg2)
        s.free()
    for step, long_groups in ((0, (1, 4)), (1, (0, 2))):
        for gi in range(len(got[0][step])):
            a, b = got[0][step][gi], got[3][step][gi]
            if gi in long_groups:
                err = float(np.abs(a - b).max())
                assert 0.0 < err <= 1e-3 * float(np.abs(b).max()), (step, gi, err)
            else:
                assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (step, gi)
    ex.close()


def test_session_validates_its_model_and_calls():
    from llama_rust_b200 import Executor, NativeCudaError, Session
    cfg = dict(n_layer=1, n_embd=256, n_head=4, n_head_kv=2, head_dim=64, n_ff=512, n_vocab=300)
    ex = Executor(0)
    tl = lw.tensor_list(cfg)
    mats = [ex.synth(dt, rows, cols, 5 + i) for i, (name, dt, rows, cols) in enumerate(tl)]
    embd = ex.synth(lw.Q4_K, cfg["n_vocab"], cfg["n_embd"], 3)
    s = _session(ex, cfg, 16, mats, embd)
    with pytest.raises(NativeCudaError):
        s.decode(1)                      # no logits yet
    with pytest.raises(NativeCudaError):
        s.prefill([300])                 # token id out of range
    with pytest.raises(NativeCudaError):
        s.prefill(list(range(17)))       # longer than the context
    s.prefill([1, 2, 3])
    with pytest.raises(NativeCudaError):
        s.decode(14)                     # 3 + 14 > 16
    ids, _ = s.decode(13)
    assert ids.shape == (13,) and s.position == 16
    s.free()
    bad = list(mats)
    bad[0] = mats[1]                     # attn_q with attn_k's shape
    with pytest.raises(NativeCudaError):
        _session(ex, cfg, 16, bad, embd)
    other = Executor(0)
    with pytest.raises(NativeCudaError):  # matrices of another executor
        _session(other, cfg, 16, mats, embd)
    other.close()
    ex.close()


def test_llama3_8b_shape_centered_greedy_tokens_on_the_device():
    """benchmark config 3 with the whole walk on the device: 512 prompt tokens, 128 greedy tokens, f32-faithful products,
    against the CPU tokens of tests/golden.  Asserted up to the first step the CPU walk decides by less than 1e-3 of the
    logit scale (its two near-ties); the outcome for all 128 is printed."""
    if not os.path.exists(GOLDEN_CENTERED):
        pytest.skip("tests/golden/config3_centered_golden.json has not been generated")
    import time
    from llama_rust_b200 import Executor
    g = json.load(open(GOLDEN_CENTERED))
    cfg = lw.LLAMA3_8B
    tl = lw.tensor_list(cfg)
    weights, embd = lw.centered_weights(cfg, g["base_seed"])
    ex = Executor(0)
    ex.set_path(3)
    mats = [ex.upload(dt, rows, cols, w) for (name, dt, rows, cols), w in zip(tl, weights)]
    embd_mat = ex.upload(lw.Q4_K, cfg["n_vocab"], cfg["n_embd"], embd)
    del weights, embd
    s = _session(ex, cfg, g["n_prompt"] + g["n_gen"], mats, embd_mat)
    prompt = lw.prompt_ids(g["n_prompt"], cfg["n_vocab"], g["prompt_seed"])
    t0 = time.perf_counter()
    s.prefill(prompt)
    t1 = time.perf_counter()
    ids, margin = s.decode(g["n_gen"])
    t2 = time.perf_counter()
    ref = np.array(g["ids"])
    n = lw.compared_prefix(ref, g["top2_margin"], g["logit_scale"])
    same = ids == ref
    first = -1 if same.all() else int(np.argmin(same))
    print(f"config 3 on the device: prefill {1e3 * (t1 - t0):.1f} ms for {g['n_prompt']} tokens, decode {1e3 * (t2 - t1) / g['n_gen']:.3f} ms per token "
          f"({g['n_gen'] / (t2 - t1):.0f} tokens/s); " + ("all 128 tokens identical" if first < 0 else
          f"first difference at token {first} (reference margin there {g['top2_margin'][first]:.3g} of scale {g['logit_scale']:.4g})"))
    assert n >= 16
    assert np.array_equal(ids[:n], ref[:n]), f"first difference at {first} of {n} decidable tokens"
    if first >= 0:
        assert g["top2_margin"][first] < 2e-2 * g["logit_scale"]
    s.free()
    ex.close()
