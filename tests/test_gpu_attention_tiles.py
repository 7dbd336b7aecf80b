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
    "keys beyond the tile kernel": nm.attention(2, 1, 776, 64, 127, 1, 40),
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
