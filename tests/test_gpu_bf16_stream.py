"""Products of layered decoders with few rows (at most 64 activation rows: tiles of 32 .. 128 weight rows, stages of 32 or 64 activation
rows) at the edges of both, gated units and sliced products among them, against the plain float64 statement."""
import numpy as np
import pytest

import nagolix_models as nm
import nagolix_plain as plain

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,ff", [(40, 24), (72, 200), (256, 1032), (512, 2048), (1032, 520)])
def test_few_rows(tmp_path, width, ff):
    from llama_rust_b200 import Executor, models
    cfg = nm.config(width, 90, [nm.attention(4, 2, 24, 40, 50, 3, 24), nm.latent(5, 16, 24, 48, 1000)], ff)
    w = nm.weights(cfg, 29, 10, nm.SHARP[nm.AUTO])
    toks = nm.tokens(65, cfg, 31)
    want = plain.forward(cfg, w, toks)
    with Executor(0) as ex:
        s = models.load(ex, nm.write(tmp_path / "m", cfg, w))
        for n in (16, 17, 31, 32, 33, 48, 63, 64, 65):
            s.reset()
            got = s.forward([(0, toks[:n])], [list(range(n))])
            assert nm.error(got, want[:n]).max() <= nm.TOLERANCE[nm.AUTO], n
        s.free()


# More tiles than SMs: gated products whose widest tiles leave rings of three stages, two blocks to an SM (33 rows and more); an input
# product of 29568 rows, which is streamed up to 32 activation rows and takes whole tiles from 33 on.
@pytest.mark.parametrize("layer,ff", [(nm.attention(2, 1, 24, 24, 50, 3, 24), 16640), (nm.attention(32, 1, 448, 448, 50, 3, 24), 0)])
def test_few_rows_of_many_tiles(tmp_path, layer, ff):
    from llama_rust_b200 import Executor, models
    cfg = nm.config(264, 90, [layer], ff)
    w = nm.weights(cfg, 29, 10, nm.SHARP[nm.AUTO])
    toks = nm.tokens(65, cfg, 31)
    want = plain.forward(cfg, w, toks)
    with Executor(0) as ex:
        s = models.load(ex, nm.write(tmp_path / "m", cfg, w))
        for n in (16, 32, 33, 64, 65):
            s.reset()
            got = s.forward([(0, toks[:n])], [list(range(n))])
            assert nm.error(got, want[:n]).max() <= nm.TOLERANCE[nm.AUTO], n
        s.free()
