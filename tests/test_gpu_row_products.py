"""The one-row products of the layer stack at the widths where a block's share of a row changes."""
import numpy as np
import pytest

import zav_cases as zc
from oracle import zavilorn as orc
from test_gpu_zavilorn import close, err, make, ok, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,ff", [
    (64, 40), (264, 2056), (520, 1032), (1040, 5000), (2056, 48), (4104, 40),   # 1 .. 8 warps on a row, 1 .. 4 chunks a thread
    (8200, 40), (72, 16392), (64, 17000), (52, 8201),                           # up to 8; rows too long; odd widths
])
def test_row_products(width, ff, dtype):
    """Tokens one by one: f32 as the other tests, bf16 weights and keys."""
    cfg = zc.config([zc.mam(6, 2, 16, 24, 4, 3, ff=ff), zc.par(ff=0)], width=width, vocab=151, emb=1.0)
    w = zc.Weights(cfg, 5)
    toks = zc.tokens(cfg, 12, 2)
    want = orc.forward(cfg, w.f64(), toks)
    m = make(cfg, w, dtype, 16)
    m.capture()
    got = run(m, toks, [])
    assert np.isfinite(got).all() and ok(err(got, want), dtype)
    close(m)


def test_longest_row():
    """The longest row that a block holds, without room for the partial sums of split rows, and one beyond."""
    from cpp_tensorlib_b200 import TlbError
    for ff in (57600, 57608):
        cfg = zc.config([zc.mam(6, 2, 16, 24, 4, 3, ff=ff)], width=64, vocab=151, emb=1.0)
        w = zc.Weights(cfg, 5)
        toks = zc.tokens(cfg, 3, 2)
        m = make(cfg, w, "bfloat16", 16)
        if ff > 57600:
            with pytest.raises(TlbError, match="does not fit"):
                run(m, toks, [])
            m.close()
            continue
        want = orc.forward(cfg, w.f64(), toks)
        got = run(m, toks, [])
        assert np.isfinite(got).all() and ok(err(got, want), "bfloat16")
        close(m)
