"""One token of the recurrent mixers at the sizes where the state's place and the split of its columns change."""
import numpy as np
import pytest

import zav_cases as zc
from oracle import zavilorn as orc
from test_gpu_zavilorn import close, err, make, ok, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("heads,groups,state,vdim,conv,norm_groups", [
    (4, 2, 16, 16, 4, 8),       # norm parts of 8
    (2, 1, 128, 128, 4, 1),     # the largest state that waits in shared memory
    (2, 1, 136, 124, 6, 2),     # above it; more than four taps
    (3, 1, 15, 21, 2, 3),       # not whole 16-byte pieces; odd parts
    (2, 2, 12, 21, 3, 2),       # whole pieces, but one column a thread
    (1, 1, 5, 260, 2, 1),       # more columns than threads, D odd
    (1, 1, 6, 1032, 2, 3),      # ... four a thread
])
def test_token_states(heads, groups, state, vdim, conv, norm_groups, dtype):
    """Tokens one by one, the state-space and the delta recurrence in turn."""
    cfg = zc.config([zc.mam(heads, groups, state, vdim, conv, norm_groups), zc.par(right=(heads, groups, state, vdim), conv=conv, ff=0)],
                    width=72, vocab=151, emb=1.0)
    w = zc.Weights(cfg, 7)
    toks = zc.tokens(cfg, 9, 2)
    want = orc.forward(cfg, w.f64(), toks)
    m = make(cfg, w, dtype, 16)
    m.capture()
    got = run(m, toks, [])
    assert np.isfinite(got).all() and ok(err(got, want), dtype)
    close(m)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("state,vdim", [
    (1, 16384),     # a state of 64 KB that does not fit beside its own values
    (1, 12788),     # the widest of one row that does
    (1, 12792),     # ... and that does not
    (1, 6900),      # the widest of one row that leaves room for two blocks an SM
    (1, 6904),      # ... and that does not
    (128, 256),     # half of the rows in shared memory
    (96, 255),      # 64 of 96 rows, one column a thread
    (63, 65),       # not whole 16-byte pieces
    (1024, 20),     # the most rows
])
def test_wide_heads(state, vdim, dtype):
    """Heads on both sides of what waits in shared memory."""
    cfg = zc.config([zc.mam(1, 1, state, vdim, 2, 1), zc.par(right=(1, 1, state, vdim), conv=2, ff=0)], width=72, vocab=151, emb=1.0)
    w = zc.Weights(cfg, 7)
    toks = zc.tokens(cfg, 6, 2)
    want = orc.forward(cfg, w.f64(), toks)
    m = make(cfg, w, dtype, 16)
    m.capture()
    got = run(m, toks, [])
    assert np.isfinite(got).all() and ok(err(got, want), dtype)
    close(m)


@pytest.mark.parametrize("width,dtype", [(896, "float32"), (912, "float32"), (1800, "bfloat16"), (1816, "bfloat16")])
def test_first_pass(width, dtype):
    """Projections of 4640 rows on both sides of 16 MiB, where the code in front of the wait changes."""
    cfg = zc.config([zc.mam(32, 4, 64, 64, 4, 2)] * 2, width=width, vocab=151, emb=1.0)
    w = zc.Weights(cfg, 7)
    toks = zc.tokens(cfg, 9, 2)
    want = orc.forward(cfg, w.f64(), toks)
    m = make(cfg, w, dtype, 16)
    m.capture()
    got = run(m, toks, [])
    assert np.isfinite(got).all() and ok(err(got, want), dtype)
    close(m)
