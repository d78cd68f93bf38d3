"""Gated linear attention over a prompt at the widths where its loads come in whole pieces or not."""
import numpy as np
import pytest

import dar_cases as dc
from oracle import daronex as orc
from test_gpu_daronex import close, err, make, ok, run, weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,dim,vdim", [
    (2, 128, 128),    # rates, keys, values and state in whole pieces
    (2, 128, 100),    # whole in front, a ragged block of columns behind
    (3, 64, 66),      # values not of 16 bytes
    (1, 120, 64),     # keys narrower than their tile
    (2, 256, 64),     # the widest tile, a thread for every row of a column
    (2, 32, 21),      # odd
])
def test_prompt_gla(heads, dim, vdim):
    """A prompt in portions with last chunks of one row and of 63, against the oracle."""
    cfg = dc.config([dc.gla(heads, dim, vdim, 16.0), dc.gla(heads, dim, vdim, 4.0, ff=0)], width=96)
    w = weights(cfg, 23)
    toks = dc.tokens(cfg, 192, 3)
    m = make(cfg, w, "bfloat16")
    got = run(m, toks, [65, 127])
    assert np.isfinite(got).all() and ok(err(got, orc.forward(cfg, w.f64(), toks)), "bfloat16")
    close(m)
