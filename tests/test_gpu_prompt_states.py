"""The state-space recurrence and the row operations of a prompt pass at the sizes where their split changes."""
import numpy as np
import pytest

import zav_cases as zc
from oracle import zavilorn as orc
from test_gpu_zavilorn import err, make, ok, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mix,cuts", [
    ((4, 2, 8, 8, 2, 1), [64, 66]),           # fewer columns than a block's, a chunk of two rows behind a state
    ((2, 1, 128, 64, 4, 1), [63, 1, 65]),     # chunks of 63, one and 64 + 1 rows
    ((3, 3, 72, 40, 5, 2), [129]),            # columns behind the last, five taps
    ((10, 5, 64, 104, 8, 2), [257, 300]),     # four and five chunks: one segment
    ((40, 2, 128, 128, 4, 1), [512, 100]),    # 160 blocks a segment: two segments, then one
    ((1, 1, 16, 32, 1, 1), [2048]),           # one block a segment: eight; no convolution
])
@pytest.mark.parametrize("width", [72, 1032, 2100])   # of the rows: one, two and four pieces a thread
def test_prompt_states(mix, cuts, width):
    """A prompt in portions against the oracle."""
    h, g, d, e, conv, parts = mix
    cfg = zc.config([zc.mam(h, g, d, e, conv, parts)], width=width, vocab=160, emb=1.0)
    w = zc.Weights(cfg, 17)
    toks = zc.tokens(cfg, sum(cuts), 4)
    m = make(cfg, w, "bfloat16", sum(cuts) + 8)
    got = run(m, toks, cuts)
    assert np.isfinite(got).all() and ok(err(got, orc.forward(cfg, w.f64(), toks)), "bfloat16")
    m.close()
