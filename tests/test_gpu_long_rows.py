"""The two products of the fp32-activation path at the sizes where they change form: one row against weight rows of 8192 columns
and more (streamed through a ring: just below, the shortest, ragged ones, the longest, beyond), and 5 rows and more (tiles of 8
to 16 rows: one tile, one row more, several), with the norms of both families behind them.  Logits against the plain oracle
with the path's 32-bit tolerance (rms 2e-5 of the logits' spread)."""
import numpy as np
import pytest

from tests import stack_util as su

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ff", [8184, 8192, 8200, 11264, 12296, 16384, 16392])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_single_tokens_and_short_portions(cuda_device, family, ff):
    if family == "keselix":
        cfg = su.model([su.attn(ff=ff)], width=600, vocab=613)
    else:
        cfg = su.bavutar([su.gqa(ff=ff)], width=604, vocab=613)
    w = su.weights(cfg, 3)
    toks = su.ids(5, 76, cfg["vocab"])
    want = su.oracle(cfg).forward(cfg, w, toks)
    rt = su.runtime(cfg, w, "f32", seq=100, max_rows=100)
    rt.start_batch(1)
    for sizes in ((1, 1, 1, 1, 5, 16, 17, 34), (4, 12, 13, 33, 6, 8)):
        rt.release(0)
        got, at = [], 0
        for n in sizes:
            got.append(su.extend(rt, 0, toks[at:at + n]))
            at += n
        assert at == len(toks)
        rt.check_device_status()
        assert su.error(np.concatenate(got), want) <= su.TOL["f32"], sizes
    rt.close()


@pytest.mark.parametrize("width", [8192, 8200, 12288, 12296])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_single_tokens_of_wide_models(cuda_device, family, width):
    """The other products of one row: input projections and the head behind a norm, both feed-forwards."""
    if family == "keselix":
        cfg = su.model([su.attn(heads=8, dim=80, ff=600)], width=width, vocab=613)
    else:
        cfg = su.bavutar([su.gqa(heads=8, dim=80, ff=600)], width=width, vocab=613)
    w = su.weights(cfg, 3)
    toks = su.ids(5, 6, cfg["vocab"])
    want = su.oracle(cfg).forward(cfg, w, toks)
    rt = su.runtime(cfg, w, "f32", seq=20, max_rows=20)
    rt.start_batch(1)
    got = np.concatenate([su.extend(rt, 0, toks[i:i + 1]) for i in range(len(toks))])
    rt.check_device_status()
    assert su.error(got, want) <= su.TOL["f32"]
    rt.close()
