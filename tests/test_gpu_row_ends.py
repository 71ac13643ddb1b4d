"""Residual rows of widths that are no multiple of 8: the padding behind a row has to stay zero whatever the row holds."""
import numpy as np
import pytest

from tests import stack_util as su

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("portion", [1, 4, 5, 20])
def test_a_row_that_was_not_finite_leaves_nothing_behind(cuda_device, portion):
    """A token whose embedding holds an infinity, in portions of every form of the few-row path (a row, up to four, and from
    five on, where the norm behind a product is a kernel of its own), then, in the same slot, a sequence without it."""
    cfg = su.bavutar([su.gqa(ff=44), su.gqa()], width=604)
    w = su.weights(cfg, 7)
    bad = dict(w)
    name = next(k for k, v in w.items() if v.shape == (cfg["vocab"], cfg["width"]) and "embed" in k)
    bad[name] = w[name].copy()
    bad[name][0, 5] = np.inf
    toks = 1 + su.ids(8, 20, cfg["vocab"] - 1)
    want = su.oracle(cfg).forward(cfg, w, toks)
    rt = su.runtime(cfg, bad, "f32", seq=60, max_rows=60)
    rt.start_batch(1)
    for at in range(0, 20, portion):
        assert not np.isfinite(su.extend(rt, 0, np.zeros(portion, np.int32))).any()
    rt.release(0)
    got = np.concatenate([su.extend(rt, 0, toks[at:at + portion]) for at in range(0, 20, portion)])
    assert su.error(got, want) <= su.TOL["f32"]
    rt.close()
