"""The product of the fp32-activation path for 2 rows and more at the edges of its tiles: 8, 16, 24 and 32 rows (one less, full,
one more, several tiles), weight rows and columns below, at and above its 64 rows and 128 columns, and K cut into pieces.  Logits
against the plain oracle with the path's 32-bit tolerance (rms 2e-5 of the logits' spread)."""
import numpy as np
import pytest

from tests import stack_util as su

pytestmark = pytest.mark.gpu

PORTIONS = [(2, 3, 4, 7), (8, 9, 15), (16, 17), (23, 24), (25, 31), (32, 33), (40, 64), (65, 96), (97, 7)]


@pytest.mark.parametrize("ff", [56, 124, 128, 136, 520])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_portions_around_the_tiles(cuda_device, family, ff):
    if family == "keselix":
        cfg = su.model([su.attn(ff=ff), su.ssm()], width=600, vocab=613)
    else:
        cfg = su.bavutar([su.gqa(ff=ff), su.delta(), su.ssd()], width=604, vocab=613)
    w = su.weights(cfg, 11)
    toks = su.ids(6, 104, cfg["vocab"])
    want = su.oracle(cfg).forward(cfg, w, toks)
    rt = su.runtime(cfg, w, "f32", seq=130, max_rows=130)
    rt.start_batch(1)
    for sizes in PORTIONS:
        rt.release(0)
        got, at = [], 0
        for n in sizes:
            n = min(n, len(toks) - at)
            got.append(su.extend(rt, 0, toks[at:at + n]))
            at += n
        rt.check_device_status()
        assert su.error(np.concatenate(got), want[:at]) <= su.TOL["f32"], sizes
    rt.close()


def test_an_infinite_activation_stays_infinite(cuda_device):
    """The pieces an fp32 number is cut into are finite parts of it; an infinity has none below its own: rows that hold one are
    not finite, the others of the same portion are what they are without it."""
    cfg = su.bavutar([su.gqa(ff=None)], width=64, vocab=77)
    w = su.weights(cfg, 5)
    name = next(k for k, v in w.items() if v.shape == (cfg["vocab"], cfg["width"]) and "embed" in k)
    bad = dict(w)
    bad[name] = w[name].copy()
    bad[name][0, 3] = np.inf
    toks = 1 + su.ids(8, 20, cfg["vocab"] - 1)
    want = su.oracle(cfg).forward(cfg, w, toks)
    toks = np.append(toks, 0).astype(toks.dtype)                   # nothing looks forward
    rt = su.runtime(cfg, bad, "f32", seq=30, max_rows=30)
    rt.start_batch(1)
    got = su.extend(rt, 0, toks)
    assert not np.isfinite(got[-1]).any()
    assert su.error(got[:-1], want) <= su.TOL["f32"]
    rt.close()
