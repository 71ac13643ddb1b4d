"""Products of one row whose weights are streamed through a ring: the widths at which the warps' shares of a row change, rows that no
share divides, one row a stage, the smallest product that goes this way, heads with padded rows, both families' norms behind it.
Logits against the plain oracle with the path's 32-bit tolerance."""
import numpy as np
import pytest

from tests import stack_util as su

pytestmark = pytest.mark.gpu
SMALLEST = 12 << 20                                       # weights of a product


@pytest.mark.parametrize("width,ff", [(1024, 6144), (1024, 12288), (1032, 12296), (1032, 16384), (1032, 16392), (2048, 3072), (2056, 6144), (3000, 4200), (4096, 3080), (4104, 3080), (8192, 1544), (8200, 1544)])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_single_tokens(cuda_device, family, width, ff):
    vocab = SMALLEST // width + 5                         # not a multiple of 4: rows of padding behind the head's
    if family == "keselix":
        cfg = su.model([su.attn(heads=8, dim=80, ff=ff)], width=width, vocab=vocab)
    else:
        cfg = su.bavutar([su.gqa(heads=8, dim=80, ff=ff)], width=width, vocab=vocab)
    w = su.weights(cfg, 3)
    toks = su.ids(5, 4, cfg["vocab"])
    want = su.oracle(cfg).forward(cfg, w, toks)
    rt = su.runtime(cfg, w, "f32", seq=20, max_rows=20)
    rt.start_batch(1)
    got = np.concatenate([su.extend(rt, 0, toks[i:i + 1]) for i in range(len(toks))])
    rt.check_device_status()
    assert su.error(got, want) <= su.TOL["f32"]
    rt.close()


@pytest.mark.parametrize("width,ff", [(592, 8192), (600, 12296), (604, 16384), (588, 8192)])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_long_rows_of_few_weights(cuda_device, family, width, ff):
    """From four rows a block on, rows of 8192 columns and more are streamed however few the weights are; with one row less not."""
    test_single_tokens(cuda_device, family, width, ff)


@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_the_same_tokens_give_the_same_bits(cuda_device, family):
    """A stage of weights is handed back before it is read if nothing has waited for its loads: most stages in the ring at once, the
    longest rows (seen in 3 of 100 tokens)."""
    layer = su.attn(heads=8, dim=80, ff=16384) if family == "keselix" else su.gqa(heads=8, dim=80, ff=16384)
    cfg = (su.model if family == "keselix" else su.bavutar)([layer], width=1032, vocab=613)
    w = su.weights(cfg, 3)
    toks = su.ids(5, 4, cfg["vocab"])
    rt = su.runtime(cfg, w, "f32", seq=20, max_rows=20)
    rt.start_batch(1)
    first = None
    for _ in range(100):
        rt.release(0)
        got = np.concatenate([su.extend(rt, 0, toks[i:i + 1]) for i in range(len(toks))])
        first = got if first is None else first
        assert np.array_equal(got, first)
    rt.check_device_status()
    rt.close()
