"""The chunked scans of matrix-state layers read records that a warp copies through a ring of three or four stages; a stage that is
handed back before its last loads have returned is overwritten under them, in a few runs of a hundred at most.  The same prompt,
many more chunks than stages and a rest, gives the same bits every time: every padded key width, both scans, few and many columns a
block (16 heads of 40 columns take blocks of 32 columns, 64 heads of 64 blocks of 64)."""
import numpy as np
import pytest

from tests import stack_util as su

pytestmark = pytest.mark.gpu

ROWS, TIMES = 333, 100


@pytest.mark.parametrize("heads,vdim", [(16, 40), (64, 64)])
@pytest.mark.parametrize("dim", [20, 64, 128, 256])
@pytest.mark.parametrize("scan", ["delta", "ssd"])
def test_the_same_prompt_gives_the_same_bits(cuda_device, scan, dim, heads, vdim):
    layer = su.delta(heads=heads, kv_heads=heads, dim=dim, vdim=vdim, ff=None) if scan == "delta" else su.ssd(heads=heads, vdim=vdim, state=dim, groups=4, norm_groups=4)
    cfg = su.bavutar([layer], width=128, vocab=77)
    w = su.weights(cfg, 9)
    toks = su.ids(2, ROWS, cfg["vocab"])
    rt = su.runtime(cfg, w, "many_rows", seq=ROWS, max_rows=ROWS)
    rt.start_batch(1)
    first = None
    for _ in range(TIMES):
        rt.release(0)
        got = su.extend(rt, 0, toks)
        first = got if first is None else first
        assert np.array_equal(got, first)
    rt.check_device_status()
    rt.close()
