"""Layer stacks on the tensor cores at widths where an output projection is cut along K and the row kernel behind it adds the
pieces: rows of every form of that kernel (up to 2048, 4096 and 8192 columns in registers, wider ones in shared memory), the
small tiles (3 rows) and the pair kernel (from 33 rows on, tiles of 64 to 256 rows and one row more).  Every position's logits
against the plain oracle with the path's tolerance (bf16 operands); a piece lost or added twice is an error of the order of the
logits themselves."""
import numpy as np
import pytest

from tests import stack_util as su

pytestmark = pytest.mark.gpu

PORTIONS = (3, 33, 65, 129, 257, 513)


@pytest.mark.parametrize("width", [512, 2056, 4096, 4104, 8192, 8200])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_output_projections_in_pieces(cuda_device, family, width):
    if family == "keselix":
        cfg = su.model([su.attn(heads=4, dim=40, vdim=128, ff=2048)], width=width, vocab=300)
    else:
        cfg = su.bavutar([su.gqa(heads=4, dim=40, vdim=128, ff=2048)], width=width, vocab=300, cap=None)
    w = su.weights(cfg, 4)
    toks = su.ids(6, sum(PORTIONS), cfg["vocab"])
    want = su.oracle(cfg).forward(cfg, w, toks)
    rt = su.runtime(cfg, w, "many_rows", seq=len(toks), max_rows=600)
    rt.start_batch(1)
    at = 0
    for n in PORTIONS:
        got = su.extend(rt, 0, toks[at:at + n])
        assert su.agrees(su.position_errors(got, want[at:at + n]), "many_rows"), n
        at += n
    rt.check_device_status()
    rt.close()
