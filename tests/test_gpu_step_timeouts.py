"""A whole-step decode kernel whose waits run out: the call reports it, and no arrival is left in the counters, where the next step
would take it for its own.  The limit is one poll, so most waits between blocks give up and return."""
import numpy as np
import pytest

from oracle import spec
from tests.test_gpu_model import _net

pytestmark = pytest.mark.gpu


def _counters(rt, layers):
    """The arrival counters of a handle, a view: they lie behind the table of layers, records of six weights and two cache pools;
    buffers begin every 256 bytes."""
    first = rt._aligned(rt.workspace) - rt.workspace.data_ptr()
    words = rt.workspace[first:].cpu().numpy()
    words = words[:words.size // 256 * 256].view(np.uint64).reshape(-1, 32)[:, :8]

    def inside(w, t):
        return (w >= t.data_ptr()) & (w < t.data_ptr() + t.numel())

    at = np.flatnonzero(inside(words[:, :6], rt.weights_arena).all(1) & inside(words[:, 6:], rt.workspace).all(1))
    assert len(at) == 1
    behind = first + 256 * int(at[0]) + (64 * layers + 255) // 256 * 256
    return rt.workspace[behind:behind + 4 * (5 * layers + 3)]


@pytest.mark.parametrize("d,heads,narrow", [(1024, 4, False), (2048, 32, False), (1024, 4, True), (512, 2, False)])
def test_no_arrival_is_left_behind(cuda_device, monkeypatch, d, heads, narrow):
    from mesh_transformer._lib import MtjError
    if narrow:
        monkeypatch.setenv("MTJ_MEGA_NARROW", "1")
    cfg = dict(spec.gptj6b_config(1), layers=4, d_model=d, n_heads=heads, n_vocab=516, seq=200, pe_rotary_dims=64, mtj_wait_limit=1)
    net = _net(cfg, spec.make_params(cfg, seed=3), cuda_device)
    ctx = np.zeros((1, 200), np.uint32)
    ctx[0, 50:] = spec.token_ids(1, 1, 150, 516)[0]
    counters = None
    for _ in range(5):
        with pytest.raises(MtjError) as err:
            net.generate(ctx, np.array([150], np.uint32), 8, {"top_p": np.zeros(1), "temp": np.ones(1)})
        assert err.value.code == 5                                            # MTJ_ERR_TIMEOUT
        net._rt.check_device_status()                                         # said once
        counters = _counters(net._rt, 4) if counters is None else counters
        assert not counters.any()
    net.close()
