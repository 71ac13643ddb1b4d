"""The projection's loss as a unit entry and as the end of an evaluation: the same kernels at the same row counts, so the same
bits.  The model's one layer adds nothing (its output weights and bias are zero), so that an evaluation's last rows are the
embedded ids."""
import numpy as np
import pytest

from oracle import spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [31, 33, 64, 65, 129, 192, 193, 257])
def test_the_unit_entry_equals_evaluation(cuda_device, rows):
    import torch
    from mesh_transformer._runtime import ShardRuntime
    torch.cuda.set_device(cuda_device)
    cfg = dict(spec.tiny_config(1, seq=260), layers=1)
    full = spec.full_weights(cfg, seed=3, stress=True)
    for leaf in ("o", "ff_out_w", "ff_out_b"):
        full["layers"][0][leaf][:] = 0
    rt = ShardRuntime(cfg, max_batch=1, max_gen=1, max_rows=260)
    rt.load_params(spec.shard_params(cfg, full))
    dev = lambda seed: torch.from_numpy(spec.token_ids(seed, 1, rows, cfg["n_vocab"]).view(np.int32)).to(cuda_device)
    obs, target = dev(1), dev(2)
    loss, correct = rt.eval_loss(obs, target, None)
    x, _ = rt.embed(obs[0])
    unit, hit = rt.projection_loss(x, target[0])
    assert torch.equal(unit, loss[0]) and torch.equal(hit, correct[0].bool())
    rt.close()
