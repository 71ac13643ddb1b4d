"""Prompts at the row counts where the pair GEMM changes its tiles, its ring or the number of pieces K is cut into: 33 rows
(the first it takes), whole and ragged 32-row chunks, tile heights on both sides of 128, one row more than a 256-row tile,
and sequences that end inside a chunk.  Logits of every position against the CPU oracle, with the path's bf16 bar (max |delta|
/ max |ref| <= 2e-2: operands rounded to 8 bits through two layers)."""
import numpy as np
import pytest

from oracle import gptj_oracle as go
from oracle import spec

pytestmark = pytest.mark.gpu

SEQ = 520


@pytest.fixture(scope="module")
def model(cuda_device):
    import torch
    torch.cuda.set_device(cuda_device)
    from mesh_transformer._runtime import ShardRuntime
    cfg = dict(spec.tiny_config(1, seq=SEQ), d_model=512, n_heads=2, pe_rotary_dims=64)
    params = spec.make_params(cfg, seed=9, stress=True)
    rt = ShardRuntime(cfg, max_batch=3, max_gen=1, max_rows=3 * SEQ)
    rt.load_params(params)
    yield cfg, params, rt
    rt.close()


@pytest.mark.parametrize("batch,T", [(1, 33), (1, 64), (1, 65), (1, 128), (1, 129), (1, 256), (1, 257), (1, 513), (3, 21), (3, 43),
                                     (2, 150), (3, 333)])
def test_prompt_logits(model, cuda_device, batch, T):
    import torch
    cfg, params, rt = model
    ids = spec.token_ids(31 + T, batch, T, cfg["n_vocab"])
    out = rt.forward_logits(torch.from_numpy(ids.view(np.int32)).to(cuda_device), None, T).cpu().numpy()
    rt.check_device_status()
    shard = go.CausalTransformerShard(cfg, params)
    for b in range(batch):
        ref = shard.logits(ids[b])
        assert np.abs(out[b] - ref).max() <= 2e-2 * np.abs(ref).max()
