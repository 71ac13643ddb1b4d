"""Prompt attention on the CUDA cores (heads of 64 columns; prompts of fewer than 32 rows) at the edges of its steps: keys 32 at a
time, 64-token pages, one query per warp or, from 2368 (row, head) pairs on, four; a key limit.  Whole models against the plain
oracle, with the models' tolerance on logits (2e-2 of the largest)."""
import numpy as np
import pytest

from oracle import gptj_oracle as go
from oracle import spec
from tests.test_gpu_model import LOGIT_TOL, _net, _rel, _wide_head_config

pytestmark = pytest.mark.gpu


def _check(cfg, params, net, batch, T, lens=None):
    import torch
    ids = spec.token_ids(T, batch, T, cfg["n_vocab"])
    rt = net._runtime(batch, 1)
    out = rt.forward_logits(torch.from_numpy(ids.view(np.int32)).to(rt.device), lens, T).cpu().numpy()
    shard = go.CausalTransformerShard(cfg, params)
    for b in range(batch):
        mask = 0 if lens is None else (np.arange(T) > int(lens[b])) * -1e10
        assert _rel(out[b], shard.logits(ids[b], mask=mask)) <= LOGIT_TOL, (batch, T, b)


def test_heads_of_64_columns(cuda_device):
    cfg = spec.tiny_config(1, seq=130)
    params = spec.make_params(cfg, seed=1, stress=True)
    net = _net(cfg, params, cuda_device)
    for T in (1, 2, 31, 32, 33, 63, 64, 65, 97, 129):
        _check(cfg, params, net, 1, T)
    _check(cfg, params, net, 3, 70, np.array([70, 33, 5], np.uint32))
    _check(cfg, params, net, 9, 67)                                       # four queries per warp, the last warp three


def test_heads_of_256_columns_in_short_prompts(cuda_device):
    cfg = _wide_head_config(40)
    params = spec.make_params(cfg, seed=1)
    net = _net(cfg, params, cuda_device)
    for T in (1, 5, 17, 31):
        _check(cfg, params, net, 1, T)
