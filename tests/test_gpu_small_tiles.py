"""Tensor-core products of up to 16 rows (tiles of 16) and of one row more: whole K, K over clusters, rows of weights and of K that fill
no tile; and decode steps of 15 to 17 sequences, whose activations are pairs of bf16 operands."""
import numpy as np
import pytest

from kernel_util import ptr
from oracle import gptj_oracle as go
from oracle import spec
from tests.test_gpu_model import LOGIT_TOL, _net, _wide_head_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(132, 64), (2048, 512), (6300, 4096), (200, 6144)])
@pytest.mark.parametrize("M", [1, 8, 15, 16, 17])
def test_product(cuda_device, M, N, K):
    """Products of bf16 are exact in fp32, so only the K sums round: each by at most 2^-23 (the unit truncates) of what is summed."""
    import torch
    from mesh_transformer._lib import check, lib
    g = torch.Generator(device=cuda_device)
    g.manual_seed(M * 7 + N)
    w = torch.randn((N, K), generator=g, device=cuda_device).to(torch.bfloat16)
    x = torch.randn((M, K), generator=g, device=cuda_device).to(torch.bfloat16)
    bias = torch.randn((N,), generator=g, device=cuda_device)
    out = torch.full((M, N), float("nan"), device=cuda_device)
    check(lib.mtj_k_gemm_tc(ptr(w), ptr(x), ptr(bias), M, N, K, ptr(out), torch.cuda.current_stream().cuda_stream))
    want = x.double() @ w.double().T + bias.double()
    bound = (x.double().abs() @ w.double().abs().T + bias.double().abs()) * (K + 1) * 2.0 ** -23
    assert bool(((out.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("batch", [15, 16, 17])
def test_decode_steps(cuda_device, batch):
    cfg = _wide_head_config(64)
    params = spec.make_params(cfg, seed=6)
    lens = np.array([1 + 4 * b % 64 for b in range(batch)], np.uint32)
    ctx = np.zeros((batch, 64), np.uint32)
    for b in range(batch):
        ctx[b, 64 - lens[b]:] = spec.token_ids(b, 1, int(lens[b]), cfg["n_vocab"])[0]
    net = _net(cfg, params, cuda_device)
    _, got = net.generate(ctx, lens, 4, {"top_p": np.zeros(batch), "temp": np.ones(batch)}, return_logits=True)
    _, ref = go.CausalTransformer(cfg, params).generate(ctx, lens, 4, return_logits=True)
    top = np.abs(ref[2]).max()
    for b in range(batch):
        for t in range(4):
            mine, want = got[2][b, t, 0], ref[2][b, t, 0]
            err = np.abs(mine - want).max()
            assert err <= LOGIT_TOL * top, (b, t)
            if got[0][b, t, 0] != ref[0][b, t, 0]:                  # only where the two best are as close as the logits are exact
                assert want.max() - want[got[0][b, t, 0]] <= 2 * err, (b, t)
                break
    net._rt.check_device_status()
    net.close()
