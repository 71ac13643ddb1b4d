"""The decode step of one sequence whose weights are streamed by a warp of their own: row and column remainders of its rings, heads
of 64 and of 256, contexts around its key ranges, evicted keys, against the oracle and the kernel that loads where it computes.

Both kernels sum in fp32 in different orders; where that turns the bf16 rounding of a cached key or value, one entry moves by at most
2^-8 of itself, and no logit by more than 2^-8 of the largest."""
import numpy as np
import pytest

from oracle import gptj_oracle as go
from oracle import spec
from tests.test_gpu_model import LOGIT_TOL, _net, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,heads,vocab", [(1024, 4, 516), (1024, 16, 50400), (1280, 5, 1004), (2304, 36, 512), (3840, 15, 776)])
def test_one_sequence(cuda_device, monkeypatch, d, heads, vocab):
    cfg = dict(spec.gptj6b_config(1), layers=2, d_model=d, n_heads=heads, n_vocab=vocab, seq=200, pe_rotary_dims=64)
    params = spec.make_params(cfg, seed=d + heads, stress=True)
    oracle = go.CausalTransformer(cfg, params)
    nets = [_net(cfg, params, cuda_device) for _ in range(2)]
    for n in (1, 14, 130, 200):
        ctx = np.zeros((1, 200), np.uint32)
        ctx[0, 200 - n:] = spec.token_ids(n, 1, n, vocab)[0]
        out = []
        for net, narrow in zip(nets, (False, True)):
            if narrow:
                monkeypatch.setenv("MTJ_MEGA_NARROW", "1")
            else:
                monkeypatch.delenv("MTJ_MEGA_NARROW", raising=False)
            _, got = net.generate(ctx, np.array([n], np.uint32), 5, {"top_p": np.zeros(1), "temp": np.ones(1)}, return_logits=True)
            net._rt.check_device_status()
            out.append(got)
        _, ref = oracle.generate(ctx, np.array([n], np.uint32), 5, return_logits=True)
        assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][0], ref[0])
        assert _rel(out[0][2], out[1][2]) <= 2.0 ** -8 and _rel(out[0][2], ref[2]) <= LOGIT_TOL
    for net in nets:
        net.close()


def test_sampled_ids_are_the_samplers_on_the_steps_logits(cuda_device):
    from mesh_transformer.sampling import nucleaus_sample
    from oracle import sampling_oracle as so
    cfg = dict(spec.gptj6b_config(1), layers=2, d_model=1024, n_heads=4, n_vocab=1004, seq=64, sampler=nucleaus_sample)
    net = _net(cfg, spec.make_params(cfg, seed=9, stress=True), cuda_device)
    ctx = spec.token_ids(2, 1, 64, 1004)
    un = np.random.default_rng(5).random((6, 1, 1004), dtype=np.float32).clip(so.TINY, None)
    opts = {"top_p": np.array([0.9]), "temp": np.array([0.8])}
    _, out = net.generate(ctx, np.array([64], np.uint32), 6, opts, return_logits=True, uniforms=un)
    for t in range(6):
        assert np.array_equal(out[0][:, t, 0], so.nucleaus_sample(un[t], out[2][:, t, 0], opts["top_p"].astype(np.float32), opts["temp"].astype(np.float32)))
    net.close()
