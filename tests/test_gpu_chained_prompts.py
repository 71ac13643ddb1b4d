"""Kernels of a pass that are launched programmatically behind one another give the same bits as kernels that start when the one
before them has ended: prompts of every form of the products, several chunks, evaluation, decoding, both families of stacks."""
import numpy as np
import pytest

from oracle import spec
from tests import stack_util as su
from tests.test_gpu_model import _net, _wide_head_config

pytestmark = pytest.mark.gpu


def _both(monkeypatch, make):
    out = []
    for off in ("1", "0"):
        monkeypatch.setenv("MTJ_NO_PDL", off)
        out.append(make())
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("rows", [20, 50, 150, 320])
def test_gptj_prompts(cuda_device, monkeypatch, rows):
    cfg = _wide_head_config(320)
    params = spec.make_params(cfg, seed=3)
    ctx = np.zeros((2, 320), np.uint32)
    lens = np.array([rows, max(1, rows // 2)], np.uint32)
    for b in range(2):
        ctx[b, 320 - lens[b]:] = spec.token_ids(b, 1, int(lens[b]), cfg["n_vocab"])[0]

    def make():
        net = _net(cfg, params, cuda_device)
        _, (toks, _, logits) = net.generate(ctx, lens, 6, {"top_p": np.zeros(2), "temp": np.ones(2)}, return_logits=True)
        ev = net.eval({"obs": ctx[:, :200], "target": ctx[:, 1:201], "ctx_length": np.array([200, 90])})
        net.close()
        return toks, logits, ev["all_loss"]
    _both(monkeypatch, make)


@pytest.mark.parametrize("path", ["f32", "few_rows", "many_rows"])
@pytest.mark.parametrize("family", ["keselix", "bavutar"])
def test_stack_prompts(cuda_device, monkeypatch, family, path):
    if family == "keselix":
        cfg = su.model([su.ssm(ff=44), su.attn(heads=4, dim=96, rot=32, vdim=128, rank=64, window=150, ff=256)], width=256, vocab=131)
    else:
        cfg = su.bavutar([su.delta(), su.gqa(heads=4, dim=128, vdim=128), su.ssd()], width=256)
    w = su.weights(cfg, 7)
    toks = su.ids(4, 300, cfg["vocab"])

    def make():
        rt = su.runtime(cfg, w, path, seq=300, max_rows=128)                 # chunks of 128 rows and a rest
        rt.start_batch(1)
        got = [su.extend(rt, 0, toks)]
        rt.release(0)
        at = 0
        for n in (1, 40, 1, 90, 3):
            got.append(su.extend(rt, 0, toks[at:at + n]))
            at += n
        rt.check_device_status()
        rt.close()
        return got
    _both(monkeypatch, make)


@pytest.mark.parametrize("model", ["gptj", "keselix", "bavutar"])
def test_chained_passes_repeat(cuda_device, monkeypatch, model):
    """A kernel that runs ahead of what it needs does so now and then: the calls above forty times, chained, against one that is not."""
    if model == "gptj":
        cfg = _wide_head_config(320)
        params = spec.make_params(cfg, seed=3)
        ctx = spec.token_ids(7, 2, 320, cfg["n_vocab"])
        lens = np.array([320, 150], np.uint32)

        def calls():
            net = _net(cfg, params, cuda_device)
            while True:
                _, (toks, _, logits) = net.generate(ctx, lens, 6, {"top_p": np.zeros(2), "temp": np.ones(2)}, return_logits=True)
                yield toks, logits, net.eval({"obs": ctx[:, :200], "target": ctx[:, 1:201], "ctx_length": np.array([200, 90])})["all_loss"]
    else:
        cfg = (su.model([su.ssm(ff=44), su.attn(heads=4, dim=96, rot=32, vdim=128, rank=64, window=150, ff=256)], width=256, vocab=131) if model == "keselix"
               else su.bavutar([su.delta(heads=16, kv_heads=16, dim=64, vdim=64), su.gqa(heads=4, dim=128, vdim=128), su.ssd(heads=16, vdim=32, state=64, groups=2)], width=256))
        w = su.weights(cfg, 7)
        toks = su.ids(4, 500, cfg["vocab"])

        def calls():
            rt = su.runtime(cfg, w, "many_rows", seq=500, max_rows=500)
            rt.start_batch(1)
            while True:
                at, got = 0, []
                for n in (300, 1, 40, 1, 90, 3):
                    got.append(su.extend(rt, 0, toks[at:at + n]))
                    at += n
                rt.check_device_status()
                rt.release(0)
                yield got
    monkeypatch.setenv("MTJ_NO_PDL", "1")
    want = next(calls())
    monkeypatch.setenv("MTJ_NO_PDL", "0")
    for _, got in zip(range(40), calls()):
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
