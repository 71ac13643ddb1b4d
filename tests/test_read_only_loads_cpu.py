"""Read-only loads (ld.global.nc, which the compiler also makes of const __restrict__ kernel parameters) are for data that nobody
writes while the kernel is there.  Cached keys and values are written by other blocks of a whole-step kernel, and whatever comes from
the kernel before it by the predecessor of a chained launch, which is still running when the kernel starts."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mesh-transformer-jax_b200", "csrc")
# written before the pass that the kernel belongs to: norms' weights, biases, the sampler's key and uniforms
CONSTANT = {"scale", "offset", "bias", "seed", "u"}


def _sources():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                yield name, f.read()


def test_cached_rows_are_read_by_coherent_loads():
    for name, text in _sources():
        for call in re.findall(r"\bld_stream\w*\(([^;]*);", text):
            assert not re.search(r"[kv]pool", call), (name, call)
        if name == "mtj_attn.cu":
            assert "ld_stream" not in text, "everything this file loads is a cached row or a predecessor's"


def test_chained_kernels_do_not_promise_that_their_inputs_rest():
    seen = 0
    for name, text in _sources():
        for m in re.finditer(r"__global__ void[^;{]*?(\w+_kernel)\(([^{;]*)\)\s*\{", text):
            body = text[m.end():text.find("\n}\n", m.end())]
            if "pdl_wait()" not in body:
                continue
            seen += 1
            promised = set(re.findall(r"const \w+\* __restrict__ (\w+)", m.group(2)))
            assert promised <= CONSTANT, (name, m.group(1), promised - CONSTANT)
    assert seen > 20
