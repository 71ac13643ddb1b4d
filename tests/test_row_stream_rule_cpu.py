"""Which products of one row are streamed: the rule says no wherever the launch would, so that such a product takes the other kernel."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mesh-transformer-jax_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include "mtj_kernels.h"
int main() {
  int n, k, ldx;
  while (scanf("%d %d %d", &n, &k, &ldx) == 3) {
    mtj::GemvArgs a = {};
    a.M = 1; a.N = n; a.K = k; a.ldx = ldx;
    printf("%d%d%d%d\\n", mtj::gemv_stream_ok(mtj::kEpiOut, a), mtj::gemv_stream_ok(mtj::kEpiSoftcap, a),
           mtj::gemv_stream_ok(mtj::kEpiSwiGLU, a), mtj::gemv_stream_ok(mtj::kEpiRelu2, a));
  }
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    import __graft_entry__ as ge
    ge.build()
    build = ge._load_build_module()
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(PROGRAM)
    lib = build.library()
    subprocess.run([build.NVCC, "-std=c++17", "-I", CSRC, str(d / "rule.cpp"), lib, "-o", str(d / "rule"), "-Xlinker", "-rpath=" + os.path.dirname(lib)], check=True)

    def ask(sizes):
        out = subprocess.run([str(d / "rule")], input="\n".join("%d %d %d" % s for s in sizes), text=True, check=True, capture_output=True).stdout.split()
        return dict(zip(sizes, out))
    return ask


def test_only_what_the_kernel_takes(rule):
    yes = [(32768, 4096, 4096), (4096, 16384, 16384), (12304, 1024, 1024), (3072, 4104, 4108), (592, 8192, 8192), (600, 16384, 16384)]
    no = [(n + dn, k + dk, ldx + dx) for n, k, ldx in yes for dn, dk, dx in ((1, 0, 0), (0, 4, 0), (0, 1, 0), (0, 0, 2), (0, 0, 1))]
    got = rule(yes + no + [(2048, 4096, 4096), (65536, 1016, 1016), (4096, 16392, 16392), (588, 8192, 8192), (592, 8184, 8184)])
    assert all(got[s] == ("1111" if s in yes else "0000") for s in got), got
