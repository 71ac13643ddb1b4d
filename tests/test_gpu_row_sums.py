"""The kernels that finish residual rows: what a row becomes does not depend on how many rows a call has, to the bit.  Calls of up to
148 rows take 512 threads a row, more rows 256; all of them add in one order.  (More than 512 rows of up to 1024 columns behind a
layer norm are summed in shared memory, in an order of their own.)"""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mesh-transformer-jax_b200", "csrc")
PROGRAM = r"""
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <vector>
#include "mtj_stack_kernels.h"
using Floats = std::vector<float>;
constexpr int kSame = 120;
// the number at column c of row r depends on nothing else; columns d .. ld - 1 are zero
static float at(uint32_t salt, uint32_t r, uint32_t c) {
  uint32_t h = (salt * 2654435761u) ^ (r * 40503u + c * 2246822519u + 374761393u);
  h ^= h >> 15; h *= 2246822519u; h ^= h >> 13; h *= 3266489917u; h ^= h >> 16;
  return static_cast<int32_t>(h) * (1.f / 2147483648.f) + 0.125f;
}
static float* up(const Floats& v) {
  float* p = nullptr;
  cudaMalloc(&p, v.size() * 4);
  cudaMemcpy(p, v.data(), v.size() * 4, cudaMemcpyHostToDevice);
  return p;
}
static Floats rows(uint32_t salt, int M, int d, int ld) {
  Floats v(static_cast<size_t>(M) * ld, 0.f);
  for (int r = 0; r < M; ++r)
    for (int c = 0; c < d; ++c) v[static_cast<size_t>(r) * ld + c] = at(salt, r, c);
  return v;
}
// the first kSame rows of x, of xn and of xn_f32 as bytes
static std::vector<char> run(bool layer, int M, int d, int ld, int planes) {
  Floats y;
  for (int p = 0; p < planes; ++p) {
    const Floats one = rows(10 + p, M, d, ld);
    y.insert(y.end(), one.begin(), one.end());
  }
  float *x = up(rows(1, M, d, ld)), *dy = up(y), *w = up(rows(2, 1, d, ld)), *b = up(rows(3, 1, d, ld)), *wn = up(rows(4, 1, d, ld)), *bn = up(rows(5, 1, d, ld));
  float* xf = up(Floats(static_cast<size_t>(M) * ld, 0.f));
  __nv_bfloat16* xn = nullptr;
  cudaMalloc(&xn, static_cast<size_t>(M) * ld * 2);
  cudaError_t e;
  if (layer) {
    mtj::ResidualLayerNormArgs a = {};
    a.x = x; a.M = M; a.d = d; a.ld = ld; a.y = dy; a.planes = planes; a.w = w; a.b = b; a.alpha = 1.5f; a.eps = 1e-5f;
    a.w_next = wn; a.b_next = bn; a.xn = xn; a.xn_f32 = xf;
    e = mtj::launch_residual_layernorm(a, nullptr, false);
  } else {
    mtj::ResidualNormArgs a = {};
    a.x = x; a.M = M; a.d = d; a.ld = ld; a.y = dy; a.planes = planes; a.w_post = w; a.mult = 0.5f; a.eps = 1e-5f;
    a.w_next = wn; a.xn = xn; a.xn_f32 = xf;
    e = mtj::launch_residual_norm(a, nullptr, false);
  }
  const size_t n = static_cast<size_t>(kSame) * ld;
  std::vector<char> out(n * 10);
  cudaMemcpy(out.data(), x, n * 4, cudaMemcpyDeviceToHost);
  cudaMemcpy(out.data() + n * 4, xf, n * 4, cudaMemcpyDeviceToHost);
  const cudaError_t e2 = cudaMemcpy(out.data() + n * 8, xn, n * 2, cudaMemcpyDeviceToHost);
  for (void* p : {static_cast<void*>(x), static_cast<void*>(dy), static_cast<void*>(w), static_cast<void*>(b), static_cast<void*>(wn), static_cast<void*>(bn),
                  static_cast<void*>(xf), static_cast<void*>(xn)}) cudaFree(p);
  if (e != cudaSuccess || e2 != cudaSuccess) out.clear();
  return out;
}
int main() {
  int layer, d, ld, planes;
  while (scanf("%d %d %d %d", &layer, &d, &ld, &planes) == 4) {
    const std::vector<char> few = run(layer, kSame, d, ld, planes);
    int same = !few.empty();
    for (int M : {148, 149, layer && ld <= 1024 ? 512 : 600}) same &= run(layer, M, d, ld, planes) == few;
    printf("%d\n", same);
  }
}
"""


@pytest.fixture(scope="module")
def same(cuda_device, tmp_path_factory):
    import __graft_entry__ as ge
    build = ge._load_build_module()
    d = tmp_path_factory.mktemp("rows")
    (d / "rows.cu").write_text(PROGRAM)
    lib = build.build()
    subprocess.run([build.NVCC, *build.FLAGS, "-I", CSRC, str(d / "rows.cu"), lib, "-o", str(d / "rows"), "-Xlinker", "-rpath=" + os.path.dirname(lib)], check=True)

    def ask(sizes):
        out = subprocess.run([str(d / "rows")], input="\n".join("%d %d %d %d" % s for s in sizes), text=True, check=True, capture_output=True).stdout.split()
        return dict(zip(sizes, out))
    return ask


def test_few_rows_and_many(same):
    sizes = [(layer, d, (d + 7) // 8 * 8, planes) for layer in (0, 1) for d in (69, 600, 1024, 2048, 2053, 4096, 4104, 8191) for planes in (1, 5, 8)]
    got = same(sizes)
    assert len(got) == len(sizes) and all(v == "1" for v in got.values()), got
