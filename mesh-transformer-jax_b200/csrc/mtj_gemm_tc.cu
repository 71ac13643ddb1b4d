// Tensor-core GEMM: host side (tensor maps, launch selection) and the two small kernels around it.  The GEMM kernels
// are in mtj_gemm_tc.cuh, their instances in mtj_gemm_tc_gptj.cu and mtj_gemm_tc_stack.cu.
#include "mtj_gemm_tc.cuh"

namespace mtj {
namespace {

template <int THREADS>
__device__ __forceinline__ float row_sum(float v, float* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  v = warp_sum(v);
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < THREADS / 32; ++i) t += red[i];
  __syncthreads();
  return t;
}

// LayerNorm of fp32 rows into bf16 (the GEMM's activation operand: hi, and lo where asked for), layers.py:17-36.  HOLD > 0:
// rows of up to 256 HOLD columns stay in registers, one read of the row with all loads in flight instead of three, and the
// weights before it; 0: wider rows, three reads.  Both add in the same order.  Few rows are bound by the loads' latency (33 of
// 4096: 5.2 us in three reads, 3.0 from registers; 33 of 1024: 2.7 and 2.2), many by how many blocks an SM holds.  (The predecessor
// of a chained launch writes x while this kernel is there: not __restrict__, which would let its loads be read-only ones.)
template <int HOLD>
__global__ void __launch_bounds__(256) ln_rows_kernel(const float* x, const float* __restrict__ scale,
                                                      const float* __restrict__ offset,
                                                      __nv_bfloat16* __restrict__ out, __nv_bfloat16* out_lo, int d) {
  __shared__ float red[8];
  float sc[HOLD > 0 ? HOLD : 1], of[HOLD > 0 ? HOLD : 1];
  if constexpr (HOLD > 0) {                              // weights do not depend on the predecessor
#pragma unroll
    for (int k = 0; k < HOLD; ++k) {
      const int i = k * 256 + static_cast<int>(threadIdx.x);
      sc[k] = i < d ? scale[i] : 0.f;
      of[k] = i < d ? offset[i] : 0.f;
    }
  }
  pdl_wait();
  pdl_launch_dependents();
  const float* xr = x + static_cast<size_t>(blockIdx.x) * d;
  __nv_bfloat16* o = out + static_cast<size_t>(blockIdx.x) * d;
  __nv_bfloat16* ol = out_lo ? out_lo + static_cast<size_t>(blockIdx.x) * d : nullptr;
  auto put = [&](int i, float xi, float mu, float rstd, float w, float b) {
    const float y = fmaf(w * rstd, xi - mu, b);
    const __nv_bfloat16 hi = __float2bfloat16_rn(y);
    o[i] = hi;
    if (ol) ol[i] = __float2bfloat16_rn(y - __bfloat162float(hi));
  };
  float s = 0.f, v = 0.f;
  if constexpr (HOLD > 0) {
    float r[HOLD];
#pragma unroll
    for (int k = 0; k < HOLD; ++k) r[k] = k * 256 + static_cast<int>(threadIdx.x) < d ? xr[k * 256 + threadIdx.x] : 0.f;
#pragma unroll
    for (int k = 0; k < HOLD; ++k) s += r[k];
    const float mu = row_sum<256>(s, red) / static_cast<float>(d);
#pragma unroll
    for (int k = 0; k < HOLD; ++k) {
      const float t = k * 256 + static_cast<int>(threadIdx.x) < d ? r[k] - mu : 0.f;
      v = fmaf(t, t, v);
    }
    const float rstd = 1.0f / sqrtf(row_sum<256>(v, red) / static_cast<float>(d) + 1e-5f);
#pragma unroll
    for (int k = 0; k < HOLD; ++k)
      if (k * 256 + static_cast<int>(threadIdx.x) < d) put(k * 256 + threadIdx.x, r[k], mu, rstd, sc[k], of[k]);
  } else {
    for (int i = threadIdx.x; i < d; i += 256) s += xr[i];
    const float mu = row_sum<256>(s, red) / static_cast<float>(d);
    for (int i = threadIdx.x; i < d; i += 256) {
      const float t = xr[i] - mu;
      v = fmaf(t, t, v);
    }
    const float rstd = 1.0f / sqrtf(row_sum<256>(v, red) / static_cast<float>(d) + 1e-5f);
    for (int i = threadIdx.x; i < d; i += 256) put(i, xr[i], mu, rstd, scale[i], offset[i]);
  }
}

// x = sum of split-K planes (in order) + bias + residual, and from the finished row the next projection's operand, the
// layer norm in bf16 (hi, and lo where asked for).  One block per row, the row in registers (HOLD float4 a thread), every
// load issued before the first sum.  The planes are in L2; bound by the latency of one round of loads and two block sums
// up to about 300 rows, by L2 above; the weights come before the wait.  It replaces two kernels: 56 rows of 4096 in 4
// planes 5.4 us against 5.1 + 4.4, 700 rows in 3 planes 14 us against 35 + 6, 8 rows in 8 planes 5.1 us against 2.4 + 4.6.
constexpr int kRowThreads = 512;
template <int HOLD>
__global__ void __launch_bounds__(kRowThreads) reduce_ln_rows_kernel(const ReduceLnArgs a) {
  __shared__ float red[kRowThreads / 32];
  const int n4 = a.d >> 2;
  auto weights = [&](const float* w, float4 (&v)[HOLD]) {
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int c = i * kRowThreads + threadIdx.x;
      v[i] = w && c < n4 ? reinterpret_cast<const float4*>(w)[c] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  float4 b[HOLD], sc[HOLD], of[HOLD];                    // they do not depend on the predecessor
  weights(a.bias, b);
  weights(a.scale, sc);
  weights(a.offset, of);
  pdl_wait();
  pdl_launch_dependents();
  const size_t row4 = static_cast<size_t>(blockIdx.x) * n4, plane4 = static_cast<size_t>(a.M) * n4;
  const float4* res = reinterpret_cast<const float4*>(a.residual) + row4;
  const float4* part = reinterpret_cast<const float4*>(a.partial) + row4;
  float4 v[HOLD], r[HOLD];
  float s = 0.f;
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    const int c = i * kRowThreads + threadIdx.x;
    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    r[i] = c < n4 ? res[c] : v[i];
  }
#pragma unroll (HOLD > 2 ? 4 : 8)
  for (int z = 0; z < a.planes; ++z) {
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int c = i * kRowThreads + threadIdx.x;
      const float4 p = c < n4 ? __ldcg(part + z * plane4 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[i].x += p.x; v[i].y += p.y; v[i].z += p.z; v[i].w += p.w;
    }
  }
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    const int c = i * kRowThreads + threadIdx.x;
    if (c >= n4) continue;
    v[i].x = v[i].x + b[i].x + r[i].x; v[i].y = v[i].y + b[i].y + r[i].y; v[i].z = v[i].z + b[i].z + r[i].z; v[i].w = v[i].w + b[i].w + r[i].w;
    reinterpret_cast<float4*>(a.out)[row4 + c] = v[i];
  }
  if (!a.scale) return;
#pragma unroll
  for (int i = 0; i < HOLD; ++i) s += (v[i].x + v[i].y) + (v[i].z + v[i].w);      // columns past the row are zero
  const float mu = row_sum<kRowThreads>(s, red) / static_cast<float>(a.d);
  float q = 0.f;
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    if (i * kRowThreads + static_cast<int>(threadIdx.x) >= n4) continue;
    const float x = v[i].x - mu, y = v[i].y - mu, z = v[i].z - mu, w = v[i].w - mu;
    q += (x * x + y * y) + (z * z + w * w);
  }
  const float rstd = 1.0f / sqrtf(row_sum<kRowThreads>(q, red) / static_cast<float>(a.d) + 1e-5f);
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    const int c = i * kRowThreads + threadIdx.x;
    if (c >= n4) continue;
    const float y[4] = {fmaf(sc[i].x * rstd, v[i].x - mu, of[i].x), fmaf(sc[i].y * rstd, v[i].y - mu, of[i].y),
                        fmaf(sc[i].z * rstd, v[i].z - mu, of[i].z), fmaf(sc[i].w * rstd, v[i].w - mu, of[i].w)};
    reinterpret_cast<uint2*>(a.xn)[row4 + c] = make_uint2(pack_bf16x2(y[0], y[1]), pack_bf16x2(y[2], y[3]));
    if (a.xn_lo) {
      float e[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) e[k] = y[k] - __bfloat162float(__float2bfloat16_rn(y[k]));
      reinterpret_cast<uint2*>(a.xn_lo)[row4 + c] = make_uint2(pack_bf16x2(e[0], e[1]), pack_bf16x2(e[2], e[3]));
    }
  }
}

int sm_count() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return n;
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  return fn;
}

}  // namespace

int gemm_tc_token_tile() { return 128; }
// Batched decode streams each weight tile once, and a block keeps only its TMA ring in flight: with fewer tiles
// than the GPU holds blocks (two per SM), K is split over a cluster of 2 or 4 blocks per tile so that the
// bytes in flight -- and with them the HBM rate -- do not fall with the tile count (tensor-parallel slices).
int gemm_tc_decode_cluster_k(int weight_rows, int M, int K) {
  if (M > 64) return 1;
  const int tiles = (weight_rows + kBM - 1) / kBM;      // one token tile
  int ck = 1;
  while (ck < 4 && tiles * ck * 2 <= 296 && K / kBK >= ck * 2 * 2) ck *= 2;
  return ck;
}

int gemm_tc_token_tile_for(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : (M <= 64 ? 64 : 128); }
// Rows from which the pair kernel takes over: above 192 always, and from 33 on where a prompt is read (not `same_sums`:
// decoding, whose kernels are chained, and evaluation, whose sums keep their order).  GPT-J-6B's two projections, us a layer:
// 56 rows 126 with the small tiles and 87 with it, 136 rows 356 and 98.
bool gemm_tc_use_wide(int M, bool same_sums) { return M > (same_sums ? 192 : 32); }
// Pieces that K is cut into, each leaving a plane of partial sums: as many as shorten the critical path by more than
// writing and adding the planes takes.  One unit is a k-block of 64, about 0.36 us: where few pairs run the round trip of the
// 192 KB of operands that a pair keeps in flight, where all run with 256-row tiles the tensor pipe (1.72 PFLOP/s); a number of a plane costs 1 ps to write and add
// where the following kernel adds the planes, and 4 ps with a kernel for it (own_sum).  4096 x
// 20480 weights: 136 rows 104 us whole, 37 us in 4 pieces; 448 rows 110 and 58 in 2; 700 rows 114 and 78 in 3; from 998
// rows on whole tiles are best.
int gemm_tc_wide_split(int M, int N, int K, bool own_sum, double least_us) {
  if (N < 2 * kBM) return 1;                           // the pair kernel's tile
  const int tiles = (M + kPBN - 1) / kPBN * ((N + 2 * kBM - 1) / (2 * kBM)), pairs = std::max(1, sm_count() / 2), nk = (K + kBK - 1) / kBK;
  int best = 1;
  double whole = 0.0, best_cost = 1e30;
  for (int s = 1; s <= 8 && (s == 1 || nk / s >= 8); ++s) {
    if ((s - 1) * ((nk + s - 1) / s) >= nk || (s > 1 && static_cast<int64_t>(s) * M * N > kWidePlaneFloats)) continue;
    const int waves = (tiles * s + pairs - 1) / pairs;
    const double planes = s > 1 ? (own_sum ? 4e-6 : 1e-6) * s * M * N / 0.36 : 0.0;
    const double cost = static_cast<double>(waves) * ((nk + s - 1) / s) + planes;
    if (s == 1) whole = cost;
    if (cost < 0.97 * best_cost && (s == 1 || 0.36 * (whole - cost) >= least_us)) {
      best = s;
      best_cost = cost;
    }
  }
  return best;
}
int64_t gemm_tc_wide_plane_floats(int max_rows, int N, int K, bool own_sum, double least_us) {
  int64_t most = 0;
  for (int M = 33; M <= max_rows && 2LL * M * N <= kWidePlaneFloats; ++M) {
    const int s = gemm_tc_wide_split(M, N, K, own_sum, least_us);
    if (s > 1) most = std::max(most, static_cast<int64_t>(s) * M * N);
  }
  return most;
}
int gemm_tc_wide_token_tile() { return kPBN / 2; }     // rows of the activation box: a tile takes two of them

cudaError_t launch_gemm_tc_wide(GemvEpilogue epi, const void* map_w, const void* map_x, const void* map_x64, const GemmTcArgs& a,
                                cudaStream_t s) {
  if (a.M <= 0 || a.N <= 0 || a.K <= 0) return cudaErrorInvalidValue;
  const CUtensorMap& mw = *static_cast<const CUtensorMap*>(map_w);
  const CUtensorMap& mx = *static_cast<const CUtensorMap*>(map_x);
  const CUtensorMap* m64 = static_cast<const CUtensorMap*>(map_x64);
  if (epi == kEpiPlain || epi == kEpiSwiGLU) return launch_gemm_tc_stack(epi, true, mw, mx, m64, a, s, false);
  if (epi == kEpiRelu2 || epi == kEpiSoftcap) return launch_gemm_tc_stack_post(epi, true, mw, mx, m64, a, s, false);
  return launch_gemm_tc_gptj(epi, true, mw, mx, m64, a, s, false);
}

cudaError_t make_tensor_map_bf16(void* map_out, const void* base, int64_t rows, int64_t K, int box_rows, int64_t ld) {
  if (ld <= 0) ld = K;
  PFN_cuTensorMapEncodeTiled_v12000 fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || (ld * 2) % 16 || ld < K || box_rows > 256) return cudaErrorInvalidValue;
  cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
  cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(kBK), static_cast<cuuint32_t>(box_rows)};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(static_cast<CUtensorMap*>(map_out), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
                  dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

cudaError_t launch_gemm_tc(GemvEpilogue epi, const void* map_w, const void* map_x, const GemmTcArgs& a,
                           cudaStream_t s, bool pdl, const void* map_x_lo) {
  if (a.M <= 0 || a.N <= 0 || a.K <= 0) return cudaErrorInvalidValue;
  const CUtensorMap& mw = *static_cast<const CUtensorMap*>(map_w);
  const CUtensorMap& mx = *static_cast<const CUtensorMap*>(map_x);
  if (epi == kEpiPlain || epi == kEpiSwiGLU)
    return map_x_lo ? cudaErrorInvalidValue : launch_gemm_tc_stack(epi, false, mw, mx, nullptr, a, s, pdl);
  if (epi == kEpiRelu2 || epi == kEpiSoftcap)
    return map_x_lo ? cudaErrorInvalidValue : launch_gemm_tc_stack_post(epi, false, mw, mx, nullptr, a, s, pdl);
  return launch_gemm_tc_gptj(epi, false, mw, mx, static_cast<const CUtensorMap*>(map_x_lo), a, s, pdl);
}

namespace {
// out[m, n] = sum_z partial[z, m, n] + bias[n] (+ residual[m, n]); fixed summation order
__global__ void splitk_reduce_kernel(const float* partial, int ksplit, int M, int N,
                                     const float* __restrict__ bias, const float* residual, float* out, int ld_out,
                                     const uint32_t* slot_sel, size_t slot_stride) {
  const size_t total = static_cast<size_t>(M) * N;
  pdl_wait();                      // the partial sums come from the predecessor kernel
  pdl_launch_dependents();
  if (slot_sel) out += static_cast<size_t>(*slot_sel & 1u) * slot_stride;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int n = static_cast<int>(i % N);
    const size_t m = i / N;
    float acc = 0.f;
    for (int z = 0; z < ksplit; ++z) acc += partial[static_cast<size_t>(z) * total + i];
    if (bias) acc += bias[n];
    if (residual) acc += residual[i];
    out[m * ld_out + n] = acc;
  }
}
}  // namespace

cudaError_t launch_splitk_reduce(const float* partial, int ksplit, int M, int N, const float* bias,
                                 const float* residual, float* out, int ld_out, const uint32_t* slot_sel,
                                 size_t slot_stride, cudaStream_t s, bool pdl) {
  const size_t total = static_cast<size_t>(M) * N;
  const int grid = static_cast<int>(std::min<size_t>((total + 255) / 256, 148 * 8));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(256);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, splitk_reduce_kernel, partial, ksplit, M, N, bias, residual, out, ld_out, slot_sel,
                            slot_stride);
}

bool reduce_ln_rows_ok(int d) { return (d & 3) == 0 && d <= 4 * 4 * kRowThreads; }

cudaError_t launch_reduce_ln_rows(const ReduceLnArgs& a, cudaStream_t s, bool pdl) {
  if (a.M <= 0 || !reduce_ln_rows_ok(a.d) || a.planes < 1 || !a.partial || !a.bias || !a.residual || !a.out || (a.scale && (!a.offset || !a.xn)))
    return cudaErrorInvalidValue;
  const dim3 grid(a.M), block(kRowThreads);
  if (a.d <= 4 * kRowThreads) return launch_pdl(reduce_ln_rows_kernel<1>, grid, block, 0, s, pdl, a);
  if (a.d <= 2 * 4 * kRowThreads) return launch_pdl(reduce_ln_rows_kernel<2>, grid, block, 0, s, pdl, a);
  return launch_pdl(reduce_ln_rows_kernel<4>, grid, block, 0, s, pdl, a);
}

cudaError_t launch_ln_rows(const float* x, const float* scale, const float* offset, __nv_bfloat16* out, int rows,
                           int d, cudaStream_t s, bool pdl, __nv_bfloat16* out_lo) {
  const dim3 grid(rows), block(256);
  if (d <= 1024) return launch_pdl(ln_rows_kernel<4>, grid, block, 0, s, pdl, x, scale, offset, out, out_lo, d);
  if (d <= 2048) return launch_pdl(ln_rows_kernel<8>, grid, block, 0, s, pdl, x, scale, offset, out, out_lo, d);
  // wide rows take the registers of more than one block in two: 512 rows of 4096 6.3 us in three reads and 5.3, 1000 7.5 and 8.7
  const bool few = rows <= 512;
  if (few && d <= 4096) return launch_pdl(ln_rows_kernel<16>, grid, block, 0, s, pdl, x, scale, offset, out, out_lo, d);
  if (few && d <= 8192) return launch_pdl(ln_rows_kernel<32>, grid, block, 0, s, pdl, x, scale, offset, out, out_lo, d);
  return launch_pdl(ln_rows_kernel<0>, grid, block, 0, s, pdl, x, scale, offset, out, out_lo, d);
}

}  // namespace mtj
