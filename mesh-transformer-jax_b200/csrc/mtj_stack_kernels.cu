// Row kernels of layer-stack models (residual + norms) and the repacking of their weights.
#include <math.h>

#include <algorithm>

#include "mtj_common.cuh"
#include "mtj_stack_kernels.h"

namespace mtj {
namespace {

constexpr int kRnThreads = 256;

__device__ __forceinline__ float rn_block_sum(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < kRnThreads / 32; ++i) t += red[i];
  __syncthreads();
  return t;
}
// The same of the row kernels' partial sums, one per float4 of a thread.  512 threads add in the order of 256, of which a thread has
// the numbers of threads t and t + 256 in turn: a row's bits do not depend on how many rows a call has.
template <int THREADS, int HOLD>
struct RowSum {
  float red[kRnThreads / 32], upper[THREADS == kRnThreads ? 1 : HOLD][kRnThreads];
  __device__ __forceinline__ float operator()(const float (&part)[HOLD]) {
    const int t = threadIdx.x;
    float v = 0.f;
    if constexpr (THREADS == kRnThreads) {
#pragma unroll
      for (int i = 0; i < HOLD; ++i) v += part[i];
      return rn_block_sum(v, red);
    }
    static_assert(THREADS == kRnThreads || THREADS == 2 * kRnThreads, "thread t adds the numbers of t + 256");
    if (t >= kRnThreads) {
#pragma unroll
      for (int i = 0; i < HOLD; ++i) upper[i][t - kRnThreads] = part[i];
    }
    __syncthreads();
    if (t < kRnThreads) {
#pragma unroll
      for (int i = 0; i < HOLD; ++i) {
        v += part[i];
        v += upper[i][t];
      }
      v = warp_sum(v);
      if ((t & 31) == 0) red[t >> 5] = v;
    }
    __syncthreads();                                         // `upper` is read; `red` is before the next sum's first barrier
    v = 0.f;
#pragma unroll
    for (int i = 0; i < kRnThreads / 32; ++i) v += red[i];
    return v;
  }
};

// Spelled out, because the compiler may fuse the sum of two products in either order and does so differently from one template to
// the next: a row's bits would depend on which of the row kernels finishes it.
__device__ __forceinline__ float dot4(const float4& a) { return fmaf(a.w, a.w, fmaf(a.z, a.z, fmaf(a.x, a.x, a.y * a.y))); }
__device__ __forceinline__ uint2 pack4(const float4& v) {
  return make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
}

// Columns from `left` on are padding and stay zero for good, whatever the row holds: a norm of a row that is not finite
// would make them NaN, and the embedding, which opens the next call, writes the columns that exist only.
__device__ __forceinline__ float4 keep(float4 v, int left) {
  if (left < 4) v = make_float4(left > 0 ? v.x : 0.f, left > 1 ? v.y : 0.f, left > 2 ? v.z : 0.f, 0.f);
  return v;
}

// The row kernels in two forms: rows of up to 8192 columns in registers (HOLD float4 a thread), every load of the row and
// of the planes issued before the first sum, because with few rows the kernel is nothing but the latency of its loads
// and sums (8 rows of 4096 in 8 planes: 12.4 us through shared memory); wider rows in shared memory.  Both add a row in the same
// order, except that the layer norm in shared memory begins a float4's squares with its second column.
//
// Rows of up to as many blocks as SMs take 512 threads, twice the loads in flight (24 rows of 2048 in 8 planes 6.1 us with 256
// threads, 5.1 with 512); above, the SMs hold fewer such blocks (1794 rows of 2048 10 us and 15.7).
constexpr int kRegCols = 8192, kFewRows = 148;

// the sum of the planes of row m, in order
template <int THREADS, int HOLD>
__device__ __forceinline__ void load_planes(const float* y, int planes, size_t m, int M, int ld, int n4, float4 (&v)[HOLD]) {
  const size_t step = static_cast<size_t>(M) * ld / 4;
  const float4* src = reinterpret_cast<const float4*>(y + m * ld);
#pragma unroll
  for (int i = 0; i < HOLD; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll(HOLD > 2 ? 4 : 8)
  for (int p = 0; p < planes; ++p) {
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int c = i * THREADS + threadIdx.x;
      const float4 w = c < n4 ? __ldcg(src + p * step + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[i].x += w.x; v[i].y += w.y; v[i].z += w.z; v[i].w += w.w;
    }
  }
}
template <int THREADS, int HOLD>
__device__ __forceinline__ void load_row(const float* row, int n4, float4 (&v)[HOLD]) {
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    const int c = i * THREADS + threadIdx.x;
    v[i] = row && c < n4 ? reinterpret_cast<const float4*>(row)[c] : make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

template <int THREADS, int HOLD>
__global__ void __launch_bounds__(THREADS) residual_norm_reg_kernel(const ResidualNormArgs a) {
  __shared__ RowSum<THREADS, HOLD> row_sum;
  float part[HOLD];
  const int n4 = a.ld >> 2;
  const size_t m = blockIdx.x;
  float4 wp[HOLD], wn[HOLD], x[HOLD];
  load_row<THREADS, HOLD>(a.y ? a.w_post : nullptr, n4, wp);          // weights do not depend on the predecessor
  load_row<THREADS, HOLD>(a.xn || a.xn_f32 ? a.w_next : nullptr, n4, wn);
  pdl_wait();
  pdl_launch_dependents();
  float4* xrow = reinterpret_cast<float4*>(a.x + (a.select ? a.select[m] : m) * a.ld);
  load_row<THREADS, HOLD>(reinterpret_cast<const float*>(xrow), n4, x);
  if (a.y) {
    float4 y[HOLD];
    load_planes<THREADS, HOLD>(a.y, a.planes, m, a.M, a.ld, n4, y);
#pragma unroll
    for (int i = 0; i < HOLD; ++i) part[i] = dot4(y[i]);
    const float rs = a.mult / sqrtf(row_sum(part) / static_cast<float>(a.d) + a.eps);
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int c = i * THREADS + threadIdx.x;
      x[i] = keep(make_float4(fmaf(y[i].x * rs, wp[i].x, x[i].x), fmaf(y[i].y * rs, wp[i].y, x[i].y), fmaf(y[i].z * rs, wp[i].z, x[i].z),
                              fmaf(y[i].w * rs, wp[i].w, x[i].w)), a.d - 4 * c);
      if (c < n4) xrow[c] = x[i];
    }
  }
#pragma unroll
  for (int i = 0; i < HOLD; ++i) part[i] = dot4(x[i]);
  const float rs = 1.0f / sqrtf(row_sum(part) / static_cast<float>(a.d) + a.eps);
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    const int c = i * THREADS + threadIdx.x;
    if (c >= n4) continue;
    const float4 v = x[i], w = wn[i];
    if (a.xn_f32) reinterpret_cast<float4*>(a.xn_f32 + m * a.ld)[c] = keep(make_float4(w.x * rs * v.x, w.y * rs * v.y, w.z * rs * v.z, w.w * rs * v.w), a.d - 4 * c);
    if (a.xn) reinterpret_cast<uint2*>(a.xn + m * a.ld)[c] = pack4(keep(make_float4(v.x * rs * w.x, v.y * rs * w.y, v.z * rs * w.z, v.w * rs * w.w), a.d - 4 * c));
    if (a.cat_f32 || a.cat_bf16) {
      const float4 e = reinterpret_cast<const float4*>(a.x0 + m * a.ld)[c];
      if (a.cat_f32) {
        float4* o = reinterpret_cast<float4*>(a.cat_f32 + m * 2 * a.ld);
        o[c] = v;
        o[n4 + c] = e;
      }
      if (a.cat_bf16) {
        uint2* o = reinterpret_cast<uint2*>(a.cat_bf16 + m * 2 * a.ld);
        o[c] = pack4(v);
        o[n4 + c] = pack4(e);
      }
    }
  }
}

template <int THREADS, int HOLD>
__global__ void __launch_bounds__(THREADS) residual_layernorm_reg_kernel(const ResidualLayerNormArgs a) {
  __shared__ RowSum<THREADS, HOLD> row_sum;
  float part[HOLD];
  const int n4 = a.ld >> 2;
  const size_t m = blockIdx.x;
  const float inv_n = 1.0f / static_cast<float>(a.d);
  float4 w[HOLD], b[HOLD], x[HOLD];
  load_row<THREADS, HOLD>(a.y ? a.w : nullptr, n4, w);                // weights do not depend on the predecessor
  load_row<THREADS, HOLD>(a.y ? a.b : nullptr, n4, b);
  pdl_wait();
  pdl_launch_dependents();
  float4* xrow = reinterpret_cast<float4*>(a.x + (a.select ? a.select[m] : m) * a.ld);
  auto norm = [&](float* mu, float* rs) {
#pragma unroll
    for (int i = 0; i < HOLD; ++i) part[i] = (x[i].x + x[i].y) + (x[i].z + x[i].w);
    *mu = __fmul_rn(row_sum(part), inv_n);               // never fused into the differences below, in no template
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int left = a.d - 4 * (i * THREADS + static_cast<int>(threadIdx.x));      // columns that exist
      part[i] = dot4(make_float4(left > 0 ? x[i].x - *mu : 0.f, left > 1 ? x[i].y - *mu : 0.f, left > 2 ? x[i].z - *mu : 0.f, left > 3 ? x[i].w - *mu : 0.f));
    }
    *rs = 1.0f / sqrtf(row_sum(part) * inv_n + a.eps);
  };
  auto scaled = [&](int c, const float4& z, float mu, float rs, const float4& w4, const float4& b4) {
    return keep(make_float4(fmaf((z.x - mu) * rs, w4.x, b4.x), fmaf((z.y - mu) * rs, w4.y, b4.y), fmaf((z.z - mu) * rs, w4.z, b4.z),
                            fmaf((z.w - mu) * rs, w4.w, b4.w)), a.d - 4 * c);
  };
  // the products of the norm in the order of the fp32 path
  auto rescaled = [&](int c, const float4& z, float mu, float rs, const float4& w4, const float4& b4) {
    return keep(make_float4(fmaf(w4.x * rs, z.x - mu, b4.x), fmaf(w4.y * rs, z.y - mu, b4.y), fmaf(w4.z * rs, z.z - mu, b4.z),
                            fmaf(w4.w * rs, z.w - mu, b4.w)), a.d - 4 * c);
  };
  float mu, rs;
  load_row<THREADS, HOLD>(reinterpret_cast<const float*>(xrow), n4, x);
  if (a.y) {
    float4 y[HOLD];
    load_planes<THREADS, HOLD>(a.y, a.planes, m, a.M, a.ld, n4, y);
#pragma unroll
    for (int i = 0; i < HOLD; ++i)
      x[i] = make_float4(fmaf(a.alpha, x[i].x, y[i].x), fmaf(a.alpha, x[i].y, y[i].y), fmaf(a.alpha, x[i].z, y[i].z), fmaf(a.alpha, x[i].w, y[i].w));
    norm(&mu, &rs);
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int c = i * THREADS + threadIdx.x;
      x[i] = scaled(c, x[i], mu, rs, w[i], b[i]);
      if (c < n4) xrow[c] = x[i];
    }
  }
  if (a.xn && !a.w_next) {
#pragma unroll
    for (int i = 0; i < HOLD; ++i) {
      const int c = i * THREADS + threadIdx.x;
      if (c < n4) reinterpret_cast<uint2*>(a.xn + m * a.ld)[c] = pack4(x[i]);
    }
  }
  if (!a.w_next) return;
  norm(&mu, &rs);
  load_row<THREADS, HOLD>(a.w_next, n4, w);
  load_row<THREADS, HOLD>(a.b_next, n4, b);
#pragma unroll
  for (int i = 0; i < HOLD; ++i) {
    const int c = i * THREADS + threadIdx.x;
    if (c >= n4) continue;
    if (a.xn) reinterpret_cast<uint2*>(a.xn + m * a.ld)[c] = pack4(scaled(c, x[i], mu, rs, w[i], b[i]));
    if (a.xn_f32) reinterpret_cast<float4*>(a.xn_f32 + m * a.ld)[c] = rescaled(c, x[i], mu, rs, w[i], b[i]);
  }
}

// Norm after the sublayer, residual add and the norm before the next sublayer, one pass over the row.  Every thread
// touches only the columns it owns, so the row lives in shared memory without barriers between the passes.
__global__ void __launch_bounds__(kRnThreads) residual_norm_kernel(const ResidualNormArgs a) {
  extern __shared__ float4 rn_row[];                   // x, then (with y) y
  __shared__ float red[kRnThreads / 32];
  pdl_wait();
  pdl_launch_dependents();
  const int n4 = a.ld >> 2;
  const size_t m = blockIdx.x;
  float4* xrow = reinterpret_cast<float4*>(a.x + (a.select ? a.select[m] : m) * a.ld);
  float ss = 0.f;
  if (a.y) {
    float4* yrow = rn_row + n4;
    float ys = 0.f;
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      float4 v = reinterpret_cast<const float4*>(a.y + m * a.ld)[i];
#pragma unroll 4
      for (int p = 1; p < a.planes; ++p) {
        const float4 w = reinterpret_cast<const float4*>(a.y + (static_cast<size_t>(p) * a.M + m) * a.ld)[i];
        v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
      }
      yrow[i] = v;
      rn_row[i] = xrow[i];
      ys += dot4(v);
    }
    const float rs = a.mult / sqrtf(rn_block_sum(ys, red) / static_cast<float>(a.d) + a.eps);
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 y = yrow[i], w = reinterpret_cast<const float4*>(a.w_post)[i];
      float4 x = rn_row[i];
      x.x = fmaf(y.x * rs, w.x, x.x);
      x.y = fmaf(y.y * rs, w.y, x.y);
      x.z = fmaf(y.z * rs, w.z, x.z);
      x.w = fmaf(y.w * rs, w.w, x.w);
      x = keep(x, a.d - 4 * i);
      rn_row[i] = x;
      xrow[i] = x;
      ss += dot4(x);
    }
  } else {
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 x = xrow[i];
      rn_row[i] = x;
      ss += dot4(x);
    }
  }
  const float rs = 1.0f / sqrtf(rn_block_sum(ss, red) / static_cast<float>(a.d) + a.eps);
  if (a.xn) {
    uint2* o = reinterpret_cast<uint2*>(a.xn + m * a.ld);
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 x = rn_row[i], w = reinterpret_cast<const float4*>(a.w_next)[i];
      o[i] = pack4(keep(make_float4(x.x * rs * w.x, x.y * rs * w.y, x.z * rs * w.z, x.w * rs * w.w), a.d - 4 * i));
    }
  }
  if (a.xn_f32) {
    float4* o = reinterpret_cast<float4*>(a.xn_f32 + m * a.ld);
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 x = rn_row[i], w = reinterpret_cast<const float4*>(a.w_next)[i];
      o[i] = keep(make_float4(w.x * rs * x.x, w.y * rs * x.y, w.z * rs * x.z, w.w * rs * x.w), a.d - 4 * i);
    }
  }
  if (a.cat_f32 || a.cat_bf16) {
    const float4* x0 = reinterpret_cast<const float4*>(a.x0 + m * a.ld);
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 x = rn_row[i], e = x0[i];
      if (a.cat_f32) {
        float4* o = reinterpret_cast<float4*>(a.cat_f32 + m * 2 * a.ld);
        o[i] = x;
        o[n4 + i] = e;
      }
      if (a.cat_bf16) {
        uint2* o = reinterpret_cast<uint2*>(a.cat_bf16 + m * 2 * a.ld);
        o[i] = pack4(x);
        o[n4 + i] = pack4(e);
      }
    }
  }
}

// The same for layers with a layer norm behind the residual sum.
__global__ void __launch_bounds__(kRnThreads) residual_layernorm_kernel(const ResidualLayerNormArgs a) {
  extern __shared__ float4 rn_row[];
  __shared__ float red[kRnThreads / 32];
  pdl_wait();
  pdl_launch_dependents();
  const int n4 = a.ld >> 2;
  const size_t m = blockIdx.x;
  float4* xrow = reinterpret_cast<float4*>(a.x + (a.select ? a.select[m] : m) * a.ld);
  const float inv_n = 1.0f / static_cast<float>(a.d);
  auto norm = [&](float sum, float* mu, float* rs) {
    *mu = __fmul_rn(rn_block_sum(sum, red), inv_n);
    float v = 0.f;
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 z = rn_row[i];
      const int left = a.d - 4 * i;                       // columns that exist
      const float dx = left > 0 ? z.x - *mu : 0.f, dy = left > 1 ? z.y - *mu : 0.f, dz = left > 2 ? z.z - *mu : 0.f, dw = left > 3 ? z.w - *mu : 0.f;
      v += fmaf(dw, dw, fmaf(dz, dz, fmaf(dy, dy, dx * dx)));                      // (not dot4's order)
    }
    *rs = 1.0f / sqrtf(rn_block_sum(v, red) * inv_n + a.eps);
  };
  auto scaled = [&](int i, float mu, float rs, const float* w, const float* b) {
    const float4 z = rn_row[i], w4 = reinterpret_cast<const float4*>(w)[i], b4 = reinterpret_cast<const float4*>(b)[i];
    return keep(make_float4(fmaf((z.x - mu) * rs, w4.x, b4.x), fmaf((z.y - mu) * rs, w4.y, b4.y), fmaf((z.z - mu) * rs, w4.z, b4.z),
                            fmaf((z.w - mu) * rs, w4.w, b4.w)), a.d - 4 * i);
  };
  float sum = 0.f, mu, rs;
  for (int i = threadIdx.x; i < n4; i += kRnThreads) {
    float4 x = xrow[i];
    if (a.y) {
      float4 y = reinterpret_cast<const float4*>(a.y + m * a.ld)[i];
#pragma unroll 4
      for (int p = 1; p < a.planes; ++p) {
        const float4 w = reinterpret_cast<const float4*>(a.y + (static_cast<size_t>(p) * a.M + m) * a.ld)[i];
        y.x += w.x; y.y += w.y; y.z += w.z; y.w += w.w;
      }
      x = make_float4(fmaf(a.alpha, x.x, y.x), fmaf(a.alpha, x.y, y.y), fmaf(a.alpha, x.z, y.z), fmaf(a.alpha, x.w, y.w));
    }
    rn_row[i] = x;
    sum += (x.x + x.y) + (x.z + x.w);
  }
  if (a.y) {
    norm(sum, &mu, &rs);
    sum = 0.f;
    for (int i = threadIdx.x; i < n4; i += kRnThreads) {
      const float4 x = scaled(i, mu, rs, a.w, a.b);
      rn_row[i] = x;
      xrow[i] = x;
      sum += (x.x + x.y) + (x.z + x.w);
      if (a.xn && !a.w_next) reinterpret_cast<uint2*>(a.xn + m * a.ld)[i] = pack4(x);
    }
  } else if (a.xn && !a.w_next) {
    for (int i = threadIdx.x; i < n4; i += kRnThreads) reinterpret_cast<uint2*>(a.xn + m * a.ld)[i] = pack4(rn_row[i]);
  }
  if (!a.w_next) return;
  norm(sum, &mu, &rs);
  for (int i = threadIdx.x; i < n4; i += kRnThreads) {
    if (a.xn) reinterpret_cast<uint2*>(a.xn + m * a.ld)[i] = pack4(scaled(i, mu, rs, a.w_next, a.b_next));
    if (!a.xn_f32) continue;
    const float4 z = rn_row[i], w4 = reinterpret_cast<const float4*>(a.w_next)[i], b4 = reinterpret_cast<const float4*>(a.b_next)[i];
    reinterpret_cast<float4*>(a.xn_f32 + m * a.ld)[i] =
        keep(make_float4(fmaf(w4.x * rs, z.x - mu, b4.x), fmaf(w4.y * rs, z.y - mu, b4.y), fmaf(w4.z * rs, z.z - mu, b4.z),
                         fmaf(w4.w * rs, z.w - mu, b4.w)), a.d - 4 * i);
  }
}

__global__ void gather_rows_bf16_kernel(const __nv_bfloat16* __restrict__ src, int ld, const int32_t* __restrict__ rows,
                                        __nv_bfloat16* __restrict__ dst) {
  const uint4* s = reinterpret_cast<const uint4*>(src + static_cast<size_t>(rows[blockIdx.x]) * ld);
  uint4* d = reinterpret_cast<uint4*>(dst + static_cast<size_t>(blockIdx.x) * ld);
  for (int i = threadIdx.x; i < ld / 8; i += blockDim.x) d[i] = s[i];
}

__global__ void copy_rows_kernel(const float4* src, float4* __restrict__ dst, int64_t n4) {
  pdl_wait();
  pdl_launch_dependents();
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += step) dst[i] = src[i];
}

__device__ __forceinline__ float load_any(const void* p, int is_bf16, int64_t i) {
  return is_bf16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(p)[i]) : static_cast<const float*>(p)[i];
}

__global__ void pack_rows_kernel(const void* src, int src_is_bf16, int N, int K, __nv_bfloat16* dst, int ld, int r0,
                                 int gin, int gout, int csplit, int cshift) {
  const int64_t total = static_cast<int64_t>(N) * K, step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step) {
    const int n = static_cast<int>(i / K), k = static_cast<int>(i % K);
    const size_t row = static_cast<size_t>(r0) + static_cast<size_t>(n / gin) * gout + n % gin;
    dst[row * ld + (k < csplit ? k : k + cshift)] = __float2bfloat16_rn(load_any(src, src_is_bf16, i));
  }
}

__global__ void neg_exp_kernel(const void* src, int src_is_bf16, int64_t n, float* dst) {
  const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += step)
    dst[i] = -expf(load_any(src, src_is_bf16, i));
}

__global__ void transpose_f32_kernel(const void* src, int src_is_bf16, int N, int K, float* dst, int ld) {
  const int64_t total = static_cast<int64_t>(N) * K, step = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += step)
    dst[static_cast<size_t>(i % K) * ld + i / K] = load_any(src, src_is_bf16, i);
}

int load_grid(int64_t n) { return static_cast<int>(std::min<int64_t>((n + 255) / 256, 4096)); }

}  // namespace

cudaError_t launch_residual_norm(const ResidualNormArgs& a, cudaStream_t s, bool pdl) {
  if (a.M <= 0 || a.d <= 0 || a.ld < a.d || (a.ld & 3)) return cudaErrorInvalidValue;
  auto go = [&](auto kernel, int threads) { return launch_pdl(kernel, dim3(a.M), dim3(threads), 0, s, pdl, a); };
  const bool few = a.M <= kFewRows;
  if (a.ld <= 2048) return few ? go(residual_norm_reg_kernel<512, 1>, 512) : go(residual_norm_reg_kernel<256, 2>, 256);
  if (a.ld <= 4096) return few ? go(residual_norm_reg_kernel<512, 2>, 512) : go(residual_norm_reg_kernel<256, 4>, 256);
  if (a.ld <= kRegCols) return few ? go(residual_norm_reg_kernel<512, 4>, 512) : go(residual_norm_reg_kernel<256, 8>, 256);
  const size_t smem = static_cast<size_t>(a.ld) * sizeof(float) * (a.y ? 2 : 1);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  static DeviceOnce once;
  cudaError_t e = once.run([&] {
    return cudaFuncSetAttribute(residual_norm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  });
  if (e != cudaSuccess) return e;
  return launch_pdl(residual_norm_kernel, dim3(a.M), dim3(kRnThreads), smem, s, pdl, a);
}

cudaError_t launch_residual_layernorm(const ResidualLayerNormArgs& a, cudaStream_t s, bool pdl) {
  if (a.M <= 0 || a.d <= 0 || a.ld < a.d || (a.ld & 3) || (a.y && (!a.w || !a.b)) || (a.w_next && !a.b_next)) return cudaErrorInvalidValue;
  auto go = [&](auto kernel, int threads) { return launch_pdl(kernel, dim3(a.M), dim3(threads), 0, s, pdl, a); };
  const bool few = a.M <= kFewRows;
  // many short rows are bound by how many blocks an SM holds, not by the latency of one row's loads: in shared memory (1500
  // rows of 512: 5.6 us there, 7.6 in registers)
  const bool many = a.M > 512 && a.ld <= 1024;
  if (!many && a.ld <= 2048) return few ? go(residual_layernorm_reg_kernel<512, 1>, 512) : go(residual_layernorm_reg_kernel<256, 2>, 256);
  if (!many && a.ld <= 4096) return few ? go(residual_layernorm_reg_kernel<512, 2>, 512) : go(residual_layernorm_reg_kernel<256, 4>, 256);
  if (!many && a.ld <= kRegCols) return few ? go(residual_layernorm_reg_kernel<512, 4>, 512) : go(residual_layernorm_reg_kernel<256, 8>, 256);
  const size_t smem = static_cast<size_t>(a.ld) * sizeof(float);
  if (smem > 200 * 1024) return cudaErrorInvalidValue;
  static DeviceOnce once;
  cudaError_t e = once.run([&] {
    return cudaFuncSetAttribute(residual_layernorm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  });
  if (e != cudaSuccess) return e;
  return launch_pdl(residual_layernorm_kernel, dim3(a.M), dim3(kRnThreads), smem, s, pdl, a);
}

cudaError_t launch_gather_rows_bf16(const __nv_bfloat16* src, int ld, const int32_t* rows, int n, __nv_bfloat16* dst,
                                    cudaStream_t s) {
  if (n <= 0 || (ld & 7)) return cudaErrorInvalidValue;
  gather_rows_bf16_kernel<<<n, 128, 0, s>>>(src, ld, rows, dst);
  return cudaGetLastError();
}

cudaError_t launch_copy_rows(const float* src, float* dst, int64_t n, cudaStream_t s, bool pdl) {
  if (n <= 0 || (n & 3)) return cudaErrorInvalidValue;
  return launch_pdl(copy_rows_kernel, dim3(static_cast<int>(std::min<int64_t>((n / 4 + 255) / 256, 1184))), dim3(256), 0, s, pdl,
                    reinterpret_cast<const float4*>(src), reinterpret_cast<float4*>(dst), n / 4);
}

cudaError_t launch_pack_rows(const void* src, int src_is_bf16, int N, int K, __nv_bfloat16* dst, int ld, int r0, int gin,
                             int gout, int csplit, int cshift, cudaStream_t s) {
  pack_rows_kernel<<<load_grid(static_cast<int64_t>(N) * K), 256, 0, s>>>(src, src_is_bf16, N, K, dst, ld, r0, gin, gout,
                                                                          csplit, cshift);
  return cudaGetLastError();
}

cudaError_t launch_neg_exp(const void* src, int src_is_bf16, int64_t n, float* dst, cudaStream_t s) {
  neg_exp_kernel<<<load_grid(n), 256, 0, s>>>(src, src_is_bf16, n, dst);
  return cudaGetLastError();
}

cudaError_t launch_transpose_f32(const void* src, int src_is_bf16, int N, int K, float* dst, int ld, cudaStream_t s) {
  transpose_f32_kernel<<<load_grid(static_cast<int64_t>(N) * K), 256, 0, s>>>(src, src_is_bf16, N, K, dst, ld);
  return cudaGetLastError();
}

}  // namespace mtj
