// What the last block of a weight-streaming product does with finished rows: the norm behind a sublayer, the residual and the
// norm before the next sublayer (GemvArgs::post_w), shared by the GEMV kernels.  The next product gets its rows normed: a norm
// in its own prologue costs every one of its blocks two more loads a column (16384 x 4096 weights 27.0 us with it, 22.7
// without; 32768 x 4096 49.7 and 41.7).  For the first T threads of a block.
#pragma once
#include "mtj_common.cuh"
#include "mtj_kernels.h"

namespace mtj {
namespace {

constexpr int kGemvThreads = 256;
constexpr int kGemvWarps = kGemvThreads / 32;

// Over the first T threads of a block (a barrier of their own: a block may have a further warp).
template <int T>
__device__ __forceinline__ void gemv_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(T) : "memory"); }
template <int T = kGemvThreads>
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = v;
  gemv_barrier<T>();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < T / 32; ++i) t += red[i];
  gemv_barrier<T>();
  return t;
}

// the row of a.out (M = 1), written by other blocks before their arrival was counted
template <int T = kGemvThreads>
__device__ __forceinline__ void finish_row(const GemvArgs& a, float* red) {
  const int n_out = a.n_valid > 0 ? a.n_valid : a.N;
  const float inv_n = 1.0f / static_cast<float>(n_out);
  // rows of up to kHold * 4 * T = 4096 numbers live in registers: one round of loads for y and x together
  constexpr int kHold = 1024 / T;
  const bool held = (n_out & 3) == 0 && n_out <= kHold * 4 * T;
  auto column = [](int i) { return 4 * (i * T + static_cast<int>(threadIdx.x)); };
  const float* row = a.out;
  float* xrow = a.post_x;
  float* xn = a.post_xn;
  if (held) {
    // (the next norm's weights as well, where a block has threads enough to hold them)
    constexpr bool kAhead = T > kGemvThreads;
    float4 y[kHold], z[kHold], w[kHold], nw[kAhead ? kHold : 1], nb[kAhead ? kHold : 1];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kHold; ++i) {
      const int c = column(i);
      const bool in = c < n_out;
      y[i] = in ? __ldcg(reinterpret_cast<const float4*>(row + c)) : zero;
      z[i] = in ? *reinterpret_cast<const float4*>(xrow + c) : zero;
      w[i] = in ? *reinterpret_cast<const float4*>(a.post_w + c) : zero;
      if (in && a.post_b) prefetch_l2(a.post_b + c);
      if (kAhead) {
        nw[kAhead ? i : 0] = in && a.post_next_w ? *reinterpret_cast<const float4*>(a.post_next_w + c) : zero;
        nb[kAhead ? i : 0] = in && a.post_next_b ? *reinterpret_cast<const float4*>(a.post_next_b + c) : zero;
      } else {
        if (in && a.post_next_w) prefetch_l2(a.post_next_w + c);
        if (in && a.post_next_b) prefetch_l2(a.post_next_b + c);
      }
    }
    auto total = [&]() {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < kHold; ++i) s += (z[i].x + z[i].y) + (z[i].z + z[i].w);
      return block_sum<T>(s, red);
    };
    auto centred = [&](float mu) {                    // sum of squared deviations
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < kHold; ++i)
        if (column(i) < n_out) {
          const float dx = z[i].x - mu, dy = z[i].y - mu, dz = z[i].z - mu, dw = z[i].w - mu;
          v += (dx * dx + dy * dy) + (dz * dz + dw * dw);
        }
      return block_sum<T>(v, red);
    };
    float mu2 = 0.f, rs2;
    if (a.post_b) {
      // layer norm of the residual sum
#pragma unroll
      for (int i = 0; i < kHold; ++i)
        z[i] = make_float4(fmaf(a.post_mult, z[i].x, y[i].x), fmaf(a.post_mult, z[i].y, y[i].y), fmaf(a.post_mult, z[i].z, y[i].z), fmaf(a.post_mult, z[i].w, y[i].w));
      const float mu = total() * inv_n;
      const float rs = 1.0f / sqrtf(centred(mu) * inv_n + a.post_eps);
#pragma unroll
      for (int i = 0; i < kHold; ++i) {
        const int c = column(i);
        if (c < n_out) {
          const float4 b = *reinterpret_cast<const float4*>(a.post_b + c);
          z[i] = make_float4(fmaf((z[i].x - mu) * rs, w[i].x, b.x), fmaf((z[i].y - mu) * rs, w[i].y, b.y),
                             fmaf((z[i].z - mu) * rs, w[i].z, b.z), fmaf((z[i].w - mu) * rs, w[i].w, b.w));
          *reinterpret_cast<float4*>(xrow + c) = z[i];
        } else {
          z[i] = zero;
        }
      }
      if (!a.post_next_w) return;
      mu2 = total() * inv_n;
      rs2 = 1.0f / sqrtf(centred(mu2) * inv_n + a.post_eps);
    } else {
      // norm after the sublayer, residual add
      float s = 0.f, q = 0.f;
#pragma unroll
      for (int i = 0; i < kHold; ++i) s += y[i].x * y[i].x + y[i].y * y[i].y + y[i].z * y[i].z + y[i].w * y[i].w;
      const float rs = a.post_mult / sqrtf(block_sum<T>(s, red) / static_cast<float>(n_out) + a.post_eps);
#pragma unroll
      for (int i = 0; i < kHold; ++i) {
        z[i] = make_float4(fmaf(y[i].x * rs, w[i].x, z[i].x), fmaf(y[i].y * rs, w[i].y, z[i].y), fmaf(y[i].z * rs, w[i].z, z[i].z), fmaf(y[i].w * rs, w[i].w, z[i].w));
        if (column(i) < n_out) *reinterpret_cast<float4*>(xrow + column(i)) = z[i];
        q += z[i].x * z[i].x + z[i].y * z[i].y + z[i].z * z[i].z + z[i].w * z[i].w;
      }
      if (!a.post_next_w) return;
      rs2 = 1.0f / sqrtf(block_sum<T>(q, red) / static_cast<float>(n_out) + a.post_eps);
    }
#pragma unroll
    for (int i = 0; i < kHold; ++i) {
      const int c = column(i);
      if (c >= n_out) continue;
      const float4 n = kAhead ? nw[kAhead ? i : 0] : *reinterpret_cast<const float4*>(a.post_next_w + c);
      const float4 o = kAhead ? nb[kAhead ? i : 0] : a.post_next_b ? *reinterpret_cast<const float4*>(a.post_next_b + c) : zero;
      *reinterpret_cast<float4*>(xn + c) = make_float4(fmaf(n.x * rs2, z[i].x - mu2, o.x), fmaf(n.y * rs2, z[i].y - mu2, o.y),
                                                       fmaf(n.z * rs2, z[i].z - mu2, o.z), fmaf(n.w * rs2, z[i].w - mu2, o.w));
    }
    return;
  }
  // each thread re-reads only what it wrote
  float mu2 = 0.f, rs2;
  if (a.post_b) {
    float s = 0.f, v = 0.f;
    for (int i = threadIdx.x; i < n_out; i += T) s += fmaf(a.post_mult, xrow[i], __ldcg(row + i));
    const float mu = block_sum<T>(s, red) * inv_n;
    for (int i = threadIdx.x; i < n_out; i += T) {
      const float z = fmaf(a.post_mult, xrow[i], __ldcg(row + i)) - mu;
      v = fmaf(z, z, v);
    }
    const float rs = 1.0f / sqrtf(block_sum<T>(v, red) * inv_n + a.post_eps);
    s = v = 0.f;
    for (int i = threadIdx.x; i < n_out; i += T) {
      const float x = fmaf((fmaf(a.post_mult, xrow[i], __ldcg(row + i)) - mu) * rs, a.post_w[i], a.post_b[i]);
      xrow[i] = x;
      s += x;
    }
    if (!a.post_next_w) return;
    mu2 = block_sum<T>(s, red) * inv_n;
    for (int i = threadIdx.x; i < n_out; i += T) v = fmaf(xrow[i] - mu2, xrow[i] - mu2, v);
    rs2 = 1.0f / sqrtf(block_sum<T>(v, red) * inv_n + a.post_eps);
  } else {
    float s = 0.f, q = 0.f;
#pragma unroll 8
    for (int i = threadIdx.x; i < n_out; i += T) {
      const float y = __ldcg(row + i);
      s = fmaf(y, y, s);
    }
    const float rs = a.post_mult / sqrtf(block_sum<T>(s, red) / static_cast<float>(n_out) + a.post_eps);
#pragma unroll 8
    for (int i = threadIdx.x; i < n_out; i += T) {
      const float v = fmaf(__ldcg(row + i) * rs, a.post_w[i], xrow[i]);
      xrow[i] = v;
      q = fmaf(v, v, q);
    }
    if (!a.post_next_w) return;
    rs2 = 1.0f / sqrtf(block_sum<T>(q, red) / static_cast<float>(n_out) + a.post_eps);
  }
  for (int i = threadIdx.x; i < n_out; i += T)
    xn[i] = fmaf(a.post_next_w[i] * rs2, xrow[i] - mu2, a.post_next_b ? a.post_next_b[i] : 0.f);
}

}  // namespace
}  // namespace mtj
