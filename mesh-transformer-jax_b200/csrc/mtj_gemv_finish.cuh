// What the last block of a weight-streaming product does with finished rows: the norm behind a sublayer and the residual
// (GemvArgs::post_w), shared by the GEMV kernels.  For the first kGemvThreads threads of a block.
#pragma once
#include "mtj_common.cuh"
#include "mtj_kernels.h"

namespace mtj {
namespace {

constexpr int kGemvThreads = 256;
constexpr int kGemvWarps = kGemvThreads / 32;

// Over the first kGemvThreads threads of a block (a barrier of their own: a block may have a further warp).
__device__ __forceinline__ void gemv_barrier() { asm volatile("bar.sync 1, %0;" ::"n"(kGemvThreads) : "memory"); }
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) red[warp] = v;
  gemv_barrier();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < kGemvWarps; ++i) t += red[i];
  gemv_barrier();
  return t;
}

// rows [m0, m0 + nb) of a.out, written by other blocks before their arrival was counted
__device__ __forceinline__ void finish_rows(const GemvArgs& a, int m0, int nb, float* red) {
  if (a.post_b) {
    // layer norm of the residual sum; the row lives in registers (kHold float4 a thread) or is read again from L2
    const int n_out = a.n_valid > 0 ? a.n_valid : a.N;
    constexpr int kHold = 4;
    const int ldo = a.ld_out > 0 ? a.ld_out : a.N;
    const float inv_n = 1.0f / static_cast<float>(n_out);
    const bool held = ((n_out | ldo | a.post_ldx) & 3) == 0 && n_out <= kHold * 4 * kGemvThreads;
    for (int bt = 0; bt < nb; ++bt) {
      const float* row = a.out + static_cast<size_t>(m0 + bt) * ldo;
      float* xrow = a.post_x + static_cast<size_t>(m0 + bt) * a.post_ldx;
      float mu2 = 0.f, rs2 = 0.f;
      if (held) {
        float4 z[kHold];
        float s = 0.f, q = 0.f;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < kHold; ++i) {
          const int c = 4 * (i * kGemvThreads + static_cast<int>(threadIdx.x));
          const bool in = c < n_out;
          const float4 y = in ? __ldcg(reinterpret_cast<const float4*>(row + c)) : zero;
          const float4 x = in ? *reinterpret_cast<const float4*>(xrow + c) : zero;
          if (in) prefetch_l2(a.post_w + c);
          if (in) prefetch_l2(a.post_b + c);
          z[i] = make_float4(fmaf(a.post_mult, x.x, y.x), fmaf(a.post_mult, x.y, y.y), fmaf(a.post_mult, x.z, y.z), fmaf(a.post_mult, x.w, y.w));
          s += (z[i].x + z[i].y) + (z[i].z + z[i].w);
        }
        auto centred = [&](float mu) {                  // sum of squared deviations
          float v = 0.f;
#pragma unroll
          for (int i = 0; i < kHold; ++i)
            if (4 * (i * kGemvThreads + static_cast<int>(threadIdx.x)) < n_out) {
              const float dx = z[i].x - mu, dy = z[i].y - mu, dz = z[i].z - mu, dw = z[i].w - mu;
              v += (dx * dx + dy * dy) + (dz * dz + dw * dw);
            }
          return v;
        };
        const float mu = block_sum(s, red) * inv_n;
        const float rs = 1.0f / sqrtf(block_sum(centred(mu), red) * inv_n + a.post_eps);
#pragma unroll
        for (int i = 0; i < kHold; ++i) {
          const int c = 4 * (i * kGemvThreads + static_cast<int>(threadIdx.x));
          if (c < n_out) {
            const float4 w = *reinterpret_cast<const float4*>(a.post_w + c), b = *reinterpret_cast<const float4*>(a.post_b + c);
            z[i] = make_float4(fmaf((z[i].x - mu) * rs, w.x, b.x), fmaf((z[i].y - mu) * rs, w.y, b.y),
                               fmaf((z[i].z - mu) * rs, w.z, b.z), fmaf((z[i].w - mu) * rs, w.w, b.w));
            *reinterpret_cast<float4*>(xrow + c) = z[i];
            q += (z[i].x + z[i].y) + (z[i].z + z[i].w);
          }
        }
        if (a.stats_out) {
          mu2 = block_sum(q, red) * inv_n;
          rs2 = 1.0f / sqrtf(block_sum(centred(mu2), red) * inv_n + a.post_eps);
        }
      } else {
        float s = 0.f, v = 0.f;
        for (int i = threadIdx.x; i < n_out; i += kGemvThreads) s += fmaf(a.post_mult, xrow[i], __ldcg(row + i));
        const float mu = block_sum(s, red) * inv_n;
        for (int i = threadIdx.x; i < n_out; i += kGemvThreads) {
          const float z = fmaf(a.post_mult, xrow[i], __ldcg(row + i)) - mu;
          v = fmaf(z, z, v);
        }
        const float rs = 1.0f / sqrtf(block_sum(v, red) * inv_n + a.post_eps);
        s = v = 0.f;
        for (int i = threadIdx.x; i < n_out; i += kGemvThreads) {
          const float x = fmaf((fmaf(a.post_mult, xrow[i], __ldcg(row + i)) - mu) * rs, a.post_w[i], a.post_b[i]);
          xrow[i] = x;                                  // each thread re-reads only what it wrote
          s += x;
        }
        if (a.stats_out) {
          mu2 = block_sum(s, red) * inv_n;
          for (int i = threadIdx.x; i < n_out; i += kGemvThreads) v = fmaf(xrow[i] - mu2, xrow[i] - mu2, v);
          rs2 = 1.0f / sqrtf(block_sum(v, red) * inv_n + a.post_eps);
        }
      }
      if (threadIdx.x == 0 && a.stats_out) {
        a.stats_out[2 * (m0 + bt)] = mu2;
        a.stats_out[2 * (m0 + bt) + 1] = rs2;
      }
    }
    return;
  }
  if (a.post_w) {
    // norm after the sublayer, residual add, and the root mean square of the new residual row
    const int n_out = a.n_valid > 0 ? a.n_valid : a.N;
    // rows of up to kHold * 4 * 256 numbers live in registers: one round of loads for y and x together
    constexpr int kHold = 4;
    const int ldo = a.ld_out > 0 ? a.ld_out : a.N;
    const bool held = ((n_out | ldo | a.post_ldx) & 3) == 0 && n_out <= kHold * 4 * kGemvThreads;
    for (int bt = 0; bt < nb; ++bt) {
      const float* row = a.out + static_cast<size_t>(m0 + bt) * ldo;
      float* xrow = a.post_x + static_cast<size_t>(m0 + bt) * a.post_ldx;
      float s = 0.f, q = 0.f;
      if (held) {
        float4 y4[kHold], x4[kHold];
#pragma unroll
        for (int i = 0; i < kHold; ++i) {
          const int c = 4 * (i * kGemvThreads + static_cast<int>(threadIdx.x));
          const bool in = c < n_out;
          y4[i] = in ? __ldcg(reinterpret_cast<const float4*>(row + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
          if (in) prefetch_l2(a.post_w + c);
          x4[i] = in ? *reinterpret_cast<const float4*>(xrow + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < kHold; ++i)
          s += y4[i].x * y4[i].x + y4[i].y * y4[i].y + y4[i].z * y4[i].z + y4[i].w * y4[i].w;
        const float rs = a.post_mult / sqrtf(block_sum(s, red) / static_cast<float>(n_out) + a.post_eps);
#pragma unroll
        for (int i = 0; i < kHold; ++i) {
          const int c = 4 * (i * kGemvThreads + static_cast<int>(threadIdx.x));
          float4 v = x4[i];
          if (c < n_out) {
            const float4 w = *reinterpret_cast<const float4*>(a.post_w + c);
            v.x = fmaf(y4[i].x * rs, w.x, v.x);
            v.y = fmaf(y4[i].y * rs, w.y, v.y);
            v.z = fmaf(y4[i].z * rs, w.z, v.z);
            v.w = fmaf(y4[i].w * rs, w.w, v.w);
            *reinterpret_cast<float4*>(xrow + c) = v;
          }
          q += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
        }
      } else {
#pragma unroll 8
        for (int i = threadIdx.x; i < n_out; i += kGemvThreads) {
          const float y = __ldcg(row + i);
          s = fmaf(y, y, s);
        }
        const float rs = a.post_mult / sqrtf(block_sum(s, red) / static_cast<float>(n_out) + a.post_eps);
#pragma unroll 8
        for (int i = threadIdx.x; i < n_out; i += kGemvThreads) {
          const float v = fmaf(__ldcg(row + i) * rs, a.post_w[i], xrow[i]);
          xrow[i] = v;
          q = fmaf(v, v, q);
        }
      }
      const float ms = block_sum(q, red) / static_cast<float>(n_out);
      if (threadIdx.x == 0) {
        a.stats_out[2 * (m0 + bt)] = 0.f;
        a.stats_out[2 * (m0 + bt) + 1] = 1.0f / sqrtf(ms + a.post_eps);
      }
    }
    return;
  }
}

}  // namespace
}  // namespace mtj
