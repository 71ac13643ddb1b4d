// fp32 activations times bf16 weights for 5 rows and more (short portions of a prompt, 32-bit runs): CUDA cores only, so
// that a product keeps fp32 inputs and fp32 sums.
//
//   y[m, n] = sum_k W[n, k] * act(x[m, k])        epilogues as in the GEMV family (no RoPE form)
//
// The GEMV kernel holds at most four rows per pass over the weights and waits for L2 in every chunk.  Here a block stages
// 64 weight rows x 256 columns and up to 16 activation rows (normed there) in shared memory, two stages deep, and multiplies
// them with packed fp32 FMAs (two columns per instruction): lanes are 8 weight rows x 4 activation rows, a thread 8 x MT / 4
// outputs, and the 8 warps of a block share the columns.  Bound by the weights' bytes up to about 8 rows and by
// shared-memory reads above (8 + MT / 2 16-byte reads per 8 MT packed FMAs).  Two blocks per SM.  K is split over blocks until there are about four per SM; the last block of a tile adds the pieces in
// order.  Width 2048, portions of 1 to 21
// rows, us a launch: 11264 x 2048 weights 66 by the GEMV kernel, 48 here; 2048 x 4096 and 5632 32, 14; 4096 x 2048 33, 18.
#include <math.h>

#include <algorithm>

#include "mtj_common.cuh"
#include "mtj_kernels.h"

namespace mtj {
namespace {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kTileN = 64, kSlab = 256;
constexpr int kWPitch = kSlab + 8, kXPitch = kSlab + 4;      // in elements: rows 4 banks apart
constexpr int kMaxTileM = 16;

__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
// two bf16 in a word -> two fp32
__device__ __forceinline__ unsigned long long widen(uint32_t w) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(w << 16), "r"(w & 0xffff0000u));
  return r;
}
__device__ __forceinline__ float sum2(unsigned long long v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return __uint_as_float(lo) + __uint_as_float(hi);
}
__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src, bool in) {
  const int bytes = in ? 16 : 0;                              // 0: zeros are written, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

template <int MT, int EPI>
__global__ void __launch_bounds__(kThreads, 2) gemm_rows_kernel(const GemvArgs a, float* planes, uint32_t* counters, int slabs_per_block) {
  constexpr bool kNorm = EPI == kEpiLogits || EPI == kEpiSwiGLU;
  constexpr int JM = MT / 4, kOut = kTileN * MT;
  extern __shared__ __align__(16) unsigned char rows_smem[];
  constexpr int kStage = kTileN * kWPitch * 2 + MT * kXPitch * 4;      // bytes: weights, then activations
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nl = lane & 7, ml = lane >> 3;
  const int n0 = blockIdx.x * kTileN, m0 = blockIdx.y * MT, rows = min(MT, a.M - m0);
  const int slabs = (a.K + kSlab - 1) / kSlab, s0 = blockIdx.z * slabs_per_block, s1 = min(slabs, s0 + slabs_per_block);
  auto w_of = [&](int slab) { return reinterpret_cast<__nv_bfloat16*>(rows_smem + ((slab - s0) & 1) * kStage); };
  auto x_of = [&](int slab) { return reinterpret_cast<float*>(rows_smem + ((slab - s0) & 1) * kStage + kTileN * kWPitch * 2); };

  auto load_w = [&](int slab) {                                // a warp takes rows warp, warp + 8, ...
    const int k = slab * kSlab + lane * 8;
    const uint32_t dst = smem_u32(w_of(slab) + warp * kWPitch + lane * 8);
#pragma unroll
    for (int i = 0; i < kTileN / kWarps; ++i) {
      const int n = i * kWarps + warp;
      const bool in = n0 + n < a.N && k < a.K;
      copy16_async(dst + i * kWarps * kWPitch * 2, a.W + (in ? static_cast<size_t>(n0 + n) * a.K + k : 0), in);
    }
  };
  // a thread stages, norms and looks up the same four columns of rows xr, xr + 4, ...
  const int xr = static_cast<int>(threadIdx.x >> 6), xc = static_cast<int>(threadIdx.x & 63) * 4;
  auto load_x = [&](int slab) {
    const int k = slab * kSlab + xc;
    const uint32_t dst = smem_u32(x_of(slab) + xr * kXPitch + xc);
#pragma unroll
    for (int r = 0; r < MT; r += 4) {
      const bool in = r + xr < rows && k < a.K;
      const int src = in ? (a.row_select ? a.row_select[m0 + r + xr] : m0 + r + xr) : 0;
      copy16_async(dst + r * kXPitch * 4, a.x + static_cast<size_t>(src) * a.ldx + (in ? k : 0), in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  load_w(s0);                                                  // weights do not depend on the predecessor
  pdl_wait();
  pdl_launch_dependents();
  load_x(s0);
  float mean[JM], rstd[JM];
  if (kNorm) {
#pragma unroll
    for (int r = 0; r < JM; ++r) {
      const int m = min(m0 + 4 * r + xr, a.M - 1), src = a.row_select ? a.row_select[m] : m;
      mean[r] = a.stats[2 * src];
      rstd[r] = a.stats[2 * src + 1];
    }
  }

  unsigned long long acc[8][JM];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < JM; ++j) acc[i][j] = 0ull;

  for (int slab = s0; slab < s1; ++slab) {
    if (slab + 1 < s1) {                                       // into the stage that the barrier below has freed
      load_w(slab + 1);
      load_x(slab + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    float* xs = x_of(slab);
    const __nv_bfloat16* ws = w_of(slab);
    if (kNorm && slab * kSlab + xc < a.K) {
      const int k = slab * kSlab + xc;
      const float4 sc = *reinterpret_cast<const float4*>(a.ln_scale + k), of = *reinterpret_cast<const float4*>(a.ln_offset + k);
#pragma unroll
      for (int r = 0; r < JM; ++r) {
        float4* p = reinterpret_cast<float4*>(xs + (4 * r + xr) * kXPitch + xc);
        const float4 v = *p;
        *p = make_float4(fmaf(sc.x * rstd[r], v.x - mean[r], of.x), fmaf(sc.y * rstd[r], v.y - mean[r], of.y),
                         fmaf(sc.z * rstd[r], v.z - mean[r], of.z), fmaf(sc.w * rstd[r], v.w - mean[r], of.w));
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int g = warp; g < kSlab / 8; g += kWarps) {           // groups of 8 columns
      ulonglong2 x0[JM], x1[JM];
#pragma unroll
      for (int j = 0; j < JM; ++j) {
        const ulonglong2* p = reinterpret_cast<const ulonglong2*>(xs + (ml + 4 * j) * kXPitch + g * 8);
        x0[j] = p[0];
        x1[j] = p[1];
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint4 w = *reinterpret_cast<const uint4*>(ws + (nl + 8 * i) * kWPitch + g * 8);
        const unsigned long long w0 = widen(w.x), w1 = widen(w.y), w2 = widen(w.z), w3 = widen(w.w);
#pragma unroll
        for (int j = 0; j < JM; ++j) {
          fma2(acc[i][j], w0, x0[j].x);
          fma2(acc[i][j], w1, x0[j].y);
          fma2(acc[i][j], w2, x1[j].x);
          fma2(acc[i][j], w3, x1[j].y);
        }
      }
    }
    __syncthreads();
  }
  // the warps' sums of the tile, [warp][m][n] where the slabs were
  float* part = reinterpret_cast<float*>(rows_smem);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < JM; ++j) part[warp * kOut + (ml + 4 * j) * kTileN + nl + 8 * i] = sum2(acc[i][j]);
  __syncthreads();
  constexpr int kPer = kOut / kThreads;                        // outputs of a thread
  float val[kPer];
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int o = e * kThreads + threadIdx.x;
    val[e] = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) val[e] += part[w * kOut + o];
  }
  if (gridDim.z > 1) {
    __shared__ bool last;
    const size_t tile = static_cast<size_t>(blockIdx.y) * gridDim.x + blockIdx.x;
    float* mine = planes + tile * gridDim.z * kOut;
#pragma unroll
    for (int e = 0; e < kPer; ++e) mine[static_cast<size_t>(blockIdx.z) * kOut + e * kThreads + threadIdx.x] = val[e];
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      last = atomicAdd(counters + tile, 1u) == gridDim.z - 1;
      if (last) counters[tile] = 0u;                           // for the next launch
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int e = 0; e < kPer; ++e) val[e] = 0.f;
#pragma unroll 4
    for (int z = 0; z < static_cast<int>(gridDim.z); ++z)
#pragma unroll
      for (int e = 0; e < kPer; ++e) val[e] += __ldcg(mine + static_cast<size_t>(z) * kOut + e * kThreads + threadIdx.x);
  }
  const int n_valid = a.n_valid > 0 ? a.n_valid : a.N;
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int o = e * kThreads + threadIdx.x, n = n0 + o % kTileN, r = o / kTileN;
    const size_t m = static_cast<size_t>(m0 + r);
    const float partner = EPI == kEpiSwiGLU ? __shfl_xor_sync(0xffffffffu, val[e], 1) : 0.f;
    if (r >= rows || n >= n_valid) continue;
    float y = val[e];
    if (EPI == kEpiSwiGLU) {
      if (!(n & 1)) a.act2[m * a.ld_out + (n >> 1)] = y / (1.0f + expf(-y)) * partner;
    } else if (EPI == kEpiRelu2) {
      y = fmaxf(y, 0.f);
      a.act2[m * a.ld_out + n] = y * y;
    } else {
      if (a.bias) y += a.bias[n];
      if (EPI == kEpiLogits) {
        if (a.softcap > 0.f) y = a.softcap * tanhf(y / a.softcap);
        a.logits[m * a.ld_logits + n] = y;
      } else {
        a.out[m * (a.ld_out > 0 ? a.ld_out : a.N) + n] = y;
      }
    }
  }
}

template <int MT, int EPI>
cudaError_t launch_one(const GemvArgs& a, float* planes, uint32_t* counters, cudaStream_t s, bool pdl) {
  constexpr int slab = 2 * (kTileN * kWPitch * 2 + MT * kXPitch * 4), sums = kWarps * kTileN * MT * 4, smem = slab > sums ? slab : sums;
  static DeviceOnce once;
  const cudaError_t e = once.run([&] { return cudaFuncSetAttribute(gemm_rows_kernel<MT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (e != cudaSuccess) return e;
  const int nt = (a.N + kTileN - 1) / kTileN, mt = (a.M + MT - 1) / MT, slabs = (a.K + kSlab - 1) / kSlab;
  const int64_t tiles = static_cast<int64_t>(nt) * mt;
  int64_t z = 1;
  if (tiles <= kGemmRowsCounters)
    z = std::max<int64_t>(1, std::min<int64_t>({slabs, 4 * 148 / tiles, kGemmRowsPlaneFloats / (tiles * kTileN * MT)}));
  const int per = static_cast<int>((slabs + z - 1) / z);
  return launch_pdl(gemm_rows_kernel<MT, EPI>, dim3(nt, mt, (slabs + per - 1) / per), dim3(kThreads), smem, s, pdl, a, planes, counters, per);
}

template <int EPI>
cudaError_t launch_epi(const GemvArgs& a, float* planes, uint32_t* counters, cudaStream_t s, bool pdl) {
  const int tiles = (a.M + kMaxTileM - 1) / kMaxTileM;
  switch (((a.M + tiles - 1) / tiles + 3) / 4) {               // even tiles: less padding; from 5 rows on 5 at least
    case 2: return launch_one<8, EPI>(a, planes, counters, s, pdl);
    case 3: return launch_one<12, EPI>(a, planes, counters, s, pdl);
    default: return launch_one<16, EPI>(a, planes, counters, s, pdl);
  }
}

}  // namespace

cudaError_t launch_gemm_rows(GemvEpilogue epi, const GemvArgs& a, float* planes, uint32_t* counters, cudaStream_t s, bool pdl) {
  if (a.M < kGemmRowsMin || a.N <= 0 || a.K <= 0 || (a.K & 7) || (a.ldx & 3) || a.post_w || a.stats_out || a.residual || a.slot_sel || !planes || !counters)
    return cudaErrorInvalidValue;
  switch (epi) {
    case kEpiOut: return launch_epi<kEpiOut>(a, planes, counters, s, pdl);
    case kEpiSwiGLU: return launch_epi<kEpiSwiGLU>(a, planes, counters, s, pdl);
    case kEpiRelu2: return launch_epi<kEpiRelu2>(a, planes, counters, s, pdl);
    case kEpiLogits: return launch_epi<kEpiLogits>(a, planes, counters, s, pdl);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mtj
