// fp32 activations times bf16 weights for a few rows (short portions of a prompt, 32-bit runs), on the tensor cores without
// giving up a bit of the activations.
//
//   y[m, n] = sum_k W[n, k] * act(x[m, k])        epilogues as in the GEMV family (no RoPE form)
//
// An fp32 number is the sum of three bf16 numbers of 8 significant bits each (cut off, not rounded: the remainders are
// exact), and a product of two bf16 numbers is exact in fp32, so W x = W hi + W mid + W lo in mma.sync.m16n8k16 with fp32
// sums.  Those sums are cut off, so a chain of them is kept to the 6 steps of one warp's 32 columns of a slab, smallest terms
// first, and added to the running sum by rounding additions: the error stays below that of a chain of fused multiply-adds.
//
// A block stages 64 weight rows x 128 columns by cp.async, four stages deep, and turns its slab of up to 32 activation rows
// into the three bf16 planes in shared memory, double buffered: one barrier per slab.  Warps are 2 halves
// of the weight rows x 4 quarters of the columns.  K is split over blocks so that the SMs are evenly busy; the last block of a
// tile adds the pieces in order.  (M is far below the 128 rows of a tcgen05 tile, whose sums could not be folded so often.)
#include <math.h>

#include <algorithm>

#include "mtj_common.cuh"
#include "mtj_kernels.h"

namespace mtj {
namespace {

constexpr int kThreads = 256;
constexpr int kTileN = 64, kSlab = 128, kKGroups = 4;
constexpr int kPitch = kSlab + 8;                            // in bf16 elements, an odd number of 16-byte units: conflict-free ldmatrix
constexpr int kPartPitch = kTileN + 4;
constexpr int kMaxTileM = 32;

__device__ __forceinline__ void copy16_async(uint32_t dst, const void* src, bool in) {
  const int bytes = in ? 16 : 0;                              // 0: zeros are written, nothing is read
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void ldsm4(uint32_t* r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, const uint32_t* b) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// the upper halves of two fp32 numbers side by side
__device__ __forceinline__ uint32_t tops(float lo, float hi) { return __byte_perm(__float_as_uint(lo), __float_as_uint(hi), 0x7632); }
// what the upper half of an fp32 number leaves of it; nothing of an infinity
__device__ __forceinline__ float below(float v) {
  const float r = v - __uint_as_float(__float_as_uint(v) & 0xffff0000u);
  return fabsf(v) == INFINITY ? 0.f : r;
}

template <int NT>
constexpr int kStagesOf = NT <= 3 ? 4 : 3;

template <int NT, int EPI>
__global__ void __launch_bounds__(kThreads, 2) gemm_rows_kernel(const GemvArgs a, float* planes, uint32_t* counters, int slabs_per_block) {
  constexpr int MT = 8 * NT, kOut = kTileN * MT, kStages = kStagesOf<NT>;
  constexpr uint32_t kStage = kTileN * kPitch * 2, kPlane = MT * kPitch * 2;      // bytes
  extern __shared__ __align__(16) unsigned char rows_smem[];                       // [stages] weights, [2][hi, mid, lo] activations
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nh = warp & 1, kg = warp >> 1;                     // this warp's weight rows and columns of a slab
  const int n0 = blockIdx.x * kTileN, m0 = blockIdx.y * MT, rows = min(MT, a.M - m0);
  const int slabs = (a.K + kSlab - 1) / kSlab, s0 = blockIdx.z * slabs_per_block, s1 = min(slabs, s0 + slabs_per_block);
  const uint32_t w_base = smem_u32(rows_smem), x_base = w_base + kStages * kStage;

  auto load_w = [&](int slab) {                                // a thread copies 16 bytes of every 16th row; past the end an empty group
    if (slab < s1) {
      const int k = slab * kSlab + (threadIdx.x & 15) * 8, r = threadIdx.x >> 4;
      const uint32_t dst = w_base + (slab - s0) % kStages * kStage + (r * kPitch + (threadIdx.x & 15) * 8) * 2;
#pragma unroll
      for (int i = 0; i < kTileN / 16; ++i) {
        const int n = n0 + i * 16 + r;
        const bool in = n < a.N && k < a.K;
        copy16_async(dst + i * 16 * kPitch * 2, a.W + (in ? static_cast<size_t>(n) * a.K + k : 0), in);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int i = 0; i < kStages - 1; ++i) load_w(s0 + i);        // weights do not depend on the predecessor
  pdl_wait();
  pdl_launch_dependents();
  // a thread turns the same four columns of rows warp, warp + 8, ... of every slab
  const float* xr[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i) {
    const int m = min(m0 + 8 * i + warp, a.M - 1);
    xr[i] = a.x + static_cast<size_t>(a.row_select ? a.row_select[m] : m) * a.ldx + lane * 4;
  }
  float4 xv[NT];
  auto load_x = [&](int slab) {
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const bool in = slab < s1 && slab * kSlab + lane * 4 < a.K;
#pragma unroll
    for (int i = 0; i < NT; ++i) xv[i] = in && 8 * i + warp < rows ? *reinterpret_cast<const float4*>(xr[i] + slab * kSlab) : zero;
  };
  load_x(s0);

  float sum[2][NT][4] = {};
  for (int slab = s0; slab < s1; ++slab) {
    const uint32_t xp = x_base + ((slab - s0) & 1) * 3 * kPlane;
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      const float4 v = xv[i];
      const float4 q = make_float4(below(v.x), below(v.y), below(v.z), below(v.w));
      const float4 t = make_float4(below(q.x), below(q.y), below(q.z), below(q.w));
      const uint32_t at = xp + ((8 * i + warp) * kPitch + lane * 4) * 2;
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at), "r"(tops(v.x, v.y)), "r"(tops(v.z, v.w)) : "memory");
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + kPlane), "r"(tops(q.x, q.y)), "r"(tops(q.z, q.w)) : "memory");
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(at + 2 * kPlane), "r"(tops(t.x, t.y)), "r"(tops(t.z, t.w)) : "memory");
    }
    load_x(slab + 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
    __syncthreads();                                           // the slab is there; the last one's stage and planes are read
    load_w(slab + kStages - 1);

    float acc[2][NT][4] = {};
    uint32_t wf[2][2][4];
    const uint32_t wp = w_base + (slab - s0) % kStages * kStage + ((nh * 32 + (lane & 15)) * kPitch + kg * 32 + (lane >> 4) * 8) * 2;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int k = 0; k < 2; ++k) ldsm4(wf[i][k], wp + i * 16 * kPitch * 2 + k * 32);
#pragma unroll
    for (int p = 2; p >= 0; --p)                               // smallest terms first
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        uint32_t xf[4];
        ldsm4(xf, xp + p * kPlane + ((j * 8 + (lane & 7)) * kPitch + kg * 32 + (lane >> 3) * 8) * 2);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          mma16816(acc[i][j], wf[i][0], xf);
          mma16816(acc[i][j], wf[i][1], xf + 2);
        }
      }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) sum[i][j][e] += acc[i][j][e];
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // the warps' sums of the tile, [columns' quarter][m][n] where the slabs were
  float* part = reinterpret_cast<float*>(rows_smem);
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        part[(kg * MT + j * 8 + (lane & 3) * 2 + (e & 1)) * kPartPitch + nh * 32 + i * 16 + (lane >> 2) + (e >> 1) * 8] = sum[i][j][e];
  __syncthreads();
  constexpr int kPer = kOut / kThreads;                        // outputs of a thread
  float val[kPer];
#pragma unroll
  for (int e = 0; e < kPer; ++e) {
    const int o = e * kThreads + threadIdx.x;
    val[e] = 0.f;
#pragma unroll
    for (int g = 0; g < kKGroups; ++g) val[e] += part[(g * MT + o / kTileN) * kPartPitch + o % kTileN];
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
      if (EPI == kEpiSoftcap) y = a.softcap * tanhf(y / a.softcap);
      else if (a.bias) y += a.bias[n];
      a.out[m * (a.ld_out > 0 ? a.ld_out : a.N) + n] = y;
    }
  }
}

template <int NT, int EPI>
cudaError_t launch_one(const GemvArgs& a, float* planes, uint32_t* counters, cudaStream_t s, bool pdl) {
  constexpr int MT = 8 * NT, ring = kStagesOf<NT> * kTileN * kPitch * 2 + 6 * MT * kPitch * 2, sums = kKGroups * MT * kPartPitch * 4,
                smem = ring > sums ? ring : sums;
  static DeviceOnce once;
  const cudaError_t e = once.run([&] { return cudaFuncSetAttribute(gemm_rows_kernel<NT, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem); });
  if (e != cudaSuccess) return e;
  const int nt = (a.N + kTileN - 1) / kTileN, mt = (a.M + MT - 1) / MT, slabs = (a.K + kSlab - 1) / kSlab;
  const int64_t tiles = static_cast<int64_t>(nt) * mt;
  // pieces of K: the fewest slab times in waves of two blocks per SM, each block counted with 1.5 of them for its start and end
  int per = slabs;
  if (tiles <= kGemmRowsCounters) {
    const int64_t fit = std::min<int64_t>(slabs, kGemmRowsPlaneFloats / (tiles * kTileN * MT));
    double best = 0;
    for (int64_t z = 1; z <= std::min<int64_t>(fit, 32); ++z) {
      const int p = static_cast<int>((slabs + z - 1) / z), blocks = (slabs + p - 1) / p;
      const double cost = static_cast<double>((tiles * blocks + 295) / 296) * (p + 1.5);
      if (z == 1 || cost < best) {
        best = cost;
        per = p;
      }
    }
  }
  return launch_pdl(gemm_rows_kernel<NT, EPI>, dim3(nt, mt, (slabs + per - 1) / per), dim3(kThreads), smem, s, pdl, a, planes, counters, per);
}

template <int EPI>
cudaError_t launch_epi(const GemvArgs& a, float* planes, uint32_t* counters, cudaStream_t s, bool pdl) {
  const int tiles = (a.M + kMaxTileM - 1) / kMaxTileM;
  switch (((a.M + tiles - 1) / tiles + 7) / 8) {               // even tiles: less padding
    case 1: return launch_one<1, EPI>(a, planes, counters, s, pdl);
    case 2: return launch_one<2, EPI>(a, planes, counters, s, pdl);
    case 3: return launch_one<3, EPI>(a, planes, counters, s, pdl);
    default: return launch_one<4, EPI>(a, planes, counters, s, pdl);
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
    case kEpiSoftcap: return launch_epi<kEpiSoftcap>(a, planes, counters, s, pdl);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace mtj
