// The GEMV for one activation row (decoding a single sequence of a layer stack): HBM-bound.
//
// gemv_kernel keeps 64 bytes per thread in flight and starts with an empty pipe in each of its waves of blocks; a product
// of 25 to 260 MB is over after 4 to 40 us, so that ramps and last waves cost a third of it.  Here one block per SM owns a
// run of rows.  A seventeenth warp streams them in stages of 16 to 32 KB, one row for each group of warps in one bulk copy (rows
// touch), through a ring of 128 KB, filled from before the wait on the predecessor.  One block per SM: with a ring of 96 KB the next product's block
// came in beside this one's, and both streams got slower (a reply of width 4096 24.4 ms, 20.2 with 160 KB, 19.6 with 128).
// The 16 others hold the activations in registers, a warp the same 512 to 1024 columns of every row that its group takes.  No
// block-wide barrier until the rows are done; the partial sums of a row are added in order.  What bounds it beside HBM is the
// number of instructions per byte (packed multiply-adds; two rows' sums cross the warp together) and, where a norm follows, the
// 4 us in which the last block does it.  Us a launch in the chained decode step, the kernels before (gemv_kernel, or a ring of
// 96 KB with scalar arithmetic and a copy per row from 8192 columns on) and this one: SwiGLU 22528 x 4096 35.6 and 26.8, squared
// relu 12288 x 4096 20.7 and 15.1, head 32768 x 4096 55 and 38.6 (6.96 TB/s), 4096 x 12288 with the norm behind it 23.3 and 20.4,
// 4096 x 8192 17.9 and 15.7.
#include <math.h>

#include <algorithm>

#include "mtj_gemv_finish.cuh"

namespace mtj {
namespace {

constexpr int kMinK = 1024, kMaxK = 16384;               // columns of a weight row
constexpr int64_t kMinWeights = 12 << 20;
constexpr int kLongK = 8192, kLeastN = 4 * 148;          // columns and rows from which fewer weights will do
constexpr int kRingBytes = 128 * 1024, kMaxRing = 8;
constexpr int kMaxSmem = 224 * 1024;
constexpr int kW = 16, kStreamThreads = 32 * kW + 32;

__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// two fp32 side by side: what the packed multiply-add takes
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
  return r;
}
__device__ __forceinline__ void fma2(F2& acc, uint32_t w, F2 x) {                 // two bf16 of a word
  F2 v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(w << 16), "r"(w & 0xffff0000u));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(v), "l"(x));
}
__device__ __forceinline__ void dot8(F2& acc, const uint4& w, const F2* x) {
  fma2(acc, w.x, x[0]);
  fma2(acc, w.y, x[1]);
  fma2(acc, w.z, x[2]);
  fma2(acc, w.w, x[3]);
}
__device__ __forceinline__ float sum2(F2 v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return __uint_as_float(lo) + __uint_as_float(hi);
}

// pieces of 8 columns of a lane, groups of warps that take the rows in turn
template <int NCH, int GROUPS, int EPI>
__global__ void __launch_bounds__(kStreamThreads, 1) gemv_stream_kernel(const GemvArgs a, int ring) {
  extern __shared__ __align__(128) unsigned char stream_smem[];
  __shared__ __align__(8) uint64_t bars[2 * kMaxRing];
  __shared__ float red[kW];
  __shared__ bool is_last;
  constexpr int kParts = kW / GROUPS, kPitch = kParts + 1;
  constexpr int kUnit = EPI == kEpiSwiGLU ? 2 : 1;               // rows that have to meet in a block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int vecs = a.K >> 3, per = (vecs + kParts - 1) / kParts;                  // 16-byte pieces of a row, of a warp
  const int units = a.N / kUnit;
  const int r0 = kUnit * static_cast<int>(static_cast<int64_t>(blockIdx.x) * units / gridDim.x);
  const int r1 = kUnit * static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * units / gridDim.x);
  const uint32_t row_bytes = static_cast<uint32_t>(a.K) * 2u, stage = row_bytes * GROUPS;
  float* part = reinterpret_cast<float*>(stream_smem + static_cast<size_t>(ring) * stage);   // [row][kPitch]
  const uint32_t bar0 = smem_u32(bars), ring0 = smem_u32(stream_smem);
  auto full = [&](int i) { return bar0 + 8u * i; };
  auto empty = [&](int i) { return bar0 + 8u * (kMaxRing + i); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < ring; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), kW);
    }
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  bool ok = true;
  int slot = 0;
  if (warp == kW) {
    if (lane == 0) {
      // weights do not depend on the predecessor
      const uint64_t pol = l2_evict_first_policy();
      uint32_t phase = 1;                                        // the first round passes
      for (int r = r0; r < r1 && ok; r += GROUPS) {
        ok = mbar_wait(empty(slot), phase);
        if (!ok) break;
        const uint32_t bytes = row_bytes * min(GROUPS, r1 - r);
        mbar_expect_tx(full(slot), bytes);
        bulk_load(ring0 + slot * stage, a.W + static_cast<size_t>(r) * a.K, bytes, full(slot), pol);
        if (++slot == ring) {
          slot = 0;
          phase ^= 1u;
        }
      }
    }
    pdl_wait();
    pdl_launch_dependents();
  } else {
    pdl_wait();
    pdl_launch_dependents();
    const int grp = warp / kParts, v0 = warp % kParts * per, mine = max(0, min(per, vecs - v0));
    const int src = a.row_select ? a.row_select[0] : 0;
    const float* xp = a.x + static_cast<size_t>(src) * a.ldx + v0 * 8 + lane * 8;
    F2 x[NCH][4];
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const bool in = c * 32 + lane < mine;
      const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
      const float4 lo = in ? *reinterpret_cast<const float4*>(xp + c * 256) : zero, hi = in ? *reinterpret_cast<const float4*>(xp + c * 256 + 4) : zero;
      x[c][0] = pack2(lo.x, lo.y); x[c][1] = pack2(lo.z, lo.w); x[c][2] = pack2(hi.x, hi.y); x[c][3] = pack2(hi.z, hi.w);
    }
    uint32_t phase = 0;
    auto dot = [&]() {                                           // this group's row of the next stage
      ok = __all_sync(0xffffffffu, mbar_wait(full(slot), phase));
      const uint4* row = reinterpret_cast<const uint4*>(stream_smem + static_cast<size_t>(slot) * stage) + grp * vecs + v0 + lane;
      F2 t0 = 0ull, t1 = 0ull;
      uint4 v[NCH];
#pragma unroll
      for (int c = 0; c < NCH; ++c) v[c] = c * 32 + lane < mine ? row[c * 32] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int c = 0; c < NCH; ++c) dot8(c & 1 ? t1 : t0, v[c], x[c]);
      const float sum = sum2(t0) + sum2(t1);
      // Every lane has the row in its registers: which lane hands the stage back hangs on every lane's sum, because an arrival
      // alone does not wait for loads that nothing has used yet, and the next rows would land under them.
      const int by = __any_sync(0xffffffffu, __float_as_uint(sum) == 0x7fc0dead) ? 1 : 0;
      if (lane == by) arrive(empty(slot));
      if (++slot == ring) {
        slot = 0;
        phase ^= 1u;
      }
      return sum;
    };
    // two rows' sums at a time: the first in lanes 0 to 15, the second in lanes 16 to 31; a wait that ran out ends the loop
    for (int r = r0 + grp; r < r1; r += 2 * GROUPS) {
      const float s0 = dot();
      float s1 = 0.f;
      const bool two = ok && r + GROUPS < r1;
      if (two) s1 = dot();
      if (!ok) break;
      float v = lane & 16 ? s1 : s0;
      v += __shfl_xor_sync(0xffffffffu, lane & 16 ? s0 : s1, 16);
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if ((lane & 15) == 0 && (lane == 0 || two)) part[(r - r0 + (lane >> 4) * GROUPS) * kPitch + warp % kParts] = v;
    }
  }
  if (!ok && lane == 0 && a.dev_err) atomicOr(a.dev_err, kDevErrTimeout);
  if (__syncthreads_or(!ok)) {
    // some wait ran out: what is still in flight gets another bounded chance to land before the block leaves
    if (threadIdx.x == 0)
      for (int i = 0; i < ring; ++i) {
        mbar_wait(full(i), 0);
        mbar_wait(full(i), 1);
      }
    __syncthreads();
  }
  const int n_valid = a.n_valid > 0 ? a.n_valid : a.N;
  for (int i = threadIdx.x; i < ((r1 - r0 + 31) & ~31); i += kStreamThreads) {    // whole warps: pairs meet by shuffle
    float val = 0.f;
    if (i < r1 - r0) {
#pragma unroll
      for (int k = 0; k < kParts; ++k) val += part[i * kPitch + k];
    }
    const float partner = __shfl_xor_sync(0xffffffffu, val, 1);
    const int n = r0 + i;
    if (i >= r1 - r0 || n >= n_valid) continue;
    if (EPI == kEpiSwiGLU) {
      if (!(n & 1)) a.act2[n >> 1] = val / (1.0f + expf(-val)) * partner;
    } else if (EPI == kEpiRelu2) {
      const float y = fmaxf(val, 0.f);
      a.act2[n] = y * y;
    } else {
      a.out[n] = EPI == kEpiSoftcap ? a.softcap * tanhf(val / a.softcap) : a.bias ? val + a.bias[n] : val;
    }
  }
  if (EPI == kEpiOut && a.post_w) {
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();                                           // what the block has stored, behind the barrier
      is_last = atomicAdd(a.counters, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (warp < kW) finish_row<32 * kW>(a, red);
    if (threadIdx.x == 0) a.counters[0] = 0u;
  }
}

int blocks_of() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return n;
}

// Groups of warps that take the rows in turn, so that a warp has 512 to 1024 columns of a row.  256 to 512 instead: a reply of
// width 4096 19.08 ms, 18.81 so; 256 at width 2048: 19.6 ms where gemv_kernel takes 17.8 and this division 16.8.
int groups_of(int K) { return K <= 1024 ? 16 : K <= 2048 ? 8 : K <= 4096 ? 4 : K <= 8192 ? 2 : 1; }

struct StreamPlan {
  int grid, ring, smem;
};
StreamPlan plan_of(GemvEpilogue epi, const GemvArgs& a) {
  const int unit = epi == kEpiSwiGLU ? 2 : 1, groups = groups_of(a.K);
  StreamPlan p;
  p.grid = std::min(blocks_of(), a.N / unit);
  p.ring = std::min(kMaxRing, kRingBytes / (2 * a.K * groups));
  const int most = unit * ((a.N / unit + p.grid - 1) / p.grid);
  p.smem = p.ring * groups * a.K * 2 + (kW / groups + 1) * most * 4;
  p.smem = std::max(p.smem, 116 * 1024);                         // one block per SM
  return p;
}

template <int NCH, int GROUPS, int EPI>
cudaError_t launch_one(const GemvArgs& a, const StreamPlan& p, cudaStream_t s, bool pdl) {
  static DeviceOnce once;
  const cudaError_t e = once.run([&] { return cudaFuncSetAttribute(gemv_stream_kernel<NCH, GROUPS, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem); });
  if (e != cudaSuccess) return e;
  return launch_pdl(gemv_stream_kernel<NCH, GROUPS, EPI>, dim3(p.grid), dim3(kStreamThreads), p.smem, s, pdl, a, p.ring);
}

template <int EPI>
cudaError_t launch_epi(const GemvArgs& a, cudaStream_t s, bool pdl) {
  const StreamPlan p = plan_of(static_cast<GemvEpilogue>(EPI), a);
  switch (groups_of(a.K)) {
    case 16: return launch_one<4, 16, EPI>(a, p, s, pdl);
    case 8: return launch_one<4, 8, EPI>(a, p, s, pdl);
    case 4: return launch_one<4, 4, EPI>(a, p, s, pdl);
    case 2: return launch_one<4, 2, EPI>(a, p, s, pdl);
    default: return a.K <= 12288 ? launch_one<3, 1, EPI>(a, p, s, pdl) : launch_one<4, 1, EPI>(a, p, s, pdl);
  }
}

}  // namespace

// One row and weights of 25 MB and more: below, the stream is over before its ring has paid for its setup (products of 8 to 24 MB
// this way too: a reply of a model of width 1024 12.0 ms against 11.8, of 2048 17.0 against 16.8 or 18.0 against 18.2).  Rows of
// 8192 columns and more earlier, from four a block on: gemv_kernel has few such rows to spread (down projections of six layers, us a
// step by gemv_kernel and this way: 600 x 8192 167 and 163, 600 x 12288 186 and 174, 768 x 12288 186 and 176, 1024 x 8192 171 and
// 174 with one family, 190 and 187 with the other).  The columns are what the warps' registers hold.
bool gemv_stream_ok(GemvEpilogue epi, const GemvArgs& a) {
  if ((a.K & 7) || (a.N & 1) || (a.ldx & 3)) return false;      // 16-byte pieces of both operands, pairs of rows
  return a.M == 1 && (epi == kEpiOut || epi == kEpiSoftcap || epi == kEpiSwiGLU || epi == kEpiRelu2) && a.K >= kMinK && a.K <= kMaxK &&
         (static_cast<int64_t>(a.N) * a.K >= kMinWeights || (a.K >= kLongK && a.N >= kLeastN)) && !a.residual && !a.slot_sel && !a.stats_out && a.ks_override == 0 && plan_of(epi, a).smem <= kMaxSmem;
}

cudaError_t launch_gemv_stream(GemvEpilogue epi, const GemvArgs& a, cudaStream_t s, bool pdl) {
  if (!gemv_stream_ok(epi, a)) return cudaErrorInvalidValue;
  switch (epi) {
    case kEpiOut: return launch_epi<kEpiOut>(a, s, pdl);
    case kEpiSwiGLU: return launch_epi<kEpiSwiGLU>(a, s, pdl);
    case kEpiRelu2: return launch_epi<kEpiRelu2>(a, s, pdl);
    default: return launch_epi<kEpiSoftcap>(a, s, pdl);
  }
}

}  // namespace mtj
