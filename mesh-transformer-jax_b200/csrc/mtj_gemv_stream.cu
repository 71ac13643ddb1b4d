// The GEMV for one activation row and long weight rows (decoding a single sequence of a layer stack): HBM-bound.
//
// gemv_kernel keeps 64 bytes per thread in flight and starts with an empty pipe in each of its waves of blocks; a product
// of 50 to 180 MB is over after 10 to 30 us, so that ramps and last waves cost a third of it.  Here one block per SM owns a
// run of rows, and each of its 8 warps the same eighth of the columns of all of them: the activations stay in registers.  A ninth warp streams the rows, one bulk copy each, through a ring of 96 KB, filled from before the wait on
// the predecessor (two such blocks fit an SM, so a kernel's ring fills while its predecessor ends).  Whole rows, because
// the copy engine takes about 70 ns for a copy of 1 KB: with a ring per warp and 1 KB pieces 184 MB took 87 us.  No
// block-wide barrier until the rows are done; the 8 partial sums of a row are added in order.
#include <math.h>

#include <algorithm>

#include "mtj_gemv_finish.cuh"

namespace mtj {
namespace {

constexpr int kMinK = 8192, kMaxK = 12288;               // columns of a weight row
constexpr int kRingBytes = 96 * 1024, kMaxRing = kRingBytes / (2 * kMinK);
constexpr int kStreamThreads = kGemvThreads + 32;

__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }

template <int NCH, int EPI>
__global__ void __launch_bounds__(kStreamThreads, 2) gemv_stream_kernel(const GemvArgs a, int ring) {
  extern __shared__ __align__(128) unsigned char stream_smem[];
  __shared__ __align__(8) uint64_t bars[2 * kMaxRing];
  __shared__ float red[kGemvWarps];
  __shared__ bool is_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int vecs = a.K >> 3, per = (vecs + kGemvWarps - 1) / kGemvWarps;          // 16-byte pieces of a row
  const int pairs = a.N >> 1;                                                      // rows go round in pairs
  const int r0 = 2 * static_cast<int>(static_cast<int64_t>(blockIdx.x) * pairs / gridDim.x);
  const int r1 = 2 * static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * pairs / gridDim.x);
  const uint32_t stage = static_cast<uint32_t>(a.K) * 2u;
  float* part = reinterpret_cast<float*>(stream_smem + static_cast<size_t>(ring) * stage);   // [row][warp]
  const uint32_t bar0 = smem_u32(bars), ring0 = smem_u32(stream_smem);
  auto full = [&](int i) { return bar0 + 8u * i; };
  auto empty = [&](int i) { return bar0 + 8u * (kMaxRing + i); };

  if (threadIdx.x == 0) {
    for (int i = 0; i < ring; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), kGemvWarps);
    }
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();
  bool ok = true;
  if (warp == kGemvWarps) {
    if (lane == 0) {
      // row r sits in slot (r - r0) % ring; weights do not depend on the predecessor
      const uint64_t pol = l2_evict_first_policy();
      int slot = 0;
      uint32_t phase = 1;                                        // the first round passes
      for (int r = r0; r < r1 && ok; ++r) {
        ok = mbar_wait(empty(slot), phase);
        if (!ok) break;
        mbar_expect_tx(full(slot), stage);
        bulk_load(ring0 + slot * stage, a.W + static_cast<size_t>(r) * a.K, stage, full(slot), pol);
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
    const int v0 = warp * per, mine = max(0, min(per, vecs - v0));
    const int src = a.row_select ? a.row_select[0] : 0;
    const float* xp = a.x + static_cast<size_t>(src) * a.ldx + v0 * 8 + lane * 8;
    float x[NCH][8];
#pragma unroll
    for (int c = 0; c < NCH; ++c) {
      const bool in = c * 32 + lane < mine;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 v = in ? *reinterpret_cast<const float4*>(xp + c * 256 + 4 * h) : zero;
        x[c][4 * h] = v.x; x[c][4 * h + 1] = v.y; x[c][4 * h + 2] = v.z; x[c][4 * h + 3] = v.w;
      }
    }
    int slot = 0;
    uint32_t phase = 0;
    // the row in the current slot times this warp's columns; hands the slot back
    auto dot = [&]() {
      ok = ok && mbar_wait(full(slot), phase);
      const uint4* rowp = reinterpret_cast<const uint4*>(stream_smem + static_cast<size_t>(slot) * stage) + v0;
      uint4 v[NCH];
#pragma unroll
      for (int c = 0; c < NCH; ++c) v[c] = c * 32 + lane < mine ? rowp[c * 32 + lane] : make_uint4(0u, 0u, 0u, 0u);
      ok = __all_sync(0xffffffffu, ok);
      __syncwarp();                                              // every lane has read the slot (a vote orders no memory)
      if (lane == 0) arrive(empty(slot));
      if (++slot == ring) {
        slot = 0;
        phase ^= 1u;
      }
      float s0 = 0.f, s1 = 0.f;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        float w8[8];
        unpack8(v[c], w8);
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          s0 = fmaf(w8[e], x[c][e], s0);
          s1 = fmaf(w8[e + 1], x[c][e + 1], s1);
        }
      }
      return s0 + s1;
    };
    // two rows' sums at a time; a wait that ran out ends the loop
    for (int r = r0; r < r1; r += 2) {
      float p0 = dot(), p1 = dot();
      if (!ok) break;
      p0 = warp_sum(p0);
      p1 = warp_sum(p1);
      if (lane == 0) {
        part[(r - r0) * kGemvWarps + warp] = p0;
        part[(r - r0 + 1) * kGemvWarps + warp] = p1;
      }
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
      for (int k = 0; k < kGemvWarps; ++k) val += part[i * kGemvWarps + k];
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
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(a.counters, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    if (warp < kGemvWarps) finish_rows(a, 0, 1, red);
    if (threadIdx.x == 0) a.counters[0] = 0u;
  }
}

int blocks_of() {
  int dev = 0, n = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 148;
  return n;
}

template <int NCH, int EPI>
cudaError_t launch_one(const GemvArgs& a, cudaStream_t s, bool pdl) {
  const int ring = kRingBytes / (a.K * 2);
  const int grid = std::min(blocks_of(), a.N / 2), rows = 2 * ((a.N / 2 + grid - 1) / grid);
  const int smem = ring * a.K * 2 + kGemvWarps * rows * 4;
  static DeviceOnce once;
  const cudaError_t e = once.run([&] { return cudaFuncSetAttribute(gemv_stream_kernel<NCH, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); });
  if (e != cudaSuccess) return e;
  return launch_pdl(gemv_stream_kernel<NCH, EPI>, dim3(grid), dim3(kStreamThreads), smem, s, pdl, a, ring);
}

template <int EPI>
cudaError_t launch_epi(const GemvArgs& a, cudaStream_t s, bool pdl) {
  const int chunks = (((a.K >> 3) + kGemvWarps - 1) / kGemvWarps + 31) / 32;      // of 32 pieces, a lane each: 4 to 6
  return chunks <= 4 ? launch_one<4, EPI>(a, s, pdl) : launch_one<6, EPI>(a, s, pdl);
}

}  // namespace

// One row, weight rows of 8192 to 12288 columns (the ring holds six rows or four, a thread's activations its registers),
// and at least four rows per block.  Us a launch in the chained decode step, this kernel and gemv_kernel: 4096 x 8192 with the
// norm behind it 14.5 and 17, 4096 x 12288 21 and 22, SwiGLU 16384 x 8192 46 and 62, squared relu 8192 x 8192 23 and 30, head
// 30002 x 8192 75 and 115.  With 4096 columns a block spends longer on a row's hand-over than its copy takes (32768 x 4096: 56
// and 53; 12288 x 4096: 23.5 and 20.6), and beyond 12288 the activations no longer fit the registers and the ring holds three
// rows (4096 x 13824 40 to 66 and 21, 4096 x 16384 66 and 24), so those stay.
bool gemv_stream_ok(GemvEpilogue epi, const GemvArgs& a) {
  return a.M == 1 && (epi == kEpiOut || epi == kEpiSoftcap || epi == kEpiSwiGLU || epi == kEpiRelu2) && a.K >= kMinK && a.K <= kMaxK &&
         a.N >= 4 * 148 && a.N <= 148 * 2048 && !a.residual && !a.slot_sel && !a.stats_out && a.ks_override == 0;
}

cudaError_t launch_gemv_stream(GemvEpilogue epi, const GemvArgs& a, cudaStream_t s, bool pdl) {
  if (!gemv_stream_ok(epi, a) || (a.K & 7) || (a.N & 1) || (a.ldx & 3)) return cudaErrorInvalidValue;
  switch (epi) {
    case kEpiOut: return launch_epi<kEpiOut>(a, s, pdl);
    case kEpiSwiGLU: return launch_epi<kEpiSwiGLU>(a, s, pdl);
    case kEpiRelu2: return launch_epi<kEpiRelu2>(a, s, pdl);
    default: return launch_epi<kEpiSoftcap>(a, s, pdl);
  }
}

}  // namespace mtj
