// The whole decode step of one sequence on one GPU as one persistent kernel, as mtj_decode_mega.cu, with the weights on a
// stream of their own.  Each block (one per SM) has four kinds of warps:
//   1 producer    walks the block's weight rows of the whole step, in the order in which they are used, through a ring of 160 KB
//                 in shared memory; it waits for free slots only, so HBM keeps working while the block waits for other blocks
//   16 streaming  multiply the ring's rows by activations that they hold in registers (a warp the same columns of every row) and
//                 leave partial sums in shared memory
//   3 finishing   finish rows (bias, rotation, cache writes, GELU, residual) and tell the other blocks
//   8 attending   one (head, key range) per block, the last one of a head merges
// The streaming warps wait for other blocks at four places per layer, of which the first alone is felt:
//     x of the layer      all rows of the last out-projection: as far as the pause outlasts the ring (3.4 us)
//     FF-in rows          in two halves: the first half's are finished everywhere while the second half's rows stream, the
//                         second half's while the out-projection's columns of the first half stream
//     attention           begins behind the Q/K/V rows, which come first, and is over when the FF-in rows and the FF columns of the
//                         out-projection have streamed; its columns come last
// Hand-overs are arrival counters as in decode_mega_kernel, every wait is bounded.  A block owns runs of rows, dealt evenly.
// What bounds it: HBM (403 MB of weights per layer of GPT-J-6B, 58 us at the 6.9 TB/s that this stream reaches), then the pause
// at x.  GPT-J-6B, us per layer with 137 / 2048 cached keys: decode_mega_kernel, whose warps stop loading in every epilogue, wait
// and attention, 76.2 / 88.5; this kernel 64.2 / 75.2 (a step 2196 -> 1857 and 2544 -> 2168 us).  On the way here: no side warps
// 98; 16 KB stages and scalar multiply-adds 101 (the streaming warps were bound by instructions); FF-in rows first, attention
// last 64.7 / 82.2; FF-in rows in one piece 66.9 / 77.3.
#include <math.h>

#include <algorithm>

#include "mtj_common.cuh"
#include "mtj_kernels.h"

namespace mtj {
namespace {

constexpr int kW = 16, kT = 32 * kW;                          // streaming warps and threads
constexpr int kEpiW = 3, kEpiT = 32 * kEpiW;                  // finishing warps and threads
constexpr int kAttW = 8, kAttT = 32 * kAttW;                  // attending warps and threads
constexpr int kThreads = kT + kEpiT + kAttT + 32;             // 28 warps: 72 registers a thread, no spills
constexpr int kRing = 5;
constexpr uint32_t kStage = 32 * 1024;
constexpr int kMaxD = 4096, kMaxFf = 16384;                   // columns that the warps' registers hold
constexpr int kMinD = 1024, kMaxSmem = 200 * 1024;            // see decode_stream_ok
constexpr int kInPitch = 9, kOutPitch = 49;                   // partial sums of a row: 8 warps; 16 for each half of FF and attention

__device__ __forceinline__ void cbar() { asm volatile("bar.sync 1, %0;" ::"n"(kT) : "memory"); }          // streaming warps
__device__ __forceinline__ void ebar() { asm volatile("bar.sync 2, %0;" ::"n"(kEpiT) : "memory"); }       // finishing warps
__device__ __forceinline__ void abar() { asm volatile("bar.sync 7, %0;" ::"n"(kAttT) : "memory"); }       // attending warps
// partial sums of product k are in place: the streaming warps go on, the finishing warps take over
template <int K>
__device__ __forceinline__ void hand_over() { asm volatile("bar.arrive %0, %1;" ::"n"(3 + K), "n"(kT + kEpiT) : "memory"); }
template <int K>
__device__ __forceinline__ void take_over() { asm volatile("bar.sync %0, %1;" ::"n"(3 + K), "n"(kT + kEpiT) : "memory"); }
__device__ __forceinline__ void arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_ready(uint32_t bar, uint32_t parity) {
  uint32_t done;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done;
}
__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void stamp(unsigned long long* t, int slot) {
  if (t && blockIdx.x == 0 && (threadIdx.x == 0 || threadIdx.x == kT)) {
    unsigned long long v;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v));
    t[slot] = v;
  }
}
// one thread of a group, behind a barrier of the group: everything the group has written is there
__device__ __forceinline__ void phase_arrive(uint32_t* counter) {
  __threadfence();
  atomicAdd(counter, 1u);
}
// one thread of a group waits (bounded) until all blocks have arrived; a barrier of the group follows
__device__ __forceinline__ void phase_poll(const uint32_t* counter, uint32_t target, uint32_t* dev_err, int limit) {
  int spins = 0;
  while (ld_acquire(counter) < target) {
    if (++spins > limit) {
      if (dev_err) atomicOr(dev_err, kDevErrTimeout);
      break;
    }
  }
  __threadfence();
}
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  cbar();
  float t = 0.f;
#pragma unroll
  for (int i = 0; i < kW; ++i) t += red[i];
  cbar();
  return t;
}
// two fp32 side by side: what the packed multiply-add takes
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
  return r;
}
__device__ __forceinline__ F2 widen(uint32_t w) {                             // two bf16 of a word
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(w << 16), "r"(w & 0xffff0000u));
  return r;
}
__device__ __forceinline__ void fma2(F2& acc, F2 a, F2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ float sum2(F2 v) {
  uint32_t lo, hi;
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
  return __uint_as_float(lo) + __uint_as_float(hi);
}
__device__ __forceinline__ void load8(const float* p, F2* f) {               // written by other blocks: from L2
  const float4 a = __ldcg(reinterpret_cast<const float4*>(p)), b = __ldcg(reinterpret_cast<const float4*>(p) + 1);
  f[0] = pack2(a.x, a.y); f[1] = pack2(a.z, a.w); f[2] = pack2(b.x, b.y); f[3] = pack2(b.z, b.w);
}
__device__ __forceinline__ void dot8(F2& acc, const uint4& w, const F2* x) {
  fma2(acc, widen(w.x), x[0]);
  fma2(acc, widen(w.y), x[1]);
  fma2(acc, widen(w.z), x[2]);
  fma2(acc, widen(w.w), x[3]);
}
// sums over the warp of two numbers: the first in lanes 0 to 15, the second in lanes 16 to 31
__device__ __forceinline__ float warp_sum2(float a, float b, int lane) {
  float v = lane & 16 ? b : a;
  v += __shfl_xor_sync(0xffffffffu, lane & 16 ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// rows [lo, hi) that this block owns of n rows from `first` on, dealt in units of `unit`
struct Span {
  int lo, hi;
};
__device__ __forceinline__ Span span_of(int first, int n, int unit) {
  const int u = n / unit;
  return {first + unit * static_cast<int>(static_cast<int64_t>(blockIdx.x) * u / gridDim.x), first + unit * static_cast<int>(static_cast<int64_t>(blockIdx.x + 1) * u / gridDim.x)};
}

template <int DH>
__global__ void __launch_bounds__(kThreads, 1) decode_stream_kernel(const MegaArgs a) {
  extern __shared__ __align__(128) unsigned char ds_smem[];
  __shared__ __align__(8) uint64_t bars[2 * kRing];
  __shared__ float red[kW];
  constexpr int kSide = 256 / DH, kParts = kAttW * kSide;        // keys side by side in a warp (a lane holds 8 columns), partial results
  __shared__ float sm_m[kParts], sm_l[kParts], sm_o[kParts][DH];
  __shared__ float wgt[64], inv_l;
  __shared__ bool is_last, merges;                               // the step's last block; the last block of a head
  __shared__ unsigned long long blk_amax;
  __shared__ uint32_t failed;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int d = a.d, dl = a.dl, ffl = a.ffl, L = a.L, K2 = dl + ffl;
  const uint32_t ring0 = smem_u32(ds_smem), bar0 = smem_u32(bars);
  auto full = [&](int i) { return bar0 + 8u * i; };
  auto empty = [&](int i) { return bar0 + 8u * (kRing + i); };
  volatile uint32_t* failed_v = &failed;
  // what this block owns, and rows per stage
  const int half = ffl / 2 & ~7;                                 // FF features of the first half
  const Span qkv = span_of(0, 3 * dl, 2), ff1 = span_of(0, half, 2), ff2 = span_of(half, ffl - half, 2), out = span_of(0, d, 1), voc = span_of(0, a.V, 2);
  const int in_rows = 2 * max(1, static_cast<int>(kStage) / (4 * d));
  const int ff_rows = max(1, static_cast<int>(kStage) / (2 * (ffl - half)));
  const int at_rows = max(1, static_cast<int>(kStage) / (2 * dl));
  // partial sums: FF-in rows of both halves (or logits), then Q/K/V rows, then the out-projection's
  float* part_ff = reinterpret_cast<float*>(ds_smem + kRing * kStage);
  float* part_ff2 = part_ff + (ff1.hi - ff1.lo) * kInPitch;
  float* part_qkv = part_ff + a.part_rows[0] * kInPitch;
  float* part_out = part_qkv + a.part_rows[1] * kInPitch;
  const uint32_t target = gridDim.x;
  uint32_t *c_x = a.sync, *c_qkv = a.sync + (L + 1), *c_af = a.sync + (2 * L + 1), *c_ff = a.sync + (3 * L + 1), *c_ff2 = a.sync + (4 * L + 2);
  const int cur = *a.cur;                                        // absolute position of this step's token

  if (threadIdx.x == 0) {
    for (int i = 0; i < kRing; ++i) {
      mbar_init(full(i), 1);
      mbar_init(empty(i), kW);
    }
    mbar_fence_init();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    failed = 0;
    blk_amax = 0ull;
  }
  __syncthreads();

  if (warp == kW + kEpiW + kAttW) {
    // ------------------------------------------------------------------------------------ the weight stream
    if (lane == 0) {
      const uint64_t pol = l2_evict_first_policy();
      int slot = 0;
      uint32_t phase = 1;                                        // the first round passes
      // a stage of n rows of `cols` columns, `ld` apart (rows that touch: one copy)
      auto push = [&](const __nv_bfloat16* w, int n, int cols, int ld) {
        if (*failed_v) return;
        if (!mbar_wait(empty(slot), phase)) {
          *failed_v = 1;
          return;
        }
        const uint32_t bytes = 2u * cols, dst = ring0 + slot * kStage;
        mbar_expect_tx(full(slot), n * bytes);
        if (cols == ld) bulk_load(dst, w, n * bytes, full(slot), pol);
        else
          for (int r = 0; r < n; ++r) bulk_load(dst + r * bytes, w + static_cast<size_t>(r) * ld, bytes, full(slot), pol);
        if (++slot == kRing) {
          slot = 0;
          phase ^= 1u;
        }
      };
      auto whole = [&](const __nv_bfloat16* w, Span s) {
        for (int r = s.lo; r < s.hi; r += in_rows) push(w + static_cast<size_t>(r) * d, min(in_rows, s.hi - r), d, d);
      };
      for (int l = 0; l < L; ++l) {
        const __nv_bfloat16 *w_in = a.layers[l].w_in, *w_out = a.layers[l].w_out;
        whole(w_in, qkv);
        whole(w_in + static_cast<size_t>(3 * dl) * d, ff1);
        whole(w_in + static_cast<size_t>(3 * dl) * d, ff2);
        for (int r = out.lo; r < out.hi; r += ff_rows) push(w_out + static_cast<size_t>(r) * K2 + dl, min(ff_rows, out.hi - r), half, K2);
        for (int r = out.lo; r < out.hi; r += ff_rows) push(w_out + static_cast<size_t>(r) * K2 + dl + half, min(ff_rows, out.hi - r), ffl - half, K2);
        for (int r = out.lo; r < out.hi; r += at_rows) push(w_out + static_cast<size_t>(r) * K2, min(at_rows, out.hi - r), dl, K2);
      }
      whole(a.proj_w, voc);
    }
    __syncwarp();
  } else if (warp < kW) {
    // ------------------------------------------------------------------------------------ streaming warps
    int slot = 0;
    uint32_t phase = 0;
    auto await = [&]() -> const unsigned char* {                 // the stage that is next
      if (!mbar_ready(full(slot), phase) && !*failed_v && !mbar_wait(full(slot), phase)) *failed_v = 1;
      return ds_smem + slot * kStage;
    };
    // Hands the stage back.  In front of it stands the store of the last sums, which hangs on a shuffle over what every lane has made
    // of the stage: that, and not the barrier, has waited for the loads (an arrival alone does not wait for loads that nothing has
    // used yet), so the reduction has to stay in front.
    auto release = [&]() {
      __syncwarp();
      if (lane == 0) arrive(empty(slot));
      if (++slot == kRing) {
        slot = 0;
        phase ^= 1u;
      }
    };
    auto phase_wait = [&](const uint32_t* counter) {
      if (threadIdx.x == 0) phase_poll(counter, target, a.dev_err, a.wait_limit);
      cbar();
    };
    // products with d columns: two groups of 8 warps take the rows in turn, a warp an eighth of the columns
    const int grp = warp >> 3, vecs = d >> 3, per = (vecs + 7) >> 3, v0 = (warp & 7) * per, mine = max(0, min(per, vecs - v0));
    F2 x[2][4];
    // x = layer norm of the residual row (this warp's columns); the norm's weights are loaded before the row is there
    auto normed = [&](const float* scale, const float* offset, const uint32_t* ready) {
      float sc[2][8], of[2][8], v[2][8];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
#pragma unroll
        for (int e = 0; e < 8; ++e) v[c][e] = sc[c][e] = of[c][e] = 0.f;
        if (c * 32 + lane < mine) {
          const int at = (v0 + c * 32 + lane) * 8;
          const float4 *s4 = reinterpret_cast<const float4*>(scale + at), *o4 = reinterpret_cast<const float4*>(offset + at);
          const float4 s0 = s4[0], s1 = s4[1], o0 = o4[0], o1 = o4[1];
          sc[c][0] = s0.x; sc[c][1] = s0.y; sc[c][2] = s0.z; sc[c][3] = s0.w; sc[c][4] = s1.x; sc[c][5] = s1.y; sc[c][6] = s1.z; sc[c][7] = s1.w;
          of[c][0] = o0.x; of[c][1] = o0.y; of[c][2] = o0.z; of[c][3] = o0.w; of[c][4] = o1.x; of[c][5] = o1.y; of[c][6] = o1.z; of[c][7] = o1.w;
        }
      }
      phase_wait(ready);
      float s = 0.f, q = 0.f;
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (c * 32 + lane < mine) {
          const float4* p = reinterpret_cast<const float4*>(a.x + (v0 + c * 32 + lane) * 8);
          const float4 x0 = __ldcg(p), x1 = __ldcg(p + 1);
          v[c][0] = x0.x; v[c][1] = x0.y; v[c][2] = x0.z; v[c][3] = x0.w; v[c][4] = x1.x; v[c][5] = x1.y; v[c][6] = x1.z; v[c][7] = x1.w;
        }
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 8; ++e) s += v[c][e];
      const float mu = block_sum(grp == 0 ? s : 0.f, red) / static_cast<float>(d);       // both groups hold the row
#pragma unroll
      for (int c = 0; c < 2; ++c)
        if (c * 32 + lane < mine)
#pragma unroll
          for (int e = 0; e < 8; ++e) q = fmaf(v[c][e] - mu, v[c][e] - mu, q);
      const float rstd = 1.0f / sqrtf(block_sum(grp == 0 ? q : 0.f, red) / static_cast<float>(d) + 1e-5f);
#pragma unroll
      for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int e = 0; e < 8; e += 2)
          x[c][e >> 1] = pack2(fmaf(sc[c][e] * rstd, v[c][e] - mu, of[c][e]), fmaf(sc[c][e + 1] * rstd, v[c][e + 1] - mu, of[c][e + 1]));
    };
    // the stream's next rows times x
    auto rows_times_x = [&](Span s, float* part) {
      for (int r0 = s.lo; r0 < s.hi; r0 += in_rows) {
        const uint4* st = reinterpret_cast<const uint4*>(await());
        const int n = min(in_rows, s.hi - r0);
        float* p = part + (r0 - s.lo) * kInPitch + (warp & 7);
        for (int r = grp; r < n; r += 4) {                       // rows r and r + 2 (a stage holds an even number)
          const uint4* row = st + r * vecs + v0;
          const bool two = r + 2 < n;
          F2 t0 = 0ull, t1 = 0ull;
#pragma unroll
          for (int c = 0; c < 2; ++c)
            if (c * 32 + lane < mine) {
              dot8(t0, row[c * 32 + lane], x[c]);
              if (two) dot8(t1, row[2 * vecs + c * 32 + lane], x[c]);
            }
          const float v = warp_sum2(sum2(t0), sum2(t1), lane);
          if ((lane & 15) == 0 && (lane == 0 || two)) p[(r + (lane >> 3)) * kInPitch] = v;
        }
        release();
      }
    };
    for (int l = 0; l < L; ++l) {
      const MegaLayer& lw = a.layers[l];
      normed(lw.ln_scale, lw.ln_offset, c_x + l);
      stamp(a.trace, 6 * l + 1);
      rows_times_x(qkv, part_qkv);
      hand_over<1>();
      rows_times_x(ff1, part_ff);
      hand_over<0>();
      rows_times_x(ff2, part_ff2);
      hand_over<3>();
      // out-projection of this block's rows: the FF columns in two halves, then the attention columns
#pragma unroll 1
      for (int k = 0; k < 3; ++k) {
        const int col0 = k == 0 ? dl : k == 1 ? dl + half : 0, cols = k == 0 ? half : k == 1 ? ffl - half : dl, step = k == 2 ? at_rows : ff_rows;
        const int pv = cols >> 3, pp = (pv + kW - 1) / kW, pv0 = warp * pp, pm = max(0, min(pp, pv - pv0));
        F2 xo[2][4];
        phase_wait(k == 0 ? c_ff + l : k == 1 ? c_ff2 + l : c_af + l);
        if (k == 0) stamp(a.trace, 6 * l + 2);
        if (k != 1) stamp(a.trace, 6 * l + 3 + k / 2);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
#pragma unroll
          for (int e = 0; e < 4; ++e) xo[c][e] = 0ull;
          if (c * 32 + lane < pm) load8(a.act2 + col0 + (pv0 + c * 32 + lane) * 8, xo[c]);
        }
        for (int r0 = out.lo; r0 < out.hi; r0 += step) {
          const uint4* st = reinterpret_cast<const uint4*>(await()) + pv0;
          const int n = min(step, out.hi - r0);
          float* p = part_out + (r0 - out.lo) * kOutPitch + k * kW + warp;
          for (int r = 0; r < n; r += 2) {
            const bool two = r + 1 < n;
            F2 t0 = 0ull, t1 = 0ull;
#pragma unroll
            for (int c = 0; c < 2; ++c)
              if (c * 32 + lane < pm) {
                dot8(t0, st[r * pv + c * 32 + lane], xo[c]);
                if (two) dot8(t1, st[(r + 1) * pv + c * 32 + lane], xo[c]);
              }
            const float v = warp_sum2(sum2(t0), sum2(t1), lane);
            if ((lane & 15) == 0 && (lane == 0 || two)) p[(r + (lane >> 4)) * kOutPitch] = v;
          }
          release();
        }
      }
      hand_over<2>();
      stamp(a.trace, 6 * l + 5);
    }
    normed(a.lnf_scale, a.lnf_offset, c_x + L);
    stamp(a.trace, 6 * L + 1);
    rows_times_x(voc, part_ff);
    hand_over<0>();
  } else if (warp < kW + kEpiW) {
    // ------------------------------------------------------------------------------------ finishing warps
    const int t = threadIdx.x - kT;
    auto arrive_at = [&](uint32_t* counter) {
      ebar();
      if (t == 0) phase_arrive(counter);
    };
    // epi(row, value, value of the other row of the pair) on one thread each
    auto finish_rows = [&](Span s, const float* part, auto epi) {
      const int n = s.hi - s.lo;
      for (int i = t; i < ((n + 31) & ~31); i += kEpiT) {
        float val = 0.f;
        if (i < n) {
#pragma unroll
          for (int k = 0; k < 8; ++k) val += part[i * kInPitch + k];
        }
        const float partner = __shfl_xor_sync(0xffffffffu, val, 1);
        if (i < n) epi(s.lo + i, val, partner);
      }
    };
    {
      // embedding: every block its own residual rows
      const int64_t id = static_cast<int64_t>(a.tokens[0]) - a.vocab_start;
      const bool hit = id >= 0 && id < a.V;
      const __nv_bfloat16* row = a.emb_w + static_cast<size_t>(hit ? id : 0) * d;
      for (int i = out.lo + t; i < out.hi; i += kEpiT) a.x[i] = (hit ? __bfloat162float(row[i]) : 0.f) + a.emb_b[i];
    }
    arrive_at(c_x);
    for (int l = 0; l < L; ++l) {
      const MegaLayer& lw = a.layers[l];
      stamp(a.trace, 6 * l + 0);
      take_over<1>();
      finish_rows(qkv, part_qkv, [&](int n, float val, float partner) {
        const int region = n / dl, nn = n - region * dl, h = nn / DH, j = nn % DH;
        float y = val;
        if (region < 2 && j < a.rot) {
          const float2 sc = a.sincos[static_cast<size_t>(cur) * (a.rot >> 1) + (j >> 1)];
          y = (j & 1) ? (val * sc.y + partner * sc.x) : (val * sc.y - partner * sc.x);
        }
        if (region == 0) {
          a.q[nn] = y;
        } else if (cur >= a.pad[0]) {
          __nv_bfloat16* pool = region == 1 ? lw.kpool : lw.vpool;
          pool[kv_offset(a.page_table, a.ring_pages, a.heads, DH, h, cur) + j] = __float2bfloat16_rn(y);
        }
      });
      arrive_at(c_qkv + l);
      take_over<0>();
      finish_rows(ff1, part_ff, [&](int f, float val, float) { a.act2[dl + f] = gelu_tanh(val + lw.b_ff[f]); });
      arrive_at(c_ff + l);
      take_over<3>();
      finish_rows(ff2, part_ff2, [&](int f, float val, float) { a.act2[dl + f] = gelu_tanh(val + lw.b_ff[f]); });
      arrive_at(c_ff2 + l);
      // out-projection: bias + residual, a thread's first row of both there before the sums are (the next layer waits for this)
      const bool owns = t < out.hi - out.lo;
      const float res0 = owns ? a.x[out.lo + t] + lw.b_out[out.lo + t] : 0.f;   // written by this thread before
      take_over<2>();
      for (int i = t; i < out.hi - out.lo; i += kEpiT) {
        float val[3] = {};
#pragma unroll
        for (int k = 0; k < kW; ++k)
#pragma unroll
          for (int j = 0; j < 3; ++j) val[j] += part_out[i * kOutPitch + j * kW + k];
        a.x[out.lo + i] = val[0] + val[1] + val[2] + (i == t ? res0 : a.x[out.lo + i] + lw.b_out[out.lo + i]);
      }
      arrive_at(c_x + l + 1);
    }
    stamp(a.trace, 6 * L + 0);
    // logits and the greedy token
    take_over<0>();
    unsigned long long best = 0ull;
    finish_rows(voc, part_ff, [&](int n, float val, float) {
      float y = val + a.proj_b[n];
      a.logits[n] = y;
      // (order key, index): the arg-max, highest index among equal logits
      if (y == 0.0f) y = 0.0f;                                   // -0 and +0 compare equal
      uint32_t k = __float_as_uint(y);
      k = (k & 0x80000000u) ? ~k : (k | 0x80000000u);
      const unsigned long long cand = (static_cast<unsigned long long>(k) << 32) | static_cast<uint32_t>(n);
      best = cand > best ? cand : best;
    });
    if (a.amax) {
#pragma unroll
      for (int o2 = 16; o2 > 0; o2 >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o2);
        best = other > best ? other : best;
      }
      if (lane == 0 && best) atomicMax(&blk_amax, best);
    }
    ebar();
    stamp(a.trace, 6 * L + 2);
  } else {
    // ------------------------------------------------------------------------------------ attending warps
    // block = (head, one of `splits` ranges of the keys that are there), all blocks as far as there are keys
    const int t = threadIdx.x - kT - kEpiT, sw = warp - kW - kEpiW;
    const int splits = a.grid_splits, split = static_cast<int>(blockIdx.x) % splits, head = static_cast<int>(blockIdx.x) / splits;
    const int start = max(a.pad[0], cur - a.window + 1), len = cur + 1 - start;
    const int range = max(2 * kParts, (len + splits - 1) / splits), nsplit = (len + range - 1) / range;
    const bool attends = head < a.heads && split < nsplit;
    const int t0 = start + split * range, t1 = min(cur + 1, t0 + range);
    for (int l = 0; l < L; ++l) {
      const MegaLayer& lw = a.layers[l];
      if (attends) {
        // towards L2 while the projections stream: the keys and values of this block, all but the newest
        constexpr int kLines = DH * 2 / 128;
        for (int i = t; i < (min(t1, cur) - t0) * kLines; i += kAttT) {
          const size_t off = kv_offset(a.page_table, a.ring_pages, a.heads, DH, head, t0 + i / kLines) + (i % kLines) * 64;
          prefetch_l2(lw.kpool + off);
          prefetch_l2(lw.vpool + off);
        }
      }
      if (attends) {                                             // uniform for the block
        if (t == 0) phase_poll(c_qkv + l, target, a.dev_err, a.wait_limit);
        abar();
        constexpr int TB = 4, kLanes = DH / 8;                   // rounds of a batch, lanes of a key
        const int side = lane / kLanes, col = lane % kLanes * 8;
        constexpr float scale = DH == 256 ? 0.0625f : 0.125f;    // 1 / sqrt(d_head), exact
        float q[8], m = -INFINITY, lsum = 0.f, o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          q[e] = __ldcg(a.q + head * DH + col + e) * scale;
          o[e] = 0.f;
        }
        const int share = (t1 - t0 + kAttW - 1) / kAttW, w0 = t0 + sw * share, w1 = min(t1, w0 + share);
        for (int tb = w0; tb < w1; tb += TB * kSide) {
          uint4 kraw[TB], vraw[TB];
#pragma unroll
          for (int k = 0; k < TB; ++k) {
            const size_t off = kv_offset(a.page_table, a.ring_pages, a.heads, DH, head, min(tb + k * kSide + side, w1 - 1)) + col;
            kraw[k] = ld_cached16(lw.kpool + off);
            vraw[k] = ld_cached16(lw.vpool + off);
          }
          float sc[TB];
#pragma unroll
          for (int k = 0; k < TB; ++k) {
            float kf[8];
            unpack8(kraw[k], kf);
            sc[k] = 0.f;
#pragma unroll
            for (int e = 0; e < 8; ++e) sc[k] = fmaf(q[e], kf[e], sc[k]);
          }
#pragma unroll
          for (int o2 = kLanes / 2; o2 > 0; o2 >>= 1)
#pragma unroll
            for (int k = 0; k < TB; ++k) sc[k] += __shfl_xor_sync(0xffffffffu, sc[k], o2);
          float mn = m;
#pragma unroll
          for (int k = 0; k < TB; ++k)
            if (tb + k * kSide + side < w1) mn = fmaxf(mn, sc[k]);
          const float corr = m == -INFINITY ? 0.f : __expf(m - mn);
          lsum *= corr;
#pragma unroll
          for (int e = 0; e < 8; ++e) o[e] *= corr;
#pragma unroll
          for (int k = 0; k < TB; ++k) {
            if (tb + k * kSide + side >= w1) continue;
            const float p = __expf(sc[k] - mn);
            float vf[8];
            unpack8(vraw[k], vf);
            lsum += p;
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = fmaf(p, vf[e], o[e]);
          }
          m = mn;
        }
        if (lane % kLanes == 0) {
          sm_m[sw * kSide + side] = m;
          sm_l[sw * kSide + side] = lsum;
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) sm_o[sw * kSide + side][col + e] = o[e];
        abar();
        const size_t pbase = static_cast<size_t>(head) * a.max_splits;
        if (t < DH) {
          float M = -INFINITY, Ls = 0.f, O = 0.f;
#pragma unroll
          for (int w = 0; w < kParts; ++w) M = fmaxf(M, sm_m[w]);
#pragma unroll
          for (int w = 0; w < kParts; ++w) {
            const float f = sm_m[w] == -INFINITY ? 0.f : __expf(sm_m[w] - M);     // no key
            Ls = fmaf(sm_l[w], f, Ls);
            O = fmaf(sm_o[w][t], f, O);
          }
          a.part_o[(pbase + split) * DH + t] = O;
          if (t == 0) {
            a.part_ml[(pbase + split) * 2] = M;
            a.part_ml[(pbase + split) * 2 + 1] = Ls;
          }
        }
        __threadfence();
        abar();
        if (t == 0) merges = atomicAdd(a.head_counters + head, 1u) == static_cast<uint32_t>(nsplit - 1);
        abar();
        if (merges) {                                            // merge the head's ranges
          __threadfence();
          if (sw == 0) {
            float ms[2], ls[2];
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
              const int i = lane + 32 * h2;
              ms[h2] = i < nsplit ? __ldcg(a.part_ml + (pbase + i) * 2) : -INFINITY;
              ls[h2] = i < nsplit ? __ldcg(a.part_ml + (pbase + i) * 2 + 1) : 0.f;
            }
            const float M = warp_max(fmaxf(ms[0], ms[1]));
            float lt = 0.f;
#pragma unroll
            for (int h2 = 0; h2 < 2; ++h2) {
              const float f = ms[h2] == -INFINITY ? 0.f : __expf(ms[h2] - M);
              wgt[lane + 32 * h2] = f;
              lt = fmaf(ls[h2], f, lt);
            }
            lt = warp_sum(lt);
            if (lane == 0) inv_l = 1.0f / lt;
          }
          abar();
          if (t < DH) {
            const float* po = a.part_o + pbase * DH + t;
            float O = 0.f;
            for (int s0 = 0; s0 < nsplit; s0 += 8) {
              float v[8];
#pragma unroll
              for (int k = 0; k < 8; ++k) v[k] = __ldcg(po + static_cast<size_t>(min(s0 + k, nsplit - 1)) * DH);
#pragma unroll
              for (int k = 0; k < 8; ++k)
                if (s0 + k < nsplit) O = fmaf(v[k], wgt[s0 + k], O);
            }
            a.act2[head * DH + t] = O * inv_l;
          }
          if (t == 0) a.head_counters[head] = 0u;
        }
      }
      if (!attends && t == 0) phase_poll(c_qkv + l, target, a.dev_err, a.wait_limit);   // keeps the layers in step
      abar();
      if (t == 0) phase_arrive(c_af + l);
    }
  }
  // The last block to finish resets the counters, writes the token and moves the position on.  A block takes its ticket when all of
  // its warps are here: once a wait has run out they are no longer in step, and an arrival behind the reset would be the next step's.
  __syncthreads();
  if (threadIdx.x == 0) {
    if (*failed_v) {
      // what is still in flight gets another bounded chance to land before the block leaves
      for (int i = 0; i < kRing; ++i) {
        mbar_wait(full(i), 0);
        mbar_wait(full(i), 1);
      }
      if (a.dev_err) atomicOr(a.dev_err, kDevErrTimeout);
    }
    if (a.amax && blk_amax) atomicMax(a.amax, blk_amax);
    __threadfence();
    is_last = atomicAdd(a.sync + (4 * L + 1), 1u) == target - 1;
  }
  __syncthreads();
  if (is_last) {
    for (int i = threadIdx.x; i < 5 * L + 3; i += kThreads) a.sync[i] = 0u;
    for (int i = threadIdx.x; i < a.heads; i += kThreads) a.head_counters[i] = 0u;
    if (a.amax && threadIdx.x == 0) {
      __threadfence();
      a.tokens_out[0] = static_cast<uint32_t>(*reinterpret_cast<volatile unsigned long long*>(a.amax));
      a.amax[0] = 0ull;
      if (a.cur_out) *a.cur_out += 1;
    }
  }
}

// shared memory of a block of G: the ring and the partial sums of the most rows that a block has (two lots of them in `rows`)
int stream_smem(const MegaArgs& a, int G, int* rows = nullptr) {
  auto most = [&](int n) { return 2 * ((n / 2 + G - 1) / G); };
  const int first = std::max(most(a.ffl / 2) + most(a.ffl - a.ffl / 2) + 16, most(a.V)), second = most(3 * a.dl);
  if (rows) {
    rows[0] = first;
    rows[1] = second;
  }
  return kRing * static_cast<int>(kStage) + 4 * ((first + second) * kInPitch + (a.d + G - 1) / G * kOutPitch);
}

template <int DH>
cudaError_t launch_stream(const MegaArgs& a, cudaStream_t s, int* grid_out) {
  static DeviceOnce once;
  static int sms_of[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  e = once.run([&] {
    const cudaError_t e2 = cudaFuncSetAttribute(decode_stream_kernel<DH>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    return e2 != cudaSuccess ? e2 : cudaDeviceGetAttribute(&sms_of[dev], cudaDevAttrMultiProcessorCount, dev);
  });
  if (e != cudaSuccess) return e;
  const int G = sms_of[dev];
  if (grid_out) *grid_out = G;
  MegaArgs b = a;
  const int smem = stream_smem(a, G, b.part_rows);
  b.grid_splits = std::min({G / a.heads, 64, a.max_splits});       // key ranges per head: one round of blocks
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;      // all blocks resident: the phase waits cannot starve
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, decode_stream_kernel<DH>, b);
}

}  // namespace

// Where the line lies: at a width of 1024 and more this kernel is at least as fast as decode_mega_kernel with 100 and 2048 cached
// keys (8 layers, 50400 logits, us a step, old -> new: 4 heads of 256 at 1024 197 -> 189 and 229 -> 225, 16 heads of 64 192 -> 190
// and 212 -> 213; at 2048 320 -> 251 and 352 -> 302; at 3072 476 -> 419 and 526 -> 444); at 512 it gains 4 % and loses 2 %, at
// 256, where a layer is all hand-overs and 8 attending warps are fewer than 16, it loses 7 % and 20 %.  Above 4096 a warp's
// share of a row outgrows its registers.  The rest is what the ring, the bulk copies and the partial sums take.
bool decode_stream_ok(const MegaArgs& a) {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return false;
  return a.world == 1 && a.B == 1 && (a.dh == 256 || a.dh == 64) && a.d >= kMinD && a.d <= kMaxD && (a.d & 7) == 0 && a.dl <= kMaxD && (a.dl & 7) == 0 &&
         a.ffl >= 16 && a.ffl <= kMaxFf && (a.ffl & 7) == 0 && (a.V & 1) == 0 && a.heads <= sms && a.max_splits >= 1 &&
         stream_smem(a, sms) <= kMaxSmem;
}

cudaError_t launch_decode_stream(const MegaArgs& a, cudaStream_t s, int* grid_out) {
  if (!decode_stream_ok(a)) return cudaErrorInvalidValue;
  return a.dh == 256 ? launch_stream<256>(a, s, grid_out) : launch_stream<64>(a, s, grid_out);
}

}  // namespace mtj
