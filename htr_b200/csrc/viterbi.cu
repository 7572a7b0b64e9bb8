// Tail-biting Viterbi search over the 16-bit bit-shift trellis: the encoder-side inverse of the decode path.
//
// For every tile (batch row) it finds the states s_0 .. s_{T-1}, s_t = ((s_{t-1} << K) & 0xFFFF) | new bits, that minimise
// sum_t w[t] * (x[t] - cb[s_t])^2 with cb[s] = float32(v(s) / rms), and -- with tail-biting -- close the stream into a circle
// (the high 16-K bits of s_0 equal the low 16-K bits of s_{T-1}), so that the rate is exactly K bits per weight.
// Same result as the reference's portable search (htr/reference.py:7-50) and its CUDA version (htr/vit_v2.py:28-73, built there
// for sm_86 / sm_120 only): same float32 operation order per candidate, first minimum wins on ties.
//
// Formulation.  The reference keeps all 65536 path costs; here only their minima over the top K bits survive a step:
//   m_{t+1}[j] = min_top ( m_t[(top << (16-2K)) | (j >> K)] + w_t * (x_t - cb[(top << (16-K)) | j])^2 ),   bp_t[j] = argmin,
// with m_0 = 0 (or, in the second pass, +inf except at the required start).  That is 2 * 2^(16-K) floats of state, which fits
// shared memory for every K (128 KB at K = 2), so one thread block owns a tile from the first step to the traceback and touches
// global memory only for the back-pointers (one byte per (step, j), second pass only; each resident block has its own region).
//
// What bounds it: per candidate the reference's operations x - c, d * d, w * (d * d), prev + ... occupy the FMA pipes for four
// cycles of a warp (packed or not), the minimum the shift/logic pipe for two.  So everything else has to go:
//  * A thread owns the same 128 states in every step, hence the same 128 codebook values: 64 of them stay in registers, 64 in shared
//    memory (one 16-byte read per four; K = 2 has no room there and recomputes them from the state hash).  Recomputing all of them
//    cost 3.5 instructions per candidate.
//  * The first pass needs no argument of the minimum except in its last step.
//  * The traceback is a chain of dependent loads; the K unknown bits per step are few enough to load two to five steps' candidates
//    at once, so a warp resolves that many steps per memory latency.
// Measured, 256 tiles (K = 2, 3, 4, 5, 6, 8): 3.91, 3.69, 3.48, 3.60, 3.82, 3.89 ms with the values recomputed and one state per
// latency in the traceback; 2.70, 1.98, 2.01, 2.10, 2.18, 2.54 ms in this form.
//
// The codebook value in float: v(s) lands in a float through the 1.5 * 2^23 mantissa trick and float32(v / rms) =
// fma(v, inv_hi, v * inv_lo) with 1/rms split in two floats -- exact for all 1021 possible v (checked by the tests against the
// oracle's table, bit for bit).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "../../include/htr_b200.h"
#include "htr_codec.cuh"

namespace htr {
namespace {

constexpr int kVitMaxT = 256;

struct VitParams {
  const float* x;
  const float* w;
  int32_t* states;
  float* total;
  uint8_t* bps;      // [tiles at once][T][2^(16-K)]
  int B, T, tailbite;
  float inv_hi, inv_lo;
};

// C: thread blocks of the cluster that share one tile (1, 2 or 4): each owns SJ / C consecutive j
template <int K, int C>
struct VitCfg {
  static constexpr int kNB = 1 << K, kSj = 1 << (16 - K);
  static constexpr int kThreads = 512, kStates = 128 / C;                 // kThreads x kStates x C = all of them
  static constexpr int kTT = kNB < 16 ? kNB : 16;                         // tops of one thread; kSub neighbouring lanes share the others
  static constexpr int kSub = kNB / kTT;
  static constexpr int kPer = kStates / kTT;                              // j of a thread
  static constexpr int kJb = K == 2 ? 4 : kPer < 8 ? kPer : 8;            // consecutive j of a group: they share their predecessor minima
  static constexpr int kGroups = kPer / kJb;                              // groups of a thread
  static constexpr int kPairs = kJb / 2;                                  // candidates are handled two at a time
  static constexpr int kBlocks = kStates / kJb;                           // (group, top) blocks of kJb states, in that order
  static constexpr int kRegBlocks = C == 1 ? kBlocks / 2 : kBlocks;       // ... whose codebook values stay in registers
  static constexpr bool kTable = C == 1 && K != 2;                        // the others': in shared memory, else from the hash
  static constexpr int kTableBytes = kTable ? 64 * kThreads * 4 : 0;
  static constexpr int kSmem = kTableBytes + 2 * kSj * 4 + 2 * kVitMaxT * 4 + kSj;   // table, two cost arrays, targets, weights, last back-pointers
  static constexpr int kLevels = K == 2 ? 5 : K <= 4 ? 3 : 2;             // steps of the traceback per memory latency: kNB^(levels-1) <= 256
};

__device__ __forceinline__ float codebook_value(uint32_t hash, float inv_hi, float inv_lo) {
  const float v = __uint_as_float(__dp4a(hash, 0x01010101u, kMagicBits - 510u)) - 12582912.0f;   // the integer v(s), exactly
  return __fmaf_rn(v, inv_hi, __fmul_rn(v, inv_lo));
}

// packed float32 pairs: one instruction, two candidates
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }

struct Best {
  float v;
  uint32_t key;      // (top << 16) | j : state order, so "smaller key" = "earlier state"
};
__device__ __forceinline__ bool better(const Best& a, const Best& b) { return a.v < b.v || (a.v == b.v && a.key < b.key); }

// one candidate: the first minimum wins, as torch.min does
template <bool ARG>
__device__ __forceinline__ void take(float val, int top, float& best, int& arg) {
  if constexpr (ARG) {
    if (val < best) { best = val; arg = top; }
  } else {
    best = fminf(best, val);
  }
}

// JB consecutive costs, or their arguments as bytes, to the same place in the shared memory of every block of the cluster
template <int C, int JB>
__device__ __forceinline__ void spread_costs(float* at, const float (&v)[JB]) {
  if constexpr (C == 1) {
    if constexpr (JB % 4 == 0) {
#pragma unroll
      for (int q = 0; q < JB / 4; ++q) *reinterpret_cast<float4*>(at + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    } else {
      *reinterpret_cast<float2*>(at) = make_float2(v[0], v[1]);
    }
  } else {
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(at);
#pragma unroll
    for (int r = 0; r < C; ++r) {
      uint32_t to;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine), "r"(r));
      if constexpr (JB % 4 == 0) {
#pragma unroll
        for (int q = 0; q < JB / 4; ++q)
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + 16 * q), "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]), "f"(v[4 * q + 3])
                       : "memory");
      } else {
        asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(to), "f"(v[0]), "f"(v[1]) : "memory");
      }
    }
  }
}
template <int C>
__device__ __forceinline__ void spread_byte(uint8_t* at, uint32_t v) {
  if constexpr (C == 1) {
    *at = (uint8_t)v;
  } else {
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(at);
#pragma unroll
    for (int r = 0; r < C; ++r) {
      uint32_t to;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine), "r"(r));
      asm volatile("st.shared::cluster.u8 [%0], %1;" ::"r"(to), "r"(v) : "memory");
    }
  }
}
// barrier of all threads that work on the tile
template <int C>
__device__ __forceinline__ void tile_sync() {
  if constexpr (C == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}

// One step of this thread's states: costs mc -> mn (of every block of the cluster) and, with ARG, the arguments to bp and lastarg
// (either may be null).
template <int K, int C, bool ARG>
__device__ __forceinline__ void vit_step(const float* __restrict__ mc, float* __restrict__ mn, float xt, float wt,
                                         const float2 (&negc)[VitCfg<K, C>::kRegBlocks * VitCfg<K, C>::kPairs], const float4* __restrict__ table, int j_first,
                                         float inv_hi, float inv_lo, uint8_t* __restrict__ bp, uint8_t* __restrict__ lastarg) {
  using Cfg = VitCfg<K, C>;
  constexpr int JB = Cfg::kJb, SH = 16 - 2 * K, TT = Cfg::kTT, SUB = Cfg::kSub, PAIRS = Cfg::kPairs;
  const int tid = threadIdx.x, sub = tid % SUB;
  const float2 xt2 = make_float2(xt, xt), wt2 = make_float2(wt, wt);
#pragma unroll
  for (int g = 0; g < Cfg::kGroups; ++g) {
    const int jbase = j_first + (g * (Cfg::kThreads / SUB) + tid / SUB) * JB;
    const float* prev_col = mc + (jbase >> K) + ((sub * TT) << SH);        // predecessor minima of this group: stride 2^(16-2K) per top
    float best[JB];
    int arg[JB];                                                          // relative to this lane's first top
#pragma unroll
    for (int b = 0; b < JB; ++b) { best[b] = INFINITY; arg[b] = 0; }
#pragma unroll
    for (int tt = 0; tt < TT; ++tt) {
      const float prev = prev_col[tt << SH];
      const int blk = g * TT + tt;
#pragma unroll
      for (int q = 0; q < (PAIRS + 1) / 2; ++q) {
        float2 nc[2];
        if (blk < Cfg::kRegBlocks) {
          nc[0] = negc[blk * PAIRS + 2 * q];
          nc[1] = negc[blk * PAIRS + (2 * q + 1 < PAIRS ? 2 * q + 1 : 2 * q)];
        } else if constexpr (Cfg::kTable) {
          const float4 f = table[((blk - Cfg::kRegBlocks) * (PAIRS / 2) + q) * Cfg::kThreads];
          nc[0] = make_float2(f.x, f.y);
          nc[1] = make_float2(f.z, f.w);
        } else {
          const uint32_t h0 = ((uint32_t)((sub * TT + tt) << (16 - K)) + (uint32_t)(jbase + 4 * q)) * kGenMul + kGenAdd;
          const float2 unmagic = make_float2(-12582912.0f, -12582912.0f), hi = make_float2(-inv_hi, -inv_hi), lo = make_float2(-inv_lo, -inv_lo);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float2 v = add2(make_float2(__uint_as_float(bytesum_add_alu(h0 + (2 * e) * kGenMul, kMagicBits - 510u)),
                                              __uint_as_float(bytesum_add(h0 + (2 * e + 1) * kGenMul, kMagicBits - 510u))), unmagic);
            nc[e] = __ffma2_rn(v, hi, mul2(v, lo));                         // -c: negation commutes with rounding
          }
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (2 * q + e >= PAIRS) break;
          const float2 d = add2(xt2, nc[e]);
          const float2 wd = mul2(wt2, mul2(d, d));
          // the last addition stays scalar: a packed multiply followed by a packed add was observed to come out fused (one
          // rounding instead of two, costs 1 ulp off the reference's), which separate scalar adds rule out
          take<ARG>(__fadd_rn(prev, wd.x), tt, best[4 * q + 2 * e], arg[4 * q + 2 * e]);
          take<ARG>(__fadd_rn(prev, wd.y), tt, best[4 * q + 2 * e + 1], arg[4 * q + 2 * e + 1]);
        }
      }
    }
    if constexpr (ARG && SUB > 1) {
#pragma unroll
      for (int b = 0; b < JB; ++b) arg[b] += sub * TT;
    }
    // neighbouring lanes hold the other tops: the smaller cost, then the smaller top
#pragma unroll
    for (int o = 1; o < SUB; o <<= 1)
#pragma unroll
      for (int b = 0; b < JB; ++b) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, best[b], o);
        if constexpr (ARG) {
          const int oa = __shfl_xor_sync(0xFFFFFFFFu, arg[b], o);
          const bool other = ov < best[b] || (ov == best[b] && oa < arg[b]);
          best[b] = other ? ov : best[b];
          arg[b] = other ? oa : arg[b];
        } else {
          best[b] = fminf(best[b], ov);
        }
      }
    if (sub == 0) {
      spread_costs<C, JB>(mn + jbase, best);
      if constexpr (ARG) {
        if (bp) {
          if constexpr (JB % 4 == 0) {
#pragma unroll
            for (int q = 0; q < JB / 4; ++q)
              *reinterpret_cast<uint32_t*>(bp + jbase + 4 * q) = (uint32_t)arg[4 * q] | ((uint32_t)arg[4 * q + 1] << 8) | ((uint32_t)arg[4 * q + 2] << 16) | ((uint32_t)arg[4 * q + 3] << 24);
          } else {
            *reinterpret_cast<uint16_t*>(bp + jbase) = (uint16_t)((uint32_t)arg[0] | ((uint32_t)arg[1] << 8));
          }
        }
        if (lastarg) {
#pragma unroll
          for (int b = 0; b < JB; ++b) spread_byte<C>(lastarg + jbase + b, (uint32_t)arg[b]);
        }
      }
    }
  }
}

template <int K, int C>
__global__ void __launch_bounds__(VitCfg<K, C>::kThreads, 1) viterbi_kernel(const VitParams p) {
  using Cfg = VitCfg<K, C>;
  constexpr int NB = Cfg::kNB, SJ = Cfg::kSj, THREADS = Cfg::kThreads, JB = Cfg::kJb, PAIRS = Cfg::kPairs;
  extern __shared__ __align__(16) unsigned char vsm[];
  float4* table = reinterpret_cast<float4*>(vsm) + threadIdx.x;
  float* m_a = reinterpret_cast<float*>(vsm + Cfg::kTableBytes);
  float* m_b = m_a + SJ;
  float* xs = m_b + SJ;
  float* ws = xs + kVitMaxT;
  uint8_t* lastarg = reinterpret_cast<uint8_t*>(ws + kVitMaxT);
  __shared__ Best s_red[32];
  __shared__ Best s_win;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = p.T;
  const int cluster = blockIdx.x / C, rank = blockIdx.x % C, j_first = rank * (SJ / C);
  uint8_t* bp = p.bps + (size_t)cluster * T * SJ;

  // the negated codebook values of this thread's states, in block order (group, top): in registers, or half of them in shared memory
  float2 negc[Cfg::kRegBlocks * PAIRS];
#pragma unroll
  for (int blk = 0; blk < (Cfg::kTable ? Cfg::kBlocks : Cfg::kRegBlocks); ++blk) {
    const int g = blk / Cfg::kTT, top = (tid % Cfg::kSub) * Cfg::kTT + blk % Cfg::kTT;
    const int jbase = j_first + (g * (THREADS / Cfg::kSub) + tid / Cfg::kSub) * JB;
    float f[JB];
#pragma unroll
    for (int e = 0; e < JB; ++e) f[e] = -codebook_value((((uint32_t)top << (16 - K)) | (uint32_t)(jbase + e)) * kGenMul + kGenAdd, p.inv_hi, p.inv_lo);
    if (blk < Cfg::kRegBlocks) {
#pragma unroll
      for (int e = 0; e < PAIRS; ++e) negc[blk * PAIRS + e] = make_float2(f[2 * e], f[2 * e + 1]);
    } else {
#pragma unroll
      for (int q = 0; q < JB / 4; ++q)
        table[((blk - Cfg::kRegBlocks) * (JB / 4) + q) * THREADS] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
    }
  }

  for (int tile = cluster; tile < p.B; tile += gridDim.x / C) {
    tile_sync<C>();                                                      // the previous tile's traceback is over; every block of the cluster runs
    for (int t = tid; t < T; t += THREADS) {
      xs[t] = p.x[(size_t)tile * T + t];
      ws[t] = p.w[(size_t)tile * T + t];
    }
    int j0 = -1;
    const int passes = p.tailbite ? 2 : 1;
    for (int pass = 0; pass < passes; ++pass) {
      const bool keep = pass == passes - 1;                              // back-pointers are needed for the last pass only
      float* mc = m_a;
      float* mn = m_b;
      for (int j = tid; j < SJ; j += THREADS) mc[j] = (j0 < 0 || j == j0) ? 0.f : INFINITY;
      tile_sync<C>();                                                    // (the other cost array may be written by the cluster from here on)
      for (int t = 0; t < T; ++t) {
        const float xt = xs[t], wt = ws[t];
        const bool last = t == T - 1;
        if (keep || last) vit_step<K, C, true>(mc, mn, xt, wt, negc, table, j_first, p.inv_hi, p.inv_lo, keep ? bp + (size_t)t * SJ : nullptr, last ? lastarg : nullptr);
        else vit_step<K, C, false>(mc, mn, xt, wt, negc, table, j_first, p.inv_hi, p.inv_lo, nullptr, nullptr);
        tile_sync<C>();
        float* sw = mc; mc = mn; mn = sw;
      }
      // mc[j] = min over top of the final costs, lastarg[j] = its first top.  First pass of a tail-biting search, or an open
      // search: the first state (in state order) of minimal cost.
      if (!(p.tailbite && keep)) {
        Best mine = {INFINITY, 0xFFFFFFFFu};
        for (int j = tid; j < SJ; j += THREADS) {
          const Best cand = {mc[j], ((uint32_t)lastarg[j] << 16) | (uint32_t)j};
          if (better(cand, mine)) mine = cand;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
          Best other = {__shfl_xor_sync(0xFFFFFFFFu, mine.v, o), __shfl_xor_sync(0xFFFFFFFFu, mine.key, o)};
          if (better(other, mine)) mine = other;
        }
        if (lane == 0) s_red[warp] = mine;
        __syncthreads();
        if (tid == 0) {
          Best win = s_red[0];
          for (int i = 1; i < THREADS / 32; ++i)
            if (better(s_red[i], win)) win = s_red[i];
          s_win = win;
        }
        __syncthreads();
        j0 = (int)(s_win.key & 0xFFFFu);                                 // low 16-K bits of the winner (j < 2^(16-K))
      }
      if (keep && warp == 0 && rank == 0) {
        // last state: with tail-biting the cheapest state whose low bits equal j0, else the overall winner
        uint32_t s = p.tailbite ? ((uint32_t)lastarg[j0] * SJ + (uint32_t)j0) : ((s_win.key >> 16) * SJ + (s_win.key & 0xFFFFu));
        int32_t* out = p.states + (size_t)tile * T;
        if (lane == 0) {
          if (p.total) p.total[tile] = p.tailbite ? mc[j0] : s_win.v;
          out[T - 1] = (int32_t)s;
        }
        // back along the path (htr/reference.py:45-49): s_{t-1} = bp_{t-1}[s_t >> K] * SJ + (s_t >> K).  The back-pointers of kLevels
        // steps are loaded together: for every value of the tops still unknown, candidate id = those tops as a number in base NB
        constexpr int LV = Cfg::kLevels;
        for (int t = T - 1; t >= 1; t -= LV) {
          constexpr int kMost = 8;                                       // loads of a lane per level: NB^(LV-1) <= 256
          uint32_t got[LV][kMost];
          int ids = 1;
#pragma unroll
          for (int l = 0; l < LV; ++l, ids *= NB) {
#pragma unroll
            for (int r = 0; r < kMost; ++r) {
              got[l][r] = 0u;
              const int id = 32 * r + lane;
              if (32 * r < ids && id < ids && t - 1 - l >= 0) {
                uint32_t low = s >> K;
#pragma unroll
                for (int k = l - 1; k >= 0; --k) low = ((((uint32_t)(id >> (k * K)) & (NB - 1)) * SJ) + low) >> K;   // the earliest step's top is the leading digit
                got[l][r] = __ldcg(bp + (size_t)(t - 1 - l) * SJ + low);
              }
            }
          }
          int id = 0;
#pragma unroll
          for (int l = 0; l < LV; ++l) {
            if (t - 1 - l < 0) break;
            uint32_t mine = got[l][0];
#pragma unroll
            for (int r = 1; r < kMost; ++r)
              if (r == id >> 5) mine = got[l][r];
            const uint32_t top = __shfl_sync(0xFFFFFFFFu, mine, id & 31);
            s = top * SJ + (s >> K);
            if (lane == 0) out[t - 1 - l] = (int32_t)s;
            id = id * NB + (int)top;
          }
        }
      }
      __syncthreads();
    }
  }
  if (C > 1) tile_sync<C>();                                              // nobody leaves while its shared memory may still be written
}

// every codebook value through the device function above (test hook)
__global__ void codebook_kernel(float* out, float inv_hi, float inv_lo) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < 65536u) out[s] = codebook_value(s * kGenMul + kGenAdd, inv_hi, inv_lo);
}

double inverse_rms() {
  static const double value = [] {
    double acc = 0.0;
    for (uint32_t s = 0; s < 65536u; ++s) {
      const double v = (double)code_value(s);
      acc += v * v;
    }
    return 1.0 / std::sqrt(acc / 65536.0);
  }();
  return value;
}

bool width_ok(int K) { return K == 2 || K == 3 || K == 4 || K == 5 || K == 6 || K == 8; }

thread_local int t_vit_cuda = 0;

// thread blocks (C = 1) or clusters that the GPU holds at once
template <int K, int C>
int resident(int* out) {
  static int cached[64] = {0};
  int dev = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return (int)cudaErrorInvalidDevice;
  if (dev >= 0 && dev < 64 && cached[dev]) { *out = cached[dev]; return 0; }
  using Cfg = VitCfg<K, C>;
  cudaError_t e = cudaFuncSetAttribute(viterbi_kernel<K, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  if (e != cudaSuccess) return (int)e;
  if constexpr (C == 1) {
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return (int)e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, viterbi_kernel<K, C>, Cfg::kThreads, Cfg::kSmem)) != cudaSuccess) return (int)e;
    per *= sms;
  } else {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(Cfg::kThreads);
    cfg.dynamicSmemBytes = Cfg::kSmem;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if ((e = cudaOccupancyMaxActiveClusters(&per, viterbi_kernel<K, C>, &cfg)) != cudaSuccess) return (int)e;
  }
  if (per < 1) return (int)cudaErrorLaunchOutOfResources;
  *out = per;
  if (dev >= 0 && dev < 64) cached[dev] = per;
  return 0;
}

// Thread blocks per tile: as many as leave every tile a cluster of its own at once (few tiles leave SMs idle otherwise; a step of a
// shared tile pays a cluster barrier and stores its costs several times: 2^(16-K) of them).  One block / two / four, ms: K = 2 1.34 / 1.01 /
// 1.14, K = 3 1.00 / 1.16 / 0.88, K = 4 1.00 / 0.81 / 0.67, K = 5 1.05 / 0.79 / 0.64, K = 8 1.28 / 1.03 / 1.00.
template <int K>
int tile_split(int B, int* split, int* at_once) {
  int one = 0, two = 0, four = 0;
  if (const int e = resident<K, 1>(&one)) return e;
  if (resident<K, 2>(&two)) { (void)cudaGetLastError(); two = 0; }
  if (resident<K, 4>(&four)) { (void)cudaGetLastError(); four = 0; }
  if (K == 2) four = 0;
  if (K == 3) two = 0;
  *split = B <= four ? 4 : B <= two ? 2 : 1;
  *at_once = *split == 4 ? four : *split == 2 ? two : one;
  return 0;
}

int split_for(int K, int B, int* split, int* at_once) {
  switch (K) {
    case 2: return tile_split<2>(B, split, at_once);
    case 3: return tile_split<3>(B, split, at_once);
    case 4: return tile_split<4>(B, split, at_once);
    case 5: return tile_split<5>(B, split, at_once);
    case 6: return tile_split<6>(B, split, at_once);
    case 8: return tile_split<8>(B, split, at_once);
  }
  return (int)cudaErrorInvalidValue;
}

template <int K, int C>
int launch_split(const VitParams& p, int tiles_at_once, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)(tiles_at_once * C));
  cfg.blockDim = dim3(VitCfg<K, C>::kThreads);
  cfg.dynamicSmemBytes = VitCfg<K, C>::kSmem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, viterbi_kernel<K, C>, p);
}
template <int K>
int launch(const VitParams& p, int split, int tiles_at_once, cudaStream_t st) {
  return split == 4 ? launch_split<K, 4>(p, tiles_at_once, st) : split == 2 ? launch_split<K, 2>(p, tiles_at_once, st) : launch_split<K, 1>(p, tiles_at_once, st);
}

}  // namespace
}  // namespace htr

using namespace htr;

extern "C" {

size_t htr_viterbi_workspace_bytes(int B, int T, int K) {
  if (!width_ok(K) || B < 1 || T < 1 || T > kVitMaxT) return 0;
  int split = 0, at_once = 0;
  if (split_for(K, B, &split, &at_once) != 0) return 0;
  const int grid = B < at_once ? B : at_once;
  return (size_t)grid * T * ((size_t)65536 >> K);
}

int htr_viterbi(const float* x, const float* w, int B, int T, int K, int tailbite, int32_t* states, float* total, void* workspace,
                size_t workspace_bytes, htr_stream_t stream) {
  if (!width_ok(K)) return HTR_ERR_BAD_K;
  if (B < 0 || T < 1 || T > kVitMaxT) return HTR_ERR_BAD_SHAPE;
  if (B == 0) return HTR_OK;
  if (!x || !w || !states) return HTR_ERR_NULL;
  int split = 0, at_once = 0;
  int e = split_for(K, B, &split, &at_once);
  if (e) { t_vit_cuda = e; return HTR_ERR_CUDA; }
  const int grid = B < at_once ? B : at_once;
  if (!workspace || workspace_bytes < (size_t)grid * T * ((size_t)65536 >> K)) return HTR_ERR_WORKSPACE;
  const double inv = inverse_rms();
  VitParams p;
  p.x = x;
  p.w = w;
  p.states = states;
  p.total = total;
  p.bps = static_cast<uint8_t*>(workspace);
  p.B = B;
  p.T = T;
  p.tailbite = tailbite ? 1 : 0;
  p.inv_hi = (float)inv;
  p.inv_lo = (float)(inv - (double)p.inv_hi);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  switch (K) {
    case 2: e = launch<2>(p, split, grid, st); break;
    case 3: e = launch<3>(p, split, grid, st); break;
    case 4: e = launch<4>(p, split, grid, st); break;
    case 5: e = launch<5>(p, split, grid, st); break;
    case 6: e = launch<6>(p, split, grid, st); break;
    case 8: e = launch<8>(p, split, grid, st); break;
  }
  if (e) { t_vit_cuda = e; return HTR_ERR_CUDA; }
  return HTR_OK;
}

int htr_viterbi_last_cuda_error(void) { return t_vit_cuda; }

int htr_codebook_f32(float* out, htr_stream_t stream) {
  if (!out) return HTR_ERR_NULL;
  const double inv = inverse_rms();
  const float hi = (float)inv, lo = (float)(inv - (double)hi);
  codebook_kernel<<<256, 256, 0, static_cast<cudaStream_t>(stream)>>>(out, hi, lo);
  const int e = (int)cudaGetLastError();
  if (e) { t_vit_cuda = e; return HTR_ERR_CUDA; }
  return HTR_OK;
}

}  // extern "C"
