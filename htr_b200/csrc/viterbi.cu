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
// shared memory for every K (128 KB at K = 2), so one thread block owns a tile from the first step to the traceback.
//
// What bounds it: per candidate the reference's operations x - c, d * d, w * (d * d), prev + ... occupy the FMA pipes for four
// cycles of a warp (packed or not), so everything else has to go:
//  * No step looks for the argument of a minimum (a comparison and two selects per candidate, half as much again as the four
//    operations).  Every kLevels-th row of minima is kept in global memory instead (1 to 11 KB a step, K = 8 to 2), and the way back computes the
//    few costs it meets again: from a state, the 2^(K kLevels) ancestors at the next kept row (vit_trace).  The first minimum of
//    three operands at a time is one instruction for two candidates.
//  * A thread owns the same states in every step, hence the same codebook values.  One block per tile or two tiles per block: three
//    quarters of them stay in registers, the rest in shared memory (one 16-byte read per four); K = 2, whose cost arrays leave no room
//    there, keeps half in registers and computes the others from the state hash.  Clusters: all in registers.
//  * More tiles than thread blocks: a block takes two tiles step by step together, so that a value from shared memory serves both and a
//    block barrier has twice the work on either side.  (Two tiles in turn, each with a barrier that is waited for only after the other
//    tile's step, were slower: 0.75 against 0.67 ms a tile and two passes.)
// Measured, ms for 256 tiles (K = 2, 3, 4, 5, 6, 8), arguments kept for every step and one tile per block -> this form: 2.71, 1.98, 2.02,
// 2.10, 2.19, 2.55 -> 1.73, 1.48, 1.42, 1.46, 1.58, 1.84; for 140 tiles 1.37, 1.00, 1.03, 1.06, 1.10, 1.28 -> 0.88, 0.86, 0.80, 0.84,
// 0.86, 1.06.  A pass of one tile takes 0.33 ms at K = 4, of which 0.27 are the four operations at the pipes' rate; the traceback 0.11 ms.
//
// The codebook value in float: v(s) lands in a float through the 1.5 * 2^23 mantissa trick and float32(v / rms) =
// fma(v, inv_hi, v * inv_lo) with 1/rms split in two floats -- exact for all 1021 possible v (checked by the tests against the
// oracle's table, bit for bit).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <type_traits>

#include "../../include/htr_b200.h"
#include "htr_codec.cuh"

namespace htr {
namespace {

constexpr int kVitMaxT = 256;

template <int V>
using Const = std::integral_constant<int, V>;

struct VitParams {
  const float* x;
  const float* w;
  int32_t* states;
  float* total;
  float* rows;       // [tiles at once][(T - 1) / kLevels][2^(16-K)]: kept cost rows
  int B, T, tailbite;
  float inv_hi, inv_lo;
  float one;         // 1, unknown to the compiler
};

// C: thread blocks of the cluster that share one tile (1, 2 or 4): each owns SJ / C consecutive j; N: tiles that a thread block
// works on step by step together
template <int K, int C, int N>
struct VitCfg {
  static constexpr int kNB = 1 << K, kSj = 1 << (16 - K);
  // (two warps a scheduler with up to 255 registers each; ms with 256 / 512 threads: K = 4, 256 tiles 1.41 / 1.47, K = 8, 60 tiles 0.76 / 0.96;
  // but K = 2, one block per tile, 0.98 / 0.87, K = 4, two 0.79 / 0.70)
  static constexpr int kThreads = (K == 2 && C == 1) || (K == 4 && C == 2) ? 512 : 256;
  static constexpr int kStates = 65536 / kThreads / C;
  static constexpr int kTT = kNB < 16 ? kNB : 16;                         // tops of one thread; kSub neighbouring lanes share the others
  static constexpr int kSub = kNB / kTT;
  static constexpr int kPer = kStates / kTT;                              // j of a thread
  static constexpr int kJb = K == 2 ? 4 : kPer < 8 ? kPer : 8;            // consecutive j of a group: they share their predecessor minima
  static constexpr int kGroups = kPer / kJb;                              // groups of a thread
  static_assert(kJb % 4 == 0, "costs are handled four at a time");
  static constexpr int kPairs = kJb / 2;                                  // candidates are handled two at a time
  static constexpr int kBlocks = kStates / kJb;                           // (group, top) blocks of kJb states, in that order
  static constexpr int kRegBlocks = C > 1 ? kBlocks : kThreads == 512 ? kBlocks / 2 : kBlocks * 3 / 4;   // ... whose codebook values stay in registers
  static constexpr bool kTable = C == 1 && K != 2;                        // the others': in shared memory, else from the hash
  static constexpr int kTableBytes = kTable ? (kBlocks - kRegBlocks) * kJb * kThreads * 4 : 0;
  static constexpr int kLevels = K == 2 ? 6 : K == 3 ? 4 : K == 4 ? 3 : K <= 6 ? 2 : 1;   // steps of the path that one kept row serves
  static constexpr int kCone = ((1 << (K * kLevels)) - 1) / (kNB - 1);     // minima on the way back from one state to a kept row
  static constexpr int kTraceThreads = K == 8 ? 32 : kThreads / N;         // (a cone of 256 states is a warp's work)
  static constexpr int kTileFloats = 2 * kSj + 2 * kVitMaxT + (kCone + 4) / 4 * 4 * 2;   // two cost arrays, targets, weights, cone: minima, tops, a state
  static constexpr int kSmem = kTableBytes + N * kTileFloats * 4;
};

__device__ __forceinline__ float codebook_value(uint32_t hash, float inv_hi, float inv_lo) {
  const float v = __uint_as_float(__dp4a(hash, 0x01010101u, kMagicBits - 510u)) - 12582912.0f;   // the integer v(s), exactly
  return __fmaf_rn(v, inv_hi, __fmul_rn(v, inv_lo));
}

// packed float32 pairs: one instruction, two candidates
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// cost of one state, the operations of vit_step one at a time
__device__ __forceinline__ float state_cost(uint32_t s, float prev, float xt, float wt, const VitParams& p) {
  const float d = __fadd_rn(xt, -codebook_value(s * kGenMul + kGenAdd, p.inv_hi, p.inv_lo));
  return __fadd_rn(prev, __fmul_rn(wt, __fmul_rn(d, d)));
}

// JB consecutive costs to the same place in the shared memory of every block of the cluster
template <int C, int JB>
__device__ __forceinline__ void spread_costs(float* at, const float (&v)[JB]) {
  if constexpr (C == 1) {
#pragma unroll
    for (int q = 0; q < JB / 4; ++q) *reinterpret_cast<float4*>(at + 4 * q) = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  } else {
    const uint32_t mine = (uint32_t)__cvta_generic_to_shared(at);
#pragma unroll
    for (int r = 0; r < C; ++r) {
      uint32_t to;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(mine), "r"(r));
#pragma unroll
      for (int q = 0; q < JB / 4; ++q)
        asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(to + 16 * q), "f"(v[4 * q]), "f"(v[4 * q + 1]), "f"(v[4 * q + 2]), "f"(v[4 * q + 3])
                     : "memory");
    }
  }
}
// barrier of all threads that work on the tile
template <int C>
__device__ __forceinline__ void tile_sync() {
  if constexpr (C == 1) {
    __syncthreads();
  } else {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  }
}
// barrier of the threads that trace one tile back
__device__ __forceinline__ void trace_sync(int id, int threads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// One step of this thread's states in N tiles at once: costs mc -> mn (of every block of the cluster).  mem: the tiles' shared memory,
// one tile behind the other; the codebook values serve all of them.
template <int K, int C, int N>
__device__ __forceinline__ void vit_step(float* __restrict__ mem, int cur, int t, float one, const float2 (&negc)[VitCfg<K, C, N>::kRegBlocks * VitCfg<K, C, N>::kPairs],
                                         const float4* __restrict__ table, int j_first, float inv_hi, float inv_lo) {
  using Cfg = VitCfg<K, C, N>;
  constexpr int JB = Cfg::kJb, SH = 16 - 2 * K, TT = Cfg::kTT, SUB = Cfg::kSub, PAIRS = Cfg::kPairs, SJ = Cfg::kSj;
  const int tid = threadIdx.x, sub = tid % SUB;
  const float* mc = mem + cur * SJ;
  float* mn = mem + (1 - cur) * SJ;
  const float2 one2 = make_float2(one, one);
  float2 xt2[N], wt2[N];
#pragma unroll
  for (int h = 0; h < N; ++h) {
    const float xt = mem[h * Cfg::kTileFloats + 2 * SJ + t], wt = mem[h * Cfg::kTileFloats + 2 * SJ + kVitMaxT + t];
    xt2[h] = make_float2(xt, xt);
    wt2[h] = make_float2(wt, wt);
  }
#pragma unroll
  for (int g = 0; g < Cfg::kGroups; ++g) {
    const int jbase = j_first + (g * (Cfg::kThreads / SUB) + tid / SUB) * JB;
    const float* prev_col = mc + (jbase >> K) + ((sub * TT) << SH);        // predecessor minima of this group: stride 2^(16-2K) per top
    float best[N][JB];
#pragma unroll
    for (int h = 0; h < N; ++h)
#pragma unroll
      for (int b = 0; b < JB; ++b) best[h][b] = INFINITY;
    // negated codebook values of two pairs of consecutive j behind one top
    auto values = [&](int tt, int q, float2 (&nc)[2]) {
      const int blk = g * TT + tt;
      if (blk < Cfg::kRegBlocks) {
        nc[0] = negc[blk * PAIRS + 2 * q];
        nc[1] = negc[blk * PAIRS + 2 * q + 1];
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
          nc[e] = __ffma2_rn(v, hi, mul2(v, lo));                           // -c: negation commutes with rounding
        }
      }
    };
    auto cost = [&](int h, float2 nc, float prev) {
      const float2 d = add2(xt2[h], nc);
      const float2 wd = mul2(wt2[h], mul2(d, d));
      // prev + wd with a rounding of its own: a packed multiply followed by a packed add was observed to come out fused (costs
      // 1 ulp off the reference's); a multiply-add by a one that the compiler does not know cannot take the multiply in
      return __ffma2_rn(wd, one2, make_float2(prev, prev));
    };
#pragma unroll
    for (int tt = 0; tt < TT; tt += 2)
#pragma unroll
      for (int q = 0; q < PAIRS / 2; ++q) {
        float2 na[2], nb[2];
        values(tt, q, na);
        values(tt + 1, q, nb);
#pragma unroll
        for (int h = 0; h < N; ++h) {
          const float pa = prev_col[h * Cfg::kTileFloats + (tt << SH)], pb = prev_col[h * Cfg::kTileFloats + ((tt + 1) << SH)];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float2 va = cost(h, na[e], pa), vb = cost(h, nb[e], pb);
            best[h][4 * q + 2 * e] = min3(best[h][4 * q + 2 * e], va.x, vb.x);
            best[h][4 * q + 2 * e + 1] = min3(best[h][4 * q + 2 * e + 1], va.y, vb.y);
          }
        }
      }
#pragma unroll
    for (int h = 0; h < N; ++h) {
      // neighbouring lanes hold the other tops
#pragma unroll
      for (int o = 1; o < SUB; o <<= 1)
#pragma unroll
        for (int b = 0; b < JB; ++b) best[h][b] = fminf(best[h][b], __shfl_xor_sync(0xFFFFFFFFu, best[h][b], o));
      if (sub == 0) spread_costs<C, JB>(mn + h * Cfg::kTileFloats + jbase, best[h]);
    }
  }
}

// Level l of a cone: of every state that l tops lead back to from s at step t, the minimum over its predecessors' tops, which lie at
// step t - l - 1.  Groups of NB candidates, one per combination of the l tops (the latest step's is the lowest digit), shared by
// `kLanes` neighbouring lanes of kThreads threads; the first top of minimal cost wins.
template <int K, int C, int N, int L, int kThreads>
__device__ __forceinline__ void vit_cone(const VitParams& p, const float* row, bool deepest, uint32_t s, float xt, float wt, float* cone, int* tops, int me) {
  using Cfg = VitCfg<K, C, N>;
  constexpr int NB = Cfg::kNB, SJ = Cfg::kSj, kGroups = 1 << (K * L), kBase = (kGroups - 1) / (NB - 1), kBelow = kBase + kGroups;
  constexpr int kWant = kThreads / kGroups < 1 ? 1 : kThreads / kGroups, kMost = NB < 32 ? NB : 32, kLanes = kWant < kMost ? kWant : kMost, kPer = NB / kLanes;
#pragma unroll
  for (int i0 = 0; i0 < kGroups * kLanes; i0 += kThreads) {
    if (kGroups * kLanes < kThreads && (me & ~31) >= kGroups * kLanes) break;   // (by warps: the shuffles stay converged)
    const int i = (i0 + me) % (kGroups * kLanes), id = i / kLanes, part = i % kLanes;   // (a group smaller than a warp: the rest of it repeats)
    const uint32_t low = (((uint32_t)id << (16 - K * L)) | (s >> (K * L))) >> K;
    float best = INFINITY;
    int top = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const int tt = part * kPer + k;
      const uint32_t st = (uint32_t)tt * SJ + low;
      const float v = state_cost(st, deepest ? row[st >> K] : cone[kBelow + id + tt * kGroups], xt, wt, p);
      if (v < best) { best = v; top = tt; }
    }
    if constexpr (kGroups == 1) {
      float least;
      asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(least) : "f"(best));
      const int at = __ffs(__ballot_sync(0xFFFFFFFFu, best == least)) - 1;   // (a NaN of `least` is not possible: every lane starts at infinity)
      top = __shfl_sync(0xFFFFFFFFu, top, at);
    } else {
#pragma unroll
      for (int o = 1; o < kLanes; o <<= 1) {
        const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o);
        const int ot = __shfl_xor_sync(0xFFFFFFFFu, top, o);
        const bool other = ov < best || (ov == best && ot < top);
        best = other ? ov : best;
        top = other ? ot : top;
      }
    }
    if (part == 0) {
      cone[kBase + id] = best;
      tops[kBase + id] = top;
    }
  }
}

// The path of one tile, backwards from the low bits j0 of its last state, by the threads me = 0 .. kThreads - 1 (barrier `bar`).
// Only the minima over the tops are kept, and of those every kLevels-th row: from a known state s_t the ancestors kLevels steps
// earlier are 2^(K kLevels) states (4096 of 65536 at K = 4), so their costs are computed again, the deepest from the kept row, and
// reduced level by level, the wide levels by all threads, the narrow ones by one warp.  Rows do not depend on the path: the next one
// is on its way while a cone is evaluated.
template <int K, int C, int N, int kThreads>
__device__ __forceinline__ void vit_trace(const VitParams& p, const float* __restrict__ rows, float* buf_a, float* buf_b, const float* xs, const float* ws,
                                          float* cone, int* tops, int j0, int32_t* __restrict__ out, int me, int bar) {
  using Cfg = VitCfg<K, C, N>;
  constexpr int NB = Cfg::kNB, SJ = Cfg::kSj, LV = Cfg::kLevels;
  constexpr int kWide = K == 8 ? 1 : K <= 3 ? LV - 2 : LV - 1;              // levels from this one on have 512 candidates and more
  const int T = p.T;
  volatile uint32_t* found = reinterpret_cast<volatile uint32_t*>(tops + Cfg::kCone);
  // row of time q (before step q) to shared memory; before the first step the costs are those the search began with
  auto fetch = [&](int q, float* to) {
    if (q > 0) {
      const float* from = rows + (size_t)((T - q) / LV - 1) * SJ;
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(to);
#pragma unroll
      for (int i = 0; i < SJ / 4; i += kThreads)
        if (SJ / 4 % kThreads == 0 || i + me < SJ / 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16u * (i + me)), "l"(from + 4 * (i + me)) : "memory");
    } else {
      for (int i = me; i < SJ; i += kThreads) to[i] = !p.tailbite || i == j0 ? 0.f : INFINITY;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint32_t s = (uint32_t)j0 << K;                                          // s_T, of which only the high bits matter
  float *row = buf_a, *next = buf_b;
  fetch(max(T - LV, 0), row);
  for (int t = T; t > 0; t -= LV) {
    const int levels = min(LV, t);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    trace_sync(bar, kThreads);                                             // the row has landed; every thread has read the state
    if (t > LV) fetch(max(t - 2 * LV, 0), next);
    auto level = [&](auto l_const, auto threads_const) {
      constexpr int L = decltype(l_const)::value;
      if (L < levels) vit_cone<K, C, N, L, decltype(threads_const)::value>(p, row, L == levels - 1, s, xs[t - L - 1], ws[t - L - 1], cone, tops, me);
    };
    if constexpr (LV - 1 >= kWide) {
      level(Const<LV - 1>{}, Const<kThreads>{});
      trace_sync(bar, kThreads);
    }
    if constexpr (LV - 2 >= kWide) {
      level(Const<LV - 2>{}, Const<kThreads>{});
      trace_sync(bar, kThreads);
    }
    if (me < 32) {
      if constexpr (kWide >= 4) { level(Const<3>{}, Const<32>{}); __syncwarp(); }
      if constexpr (kWide >= 3) { level(Const<2>{}, Const<32>{}); __syncwarp(); }
      if constexpr (kWide >= 2) { level(Const<1>{}, Const<32>{}); __syncwarp(); }
      level(Const<0>{}, Const<32>{});
      __syncwarp();
      int id = 0;
#pragma unroll
      for (int l = 0; l < LV; ++l) {
        if (l < levels) {
          const int top = tops[((1 << (K * l)) - 1) / (NB - 1) + id];
          s = (uint32_t)top * SJ + (s >> K);
          if (me == l) out[t - 1 - l] = (int32_t)s;
          id += top << (K * l);
        }
      }
      if (me == 0) *found = s;
    }
    trace_sync(bar, kThreads);
    s = *found;
    float* sw = row; row = next; next = sw;
  }
}

template <int K, int C, int N>
__global__ void __launch_bounds__(VitCfg<K, C, N>::kThreads, 1) viterbi_kernel(const VitParams p) {
  using Cfg = VitCfg<K, C, N>;
  constexpr int NB = Cfg::kNB, SJ = Cfg::kSj, THREADS = Cfg::kThreads, JB = Cfg::kJb, PAIRS = Cfg::kPairs;
  static_assert(N == 1 || C == 1, "tiles are interleaved by single thread blocks");
  extern __shared__ __align__(16) unsigned char vsm[];
  float4* table = reinterpret_cast<float4*>(vsm) + threadIdx.x;
  auto tile_mem = [&](int h) { return reinterpret_cast<float*>(vsm + Cfg::kTableBytes) + h * Cfg::kTileFloats; };
  __shared__ float s_red[THREADS / 32];
  __shared__ unsigned s_key;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int T = p.T, kept = (T - 1) / Cfg::kLevels;
  const int at_once = gridDim.x / C * N, cluster = blockIdx.x / C, rank = blockIdx.x % C, j_first = rank * (SJ / C);

  // the negated codebook values of this thread's states, in block order (group, top): in registers, the last ones in shared memory where there is a table
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

  for (int first = cluster; first < p.B; first += at_once) {
    const int tiles = N > 1 && first + (at_once / N) < p.B ? N : 1;        // tiles first, first + at_once / N
    tile_sync<C>();                                                        // the previous tiles' traceback is over; every block of the cluster runs
    for (int i = tid; i < N * T; i += THREADS) {
      const int h = N > 1 && i >= T ? 1 : 0, t = i - h * T;
      const size_t from = (size_t)(first + (h < tiles ? h : 0) * (at_once / N)) * T + t;   // (a lone tile runs twice)
      float* xs = tile_mem(h) + 2 * SJ;
      xs[t] = p.x[from];
      xs[kVitMaxT + t] = p.w[from];
    }
    int j0[N];
    float cost[N];
#pragma unroll
    for (int h = 0; h < N; ++h) { j0[h] = -1; cost[h] = 0.f; }
    const int passes = p.tailbite ? 2 : 1;
    for (int pass = 0; pass < passes; ++pass) {
      const bool keep = pass == passes - 1;                                // cost rows are needed for the last pass only
#pragma unroll
      for (int h = 0; h < N; ++h)
        for (int j = tid; j < SJ; j += THREADS) tile_mem(h)[j] = (j0[h] < 0 || j == j0[h]) ? 0.f : INFINITY;
      tile_sync<C>();                                                      // (the other cost array may be written by the cluster from here on)
      int cur = 0;                                                         // which of the two cost arrays a step reads
      int until_row = keep ? (T - 1) % Cfg::kLevels : T;                   // steps until one whose minima are kept: row q with (T - q) % kLevels = 0
      int row_at = kept - 1;
      for (int t = 0; t < T; ++t) {
        vit_step<K, C, N>(tile_mem(0), cur, t, p.one, negc, table, j_first, p.inv_hi, p.inv_lo);
        if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the array that the next step writes has left
        tile_sync<C>();
        if (until_row-- == 0) {
          // a row to keep: this block's part of it leaves beside the next step (stored by the threads, a cluster's barrier waited for it)
          if (tid == 0 && row_at >= 0) {
            asm volatile("fence.proxy.async;" ::: "memory");
#pragma unroll
            for (int h = 0; h < N; ++h)
              asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(p.rows + ((size_t)(cluster * N + h) * kept + row_at) * SJ + j_first),
                           "r"((uint32_t)__cvta_generic_to_shared(tile_mem(h) + (1 - cur) * SJ + j_first)), "n"(SJ / C * 4)
                           : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
          until_row = Cfg::kLevels - 1;
          --row_at;
        }
        cur = 1 - cur;
      }
#pragma unroll
      for (int h = 0; h < N; ++h) {
        if (h >= tiles) break;
        const float *fin = tile_mem(h) + cur * SJ, *before = tile_mem(h) + (1 - cur) * SJ, *xs = tile_mem(h) + 2 * SJ;
        if (p.tailbite && keep) {
          cost[h] = fin[j0[h]];
          continue;
        }
        // First pass of a tail-biting search, or an open search: the first state (in state order) of minimal cost.  The minima say
        // which low bits reach it; those states' tops are looked up again from the costs before the last step.
        float least = INFINITY;
        for (int j = tid; j < SJ; j += THREADS) least = fminf(least, fin[j]);
#pragma unroll
        for (int o = 16; o; o >>= 1) least = fminf(least, __shfl_xor_sync(0xFFFFFFFFu, least, o));
        if (lane == 0) s_red[warp] = least;
        if (tid == 0) s_key = 0xFFFFFFFFu;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < THREADS / 32; ++i) least = fminf(least, s_red[i]);
        for (int j = tid; j < SJ; j += THREADS) {
          if (fin[j] != least) continue;
          float best = INFINITY;
          int top = 0;
#pragma unroll 1
          for (int tt = 0; tt < NB; ++tt) {
            const uint32_t st = (uint32_t)tt * SJ + (uint32_t)j;
            const float v = state_cost(st, before[st >> K], xs[T - 1], xs[kVitMaxT + T - 1], p);
            if (v < best) { best = v; top = tt; }
          }
          atomicMin(&s_key, (unsigned)top * SJ + (unsigned)j);
        }
        __syncthreads();
        j0[h] = (int)(s_key & (SJ - 1));                                   // low 16-K bits of the winner
        cost[h] = least;
        __syncthreads();
      }
    }
    if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    __threadfence();                                                       // the kept rows are read through L2
    tile_sync<C>();
    const int h = tid / Cfg::kTraceThreads, me = tid % Cfg::kTraceThreads;
    if (rank == 0 && h < tiles) {
      const int tile = first + h * (at_once / N);
      float *mem = tile_mem(h), *cone = mem + 2 * SJ + 2 * kVitMaxT;
      int jt = j0[0];
      float total = cost[0];
#pragma unroll
      for (int i = 1; i < N; ++i)
        if (i == h) { jt = j0[i]; total = cost[i]; }
      vit_trace<K, C, N, Cfg::kTraceThreads>(p, p.rows + (size_t)(cluster * N + h) * kept * SJ, mem, mem + SJ, mem + 2 * SJ, mem + 2 * SJ + kVitMaxT, cone,
                                             reinterpret_cast<int*>(cone + (Cfg::kCone + 4) / 4 * 4), jt, p.states + (size_t)tile * T, me, 1 + h);
      if (me == 0 && p.total) p.total[tile] = total;
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

// tiles that the GPU works on at once, in thread blocks (C = 1) of N tiles or in clusters of C
template <int K, int C, int N>
int resident(int* out) {
  static int cached[64] = {0};
  int dev = 0, sms = 0, per = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return (int)cudaErrorInvalidDevice;
  if (dev >= 0 && dev < 64 && cached[dev]) { *out = cached[dev]; return 0; }
  using Cfg = VitCfg<K, C, N>;
  cudaError_t e = cudaFuncSetAttribute(viterbi_kernel<K, C, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmem);
  if (e != cudaSuccess) return (int)e;
  if constexpr (C == 1) {
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return (int)e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, viterbi_kernel<K, C, N>, Cfg::kThreads, Cfg::kSmem)) != cudaSuccess) return (int)e;
    per *= sms * N;
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
    if ((e = cudaOccupancyMaxActiveClusters(&per, viterbi_kernel<K, C, N>, &cfg)) != cudaSuccess) return (int)e;
  }
  if (per < 1) return (int)cudaErrorLaunchOutOfResources;
  *out = per;
  if (dev >= 0 && dev < 64) cached[dev] = per;
  return 0;
}

// Which form searches the first `tiles` of B tiles: `split` thread blocks per tile, `pair` tiles per thread block.  The rest, if any, is
// planned by itself; it needs no more memory for kept rows.
struct VitPlan {
  int split, pair, tiles, blocks;   // blocks: thread blocks of the launch
  size_t rows_bytes;
};

template <int K>
constexpr bool kPairs2 = K >= 3;  // two tiles' cost arrays fit beside the codebook values

// Thread blocks per tile: as many as leave every tile a cluster of its own at once (few tiles leave SMs idle otherwise; a step of a
// shared tile pays a cluster barrier and stores its costs several times: 2^(16-K) of them, so that K = 2 gains nothing from four and K = 3
// nothing from either).  One block / two / four, ms: K = 3 0.85 / 0.91 / 0.85, K = 4 0.80 / 0.70 / 0.63, K = 5 0.84 / 0.70 / 0.56, K = 6
// 0.86 / 0.68 / 0.58, K = 8 1.06 / 0.76 / 0.68.
template <int K>
constexpr int kMostSplit = K == 2 ? 2 : K == 3 ? 1 : 4;
template <int K>
int plan(int B, int T, VitPlan* out) {
  int one = 0, two = 0, four = 0, pairs = 0;
  if (const int e = resident<K, 1, 1>(&one)) return e;
  if constexpr (kMostSplit<K> >= 2)
    if (resident<K, 2, 1>(&two)) { (void)cudaGetLastError(); two = 0; }
  if constexpr (kMostSplit<K> >= 4)
    if (resident<K, 4, 1>(&four)) { (void)cudaGetLastError(); four = 0; }
  if constexpr (kPairs2<K>)
    if (const int e = resident<K, 1, 2>(&pairs)) return e;
  VitPlan p = {1, 1, B, 0, 0};
  int tiles = 0;                                                           // with kept rows of their own
  if (B > one && pairs > 0) {
    p.pair = 2;
    if (B > pairs && B % pairs <= one) p.tiles = B - B % pairs;            // the last few in a form of their own
    p.blocks = pairs / 2 < p.tiles ? pairs / 2 : p.tiles;
    tiles = 2 * p.blocks;
  } else {
    p.split = B <= four ? 4 : B <= two ? 2 : 1;
    tiles = p.split > 1 || B < one ? B : one;
    p.blocks = tiles * p.split;
  }
  const int kept = (T - 1) / VitCfg<K, 1, 1>::kLevels;
  p.rows_bytes = (size_t)tiles * (kept > 0 ? kept : 1) * ((size_t)65536 >> K) * sizeof(float) + 16;   // (rows start on 16 bytes)
  *out = p;
  return 0;
}

int plan_for(int K, int B, int T, VitPlan* out) {
  switch (K) {
    case 2: return plan<2>(B, T, out);
    case 3: return plan<3>(B, T, out);
    case 4: return plan<4>(B, T, out);
    case 5: return plan<5>(B, T, out);
    case 6: return plan<6>(B, T, out);
    case 8: return plan<8>(B, T, out);
  }
  return (int)cudaErrorInvalidValue;
}

template <int K, int C, int N>
int launch_form(const VitParams& p, int blocks, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3(VitCfg<K, C, N>::kThreads);
  cfg.dynamicSmemBytes = VitCfg<K, C, N>::kSmem;
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = C > 1 ? 1 : 0;
  return (int)cudaLaunchKernelEx(&cfg, viterbi_kernel<K, C, N>, p);
}
template <int K>
int launch(const VitParams& p, const VitPlan& plan, cudaStream_t st) {
  if constexpr (kPairs2<K>)
    if (plan.pair == 2) return launch_form<K, 1, 2>(p, plan.blocks, st);
  if constexpr (kMostSplit<K> >= 4)
    if (plan.split == 4) return launch_form<K, 4, 1>(p, plan.blocks, st);
  if constexpr (kMostSplit<K> >= 2)
    if (plan.split == 2) return launch_form<K, 2, 1>(p, plan.blocks, st);
  return launch_form<K, 1, 1>(p, plan.blocks, st);
}

}  // namespace
}  // namespace htr

using namespace htr;

extern "C" {

size_t htr_viterbi_workspace_bytes(int B, int T, int K) {
  if (!width_ok(K) || B < 1 || T < 1 || T > kVitMaxT) return 0;
  VitPlan plan;
  return plan_for(K, B, T, &plan) == 0 ? plan.rows_bytes : 0;
}

int htr_viterbi(const float* x, const float* w, int B, int T, int K, int tailbite, int32_t* states, float* total, void* workspace,
                size_t workspace_bytes, htr_stream_t stream) {
  if (!width_ok(K)) return HTR_ERR_BAD_K;
  if (B < 0 || T < 1 || T > kVitMaxT) return HTR_ERR_BAD_SHAPE;
  if (B == 0) return HTR_OK;
  if (!x || !w || !states) return HTR_ERR_NULL;
  VitPlan plan;
  int e = plan_for(K, B, T, &plan);
  if (e) { t_vit_cuda = e; return HTR_ERR_CUDA; }
  if (!workspace || workspace_bytes < plan.rows_bytes) return HTR_ERR_WORKSPACE;
  const double inv = inverse_rms();
  VitParams p;
  p.rows = reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(workspace) + 15) & ~(uintptr_t)15);
  p.T = T;
  p.tailbite = tailbite ? 1 : 0;
  p.inv_hi = (float)inv;
  p.inv_lo = (float)(inv - (double)p.inv_hi);
  p.one = 1.0f;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  for (int done = 0; !e && done < B; done += plan.tiles) {                   // (launches of one stream share the kept rows in turn)
    if (done > 0 && (e = plan_for(K, B - done, T, &plan))) break;
    p.x = x + (size_t)done * T;
    p.w = w + (size_t)done * T;
    p.states = states + (size_t)done * T;
    p.total = total ? total + done : nullptr;
    p.B = plan.tiles;
    switch (K) {
      case 2: e = launch<2>(p, plan, st); break;
      case 3: e = launch<3>(p, plan, st); break;
      case 4: e = launch<4>(p, plan, st); break;
      case 5: e = launch<5>(p, plan, st); break;
      case 6: e = launch<6>(p, plan, st); break;
      case 8: e = launch<8>(p, plan, st); break;
    }
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
