// Packed GEMV for one activation row in a chain of dependent launches: one thread block per SM, decode and finishing overlapped.
//
//   y = sv * Ho( diag(scale * CB) * V * Hi(su * x) ),  V[i,j] = bytesum(h_ij) - 510      (the linear of packed_gemv.cuh)
//
// What bounds a dependent launch: the decode at an SM's issue rate, and what no
// weight is decoded in -- the release behind the predecessor, the staging of the activations, the hand-over of partial sums, the
// tail.  packed_gemv.cuh with three small thread blocks per SM hides those parts of overlapping launches from one another, but in a
// chain they add up, its blocks get 7 or 8 units each where 6.9 would do, and a scheduler serves its oldest warps first, so that
// the three blocks of an SM end one after the other and the last one decodes alone (12288x4096: 10 to 23 us).  Here
//  * every SM gets an even run of 128 x 128 blocks (flat over the row blocks), 16 decode warps take alternate blocks in two groups
//    (a barrier per trip to keep the warps of a group together cost 4 to 8 %);
//  * activations are staged once per SM, from one load per value also where a norm is folded in (the row stays in registers between
//    its sum of squares and the transform);
//  * at the end of a row block the decode warps leave their sums in shared memory and go on; four finisher warps add them, publish
//    and finish;
//  * a weight costs half an instruction less: its byte sum, as the bits of a float, is a subnormal number (n * 2^-149 exactly), and
//    multiplied with activations staged times 2^80 it needs neither a magic constant nor its subtraction.  The constant 510 goes in
//    per 16 columns, as -510 times their sum added to the accumulator first, so that the sums stay centred (no cancellation at the end).
// Every launch runs its code from cold instruction caches, so that what stands on the way to the first loads and behind the wait costs more
// than its instructions: run boundaries need no division (host, or the reciprocal of the blocks per row block), and the staging is
// compiled for one, two, five and seven blocks a warp instead of seven with most of them skipped (1024x4096 K4 4.65 -> 4.13, 4096x12288
// K4 12.7 -> 12.4, 1024x2048 K3 4.15 -> 3.63 us).  A round on zeros before the wait, as in the activation transform of the GEMM,
// was slower here (4.65 -> 6.5): a thread block starts when its SM is free, shortly before the wait ends.
// us per launch in a chain, bf16, packed_gemv.cuh -> here: 1024x4096 K4 6.4 -> 4.1, 4096x12288 K4 13.8 -> 12.4, 151936x4096 K4
// 131 -> 105 (5.9e12 weights a second, 20 per cycle and SM).
// Range.  A transformed activation beyond 2^46 overflows under the factor 2^80, and where all of a row lie below 2^-56 the products sink into the
// subnormals.  Both show in the sums of a row block: then all 128 are infinite, or all below 2^-33.  The barrier before the epilogue votes
// on that (the only cost to other rows: half a per cent), and such a row block is summed again by the finishers alone, slowly and
// without the factor (gemv1_any_range), so that the range of the results is that of packed_gemv.cuh.  Looking at the activations instead costs
// launches of the usual range 1 to 4 %: a vote at the barrier before the decode, votes of the staging warps and a second run of the
// thread block under another factor, a scan of the staged row by the finishers.
#pragma once
#include "packed_gemv.cuh"

namespace htr {

constexpr int kG1DecodeWarps = 16, kG1FinishWarps = 4, kG1Warps = kG1DecodeWarps + kG1FinishWarps, kG1Threads = kG1Warps * 32;
constexpr int kG1Alu = 2;                                    // byte sums of four that go to the shift/logic pipe (1, 3, 4: 2 to 3 % slower)
constexpr int kG1MaxCols = 16384;                            // staged activations of a row: 64 KB
constexpr float kG1Up = 1.2089258196146292e24f;              // 2^80: staged activations
constexpr float kG1Down = 1.6940658945086007e-21f;           // 2^-69 = 2^80 * 2^-149: unit of the accumulators
constexpr float kG1Out = 5.902958103587057e20f;              // 2^69
// A sum of at least this shows that its activations kept their bits: one of them, transformed, is then at least 2^-33 / (16384 columns * 510
// * 1.1) = 2^-56, and products near that are rounded at 2^-80, 2^-24 of the largest.
constexpr float kG1Least = 1.1641532e-10f;                   // 2^-33

template <int K>
struct G1Ring {
  static constexpr int tile_bytes = 32 * K, slot_bytes = 8 * tile_bytes;      // one warp, one trip: four strips x two units
  static constexpr int slots = K <= 3 ? 5 : K <= 5 ? 4 : 3;
  static constexpr int bytes = kG1DecodeWarps * slots * slot_bytes;
};
template <int K>
constexpr int gemv1_smem_bytes(int n) { return G1Ring<K>::bytes + n * 4 + (n / 16) * 4; }

template <int ID, int COUNT>
__device__ __forceinline__ void named_sync() {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(COUNT) : "memory");
}
__device__ __forceinline__ void named_sync_at(int id, int count) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void named_arrive_at(int id, int count) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

// 32 weights (two tile rows x 16 columns) of a lane against the tile's staged activations
template <int K, int ALU4>
__device__ __forceinline__ void unit_fma_subnormal(const uint32_t (&V)[K + 1], const float* __restrict__ xs, float offset, float2 (&acc)[2]) {
  uint32_t s[32];
  unit_states<K>(V, s);
  acc[0].x += offset;
  acc[1].x += offset;
#pragma unroll
  for (int quad = 0; quad < 4; ++quad) {
    const float4 xv = *reinterpret_cast<const float4*>(xs + quad * 4);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c0 = staged_col_inv<K>(quad * 4 + half * 2), c1 = staged_col_inv<K>(quad * 4 + half * 2 + 1);
      const float2 xp = half ? make_float2(xv.z, xv.w) : make_float2(xv.x, xv.y);
#pragma unroll
      for (int rr = 0; rr < 2; ++rr) {
        const uint32_t h0 = s[rr * 16 + c0] * kGenMul + kGenAdd, h1 = s[rr * 16 + c1] * kGenMul + kGenAdd;
        const uint32_t b0 = (2 * half + 2 * rr) % 4 < ALU4 ? bytesum_add_alu(h0, 0u) : bytesum_add(h0, 0u);
        const uint32_t b1 = (2 * half + 2 * rr + 1) % 4 < ALU4 ? bytesum_add_alu(h1, 0u) : bytesum_add(h1, 0u);
        acc[rr] = __ffma2_rn(make_float2(__uint_as_float(b0), __uint_as_float(b1)), xp, acc[rr]);
      }
    }
  }
}

// barrier of the finishers; true where any of them brings true
__device__ __forceinline__ bool finishers_any(bool mine) {
  int any;
  __syncwarp();
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.or.pred p, 5, %2, q;\n\tselp.s32 %0, 1, 0, p;\n\t}"
               : "=r"(any)
               : "r"((int)mine), "n"(kG1FinishWarps * 32)
               : "memory");
  return any != 0;
}

// The sum of row r of row block rb over all its columns, by the finishers alone and without the factor 2^80: for activations whose sums
// left the range of the fast form (see Range above).  Four 128-column blocks at a time; f holds their transformed activations.
template <int K>
static __device__ __noinline__ float gemv1_any_range(const GemvParams& p, float (*f)[128], int rb, int r) {
  const int nt = p.nt, n = nt * 16, HB = nt >> 3, lane = r & 31, fw = r >> 5, q = (r & 15) >> 1;
  float ss = 0.f;
  bool some = false;                                         // (a row of zeros ends here: its sums are zeros as they are)
  for (int col = 4 * r; col < n; col += 4 * kG1FinishWarps * 32) {
    const float4 v = load_x(p.x, 0, col, p.n_in, p.dtype);
    ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    some = some || v.x != 0.f || v.y != 0.f || v.z != 0.f || v.w != 0.f;
  }
  if (!finishers_any(some)) return 0.f;
  float inv = 0.f;
  if (p.prologue == 1) {
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(kFullWarp, ss, o);
    if (lane == 0) f[0][fw] = ss;
    named_sync<5, kG1FinishWarps * 32>();
    inv = rsqrtf((f[0][0] + f[0][1] + f[0][2] + f[0][3]) / (float)n + p.eps);
    named_sync<5, kG1FinishWarps * 32>();
  }
  const uint32_t* strip = p.qw + (size_t)(rb * 8 + (r >> 4)) * nt * (8 * K);
  float sum = 0.f;
#pragma unroll 1
  for (int first = 0; first < HB; first += kG1FinishWarps) {
    const int hb = first + fw, col = hb * 128 + 4 * lane;
    if (hb < HB) {
      float4 x4 = load_x(p.x, 0, col, p.n_in, p.dtype);
      if (p.prologue == 1) x4 = norm_x(x4, __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p.norm_w) + col)), inv);
      const unsigned sg = sign_nibble(p.su, hb * 32 + lane);
      float v[4] = {flip(x4.x, sg & 1u), flip(x4.y, (sg >> 1) & 1u), flip(x4.z, (sg >> 2) & 1u), flip(x4.w, sg >> 3)};
      wht128(v, lane);
#pragma unroll
      for (int k = 0; k < 4; ++k) f[fw][4 * lane + k] = v[k] * kInvSqrt128;
    }
    named_sync<5, kG1FinishWarps * 32>();
#pragma unroll 1
    for (int tile = 0; tile < 8 * min(kG1FinishWarps, HB - first); ++tile) {
      uint32_t V[K + 1], s[32];
      read_unit_words<K>(strip + (size_t)(first * 8 + tile) * (8 * K), q, V);
      unit_states<K>(V, s);
      float part = 0.f;
#pragma unroll
      for (int c = 0; c < 16; ++c) {
        const uint32_t h = (r & 1 ? s[16 + c] : s[c]) * kGenMul + kGenAdd;
        part += (float)((int)bytesum_add(h, 0u) - 510) * f[tile >> 3][(tile & 7) * 16 + c];
      }
      sum += part;
    }
    named_sync<5, kG1FinishWarps * 32>();
  }
  return sum;
}

// HELD: 128-column blocks of activations that a warp stages at most
template <int K, int HELD>
__global__ void __launch_bounds__(kG1Threads, 1) packed_gemv1_kernel(const __grid_constant__ GemvParams p) {
  using Ring = G1Ring<K>;
  constexpr int kTileBytes = Ring::tile_bytes, kSlotBytes = Ring::slot_bytes, R = Ring::slots;
  extern __shared__ __align__(128) unsigned char dyn_smem[];
  __shared__ __align__(16) float s_red[2][kG1DecodeWarps][64];   // sums of a row block: [buffer][decode warp][its 64 rows]
  __shared__ __align__(16) float ytil[128];
  __shared__ float s_ss[kG1Warps];
  __shared__ int s_arrival;
  __shared__ __align__(16) float s_any[kG1FinishWarps][128];   // gemv1_any_range
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nt = p.nt, n = nt * 16, HB = nt >> 3;
  // (no divisions on the way to the first loads: a few dozen cold instructions each)
  const EvenRuns runs(p.run_q, p.run_rem, 0);
  const int u_begin = runs.begin(blockIdx.x), u_end = runs.begin(blockIdx.x + 1);
  const auto row_block = [&](int u) { return p.hb_magic ? (int)__umulhi((unsigned)u, p.hb_magic) : u; };
  const int rb0 = row_block(u_begin), hb0 = u_begin - rb0 * HB;
  float* xs = reinterpret_cast<float*>(dyn_smem + Ring::bytes);  // [n] staged activations, by column
  float* xoff = xs + n;                                          // [n / 16] offset of every tile

  // ---- decode warps: copy cursor over every second block of the run (warp = 64 rows h x tile column c of either unit)
  const int h = warp & 1, c = (warp >> 1) & 3, group = warp >> 3, g = lane >> 3, q = lane & 7;
  const unsigned char* my_ring = dyn_smem + ((warp < kG1DecodeWarps ? warp : 0) * R * 8 + g) * kTileBytes;
  const uint32_t ring_dst = (uint32_t)__cvta_generic_to_shared(my_ring) + q * 16;
  const int on_tail = (q + 8 * ((2 * K - 1) / 8) < 2 * K) ? -1 : 0;
  const size_t next_strip = (size_t)7 * nt * kTileBytes * (HB == 1 ? 2 : 1);
  int pf_left = 0, pf_in_rb = 1;
  const char* pf = nullptr;
  auto fetch = [&](uint32_t at) {
    GemvTripCopies<K, 0, 0>::run(ring_dst + at, pf, pf_left, pf_left & on_tail);
    pf_left -= 2;
    const bool wrap = pf_in_rb <= 2;
    pf_in_rb += wrap ? HB - 2 : -2;
    pf += wrap ? next_strip + 16 * kTileBytes : (size_t)(16 * kTileBytes);
    async_commit();
  };
  if (warp < kG1DecodeWarps) {
    const bool next = hb0 + group >= HB;                     // (HB = 1: the second group begins in the next row block)
    const int rb = rb0 + (next ? 1 : 0), hb = next ? 0 : hb0 + group;
    pf_left = max(u_end - u_begin - group, 0);
    pf_in_rb = HB - hb;
    pf = reinterpret_cast<const char*>(p.qw) + ((size_t)(rb * 8 + 4 * h + g) * nt + (size_t)hb * 8 + c) * kTileBytes + q * 16;
#pragma unroll
    for (int i = 0; i < R - 1; ++i) fetch(i * kSlotBytes);   // the weights do not depend on the preceding kernel
  }
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // ---- activations of every column this thread block meets: `count` blocks from its first one on, around the end of the row.
  // A warp takes every 20th; signs and norm weights do not depend on the preceding kernel and are fetched before the wait
  constexpr int kHeld = HELD;
  const int count = min(u_end - u_begin, HB);
  auto block_at = [&](int i) { const int hb = hb0 + warp + kG1Warps * i; return hb >= HB ? hb - HB : hb; };
  unsigned signs[kHeld];
  uint2 gain[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    signs[i] = 0u;
    gain[i] = make_uint2(0u, 0u);
    if (warp + kG1Warps * i < count) {
      // (in assembly so that nothing waits for the byte here)
      asm volatile("ld.global.nc.u8 %0, [%1];" : "=r"(signs[i]) : "l"(p.su + block_at(i) * 16 + (lane >> 1)));
      if (p.prologue == 1) gain[i] = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(p.norm_w) + block_at(i) * 128 + 4 * lane));
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");

  auto stage = [&](int hb, unsigned sg, float4 x4) {
    float v[4] = {flip(x4.x, sg & 1u), flip(x4.y, (sg >> 1) & 1u), flip(x4.z, (sg >> 2) & 1u), flip(x4.w, sg >> 3)};
    wht128(v, lane);
    float* dst = xs + hb * 128 + (lane >> 2) * 16;
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float f = v[k] * kInvSqrt128;
      dst[staged_col<K>(4 * (lane & 3) + k)] = f * kG1Up;
      sum += f;
    }
    sum += __shfl_xor_sync(kFullWarp, sum, 1);
    sum += __shfl_xor_sync(kFullWarp, sum, 2);
    if ((lane & 3) == 0) xoff[hb * 8 + (lane >> 2)] = -510.0f * sum * kG1Down;
  };
  float4 held[kHeld];                                        // every load of a warp is in flight before the first is used
  if (p.prologue == 1) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < kHeld; ++i)                          // the whole row, for its sum of squares
      held[i] = warp + kG1Warps * i < HB ? load_quad(p.x, block_at(i) * 128 + 4 * lane, p.dtype) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kHeld; ++i) ss += held[i].x * held[i].x + held[i].y * held[i].y + held[i].z * held[i].z + held[i].w * held[i].w;
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(kFullWarp, ss, o);
    if (lane == 0) s_ss[warp] = ss;
    __syncthreads();
    float tot = 0.f;
#pragma unroll
    for (int k = 0; k < kG1Warps; ++k) tot += s_ss[k];
    const float inv = rsqrtf(tot / (float)n + p.eps);
#pragma unroll
    for (int i = 0; i < kHeld; ++i) held[i] = norm_x(held[i], gain[i], inv);
  } else {                                                   // (other prologues and the residual form do not come here)
#pragma unroll
    for (int i = 0; i < kHeld; ++i)
      if (warp + kG1Warps * i < count) held[i] = load_x(p.x, 0, block_at(i) * 128 + 4 * lane, p.n_in, p.dtype);
  }
#pragma unroll
  for (int i = 0; i < kHeld; ++i)
    if (warp + kG1Warps * i < count) stage(block_at(i), (signs[i] >> (4 * (lane & 1))) & 15u, held[i]);
  __syncthreads();

  if (warp < kG1DecodeWarps) {
    float2 acc[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    uint32_t at = 0u, refill = (R - 1) * kSlotBytes;         // ring slots of this trip and of the one before it
    int seg = 0, u = u_begin + group;
    for (int start = u_begin; start < u_end; ++seg) {
      const int rb = rb0 + seg, stop = min(u_end, (rb + 1) * HB);
      const float* xt = xs + (u - rb * HB) * 128 + c * 16;
      const float* ot = xoff + (u - rb * HB) * 8 + c;
#pragma unroll 1
      for (; u < stop; u += 2) {
        async_wait<R - 2>();                                 // this trip's words have landed (own copies) ...
        __syncwarp();                                        // ... and those of the other lanes; the slot before it is free
        fetch(refill);
        const uint32_t* tiles = reinterpret_cast<const uint32_t*>(my_ring + at);
        refill = at;
        at = at == (R - 1) * kSlotBytes ? 0u : at + kSlotBytes;
        uint32_t V[K + 1];
        read_unit_words<K>(tiles, q, V);
        unit_fma_subnormal<K, kG1Alu>(V, xt, ot[0], acc);
        read_unit_words<K>(tiles + 8 * K * 4, q, V);
        unit_fma_subnormal<K, kG1Alu>(V, xt + 64, ot[4], acc);
        xt += 256;
        ot += 16;
      }
      // ---- this warp's part of row block rb: leave it for the finishers (two buffers)
      const int buf = seg & 1;
      if (seg >= 2) named_sync_at(3 + buf, kG1Threads);
      *reinterpret_cast<float2*>(&s_red[buf][warp][g * 16 + 2 * q]) = make_float2(acc[0].x + acc[0].y, acc[1].x + acc[1].y);
      acc[0] = acc[1] = make_float2(0.f, 0.f);
      named_arrive_at(1 + buf, kG1Threads);
      start = stop;
    }
    async_wait<0>();
    return;
  }

  // ---- finishers: thread r owns row r of the row block
  const int r = tid - kG1DecodeWarps * 32, segs = row_block(u_end - 1) - rb0 + 1;
  for (int seg = 0; seg < segs; ++seg) {
    const int rb = rb0 + seg, buf = seg & 1;
    const int first = runs.owner(rb * HB), contributors = runs.owner((rb + 1) * HB - 1) - first + 1;
    // operands of the epilogue are fetched now so that their latency hides behind the hand-over
    const int row0 = rb * 128 + 4 * lane;
    const uint2 sc_raw = __ldg(reinterpret_cast<const uint2*>(p.scales + row0));
    const unsigned sv_bits = sign_nibble(p.sv, rb * 32 + lane);
    float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < 32 && row0 < p.m_out && p.bias) bias4 = load_quad(p.bias, row0, p.dtype);
    named_sync_at(1 + buf, kG1Threads);
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kG1DecodeWarps / 2; ++w) sum += s_red[buf][2 * w + (r >> 6)][r & 63];
    if (seg + 2 < segs) named_arrive_at(3 + buf, kG1Threads);
    bool finish = true;
    if (contributors > 1) {
      // a thread block has two partials: its first row block's and that of a later one (only its last is read by others)
      __stcg(p.part + (size_t)(2 * blockIdx.x + (seg > 0 ? 1 : 0)) * 128 + r, sum);
      named_sync<5, kG1FinishWarps * 32>();
      if (r == 0) {
        __threadfence();                                     // the partials of the thread block (ordered by the barrier) before the arrival
        s_arrival = atomicAdd(p.counters + rb, 1);           // (they are read with loads served by L2, after this atomic)
      }
      named_sync<5, kG1FinishWarps * 32>();
      finish = s_arrival == contributors - 1;
      if (finish) {
        if (r == 0) p.counters[rb] = 0;
        const int head = runs.begin(first) < rb * HB ? 1 : 0;
        const float* slot0 = p.part + (size_t)(2 * first) * 128 + r;
        sum = 0.f;
        for (int base = 0; base < contributors; base += 8) { // loads in flight together, added in thread-block order
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = base + j < contributors ? __ldcg(slot0 + (size_t)(base + j == 0 ? head : 2 * (base + j)) * 128) : 0.f;
#pragma unroll
          for (int j = 0; j < 8; ++j) sum += v[j];
        }
      }
    }
    if (!finish) continue;
    sum *= kG1Out;
    ytil[r] = sum;
    if (!finishers_any(fabsf(sum) >= kG1Least && fabsf(sum) <= 3.402823466e38f)) {
      sum = gemv1_any_range<K>(p, s_any, rb, r);
      ytil[r] = sum;
      named_sync<5, kG1FinishWarps * 32>();
    }
    if (r < 32) {
      const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&sc_raw.x)), s23 = __half22float2(*reinterpret_cast<const __half2*>(&sc_raw.y));
      const float4 y4 = *reinterpret_cast<const float4*>(ytil + 4 * lane);
      float v[4] = {y4.x * (s01.x * p.cb), y4.y * (s01.y * p.cb), y4.z * (s23.x * p.cb), y4.w * (s23.y * p.cb)};
      wht128(v, lane);
      float4 o = make_float4(flip(v[0] * kInvSqrt128, sv_bits & 1u) + bias4.x, flip(v[1] * kInvSqrt128, (sv_bits >> 1) & 1u) + bias4.y,
                             flip(v[2] * kInvSqrt128, (sv_bits >> 2) & 1u) + bias4.z, flip(v[3] * kInvSqrt128, sv_bits >> 3) + bias4.w);
      if (row0 < p.m_out) store_quad(p.y, row0, p.dtype, o);
    }
    // (ytil is written again only behind the next barrier with the decode warps, which warp 0 reaches after this)
  }
}

// host side, defined once per K in packed_gemv_k*.cu
template <int K>
int launch_packed_gemv1(const GemvParams& p, int grid, cudaStream_t stream);

}  // namespace htr
