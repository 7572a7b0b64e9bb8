// C entry points of the tensor-core packed GEMM (batches of up to 256 activation rows per call).
#include <cmath>
#include <type_traits>

#include "packed_gemm_tc.cuh"

namespace htr {

// ------------------------------------------------------------------------------------------------
// Activation transform for the GEMM: xt = H128(su * x) / sqrt(128) / tok as one or two fp16 planes, their sums, tok.
// Output layout = the B operand tiles of the GEMM, one contiguous block per 128 columns of x:
//   xb[64-column unit][column group g][k-group kc][column r][8 k]   column = g*8 + r: activation row (hi plane), np + row (lo plane)
// with the k order of the A operand inside a unit (packed_gemm_tc.cuh): position 16 j + 4 c + e holds column 16 c + 4 j + e.
// A thread block transforms one slice of one activation row, after finding the range of the whole row itself (16 bytes per load; cheaper
// than an exchange between slices).  xsum[row][i] holds the sum of the i-th 8 `per` blocks.  Butterflies go from the lowest column bit to
// the highest, and sums are formed over four columns of every eighth block, the 32 fours of a block (halves, quarters, ...) and eight
// blocks one after another, whatever the form and the grid: dozens of bf16 layers turn another order into percents.  Columns from n_in
// on read as zeros; B columns of the padded batch that have no row stay as they are: they reach only accumulator columns that nobody reads.
//
// What bounds it: latency -- of the wait for the kernel before it, of the row, of instructions that nobody has fetched yet (a kernel this
// short runs every line once) -- and the stores, 16 bytes apart by the B layout, a line of L1 each.  Two forms:
//  * one block per warp and turn, a thread block per sum: four columns a lane, so that a value crosses lanes five times, and every block of
//    a short row has a warp of its own;
//  * four blocks per warp, eight lanes each, a lane the 16 columns of one tile: a value crosses lanes three times, and one thread block takes
//    a whole row or half of one.  Few thread blocks matter before a GEMM in clusters: those that do not fit on the SMs that the GEMM before
//    leaves free keep its successor's clusters waiting.
// us for transform + GEMM in a chain (graph) and behind an elementwise kernel, one block per warp / four: 1024x640 K4 16 rows 5.3, 7.2 / 5.7,
// 7.3; 2048x2048 K4 96 rows 9.7, 11.5 / 10.3, 12.1; 4096x4096 K4 37 rows 11.8, 12.1 / 9.6, 12.8; 4096x12288 K5 16 rows 20.9, 21.4 / 17.7, 19.8.
// (All warps through the code once on zeros before the wait, to fetch its instructions: nothing in a chain, where the wait is long, and 0.7 to
// 1.7 us more behind a kernel that lets its successors go at its end only; 4096x12288 K5 16 rows 17.7, 21.4.)
//
// Range scale of a row: the power of two 2^k with max|x| * sqrt(128) in (2^13, 2^14] * 2^k, in both directions, so that neither a large
// row leaves the fp16 range nor a small one sinks into its subnormals (fp16 numbers are 2^-24 apart below 2^-14: unscaled, a row of
// rms 1e-5 kept 9 bits).  |H128 x| / sqrt(128) <= sqrt(128) * max|x|.  k stays in [-120, 118], so that the scale, its reciprocal and
// their products with 1/sqrt(128) are normal float32 numbers; two planes carry 4e-8 (2-norm) down to rows of rms 1e-36, 3e-7 at 3e-38.
// The epilogue multiplies by 2^k last, so that the steps before it see ordinary magnitudes.
__device__ __forceinline__ float range_scale(float mx) {
  const uint32_t bits = __float_as_uint(mx * (11.32f / 16384.f));
  const uint32_t e = (bits >> 23) + ((bits & 0x7FFFFFu) != 0u);   // rounded up; inf and NaN end at the upper limit, zero at the lower
  return __uint_as_float(min(max(e, 127u - 120u), 127u + 118u) << 23);
}

constexpr int kRhtWarps = 24, kRhtBlocks = 512;              // (blocks of a slice: longer rows take more slices)

template <int DT>
__global__ void __launch_bounds__(1024) rht_f16_kernel(const void* __restrict__ x, int np, int n, int n_in, int planes,
                                                                 const uint8_t* __restrict__ su, __half* __restrict__ xb, float* __restrict__ xsum,
                                                                 float* __restrict__ tok, int per) {
  __shared__ unsigned red_top[kRhtWarps];
  __shared__ float block_sum[kRhtBlocks];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the GEMM may start fetching packed words now
  const int r = blockIdx.x, slice = blockIdx.y, slices = gridDim.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const int blocks = n >> 7, sums = (blocks + 8 * per - 1) / (8 * per), own = (sums + slices - 1) / slices;   // sums of a row, of this slice
  const int u = (lane >> 2) & 1, c = lane & 3;               // this lane's tile inside a block of a group
  const int ncols = np * planes;
  // column 16 c + 4 j + e of unit u goes to position 16 j + 4 c + e
  __half* const out = xb + (size_t)u * ncols * 64 + (size_t)(r >> 3) * 512 + (r & 7) * 8 + (c >> 1) * 64 + 4 * (c & 1);
  const size_t to_lo = (size_t)(np >> 3) * 512;
  constexpr int kPer16 = DT == HTR_DTYPE_F32 ? 4 : 8;        // elements in 16 bytes
  const char* const row = static_cast<const char*>(x) + (size_t)r * n_in * (16 / kPer16);
  const int first = 8 * per * slice * own, col0 = 64 * u + 16 * c;
  asm volatile("griddepcontrol.wait;" ::: "memory");         // x may come from the preceding kernel, the last GEMM may still read xb
  // range of the whole row: magnitudes of floats compare like their bit patterns, so 16-bit pairs take the packed integer maximum
  uint32_t top = 0u;
  const uint4* row16 = reinterpret_cast<const uint4*>(row);
#pragma unroll 1                                             // (few turns, and every line is fetched cold: by four, 4096x12288 K5, 16 rows 17.7 -> 18.0 us)
  for (int e = threadIdx.x; e < n_in / kPer16; e += blockDim.x) {
    const uint4 v = __ldg(row16 + e);
    if constexpr (DT == HTR_DTYPE_F32) {
      constexpr uint32_t m = 0x7FFFFFFFu;
      top = max(max(top, v.x & m), max(v.y & m, max(v.z & m, v.w & m)));
    } else {
      constexpr uint32_t m = 0x7FFF7FFFu;
      top = __vmaxu2(__vmaxu2(top, v.x & m), __vmaxu2(v.y & m, __vmaxu2(v.z & m, v.w & m)));
    }
  }
  if constexpr (DT != HTR_DTYPE_F32) top = max(top >> 16, top & 0xFFFFu);
  top = __reduce_max_sync(kFullWarp, top);
  if (lane == 0) red_top[warp] = top;
  __syncthreads();
  top = __reduce_max_sync(kFullWarp, lane < warps ? red_top[lane] : 0u);
  float mx;
  if constexpr (DT == HTR_DTYPE_F32) mx = __uint_as_float(top);
  else if constexpr (DT == HTR_DTYPE_BF16) mx = __uint_as_float(top << 16);
  else mx = __half2float(__ushort_as_half((unsigned short)top));
  const float scale = range_scale(mx), inv = kInvSqrt128 / scale;
#pragma unroll 1
  for (int g = warp; g < 2 * own; g += warps) {              // half of the blocks of a sum: four of every eight
    float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
    for (int i8 = 0; i8 < per; ++i8) {
      const int hb = first + 8 * (per * (g >> 1) + i8) + 4 * (g & 1) + (lane >> 3);
      float2 v[8];
      const int col = hb * 128 + col0;
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const float4 q = hb < blocks && col + 4 * h < n_in ? load_quad(row, col + 4 * h, DT) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[2 * h] = make_float2(q.x, q.y);
        v[2 * h + 1] = make_float2(q.z, q.w);
      }
      const int byte = hb < blocks ? col >> 3 : 0;
      const uint32_t signs = (uint32_t)su[byte] | ((uint32_t)su[byte + 1] << 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = make_float2(flip(v[i].x, (signs >> (2 * i)) & 1u), flip(v[i].y, (signs >> (2 * i + 1)) & 1u));
#pragma unroll
      for (int i = 0; i < 8; ++i) v[i] = make_float2(v[i].x + v[i].y, v[i].x - v[i].y);
      const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
      for (int bit = 1; bit < 8; bit <<= 1)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (!(i & bit)) {
            const float2 a = v[i], b = v[i | bit];
            v[i] = __fadd2_rn(a, b);
            v[i | bit] = __ffma2_rn(b, minus, a);                    // a - b, as rounded
          }
#pragma unroll
      for (int bit = 1; bit < 8; bit <<= 1) {
        const float sgn = (lane & bit) ? -1.0f : 1.0f;               // the upper partner of a butterfly keeps (other - own)
#pragma unroll
        for (int i = 0; i < 8; ++i)
          v[i] = make_float2(fmaf(sgn, v[i].x, __shfl_xor_sync(kFullWarp, v[i].x, bit)), fmaf(sgn, v[i].y, __shfl_xor_sync(kFullWarp, v[i].y, bit)));
      }
      __half* const at = out + (size_t)hb * ncols * 128;
      const bool store = hb < blocks;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        __half2 hi[2], lo[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 t = __fmul2_rn(v[2 * j + e], make_float2(inv, inv));
          hi[e] = __float22half2_rn(t);
          const float2 back = __half22float2(hi[e]);
          lo[e] = __float22half2_rn(__ffma2_rn(back, minus, t));
          const float2 rest = __half22float2(lo[e]);
          sum[j] += planes == 2 ? back.x + rest.x : back.x;          // exactly what the MMA will see
          sum[j] += planes == 2 ? back.y + rest.y : back.y;
        }
        if (store) *reinterpret_cast<uint2*>(at + 128 * j) = *reinterpret_cast<const uint2*>(hi);
        if (store && planes == 2) *reinterpret_cast<uint2*>(at + 128 * j + to_lo) = *reinterpret_cast<const uint2*>(lo);
      }
    }
    // the sum over the fours of a block, index 4 w + j in lane w: bits 4 and 3 by an exchange of halves (a lane keeps what its own bit says),
    // then bits 2, 1 and 0
    const int w = lane & 7;
    const bool upper = w & 4, second = w & 2;
    float a = (upper ? sum[2] : sum[0]) + __shfl_xor_sync(kFullWarp, upper ? sum[0] : sum[2], 4);
    const float b = (upper ? sum[3] : sum[1]) + __shfl_xor_sync(kFullWarp, upper ? sum[1] : sum[3], 4);
    a = (second ? b : a) + __shfl_xor_sync(kFullWarp, second ? a : b, 2);
    a += __shfl_xor_sync(kFullWarp, a, 1);
    a += __shfl_xor_sync(kFullWarp, a, 4);
    a += __shfl_xor_sync(kFullWarp, a, 2);
    if (w == 0) block_sum[4 * g + (lane >> 3)] = a;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < own; i += blockDim.x) {
    float all = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) all += block_sum[8 * i + k];
    const int at = slice * own + i;
    if (at < sums) xsum[(size_t)r * sums + at] = all;
  }
  if (slice == 0 && threadIdx.x == 0) tok[r] = scale;
}

// One block per warp and turn: grid (rows, sums of a row), 8 warps
template <int DT>
__global__ void __launch_bounds__(256) rht_f16_short_kernel(const void* __restrict__ x, int np, int n, int n_in, int planes,
                                                            const uint8_t* __restrict__ su, __half* __restrict__ xb, float* __restrict__ xsum,
                                                            float* __restrict__ tok, int per) {
  __shared__ float red[8];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");   // the GEMM may start fetching packed words now
  const int r = blockIdx.x, slice = blockIdx.y, slices = gridDim.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int blocks = n >> 7;
  const int hb0 = slice * 8 * per + warp;                    // this warp's 128-column blocks: hb0, hb0 + 8, ... (`per` of them)
  const int ncols = np * planes;
  const size_t unit_halves = (size_t)ncols * 64;
  const size_t col_hi = (size_t)(r >> 3) * 512 + (r & 7) * 8, col_lo = (size_t)((np + r) >> 3) * 512 + ((np + r) & 7) * 8;
  // four consecutive columns 4 lane .. + 3 of a block: tile c = (lane % 16) / 4, step j = lane % 4 of unit lane / 16
  const int c = (lane & 15) >> 2, j = lane & 3;
  const size_t in_unit = (size_t)(2 * j + (c >> 1)) * 64 + 4 * (c & 1);
  auto tile_offset = [&](int hb) { return (size_t)(2 * hb + (lane >> 4)) * unit_halves + in_unit; };
  const unsigned sg_first = hb0 < blocks ? sign_nibble(su, hb0 * 32 + lane) : 0u;   // the signs do not depend on earlier kernels
  asm volatile("griddepcontrol.wait;" ::: "memory");         // x may come from the preceding kernel, the last GEMM may still read xb
  // this lane's values of its first block: the load is in flight beside those of the scan
  auto values = [&](int hb) {
    const int col = hb * 128 + 4 * lane;
    return hb < blocks && col < n_in ? load_quad(x, (size_t)r * n_in + col, DT) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  const float4 first = values(hb0);
  // range of the whole row: magnitudes of floats compare like their bit patterns, so 16-bit pairs take the packed integer maximum
  uint32_t top = 0u;
  constexpr int kPer16 = DT == HTR_DTYPE_F32 ? 4 : 8;        // elements in 16 bytes
  const uint4* row16 = reinterpret_cast<const uint4*>(static_cast<const char*>(x) + (size_t)r * n_in * (16 / kPer16));
#pragma unroll 8
  for (int e = tid; e < n_in / kPer16; e += 256) {
    const uint4 v = __ldg(row16 + e);
    if constexpr (DT == HTR_DTYPE_F32) {
      constexpr uint32_t m = 0x7FFFFFFFu;
      top = max(max(top, v.x & m), max(v.y & m, max(v.z & m, v.w & m)));
    } else {
      constexpr uint32_t m = 0x7FFF7FFFu;
      top = __vmaxu2(__vmaxu2(top, v.x & m), __vmaxu2(v.y & m, __vmaxu2(v.z & m, v.w & m)));
    }
  }
  if constexpr (DT != HTR_DTYPE_F32) top = max(top >> 16, top & 0xFFFFu);
  top = __reduce_max_sync(kFullWarp, top);
  if (lane == 0) red[warp] = __uint_as_float(top);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 8; ++k) top = max(top, __float_as_uint(red[k]));
  float mx;
  if constexpr (DT == HTR_DTYPE_F32) mx = __uint_as_float(top);
  else if constexpr (DT == HTR_DTYPE_BF16) mx = __uint_as_float(top << 16);
  else mx = __half2float(__ushort_as_half((unsigned short)top));
  const float scale = range_scale(mx);
  if (tid == 0 && slice == 0) tok[r] = scale;
  const float inv = kInvSqrt128 / scale;
  float sum = 0.f;
#pragma unroll 2
  for (int i = 0; i < per; ++i) {
    const int hb = hb0 + 8 * i;
    if (hb >= blocks) break;                                 // warp-uniform: the shuffles inside stay converged
    const float4 mine = i == 0 ? first : values(hb);         // (second touch: L1)
    const unsigned sg = i == 0 ? sg_first : sign_nibble(su, hb * 32 + lane);
    float v[4] = {flip(mine.x, sg & 1u), flip(mine.y, (sg >> 1) & 1u), flip(mine.z, (sg >> 2) & 1u), flip(mine.w, sg >> 3)};
    wht128(v, lane);
    __half hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float t = v[k] * inv;
      hi[k] = __float2half_rn(t);
      lo[k] = __float2half_rn(t - __half2float(hi[k]));
      sum += planes == 2 ? __half2float(hi[k]) + __half2float(lo[k]) : __half2float(hi[k]);   // exactly what the MMA will see
    }
    const size_t at = tile_offset(hb);
    *reinterpret_cast<uint2*>(xb + at + col_hi) = *reinterpret_cast<const uint2*>(hi);
    if (planes == 2) *reinterpret_cast<uint2*>(xb + at + col_lo) = *reinterpret_cast<const uint2*>(lo);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFullWarp, sum, o);
  __syncthreads();
  if (lane == 0) red[warp] = sum;
  __syncthreads();
  if (tid == 0) {
    float s = 0.f;
    for (int k = 0; k < 8; ++k) s += red[k];
    xsum[(size_t)r * slices + slice] = s;
  }
}

// ------------------------------------------------------------------------------------------------
// Plan of a mixture-of-experts step for the grouped GEMM: the (token, slot) pairs sorted by expert and cut into tiles of up to
// kGroupRows pairs, so that an expert's weights are decoded once per tile instead of once per pair.  One thread block; a warp
// takes every 32nd expert and finds its pairs, in order, with one ballot per 32 route entries (a few hundred to a few thousand
// entries: the launch is what it costs).  Entries outside the tables and absent experts (null weight) get no tile.
// slot_of[pair] (behind the plan) = tile * kGroupRows + row, or -1.
constexpr int kPlanThreads = 1024;
__global__ void __launch_bounds__(kPlanThreads) route_plan_kernel(const long long* __restrict__ route, int count, int experts, const uint32_t* const* qw,
                                                                  int* __restrict__ plan, int cap) {
  extern __shared__ int plan_smem[];                         // [experts] pairs, then first tile of every expert; [count] routes
  int* first_tile = plan_smem;
  int* ids = plan_smem + experts;
  __shared__ int warp_sum[kPlanThreads / 32];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");         // the route comes from the router's kernel, the last step may still read the plan
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int* slot_of = plan + group_plan_ints(cap);
  for (int i = tid; i < count; i += kPlanThreads) {
    const long long e = route[i];
    const bool ok = e >= 0 && e < experts && qw[e] != nullptr;
    ids[i] = ok ? (int)e : -1;
    if (!ok) slot_of[i] = -1;
  }
  __syncthreads();
  for (int e = warp; e < experts; e += kPlanThreads / 32) {
    int n = 0;
    for (int base = 0; base < count; base += 32) n += __popc(__ballot_sync(kFullWarp, base + lane < count && ids[base + lane] == e));
    if (lane == 0) first_tile[e] = (n + kGroupRows - 1) / kGroupRows;
  }
  __syncthreads();
  // exclusive sum of the tile counts over the experts
  int running = 0;
  for (int base = 0; base < experts; base += kPlanThreads) {
    const int e = base + tid, own = e < experts ? first_tile[e] : 0;
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(kFullWarp, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warp_sum[warp] = incl;
    __syncthreads();
    int before = 0, all = 0;
    for (int w = 0; w < kPlanThreads / 32; ++w) {
      if (w < warp) before += warp_sum[w];
      all += warp_sum[w];
    }
    __syncthreads();
    if (e < experts) first_tile[e] = running + before + incl - own;
    running += all;
  }
  __syncthreads();
  if (tid == 0) plan[0] = running;
  for (int e = warp; e < experts; e += kPlanThreads / 32) {
    const int t0 = first_tile[e];
    int n = 0;
    for (int base = 0; base < count; base += 32) {
      const bool hit = base + lane < count && ids[base + lane] == e;
      const unsigned mask = __ballot_sync(kFullWarp, hit);
      if (hit) {
        const int at = n + __popc(mask & ((1u << lane) - 1u)), t = t0 + at / kGroupRows, j = at % kGroupRows;
        plan[4 + 2 * cap + t * kGroupRows + j] = base + lane;
        slot_of[base + lane] = t * kGroupRows + j;
      }
      n += __popc(mask);
    }
    for (int t = lane; t < (n + kGroupRows - 1) / kGroupRows; t += 32) {
      plan[4 + t0 + t] = e;
      plan[4 + cap + t0 + t] = min(kGroupRows, n - t * kGroupRows);
    }
  }
}

// Activation transform of the grouped GEMM: one thread block per (token, slot) pair, two fp16 planes (the float32 activations of the
// routed GEMV must not lose precision here), B operand tiles per plan tile as in rht_f16_kernel.  The row stays in registers
// between the range scan and the transform.  SWIGLU: the row is [gate | up] of 2n bf16 values and the linear sees silu(gate) * up
// with the roundings of the unfused operators.  Columns of B without a pair are left as they are: they reach only accumulator
// columns that nobody reads.
constexpr int kGroupRhtWarps = 16, kGroupRhtBlocks = 8;      // n <= 16 * 8 * 128
template <bool SWIGLU>
__global__ void __launch_bounds__(kGroupRhtWarps * 32) rht_group_kernel(const void* __restrict__ x, int dtype, int x_div, long long x_stride, int n,
                                                                        const int* __restrict__ plan, int cap, const uint8_t* const* su_table,
                                                                        __half* __restrict__ xb, float* __restrict__ xsum, float* __restrict__ tok) {
  __shared__ float red[kGroupRhtWarps];
  // in this order: the GEMM behind this kernel starts when every thread block has come here, and then the plan, which an earlier kernel
  // wrote, is complete, so that it can look up its experts and fetch their words while this kernel still works
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int pair = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, blocks = n >> 7;
  const int slot = __ldcg(plan + group_plan_ints(cap) + pair);
  if (slot < 0) return;                                      // no expert here (the whole thread block): nobody may have written the row
  const size_t row = (size_t)(pair / x_div) * x_stride;
  float v[kGroupRhtBlocks][4];
  float mx = 0.f;
#pragma unroll
  for (int i = 0; i < kGroupRhtBlocks; ++i) {
    const int hb = warp + kGroupRhtWarps * i, col = hb * 128 + 4 * lane;
    if (hb >= blocks) break;
    float4 q = load_quad(x, row + col, dtype);
    if constexpr (SWIGLU) {
      const float4 u = load_quad(x, row + n + col, dtype);
      const auto rnd = [](float f) { return __bfloat162float(__float2bfloat16_rn(f)); };
      q = make_float4(rnd(rnd(q.x / (1.f + __expf(-q.x))) * u.x), rnd(rnd(q.y / (1.f + __expf(-q.y))) * u.y), rnd(rnd(q.z / (1.f + __expf(-q.z))) * u.z),
                      rnd(rnd(q.w / (1.f + __expf(-q.w))) * u.w));
    }
    v[i][0] = q.x; v[i][1] = q.y; v[i][2] = q.z; v[i][3] = q.w;
    mx = fmaxf(mx, fmaxf(fmaxf(fabsf(q.x), fabsf(q.y)), fmaxf(fabsf(q.z), fabsf(q.w))));
  }
  // the signs come from the end of a chain, slot -> expert -> signs, beside the row's loads: they are needed behind the barrier only
  const int t = slot / kGroupRows, r = slot % kGroupRows;
  const uint8_t* su = su_table[group_expert(plan, cap, t)];
  unsigned sg[kGroupRhtBlocks];
#pragma unroll
  for (int i = 0; i < kGroupRhtBlocks; ++i) {
    const int hb = warp + kGroupRhtWarps * i;
    sg[i] = hb < blocks ? sign_nibble(su, hb * 32 + lane) : 0u;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(kFullWarp, mx, o));
  if (lane == 0) red[warp] = mx;
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kGroupRhtWarps; ++k) mx = fmaxf(mx, red[k]);
  const float scale = range_scale(mx);
  if (tid == 0) tok[slot] = scale;
  const float inv = kInvSqrt128 / scale;
  const int c = (lane & 15) >> 2, j = lane & 3;
  constexpr size_t unit_halves = 2 * kGroupRows * 64;
  __half* out = xb + (size_t)t * (2 * blocks) * unit_halves + (size_t)(2 * j + (c >> 1)) * 64 + 4 * (c & 1);
  const size_t col_hi = (size_t)(r >> 3) * 512 + (r & 7) * 8, col_lo = col_hi + (kGroupRows >> 3) * 512;
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < kGroupRhtBlocks; ++i) {
    const int hb = warp + kGroupRhtWarps * i;
    if (hb >= blocks) break;                                 // warp-uniform
#pragma unroll
    for (int k = 0; k < 4; ++k) v[i][k] = flip(v[i][k], (sg[i] >> k) & 1u);
    wht128(v[i], lane);
    __half hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float f = v[i][k] * inv;
      hi[k] = __float2half_rn(f);
      lo[k] = __float2half_rn(f - __half2float(hi[k]));
      sum += __half2float(hi[k]) + __half2float(lo[k]);      // exactly what the MMA will see
    }
    __half* at = out + (size_t)(2 * hb + (lane >> 4)) * unit_halves;
    *reinterpret_cast<uint2*>(at + col_hi) = *reinterpret_cast<const uint2*>(hi);
    *reinterpret_cast<uint2*>(at + col_lo) = *reinterpret_cast<const uint2*>(lo);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(kFullWarp, sum, o);
  __syncthreads();
  if (lane == 0) red[warp] = sum;
  __syncthreads();
  if (tid == 0) {
    float s = 0.f;
    for (int k = 0; k < kGroupRhtWarps; ++k) s += red[k];
    xsum[slot] = s;
  }
}

template <typename... P, typename... A>
int launch_chained(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // resident early, waits before its first read
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, args...);
}

// blocks that a lane of the transform adds up one after another, and the sums that it leaves of a row
int gemm_rht_per(int np, int n) { return min(max(np / 48, 1), (n + 1023) / 1024); }
int gemm_xsums(int np, int n) { return (n / 128 + 8 * gemm_rht_per(np, n) - 1) / (8 * gemm_rht_per(np, n)); }

// Form, slices of a row and warps of the transform's thread blocks before a GEMM of `grid` thread blocks.  Below 2560 columns one block per
// warp is better (figures above), but for more than 128 rows of 2048 columns and more (2048x2048 K4, 200 rows: 14.8 / 14.0 us in a chain; at 2560
// columns, 48 rows, 10.1 / 9.5).  The rest is about the SMs that a GEMM in clusters leaves free, `idle`, taken from the GEMM that comes: in a
// chain of layers the one before is most often like it, and behind another kernel the transform finds the GPU empty and the numbers matter
// little.  An SM holds one thread block of 24 warps, two of 16 or four of 8 at 64 registers a thread.
//  * Two turns of the scan, whatever the slices: 8 warps up to 4096 columns (more rows than 64 take 16: 4096x4096 K4, 96 rows 14.8 / 13.9), 16 up
//    to 8192, 24 beyond (512x13568 K3, 2 rows, 8 / 24: 8.4 / 7.8).  More than 128 rows fill the SMs with 16 (4096x12288 K5, 200 rows, 24 / 16:
//    36.7 / 34.2).
//  * Two slices where all fit (4096x12288 K5, 8 rows, 1 / 2: 18.6 / 17.2), four for long rows if they do (1024x16256 K4, 2 rows, 2 / 4: 11.2 / 10.4),
//    and two where one would not fit either (4096x12288 37 rows 22.3 / 21.5; 4096x8192 K3, 48 rows 17.6 / 16.6); between the two one slice, all
//    of them at once (4096x8192 K3, 24 rows 14.4 / 15.7).
//  * Where the GEMM before leaves no SM free, the transform comes when all of them are: larger thread blocks (12288x4096 K2, 11 rows, 8 / 24 warps:
//    19.9 / 18.5), and more for few rows (2 rows, one slice of 8 / four: 18.4 / 18.1; 7168x15104 K8, 13 float32 rows, two / four of 24: 36.5 /
//    35.2) and long ones (18560x13696 K3, 16 rows, one / two: 64.3 / 62.4).
struct RhtShape {
  bool quad;                                                 // four blocks per warp
  int slices, warps;
  RhtShape(int rows, int np, int n, int grid, int sms) {
    const int groups = (n + 511) / 512, idle = sms - grid;
    const bool full = idle < 4, all_fit = !full && 2 * rows <= idle;
    quad = n >= 2560 || (n >= 2048 && rows > 128);
    slices = gemm_xsums(np, n);
    warps = 8;
    if (!quad) return;
    const bool four = full ? rows <= (groups > 16 ? 16 : 4) : groups > 16 && 4 * rows < idle;
    if (full && four && groups <= 16) warps = 8;
    else if (rows > 128) warps = 16;
    else if (full || groups > 16) warps = 24;
    else warps = groups <= 8 && rows <= 64 ? 8 : 16;
    if (four) slices = 4;
    else if (full) slices = groups > 16 && rows <= 64 ? 2 : 1;
    else if (warps == 24) slices = all_fit || (rows > idle && rows <= 64) ? 2 : 1;
    else slices = all_fit || (groups > 8 && rows > 2 * idle && rows <= 128) ? 2 : 1;
    const int least = (n + 128 * kRhtBlocks - 1) / (128 * kRhtBlocks);
    if (slices < least) slices = least;
  }
};

int run_rht_f16(const void* x, int dtype, int rows, int np, int n, int n_in, int planes, const RhtShape& shape, const uint8_t* su, __half* xb,
                float* xsum, float* tok, cudaStream_t st) {
  const dim3 grid(rows, shape.slices);
  const int threads = 32 * shape.warps, per = gemm_rht_per(np, n);
  const auto launch = [&](auto type) {
    constexpr int DT = decltype(type)::value;
    return launch_chained(shape.quad ? rht_f16_kernel<DT> : rht_f16_short_kernel<DT>, grid, threads, 0, st, x, np, n, n_in, planes, su, xb, xsum, tok, per);
  };
  switch (dtype) {
    case HTR_DTYPE_BF16: return launch(std::integral_constant<int, HTR_DTYPE_BF16>{});
    case HTR_DTYPE_F16: return launch(std::integral_constant<int, HTR_DTYPE_F16>{});
    default: return launch(std::integral_constant<int, HTR_DTYPE_F32>{});
  }
}

namespace {

thread_local int t_gemm_cuda = 0;
thread_local int t_gemm_withhold = 0;                      // (htr_gemm_withhold_tile)
constexpr size_t kCounterRegion = 1 << 16;   // same fixed counter region as the GEMV workspace
constexpr size_t kErrorRegion = 256;

struct GemmPlan {
  int np, rbs, hb, split, grid, stages, smem, sms, inbox;
  size_t off_xb, off_xsum, off_tok, off_part, total;
};

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

bool width_ok(int K) { return K == 2 || K == 3 || K == 4 || K == 5 || K == 6 || K == 8; }

double codebook_scale() {
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

int gemm_clusters(int K, int smem, int split) {
  switch (K) {
    case 2: return packed_gemm_tc_clusters<2>(smem, split);
    case 3: return packed_gemm_tc_clusters<3>(smem, split);
    case 4: return packed_gemm_tc_clusters<4>(smem, split);
    case 5: return packed_gemm_tc_clusters<5>(smem, split);
    case 6: return packed_gemm_tc_clusters<6>(smem, split);
    case 8: return packed_gemm_tc_clusters<8>(smem, split);
  }
  return 0;
}

int launch_gemm(int K, const GemmParams& p, int grid, int smem, cudaStream_t st) {
  switch (K) {
    case 2: return launch_packed_gemm_tc<2>(p, grid, smem, st);
    case 3: return launch_packed_gemm_tc<3>(p, grid, smem, st);
    case 4: return launch_packed_gemm_tc<4>(p, grid, smem, st);
    case 5: return launch_packed_gemm_tc<5>(p, grid, smem, st);
    case 6: return launch_packed_gemm_tc<6>(p, grid, smem, st);
    case 8: return launch_packed_gemm_tc<8>(p, grid, smem, st);
  }
  return (int)cudaErrorInvalidValue;
}

// activation rows per launch after padding: accumulator columns come in multiples of 16
int padded_rows(int M, int planes) { return planes == 2 ? (M + 7) / 8 * 8 : (M + 15) / 16 * 16; }

int device_sms() {                                        // 0: a CUDA error
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  static int seen_sms[64] = {0};                          // a device fact: asked once (every caller would store the same number)
  if (dev >= 0 && dev < 64) sms = seen_sms[dev];
  if (sms <= 0) {
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 0;
    if (dev >= 0 && dev < 64) seen_sms[dev] = sms;
  }
  return sms;
}

// Stages of a launch, as many as tensor memory and `budget` bytes of shared memory hold, and the shared memory of its two rings; 0: fewer than two
int gemm_stages(int np, int planes, int K, int budget, int* smem) {
  int stages = (kGemmTmemCols - gemm_acc_cols(np * planes)) / 64;
  if (stages > kGemmMaxStages) stages = kGemmMaxStages;
  while (stages > 1 && gemm_smem_bytes(np, planes, stages, gemm_word_bytes(K)) > budget) --stages;
  *smem = gemm_smem_bytes(np, planes, stages, gemm_word_bytes(K));
  return stages < 2 || *smem > budget ? 0 : stages;
}

int make_gemm_plan(int M, int m, int n, int K, int planes, GemmPlan* out) {
  GemmPlan g;
  g.sms = device_sms();
  if (g.sms <= 0) return HTR_ERR_CUDA;
  g.np = padded_rows(M, planes);
  g.rbs = m / 128;
  g.hb = n / 128;
  const int ncols = g.np * planes;
  if (ncols > kGemmMaxCols) return HTR_ERR_TOO_LARGE;
  // one thread block per SM
  const int words = gemm_word_bytes(K), budget = kGemmSmem;
  g.stages = gemm_stages(g.np, planes, K, budget, &g.smem);
  if (g.stages == 0) return HTR_ERR_TOO_LARGE;
  // Three forms, by their cost in units of one decoded 128 x 128 block (0.43 us, or as long as the MMAs of a wide batch take):
  //  * up to sixteen thread blocks share a row block as a cluster and reduce on chip;
  //  * a thread block takes a whole row block, in as many waves as there are row blocks per SM: its decode warps finish it from shared
  //    memory, about four blocks' time and a thirtieth of one per activation row;
  //  * every thread block of the GPU takes an even run (flat) and a row block's partial sums meet in global memory at one last arriver:
  //    nine blocks' time for the hand-over (measured 2 to 3 us) and the partials, which that one reads row by row.  Row blocks inside a
  //    run are finished by four warps beside the decode, half a block's time per activation row: many rows wait for them.
  // us, flat / whole row blocks: 28672x1024, 64 rows 31.6 / 18.8; 151936x4096, 32 rows 146 / 171; 12288x4096, 64 rows 23.7 / 25.0, 160 rows
  // 34.3 / 32.3, 200 rows 39.8 / 33.8, 256 rows 48.8 / 44.7; flat / clusters: 2048x2048, 8 / 200 rows 11.8 / 6.7, 35.1 / 14.6.
  // (Beyond 128 rows a partial is read at less than half the rate: 12288x4096, 128 rows 29.7 / 29.9, 160 rows 34.3 / 32.3.)
  // The tensor cores cut each sum off towards zero, so the error of a result grows with the blocks that one accumulator takes: 2048x4096,
  // float32, 2 / 8 / 32 blocks 3.5e-6 / 1.1e-5 / 4.1e-5 (2-norm, normal activations), five times that where the activations have a mean.
  // A change of these terms that gives float32 rows longer sums loses precision; beyond 128 rows there is one plane, whose own rounding
  // (2e-4) hides it.
  const double unit = ncols > 192 ? 1.2 : 1.0;
  const long long slots = g.sms, units = (long long)g.rbs * g.hb;
  const long long flat_grid = slots < units ? slots : units, flat_run = (units + flat_grid - 1) / flat_grid;
  const double beside = (double)(flat_run / g.hb) * M * 0.5;
  double best = (flat_run * unit > beside ? flat_run * unit : beside) + 9 + (double)((g.hb / flat_run + 1) * g.np) / (g.np > 128 ? 32 : 84);
  g.split = 0;
  for (int s = (int)(slots / g.rbs < 16 ? slots / g.rbs : 16); s >= 2; --s) {
    const double cost = (double)((g.hb + s - 1) / s) * unit;
    if (s <= g.hb && cost < best && gemm_clusters(K, g.smem, s) >= g.rbs) {
      g.split = s;
      best = cost;
    }
  }
  const long long waves = (g.rbs + slots - 1) / slots;
  if (waves * (g.hb * unit + M / 30.0) + (waves - 1) * 4 < best) g.split = 1;
  g.grid = g.split > 0 ? g.rbs * g.split : (int)flat_grid;
  // A cluster's partials are sent to the thread blocks that finish their rows where an inbox of np x 512 bytes fits beside the rings, with
  // fewer stages of B if need be (a run needs no more than it has blocks).  us, fetched from where they were made / sent: 4096x12288 K3 4
  // rows 17.1 / 16.6, 4096x4096 K4 32 rows 9.5 / 8.8, 2048x2048 K4 64 rows 8.3 / 7.4, 640x1024 K4 64 rows 7.4 / 6.6; but 768x384 K2 137 rows
  // 8.6 / 9.4: a number sent is an instruction of its own, and at many rows they outweigh the barriers.
  g.inbox = 0;
  if (g.split > 1 && g.np <= 64) {
    const int inbox_bytes = g.split * ((g.np + g.split - 1) / g.split) * 512, run = (g.hb + g.split - 1) / g.split, least = run < 2 ? 2 : run < 4 ? run : 4;
    int stages = g.stages;
    while (stages > least && gemm_smem_bytes(g.np, planes, stages, words) + inbox_bytes > budget) --stages;
    const int smem = gemm_smem_bytes(g.np, planes, stages, words);
    if (smem + inbox_bytes <= budget) {
      g.stages = stages;
      g.inbox = smem - 128;                                  // (behind the words; the last 128 bytes are for the alignment of the first)
      g.smem = smem + inbox_bytes;
    }
  }
  size_t off = kCounterRegion + kErrorRegion;
  g.off_xb = off; off += align256((size_t)ncols * n * 2);
  g.off_xsum = off; off += align256((size_t)g.np * gemm_xsums(g.np, n) * 4);
  g.off_tok = off; off += align256((size_t)g.np * 4);
  g.off_part = off;
  if (g.split == 0) off += align256((size_t)g.grid * 2 * g.np * 128 * 4);
  g.total = off;
  *out = g;
  return HTR_OK;
}

}  // namespace
}  // namespace htr

using namespace htr;

extern "C" {

static size_t plan_bytes(int M, int m, int n, int K, int planes) {
  GemmPlan g;
  return make_gemm_plan(M, m, n, K, planes, &g) == HTR_OK ? g.total : 0;
}

size_t htr_linear_gemm_workspace_bytes(int M, int m, int n, int K) {
  if (!width_ok(K) || M < 1 || M > HTR_GEMM_MAX_ROWS || m <= 0 || n <= 0 || m % 128 || n % 128) return 0;
  // the scratch of either activation form (one or two fp16 planes) must fit
  const size_t b1 = plan_bytes(M, m, n, K, 1), b2 = plan_bytes(M > HTR_GEMM_MAX_ROWS_F32 ? HTR_GEMM_MAX_ROWS_F32 : M, m, n, K, 2);
  if (!b1 || !b2) return 0;
  return b1 > b2 ? b1 : b2;
}

// fp16 planes of the activations: two (hi + lo, 22 bits) for float32 inputs, for callers that ask, and for up to 8 rows, which fill the
// 16 accumulator columns of the smallest MMA either way; else one
static int gemm_planes(int dtype, int M, bool fine) { return dtype == HTR_DTYPE_F32 || fine || M <= 8 ? 2 : 1; }

static int gemm_launch(const void* x, int dtype, int M, int n_in, const void* qweight, int mt, int nt, int K, const void* scales, const uint8_t* su,
                       const uint8_t* sv, const void* bias, void* y, int m_out, bool fine, void* const* peer_y, int npeer, int64_t peer_offset,
                       void* workspace, size_t workspace_bytes, htr_stream_t stream);

int htr_linear_gemm(const void* x, int dtype, int M, const void* qweight, int mt, int nt, int K, const void* scales, const uint8_t* su,
                    const uint8_t* sv, const void* bias, void* y, void* workspace, size_t workspace_bytes, htr_stream_t stream) {
  return gemm_launch(x, dtype, M, nt * 16, qweight, mt, nt, K, scales, su, sv, bias, y, mt * 16, false, nullptr, 0, 0, workspace, workspace_bytes, stream);
}

int htr_linear_gemm_padded(const void* x, int dtype, int M, int n_in, const void* qweight, int mt, int nt, int K, const void* scales, const uint8_t* su,
                           const uint8_t* sv, const void* bias, void* y, int m_out, void* workspace, size_t workspace_bytes, htr_stream_t stream) {
  if (mt <= 0 || nt <= 0 || M > HTR_GEMM_MAX_ROWS_F32) return HTR_ERR_BAD_SHAPE;
  if (n_in < 8 || n_in > nt * 16 || n_in % 8 || m_out < 8 || m_out > mt * 16 || m_out % 8) return HTR_ERR_BAD_SHAPE;
  return gemm_launch(x, dtype, M, n_in, qweight, mt, nt, K, scales, su, sv, bias, y, m_out, true, nullptr, 0, 0, workspace, workspace_bytes, stream);
}

int htr_linear_gemm_peers(const void* x, int dtype, int M, const void* qweight, int mt, int nt, int K, const void* scales, const uint8_t* su,
                          const uint8_t* sv, const void* bias, void* const* peer_y, int npeer, int64_t peer_offset, void* workspace,
                          size_t workspace_bytes, htr_stream_t stream) {
  if (npeer < 1 || npeer > 8 || !peer_y || peer_offset < 0 || (peer_offset & 7)) return HTR_ERR_BAD_SHAPE;
  for (int i = 0; i < npeer; ++i)
    if (!peer_y[i] || (reinterpret_cast<uintptr_t>(peer_y[i]) & 15u)) return peer_y[i] ? HTR_ERR_ALIGNMENT : HTR_ERR_NULL;
  return gemm_launch(x, dtype, M, nt * 16, qweight, mt, nt, K, scales, su, sv, bias, nullptr, mt * 16, false, peer_y, npeer, peer_offset, workspace,
                     workspace_bytes, stream);
}

static int gemm_launch(const void* x, int dtype, int M, int n_in, const void* qweight, int mt, int nt, int K, const void* scales, const uint8_t* su,
                       const uint8_t* sv, const void* bias, void* y, int m_out, bool fine, void* const* peer_y, int npeer, int64_t peer_offset,
                       void* workspace, size_t workspace_bytes, htr_stream_t stream) {
  if (!width_ok(K)) return HTR_ERR_BAD_K;
  if (dtype < HTR_DTYPE_BF16 || dtype > HTR_DTYPE_F32) return HTR_ERR_BAD_DTYPE;
  if (M < 0 || M > HTR_GEMM_MAX_ROWS || mt <= 0 || nt <= 0 || mt % 8 || nt % 8) return HTR_ERR_BAD_SHAPE;
  if (mt / 8 > (int)(kCounterRegion / 4)) return HTR_ERR_TOO_LARGE;
  if (M == 0) return HTR_OK;
  if (!x || !qweight || !scales || !su || !sv || (!y && npeer == 0)) return HTR_ERR_NULL;
  const auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(x) || !a16(qweight) || !a16(y) || (bias && !a16(bias)) || !a16(workspace) || !a16(scales)) return HTR_ERR_ALIGNMENT;
  const int m = mt * 16, n = nt * 16;
  GemmPlan g;
  const int planes = gemm_planes(dtype, M, fine);
  if (planes == 2 && M > HTR_GEMM_MAX_ROWS_F32) return HTR_ERR_BAD_SHAPE;
  const int rc = make_gemm_plan(M, m, n, K, planes, &g);
  if (rc != HTR_OK) return rc;
  if (!workspace || workspace_bytes < g.total) return HTR_ERR_WORKSPACE;
  char* ws = static_cast<char*>(workspace);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  GemmParams p;
  p.qw = static_cast<const uint32_t*>(qweight);
  p.scales = static_cast<const __half*>(scales);
  p.sv = sv;
  p.bias = bias;
  p.y = y;
  p.xb = reinterpret_cast<const __half*>(ws + g.off_xb);
  p.xsum = reinterpret_cast<const float*>(ws + g.off_xsum);
  p.tok = reinterpret_cast<const float*>(ws + g.off_tok);
  p.part = reinterpret_cast<float*>(ws + g.off_part);
  p.counters = reinterpret_cast<int*>(ws);
  p.error = reinterpret_cast<int*>(ws + kCounterRegion);
  p.rows = M;
  p.np = g.np;
  p.planes = planes;
  p.mt = mt;
  p.nt = nt;
  p.dtype = dtype;
  p.hb = g.hb;
  p.split = g.split;
  p.run_q = g.split > 0 ? g.hb / g.split : g.rbs * g.hb / g.grid;
  p.run_rem = g.split > 0 ? g.hb % g.split : g.rbs * g.hb % g.grid;
  p.part_magic = g.split > 0 ? part_reciprocal(g.split) : 0;
  p.inbox = g.inbox;
  p.stages = g.stages;
  p.withhold = t_gemm_withhold;
  p.m_out = m_out;
  const RhtShape shape(M, g.np, n, g.grid, g.sms);
  p.xsum_slices = gemm_xsums(g.np, n);
  p.cb = (float)codebook_scale();
  p.plan = nullptr;
  p.npeer = npeer;
  p.peer_offset = peer_offset;
  for (int i = 0; i < 8; ++i) p.peer_y[i] = i < npeer ? peer_y[i] : nullptr;
  int e = run_rht_f16(x, dtype, M, g.np, n, n_in, planes, shape, su, reinterpret_cast<__half*>(ws + g.off_xb), reinterpret_cast<float*>(ws + g.off_xsum),
                      reinterpret_cast<float*>(ws + g.off_tok), st);
  if (e) { t_gemm_cuda = e; return HTR_ERR_CUDA; }
  e = launch_gemm(K, p, g.grid, g.smem, st);
  if (e) t_gemm_cuda = e;
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_linear_gemm_shape(int dtype, int M, int m, int n, int K, int* shape) {
  if (!width_ok(K)) return HTR_ERR_BAD_K;
  if (dtype < HTR_DTYPE_BF16 || dtype > HTR_DTYPE_F32) return HTR_ERR_BAD_DTYPE;
  const int planes = gemm_planes(dtype, M, false);
  if (M < 1 || M > (planes == 2 ? HTR_GEMM_MAX_ROWS_F32 : HTR_GEMM_MAX_ROWS) || m <= 0 || n <= 0 || m % 128 || n % 128) return HTR_ERR_BAD_SHAPE;
  if (!shape) return HTR_ERR_NULL;
  GemmPlan g;
  const int rc = make_gemm_plan(M, m, n, K, planes, &g);
  if (rc != HTR_OK) return rc;
  const RhtShape r(M, g.np, n, g.grid, g.sms);
  const int all[5] = {g.split, g.grid, r.quad ? 1 : 0, r.slices, r.warps};
  for (int i = 0; i < 5; ++i) shape[i] = all[i];
  return HTR_OK;
}

// ---- grouped form: the experts of a mixture-of-experts step
static int group_cap(int count, int table_rows) {
  const int most = table_rows + count / kGroupRows;          // every expert may end in a part tile
  return count < most ? count : most;
}

struct GroupLayout {
  int cap, stages, smem, grid;
  size_t off_xb, off_xsum, off_tok, off_part, total;
};

static int group_layout(int count, int table_rows, int m, int n, int K, GroupLayout* g) {
  if (count < 1 || count > 4096 || table_rows < 1 || table_rows + count > 12288 || n > kGroupRhtWarps * kGroupRhtBlocks * 128) return HTR_ERR_TOO_LARGE;
  g->cap = group_cap(count, table_rows);
  if (g->cap > kGroupMaxTiles || (long long)g->cap * (m / 128) > (int)(kCounterRegion / 4) || (long long)g->cap * (m / 128) * (n / 128) > 0x3FFFFFFF)
    return HTR_ERR_TOO_LARGE;
  g->stages = gemm_stages(kGroupRows, 2, K, kGemmGroupSmem, &g->smem);
  if (g->stages == 0) return HTR_ERR_TOO_LARGE;
  g->grid = device_sms();
  if (g->grid <= 0) return HTR_ERR_CUDA;
  size_t off = kCounterRegion + kErrorRegion;
  g->off_xb = off; off += align256((size_t)g->cap * n * (2 * kGroupRows) * 2);
  g->off_xsum = off; off += align256((size_t)g->cap * kGroupRows * 4);
  g->off_tok = off; off += align256((size_t)g->cap * kGroupRows * 4);
  g->off_part = off; off += align256((size_t)g->grid * 2 * kGroupRows * 128 * 4);
  g->total = off;
  return HTR_OK;
}

size_t htr_route_plan_bytes(int count, int table_rows) {
  if (count < 1 || count > 4096 || table_rows < 1 || table_rows + count > 12288) return 0;
  return align256(((size_t)group_plan_ints(group_cap(count, table_rows)) + count) * sizeof(int));
}

int htr_route_plan(const int64_t* route, int count, int table_rows, const void* const* qweight_table, void* plan, size_t plan_bytes,
                   htr_stream_t stream) {
  const size_t need = htr_route_plan_bytes(count, table_rows);
  if (need == 0) return HTR_ERR_TOO_LARGE;
  if (!route || !qweight_table || !plan) return HTR_ERR_NULL;
  if (plan_bytes < need) return HTR_ERR_WORKSPACE;
  const int e = launch_chained(route_plan_kernel, dim3(1), kPlanThreads, (size_t)(table_rows + count) * sizeof(int), static_cast<cudaStream_t>(stream),
                               reinterpret_cast<const long long*>(route), count, table_rows, reinterpret_cast<const uint32_t* const*>(qweight_table),
                               static_cast<int*>(plan), group_cap(count, table_rows));
  if (e) { t_gemm_cuda = e; return HTR_ERR_CUDA; }
  return HTR_OK;
}

size_t htr_linear_routed_gemm_workspace_bytes(int count, int table_rows, int m, int n, int K) {
  if (!width_ok(K) || m <= 0 || n <= 0 || m % 128 || n % 128) return 0;
  GroupLayout g;
  return group_layout(count, table_rows, m, n, K, &g) == HTR_OK ? g.total : 0;
}

int htr_linear_routed_gemm(const void* x, int dtype, int x_div, int64_t x_row_stride, const void* plan, int count, int table_rows,
                           const void* const* qweight_table, const void* const* scales_table, const uint8_t* const* su_table,
                           const uint8_t* const* sv_table, int mt, int nt, int K, void* y, int prologue, void* workspace, size_t workspace_bytes,
                           htr_stream_t stream) {
  if (!width_ok(K)) return HTR_ERR_BAD_K;
  if (dtype < HTR_DTYPE_BF16 || dtype > HTR_DTYPE_F32) return HTR_ERR_BAD_DTYPE;
  if (prologue == HTR_PROLOGUE_SWIGLU && dtype != HTR_DTYPE_BF16) return HTR_ERR_BAD_DTYPE;
  if (x_div < 1 || x_row_stride < 0 || x_row_stride % 4 || mt <= 0 || nt <= 0 || mt % 8 || nt % 8 || (prologue != HTR_PROLOGUE_NONE && prologue != HTR_PROLOGUE_SWIGLU))
    return HTR_ERR_BAD_SHAPE;
  if (!x || !y || !plan || !qweight_table || !scales_table || !su_table || !sv_table) return HTR_ERR_NULL;
  const auto a16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; };
  if (!a16(x) || !a16(y) || !a16(workspace) || !a16(plan)) return HTR_ERR_ALIGNMENT;
  const int m = mt * 16, n = nt * 16;
  GroupLayout g;
  const int rc = group_layout(count, table_rows, m, n, K, &g);
  if (rc != HTR_OK) return rc;
  if (!workspace || workspace_bytes < g.total) return HTR_ERR_WORKSPACE;
  char* ws = static_cast<char*>(workspace);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  __half* xb = reinterpret_cast<__half*>(ws + g.off_xb);
  float *xsum = reinterpret_cast<float*>(ws + g.off_xsum), *tok = reinterpret_cast<float*>(ws + g.off_tok);
  const int* pl = static_cast<const int*>(plan);
  int e = prologue == HTR_PROLOGUE_SWIGLU
              ? launch_chained(rht_group_kernel<true>, dim3(count), kGroupRhtWarps * 32, 0, st, x, dtype, x_div, (long long)x_row_stride, n, pl, g.cap, su_table, xb, xsum, tok)
              : launch_chained(rht_group_kernel<false>, dim3(count), kGroupRhtWarps * 32, 0, st, x, dtype, x_div, (long long)x_row_stride, n, pl, g.cap, su_table, xb, xsum, tok);
  if (e) { t_gemm_cuda = e; return HTR_ERR_CUDA; }
  GemmParams p = {};
  p.y = y;
  p.xb = xb;
  p.xsum = xsum;
  p.tok = tok;
  p.part = reinterpret_cast<float*>(ws + g.off_part);
  p.counters = reinterpret_cast<int*>(ws);
  p.error = reinterpret_cast<int*>(ws + kCounterRegion);
  p.rows = p.np = kGroupRows;
  p.planes = 2;
  p.mt = mt;
  p.nt = nt;
  p.m_out = m;
  p.dtype = dtype;
  p.hb = n / 128;
  p.stages = g.stages;
  p.withhold = t_gemm_withhold;
  p.xsum_slices = 1;
  p.cb = (float)codebook_scale();
  p.plan = pl;
  p.tile_cap = g.cap;
  p.rb_per_tile = m / 128;
  p.g_qw = reinterpret_cast<const uint32_t* const*>(qweight_table);
  p.g_scales = reinterpret_cast<const __half* const*>(scales_table);
  p.g_sv = sv_table;
  e = launch_gemm(K, p, g.grid, g.smem, st);
  if (e) t_gemm_cuda = e;
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_linear_gemm_last_cuda_error(void) { return t_gemm_cuda; }

size_t htr_linear_gemm_error_offset(void) { return kCounterRegion; }

void htr_gemm_withhold_tile(int block) { t_gemm_withhold = block < 0 ? 0 : block + 1; }

}  // extern "C"
