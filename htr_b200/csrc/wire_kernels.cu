// Hooks around the wire format: raw integer decode, the stand-alone activation transform and the
// original-basis weight materialisation.  None of them is on the decode hot path (the packed GEMV fuses
// what it needs); they exist so that each stage can be compared with the CPU decoder on its own.
#include "htr_codec.cuh"
#include "htr_common.cuh"

namespace htr {

// ------------------------------------------------------------------------------------------------
// int16 v(s_t) for every step of every tile, [ntiles, 256] in stream order.  One thread = one row pair.
template <int K>
__global__ void __launch_bounds__(256) decode_raw_kernel(const uint32_t* __restrict__ qw, int16_t* __restrict__ out, long long ntiles) {
  const long long unit = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (unit >= ntiles * 8) return;
  const long long tile = unit >> 3;
  const int q = (int)(unit & 7);
  const uint32_t* words = qw + tile * (8 * K);
  uint32_t V[K + 1];
  V[0] = words[history_word<K>(q)];
#pragma unroll
  for (int k = 0; k < K; ++k) V[k + 1] = words[q * K + k];
  uint32_t s[32];
  unit_states<K>(V, s);
  uint4* dst = reinterpret_cast<uint4*>(out + tile * 256 + q * 32);
#pragma unroll
  for (int v4 = 0; v4 < 4; ++v4) {
    uint32_t packed[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const uint32_t lo = (uint32_t)code_value(s[v4 * 8 + 2 * e]) & 0xFFFFu, hi = (uint32_t)code_value(s[v4 * 8 + 2 * e + 1]) & 0xFFFFu;
      packed[e] = lo | (hi << 16);
    }
    dst[v4] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  }
}

// ------------------------------------------------------------------------------------------------
// xt[r, 128b + :] = H128/sqrt(128) (su * x[r, 128b + :]).  One warp per (row, 128-column block).
__global__ void __launch_bounds__(256) rht_kernel(const void* __restrict__ x, int dtype, int M, int n, const uint8_t* __restrict__ su,
                                                  float* __restrict__ xt) {
  const int lane = threadIdx.x & 31;
  const long long item = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int blocks = n >> 7;
  if (item >= (long long)M * blocks) return;
  const int r = (int)(item / blocks), hb = (int)(item % blocks);
  const size_t at = (size_t)r * n + hb * 128 + 4 * lane;
  const float4 xv = load_quad(x, at, dtype);
  const unsigned sg = sign_nibble(su, hb * 32 + lane);
  float v[4] = {flip(xv.x, sg & 1u), flip(xv.y, (sg >> 1) & 1u), flip(xv.z, (sg >> 2) & 1u), flip(xv.w, sg >> 3)};
  wht128(v, lane);
  *reinterpret_cast<float4*>(xt + at) = make_float4(v[0] * kInvSqrt128, v[1] * kInvSqrt128, v[2] * kInvSqrt128, v[3] * kInvSqrt128);
}

// ------------------------------------------------------------------------------------------------
// W block (128 x 128) = sv * Ho Q Hi * su, one thread block of 128 threads per block: 14 butterfly stages and the decode per weight.
// What bounds it: the 14 additions (the FMA pipes take 124 of them per cycle and SM: 20 us at 4096 x 12288), then the decode
// (6 us); 100 MB of bf16 output take 15 us.  So every stage runs in registers, two elements per instruction where they are
// independent, and the block crosses shared memory once:
//   phase 1  thread = a row pair (q) of one strip x 64 columns (four tiles): 128 values, seven index bits in registers -- four
//            column bits and two tile bits as packed pairs (row 2q, row 2q+1), then the row bit;
//   phase 2  thread = columns c, c + 64 of the 64 rows of one parity: the six row bits as packed pairs (c, c + 64), then the last
//            column bit, signs, cast, store.
// The exchange buffer swaps 16-byte groups by row pair so that both sides are free of bank conflicts.  A register of the 16-bit results holds
// one column of two rows; the neighbour lane has the next column, and one shuffle and one byte permutation leave two adjacent columns of
// one row in each, for one store (with a register of two columns of one row, two selections more per pair of values and half a shuffle less).
// Measured, bf16: 4096 x 12288 K4 52.5 -> 48.1 us for that exchange, 28672 x 8192 K4 230 -> 208; one value per shuffle and shared-memory access
// with scalar stores took 108.  A quarter of the stalls are instruction fetches of the unrolled body, so that instructions count twice.
// Without gain: words of the next wave's blocks prefetched to L2, magic constants cancelled in the first butterfly (50 us).
constexpr int kDqThreads = 128;
constexpr int kDqSmem = 128 * 128 * 4;

__device__ __forceinline__ int dq_at(int row, int col) { return row * 128 + ((((col >> 2) ^ ((row >> 1) & 7)) << 2) | (col & 3)); }

// butterflies over index bit BIT of N packed pairs
template <int N, int BIT>
__device__ __forceinline__ void dq_stage(float2 (&v)[N]) {
  const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
  for (int i = 0; i < N; ++i)
    if (!(i & (1 << BIT))) {
      const float2 a = v[i], b = v[i | (1 << BIT)];
      v[i] = __fadd2_rn(a, b);
      v[i | (1 << BIT)] = __ffma2_rn(b, minus, a);           // a - b, exactly as rounded
    }
}

template <int K, int OUT>
__global__ void __launch_bounds__(kDqThreads, 3) dequant_w_kernel(const uint32_t* __restrict__ qw, const __half* __restrict__ scales,
                                                                  const uint8_t* __restrict__ su, const uint8_t* __restrict__ sv, float cb,
                                                                  void* __restrict__ W, int nt) {
  extern __shared__ __align__(16) float blk[];               // [128][128], groups of four columns swapped by row pair
  __shared__ __align__(16) uint32_t s_sign[OUT == HTR_DTYPE_F32 ? 128 : 64];   // sign masks: of a row, or of two rows of one parity in halves
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cbk = blockIdx.x, rb = blockIdx.y, n = nt * 16;
  if constexpr (OUT == HTR_DTYPE_F32) {
    s_sign[(tid & 1) * 64 + (tid >> 1)] = ((sv[rb * 16 + (tid >> 3)] >> (tid & 7)) & 1) << 31;
  } else if (tid < 64) {                                     // rows 4 i + parity, 4 i + parity + 2
    const unsigned b = sv[rb * 16 + ((tid & 31) >> 1)] >> (4 * (tid & 1) + (tid >> 5));
    s_sign[tid] = ((b & 1) << 15) | ((b & 4) << 29);
  }
  {
    const int q = lane & 7, half = (lane >> 3) & 1, strip = 2 * warp + (lane >> 4);
    const uint32_t* words = qw + ((size_t)(rb * 8 + strip) * nt + (size_t)(cbk * 8 + half * 4)) * (8 * K) + q * K;
    uint32_t own[4][K];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const uint32_t* w = words + t * (8 * K);
      if constexpr (K % 4 == 0) {
#pragma unroll
        for (int i = 0; i < K / 4; ++i) {
          const uint4 r = __ldg(reinterpret_cast<const uint4*>(w) + i);
          own[t][4 * i] = r.x; own[t][4 * i + 1] = r.y; own[t][4 * i + 2] = r.z; own[t][4 * i + 3] = r.w;
        }
      } else if constexpr (K % 2 == 0) {
#pragma unroll
        for (int i = 0; i < K / 2; ++i) {
          const uint2 r = __ldg(reinterpret_cast<const uint2*>(w) + i);
          own[t][2 * i] = r.x; own[t][2 * i + 1] = r.y;
        }
      } else {
#pragma unroll
        for (int i = 0; i < K; ++i) own[t][i] = __ldg(w + i);
      }
    }
    const int row = strip * 16 + 2 * q;
    const float2 sc = make_float2(__half2float(scales[rb * 128 + row]), __half2float(scales[rb * 128 + row + 1]));
    const float2 s2 = make_float2(sc.x * cb * (1.0f / 128.0f), sc.y * cb * (1.0f / 128.0f));
    const float2 unbias = make_float2(-kMagic, -kMagic);
    float2 v[64];                                            // [tile][column] of (row, row + 1)
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      uint32_t V[K + 1], s[32];
#pragma unroll
      for (int i = 0; i < K; ++i) V[i + 1] = own[t][i];
      V[0] = __shfl_sync(kFullWarp, own[t][K - 1], (lane & 24) | ((q - 1) & 7));   // last word of the row pair before
      unit_states<K>(V, s);
#pragma unroll
      for (int u = 0; u < 16; ++u)
        v[t * 16 + u] = __fmul2_rn(__fadd2_rn(make_float2(__uint_as_float(code_magic_bits_alu(s[u])), __uint_as_float(code_magic_bits(s[16 + u]))), unbias), s2);
    }
    dq_stage<64, 0>(v);
    dq_stage<64, 1>(v);
    dq_stage<64, 2>(v);
    dq_stage<64, 3>(v);
    dq_stage<64, 4>(v);
    dq_stage<64, 5>(v);
#pragma unroll
    for (int g = 0; g < 16; ++g) {
      const float2 *p = v + 4 * g;
      const int col = half * 64 + 4 * g;
      *reinterpret_cast<float4*>(blk + dq_at(row, col)) = make_float4(p[0].x + p[0].y, p[1].x + p[1].y, p[2].x + p[2].y, p[3].x + p[3].y);
      *reinterpret_cast<float4*>(blk + dq_at(row + 1, col)) = make_float4(p[0].x - p[0].y, p[1].x - p[1].y, p[2].x - p[2].y, p[3].x - p[3].y);
    }
  }
  __syncthreads();
  const int parity = warp >> 1, c = (warp & 1) * 32 + lane;
  float2 v[64];                                              // row 2i + parity, columns (c, c + 64)
#pragma unroll
  for (int i = 0; i < 64; ++i) v[i] = make_float2(blk[dq_at(2 * i + parity, c)], blk[dq_at(2 * i + parity, c + 64)]);
  dq_stage<64, 0>(v);
  dq_stage<64, 1>(v);
  dq_stage<64, 2>(v);
  dq_stage<64, 3>(v);
  dq_stage<64, 4>(v);
  dq_stage<64, 5>(v);
  const int gc = cbk * 128 + c;
  const uint32_t su0 = (su[gc >> 3] >> (gc & 7)) & 1u, su1 = (su[(gc + 64) >> 3] >> (gc & 7)) & 1u;
  const size_t row0 = (size_t)rb * 128 + parity;
  if constexpr (OUT == HTR_DTYPE_F32) {
    const uint32_t* masks = s_sign + parity * 64;
#pragma unroll
    for (int i = 0; i < 64; i += 4) {
      const uint4 m4 = *reinterpret_cast<const uint4*>(masks + i);
      const uint32_t m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 a = v[i + k];
        float* dst = static_cast<float*>(W) + (row0 + 2 * (i + k)) * n + gc;
        dst[0] = __uint_as_float(__float_as_uint(a.x + a.y) ^ (m[k] ^ (su0 << 31)));
        dst[64] = __uint_as_float(__float_as_uint(a.x - a.y) ^ (m[k] ^ (su1 << 31)));
      }
    }
  } else {
    // a register takes one column of two rows; the even lane stores the first row of its column and its neighbour's, the odd lane the second
    const uint32_t* masks = s_sign + parity * 32;
    const uint32_t flip0 = su0 * 0x80008000u, flip1 = su1 * 0x80008000u, pick = lane & 1 ? 0x3276u : 0x5410u;
    uint16_t* dst = static_cast<uint16_t*>(W) + (row0 + 2 * (lane & 1)) * n + (gc & ~1);
    const auto narrow = [](float lo, float hi) {
      if constexpr (OUT == HTR_DTYPE_BF16) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
      } else {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t*>(&h);
      }
    };
#pragma unroll
    for (int i = 0; i < 64; i += 8) {
      const uint4 m4 = *reinterpret_cast<const uint4*>(masks + i / 2);
      const uint32_t m[4] = {m4.x, m4.y, m4.z, m4.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 a = v[i + 2 * k], b = v[i + 2 * k + 1];
        const uint32_t w0 = narrow(a.x + a.y, b.x + b.y) ^ m[k] ^ flip0, w1 = narrow(a.x - a.y, b.x - b.y) ^ m[k] ^ flip1;
        uint32_t* at = reinterpret_cast<uint32_t*>(dst + (size_t)(2 * (i + 2 * k)) * n);
        at[0] = __byte_perm(w0, __shfl_xor_sync(kFullWarp, w0, 1), pick);
        at[32] = __byte_perm(w1, __shfl_xor_sync(kFullWarp, w1, 1), pick);
      }
    }
  }
}

template <int K>
static int launch_decode_raw(const uint32_t* qw, int16_t* out, long long ntiles, cudaStream_t st) {
  const long long blocks = (ntiles * 8 + 255) / 256;
  decode_raw_kernel<K><<<(unsigned)blocks, 256, 0, st>>>(qw, out, ntiles);
  return (int)cudaGetLastError();
}

template <int K, int OUT>
static int launch_dequant_w_as(const uint32_t* qw, const __half* scales, const uint8_t* su, const uint8_t* sv, float cb, void* W, int mt, int nt,
                               cudaStream_t st) {
  static bool allowed[64] = {false};                         // shared memory beyond 48 KB: opted in once per device
  int dev = 0;
  if (const cudaError_t e = cudaGetDevice(&dev)) return (int)e;
  if (dev < 0 || dev >= 64 || !allowed[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(dequant_w_kernel<K, OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDqSmem);
    if (e != cudaSuccess) return (int)e;
    if (dev >= 0 && dev < 64) allowed[dev] = true;
  }
  dequant_w_kernel<K, OUT><<<dim3(nt / 8, mt / 8), kDqThreads, kDqSmem, st>>>(qw, scales, su, sv, cb, W, nt);
  return (int)cudaGetLastError();
}

template <int K>
static int launch_dequant_w(const uint32_t* qw, const __half* scales, const uint8_t* su, const uint8_t* sv, float cb, void* W,
                            int out_dtype, int mt, int nt, cudaStream_t st) {
  switch (out_dtype) {
    case HTR_DTYPE_BF16: return launch_dequant_w_as<K, HTR_DTYPE_BF16>(qw, scales, su, sv, cb, W, mt, nt, st);
    case HTR_DTYPE_F16: return launch_dequant_w_as<K, HTR_DTYPE_F16>(qw, scales, su, sv, cb, W, mt, nt, st);
    default: return launch_dequant_w_as<K, HTR_DTYPE_F32>(qw, scales, su, sv, cb, W, mt, nt, st);
  }
}

int run_decode_raw(int K, const uint32_t* qw, int16_t* out, long long ntiles, cudaStream_t st) {
  switch (K) {
    case 2: return launch_decode_raw<2>(qw, out, ntiles, st);
    case 3: return launch_decode_raw<3>(qw, out, ntiles, st);
    case 4: return launch_decode_raw<4>(qw, out, ntiles, st);
    case 5: return launch_decode_raw<5>(qw, out, ntiles, st);
    case 6: return launch_decode_raw<6>(qw, out, ntiles, st);
    case 8: return launch_decode_raw<8>(qw, out, ntiles, st);
  }
  return (int)cudaErrorInvalidValue;
}

int run_rht(const void* x, int dtype, int M, int n, const uint8_t* su, float* xt, cudaStream_t st) {
  const long long warps = (long long)M * (n >> 7);
  const long long blocks = (warps + 7) / 8;
  rht_kernel<<<(unsigned)blocks, 256, 0, st>>>(x, dtype, M, n, su, xt);
  return (int)cudaGetLastError();
}

int run_dequant_w(int K, const uint32_t* qw, const __half* scales, const uint8_t* su, const uint8_t* sv, float cb, void* W,
                  int out_dtype, int mt, int nt, cudaStream_t st) {
  switch (K) {
    case 2: return launch_dequant_w<2>(qw, scales, su, sv, cb, W, out_dtype, mt, nt, st);
    case 3: return launch_dequant_w<3>(qw, scales, su, sv, cb, W, out_dtype, mt, nt, st);
    case 4: return launch_dequant_w<4>(qw, scales, su, sv, cb, W, out_dtype, mt, nt, st);
    case 5: return launch_dequant_w<5>(qw, scales, su, sv, cb, W, out_dtype, mt, nt, st);
    case 6: return launch_dequant_w<6>(qw, scales, su, sv, cb, W, out_dtype, mt, nt, st);
    case 8: return launch_dequant_w<8>(qw, scales, su, sv, cb, W, out_dtype, mt, nt, st);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace htr
