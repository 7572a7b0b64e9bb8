// Small fused kernels of the decoder harness (the non-linear glue between packed linears in a decode step):
// residual add + RMSNorm, rotary embedding + KV-cache write, single-query grouped-query attention, SwiGLU.
// They exist so that a decode step is a short chain of launches around the packed GEMVs instead of dozens of
// framework kernels; every one is launched with programmatic stream serialisation, signals its dependents at once and
// waits for its predecessor before touching data, so the next packed GEMV prefetches its weights while these run.
// bf16 activations, float32 arithmetic.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/htr_b200.h"
#include "htr_common.cuh"

namespace {

__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = 0.f;
  for (int i = 0; i < nw; ++i) t += red[i];
  return t;
}

__device__ __forceinline__ float block_max(float v, float* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float t = -3.0e38f;
  for (int i = 0; i < nw; ++i) t = fmaxf(t, red[i]);
  return t;
}

// resid += delta (if any); out = rmsnorm(resid) * w.  One CTA per row; the row stays in registers between the two passes
// (h <= 8192: up to 16 bf16 pairs per thread).
__global__ void __launch_bounds__(256) add_rmsnorm_kernel(__nv_bfloat16* __restrict__ resid, const __nv_bfloat16* __restrict__ delta,
                                                          const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ out, int h, float eps) {
  __shared__ float red[8];
  pdl_enter();
  const size_t row = (size_t)blockIdx.x * h;
  constexpr int kMaxPairs = 16;
  float2 v[kMaxPairs];
  float2 g[kMaxPairs];
  float ss = 0.f;
#pragma unroll
  for (int j = 0; j < kMaxPairs; ++j) {
    const int i = (threadIdx.x + j * 256) * 2;
    v[j] = make_float2(0.f, 0.f);
    g[j] = make_float2(0.f, 0.f);
    if (i < h) {
      v[j] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(resid + row + i));
      g[j] = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(w + i));
      if (delta) {
        const float2 d = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(delta + row + i));
        const __nv_bfloat162 r = __floats2bfloat162_rn(v[j].x + d.x, v[j].y + d.y);
        *reinterpret_cast<__nv_bfloat162*>(resid + row + i) = r;
        v[j] = __bfloat1622float2(r);                   // the norm sees the stored (rounded) residual, as a framework would
      }
      ss += v[j].x * v[j].x + v[j].y * v[j].y;
    }
  }
  const float inv = rsqrtf(block_sum(ss, red) / (float)h + eps);
#pragma unroll
  for (int j = 0; j < kMaxPairs; ++j) {
    const int i = (threadIdx.x + j * 256) * 2;
    if (i < h) {
      // normalise, round to bf16, then scale: the order of the unfused reference ops
      const float2 nf = __bfloat1622float2(__floats2bfloat162_rn(v[j].x * inv, v[j].y * inv));
      *reinterpret_cast<__nv_bfloat162*>(out + row + i) = __floats2bfloat162_rn(nf.x * g[j].x, nf.y * g[j].y);
    }
  }
}

// rotary embedding of q and k (interleaved pairs), k and v written into the cache rows pos[t].  grid (heads_q + 2*heads_kv, T), D/2 threads.
__global__ void rope_cache_kernel(const __nv_bfloat16* __restrict__ qkv, const long long* __restrict__ pos, const float* __restrict__ cosv,
                                  const float* __restrict__ sinv, __nv_bfloat16* __restrict__ q_out, __nv_bfloat16* __restrict__ k_cache,
                                  __nv_bfloat16* __restrict__ v_cache, int hq, int hkv, int D, int capacity, int* __restrict__ status) {
  pdl_enter();
  const int head = blockIdx.x, t = blockIdx.y, i = threadIdx.x;           // pair index i: elements 2i, 2i+1
  const long long p = pos[t];
  if (p < 0 || p >= capacity) {                                           // a position outside the cache: nothing is read or written
    if (status && i == 0 && head == 0) atomicOr(status, 1);
    return;
  }
  const size_t row = (size_t)t * (hq + 2 * hkv) * D;
  const __nv_bfloat162 in = *reinterpret_cast<const __nv_bfloat162*>(qkv + row + (size_t)head * D + 2 * i);
  if (head >= hq + hkv) {                                                 // v: plain copy into the cache
    *reinterpret_cast<__nv_bfloat162*>(v_cache + ((size_t)p * hkv + (head - hq - hkv)) * D + 2 * i) = in;
    return;
  }
  const float2 v = __bfloat1622float2(in);
  const float c = cosv[(size_t)p * (D / 2) + i], s = sinv[(size_t)p * (D / 2) + i];
  const __nv_bfloat162 r = __floats2bfloat162_rn(v.x * c - v.y * s, v.x * s + v.y * c);
  if (head < hq) *reinterpret_cast<__nv_bfloat162*>(q_out + ((size_t)t * hq + head) * D + 2 * i) = r;
  else *reinterpret_cast<__nv_bfloat162*>(k_cache + ((size_t)p * hkv + (head - hq)) * D + 2 * i) = r;
}

// out[t, head, :] = softmax(q . K[0..pos[t]] / sqrt(D)) V.  grid (heads_q, T), 128 threads, D == 128, positions < min(capacity,
// HTR_DEC_MAX_LEN); a row whose position lies outside gets zeros and sets the status word.
// Scores: one thread per position (128 positions per pass, the 256-byte key row read as sixteen 16-byte loads);
// values: one thread per dimension, eight positions in flight.
__global__ void __launch_bounds__(128) attention_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_cache,
                                                        const __nv_bfloat16* __restrict__ v_cache, const long long* __restrict__ pos,
                                                        __nv_bfloat16* __restrict__ out, int hq, int hkv, int capacity, int* __restrict__ status) {
  constexpr int D = 128;
  __shared__ __align__(16) float sq[D];
  __shared__ float sc[HTR_DEC_MAX_LEN];
  __shared__ float red[4];
  pdl_enter();
  const int head = blockIdx.x, t = blockIdx.y, tid = threadIdx.x;
  const int kvh = head / (hq / hkv);
  const long long pt = pos[t];
  if (pt < 0 || pt >= capacity || pt >= HTR_DEC_MAX_LEN) {                // the whole CTA takes this branch: no barrier is skipped by a part of it
    if (status && tid == 0 && head == 0) atomicOr(status, 2);
    out[((size_t)t * hq + head) * D + tid] = __float2bfloat16_rn(0.f);
    return;
  }
  const int len = (int)pt + 1;
  sq[tid] = bf(q[((size_t)t * hq + head) * D + tid]) * 0.08838834764831845f;   // 1/sqrt(128)
  __syncthreads();
  float mx = -3.0e38f;
  for (int p = tid; p < len; p += 128) {
    const uint4* kr = reinterpret_cast<const uint4*>(k_cache + ((size_t)p * hkv + kvh) * D);
    float d = 0.f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 raw = __ldg(kr + c);
      const float4 q0 = *reinterpret_cast<const float4*>(sq + 8 * c), q1 = *reinterpret_cast<const float4*>(sq + 8 * c + 4);
      const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
      const float2 e = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.z)), f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.w));
      d += a.x * q0.x + a.y * q0.y + b.x * q0.z + b.y * q0.w + e.x * q1.x + e.y * q1.y + f.x * q1.z + f.y * q1.w;
    }
    sc[p] = d;
    mx = fmaxf(mx, d);
  }
  mx = block_max(mx, red);
  float sum = 0.f;
  for (int p = tid; p < len; p += 128) {
    const float e = __expf(sc[p] - mx);
    sc[p] = e;
    sum += e;
  }
  sum = block_sum(sum, red);
  const __nv_bfloat16* vcol = v_cache + (size_t)kvh * D + tid;
  float acc = 0.f;
  int p = 0;
  for (; p + 8 <= len; p += 8) {
    float vv[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) vv[j] = bf(vcol[(size_t)(p + j) * hkv * D]);
#pragma unroll
    for (int j = 0; j < 8; ++j) acc += sc[p + j] * vv[j];
  }
  for (; p < len; ++p) acc += sc[p] * bf(vcol[(size_t)p * hkv * D]);
  out[((size_t)t * hq + head) * D + tid] = __float2bfloat16_rn(acc / sum);
}

// Single-token step: rotary embedding, cache write and attention of up to four query heads of one key/value head in one kernel.
// grid (4 * heads_kv, ceil(group / 4)), clusters of 4 thread blocks of 256 threads, D == 128.
// What bounds it: at a few hundred positions not the bytes (400 KB) but a chain of dependent loads, one after the other in one block
// per query head: position -> rotation -> scores -> values, eight rows at a time, 17 us at position 200.  So
//  * a cluster shares the positions of a key/value head (block r takes positions r, r + 4, ...) and a block serves the whole group of
//    query heads, so that each key and value row is read once;
//  * the rows of a block do not depend on the length, so the first keys and values (256 positions of the cluster) are copied to shared
//    memory right after the wait, while the position and the new row arrive; later ones follow two buffers ahead;
//  * the rows are usually in DRAM by then: before the wait the position is read as a hint, to bring them to L2 and
//    to load the rotation, which is loaded again if the position turns out to be another.
// The order of every float32 sum is fixed and does not depend on the split: a score is one thread's sum along the row, the value rows
// are added in four streams (positions t = r mod 4, a block each), and the weights as 128 threads would, then over their lanes and
// warps.  A decoder of dozens of bf16 layers turns one other rounding into another result of percents (no worse a one), so this order
// stays and results with it.  Block h
// of the cluster adds up and finishes query head h of the group: scores and streams meet in its shared memory.
// A token of a small decoder (12 layers of hidden 2048, 16 / 4 heads; with the other changes to its step) at position 200: 612 -> 431 us, at
// position 900: 1247 -> 507.
constexpr int kAttSplit = 4, kAttHeads = 4, kAttThreads = 256, kAttWarps = kAttThreads / 32;
constexpr int kAttRows = 64, kAttPitch = 272;                // positions of a buffer; bytes of a row in it (17 x 16: no bank conflicts)
constexpr int kAttLocal = HTR_DEC_MAX_LEN / kAttSplit;       // positions of one thread block at most
constexpr int kAttBuffer = kAttRows * kAttPitch, kAttSmem = 4 * kAttBuffer;

__device__ __forceinline__ void cluster_write(float* mine, unsigned rank, float v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

__global__ void __cluster_dims__(kAttSplit, 1, 1) __launch_bounds__(kAttThreads, 1)
    rope_attention_kernel(const __nv_bfloat16* __restrict__ qkv, const long long* __restrict__ pos, const float* __restrict__ cosv,
                          const float* __restrict__ sinv, __nv_bfloat16* k_cache, __nv_bfloat16* v_cache,
                          __nv_bfloat16* __restrict__ out, int hq, int hkv, int capacity, int* __restrict__ status) {
  constexpr int D = 128, S = kAttSplit, H = kAttHeads;
  static_assert(S == H && kAttThreads == kAttRows * H, "a block finishes one head; a thread per position and head");
  extern __shared__ __align__(16) unsigned char rows[];        // two buffers of keys, two of values
  __shared__ __align__(16) float sq[H][D];
  __shared__ __align__(16) float sk[D], sv[D];
  __shared__ float sc[H][kAttLocal];                            // scores of this block's positions
  __shared__ float all[HTR_DEC_MAX_LEN];                        // from the cluster, for the head this block finishes: scores ...
  __shared__ float part[S][D];                                  // ... and weighted sums
  __shared__ float in_m[H][S * 2];                              // largest scores: two warps per head and block
  __shared__ float red[4];
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  htr::cluster_arrive_relaxed();                                  // this block runs: its shared memory may be written (waited for below)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % S, kvh = blockIdx.x / S, rep = hq / hkv, head0 = kvh * rep + blockIdx.y * H;
  const int nh = min(H, rep - (int)blockIdx.y * H);            // query heads of this cluster
  const int limit = min(capacity, HTR_DEC_MAX_LEN);
  const size_t stride = (size_t)hkv * D;
  const __nv_bfloat16 *kbase = k_cache + (size_t)kvh * D, *vbase = v_cache + (size_t)kvh * D;
  const int pair = tid & 63;
  // ---- before the predecessor is done: hints only (the position may still be written)
  long long hint = *reinterpret_cast<const volatile long long*>(pos);
  if (hint < 0 || hint >= limit) hint = 0;
  float c = cosv[(size_t)hint * (D / 2) + pair], s = sinv[(size_t)hint * (D / 2) + pair];
  for (int i = tid >> 2; i * S + rank < hint; i += kAttThreads / 4) {   // four threads per position: both 128-byte lines of key and value
    const __nv_bfloat16* row = (tid & 2 ? vbase : kbase) + (size_t)(i * S + rank) * stride + (tid & 1) * 64;
    asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // ---- everything whose address is known, at once
  const long long p0 = *reinterpret_cast<const volatile long long*>(pos);
  // items 0..3: query heads, 4: the new key, 5: the new value; a thread takes its 64-thread group's and the one four further on
  __nv_bfloat162 raw[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int who = (tid >> 6) + 4 * k;
    const int src_head = who < H ? head0 + min(who, nh - 1) : who == 4 ? hq + kvh : hq + hkv + kvh;
    if (who < 6) raw[k] = *reinterpret_cast<const __nv_bfloat162*>(qkv + (size_t)src_head * D + 2 * pair);
  }
  const uint32_t rows_at = (uint32_t)__cvta_generic_to_shared(rows);
  // positions [64 chunk, 64 chunk + 64) of this block below `end` into a buffer (16 threads per row); commits a group, also an empty one
  auto copy_rows = [&](const __nv_bfloat16* base, int buffer, int chunk, int end) {
#pragma unroll
    for (int k = 0; k < kAttRows * 16 / kAttThreads; ++k) {
      const int row = k * (kAttThreads / 16) + (tid >> 4), i = chunk * kAttRows + row;
      if (i < end)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(rows_at + buffer * kAttBuffer + row * kAttPitch + (tid & 15) * 16),
                     "l"(base + (size_t)(i * S + rank) * stride + (tid & 15) * 8) : "memory");
    }
    copy_commit();
  };
  const int local_limit = (limit - rank + S - 1) / S;           // positions of this block inside the caches
  copy_rows(kbase, 0, 0, local_limit);
  copy_rows(vbase, 2, 0, local_limit);
  if (p0 < 0 || p0 >= limit) {                                  // outside the cache: no cache row is touched, zeros come out (the whole cluster)
    if (status && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) atomicOr(status, 4);
    for (int x = tid; x < nh * D && rank == 0; x += kAttThreads) out[(size_t)head0 * D + x] = __float2bfloat16_rn(0.f);
    copy_wait<0>();
    htr::cluster_wait();
    return;
  }
  const int p = (int)p0, mine = (p + S - 1 - rank) / S;         // cached positions of this block (the new one does not come through the cache)
  copy_rows(kbase, 1, 1, mine);
  copy_rows(vbase, 3, 1, mine);
  const bool owner = p % S == rank;                             // of the new position
  if (p != (int)hint) {
    c = cosv[(size_t)p * (D / 2) + pair];
    s = sinv[(size_t)p * (D / 2) + pair];
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const int who = (tid >> 6) + 4 * k;
    if (who >= 6) continue;
    const float2 v = __bfloat1622float2(raw[k]);
    const __nv_bfloat162 r = who == 5 ? raw[k] : __floats2bfloat162_rn(v.x * c - v.y * s, v.x * s + v.y * c);
    const float2 f = __bfloat1622float2(r);
    if (who < H) {
      *reinterpret_cast<float2*>(&sq[who][2 * pair]) = make_float2(f.x * 0.08838834764831845f, f.y * 0.08838834764831845f);   // 1/sqrt(128)
    } else {
      *reinterpret_cast<float2*>((who == 4 ? sk : sv) + 2 * pair) = f;
      if (owner && blockIdx.y == 0)
        *reinterpret_cast<__nv_bfloat162*>((who == 4 ? k_cache : v_cache) + ((size_t)p * hkv + kvh) * D + 2 * pair) = r;
    }
  }
  // ---- scores: warps 2h and 2h + 1 take head h, a thread one position of a buffer
  const int h = warp >> 1, half = warp & 1, chunks = (mine + kAttRows - 1) / kAttRows;
  float mx = -3.0e38f;
  copy_wait<3>();
  __syncthreads();
  htr::cluster_wait();                                           // every block of the cluster has started
  if (owner && half == 0) {                                     // of the new position: four dimensions per lane
    const float4 k4 = *reinterpret_cast<const float4*>(sk + 4 * lane), q4 = *reinterpret_cast<const float4*>(&sq[h][4 * lane]);
    float d = k4.x * q4.x + k4.y * q4.y + k4.z * q4.z + k4.w * q4.w;
#pragma unroll
    for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
    if (lane == 0) cluster_write(&all[p], h, d);
    mx = d;
  }
  for (int chunk = 0; chunk < chunks; ++chunk) {
    if (chunk > 0) {                                            // (groups after this chunk's: values 1 and keys 2, then keys chunk + 1)
      if (chunk == 1) copy_wait<2>();
      else copy_wait<1>();
      __syncthreads();
    }
    const int row = half * 32 + lane, i = chunk * kAttRows + row;
    if (i < mine) {
      const uint4* kr = reinterpret_cast<const uint4*>(rows + (chunk & 1) * kAttBuffer + row * kAttPitch);
      float d = 0.f;
#pragma unroll
      for (int x = 0; x < 16; ++x) {
        const uint4 raw4 = kr[x];
        const float4 q0 = *reinterpret_cast<const float4*>(&sq[h][8 * x]), q1 = *reinterpret_cast<const float4*>(&sq[h][8 * x + 4]);
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw4.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw4.y));
        const float2 e = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw4.z)), f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw4.w));
        d += a.x * q0.x + a.y * q0.y + b.x * q0.z + b.y * q0.w + e.x * q1.x + e.y * q1.y + f.x * q1.z + f.y * q1.w;
      }
      sc[h][i] = d;
      cluster_write(&all[i * S + rank], h, d);
      mx = fmaxf(mx, d);
    }
    if (chunks > 1) {
      __syncthreads();                                          // the buffer is free
      copy_rows(kbase, chunk & 1, chunk + 2, mine);
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  if (lane < S) cluster_write(&in_m[h][rank * 2 + half], lane, mx);
  copy_wait<0>();
  htr::cluster_sync();
  mx = in_m[h][0];
#pragma unroll
  for (int r = 1; r < 2 * S; ++r) mx = fmaxf(mx, in_m[h][r]);
  // ---- values: a warp sums half of the dimensions for its head, position after position; a lane holds two dimensions
  float a0 = 0.f, a1 = 0.f;
  for (int chunk = 0; chunk < chunks; ++chunk) {
    if (chunk > 1) {
      copy_wait<1>();
      __syncthreads();
    }
    const unsigned char* vr = rows + (2 + (chunk & 1)) * kAttBuffer + half * 128 + lane * 4;
    for (int base = chunk * kAttRows; base < min(mine, (chunk + 1) * kAttRows); base += 32, vr += 32 * kAttPitch) {
      const float e = base + lane < mine ? __expf(sc[h][base + lane] - mx) : 0.f;
      const int n = min(32, mine - base);
      if (n == 32) {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float w = __shfl_sync(0xFFFFFFFFu, e, j);
          const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(vr + j * kAttPitch));
          a0 += w * v.x; a1 += w * v.y;
        }
      } else {
#pragma unroll 4
        for (int j = 0; j < n; ++j) {
          const float w = __shfl_sync(0xFFFFFFFFu, e, j);
          const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(vr + j * kAttPitch));
          a0 += w * v.x; a1 += w * v.y;
        }
      }
    }
    if (chunks > 2) {
      __syncthreads();
      copy_rows(vbase, 2 + (chunk & 1), chunk + 2, mine);
    }
  }
  cluster_write(&part[rank][half * 64 + 2 * lane], h, a0);
  cluster_write(&part[rank][half * 64 + 2 * lane + 1], h, a1);
  // ---- the head this block finishes: sum of its weights, then the streams and the new row
  float mo = in_m[rank][0];
#pragma unroll
  for (int r = 1; r < 2 * S; ++r) mo = fmaxf(mo, in_m[rank][r]);
  if (tid < D) {
    float sum = 0.f;
    for (int t = tid; t <= p; t += D) sum += __expf(all[t] - mo);
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) red[warp] = sum;
  }
  copy_wait<0>();
  htr::cluster_sync();
  if (tid < D && rank < nh) {
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < 4; ++w) sum += red[w];
    const float last = __expf(all[p] - mo);
    const float acc = part[0][tid] + part[1][tid] + part[2][tid] + part[3][tid] + last * sv[tid];
    out[(size_t)(head0 + rank) * D + tid] = __float2bfloat16_rn(acc / sum);
  }
}

// out = silu(gate) * up, gu = [T, 2I] with the gate half first
__global__ void __launch_bounds__(256) swiglu_kernel(const __nv_bfloat16* __restrict__ gu, __nv_bfloat16* __restrict__ out, int I, int total) {
  pdl_enter();
  const int idx = (blockIdx.x * 256 + threadIdx.x) * 2;
  if (idx >= total) return;
  const int t = idx / I, j = idx - t * I;
  const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gu + (size_t)t * 2 * I + j));
  const float2 u = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gu + (size_t)t * 2 * I + I + j));
  // silu rounded to bf16 before the product, as the unfused ops do
  const __nv_bfloat162 s = __floats2bfloat162_rn(g.x / (1.f + __expf(-g.x)), g.y / (1.f + __expf(-g.y)));
  const float2 sf = __bfloat1622float2(s);
  *reinterpret_cast<__nv_bfloat162*>(out + (size_t)t * I + j) = __floats2bfloat162_rn(sf.x * u.x, sf.y * u.y);
}

template <typename Kern, typename... Args>
int launch_pdl(Kern kern, dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace

extern "C" {

int htr_dec_add_rmsnorm(void* resid, const void* delta, const void* weight, void* out, int rows, int h, float eps, htr_stream_t stream) {
  if (rows <= 0) return HTR_OK;
  if (!resid || !weight || !out) return HTR_ERR_NULL;
  if (h <= 0 || h % 2 || h > 8192) return HTR_ERR_BAD_SHAPE;
  const int e = launch_pdl(add_rmsnorm_kernel, dim3(rows), dim3(256), 0, static_cast<cudaStream_t>(stream), static_cast<__nv_bfloat16*>(resid),
                           static_cast<const __nv_bfloat16*>(delta), static_cast<const __nv_bfloat16*>(weight), static_cast<__nv_bfloat16*>(out), h, eps);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_dec_rope_cache(const void* qkv, const int64_t* pos, const float* cosv, const float* sinv, void* q_out, void* k_cache, void* v_cache,
                       int rows, int q_heads, int kv_heads, int head_dim, int capacity, int* status, htr_stream_t stream) {
  if (rows <= 0) return HTR_OK;
  if (!qkv || !pos || !cosv || !sinv || !q_out || !k_cache || !v_cache) return HTR_ERR_NULL;
  if (head_dim <= 0 || head_dim % 2 || head_dim > 2048 || q_heads <= 0 || kv_heads <= 0 || capacity <= 0) return HTR_ERR_BAD_SHAPE;
  const int e = launch_pdl(rope_cache_kernel, dim3(q_heads + 2 * kv_heads, rows), dim3(head_dim / 2), 0, static_cast<cudaStream_t>(stream),
                           static_cast<const __nv_bfloat16*>(qkv), reinterpret_cast<const long long*>(pos), cosv, sinv,
                           static_cast<__nv_bfloat16*>(q_out), static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), q_heads,
                           kv_heads, head_dim, capacity, status);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_dec_attention(const void* q, const void* k_cache, const void* v_cache, const int64_t* pos, void* out, int rows, int q_heads,
                      int kv_heads, int head_dim, int capacity, int* status, htr_stream_t stream) {
  if (rows <= 0) return HTR_OK;
  if (!q || !k_cache || !v_cache || !pos || !out) return HTR_ERR_NULL;
  if (head_dim != 128 || q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads || capacity <= 0) return HTR_ERR_BAD_SHAPE;
  const int e = launch_pdl(attention_kernel, dim3(q_heads, rows), dim3(128), 0, static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(q),
                           static_cast<const __nv_bfloat16*>(k_cache), static_cast<const __nv_bfloat16*>(v_cache),
                           reinterpret_cast<const long long*>(pos), static_cast<__nv_bfloat16*>(out), q_heads, kv_heads, capacity, status);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_dec_rope_attention(const void* qkv, const int64_t* pos, const float* cosv, const float* sinv, void* k_cache, void* v_cache, void* out,
                           int q_heads, int kv_heads, int head_dim, int capacity, int* status, htr_stream_t stream) {
  if (!qkv || !pos || !cosv || !sinv || !k_cache || !v_cache || !out) return HTR_ERR_NULL;
  if (head_dim != 128 || q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads || capacity <= 0) return HTR_ERR_BAD_SHAPE;
  static bool allowed[64] = {false};                      // shared memory beyond 48 KB: opted in once per device
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return HTR_ERR_CUDA;
  if (dev < 0 || dev >= 64 || !allowed[dev]) {
    if (cudaFuncSetAttribute(rope_attention_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kAttSmem) != cudaSuccess) return HTR_ERR_CUDA;
    if (dev >= 0 && dev < 64) allowed[dev] = true;
  }
  const int e = launch_pdl(rope_attention_kernel, dim3(kAttSplit * kv_heads, (q_heads / kv_heads + kAttHeads - 1) / kAttHeads), dim3(kAttThreads),
                           kAttSmem, static_cast<cudaStream_t>(stream),
                           static_cast<const __nv_bfloat16*>(qkv), reinterpret_cast<const long long*>(pos), cosv, sinv,
                           static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), static_cast<__nv_bfloat16*>(out), q_heads,
                           kv_heads, capacity, status);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_dec_swiglu(const void* gate_up, void* out, int rows, int intermediate, htr_stream_t stream) {
  if (rows <= 0) return HTR_OK;
  if (!gate_up || !out) return HTR_ERR_NULL;
  if (intermediate <= 0 || intermediate % 2) return HTR_ERR_BAD_SHAPE;
  const int total = rows * intermediate;
  const int e = launch_pdl(swiglu_kernel, dim3((total / 2 + 255) / 256), dim3(256), 0, static_cast<cudaStream_t>(stream),
                           static_cast<const __nv_bfloat16*>(gate_up), static_cast<__nv_bfloat16*>(out), intermediate, total);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

}  // extern "C"
