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
//  * the rows of a block do not depend on the length, so the first keys and values (256 positions of the cluster) are loaded right
//    after the wait, together with the position and the new row;
//  * the rows are usually in DRAM by then: before the wait the position is read as a hint, to bring them to L2 and
//    to load the rotation, which is loaded again if the position turns out to be another.
// The cluster's partial softmax results meet in distributed shared memory; block h % 4 finishes query head h of the group.  Same
// roundings as rope_cache_kernel + attention_kernel up to the order of the float32 sums.  A token of the 36-layer decoder at position
// 200: 2.97 -> 2.52 ms; of a small one (12 layers, 16 / 4 heads) at position 900: 1.10 -> 0.46 ms.
constexpr int kAttSplit = 4, kAttHeads = 4, kAttThreads = 256, kAttWarps = kAttThreads / 32;
constexpr int kAttLocal = HTR_DEC_MAX_LEN / kAttSplit;       // positions of one thread block at most

__device__ __forceinline__ void unpack8(const uint4 raw, float (&f)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}
__device__ __forceinline__ void cluster_write(float* mine, unsigned rank, float v) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

__global__ void __cluster_dims__(kAttSplit, 1, 1) __launch_bounds__(kAttThreads, 1)
    rope_attention_kernel(const __nv_bfloat16* __restrict__ qkv, const long long* __restrict__ pos, const float* __restrict__ cosv,
                          const float* __restrict__ sinv, __nv_bfloat16* __restrict__ k_cache, __nv_bfloat16* __restrict__ v_cache,
                          __nv_bfloat16* __restrict__ out, int hq, int hkv, int capacity, int* __restrict__ status) {
  constexpr int D = 128, S = kAttSplit, H = kAttHeads;
  __shared__ __align__(16) float sq[H][D];
  __shared__ __align__(16) float sk[D], sv[D];
  __shared__ float sc[H][kAttLocal];
  __shared__ __align__(16) float part[kAttWarps][H][D];
  __shared__ float s_m[H], s_l[H];
  __shared__ float in_out[H][S][D], in_m[H][S], in_l[H][S];    // what the blocks of the cluster found for this block's query heads
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // this block runs: its shared memory may be written (waited for below)
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
  const int sub = lane >> 3, e = lane & 7;                     // scores: eight lanes per position, 16 dimensions each
  constexpr int kKeys = 2;                                      // key rows of a lane group in flight
  uint4 kr[kKeys][2];
  auto load_keys = [&](int base, int end) {
#pragma unroll
    for (int k = 0; k < kKeys; ++k) {
      const int i = base + (k * kAttWarps + warp) * 4 + sub;
      kr[k][0] = kr[k][1] = make_uint4(0u, 0u, 0u, 0u);
      if (i < end) {
        const uint4* row = reinterpret_cast<const uint4*>(kbase + (size_t)(i * S + rank) * stride + e * 16);
        kr[k][0] = row[0];
        kr[k][1] = row[1];
      }
    }
  };
  constexpr int kAhead = 8;                                     // value rows of a warp in flight: warp, warp + 8, ... of the block
  uint2 vr[kAhead];
  auto load_values = [&](int base, int end) {
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int i = base + warp + kAttWarps * j;
      vr[j] = i < end ? *reinterpret_cast<const uint2*>(vbase + (size_t)(i * S + rank) * stride + 4 * lane) : make_uint2(0u, 0u);
    }
  };
  const int local_limit = (limit - rank + S - 1) / S;           // positions of this block inside the caches
  load_keys(0, local_limit);
  load_values(0, local_limit);
  if (p0 < 0 || p0 >= limit) {                                  // outside the cache: no cache row is touched, zeros come out (the whole cluster)
    if (status && tid == 0 && blockIdx.x == 0 && blockIdx.y == 0) atomicOr(status, 4);
    for (int x = tid; x < nh * D && rank == 0; x += kAttThreads) out[(size_t)head0 * D + x] = __float2bfloat16_rn(0.f);
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    return;
  }
  const int p = (int)p0, mine = p >= rank ? (p - rank) / S + 1 : 0;   // positions of this block
  const bool owner = p % S == rank;                             // of the new position, its last
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
  __syncthreads();
  // ---- scores
  for (int base = 0; base < mine; base += kKeys * kAttWarps * 4) {
    if (base > 0) load_keys(base, mine - owner);               // (the new row does not come through the cache)
#pragma unroll
    for (int k = 0; k < kKeys; ++k) {
      const int i = base + (k * kAttWarps + warp) * 4 + sub;
      if (base + (k * kAttWarps + warp) * 4 >= mine) break;      // warp-uniform
      float kf[16];
      unpack8(kr[k][0], *reinterpret_cast<float(*)[8]>(kf));
      unpack8(kr[k][1], *reinterpret_cast<float(*)[8]>(kf + 8));
      if (owner && i == mine - 1) {
#pragma unroll
        for (int d = 0; d < 16; ++d) kf[d] = sk[e * 16 + d];
      }
#pragma unroll
      for (int h = 0; h < H; ++h) {
        float dot = 0.f;
#pragma unroll
        for (int d = 0; d < 16; d += 4) {
          const float4 q = *reinterpret_cast<const float4*>(&sq[h][e * 16 + d]);
          dot += kf[d] * q.x + kf[d + 1] * q.y + kf[d + 2] * q.z + kf[d + 3] * q.w;
        }
#pragma unroll
        for (int o = 4; o; o >>= 1) dot += __shfl_xor_sync(0xFFFFFFFFu, dot, o);
        if (e == h && i < mine) sc[h][i] = dot;
      }
    }
  }
  __syncthreads();
  if (warp < H) {                                               // softmax of this block's positions, one warp per head
    float mx = -3.0e38f, sum = 0.f;
    for (int i = lane; i < mine; i += 32) mx = fmaxf(mx, sc[warp][i]);
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    for (int i = lane; i < mine; i += 32) {
      const float w = __expf(sc[warp][i] - mx);
      sc[warp][i] = w;
      sum += w;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    if (lane == 0) {
      s_m[warp] = mx;
      s_l[warp] = sum;
    }
  }
  __syncthreads();
  // ---- values: a lane holds four dimensions of a row, for all heads
  float acc[H][4];
#pragma unroll
  for (int h = 0; h < H; ++h) acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f;
  for (int base = 0; base < mine; base += kAttWarps * kAhead) {
    if (base > 0) load_values(base, mine - owner);
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const int i = base + warp + kAttWarps * j;
      if (i >= mine) break;
      float4 v = make_float4(__uint_as_float(vr[j].x << 16), __uint_as_float(vr[j].x & 0xFFFF0000u), __uint_as_float(vr[j].y << 16),
                             __uint_as_float(vr[j].y & 0xFFFF0000u));
      if (owner && i == mine - 1) v = *reinterpret_cast<const float4*>(sv + 4 * lane);
#pragma unroll
      for (int h = 0; h < H; ++h) {
        const float w = sc[h][i];
        acc[h][0] += w * v.x; acc[h][1] += w * v.y; acc[h][2] += w * v.z; acc[h][3] += w * v.w;
      }
    }
  }
#pragma unroll
  for (int h = 0; h < H; ++h) *reinterpret_cast<float4*>(&part[warp][h][4 * lane]) = make_float4(acc[h][0], acc[h][1], acc[h][2], acc[h][3]);
  __syncthreads();
  asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // every block of the cluster has started
  for (int x = tid; x < H * D; x += kAttThreads) {
    const int h = x >> 7, d = x & 127;
    float o = 0.f;
#pragma unroll
    for (int w = 0; w < kAttWarps; ++w) o += part[w][h][d];
    cluster_write(&in_out[h][rank][d], h % S, o);
  }
  if (tid < H) {
    cluster_write(&in_m[tid][rank], tid % S, s_m[tid]);
    cluster_write(&in_l[tid][rank], tid % S, s_l[tid]);
  }
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  for (int x = tid; x < H / S * D; x += kAttThreads) {
    const int h = (x >> 7) * S + rank, d = x & 127;
    if (h >= nh) break;
    float mx = in_m[h][0];
#pragma unroll
    for (int r = 1; r < S; ++r) mx = fmaxf(mx, in_m[h][r]);
    float sum = 0.f, acc_o = 0.f;
#pragma unroll
    for (int r = 0; r < S; ++r) {
      const float w = __expf(in_m[h][r] - mx);                  // (a block without positions: m = -3e38, weight zero)
      sum += w * in_l[h][r];
      acc_o += w * in_out[h][r][d];
    }
    out[(size_t)(head0 + h) * D + d] = __float2bfloat16_rn(acc_o / sum);
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
int launch_pdl(Kern kern, dim3 grid, dim3 block, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
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
  const int e = launch_pdl(add_rmsnorm_kernel, dim3(rows), dim3(256), static_cast<cudaStream_t>(stream), static_cast<__nv_bfloat16*>(resid),
                           static_cast<const __nv_bfloat16*>(delta), static_cast<const __nv_bfloat16*>(weight), static_cast<__nv_bfloat16*>(out), h, eps);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_dec_rope_cache(const void* qkv, const int64_t* pos, const float* cosv, const float* sinv, void* q_out, void* k_cache, void* v_cache,
                       int rows, int q_heads, int kv_heads, int head_dim, int capacity, int* status, htr_stream_t stream) {
  if (rows <= 0) return HTR_OK;
  if (!qkv || !pos || !cosv || !sinv || !q_out || !k_cache || !v_cache) return HTR_ERR_NULL;
  if (head_dim <= 0 || head_dim % 2 || head_dim > 2048 || q_heads <= 0 || kv_heads <= 0 || capacity <= 0) return HTR_ERR_BAD_SHAPE;
  const int e = launch_pdl(rope_cache_kernel, dim3(q_heads + 2 * kv_heads, rows), dim3(head_dim / 2), static_cast<cudaStream_t>(stream),
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
  const int e = launch_pdl(attention_kernel, dim3(q_heads, rows), dim3(128), static_cast<cudaStream_t>(stream), static_cast<const __nv_bfloat16*>(q),
                           static_cast<const __nv_bfloat16*>(k_cache), static_cast<const __nv_bfloat16*>(v_cache),
                           reinterpret_cast<const long long*>(pos), static_cast<__nv_bfloat16*>(out), q_heads, kv_heads, capacity, status);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

int htr_dec_rope_attention(const void* qkv, const int64_t* pos, const float* cosv, const float* sinv, void* k_cache, void* v_cache, void* out,
                           int q_heads, int kv_heads, int head_dim, int capacity, int* status, htr_stream_t stream) {
  if (!qkv || !pos || !cosv || !sinv || !k_cache || !v_cache || !out) return HTR_ERR_NULL;
  if (head_dim != 128 || q_heads <= 0 || kv_heads <= 0 || q_heads % kv_heads || capacity <= 0) return HTR_ERR_BAD_SHAPE;
  const int e = launch_pdl(rope_attention_kernel, dim3(kAttSplit * kv_heads, (q_heads / kv_heads + kAttHeads - 1) / kAttHeads), dim3(kAttThreads), static_cast<cudaStream_t>(stream),
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
  const int e = launch_pdl(swiglu_kernel, dim3((total / 2 + 255) / 256), dim3(256), static_cast<cudaStream_t>(stream),
                           static_cast<const __nv_bfloat16*>(gate_up), static_cast<__nv_bfloat16*>(out), intermediate, total);
  return e ? HTR_ERR_CUDA : HTR_OK;
}

}  // extern "C"
