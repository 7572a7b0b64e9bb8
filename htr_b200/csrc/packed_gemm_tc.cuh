// Packed GEMM for batches on sm_100a: decoded tiles feed tcgen05.mma from tensor memory, accumulators live there too.
//
//   Y[j, i] = sum_k Xt[j, k] * V[i, k]   for one 128-row block i of the weight, activation rows j (up to 256 per launch)
//
// Replaces the reference's prefill route (dequant_w to bf16 in DRAM + library GEMM, htr/ops.py:89-93, kernels
// htr_kernels.cu:658-903): the packed words are decoded once per launch straight into the A operand and never reach memory as
// 16-bit weights.
//
// Operands.  A holds the codebook integers as exact fp16 values 1024 + bytesum (the fp16 bit pattern 0x6400 + bytesum needs no
// conversion instruction); the constant 1534 = 1024 + 510 is removed in the epilogue with the row sums of the activations, as the
// reference does (htr_kernels.cu:312-313).  B holds the transformed activations as one fp16 plane `hi`, or two, hi and
// lo = fp16(xt - hi), concatenated along N, so that the products carry ~22 bits of the activations; the two accumulator halves are
// added after the MMA.  A per-row power-of-two scale puts |xt| just inside the fp16 range (htr_kernels.cu:205-206; here small rows are
// scaled up as well).
//
// What bounds it: producing A.  A weight costs about four issue slots (window, hash multiply-add, byte sum, half a pack) whatever
// the batch, so the goal is that the decode warps do nothing else.  Two properties of the layout serve that:
//  * A lives in tensor memory, not in shared memory.  An fp16 weight that is stored to and fetched from shared memory takes 4 of
//    its 128 bytes per cycle and SM, a bound of 32 weights per cycle by itself beside B and the packed words; the tensor-memory
//    path carries A alone (the MMA fetches 4 KB in 32 cycles: 64 weights per cycle).
//  * tcgen05.st.16x256b gives a thread a piece of two rows, which is the decode unit (a row pair of one tile, whose 32 windows
//    share words): lane (g, c) decodes rows 2g, 2g+1 of tile c of a 16-row strip's four tiles and one store per unit places them.
//    Tensor-memory lane l < 8 of a strip holds weight row 2l, lane 8 + l row 2l + 1, and MMA step j takes columns 4j..4j+3 of each
//    of the four tiles; the activation transform writes B in that k order.
// The packed words take a ring per warp (16-byte cp.async, all slots but one in flight): plain loads into registers one block ahead
// keep 16 KB per SM in flight and measured 12 weights per cycle and SM, the ring 17 over the launch of an LM head (151936x4096 K4, 8 rows: 622
// million weights in 127 us; the same at any depth from 3 slots on), at 80 % of the issue slots: 5.6 instructions a weight over the launch, of
// which the decode unit is about four.
//
// Roles (22 warps, one thread block per SM).  Warps 0-15 decode, as two groups of eight that take alternate 128-column blocks;
// inside a group warp w owns tensor-memory quadrant w % 4 and strip 2 (w % 4) + (w / 4) % 2.  One lane of warp 16 brings the B tile
// of each block (one bulk copy, completion counted on an mbarrier); one lane of warp 17 issues the eight MMAs of a block.  Stage s of
// the ring is {64 tensor-memory columns of A, one B tile} with full[s] and freed[s] (tcgen05.commit); with up to seven
// stages the decode runs ahead while the activation transform before the launch still works and while an accumulator is read.
// Warps 18-21 finish the row blocks of a flat run: they move the accumulator to a partial sum in memory and, where it is the last, add the
// partials, apply scales, output transform and signs, and store.  (Done by the decode warps, that chain of dependent loads cost 12 000
// cycles per row block, a fifth of the LM head at 8 rows.)  The last row block of a run is finished by all warps.
// A thread block with one row block, or a part of one (clusters, whole row blocks), has no use for them: its decode warps fetch what
// their rows need (scales, signs, activation sums, lane i those of the i-th row) behind their last block, beside the last MMAs, move the
// accumulator, four warps per quadrant, and finish.  With the finishers in their place a row waited for its own loads and 200 rows left
// tensor memory one column group at a time.  us, before -> after: 32768x256, 8 / 200 rows 11.9 -> 10.0, 34.6 -> 24.8; 4096x4096, 8 / 256 rows
// 9.9 -> 9.0, 25.9 -> 22.8; 2048x2048, 8 rows 7.5 -> 6.7; 4096x12288, 128 rows 27.5 -> 25.0 (each before the inbox below).
//
// Decomposition.  Work = (row block) x (128-column blocks).  Where the row blocks are few, `split` thread blocks share one as a
// cluster: each sends its partial sums of a row into the shared memory of the one that finishes that row (st.async, up to 64 rows), or,
// where no inbox fits or the rows are many, fetches the others' between two cluster barriers.  4096x12288 K3, 4 rows: 17.1 -> 16.5 us
// for the inbox.  Else every thread block takes an even contiguous run that may cross row blocks (flat), publishes a partial [np][128]
// per row block it touches, and the last arriver adds them in thread-block order.  Both are deterministic and nobody waits for another
// thread block except inside a cluster.  One thread block per SM, not two: the partial sums of a row block are half as many, and no SM
// waits for the slower of two.
//
// Every wait on an mbarrier is bounded: when it expires the thread block records an error code, stops issuing work, waits (bounded)
// for its copies and MMAs in flight, writes NaN into the rows it owed, frees its tensor memory and returns; the host sees the code
// in the workspace header.
#pragma once
#include "htr_codec.cuh"
#include "htr_common.cuh"

namespace htr {

constexpr int kGemmMaxStages = 7;
constexpr int kGemmDecodeWarps = 16, kGemmGroupWarps = 8;
constexpr int kGemmFinishWarps = 4;
constexpr int kGemmWarps = kGemmDecodeWarps + 2 + kGemmFinishWarps;
constexpr int kGemmThreads = kGemmWarps * 32;
constexpr int kGemmTmemCols = 512;                          // the accumulator first, then 64 columns of A per stage
constexpr int kGemmSmem = 226 * 1024, kGemmGroupSmem = 220 * 1024;   // dynamic shared memory that a launch may ask for (grouped: beside 4 KB of tables)
constexpr int kGemmMaxCols = 256;                           // accumulator columns (activation rows x planes) per launch
constexpr int kLbo = 128;                                   // bytes between core matrices of B adjacent in K
constexpr int kSboB = 1024;                                 // bytes between its 8-column groups (64 k x 8 columns x 2 bytes)
constexpr unsigned kSleepNs = 100u;                         // between polls of a role that is ahead of the decode warps
constexpr unsigned kSpinLimit = 2000000u;                   // iterations of a try_wait loop before giving up

struct GemmParams {
  const uint32_t* qw;
  const __half* scales;
  const uint8_t* sv;
  const void* bias;
  void* y;
  const __half* xb;       // transformed activations in B tile layout (see rht_f16_kernel): columns 0..np-1 = hi plane of the
                          // activation rows, np..2np-1 = lo plane (planes == 2)
  const float* xsum;      // [np][xsum_slices] sums over k (per slice of the transform) of the planes in use
  const float* tok;       // [np] power-of-two range scale per activation row
  float* part;            // [thread blocks][2][np][128]: flat form, the partial of a thread block's first row block and of a later one
  int* counters;          // [row blocks]
  int* error;             // one word: first failure code seen by any thread block (0 = none)
  int rows, np;           // activation rows present / padded (to 16, or 8 with two planes)
  int planes;
  int mt, nt;
  int m_out;              // rows of the weight that are written (row stride of y, length of bias)
  int dtype;
  int hb;                 // 128-column blocks per row block (n / 128)
  int split;              // > 0: thread blocks per row block (cluster form); 0: flat ranges
  int run_q, run_rem;     // blocks of a thread block's run: run_q, one more for the first run_rem (cluster form: hb / split and the remainder,
                          // parts from block part * hb / split on)
  int part_magic;         // part_reciprocal(split)
  int inbox;              // > 0: offset in shared memory where a thread block of a cluster receives the partial sums of its rows; 0: the
                          // partials stay where they are and are fetched from there (many activation rows)
  int stages;
  int withhold;           // test hook: the B tile of block withhold - 1 of the launch is never fetched (0: none)
  int xsum_slices;
  float cb;
  // Grouped form (GROUP instantiations: the experts of a mixture-of-experts step): the problems are the tiles of a device-side plan
  // (route_plan_kernel in gemm_api.cu), each an expert and up to kGroupRows (token, slot) pairs; row blocks are numbered tile-major,
  // xb holds one B operand per tile, xsum / tok kGroupRows entries per tile, and activation row j of tile t is output row pair(t, j).
  const int* plan;
  int tile_cap;           // tiles the plan has room for
  int rb_per_tile;
  const uint32_t* const* g_qw;
  const __half* const* g_scales;
  const uint8_t* const* g_sv;
  // row-shard form: the output rows go, with plain peer stores, to element offset peer_offset + j * m + row of every buffer in
  // peer_y (the gather buffers of all ranks of an NVLink box as mapped into this process) instead of y
  void* peer_y[8];
  int npeer;
  long long peer_offset;
};

// layout of the plan (ints): tile count, three spare, then per tile the expert, the number of pairs, and kGroupRows pair numbers
constexpr int kGroupRows = 16, kGroupMaxTiles = 512;
__host__ __device__ inline int group_plan_ints(int cap) { return 4 + cap * (2 + kGroupRows); }
__device__ __forceinline__ int group_tiles(const int* plan) { return __ldcg(plan); }
__device__ __forceinline__ int group_expert(const int* plan, int, int t) { return __ldcg(plan + 4 + t); }
__device__ __forceinline__ int group_count(const int* plan, int cap, int t) { return __ldcg(plan + 4 + cap + t); }
__device__ __forceinline__ const int* group_pairs(const int* plan, int cap, int t) { return plan + 4 + 2 * cap + t * kGroupRows; }

__device__ __forceinline__ void gemm_store_rows(const GemmParams& p, int j, int row0, float4 o) {
  if (p.npeer == 0) {
    if (row0 < p.m_out) store_quad(p.y, (size_t)j * p.m_out + row0, p.dtype, o);
  } else {
#pragma unroll 1
    for (int pe = 0; pe < p.npeer; ++pe) store_quad(p.peer_y[pe], (size_t)p.peer_offset + (size_t)j * p.m_out + row0, p.dtype, o);
  }
}

// One lane of the (converged) warp.  The branch on elect.sync tells the compiler that one thread runs it, so the operands of
// tcgen05 and bulk-copy instructions go to uniform registers once; behind `lane == 0` every MMA took 125 cycles to issue, behind
// the election 50 (measured back to back at N = 16..64, A in tensor memory).
__device__ __forceinline__ bool elect_one() {
  uint32_t is;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(is));
  return is != 0;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t umma_desc_b(uint32_t smem_addr) {
  // start address, LBO, SBO in 16-byte units; descriptor version 1 (sm_100); layout type 0 = no swizzle
  return (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)((kLbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((kSboB >> 4) & 0x3FFF) << 32) |
         (1ull << 46);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// CLUSTER: what is waited for was written by other thread blocks of the cluster (the default acquires from this one's threads alone)
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity, unsigned hint_ns) {
  uint32_t done;
  if constexpr (CLUSTER)
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity), "r"(hint_ns)
        : "memory");
  return done != 0;
}
// (a role that waits most of the time sleeps between polls: the issue slots are the decode warps')
template <bool CLUSTER = false>
static __device__ __noinline__ bool mbar_wait_slow(uint32_t bar, uint32_t parity, const volatile int* fail, unsigned sleep_ns) {
  for (unsigned it = 0; it < kSpinLimit; ++it) {
    if (mbar_try<CLUSTER>(bar, parity, 1000u)) return true;
    if ((it & 255u) == 255u && fail && *fail) return false;
    if (sleep_ns) __nanosleep(sleep_ns);
  }
  return false;
}
// bounded wait for the phase with the given parity; false when the limit ran out or another role has already failed
// (`fail` null: no early exit -- used on the failure path to let copies and MMAs in flight drain)
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, const volatile int* fail, unsigned sleep_ns = 0) {
  return mbar_try<CLUSTER>(bar, parity, 1000u) || mbar_wait_slow<CLUSTER>(bar, parity, fail, sleep_ns);
}

// global -> shared bulk copy (16-byte aligned, size a multiple of 16), completion counted in bytes on an mbarrier
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
               "r"(bar)
               : "memory");
}

// D[128 x N] (+)= A[128 x 16 f16, tensor memory] * B[N x 16 f16, shared memory]
__device__ __forceinline__ void umma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
      "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// 16 lanes x 32 columns of tensor memory from one warp: registers 4j, 4j+1 of lane (g, c) = columns 8j + 2c, +1 of row g,
// registers 4j+2, 4j+3 the same of row g + 8
__device__ __forceinline__ void tmem_store_strip(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
               "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
               "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
               : "memory");
}

// one float to the same place in the shared memory of thread block `rank` of the cluster, counted in bytes on its mbarrier
__device__ __forceinline__ void send_partial(uint32_t at, uint32_t bar, int rank, float v) {
  asm volatile(
      "{\n\t.reg .b32 a, b;\n\tmapa.shared::cluster.u32 a, %0, %2;\n\tmapa.shared::cluster.u32 b, %1, %2;\n\t"
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [a], %3, [b];\n\t}" ::"r"(at),
      "r"(bar), "r"(rank), "f"(v)
      : "memory");
}

// 8 consecutive accumulator columns of this thread's tensor-memory lane (complete after tcgen05.wait::ld)
__device__ __forceinline__ void tmem_load8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// dynamic shared memory: the B ring (the cluster form reuses it for the [np][128] float partial of the thread block), then the
// packed-word rings of the decode warps (`words` bytes)
__host__ __device__ constexpr int gemm_stage_bytes(int ncols) { return ncols * 256; }
__host__ __device__ constexpr int gemm_ring_bytes(int np, int planes, int stages) {
  const int ring = stages * gemm_stage_bytes(np * planes), result = np * 128 * 4;
  return ring > result ? ring : result;
}
__host__ __device__ constexpr int gemm_smem_bytes(int np, int planes, int stages, int words) { return gemm_ring_bytes(np, planes, stages) + words + 128; }
__host__ __device__ inline int gemm_acc_cols(int ncols) { return ncols < 32 ? 32 : ncols; }

// ---- packed-word ring of a decode warp: one slot = the tiles of its strip in one 128-column block (two units of four tiles).
// A lane reads the words of row pair g of tile c; for K a multiple of 4 the 16-byte chunks of a tile are stored in an order that
// spreads the eight lanes of a read phase (two g, four c) over all banks.
template <int K>
struct GemmRing {
  static constexpr int slot_bytes = 256 * K;
  static constexpr int slots = K <= 3 ? 6 : K <= 5 ? 4 : 3;  // 40 to 64 KB in flight per SM
  static constexpr int bytes = kGemmDecodeWarps * slots * slot_bytes;
  static constexpr int chunks = slot_bytes / 16, copies = (chunks + 31) / 32;
};
// position (in 16-byte chunks, inside the four tiles of a unit) of chunk ch of tile c
template <int K>
__device__ __forceinline__ int ring_chunk(int c, int ch) {
  if constexpr (K == 4) return c * 8 + (ch ^ (2 * c));
  else if constexpr (K == 8) return c * 16 + (ch ^ ((c & 1) | ((c & 2) << 1)));
  else return c * 2 * K + ch;
}
template <int K>
__device__ __forceinline__ void read_own_words(const unsigned char* unit, int c, int g, uint32_t (&V)[K]) {
  if constexpr (K % 4 == 0) {
#pragma unroll
    for (int i = 0; i < K / 4; ++i) {
      const uint4 t = *reinterpret_cast<const uint4*>(unit + 16 * ring_chunk<K>(c, (K / 4) * g + i));
      V[4 * i] = t.x; V[4 * i + 1] = t.y; V[4 * i + 2] = t.z; V[4 * i + 3] = t.w;
    }
  } else if constexpr (K % 2 == 0) {
#pragma unroll
    for (int i = 0; i < K / 2; ++i) {
      const uint2 t = *reinterpret_cast<const uint2*>(unit + c * (32 * K) + g * (4 * K) + 8 * i);
      V[2 * i] = t.x; V[2 * i + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int i = 0; i < K; ++i) V[i] = *reinterpret_cast<const uint32_t*>(unit + c * (32 * K) + g * (4 * K) + 4 * i);
  }
}

// 32 codebook integers of a lane unit as fp16 pairs (1024 + bytesum), in the register order of tmem_store_strip
template <int K>
__device__ __forceinline__ void decode_unit(const uint32_t (&own)[K], int lane, uint32_t (&out)[16]) {
  uint32_t V[K + 1], s[32];
#pragma unroll
  for (int i = 0; i < K; ++i) V[i + 1] = own[i];
  V[0] = __shfl_sync(kFullWarp, own[K - 1], (lane - 4) & 31);          // last word of the row pair before, circularly inside the tile
  unit_states<K>(V, s);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int rr = 0; rr < 2; ++rr)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = rr * 16 + 4 * j + 2 * h;
        const uint32_t lo = bytesum_add(s[t] * kGenMul + kGenAdd, 0x6400u), hi = bytesum_add(s[t + 1] * kGenMul + kGenAdd, 0x6400u);
        // the pack goes to whichever pipe the width leaves free: shift/logic (PRMT) or multiply (IMAD)
        const bool alu = PairStride<K>::value > 1 || h == 0;
        out[4 * j + 2 * rr + h] = alu ? __byte_perm(lo, hi, 0x5410) : hi * 65536u + lo;
      }
}

// barrier of the finisher warps; true where every thread brought true
__device__ __forceinline__ bool finishers_all(bool mine) {
  int all;
  __syncwarp();
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbar.red.and.pred p, 1, %2, q;\n\tselp.s32 %0, 1, 0, p;\n\t}"
               : "=r"(all)
               : "r"((int)mine), "n"(kGemmFinishWarps * 32)
               : "memory");
  return all != 0;
}

// ---- finishing of a row block: one warp per activation row, lane holds rows 4 lane .. + 3 of the block
struct GemmTail {
  float s[4];                                               // row scales times the codebook's
  unsigned sv_bits;
  float4 bias;
  int row0;                                                 // row of this problem's weight
  int rows;                                                 // activation rows
  int base;                                                 // of its entries of xsum and tok
  const int* pairs;                                         // grouped form: output row of every activation row
  template <bool GROUP>
  __device__ __forceinline__ void load(const GemmParams& p, int rb, int lane) {
    const __half* scales = p.scales;
    const uint8_t* sv = p.sv;
    rows = p.rows;
    base = 0;
    pairs = nullptr;
    if constexpr (GROUP) {
      const int t = rb / p.rb_per_tile, e = group_expert(p.plan, p.tile_cap, t);
      rb -= t * p.rb_per_tile;
      scales = p.g_scales[e];
      sv = p.g_sv[e];
      rows = group_count(p.plan, p.tile_cap, t);
      base = t * kGroupRows;
      pairs = group_pairs(p.plan, p.tile_cap, t);
    }
    row0 = rb * 128 + 4 * lane;
    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(scales + row0));
    const float2 s01 = __half22float2(*reinterpret_cast<const __half2*>(&raw.x)), s23 = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
    s[0] = s01.x * p.cb; s[1] = s01.y * p.cb; s[2] = s23.x * p.cb; s[3] = s23.y * p.cb;
    sv_bits = sign_nibble(sv, rb * 32 + lane);
    bias = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.bias && row0 < p.m_out) bias = load_quad(p.bias, row0, p.dtype);
  }
};
// this lane's share of the row sum of the activations; the warp adds the shares (a fixed tree: results do not depend on scheduling)
__device__ __forceinline__ float gemm_xsum_share(const GemmParams& p, int j, int lane) {
  float xs = 0.f;
  for (int y = lane; y < p.xsum_slices; y += 32) xs += __ldcg(p.xsum + (size_t)j * p.xsum_slices + y);
  return xs;
}
__device__ __forceinline__ float gemm_xsum_total(float xs) {
#pragma unroll
  for (int o = 16; o; o >>= 1) xs += __shfl_xor_sync(kFullWarp, xs, o);
  return xs;
}
// xs: the whole row sum of the activations
__device__ __forceinline__ void gemm_finish_row(const GemmParams& p, const GemmTail& t, int j, int lane, float4 r4, float xs, float tok) {
  const float off = 1534.0f * xs, out = kInvSqrt128 * tok;  // (the range scale last: a row scale times a small tok could underflow)
  float v[4] = {(r4.x - off) * t.s[0], (r4.y - off) * t.s[1], (r4.z - off) * t.s[2], (r4.w - off) * t.s[3]};
  wht128(v, lane);
  gemm_store_rows(p, t.pairs ? __ldcg(t.pairs + j) : j, t.row0,
                  make_float4(flip(v[0] * out, t.sv_bits & 1u) + t.bias.x, flip(v[1] * out, (t.sv_bits >> 1) & 1u) + t.bias.y,
                              flip(v[2] * out, (t.sv_bits >> 2) & 1u) + t.bias.z, flip(v[3] * out, t.sv_bits >> 3) + t.bias.w));
}

// rows j0, j0 + step, ... of row block rb from the partial sums of thread blocks first .. first + contributors - 1, added in that
// order.  Two rows at a time: the loads of both are in flight together.  head: which partial of thread block `first`.
template <bool GROUP>
__device__ __forceinline__ void gemm_finish_flat(const GemmParams& p, int rb, int first, int contributors, int head, int j0, int step, int lane) {
  GemmTail tail;
  tail.load<GROUP>(p, rb, lane);
  const float4* slot0 = reinterpret_cast<const float4*>(p.part + (size_t)(2 * first) * ((size_t)p.np * 128)) + lane;
  const size_t stride = (size_t)p.np * 32;
  for (int j = j0; j < tail.rows; j += 2 * step) {
    const int jb = j + step < tail.rows ? j + step : j;
    const float xa = gemm_xsum_share(p, tail.base + j, lane), xb = gemm_xsum_share(p, tail.base + jb, lane);
    const float ta = __ldcg(p.tok + tail.base + j), tb = __ldcg(p.tok + tail.base + jb);
    float4 ra = make_float4(0.f, 0.f, 0.f, 0.f), rb4 = ra;
    for (int base = 0; base < contributors; base += 4) {
      float4 va[4], vb[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = base + q;
        const float4* src = slot0 + (size_t)(i == 0 ? head : 2 * i) * stride;
        va[q] = i < contributors ? __ldcg(src + j * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
        vb[q] = i < contributors ? __ldcg(src + jb * 32) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        ra.x += va[q].x; ra.y += va[q].y; ra.z += va[q].z; ra.w += va[q].w;
        rb4.x += vb[q].x; rb4.y += vb[q].y; rb4.z += vb[q].z; rb4.w += vb[q].w;
      }
    }
    gemm_finish_row(p, tail, j, lane, ra, gemm_xsum_total(xa), ta);
    if (jb != j) gemm_finish_row(p, tail, jb, lane, rb4, gemm_xsum_total(xb), tb);
  }
}

template <int K, bool GROUP>
__global__ void __launch_bounds__(kGemmThreads, 1) packed_gemm_tc_kernel(const GemmParams p) {
  extern __shared__ __align__(128) unsigned char gsm[];
  __shared__ __align__(8) unsigned long long s_full[kGemmMaxStages], s_freed[kGemmMaxStages], s_done, s_drained, s_inbox, s_nobody;
  __shared__ uint32_t s_tmem;
  __shared__ int s_arrival;
  __shared__ int s_owed[kGemmFinishWarps];                  // row blocks below it have been delivered by the finisher warp
  __shared__ volatile int s_fail;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  constexpr int DW = kGemmDecodeWarps;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int np = p.np, ncols = p.planes * np;               // accumulator columns: hi plane, then lo plane if present
  const int nt = p.nt, HB = p.hb, NS = p.stages;
  int tiles = 1;
  if constexpr (GROUP) tiles = group_tiles(p.plan);         // (complete: the transform before this launch lets it start only then)
  const int U = (GROUP ? tiles * p.rb_per_tile : p.mt >> 3) * HB;
  EvenRuns runs(p.run_q, p.run_rem, 0);
  if constexpr (GROUP) runs = EvenRuns(U, gridDim.x);
  // first row block and first block in it of the run (cluster form: its only row block; divisions cost a start of cold instructions)
  int rb0, hb0, part_id = 0, part = 0, u_begin, u_end;
  if (!GROUP && p.split > 0) {
    rb0 = blockIdx.x;
    if (p.split > 1) {
      asm("mov.u32 %0, %%clusterid.x;" : "=r"(rb0));
      asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(part_id));
    }
    // The last part is always one of the longer ones: it goes to the first thread block of the cluster, which starts first (2944x1664 K6, 37
    // rows: 8.3 -> 8.0 us)
    part = p.split - 1 - part_id;
    hb0 = part_begin(part, p.run_q, p.run_rem, p.part_magic);
    u_begin = rb0 * HB + hb0;
    u_end = rb0 * HB + part_begin(part + 1, p.run_q, p.run_rem, p.part_magic);
  } else {
    u_begin = runs.begin(blockIdx.x);
    u_end = runs.begin(blockIdx.x + 1);
    rb0 = u_begin / HB;
    hb0 = u_begin - rb0 * HB;
  }
  if (GROUP && u_begin == u_end) {                          // fewer blocks than thread blocks (an empty plan among others)
    // not before the transform has: with an empty plan the grid would be over, and what comes behind it free to write, while that still reads
    asm volatile("griddepcontrol.wait;" ::: "memory");
    return;
  }
  const int b_tile_bytes = ncols * 256;
  unsigned char* ring = gsm + (128 - (smem_u32(gsm) & 127)) % 128;
  const uint32_t ring_addr = smem_u32(ring);
  const int a_col = gemm_acc_cols(ncols);

  if (warp == kGemmWarps - 2) {                             // (not a warp whose first words are on the way)
    if (lane < kGemmMaxStages) {
      mbar_init(smem_u32(&s_full[lane]), kGemmGroupWarps + 1);          // the warps of the group that decodes the block, and the B
                                                                        // lane's arrive.expect_tx (with the bytes of the tile)
      mbar_init(smem_u32(&s_freed[lane]), 1);                           // tcgen05.commit
    }
    if (lane == 0) {
      mbar_init(smem_u32(&s_done), 1);                                  // tcgen05.commit: the MMAs of a row block have retired
      mbar_init(smem_u32(&s_drained), kGemmFinishWarps);                // one arrival per finisher warp: its accumulator has been read
      if (GROUP) mbar_init(smem_u32(&s_nobody), DW);                    // before the first block of a warp
      mbar_init(smem_u32(&s_inbox), 1);                                 // the partial sums of this thread block's rows, from the whole cluster
      s_fail = 0;
      for (int i = 0; i < kGemmFinishWarps; ++i) s_owed[i] = rb0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    if (!GROUP && p.inbox > 0 && lane == 0) mbar_expect_tx(smem_u32(&s_inbox), (uint32_t)(p.split * ((p.rows - part_id + p.split - 1) / p.split) * 512));
  }
  if (!GROUP && p.inbox > 0) cluster_arrive();   // (waited for before the first partial is sent)
  if (warp == DW + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"((uint32_t)kGemmTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __shared__ const uint32_t* s_qw[GROUP ? kGroupMaxTiles : 1];   // packed words of every tile's expert
  if constexpr (GROUP) {
    for (int t = tid; t < tiles; t += kGemmThreads) s_qw[t] = p.g_qw[group_expert(p.plan, p.tile_cap, t)];
    __syncthreads();
  }
  if (!GROUP && warp == kGemmWarps - 1 && lane < 6) {
    // the row scales and signs of the first and the last row block are needed at the very end, in a chain of dependent loads:
    // bring them to L2 now (256 bytes of scales and 16 of signs per row block)
    const size_t rb = lane & 1 ? (u_end - 1) / HB : rb0;
    const char* at = lane < 4 ? reinterpret_cast<const char*>(p.scales + rb * 128) + (lane >> 1) * 128 : reinterpret_cast<const char*>(p.sv + rb * 16);
    asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
  }

  // cluster form: what a decode warp needs to finish its rows j0, j0 + split * DW, ... (at most sixteen) of the one row block
  GemmTail tail;
  float xs_of = 0.f, tok_of = 0.f;                          // lane i: activation sum and scale of the i-th of these rows
  if (warp < DW) {
    // ================= decode warps
    const int quad = warp & 3, half = (warp >> 2) & 1, strip = 2 * quad + half, group = warp >> 3;
    const int g = lane >> 2, c = lane & 3;
    using Ring = GemmRing<K>;
    constexpr int R = Ring::slots;
    const unsigned char* words = ring + gemm_ring_bytes(np, p.planes, NS) + warp * (R * Ring::slot_bytes);
    // copy cursor: every second block of the run, across row blocks; past the end of the run the copies are predicated off
    uint32_t cp_dst[Ring::copies];
#pragma unroll
    for (int i = 0; i < Ring::copies; ++i) {
      const int ch = lane + 32 * i, unit = ch / (8 * K), within = ch % (8 * K);
      cp_dst[i] = smem_u32(words) + unit * (128 * K) + 16 * ring_chunk<K>(within / (2 * K), within % (2 * K));
    }
    // from the end of a strip's row to the same strip of the next row block (a row of one block is left twice per step of two)
    const size_t next_strip = (size_t)7 * nt * (32 * K) * (HB == 1 ? 2 : 1);
    int pf_left = u_end - u_begin - group, pf_in_rb, pf_rb;
    const char* pf;
    auto strip_row = [&](int rb) {                          // this lane's first chunk of this warp's strip of row block rb
      const uint32_t* base = p.qw;
      if constexpr (GROUP) {
        const int t = min(rb / p.rb_per_tile, tiles - 1);    // (past the last tile nothing is copied any more)
        rb -= t * p.rb_per_tile;
        base = s_qw[t];
      }
      return reinterpret_cast<const char*>(base) + (size_t)(rb * 8 + strip) * nt * (32 * K) + lane * 16;
    };
    {
      int hb = hb0 + group;
      pf_rb = rb0;
      while (hb >= HB) { hb -= HB; ++pf_rb; }
      pf = strip_row(pf_rb) + (size_t)hb * (256 * K);
      pf_in_rb = HB - hb;
    }
    auto fetch = [&](uint32_t at) {
#pragma unroll
      for (int i = 0; i < Ring::copies; ++i) {
        const int on = (32 * i + 32 <= Ring::chunks || lane + 32 * i < Ring::chunks) ? pf_left : 0;
        asm volatile("{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %2, 0;\n\t@p cp.async.cg.shared.global [%0], [%1], 16;\n\t}" ::"r"(cp_dst[i] + at),
                     "l"(pf + 512 * i), "r"(on)
                     : "memory");
      }
      pf_left -= 2;
      if constexpr (GROUP) {
        pf += 512 * K;
        pf_in_rb -= 2;
        if (pf_in_rb <= 0) {
          while (pf_in_rb <= 0) { pf_in_rb += HB; ++pf_rb; }
          pf = strip_row(pf_rb) + (size_t)(HB - pf_in_rb) * (256 * K);
        }
      } else {
        const bool wrap = pf_in_rb <= 2;
        pf_in_rb += wrap ? HB - 2 : -2;
        pf += wrap ? next_strip + 512 * K : (size_t)(512 * K);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int i = 0; i < R - 1; ++i) fetch(i * Ring::slot_bytes);   // the weights do not depend on the preceding kernel
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();                                        // the barriers and the tensor-memory address are visible from here on
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t a_addr = s_tmem + ((uint32_t)(32 * quad + 16 * half) << 16) + (uint32_t)a_col;
    // (this loop is what bounds the kernel: no branches but the two below, no divisions, no counters beside the ring positions)
    uint32_t at = 0u, refill = (R - 1) * Ring::slot_bytes;  // ring slots of this block and of the one before it
    int stage = group;
    uint32_t parity = 1u;                                   // of freed[stage]: passes at once on the first round
    // A stage is told of when its stores have landed: behind the second one, or (experts) half a block later, while the next block is decoded.
    // The wait leaves issue slots empty, but the MMAs lose half a block at every boundary of row blocks: us, at once / later, 16 tokens
    // on 64 experts 272 / 268, 4096x12288 K3 4 rows 16.6 / 16.2, but 12288x4096 K2 64 rows 22.9 / 23.2, 151936x4096 K4 8 rows 127.3 / 127.9
    // (and choosing at run time costs 2 % by itself).
    uint32_t stored = GROUP ? smem_u32(&s_nobody) : 0u;     // full[] of the stage stored last
    auto deliver = [&](uint32_t to) {
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(to);
    };
    bool ok = true;
#pragma unroll 1
    for (int left = u_end - u_begin - group; left > 0; left -= 2) {
      asm volatile("cp.async.wait_group %0;" ::"n"(R - 2) : "memory");   // this block's words have landed (own copies) ...
      __syncwarp();                                                       // ... and those of the other lanes; the slot before it is free
      fetch(refill);
      const unsigned char* blk = words + at;
      refill = at;
      at = at == (R - 1) * Ring::slot_bytes ? 0u : at + Ring::slot_bytes;
      uint32_t V[K], w[16];
      read_own_words<K>(blk, c, g, V);
      decode_unit<K>(V, lane, w);
      if constexpr (GROUP) deliver(stored);
      // the MMAs that read this stage NS blocks ago must have retired
      const uint32_t bar = smem_u32(&s_freed[0]) + 8u * stage;
      if (!__all_sync(kFullWarp, mbar_try(bar, parity, 1000u)) && !__all_sync(kFullWarp, mbar_wait_slow(bar, parity, &s_fail, 0u))) {
        s_fail = 1;                                          // (before anything else that the MMA lane could take for progress)
        ok = false;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      tmem_store_strip(a_addr + 64 * stage, w);
      read_own_words<K>(blk + 128 * K, c, g, V);
      decode_unit<K>(V, lane, w);
      tmem_store_strip(a_addr + 64 * stage + 32, w);
      if constexpr (GROUP) stored = smem_u32(&s_full[0]) + 8u * stage;
      else deliver(smem_u32(&s_full[0]) + 8u * stage);
      const bool around = stage + 2 >= NS;
      stage += around ? 2 - NS : 2;
      parity ^= around ? 1u : 0u;
    }
    if constexpr (GROUP)
      if (ok) deliver(stored);                               // (a warp that gave up has told of all it stored: another arrival counts for the next round)
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (!GROUP && p.split > 0) {
      // these loads, and the wait for the transform that they need, lie beside the last MMAs; then the accumulator goes to the ring as
      // the thread block's partial [np][128], hi + lo added: four warps of a quadrant take alternate groups of 8 columns
      asm volatile("griddepcontrol.wait;" ::: "memory");
      tail.load<false>(p, rb0, lane);
      const int j = part_id + p.split * (warp + lane * DW);
      if (j < p.rows) {
        float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
        for (int y = 0; y < p.xsum_slices; y += 4)
#pragma unroll
          for (int q = 0; q < 4; ++q) part[q] += y + q < p.xsum_slices ? __ldcg(p.xsum + (size_t)j * p.xsum_slices + y + q) : 0.f;
        xs_of = (part[0] + part[2]) + (part[1] + part[3]);
        tok_of = __ldcg(p.tok + j);
      }
      ok = ok && __all_sync(kFullWarp, mbar_wait(smem_u32(&s_done), 0u, &s_fail));
      ok = __all_sync(kFullWarp, ok && !s_fail);             // (an MMA lane that gave up says so before it commits what it had issued)
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int li = lane & 15, row = 32 * quad + (lane & 16) + (li < 8 ? 2 * li : 2 * li - 15);   // weight row of this tensor-memory lane
      const uint32_t acc_addr = s_tmem + ((uint32_t)(32 * quad) << 16);
      if (p.inbox > 0) {
        const uint32_t inbox = smem_u32(ring) + (uint32_t)p.inbox, own_rows = (np + p.split - 1) / p.split;
        cluster_wait();   // every thread block's inbox is ready
        for (int j0 = 8 * (warp >> 2); j0 < np; j0 += 2 * DW) {
          uint32_t hi[8], lo[8];
          if (ok) {
            tmem_load8(acc_addr + j0, hi);
            if (p.planes == 2) tmem_load8(acc_addr + np + j0, lo);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          }
          int index = j0 / p.split, owner = j0 - index * p.split;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float v = p.planes == 2 ? __uint_as_float(hi[i]) + __uint_as_float(lo[i]) : __uint_as_float(hi[i]);
            if (!ok) v = __uint_as_float(0x7FC00000u);       // a bounded wait gave up: NaN, so that the row carries it whoever finishes it
            if (j0 + i < p.rows) send_partial(inbox + ((part * own_rows + index) * 128 + row) * 4, smem_u32(&s_inbox), owner, v);
            if (++owner == p.split) { owner = 0; ++index; }
          }
        }
      } else if (ok) {
        float* mine = reinterpret_cast<float*>(ring);
        for (int j0 = 8 * (warp >> 2); j0 < np; j0 += 2 * DW) {
          uint32_t hi[8], lo[8];
          tmem_load8(acc_addr + j0, hi);
          if (p.planes == 2) tmem_load8(acc_addr + np + j0, lo);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int i = 0; i < 8; ++i) mine[(j0 + i) * 128 + row] = p.planes == 2 ? __uint_as_float(hi[i]) + __uint_as_float(lo[i]) : __uint_as_float(hi[i]);
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (!ok) s_fail = 1;
  } else {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == DW) {
      // ================= B lane: one bulk copy per 128-column block (the activation transform wrote the tiles contiguously)
      if (elect_one()) {
        asm volatile("griddepcontrol.wait;" ::: "memory");  // the transformed activations come from the preceding kernel
        int s = 0, issued = 0, hb = hb0;
        int rb_left = GROUP ? p.rb_per_tile - rb0 % p.rb_per_tile : 0;   // row blocks of this tile still to come, this one included
        const char* xb = reinterpret_cast<const char*>(p.xb);
        if constexpr (GROUP) xb += (size_t)(rb0 / p.rb_per_tile) * HB * b_tile_bytes;
        uint32_t use = 0u;
        for (int u = u_begin; u < u_end; ++u) {
          if (use > 0 && !mbar_wait(smem_u32(&s_freed[s]), (use - 1u) & 1u, &s_fail, kSleepNs)) { s_fail = 1; break; }
          const uint32_t bar = smem_u32(&s_full[s]);
          if (u + 1 != p.withhold) {
            mbar_expect_tx(bar, (uint32_t)b_tile_bytes);
            bulk_load(ring_addr + s * b_tile_bytes, xb + (size_t)hb * b_tile_bytes, (uint32_t)b_tile_bytes, bar);
            ++issued;
          }
          if (++hb == HB) {
            hb = 0;
            if (GROUP && --rb_left == 0) {
              rb_left = p.rb_per_tile;
              xb += (size_t)HB * b_tile_bytes;
            }
          }
          if (++s == NS) { s = 0; ++use; }
        }
        if (s_fail) {
          // copies still in flight write into this thread block's shared memory, and the decode warps' arrivals may never come to
          // complete their barriers: give the copies far longer than a copy takes
          if (issued) __nanosleep(1000000u);
        }
      }
    } else if (warp == DW + 1) {
      // ================= MMA lane
      if (elect_one()) {
        const uint32_t tmem = s_tmem;
        // instruction descriptor: D = f32, A = B = f16, both K-major, M = 128, N = ncols
        const uint32_t idesc = (1u << 4) | ((uint32_t)(ncols >> 3) << 17) | ((128u >> 4) << 24);
        const uint64_t desc0 = umma_desc_b(ring_addr);
        int s = 0, seg = 0;
        uint32_t ph = 0u;
        bool ok = true;
        for (int u = u_begin; u < u_end && ok; ++seg) {
          const int stop = min(u_end, (rb0 + seg + 1) * HB);
          if (seg > 0 && !mbar_wait(smem_u32(&s_drained), (uint32_t)(seg - 1) & 1u, &s_fail)) { ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          uint32_t fresh = 0u;                               // 0: the first MMA of a row block overwrites the accumulator
          for (; u < stop; ++u) {
            if (!mbar_wait(smem_u32(&s_full[s]), ph, &s_fail)) { ok = false; break; }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t desc = desc0 + (uint64_t)(s * (b_tile_bytes >> 4));   // (shared memory addresses fit the field: no carry)
            const uint32_t a_addr = tmem + (uint32_t)(a_col + 64 * s);
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
              for (int j = 0; j < 4; ++j)
                umma_f16_ts(tmem, a_addr + 32 * q + 8 * j, desc + (uint64_t)(q * (b_tile_bytes >> 5) + j * ((2 * kLbo) >> 4)), idesc, (q | j) ? 1u : fresh);
            fresh = 1u;
            umma_commit(smem_u32(&s_freed[s]));
            if (++s == NS) { s = 0; ph ^= 1u; }
          }
          if (!ok) break;
          umma_commit(smem_u32(&s_done));                    // covers every MMA issued so far
        }
        if (!ok) {
          s_fail = 1;                                        // the other threads stop waiting at once ...
          __threadfence_block();
          umma_commit(smem_u32(&s_done));
          mbar_wait(smem_u32(&s_done), (uint32_t)seg & 1u, nullptr);   // ... this one lets the MMAs in flight retire first
        }
      }
    } else if (GROUP || p.split == 0) {
      // ================= finishers (cluster form: the decode warps do that)
      const int fw = warp - (DW + 2), quad = warp & 3;
      const uint32_t acc_addr = s_tmem + ((uint32_t)(32 * quad) << 16);
      const int li = lane & 15, row = 32 * quad + (lane & 16) + (li < 8 ? 2 * li : 2 * li - 15);   // weight row of this tensor-memory lane
      bool ok = true, predecessor_done = false;
      int seg = 0;
      for (int u = u_begin; u < u_end; ++seg) {
        const int rb = rb0 + seg, stop = (rb + 1) * HB;
        ok = __all_sync(kFullWarp, mbar_wait(smem_u32(&s_done), (uint32_t)seg & 1u, &s_fail, kSleepNs));
        if (s_fail) ok = false;
        if (!ok) s_fail = 1;
        // all finishers go on together or none does (they meet in barriers below)
        if (!finishers_all(ok)) { ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!predecessor_done) {
          asm volatile("griddepcontrol.wait;" ::: "memory");   // scratch and outputs of earlier launches
          predecessor_done = true;
        }
        // accumulator -> partial [np][128], hi + lo added here.  A thread block has two partials: its first row block's, which other
        // thread blocks may read, and one for all later ones (of which only the last is read by others)
        float* mine = p.part + (size_t)(2 * blockIdx.x + (seg > 0 ? 1 : 0)) * ((size_t)np * 128);
        for (int j0 = 0; j0 < np; j0 += 8) {
          uint32_t hi[8], lo[8];
          tmem_load8(acc_addr + j0, hi);
          if (p.planes == 2) tmem_load8(acc_addr + np + j0, lo);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float v = p.planes == 2 ? __uint_as_float(hi[j]) + __uint_as_float(lo[j]) : __uint_as_float(hi[j]);
            __stcg(mine + (j0 + j) * 128 + row, v);
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&s_drained));    // the MMAs of the next row block may start
        if (stop >= u_end) break;                            // the last row block: all warps finish it, below
        // only the run's first row block can have other contributors here, thread blocks before this one
        const int first = runs.owner(rb * HB), contributors = blockIdx.x - first + 1;
        bool finish = true;
        finishers_all(true);
        if (contributors > 1) {
          if (fw == 0 && lane == 0) {
            __threadfence();                                 // the partials of the whole thread block (ordered by the barrier) before the arrival
            s_arrival = atomicAdd(p.counters + rb, 1);       // (they are read with loads served by L2, after this atomic)
          }
          finishers_all(true);
          finish = s_arrival == contributors - 1;
          if (finish && fw == 0 && lane == 0) p.counters[rb] = 0;
        }
        if (finish) gemm_finish_flat<GROUP>(p, rb, first, contributors, runs.begin(first) < rb * HB ? 1 : 0, fw, kGemmFinishWarps, lane);
        __syncwarp();
        if (lane == 0) s_owed[fw] = rb + 1;
        finishers_all(true);                                 // the partial has been read by all of them: it may be written again
        u = stop;
      }
      if (!ok) s_fail = 1;
    }
    __syncwarp();
    if (!GROUP && p.inbox > 0) cluster_wait();   // (its arrival; complete long ago)
  }
  if (!GROUP && p.inbox > 0) {
    // ---- reduction inside the cluster: every thread block has sent its partials of row j to thread block j % split, which adds them in the
    // order of the parts and finishes the row.  (Partials fetched from where they were made wait for a barrier of the cluster before and one
    // after, so that nobody leaves too early, 1.5 us together.)
    if (warp < DW) {
      // A peer whose own wait gave up still sends, but up to two of its limits later, and into shared memory that must not be gone by then.
      bool here = mbar_wait<true>(smem_u32(&s_inbox), 0u, nullptr);
      for (int limit = 0; limit < 3 && !here; ++limit) here = mbar_wait<true>(smem_u32(&s_inbox), 0u, nullptr);
      here = __all_sync(kFullWarp, here);
      const int own_rows = (np + p.split - 1) / p.split, row_first = part_id + p.split * warp;
      const float4* in = reinterpret_cast<const float4*>(ring + p.inbox) + lane;
      for (int i = 0; row_first + i * (p.split * DW) < p.rows; ++i) {
        float4 r4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int r = 0; r < p.split; ++r) {
          const float4 v = in[(r * own_rows + warp + i * DW) * 32];
          r4.x += v.x; r4.y += v.y; r4.z += v.z; r4.w += v.w;
        }
        if (!here) r4.x = r4.y = r4.z = r4.w = __uint_as_float(0x7FC00000u);
        gemm_finish_row(p, tail, row_first + i * (p.split * DW), lane, r4, __shfl_sync(kFullWarp, xs_of, i), __shfl_sync(kFullWarp, tok_of, i));
      }
      if (!here) s_fail = 1;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && s_fail) atomicCAS(p.error, 0, 1);
    if (warp == DW + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"((uint32_t)kGemmTmemCols) : "memory");
    return;
  }
  __syncthreads();
  const bool bad = s_fail != 0;
  if (bad && tid == 0) atomicCAS(p.error, 0, 1);

  if (!GROUP && p.split > 0) {
    // ---- split reduction inside the cluster: every thread block keeps its partial [np][128] where it is; thread block r of the
    // cluster sums rows r, r + split, ... over all of them (in the order of the parts) and finishes those rows itself
    float* result = reinterpret_cast<float*>(ring);
    if (bad)                                                 // a bounded wait gave up: the rows come out as NaN, beside the error word
      for (int e = tid; e < np * 128; e += kGemmThreads) result[e] = __uint_as_float(0x7FC00000u);
    if (p.split > 1) {
      cluster_sync();
    } else if (bad) {
      __syncthreads();
    }
    if (warp < DW) {
      const uint32_t result_addr = smem_u32(result) + (uint32_t)lane * 16u;
      const int row_first = part_id + p.split * warp;
      for (int i = 0; row_first + i * (p.split * DW) < p.rows; ++i) {
        const int j = row_first + i * (p.split * DW);
        float4 r4 = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < p.split; ++r) {
          uint32_t remote;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(result_addr + (uint32_t)j * 512u), "r"(p.split - 1 - r));
          float4 v;
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(remote) : "memory");
          r4.x += v.x; r4.y += v.y; r4.z += v.z; r4.w += v.w;
        }
        gemm_finish_row(p, tail, j, lane, r4, __shfl_sync(kFullWarp, xs_of, i), __shfl_sync(kFullWarp, tok_of, i));
      }
    }
    if (p.split > 1) {                                       // nobody leaves while its shared memory may still be read
      cluster_sync();
    }
  } else {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const int rb = (u_end - 1) / HB;
    bool finish = !bad;
    const int first = runs.owner(rb * HB), contributors = runs.owner((rb + 1) * HB - 1) - first + 1;
    if (!bad && contributors > 1) {
      if (tid == 0) {
        __threadfence();                                    // the partials of the whole thread block (ordered by the barrier above) before the arrival
        s_arrival = atomicAdd(p.counters + rb, 1);
      }
      __syncthreads();
      finish = s_arrival == contributors - 1;
      if (finish && tid == 0) p.counters[rb] = 0;
    }
    if (finish) gemm_finish_flat<GROUP>(p, rb, first, contributors, runs.begin(first) < rb * HB ? 1 : 0, warp, kGemmWarps, lane);
    if (bad) {
      // the row blocks this thread block still owed never complete (nobody arrives for them): their rows come out as NaN
      const float nan = __uint_as_float(0x7FC00000u);
      for (int b = min(min(s_owed[0], s_owed[1]), min(s_owed[2], s_owed[3])); b <= rb; ++b) {
        GemmTail tail;
        tail.load<GROUP>(p, b, lane);
        for (int j = warp; j < tail.rows; j += kGemmWarps) gemm_store_rows(p, tail.pairs ? tail.pairs[j] : j, tail.row0, make_float4(nan, nan, nan, nan));
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == DW + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(s_tmem), "r"((uint32_t)kGemmTmemCols) : "memory");
}

template <int K>
int launch_packed_gemm_tc(const GemmParams& p, int grid, int smem, cudaStream_t st);   // p.plan set: the grouped form
// clusters of `split` thread blocks that the GPU holds at once (0: none), for the cluster form of the plan
template <int K>
int packed_gemm_tc_clusters(int smem, int split);
// bytes of the packed-word rings of a thread block
inline int gemm_word_bytes(int K) {
  switch (K) {
    case 2: return GemmRing<2>::bytes;
    case 3: return GemmRing<3>::bytes;
    case 4: return GemmRing<4>::bytes;
    case 5: return GemmRing<5>::bytes;
    case 6: return GemmRing<6>::bytes;
    default: return GemmRing<8>::bytes;
  }
}

}  // namespace htr
