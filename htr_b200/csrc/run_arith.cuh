// Which part of the work a thread block has, and quotients without divisions for it: an integer division is dozens of cold instructions
// (64 bits: a subroutine) at the start of every thread block and between its last sum and its partial.  Everything here also compiles as
// host code (tests/host_runs_check.cpp compares it with exact division).
#pragma once
#include <cstdint>

#include "htr_codec.cuh"

namespace htr {

// Quotients come as the upper product with ceil(2^32 / divisor), exact while dividend times divisor stays below 2^32 (0 stands for the
// divisor 1), or from a float32 guess that is then corrected.
inline unsigned reciprocal(int divisor) { return divisor > 1 ? (unsigned)((0x100000000ull + divisor - 1) / divisor) : 0u; }
HTR_HD int quotient(int x, unsigned magic) {
#if defined(__CUDA_ARCH__)
  return magic ? (int)__umulhi((unsigned)x, magic) : x;
#else
  return magic ? (int)(((uint64_t)(unsigned)x * magic) >> 32) : x;
#endif
}
HTR_HD int quotient(int x, int divisor, float per_divisor) {
  int q = (int)((float)x * per_divisor);
  while (q * divisor > x) --q;
  while (x - q * divisor >= divisor) ++q;
  return q;
}

// even contiguous runs of `units` over `grid` thread blocks: the first `rem` of them hold one more
struct EvenRuns {
  int q, rem;
  HTR_HD EvenRuns(int quotient, int remainder, int) : q(quotient), rem(remainder) {}   // divided elsewhere
  HTR_HD EvenRuns(int units, int grid) : q(units / grid), rem(units - (units / grid) * grid) {}
  HTR_HD int begin(int b) const { return b * q + (b < rem ? b : rem); }
  HTR_HD int owner(int u) const { return u < rem * (q + 1) ? u / (q + 1) : rem + (u - rem * (q + 1)) / q; }
};

// owner of unit x when thread block b of G starts at floor(b*U/G)
HTR_HD int unit_owner(long long x, long long G, long long U) { return (int)(((x + 1) * G - 1) / U); }
// The same runs without a division: U / G and U % G, reciprocal(G) (b * rem * G stays below G^3: G up to 1625), and G / U
struct FlatRuns {
  int q, rem;
  unsigned grid_magic;
  float per_unit;
  HTR_HD FlatRuns(int quotient, int remainder, unsigned magic, float blocks_per_unit)
      : q(quotient), rem(remainder), grid_magic(magic), per_unit(blocks_per_unit) {}
  HTR_HD int begin(int b) const { return b * q + quotient(b * rem, grid_magic); }
  HTR_HD int owner(int x) const {
    int b = (int)(((float)x + 0.5f) * per_unit);
    while (begin(b) > x) --b;
    while (begin(b + 1) <= x) ++b;
    return b;
  }
};

// first of the blocks of part `part` where `split` parts share q * split + rem blocks: floor(part * blocks / split), the quotient of the remainders
// from magic = part_reciprocal(split) (exact: at most 16 * 15 by at most 16)
inline int part_reciprocal(int split) { return (65536 + split - 1) / split; }
HTR_HD int part_begin(int part, int q, int rem, int magic) { return part * q + ((part * rem * magic) >> 16); }

}  // namespace htr
