// Shared pieces of the register/ballot form of the per-strand steps (mg_dual.cuh), which replace
// the sorts and scans over shared arrays of process_strand (mg_kernels.cuh) for reads of up to
// kLeanQ bases:
//
//   seeds / probe          one lane per seed; found index = popc of the found ballot below it
//   occurrence filter      per posting, the bitmask of found indices where its reference occurs;
//                          the longest run of set bits is that reference's occMax
//                          (Analyser.cpp:2057-2115)
//   sort (ref, pos, q)     rank sort of the kept postings (keys are distinct)
//   diagonal runs          run starts as a bit mask; run length = i - last start + 1
//                          (Analyser.cpp:2337-2490)
//   scoring                head/tail walks, coverage and scores in k_finish_dual (mg_lib.cu), from
//                          one record per run end (MatrixCPU.cpp:18-214)
#pragma once
#include "mg_kernels.cuh"

namespace mg {

constexpr int kLeanQ = 320;  // longest read of the register/ballot form

__device__ __forceinline__ int longest_run(uint32_t m) {
  int r = 0;
  while (m) {
    m &= m >> 1;
    r++;
  }
  return r;
}

// upper_dev on each byte of w: bytes 0x61..0x7F lose 0x20.
__device__ __forceinline__ uint32_t upper4(uint32_t w) {
  const uint32_t m = (((w & 0x7F7F7F7Fu) + 0x1F1F1F1Fu) & ~w) & 0x80808080u;
  return w - (m >> 2);
}
// Whether all four bytes of w (upper case) are in ACGT: two bits of a byte pick the letter that it
// has to be.
__device__ __forceinline__ bool acgt4(uint32_t w) {
  const uint32_t c = (w >> 1) & 0x03030303u;  // A 0, C 1, T 2, G 3
  const uint32_t t = c | (c >> 4);
  return __byte_perm(0x47544341u, 0, (t & 0xFFu) | ((t >> 8) & 0xFF00u)) == w;
}
// Complement of four ACGT bytes: A and T differ in 0x15, C and G (bit 1 set) in 0x04.
__device__ __forceinline__ uint32_t comp4(uint32_t w) { return w ^ 0x15151515u ^ (((w >> 1) & 0x01010101u) * 0x11u); }

}  // namespace mg
