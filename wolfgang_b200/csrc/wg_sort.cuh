// wg_sort.cuh -- sort keys as 64-bit order-preserving codes, and one stable
// radix pass per 8 code bits (wg_sort.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "wg_common.cuh"

namespace wgo {

// How a key of B varying bits (most significant first, packed into words)
// becomes a 64-bit code that sorts like it:
//   exact  B <= 64: the bits themselves;
//   else   each set bit is coded by its gap to the previous one, as in
//          Golomb-Rice coding with parameter k (S. W. Golomb, "Run-length
//          encodings", IEEE Trans. Inf. Theory 12, 1966; R. F. Rice, JPL
//          79-22, 1979) but with the remainder complemented: q = gap >> k zeros, a one, then
//          the k low bits of ~gap.  A smaller gap gives a larger code, so
//          codes compare like the keys; k = 0 is the plain bits.  A sparse
//          key's first ten or so set bits fit in 64 bits, where 64 plain bits
//          of it would hold two or three.
// A code that is cut off at 64 bits may be shared by different keys.
struct CodeSpec {
  int B;      // varying key bits
  int words;  // words of a packed key
  int k;      // Rice parameter
  int nb;     // code bits in use (the low ones)
  bool exact;
};

// word(w) gives the packed key's w-th word.  *whole: the code tells this key
// from every other one.  more > 0: the code goes on for that many bits, of
// which the last 64 are returned (which order keys that agree in the ones before).
template <class Word>
__device__ __forceinline__ uint64_t key_code(const CodeSpec& c, Word&& word, bool* whole, int more = 0) {
  if (c.exact) {
    *whole = true;
    return c.B == 0 ? 0 : word(0) >> (64 - c.B);
  }
  uint64_t code = 0;
  int room = c.nb + more;  // code bits left
  int next = 0;     // place behind the last coded bit
  const uint32_t low = (1u << c.k) - 1u;
  for (int w = 0; w < c.words; ++w) {
    const uint64_t v64 = word(w);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      // 32 bits at a time: 64-bit scans and masks take twice the instructions
      uint32_t v = static_cast<uint32_t>(half ? v64 : v64 >> 32);
      const int base = 64 * w + 32 * half;
      while (v) {
        const int lz = __clz(static_cast<int>(v));
        const uint32_t gap = static_cast<uint32_t>(base + lz - next);
        room -= static_cast<int>(gap >> c.k);
        if (room <= 0) {
          *whole = false;
          return code;
        }
        const uint32_t piece = (1u << c.k) | (~gap & low);
        room -= c.k + 1;
        next = base + lz + 1;
        if (room <= 0) {
          *whole = room == 0 && next >= c.B;
          return code | (piece >> -room);
        }
        if (more == 0 || room < 64) code |= static_cast<uint64_t>(piece) << room;
        v &= ~(0x80000000u >> lz);
      }
    }
  }
  // another set bit would have to leave every code bit that is left zero
  *whole = static_cast<long long>(next) + (static_cast<long long>(room) << c.k) >= c.B;
  return code;
}

constexpr int kDigits = 256;
constexpr int kMaxPasses = 8;
constexpr int kHistCopies = 4;  // lanes l with equal l % 4 share a histogram copy

// Adds an item's digits to the CTA's histograms sh[pass][digit][copy].  Zeros
// are left out (radix_base_kernel knows n): the codes of short keys end in
// them, and a warp's equal digits are added one after another.
__device__ __forceinline__ void count_digits(uint32_t* sh, uint64_t code, int passes) {
  const uint32_t copy = threadIdx.x & (kHistCopies - 1);
#pragma unroll 1
  for (int p = 0; p < passes; ++p) {
    const int d = static_cast<int>((code >> (8 * p)) & 255u);
    if (d) atomicAdd(&sh[(p * kDigits + d) * kHistCopies + copy], 1u);
  }
}

__device__ __forceinline__ void clear_digits(uint32_t* sh, int passes) {
  for (int i = threadIdx.x; i < passes * kDigits * kHistCopies; i += blockDim.x) sh[i] = 0;
}

__device__ __forceinline__ void store_digits(const uint32_t* sh, int passes, uint32_t* hist) {
  for (int i = threadIdx.x; i < passes * kDigits; i += blockDim.x) {
    uint32_t s = 0;
#pragma unroll
    for (int c = 0; c < kHistCopies; ++c) s += sh[i * kHistCopies + c];
    if (s) atomicAdd(hist + i, s);
  }
}

constexpr size_t digit_smem(int passes) { return sizeof(uint32_t) * kDigits * kHistCopies * static_cast<size_t>(passes); }

// Device words that a sort writes for the host.
struct SortControl {
  uint32_t ticket[kMaxPasses];  // next tile of each pass
  uint32_t timeout;             // a look-back gave up: codes and item numbers are not all in place, nothing may follow them
  uint32_t mixed;               // a run of equal codes needs the full keys
  uint32_t infinite;            // some |c| is infinite
  uint32_t survivors;
};

// Buffers of one sort of n (code, index) pairs.  The pairs are in k0 / i0
// (i0 unset before the first pass: item i is at place i) and end in k0 / i0.
struct PairBuffers {
  uint64_t *k0, *k1;
  uint32_t *i0, *i1;
  uint32_t* hist;               // [kMaxPasses][256] digit counts, zeroed before counting
  unsigned long long* status;   // [tiles][256], zeroed once per sort
  SortControl* control;         // zeroed before counting
};

size_t pair_tiles(size_t n);

// `count` stable radix passes over the low 8 * count bits of the codes; the
// histograms must hold the digits' counts.  implied: item i of the first pass
// carries index i, i0 is not read.
void sort_pairs(size_t n, PairBuffers& b, int count, bool implied, cudaStream_t s);

// Bits in which the keys of one or two term lists vary, and how many are set.
struct KeyBits {
  bool side_by_side;  // two lists: the keys are XORs of one of each
  int K;              // key words (2 per mask word)
  int B;              // varying bits
  double density;     // mean share of set bits among the varying ones
  std::vector<int> vary;  // varying bits per key word
  wg::Scratch masks;      // device: the same as masks (K words)
};
CodeSpec choose_code(const KeyBits& kb, size_t n);

}  // namespace wgo
