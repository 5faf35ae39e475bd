// wg_simplify.cu -- all-pairs Pauli products and simplify (sort, reduce, cull).
//
// Semantics (reference src/simplify.cpp:147-430, src/multiply.cpp:73-402):
//  * product (l, r): x = lx ^ rx, z = lz ^ rz,
//      e = sum_w popc(x&z) - popc(lx&lz) - popc(rx&rz) + 2 popc(lx&rz)  (mod 4),
//      c = (cl * cr) * i^e, with std::complex<double> rounding;
//    products are numbered l*n_r + r (nested-loop order, lhs outer).
//  * simplify: equal keys are summed in input order, kept iff
//    |sum| > atol + rtol*max|c_in| (|.| = glibc hypot), emitted in canonical
//    key order (x0, z0, x1, z1, ... as unsigned words).
//
// An item is a term, or a product known by its number: neither a product's
// key nor its coefficient is ever stored, both are formed from the operands
// (which stay in L2) where they are needed.
//
//  * up to 8,192 items: one CTA does all of it in one launch (small_kernel);
//  * above: each item's key becomes a 64-bit code that sorts like it
//    (wg_sort.cuh); a stable radix sort of (code, item) pairs; then
//    reduce_kernel, a CTA per 1,024 sorted items, finds the runs of equal
//    codes, puts the rare run of unequal keys in order, sums every key's items
//    left to right (stability keeps them in input order, the reference's order
//    and rounding) and culls; write_kernel forms the survivors' keys at their
//    ranks.  Keys whose codes tie too often are sorted by all their words.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>

#include "wg_common.cuh"
#include "wg_scan.cuh"
#include "wg_sort.cuh"
#include "wg_sort_block.cuh"

namespace {

using wgd::c128;
using namespace wgo;

constexpr int kThreads = 256;

// Raw products in nested-loop order; W words a mask (W < 0: any width, Wrt).  Bound by
// the writes: 16,777,216 products of 100 qubits 185 us, 4.4 TB/s (238 with 8-byte stores
// and CTAs for one wave and a third); 9,000,000 of 150 qubits 239 (258).
template <int W>
__global__ void __launch_bounds__(kThreads) products_kernel(
    const uint64_t* __restrict__ lx, const uint64_t* __restrict__ lz, const double* __restrict__ lc, size_t n_l,
    const uint64_t* __restrict__ rx, const uint64_t* __restrict__ rz, const double* __restrict__ rc, size_t n_r,
    int Wrt, uint64_t* __restrict__ out_x, uint64_t* __restrict__ out_z, double* __restrict__ out_c) {
  const size_t P = n_l * n_r;
  const int WW = W >= 0 ? W : Wrt;
  for (size_t p = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; p < P;
       p += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t l = p / n_r;
    const size_t r = p - l * n_r;
    unsigned e = 0;
    auto word = [&](int w, uint64_t& px, uint64_t& pz) {
      const uint64_t ax = __ldg(lx + l * WW + w), az = __ldg(lz + l * WW + w);
      const uint64_t bx = __ldg(rx + r * WW + w), bz = __ldg(rz + r * WW + w);
      px = ax ^ bx;
      pz = az ^ bz;
      e += __popcll(px & pz) - __popcll(ax & az) - __popcll(bx & bz) + 2u * __popcll(ax & bz);
    };
    auto coefficient = [&] {
      const c128 a{__ldg(lc + 2 * l), __ldg(lc + 2 * l + 1)};
      const c128 b{__ldg(rc + 2 * r), __ldg(rc + 2 * r + 1)};
      return wgd::rotate(wgd::cmul(a, b), e);
    };
    if constexpr (W == 2) {
      uint64_t x0, z0, x1, z1;
      word(0, x0, z0);
      word(1, x1, z1);
      reinterpret_cast<ulonglong2*>(out_x)[p] = make_ulonglong2(x0, x1);
      reinterpret_cast<ulonglong2*>(out_z)[p] = make_ulonglong2(z0, z1);
    } else {
      for (int w = 0; w < WW; ++w) {
        uint64_t px, pz;
        word(w, px, pz);
        out_x[p * WW + w] = px;
        out_z[p * WW + w] = pz;
      }
    }
    const c128 c = coefficient();
    reinterpret_cast<double2*>(out_c)[p] = make_double2(c.re, c.im);
  }
}

// ------------------------------------------------------------- items

// The mask words of one operand, in key order (x0, z0, x1, z1, ...).
struct OperandWords {
  const uint64_t* x;
  const uint64_t* z;
  int W;
  __device__ __forceinline__ uint64_t operator()(size_t t, int k) const {
    return __ldg((k & 1 ? z : x) + t * W + (k >> 1));
  }
};

// i / n as a multiplication: div = floor((2^64 - 1) / n) + 1 is exact for
// i, n < 2^32; n = 1 divides trivially.
struct Divide {
  uint32_t n;
  uint64_t div;
  explicit Divide(size_t d) : n(static_cast<uint32_t>(d)), div(d > 1 ? ~0ull / d + 1 : 0ull) {}
  __device__ __forceinline__ void split(uint32_t i, uint32_t& q, uint32_t& r) const {
    q = n == 1 ? i : static_cast<uint32_t>(__umul64hi(static_cast<uint64_t>(i), div));
    r = i - q * n;
  }
};

// Item i is term i of one operator.  W: mask words, 0 for any number.
template <int W>
struct TermItems {
  const uint64_t* x;
  const uint64_t* z;
  const double* c;
  int Wrt;
  const uint64_t* bits;  // packed keys [t][words]
  int words;
  __device__ __forceinline__ uint64_t packed(uint32_t i, int w) const { return __ldg(bits + size_t(i) * words + w); }
  __device__ __forceinline__ uint64_t key(uint32_t i, int k) const {
    const int WW = W > 0 ? W : Wrt;
    return __ldg((k & 1 ? z : x) + size_t(i) * WW + (k >> 1));
  }
  __device__ __forceinline__ c128 coefficient(uint32_t i) const {
    return {__ldg(c + 2 * size_t(i)), __ldg(c + 2 * size_t(i) + 1)};
  }
  __device__ __forceinline__ void store(uint32_t i, size_t o, uint64_t* ox, uint64_t* oz) const {
    const int WW = W > 0 ? W : Wrt;
    for (int w = 0; w < WW; ++w) {
      ox[o * WW + w] = __ldg(x + size_t(i) * WW + w);
      oz[o * WW + w] = __ldg(z + size_t(i) * WW + w);
    }
  }
};

// Item i is the product of lhs term i / n_r and rhs term i % n_r.  The operand
// records are [x0 z0 x1 z1 ... | re im], read 16 bytes at a time.
template <int W>
struct ProductItems {
  const uint64_t* lrec;
  const uint64_t* rrec;
  int Wrt;
  Divide by;
  const uint64_t* lbits;  // packed operand keys [t][words]
  const uint64_t* rbits;
  int words;
  __device__ __forceinline__ uint64_t packed(uint32_t i, int w) const {
    uint32_t l, r;
    by.split(i, l, r);
    return __ldg(lbits + size_t(l) * words + w) ^ __ldg(rbits + size_t(r) * words + w);
  }
  __device__ __forceinline__ c128 coefficient(uint32_t i) const {
    const int WW = W > 0 ? W : Wrt;
    uint32_t l, r;
    by.split(i, l, r);
    const ulonglong2* a = reinterpret_cast<const ulonglong2*>(lrec) + size_t(l) * (WW + 1);
    const ulonglong2* b = reinterpret_cast<const ulonglong2*>(rrec) + size_t(r) * (WW + 1);
    unsigned e = 0;
#pragma unroll
    for (int w = 0; w < WW; ++w) {
      const ulonglong2 p = __ldg(a + w), q = __ldg(b + w);
      e += __popcll((p.x ^ q.x) & (p.y ^ q.y)) - __popcll(p.x & p.y) - __popcll(q.x & q.y) + 2u * __popcll(p.x & q.y);
    }
    const double2 u = __ldg(reinterpret_cast<const double2*>(a + WW));
    const double2 v = __ldg(reinterpret_cast<const double2*>(b + WW));
    return wgd::rotate(wgd::cmul(c128{u.x, u.y}, c128{v.x, v.y}), e);
  }
  __device__ __forceinline__ void store(uint32_t i, size_t o, uint64_t* ox, uint64_t* oz) const {
    const int WW = W > 0 ? W : Wrt;
    uint32_t l, r;
    by.split(i, l, r);
    const ulonglong2* a = reinterpret_cast<const ulonglong2*>(lrec) + size_t(l) * (WW + 1);
    const ulonglong2* b = reinterpret_cast<const ulonglong2*>(rrec) + size_t(r) * (WW + 1);
    if constexpr (W == 2) {
      const ulonglong2 p = __ldg(a), q = __ldg(b), u = __ldg(a + 1), v = __ldg(b + 1);
      reinterpret_cast<ulonglong2*>(ox)[o] = make_ulonglong2(p.x ^ q.x, u.x ^ v.x);
      reinterpret_cast<ulonglong2*>(oz)[o] = make_ulonglong2(p.y ^ q.y, u.y ^ v.y);
    } else {
      for (int w = 0; w < WW; ++w) {
        const ulonglong2 p = __ldg(a + w), q = __ldg(b + w);
        ox[o * WW + w] = p.x ^ q.x;
        oz[o * WW + w] = p.y ^ q.y;
      }
    }
  }
};

// Both operands' records and packed keys (blockIdx.y: the operand).
struct Operand {
  OperandWords words;
  const double* c;
  size_t n;
  uint64_t* rec;   // null: packed keys only
  uint64_t* bits;
};

__global__ void __launch_bounds__(kThreads) pack_kernel(Operand a, Operand b, int W,
                                                        const unsigned long long* __restrict__ masks, int words) {
  const Operand& p = blockIdx.y == 0 ? a : b;
  for (size_t t = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; t < p.n;
       t += static_cast<size_t>(gridDim.x) * blockDim.x) {
    if (p.rec) {
      uint64_t* rec = p.rec + t * (2 * W + 2);
      for (int k = 0; k < 2 * W; ++k) rec[k] = p.words(t, k);
      rec[2 * W] = static_cast<uint64_t>(__double_as_longlong(p.c[2 * t]));
      rec[2 * W + 1] = static_cast<uint64_t>(__double_as_longlong(p.c[2 * t + 1]));
    }
    pack_key(masks, 2 * W, [&](int k) { return p.words(t, k); },
             [&](int w, uint64_t v) { p.bits[t * words + w] = v; }, words);
  }
}

// Every item's code, and the digit counts of all radix passes.  Bound by the ALU
// for wide keys (the loop over a key's set bits: 1.8 ms for 67,108,864 products of
// 100 qubits), else by the shared-memory atomics, one per item and pass (0.09 ms for
// 16,777,216 products of 20).
template <class Items>
__global__ void __launch_bounds__(kThreads) code_kernel(Items items, uint32_t n, CodeSpec spec, int passes,
                                                        uint64_t* __restrict__ code, uint32_t* hist) {
  extern __shared__ uint32_t sh[];
  clear_digits(sh, passes);
  __syncthreads();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    bool whole;
    const uint64_t c = key_code(spec, [&](int w) { return items.packed(static_cast<uint32_t>(i), w); }, &whole);
    code[i] = c;
    count_digits(sh, c, passes);
  }
  __syncthreads();
  store_digits(sh, passes, hist);
}

// The top 8 * passes bits of one packed word as code, read through the order
// so far (none: item order).
template <class Items>
__global__ void __launch_bounds__(kThreads) word_kernel(Items items, uint32_t n, int w, int passes,
                                                        const uint32_t* __restrict__ order,
                                                        uint64_t* __restrict__ code, uint32_t* hist) {
  extern __shared__ uint32_t sh[];
  clear_digits(sh, passes);
  __syncthreads();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint64_t c = items.packed(order ? order[i] : static_cast<uint32_t>(i), w) >> (64 - 8 * passes);
    code[i] = c;
    count_digits(sh, c, passes);
  }
  __syncthreads();
  store_digits(sh, passes, hist);
}

// ------------------------------------------------------------- thresholds

// 0 fixed; 1 atol + rtol * max|c|; 2 atol, unless some |c| is infinite (then
// atol + 0 * inf is NaN and nothing survives).  max: bits of the largest |c|
// (non-negative doubles order like their bits; a NaN never replaces it).
struct Threshold {
  int mode;
  double atol, rtol, fixed;
  const unsigned long long* max;
  __device__ __forceinline__ double value() const {
    // one product, one sum, no contraction (src/simplify.cpp:156-160)
    if (mode == 1) return __dadd_rn(atol, __dmul_rn(rtol, __longlong_as_double(static_cast<long long>(*max))));
    return mode == 0 ? fixed : atol;
  }
};

// |c| > thr; without NaNs the rounded |c| is never below max(|re|, |im|), so
// most sums are decided without the full hypot
__device__ __forceinline__ bool above(c128 c, double thr) {
  const bool plain = !isnan(c.re) && !isnan(c.im);
  return (plain && (fabs(c.re) > thr || fabs(c.im) > thr)) || wgd::hypot_ref(c.re, c.im) > thr;
}

__device__ __noinline__ bool infinite_magnitude(double re, double im) { return isinf(wgd::hypot_ref(re, im)); }

__device__ __forceinline__ bool infinite(c128 c) {
  return !(fabs(c.re) <= 0x1p1022 && fabs(c.im) <= 0x1p1022) && infinite_magnitude(c.re, c.im);
}

template <class Items>
__global__ void __launch_bounds__(kThreads) max_abs_kernel(Items items, uint32_t n,
                                                           unsigned long long* __restrict__ max_bits) {
  double mx = 0.0;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const c128 c = items.coefficient(static_cast<uint32_t>(i));
    const double a = wgd::hypot_ref(c.re, c.im);
    if (mx < a) mx = a;  // std::max semantics: a NaN never replaces the running max
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    const double other = __shfl_xor_sync(0xffffffffu, mx, o);
    if (mx < other) mx = other;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(max_bits, static_cast<unsigned long long>(__double_as_longlong(mx)));
}

// ------------------------------------------------------------- reduction

// How equal keys are recognised in the sorted order:
enum Equal : int {
  kByCode = 0,   // the code is the key
  kChecked = 1,  // equal codes, and the keys compared where a code can tie
  kByKey = 2,    // the packed words (sorted by all of them)
};

constexpr int kTile = 1024;        // sorted items whose runs a CTA owns
constexpr int kBeyond = 256;       // items of its last run that it also stages
constexpr int kSpan = kTile + kBeyond;
constexpr int kSpanWords = kSpan / 32;
constexpr int kMixedRun = 16;      // a longer run of equal codes and unequal keys is sorted by the whole CTA
constexpr int kMixedRuns = kSpan / (kMixedRun + 1) + 1;
constexpr int kSortSpan = 2048;    // kSpan, up to the next power of two

// Long mixed runs, sorted by the code bits behind the first ones.
struct MixedSmem {
  uint64_t code[kSortSpan];
  uint16_t at[kSortSpan];
};

struct ReduceSmem {
  union {
    double2 c[kSpan];
    MixedSmem mixed_run;  // before the coefficients are formed
  };
  uint32_t idx[kSpan];
  uint32_t head[kSpanWords];
  uint32_t keep[kSpanWords];
  uint32_t rank[kSpanWords + 1];
  uint32_t end;
  uint32_t runs;
  uint32_t run[kMixedRuns];  // first item << 16 | end
};

__device__ __forceinline__ int next_bit(const uint32_t* bits, int words, int p) {
  int w = p >> 5;
  if (w >= words) return 32 * words;
  uint32_t m = bits[w] & (0xffffffffu << (p & 31));
  while (!m) {
    if (++w == words) return 32 * words;
    m = bits[w];
  }
  return 32 * w + __ffs(m) - 1;
}

template <class Items>
__device__ __forceinline__ int compare_items(const Items& items, uint32_t a, uint32_t b, int words) {
  for (int w = 0; w < words; ++w) {
    const uint64_t u = items.packed(a, w), v = items.packed(b, w);
    if (u != v) return u < v ? -1 : 1;
  }
  return 0;
}

// rank[w] = set bits below word w; rank[words] = all.  One warp.
__device__ __forceinline__ void rank_bits(const uint32_t* bits, int words, uint32_t* rank) {
  const int lane = threadIdx.x & 31;
  uint32_t run = 0;
  for (int w0 = 0; w0 < words; w0 += 32) {
    const uint32_t c = w0 + lane < words ? __popc(bits[w0 + lane]) : 0;
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (w0 + lane < words) rank[w0 + lane] = run + incl - c;
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (lane == 0) rank[words] = run;
}

// Puts a run [a, b) of equal codes and unequal keys in stable key order and
// marks where its keys start; false: the further code bits do not tell all of
// its keys apart.  All threads of the CTA.
template <class Items>
__device__ bool sort_mixed_run(const Items& items, const CodeSpec& spec, ReduceSmem& sm, int a, int b) {
  const int tid = threadIdx.x, m = b - a;
  uint64_t* code = sm.mixed_run.code;
  uint16_t* at = sm.mixed_run.at;
  int size = 32;
  while (size < m) size *= 2;
  __syncthreads();
  for (int q = tid; q < size; q += kThreads) {
    bool whole;
    code[q] = q < m ? key_code(spec, [&](int w) { return items.packed(sm.idx[a + q], w); }, &whole, 64) : ~0ull;
    at[q] = static_cast<uint16_t>(q);
  }
  // bitonic sort by (code, place)
  for (int k = 2; k <= size; k *= 2)
    for (int j = k / 2; j > 0; j /= 2) {
      __syncthreads();
      for (int q = tid; q < size; q += kThreads) {
        const int r = q ^ j;
        if (r < q) continue;
        const uint64_t u = code[q], v = code[r];
        const uint16_t x = at[q], y = at[r];
        const bool greater = u != v ? u > v : x > y;
        if (greater == ((q & k) == 0)) {
          code[q] = v;
          code[r] = u;
          at[q] = y;
          at[r] = x;
        }
      }
    }
  __syncthreads();
  uint32_t moved[kSpan / kThreads];
#pragma unroll
  for (int e = 0; e < kSpan / kThreads; ++e) {
    const int q = tid + e * kThreads;
    moved[e] = q < m ? sm.idx[a + at[q]] : 0;
  }
  __syncthreads();
#pragma unroll
  for (int e = 0; e < kSpan / kThreads; ++e) {
    const int q = tid + e * kThreads;
    if (q < m) sm.idx[a + q] = moved[e];
  }
  __syncthreads();
  bool ok = true;
  for (int q = 1 + tid; q < m; q += kThreads) {
    if (code[q] != code[q - 1]) atomicOr(&sm.head[(a + q) >> 5], 1u << ((a + q) & 31));
    else ok &= compare_items(items, sm.idx[a + q], sm.idx[a + q - 1], spec.words) == 0;
  }
  return ok;
}

// A CTA owns the runs that start in its tile.  Coefficients are formed by all
// threads and left in shared memory, then a thread per run adds its run up:
// the loads of a long run are spread over the CTA and only its additions stay
// in sequence (one thread gathering a whole run from memory took 3.0 ms for
// 5,000,000 terms of 100,000 keys; this takes 0.22 ms).  Bound by the gathers of
// the operands' records, which live in L1 and L2: tiles of 1,024 leave L1 the
// room for them that tiles of 2,048 take (0.33 against 0.38 ms for 4,096 x 4,096
// products).
template <int EQUAL, class Items>
__global__ void __launch_bounds__(kThreads, 4) reduce_kernel(Items items, const uint64_t* __restrict__ code,
                                                             const uint32_t* __restrict__ idx, uint32_t n,
                                                             CodeSpec spec, Threshold threshold,
                                                             uint32_t* __restrict__ out_idx,
                                                             double2* __restrict__ out_c,
                                                             uint32_t* __restrict__ counts,
                                                             uint32_t* __restrict__ starts, SortControl* ctl) {
  extern __shared__ __align__(16) unsigned char raw[];
  ReduceSmem& sm = *reinterpret_cast<ReduceSmem*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (ctl->timeout) {  // item numbers are not all in place
    if (tid == 0) counts[blockIdx.x] = 0;
    return;
  }
  const size_t t0 = static_cast<size_t>(blockIdx.x) * kTile;
  const int own = static_cast<int>(min(static_cast<size_t>(kTile), n - t0));
  const double thr = threshold.value();
  for (int p = tid; p < kSpan; p += kThreads) {
    const size_t g = t0 + p;
    bool head = true;  // past the end: ends the last run
    if (g < n) {
      const uint32_t i = idx[g];
      sm.idx[p] = i;
      if (g > 0) {
        if (EQUAL == kByKey) head = compare_items(items, i, idx[g - 1], spec.words) != 0;
        else head = code[g] != code[g - 1];
      }
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, head);
    if (lane == 0) sm.head[p >> 5] = bits;
  }
  for (int w = tid; w < kSpanWords; w += kThreads) sm.keep[w] = 0;
  __syncthreads();
  const int first = next_bit(sm.head, kSpanWords, 0);
  if (first >= own) {  // inside another tile's run
    if (tid == 0) counts[blockIdx.x] = 0;
    return;
  }
  int last = own - 1;
  {
    int w = last >> 5;
    uint32_t m = sm.head[w] & (0xffffffffu >> (31 - (last & 31)));
    while (!m) m = sm.head[--w];
    last = 32 * w + 31 - __clz(m);
  }
  int end = next_bit(sm.head, kSpanWords, last + 1);
  const bool open = end == kSpan && t0 + kSpan < n && [&] {
    // the last run may go on behind the staged items
    const size_t g = t0 + kSpan;
    if (EQUAL == kByKey) return compare_items(items, idx[g], idx[g - 1], spec.words) == 0;
    return code[g] == code[g - 1];
  }();
  if (open) end = last;
  // runs whose code may stand for several keys
  if (EQUAL == kChecked) {
    if (tid == 0) sm.runs = 0;
    uint32_t heads = 0;  // the run starts among this thread's places, before any are added
    for (int p = first + tid, j = 0; p < min(end, kTile); p += kThreads, ++j)
      heads |= ((sm.head[p >> 5] >> (p & 31)) & 1u) << j;
    __syncthreads();
    for (int p = first + tid; heads; p += kThreads, heads >>= 1) {
      if (!(heads & 1u)) continue;
      const int e = next_bit(sm.head, kSpanWords, p + 1);
      if (e - p == 1) continue;
      bool whole, mixed = false;
      const uint32_t h = sm.idx[p];
      (void)key_code(spec, [&](int w) { return items.packed(h, w); }, &whole);
      if (!whole)
        for (int q = p + 1; q < e && !mixed; ++q) mixed = compare_items(items, h, sm.idx[q], spec.words) != 0;
      if (!mixed) continue;
      if (e - p > kMixedRun) {
        sm.run[atomicAdd(&sm.runs, 1u)] = static_cast<uint32_t>(p) << 16 | static_cast<uint32_t>(e);
        continue;
      }
      // stable insertion sort by key
      for (int q = p + 1; q < e; ++q) {
        const uint32_t i = sm.idx[q];
        int r = q;
        for (; r > p && compare_items(items, sm.idx[r - 1], i, spec.words) > 0; --r) sm.idx[r] = sm.idx[r - 1];
        sm.idx[r] = i;
      }
      // other threads look for their runs' ends before this run's first item
      for (int q = p + 1; q < e; ++q)
        if (compare_items(items, sm.idx[q - 1], sm.idx[q], spec.words) != 0)
          atomicOr(&sm.head[q >> 5], 1u << (q & 31));
    }
    __syncthreads();
    const uint32_t runs = sm.runs;
    for (uint32_t r = 0; r < runs; ++r)
      if (!sort_mixed_run(items, spec, sm, static_cast<int>(sm.run[r] >> 16), static_cast<int>(sm.run[r] & 0xffffu)))
        ctl->mixed = 1;
    __syncthreads();
  }
  bool inf = false;
  for (int p = first + tid; p < end; p += kThreads) {
    const c128 c = items.coefficient(sm.idx[p]);
    inf |= infinite(c);
    sm.c[p] = make_double2(c.re, c.im);
  }
  __syncthreads();
  for (int p = first + tid; p < end; p += kThreads) {
    if (!((sm.head[p >> 5] >> (p & 31)) & 1u)) continue;
    const int e = next_bit(sm.head, kSpanWords, p + 1);
    c128 acc{0.0, 0.0};
    for (int q = p; q < e; ++q) {
      const double2 v = sm.c[q];
      acc = wgd::cadd(acc, c128{v.x, v.y});
    }
    sm.c[p] = make_double2(acc.re, acc.im);
    if (above(acc, thr)) atomicOr(&sm.keep[p >> 5], 1u << (p & 31));
  }
  __syncthreads();
  if (warp == 0) rank_bits(sm.keep, kSpanWords, sm.rank);
  __syncthreads();
  // survivors from the tile's first run on: no more than it has items, so the tiles' lie one behind another
  const size_t o0 = t0 + first;
  for (int p = tid; p < kSpan; p += kThreads) {
    const uint32_t k = sm.keep[p >> 5];
    if (!((k >> (p & 31)) & 1u)) continue;
    const size_t o = o0 + sm.rank[p >> 5] + __popc(k & ((1u << (p & 31)) - 1u));
    out_idx[o] = sm.idx[p];
    out_c[o] = sm.c[p];
  }
  uint32_t kept = sm.rank[kSpanWords];
  if (open) {
    // the open run, kTile items at a time; thread 0 carries the sum
    const uint32_t h = sm.idx[last];
    bool whole = true;
    if (EQUAL == kChecked) (void)key_code(spec, [&](int w) { return items.packed(h, w); }, &whole);
    c128 acc{0.0, 0.0};
    bool mixed = false;
    for (size_t g0 = t0 + last;; g0 += kTile) {
      __syncthreads();
      if (tid == 0) sm.end = kTile;
      __syncthreads();
      for (int p = tid; p < kTile; p += kThreads) {
        const size_t g = g0 + p;
        bool out = g >= n;
        if (!out) {
          const uint32_t i = idx[g];
          if (EQUAL == kByKey) out = compare_items(items, i, h, spec.words) != 0;
          else out = code[g] != code[t0 + last];
          if (!out) {
            if (!whole) mixed |= compare_items(items, i, h, spec.words) != 0;
            const c128 c = items.coefficient(i);
            inf |= infinite(c);
            sm.c[p] = make_double2(c.re, c.im);
          }
        }
        if (out) {
          atomicMin(&sm.end, static_cast<uint32_t>(p));
          break;
        }
      }
      __syncthreads();
      const int m = static_cast<int>(sm.end);
      if (tid == 0)
        for (int q = 0; q < m; ++q) acc = wgd::cadd(acc, c128{sm.c[q].x, sm.c[q].y});
      if (m < kTile) break;
    }
    if (mixed) ctl->mixed = 1;
    if (tid == 0 && above(acc, thr)) {
      out_idx[o0 + kept] = h;
      out_c[o0 + kept] = make_double2(acc.re, acc.im);
      ++kept;
    }
  }
  if (inf) ctl->infinite = 1;
  if (tid == 0) {
    counts[blockIdx.x] = kept;
    starts[blockIdx.x] = static_cast<uint32_t>(o0);
  }
}

// The survivors of each tile at their ranks: a CTA per tile.
template <class Items>
__global__ void __launch_bounds__(kThreads) write_kernel(Items items, const uint32_t* __restrict__ sidx,
                                                         const double2* __restrict__ sc,
                                                         const uint32_t* __restrict__ counts,
                                                         const uint32_t* __restrict__ starts,
                                                         const uint32_t* __restrict__ offsets,
                                                         uint64_t* __restrict__ ox, uint64_t* __restrict__ oz,
                                                         double2* __restrict__ oc) {
  const uint32_t m = counts[blockIdx.x];
  if (m == 0) return;
  const size_t o0 = offsets[blockIdx.x], i0 = starts[blockIdx.x];
#pragma unroll 4
  for (uint32_t r = threadIdx.x; r < m; r += kThreads) {
    items.store(sidx[i0 + r], o0 + r, ox, oz);
    oc[o0 + r] = sc[i0 + r];
  }
}

// ------------------------------------------------------------- one CTA

// Everything for at most kBlockSortItems items in one launch: at this size the
// time is that of launches and of the host's waits, not of the work (48 x 40
// products on 16 qubits: 226 us in 20 launches and three waits, 60 us in one
// launch and one wait).
struct SmallSmem {
  BlockSort sort;
  double2 c[kBlockSortItems];
  uint32_t head[kBlockSortItems / 32];
  uint32_t keep[kBlockSortItems / 32];
  uint32_t rank[kBlockSortItems / 32 + 1];
  unsigned long long max;
  uint32_t infinite;
};

// The items' keys and coefficients straight from the operands (rhs absent: the
// lhs terms themselves).
struct SmallItems {
  OperandWords lhs, rhs;
  const double* lc;
  const double* rc;
  Divide by;
  bool products;
};

__global__ void __launch_bounds__(kBlockSortThreads) small_kernel(SmallItems in, int n, int W, Threshold threshold,
                                                                 uint64_t* keys, uint64_t* __restrict__ ox,
                                                                 uint64_t* __restrict__ oz, double2* __restrict__ oc,
                                                                 SortControl* ctl) {
  extern __shared__ __align__(16) unsigned char raw[];
  SmallSmem& sm = *reinterpret_cast<SmallSmem*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, K = 2 * W;
  // keys, word by word: keys[k * n + i]
  for (int i = tid; i < n; i += kBlockSortThreads) {
    uint32_t l = i, r = 0;
    if (in.products) in.by.split(i, l, r);
    for (int k = 0; k < K; ++k) {
      uint64_t v = in.lhs(l, k);
      if (in.products) v ^= in.rhs(r, k);
      keys[k * n + i] = v;
    }
  }
  if (tid == 0) {
    sm.max = 0;
    sm.infinite = 0;
  }
  __syncthreads();
  const uint16_t* order = block_sort(sm.sort, n, K, [&](int k, int i) { return keys[k * n + i]; });
  double mx = 0.0;
  bool inf = false;
  for (int p = tid; p < kBlockSortItems; p += kBlockSortThreads) {
    bool head = true;  // past the end: ends the last run
    if (p < n) {
      const int i = order[p];
      if (p > 0) {
        const int j = order[p - 1];
        head = false;
        for (int k = 0; k < K && !head; ++k) head = keys[k * n + i] != keys[k * n + j];
      }
      c128 c;
      if (in.products) {
        uint32_t l, r;
        in.by.split(i, l, r);
        unsigned e = 0;
        for (int w = 0; w < W; ++w) {
          const uint64_t ax = in.lhs(l, 2 * w), az = in.lhs(l, 2 * w + 1);
          const uint64_t bx = in.rhs(r, 2 * w), bz = in.rhs(r, 2 * w + 1);
          e += __popcll((ax ^ bx) & (az ^ bz)) - __popcll(ax & az) - __popcll(bx & bz) + 2u * __popcll(ax & bz);
        }
        c = wgd::rotate(wgd::cmul(c128{in.lc[2 * l], in.lc[2 * l + 1]}, c128{in.rc[2 * r], in.rc[2 * r + 1]}), e);
      } else {
        c = {in.lc[2 * i], in.lc[2 * i + 1]};
      }
      sm.c[p] = make_double2(c.re, c.im);
      inf |= infinite(c);
      if (threshold.mode == 1) {
        const double a = wgd::hypot_ref(c.re, c.im);
        if (mx < a) mx = a;
      }
    }
    const uint32_t bits = __ballot_sync(0xffffffffu, head);
    if (lane == 0) {
      sm.head[p >> 5] = bits;
      sm.keep[p >> 5] = 0;
    }
  }
  if (mx > 0.0) atomicMax(&sm.max, static_cast<unsigned long long>(__double_as_longlong(mx)));
  if (inf) sm.infinite = 1;
  __syncthreads();
  threshold.max = &sm.max;
  const double thr = threshold.value();
  for (int p = tid; p < n; p += kBlockSortThreads) {
    if (!((sm.head[p >> 5] >> (p & 31)) & 1u)) continue;
    const int e = min(n, next_bit(sm.head, kBlockSortItems / 32, p + 1));
    c128 acc{0.0, 0.0};
    for (int q = p; q < e; ++q) acc = wgd::cadd(acc, c128{sm.c[q].x, sm.c[q].y});
    sm.c[p] = make_double2(acc.re, acc.im);
    if (above(acc, thr)) atomicOr(&sm.keep[p >> 5], 1u << (p & 31));
  }
  __syncthreads();
  if (warp == 0) rank_bits(sm.keep, kBlockSortItems / 32, sm.rank);
  __syncthreads();
  for (int p = tid; p < n; p += kBlockSortThreads) {
    const uint32_t k = sm.keep[p >> 5];
    if (!((k >> (p & 31)) & 1u)) continue;
    const size_t o = sm.rank[p >> 5] + __popc(k & ((1u << (p & 31)) - 1u));
    const int i = order[p];
    for (int w = 0; w < W; ++w) {
      ox[o * W + w] = keys[(2 * w) * n + i];
      oz[o * W + w] = keys[(2 * w + 1) * n + i];
    }
    oc[o] = sm.c[p];
  }
  if (tid == 0) {
    ctl->survivors = sm.rank[kBlockSortItems / 32];
    ctl->infinite = sm.infinite;
  }
}

// ------------------------------------------------------------- host driver

struct Outputs {
  uint64_t** x;
  uint64_t** z;
  double** c;
  size_t* n;
};

SortControl read_control(const SortControl* dev, cudaStream_t s) {
  SortControl h{};
  wg::check_cuda(cudaMemcpyAsync(&h, dev, sizeof(h), cudaMemcpyDeviceToHost, s), "read sort state");
  wg::check_cuda(cudaStreamSynchronize(s), "read sort state");
  if (h.timeout) throw wg::Error(WG_ERR_TIMEOUT, "radix sort: a tile waited too long for its predecessors");
  return h;
}

void run_small(const SmallItems& in, size_t n, int W, const Threshold& thr, const Outputs& out, cudaStream_t s) {
  wg::allow_smem(small_kernel, sizeof(SmallSmem));
  wg::Scratch keys(std::max<size_t>(16, sizeof(uint64_t) * 2 * W * n), s), control(sizeof(SortControl), s);
  // outputs for every item: the count is known only with the result
  wg::Scratch ox(sizeof(uint64_t) * W * n, s), oz(sizeof(uint64_t) * W * n, s), oc(sizeof(double) * 2 * n, s);
  auto* ctl = control.as<SortControl>();
  wg::check_cuda(cudaMemsetAsync(ctl, 0, sizeof(SortControl), s), "clear sort state");
  WG_TIMED("small_kernel", s,
    small_kernel<<<1, kBlockSortThreads, sizeof(SmallSmem), s>>>(in, static_cast<int>(n), W, thr, keys.as<uint64_t>(),
                                                               ox.as<uint64_t>(), oz.as<uint64_t>(),
                                                               oc.as<double2>(), ctl));
  wg::check_launch("launch small simplify");
  const SortControl h = read_control(ctl, s);
  if (h.survivors == 0 || (thr.mode == 2 && h.infinite)) return;
  // Blocks for all items are handed out unless more than kSpare bytes of them would
  // never be used: exact ones take three allocations, copies and a wait (15 us).
  const size_t U = h.survivors;
  constexpr size_t kSpare = size_t{64} << 10;
  if ((n - U) * (16 * static_cast<size_t>(W) + 16) > kSpare) {
    auto exact = [&](wg::Scratch& all, size_t bytes) {
      wg::Scratch own(bytes, s);
      wg::check_cuda(cudaMemcpyAsync(own.get(), all.get(), bytes, cudaMemcpyDeviceToDevice, s), "copy small result");
      std::swap(all, own);
    };
    if (W > 0) {
      exact(ox, sizeof(uint64_t) * W * U);
      exact(oz, sizeof(uint64_t) * W * U);
    }
    exact(oc, sizeof(double) * 2 * U);
    wg::check_cuda(cudaStreamSynchronize(s), "copy small result");
  }
  *out.n = U;
  *out.x = static_cast<uint64_t*>(ox.detach());
  *out.z = static_cast<uint64_t*>(oz.detach());
  *out.c = static_cast<double*>(oc.detach());
}

// Pieces of one block of device memory: of the device's workspace for large
// calls, whose blocks would fragment the pool, else of the pool.
class Pieces {
 public:
  Pieces(int device, size_t bytes, cudaStream_t s) : s_(s) {
    if (bytes >= (size_t{64} << 20)) {
      ws_.reset(new wg::Workspace(device, bytes, s));
      p_ = static_cast<char*>(ws_->take(bytes));
    } else {
      block_.reset(bytes, s);
      p_ = static_cast<char*>(block_.get());
    }
  }
  ~Pieces() {
    // the next holder of the workspace may use another stream
    if (ws_) (void)cudaStreamSynchronize(s_);
  }
  Pieces(const Pieces&) = delete;
  Pieces& operator=(const Pieces&) = delete;
  template <typename T>
  T* take(size_t count) {
    T* out = reinterpret_cast<T*>(p_);
    p_ += wg::Workspace::rounded(sizeof(T) * count);
    return out;
  }

 private:
  cudaStream_t s_;
  std::unique_ptr<wg::Workspace> ws_;
  wg::Scratch block_;
  char* p_;
};

// Sorts and reduces n items; `where` points the items at their packed keys.
// Wide keys go by their codes under WG_SORT_AUTO only.  Returns what sorted them, for
// wg_last_sort_algorithm: WG_SORT_LSD their own bits, WG_SORT_BUCKET their codes.
template <class Items>
int sort_reduce(int device, int W, Items items, uint32_t n, const CodeSpec& spec, Threshold thr,
                Pieces& mem, const Outputs& out, cudaStream_t s) {
  const int passes = (spec.nb + 7) / 8;
  const size_t tiles = pair_tiles(n), parts = (static_cast<size_t>(n) + kTile - 1) / kTile;
  // Sums take the place of one code array and sums' items that of one item array:
  // the codes of the sorted order are to end in the other.
  PairBuffers b{};
  auto* codes = mem.take<uint64_t>(n);
  auto* sc = mem.take<double2>(n);
  b.k0 = codes;
  b.k1 = reinterpret_cast<uint64_t*>(sc);
  if (passes % 2) std::swap(b.k0, b.k1);
  b.i0 = mem.take<uint32_t>(n);
  b.i1 = mem.take<uint32_t>(n);
  auto* counts = mem.take<uint32_t>(parts);
  auto* starts = mem.take<uint32_t>(parts);
  auto* offsets = mem.take<uint32_t>(parts);
  auto* scan = mem.take<uint32_t>(wgs::scan_workspace(parts));
  auto* max_bits = mem.take<unsigned long long>(1);
  // cleared together: status, digit counts, control
  auto* zero = mem.take<char>(sizeof(uint64_t) * kDigits * tiles + sizeof(uint32_t) * kDigits * kMaxPasses + sizeof(SortControl));
  const size_t zero_bytes = sizeof(uint64_t) * kDigits * tiles + sizeof(uint32_t) * kDigits * kMaxPasses + sizeof(SortControl);
  b.status = reinterpret_cast<unsigned long long*>(zero);
  b.hist = reinterpret_cast<uint32_t*>(b.status + kDigits * tiles);
  b.control = reinterpret_cast<SortControl*>(b.hist + kDigits * kMaxPasses);
  const unsigned g = wg::grid_for(n, kThreads, device, 6);
  thr.max = max_bits;
  if (thr.mode == 1) {
    wg::check_cuda(cudaMemsetAsync(max_bits, 0, sizeof(*max_bits), s), "clear max");
    WG_TIMED("max_abs_kernel", s, max_abs_kernel<<<g, kThreads, 0, s>>>(items, n, max_bits));
    wg::check_launch("launch max abs");
  }
  auto reduce = [&](auto* kernel) {
    wg::allow_smem(kernel, sizeof(ReduceSmem));
    WG_TIMED("reduce_kernel", s,
      kernel<<<static_cast<unsigned>(parts), kThreads, sizeof(ReduceSmem), s>>>(items, b.k0, b.i0, n, spec, thr, b.i1,
                                                                              sc, counts, starts, b.control));
    wg::check_launch("launch reduce");
    wgs::exclusive_scan_ws<uint32_t>(counts, offsets, parts, &b.control->survivors, scan, s);
    return read_control(b.control, s);
  };
  SortControl h{};
  h.mixed = !spec.exact && wg::sort_algorithm() != WG_SORT_AUTO;
  if (!h.mixed) {
    wg::check_cuda(cudaMemsetAsync(zero, 0, zero_bytes, s), "clear sort state");
    wg::allow_smem(code_kernel<Items>, digit_smem(kMaxPasses));
    WG_TIMED("code_kernel", s,
      code_kernel<<<g, kThreads, digit_smem(passes), s>>>(items, n, spec, passes, b.k0, b.hist));
    wg::check_launch("launch codes");
    sort_pairs(n, b, passes, true, s);
    h = spec.exact ? reduce(reduce_kernel<kByCode, Items>) : reduce(reduce_kernel<kChecked, Items>);
  }
  const int algo = spec.exact || h.mixed ? WG_SORT_LSD : WG_SORT_BUCKET;
  if (h.mixed) {
    wg::allow_smem(word_kernel<Items>, digit_smem(kMaxPasses));
    for (int w = spec.words - 1; w >= 0; --w) {
      const int count = (std::min(64, spec.B - 64 * w) + 7) / 8;
      wg::check_cuda(cudaMemsetAsync(zero, 0, zero_bytes, s), "clear sort state");
      WG_TIMED("word_kernel", s,
        word_kernel<<<g, kThreads, digit_smem(count), s>>>(items, n, w, count, w == spec.words - 1 ? nullptr : b.i0,
                                                              b.k0, b.hist));
      wg::check_launch("launch key word");
      sort_pairs(n, b, count, w == spec.words - 1, s);
      (void)read_control(b.control, s);
    }
    h = reduce(reduce_kernel<kByKey, Items>);
  }
  const size_t U = thr.mode == 2 && h.infinite ? 0 : h.survivors;
  *out.n = U;
  if (U == 0) return algo;
  wg::Scratch ox(sizeof(uint64_t) * W * U, s), oz(sizeof(uint64_t) * W * U, s), oc(sizeof(double) * 2 * U, s);
  WG_TIMED("write_kernel", s,
    write_kernel<<<static_cast<unsigned>(parts), kThreads, 0, s>>>(items, b.i1, sc, counts, starts, offsets,
                                                                 ox.as<uint64_t>(),
                                                                 oz.as<uint64_t>(), oc.as<double2>()));
  wg::check_launch("launch simplify output");
  wg::check_cuda(cudaStreamSynchronize(s), "synchronize simplify");
  *out.x = static_cast<uint64_t*>(ox.detach());
  *out.z = static_cast<uint64_t*>(oz.detach());
  *out.c = static_cast<double*>(oc.detach());
  return algo;
}

// Bytes that sort_reduce takes from its Pieces.
size_t sort_reduce_bytes(size_t n) {
  using WS = wg::Workspace;
  const size_t tiles = pair_tiles(n), parts = (n + kTile - 1) / kTile;
  return WS::rounded(8 * n) + WS::rounded(16 * n) + 2 * WS::rounded(4 * n) + 3 * WS::rounded(4 * parts) +
         WS::rounded(4 * wgs::scan_workspace(parts)) +
         WS::rounded(8) + WS::rounded(8 * kDigits * tiles + 4 * kDigits * kMaxPasses + sizeof(SortControl));
}

void simplify_terms(int device, int W, const uint64_t* x, const uint64_t* z, const double* c, size_t n,
                    const Threshold& thr, const Outputs& out, cudaStream_t s) {
  const OperandWords words{x, z, W};
  if (n <= static_cast<size_t>(kBlockSortItems)) {
    run_small(SmallItems{words, words, c, c, Divide(1), false}, n, W, thr, out, s);
    wg::note_sort(WG_SORT_LSD);
    return;
  }
  const KeyBits kb = key_bits(device, 2 * W, n, words, size_t{0}, words, s);
  const CodeSpec spec = choose_code(kb, n);
  const size_t packed = wg::Workspace::rounded(sizeof(uint64_t) * spec.words * n);
  Pieces mem(device, packed + sort_reduce_bytes(n), s);
  auto* bits = mem.take<uint64_t>(spec.words * n);
  const Operand op{words, c, n, nullptr, bits};
  WG_TIMED("pack_kernel", s,
    pack_kernel<<<wg::grid_for(n, kThreads, device, 8), kThreads, 0, s>>>(op, op, W, kb.masks.as<unsigned long long>(),
                                                                        spec.words));
  wg::check_launch("launch pack");
  const uint32_t n32 = static_cast<uint32_t>(n);
  auto go = [&](auto items) { wg::note_sort(sort_reduce(device, W, items, n32, spec, thr, mem, out, s)); };
  if (W == 1) go(TermItems<1>{x, z, c, 1, bits, spec.words});
  else if (W == 2) go(TermItems<2>{x, z, c, 2, bits, spec.words});
  else go(TermItems<0>{x, z, c, W, bits, spec.words});
}

void simplify_products(int device, int W, const uint64_t* lx, const uint64_t* lz, const double* lc, size_t n_l,
                       const uint64_t* rx, const uint64_t* rz, const double* rc, size_t n_r, const Threshold& thr,
                       const Outputs& out, cudaStream_t s) {
  const size_t P = n_l * n_r;
  const OperandWords l{lx, lz, W}, r{rx, rz, W};
  if (P <= static_cast<size_t>(kBlockSortItems)) {
    run_small(SmallItems{l, r, lc, rc, Divide(n_r), true}, P, W, thr, out, s);
    wg::note_sort(WG_SORT_LSD);
    return;
  }
  const KeyBits kb = key_bits(device, 2 * W, n_l, l, n_r, r, s);
  const CodeSpec spec = choose_code(kb, P);
  using WS = wg::Workspace;
  const size_t rec = 2 * static_cast<size_t>(W) + 2;
  Pieces mem(device, WS::rounded(8 * rec * n_l) + WS::rounded(8 * rec * n_r) + WS::rounded(8 * spec.words * n_l) +
                         WS::rounded(8 * spec.words * n_r) + sort_reduce_bytes(P), s);
  const Operand a{l, lc, n_l, mem.take<uint64_t>(rec * n_l), mem.take<uint64_t>(spec.words * n_l)};
  const Operand b{r, rc, n_r, mem.take<uint64_t>(rec * n_r), mem.take<uint64_t>(spec.words * n_r)};
  const dim3 grid(wg::grid_for(std::max(n_l, n_r), kThreads, device, 4), 2);
  WG_TIMED("pack_kernel", s,
    pack_kernel<<<grid, kThreads, 0, s>>>(a, b, W, kb.masks.as<unsigned long long>(), spec.words));
  wg::check_launch("launch pack");
  const uint32_t n32 = static_cast<uint32_t>(P);
  auto go = [&](auto items) { wg::note_sort(sort_reduce(device, W, items, n32, spec, thr, mem, out, s)); };
  const Divide by(n_r);
  if (W == 1) go(ProductItems<1>{a.rec, b.rec, 1, by, a.bits, b.bits, spec.words});
  else if (W == 2) go(ProductItems<2>{a.rec, b.rec, 2, by, a.bits, b.bits, spec.words});
  else go(ProductItems<0>{a.rec, b.rec, W, by, a.bits, b.bits, spec.words});
}

void validate_tolerances(double atol, double rtol) {
  // src/simplify.cpp:148-150
  if (atol < 0.0 || rtol < 0.0 || !std::isfinite(atol) || !std::isfinite(rtol))
    wg::throw_invalid("simplify tolerances must be non-negative finite values");
}

template <int W>
void launch_products(const uint64_t* lx, const uint64_t* lz, const double* lc, size_t n_l, const uint64_t* rx,
                     const uint64_t* rz, const double* rc, size_t n_r, int Wrt, uint64_t* ox, uint64_t* oz,
                     double* oc, int device, cudaStream_t s) {
  const unsigned g = wg::grid_for(n_l * n_r, kThreads, device, 64);  // ten waves: the last one does not count
  WG_TIMED("products_kernel", s,
    products_kernel<W><<<g, kThreads, 0, s>>>(lx, lz, lc, n_l, rx, rz, rc, n_r, Wrt, ox, oz, oc));
  wg::check_launch("launch products");
}

}  // namespace

extern "C" {

int wg_simplify(int device, size_t words, size_t n_terms, const uint64_t* x, const uint64_t* z,
                const double* coeffs, double atol, double rtol, uint64_t** out_x, uint64_t** out_z,
                double** out_coeffs, size_t* out_terms, wg_stream_t stream) {
  return wg::guarded([&] {
    validate_tolerances(atol, rtol);
    *out_x = *out_z = nullptr;
    *out_coeffs = nullptr;
    *out_terms = 0;
    if (n_terms == 0) return;
    if (n_terms > 0xffffffffull) wg::throw_invalid("simplify supports at most 2^32-1 terms on the device");
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    const int W = static_cast<int>(words);
    const int thr_mode = rtol > 0.0 ? 1 : 2;
    if (wg::sort_algorithm() == WG_SORT_BUCKET &&
        wg::bucket_simplify(device, W, x, z, coeffs, n_terms, thr_mode, atol, rtol, out_x, out_z, out_coeffs,
                            out_terms, s)) {
      wg::note_sort(WG_SORT_BUCKET);
      return;
    }
    simplify_terms(device, W, x, z, coeffs, n_terms, Threshold{thr_mode, atol, rtol, 0.0, nullptr},
                   Outputs{out_x, out_z, out_coeffs, out_terms}, s);
  });
}

int wg_pauli_products(int device, size_t words, const uint64_t* lhs_x, const uint64_t* lhs_z, const double* lhs_c,
                      size_t n_lhs, const uint64_t* rhs_x, const uint64_t* rhs_z, const double* rhs_c,
                      size_t n_rhs, int mode, double atol, double rtol, uint64_t** out_x, uint64_t** out_z,
                      double** out_coeffs, size_t* out_terms, wg_stream_t stream) {
  return wg::guarded([&] {
    if (mode != WG_PRODUCTS_RAW && mode != WG_PRODUCTS_SIMPLIFY && mode != WG_PRODUCTS_FUSED)
      wg::throw_invalid("products mode must be raw, simplify or fused");
    if (mode == WG_PRODUCTS_SIMPLIFY) validate_tolerances(atol, rtol);
    *out_x = *out_z = nullptr;
    *out_coeffs = nullptr;
    *out_terms = 0;
    const size_t P = wg::checked_mul(n_lhs, n_rhs, "matmul intermediate term count");
    if (P == 0) return;
    if (P > 0xffffffffull) wg::throw_invalid("matmul intermediate term count exceeds the device index range (2^32-1)");
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    const int W = static_cast<int>(words);
    if (mode == WG_PRODUCTS_RAW) {
      wg::Scratch ox(sizeof(uint64_t) * P * words, s), oz(sizeof(uint64_t) * P * words, s),
          oc(sizeof(double) * 2 * P, s);
      auto* launch = W == 0 ? launch_products<0> : W == 1 ? launch_products<1> : W == 2 ? launch_products<2>
                                                                                       : launch_products<-1>;
      launch(lhs_x, lhs_z, lhs_c, n_lhs, rhs_x, rhs_z, rhs_c, n_rhs, W, ox.as<uint64_t>(), oz.as<uint64_t>(),
             oc.as<double>(), device, s);
      wg::check_cuda(cudaStreamSynchronize(s), "synchronize products");
      *out_x = static_cast<uint64_t*>(ox.detach());
      *out_z = static_cast<uint64_t*>(oz.detach());
      *out_coeffs = static_cast<double*>(oc.detach());
      *out_terms = P;
      return;
    }
    // The fused hash path of the reference culls at a hard-coded 1e-12
    // (src/multiply.cpp:144, :226); simplify() uses atol + rtol*max|c|.
    const int thr_mode = mode == WG_PRODUCTS_FUSED ? 0 : (rtol > 0.0 ? 1 : 2);
    if (wg::sort_algorithm() == WG_SORT_BUCKET &&
        wg::bucket_products(device, W, lhs_x, lhs_z, lhs_c, n_lhs, rhs_x, rhs_z, rhs_c, n_rhs, thr_mode, atol, rtol,
                            1.0e-12, out_x, out_z, out_coeffs, out_terms, s)) {
      wg::note_sort(WG_SORT_BUCKET);
      return;
    }
    simplify_products(device, W, lhs_x, lhs_z, lhs_c, n_lhs, rhs_x, rhs_z, rhs_c, n_rhs,
                      Threshold{thr_mode, atol, rtol, 1.0e-12, nullptr},
                      Outputs{out_x, out_z, out_coeffs, out_terms}, s);
  });
}

}  // extern "C"
