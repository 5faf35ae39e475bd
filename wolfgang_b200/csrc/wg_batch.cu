// wg_batch.cu -- prepared batches of Pauli products: many lhs_p * rhs_p pairs
// of uneven sizes, simplified, in one capturable sequence of launches.
//
// Every pair's result is PauliSum::matmul(simplify) of the reference
// (src/multiply.cpp:73-402, src/simplify.cpp:147-430): products (l, r) in
// nested-loop order, equal keys summed left to right in that order, culled at
// |sum| > thr, emitted in canonical key order.  What a product's key and
// phase are depends only on the operands' masks, so the batch splits the work
// the way a sparse factorisation splits symbolic from numeric work:
//
//  create (symbolic, once): every product of every pair gets the key
//    (pair, x0, z0, ..., x_{W-1}, z_{W-1}); one stable LSD radix sort over all
//    pairs' products groups equal keys of a pair, in nested-loop order; each
//    sorted product keeps its pair-local index and phase (one 32-bit code),
//    each run of equal keys (a segment) its start, pair and key.  All scratch
//    of the numeric pass and the outputs (one slot per segment) are sized here.
//  run (numeric, any number of times): one pass over the products, a CTA per
//    1,024 of them: coefficients formed from the operands' current coefficient
//    buffers, runs summed in order, sums culled (atol + rtol*max|c| over the
//    pair's products, or the fused path's 1e-12) and written with their keys to
//    the slots they have if nothing of their pair is culled.  Pairs of which
//    something was are written once more, at the survivors' ranks.  No
//    allocation, no host copy, no host synchronisation: a run can be captured
//    in a CUDA graph and replayed after the coefficients change.
//
// Sizes: each pair has at most 2^30 products (index and phase share 32 bits)
// and the batch fewer than 2^32 products in all.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "wg_common.cuh"
#include "wg_scan.cuh"

namespace {

using wgd::c128;

constexpr int kThreads = 256;

// Operand masks of one pair (create only).
struct PairMasks {
  const uint64_t* lx;
  const uint64_t* lz;
  const uint64_t* rx;
  const uint64_t* rz;
  uint64_t n_r;
  uint64_t item_base;  // first product of the pair in the batch
};

// What a run needs of one pair.  q / n_r is computed as the high word of
// q * div_m (div_m = floor((2^64 - 1) / n_r) + 1, exact for q, n_r < 2^32;
// n_r = 1 divides trivially).
struct PairNum {
  const double* lc;
  const double* rc;
  uint64_t n_r;
  uint64_t div_m;
  uint64_t seg_base;  // first segment of the pair = first output slot
  uint64_t n_seg;
  uint64_t item_end;  // end of the pair's (sorted) products
};

// How a run forms each pair's largest |product| (the rtol threshold):
enum MaxMode : int {
  kMaxNone = 0,  // fused mode: fixed threshold
  kMaxInf = 1,   // rtol == 0: atol + 0 * max is atol unless some |product| is infinite
  kMaxFull = 2,  // rtol > 0: the maximum itself
};

// ------------------------------------------------------------- symbolic pass

// Keys of every product: word 0 = pair, then the canonical key words (SoA);
// code = pair-local product index << 2 | phase exponent (mod 4).
__global__ void pbatch_keys_kernel(const PairMasks* __restrict__ pairs, const uint64_t* __restrict__ item_base,
                                   uint32_t n_pairs, size_t N, int W, uint64_t* __restrict__ keys,
                                   uint32_t* __restrict__ idx, uint32_t* __restrict__ code) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < N;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    // the last pair whose first product is at or before i (empty pairs share bases)
    uint32_t lo = 0, hi = n_pairs;
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (item_base[mid] <= i) lo = mid;
      else hi = mid;
    }
    const PairMasks P = pairs[lo];
    const uint64_t q = i - P.item_base;
    const uint64_t l = q / P.n_r, r = q - l * P.n_r;
    keys[i] = lo;
    unsigned e = 0;
    for (int w = 0; w < W; ++w) {
      const uint64_t ax = P.lx[l * W + w], az = P.lz[l * W + w];
      const uint64_t bx = P.rx[r * W + w], bz = P.rz[r * W + w];
      const uint64_t px = ax ^ bx, pz = az ^ bz;
      keys[static_cast<size_t>(1 + 2 * w) * N + i] = px;
      keys[static_cast<size_t>(2 + 2 * w) * N + i] = pz;
      e += __popcll(px & pz) - __popcll(ax & az) - __popcll(bx & bz) + 2u * __popcll(ax & bz);
    }
    code[i] = static_cast<uint32_t>(q << 2) | (e & 3u);
    idx[i] = static_cast<uint32_t>(i);
  }
}

__global__ void pbatch_gather_kernel(const uint32_t* __restrict__ idx, const uint32_t* __restrict__ in, size_t N,
                                     uint32_t* __restrict__ out) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < N;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = in[idx[i]];
}

__global__ void pbatch_head_kernel(const uint64_t* __restrict__ keys, size_t N, int K, uint32_t* __restrict__ flags) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < N;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    uint32_t head = i == 0;
    for (int k = 0; k < K && !head; ++k)
      head = keys[static_cast<size_t>(k) * N + i] != keys[static_cast<size_t>(k) * N + i - 1];
    flags[i] = head;
  }
}

// Per segment: start, pair and key (AoS, x words then z words).
__global__ void pbatch_segments_kernel(const uint32_t* __restrict__ flags, const uint32_t* __restrict__ segid,
                                       const uint64_t* __restrict__ keys, size_t N, int W,
                                       uint32_t* __restrict__ seg_start, uint32_t* __restrict__ seg_pair,
                                       uint64_t* __restrict__ seg_keys) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < N;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    if (!flags[i]) continue;
    const size_t s = segid[i];
    seg_start[s] = static_cast<uint32_t>(i);
    seg_pair[s] = static_cast<uint32_t>(keys[i]);
    for (int w = 0; w < W; ++w) {
      seg_keys[s * (2 * W) + w] = keys[static_cast<size_t>(1 + 2 * w) * N + i];
      seg_keys[s * (2 * W) + W + w] = keys[static_cast<size_t>(2 + 2 * w) * N + i];
    }
  }
}

// Segments per pair (segments of a pair are contiguous: one atomic per
// warp-run of equal pairs).
__global__ void pbatch_count_kernel(const uint32_t* __restrict__ seg_pair, size_t S, unsigned* __restrict__ cnt) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t base = static_cast<size_t>(blockIdx.x) * blockDim.x; base < S; base += stride) {
    const size_t s = base + threadIdx.x;
    const uint32_t p = s < S ? seg_pair[s] : 0xffffffffu;
    const unsigned peers = __match_any_sync(0xffffffffu, p);
    if (s < S && (threadIdx.x & 31) == static_cast<unsigned>(__ffs(peers) - 1)) atomicAdd(cnt + p, __popc(peers));
  }
}

// ------------------------------------------------------------- numeric pass

// The magnitude of a product, out of line: kMaxInf needs it only for the rare
// product with a part beyond 2^1022 or not finite.
__device__ __noinline__ double product_magnitude(double re, double im) { return wgd::hypot_ref(re, im); }

// What a run learns of its pairs (cleared by every run).
struct PairRun {
  unsigned long long max;  // bits of the largest |product|, as far as the mode needs it
  uint32_t culled;         // something of the pair is culled
  uint32_t below;          // survivors in its first segment's tile below that segment
};

// Sums that the pass leaves for its repetition: those of the tiles in which it
// found a pair with culled sums.
struct SavedSums {
  double2* sum;     // [segments]
  uint32_t* saved;  // [tiles]
};

// The pair of sorted position j, one of lo to hi.
__device__ __forceinline__ uint32_t pair_within(const PairNum* __restrict__ pairs, uint32_t lo, uint32_t hi, uint64_t j) {
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (j < pairs[mid].item_end) hi = mid;
    else lo = mid + 1;
  }
  return lo;
}

constexpr int kTile = 1024;      // products whose segments a CTA owns: those that start there

// Products of a warp of pbatch_max_kernel, ROUND of a lane in flight together.
template <int ROUND>
constexpr int kMaxItems = ROUND == 1 ? 32 : 64 * ROUND;

// rtol > 0: each pair's largest |product|, ahead of the pass that needs it
// (non-negative doubles order like their bits; a NaN never replaces the running
// maximum, std::max's rule).  A warp takes consecutive products.  The hypot is
// formed only of products that may exceed what is known: |c| <= sqrt(2) max(|re|,
// |im|), and a NaN fails the comparison.  18,000,000 products of 20,000 pairs
// 0.16 ms (0.46 with a look and an atomic by every product).  ROUND = 1 where there
// are few products: what counts then is the chain of one warp's loads.
template <int ROUND>
__global__ void __launch_bounds__(kThreads, ROUND == 1 ? 8 : 4) pbatch_max_kernel(const PairNum* __restrict__ pairs,
                                                              const uint32_t* __restrict__ tile_seg,
                                                              const uint32_t* __restrict__ seg_pair,
                                                              const uint32_t* __restrict__ code, size_t N,
                                                              PairRun* run) {
  const int lane = threadIdx.x & 31;
  const size_t warps = static_cast<size_t>(gridDim.x) * (kThreads / 32);
  auto known = [&](uint32_t p) { return __longlong_as_double(static_cast<long long>(__ldcg(&run[p].max))); };
  // of the lanes that come here together for one pair, those with the largest upper half
  auto put = [&](uint32_t p, double m) {
    const uint32_t peers = __match_any_sync(__activemask(), p), high = static_cast<uint32_t>(__double2hiint(m));
    if (__reduce_max_sync(peers, high) == high && m > 0.0)
      atomicMax(&run[p].max, static_cast<unsigned long long>(__double_as_longlong(m)));
  };
  for (size_t w = (blockIdx.x * static_cast<size_t>(kThreads) + threadIdx.x) >> 5; w * kMaxItems<ROUND> < N; w += warps) {
    const size_t j0 = w * kMaxItems<ROUND>, end = min(N, j0 + kMaxItems<ROUND>);
    // the pairs of the segments that start in the tile, and of the one that reaches into it
    const size_t tile = j0 / kTile;
    const uint32_t first = tile_seg[tile], past = tile_seg[tile + 1];
    const uint32_t lo = seg_pair[first ? first - 1 : 0], hi = seg_pair[past - 1];
    uint32_t p = pair_within(pairs, lo, hi, min(j0 + lane, end - 1));
    double most = known(p), best = 0.0;  // best: what this lane found above what was known
    for (size_t j = j0 + lane; j - lane < end; j += 32 * ROUND) {
      uint32_t own[ROUND], c[ROUND];
      double2 u[ROUND], v[ROUND];
#pragma unroll
      for (int k = 0; k < ROUND; ++k) c[k] = __ldg(code + min(j + 32 * k, end - 1));
#pragma unroll
      for (int k = 0; k < ROUND; ++k) {
        own[k] = pair_within(pairs, k ? own[k - 1] : p, hi, min(j + 32 * k, end - 1));
        const PairNum& P = pairs[own[k]];
        const uint32_t nr = static_cast<uint32_t>(P.n_r), q = c[k] >> 2;  // below 2^30
        const uint32_t l = nr == 1 ? q : static_cast<uint32_t>(__umul64hi(static_cast<uint64_t>(q), P.div_m));
        u[k] = __ldg(reinterpret_cast<const double2*>(P.lc) + l);
        v[k] = __ldg(reinterpret_cast<const double2*>(P.rc) + (q - l * nr));
      }
#pragma unroll
      for (int k = 0; k < ROUND; ++k) {
        // behind the end: the last product once more
        if (own[k] != p) {
          put(p, best);
          p = own[k];
          most = known(p);
          best = 0.0;
        }
        const c128 t = wgd::cmul(c128{u[k].x, u[k].y}, c128{v[k].x, v[k].y});  // the phase leaves |c| as it is
        if (1.5 * fabs(t.re) <= most && 1.5 * fabs(t.im) <= most) continue;
        const double m = product_magnitude(t.re, t.im);
        if (m > most) most = best = m;
      }
    }
    __syncwarp();
    put(p, best);
  }
}

// The pairs' counts, spread over the launch (kept holds the survivors before each
// tile where something was culled).  rtol = 0 (`infinite`): a pair with an infinite
// |product| has the threshold atol + 0 * inf, a NaN, and keeps nothing.
__device__ __forceinline__ void write_counts(const PairNum* __restrict__ pairs, uint32_t n_pairs,
                                             const uint32_t* __restrict__ tile_of, bool infinite, const PairRun* run,
                                             const uint32_t* kept, uint32_t tiles, uint64_t* __restrict__ counts) {
  for (uint64_t p = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; p < n_pairs;
       p += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    uint64_t c = pairs[p].n_seg;
    if (c && run[p].culled) {
      // up to where the next pair with segments begins
      uint64_t q = p + 1;
      while (q < n_pairs && pairs[q].n_seg == 0) ++q;
      const uint32_t end = q < n_pairs ? kept[tile_of[q]] + run[q].below : kept[tiles];
      c = end - (kept[tile_of[p]] + run[p].below);
    }
    if (infinite && isinf(__longlong_as_double(static_cast<long long>(run[p].max)))) c = 0;
    counts[p] = c;
  }
}

constexpr int kStage = kTile + kThreads;  // products staged at a time

// The numeric pass.  All threads form products (coalesced codes, gathers of
// the operands' coefficients in flight together), a thread per segment adds its
// products up from shared memory.  REDO: the pairs with culled segments again,
// at the survivors' ranks (offset: survivors of all tiles before).  WT = W for 1
// or 2 mask words (16-byte loads and stores), 0 for any width.
// Bound by the latency and L1 lookups of the gathers (half of the products'
// coefficients come from L2).  47,800,000 products of 64 pairs on 64 qubits:
// 0.91 ms and 0.03 ms for the repetition's early exits.  Before, a thread per
// segment chased start, code and coefficients one after another (0.99 ms), and
// cull, scan and write-out re-read every sum (0.65 ms).  Where a tile's pairs are
// known to have culled sums by the time it is done, it keeps its sums for the
// repetition, and leaves out the writing if the tile has one pair only: 98,600,000
// products of 64 squares on 64 qubits, 5,200,000 of 39,750,000 sums culled, 2.8 ms
// (4.7 ms with all products formed twice and a mark by every culled sum; 2.9 ms in
// four passes).  Ranks from a look-back
// over the tiles measured 2.7 ms: the tiles of one large pair wait for one
// another in a chain.
template <int WT, int MAX, bool REDO>
__global__ void __launch_bounds__(kThreads, 4) pbatch_pass_kernel(
    const PairNum* __restrict__ pairs, uint32_t n_pairs, const uint32_t* __restrict__ tile_seg, const uint32_t* __restrict__ seg_start,
    const uint32_t* __restrict__ seg_pair, const uint64_t* __restrict__ seg_keys, const uint32_t* __restrict__ code,
    int Wrt, double atol, double rtol, PairRun* run, uint32_t* any, uint32_t* __restrict__ kept,
    const uint32_t* __restrict__ tile_of, uint64_t* __restrict__ ox, uint64_t* __restrict__ oz,
    double2* __restrict__ oc, uint64_t* __restrict__ counts, SavedSums keeper) {
  if (REDO) {
    write_counts(pairs, n_pairs, tile_of, MAX == kMaxInf, run, kept, gridDim.x, counts);
    if (*any == 0) return;
  }
  __shared__ double2 prod[kStage];
  __shared__ uint32_t bits[kTile / 32];
  __shared__ uint32_t rank[kTile / 32 + 1];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int W = WT > 0 ? WT : Wrt;
  const uint32_t s0 = tile_seg[blockIdx.x], s1 = tile_seg[blockIdx.x + 1];
  if (s0 == s1) {
    if (!REDO && tid == 0) kept[blockIdx.x] = keeper.saved[blockIdx.x] = 0;
    return;
  }
  if (REDO) {
    // nothing to do unless a pair of the tile has culled segments
    bool redo = false;
    for (uint32_t p = seg_pair[s0] + tid; p <= seg_pair[s1 - 1]; p += kThreads) redo |= run[p].culled != 0;
    if (!__syncthreads_or(redo)) return;
  }
  const uint32_t j0 = seg_start[s0], j1 = seg_start[s1];
  const uint32_t staged = min(j1 - j0, static_cast<uint32_t>(kStage));
  const uint32_t p0 = seg_pair[s0], p1 = seg_pair[s1 - 1];  // the tile's first and last pair
  const bool hint = !REDO && __ldcg(any) != 0;
  const bool again = REDO && keeper.saved[blockIdx.x] != 0;
  // products [from, from + count) of pairs p to p1 into prod[0..]; the loads of
  // a thread's products are in flight together
  auto stage = [&](uint32_t p, uint32_t from, uint32_t count) {
    constexpr int kPer = kStage / kThreads;
    uint32_t c[kPer], own[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t i = k * kThreads + tid;
      c[k] = i < count ? __ldg(code + from + i) : 0;
    }
    double2 u[kPer], v[kPer];
    auto gather = [&](const PairNum& P, int k) {
      const uint32_t nr = static_cast<uint32_t>(P.n_r), q = c[k] >> 2;  // below 2^30
      const uint32_t l = nr == 1 ? q : static_cast<uint32_t>(__umul64hi(static_cast<uint64_t>(q), P.div_m));
      u[k] = __ldg(reinterpret_cast<const double2*>(P.lc) + l);
      v[k] = __ldg(reinterpret_cast<const double2*>(P.rc) + (q - l * nr));
    };
    if (p == p1) {  // with the pair's fields in registers; searched as below 948 against 916 us for 47,800,000 products
      const PairNum P = pairs[p];
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        own[k] = p;
        gather(P, k);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kPer; ++k) {
        const uint32_t i = k * kThreads + tid;
        if (i < count) p = pair_within(pairs, p, p1, from + i);
        own[k] = p;
        gather(pairs[p], k);
      }
    }
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
      const uint32_t i = k * kThreads + tid;
      if (i >= count) break;
      const c128 t = wgd::rotate(wgd::cmul(c128{u[k].x, u[k].y}, c128{v[k].x, v[k].y}), c[k] & 3u);
      prod[i] = make_double2(t.re, t.im);
      // with rtol = 0 only a magnitude that may be infinite matters (a part
      // beyond 2^1022 or not finite): a finite maximum leaves the threshold at atol
      if (!REDO && MAX == kMaxInf && !(fabs(t.re) <= 0x1p1022 && fabs(t.im) <= 0x1p1022)) {
        const double m = product_magnitude(t.re, t.im);
        if (m > 0.0) atomicMax(&run[own[k]].max, static_cast<unsigned long long>(__double_as_longlong(m)));
      }
    }
  };
  constexpr int kRounds = kTile / kThreads;
  c128 sum[kRounds];
  uint32_t pair[kRounds], begin[kRounds], end[kRounds];
  bool keep[kRounds];
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const uint32_t s = min(s0 + k * kThreads + tid, s1 - 1);
    pair[k] = __ldg(seg_pair + s);
    begin[k] = __ldg(seg_start + s) - j0;
    end[k] = __ldg(seg_start + s + 1) - j0;
  }
  if (!again) stage(p0, j0, staged);
  __syncthreads();
  ulonglong2 key[WT == 1 ? kRounds : 1];  // on their way while the sums are formed
  if constexpr (WT == 1) {
#pragma unroll
    for (int k = 0; k < kRounds; ++k)
      key[k] = __ldg(reinterpret_cast<const ulonglong2*>(seg_keys) + min(s0 + k * kThreads + tid, s1 - 1));
  }
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    sum[k] = {0.0, 0.0};
    if (s0 + k * kThreads + tid >= s1) continue;
    if (again) {
      const double2 v = __ldcs(keeper.sum + s0 + k * kThreads + tid);
      sum[k] = {v.x, v.y};
      continue;
    }
    const uint32_t e = min(end[k], staged);
    for (uint32_t q = begin[k]; q < e; ++q) sum[k] = wgd::cadd(sum[k], c128{prod[q].x, prod[q].y});
  }
  // the last segment may go on behind the staged products: all threads form
  // them, its thread goes on adding
  for (uint32_t from = j0 + staged; !again && from < j1; from += kStage) {
    const uint32_t count = min(j1 - from, static_cast<uint32_t>(kStage));
    __syncthreads();
    stage(p1, from, count);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kRounds; ++k)
      if (s0 + k * kThreads + tid == s1 - 1)
        for (uint32_t q = 0; q < count; ++q) sum[k] = wgd::cadd(sum[k], c128{prod[q].x, prod[q].y});
  }
  // pairs that other tiles have found culled sums of, as far as is known (of the first 256)
  const bool known = hint && static_cast<uint32_t>(tid) <= p1 - p0 && __ldcg(&run[p0 + tid].culled) != 0;
  bool culls = known;
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    keep[k] = false;
    if (s0 + k * kThreads + tid < s1) {
      const c128 acc = sum[k];
      const uint32_t p = pair[k];
      double thr = 1.0e-12;  // the fused path's fixed cull (src/multiply.cpp:144, :226)
      // atol + rtol * max|c| with one rounding each (src/simplify.cpp:156-160)
      if (MAX == kMaxInf) thr = atol;
      else if (MAX == kMaxFull)
        thr = __dadd_rn(atol, __dmul_rn(rtol, __longlong_as_double(static_cast<long long>(run[p].max))));
      // without NaNs the rounded |s| is never below max(|re|, |im|): most sums are
      // decided without the full hypot
      const bool plain = !isnan(acc.re) && !isnan(acc.im);
      keep[k] = (plain && (fabs(acc.re) > thr || fabs(acc.im) > thr)) || wgd::hypot_ref(acc.re, acc.im) > thr;
      if (!REDO && !keep[k]) {
        if (p0 != p1 && __ldcg(&run[p].culled) == 0) run[p].culled = 1;
        culls = true;
      }
    }
    const uint32_t v = __ballot_sync(0xffffffffu, keep[k]);
    if (lane == 0) bits[k * (kThreads / 32) + warp] = v;
  }
  const bool save = __syncthreads_or(culls) && !REDO;
  if (save) {
    // a store by every thread with a culled sum would take its turn in L2: 2 ms for 5,000,000
    if (tid == 0) {
      if (p0 == p1 && !known) run[p0].culled = 1;
      if (__ldcg(any) == 0) *any = 1;
    }
#pragma unroll
    for (int k = 0; k < kRounds; ++k) {
      const uint32_t s = s0 + k * kThreads + tid;
      if (s < s1) __stcs(keeper.sum + s, make_double2(sum[k].re, sum[k].im));
    }
  }
  if (!REDO && tid == 0) keeper.saved[blockIdx.x] = save;
  if (warp == 0) {
    static_assert(kTile / 32 == 32, "one warp scans the tile");
    const uint32_t c = __popc(bits[lane]);
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    rank[lane] = incl - c;
    if (lane == 31) {
      rank[32] = incl;
      if (!REDO) kept[blockIdx.x] = incl;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kRounds; ++k) {
    const uint32_t i = k * kThreads + tid, s = s0 + i;
    if (s >= s1) continue;
    const uint32_t p = pair[k];
    const uint64_t base = pairs[p].seg_base;
    const uint32_t below = rank[i >> 5] + __popc(bits[i >> 5] & ((1u << lane) - 1u));
    size_t o = s;
    if (!REDO) {
      if (s == base) run[p].below = below;
    } else {
      if (!run[p].culled) continue;
      // kept holds the survivors of all tiles before
      o = base + (kept[blockIdx.x] + below) - (kept[tile_of[p]] + run[p].below);
    }
    if (!keep[k] || (save && p0 == p1)) continue;  // one pair: the repetition writes all of it
    if constexpr (WT == 1) {
      ox[o] = key[k].x;
      oz[o] = key[k].y;
    } else if constexpr (WT == 2) {
      reinterpret_cast<ulonglong2*>(ox)[o] = __ldg(reinterpret_cast<const ulonglong2*>(seg_keys) + 2 * size_t(s));
      reinterpret_cast<ulonglong2*>(oz)[o] = __ldg(reinterpret_cast<const ulonglong2*>(seg_keys) + 2 * size_t(s) + 1);
    } else {
      for (int w = 0; w < W; ++w) {
        ox[o * W + w] = seg_keys[size_t(s) * (2 * W) + w];
        oz[o * W + w] = seg_keys[size_t(s) * (2 * W) + W + w];
      }
    }
    oc[o] = make_double2(sum[k].re, sum[k].im);
  }
}

// One CTA, between the pass and its repetition: where something was culled, the
// tiles' survivor counts become the survivors before each tile.
__global__ void __launch_bounds__(1024) pbatch_scan_kernel(const uint32_t* __restrict__ any, uint32_t* kept,
                                                           size_t tiles) {
  constexpr int kPer = 8;  // consecutive tiles of a thread
  __shared__ uint32_t sums[32];
  if (!*any) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t carry = 0;
  for (size_t t0 = 0; t0 < tiles; t0 += 1024 * kPer) {
    uint32_t c[kPer], sum = 0;
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const size_t t = t0 + static_cast<size_t>(tid) * kPer + e;
      c[e] = t < tiles ? kept[t] : 0;
    }
#pragma unroll
    for (int e = 0; e < kPer; ++e) sum += c[e];
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    uint32_t at = carry + incl - sum;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) at += sums[w];
      carry += sums[w];
    }
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const size_t t = t0 + static_cast<size_t>(tid) * kPer + e;
      if (t < tiles) kept[t] = at;
      at += c[e];
    }
    __syncthreads();
  }
  if (tid == 0) kept[tiles] = carry;
}

}  // namespace

// Allocations of a batch come from the device pool on the legacy default
// stream; create ends with a device synchronisation, so they are complete
// before any stream uses them, and destroy synchronises the device first.
struct wg_products_batch_s {
  int device = 0;
  int W = 0;
  int mode = WG_PRODUCTS_SIMPLIFY;
  double atol = 0.0, rtol = 0.0;
  size_t n_pairs = 0, N = 0, S = 0;
  std::vector<uint64_t> seg_base, n_seg;
  wg::Scratch pairs;            // PairNum[n_pairs]
  wg::Scratch code;             // uint32[N]: sorted products' index << 2 | phase
  wg::Scratch seg_start;        // uint32[S + 1]
  wg::Scratch seg_pair;         // uint32[S]
  wg::Scratch seg_keys;         // uint64[S][2W]
  wg::Scratch tile_seg;         // uint32[tiles + 1]: first segment that starts in a tile
  wg::Scratch tile_of;          // uint32[n_pairs]: tile of a pair's first segment
  wg::Scratch run, kept;        // PairRun[n_pairs] and `any`, cleared by every run; uint32[tiles + 1]
  wg::Scratch sums, saved;      // double2[S], uint32[tiles]: SavedSums
  size_t tiles = 0;
  wg::Scratch out_x, out_z, out_c, counts;
};

namespace {

void build_batch(wg_products_batch_s& b, const uint64_t* const* lhs_x, const uint64_t* const* lhs_z,
                 const double* const* lhs_c, const size_t* n_lhs, const uint64_t* const* rhs_x,
                 const uint64_t* const* rhs_z, const double* const* rhs_c, const size_t* n_rhs) {
  const int device = b.device;
  const int W = b.W;
  const size_t np = b.n_pairs;
  cudaStream_t s = nullptr;  // see the note above wg_products_batch_s
  std::vector<PairMasks> masks(np);
  std::vector<PairNum> nums(np);
  std::vector<uint64_t> item_base(np + 1, 0);
  for (size_t p = 0; p < np; ++p) {
    const size_t P = wg::checked_mul(n_lhs[p], n_rhs[p], "matmul intermediate term count");
    if (P > (size_t{1} << 30))
      wg::throw_invalid("a product batch takes at most 2^30 products per pair (pair " + std::to_string(p) +
                        " has " + std::to_string(P) + "); use wg_pauli_products for it");
    if (P > 0) {
      if (!lhs_c[p] || !rhs_c[p]) wg::throw_invalid("product batch pair has a null coefficient buffer");
      // runs read a coefficient (re, im) as one 16-byte load
      if ((reinterpret_cast<uintptr_t>(lhs_c[p]) | reinterpret_cast<uintptr_t>(rhs_c[p])) & 15u)
        wg::throw_invalid("product batch coefficient buffers must be 16-byte aligned (complex128 arrays)");
      if (W > 0 && (!lhs_x[p] || !lhs_z[p] || !rhs_x[p] || !rhs_z[p]))
        wg::throw_invalid("product batch pair has a null mask buffer");
    }
    masks[p] = PairMasks{lhs_x[p], lhs_z[p], rhs_x[p], rhs_z[p], n_rhs[p], item_base[p]};
    const uint64_t div_m = n_rhs[p] > 1 ? ~0ull / n_rhs[p] + 1 : 0ull;
    item_base[p + 1] = item_base[p] + P;
    nums[p] = PairNum{lhs_c[p], rhs_c[p], n_rhs[p], div_m, 0, 0, item_base[p + 1]};
    if (item_base[p + 1] > 0xffffffffull) wg::throw_invalid("a product batch takes fewer than 2^32 products in all");
  }
  const size_t N = item_base[np];
  b.N = N;
  b.seg_base.assign(np, 0);
  b.n_seg.assign(np, 0);
  if (N == 0) {
    b.S = 0;
  } else {
    const int K = 1 + 2 * W;
    wg::Scratch dmasks(sizeof(PairMasks) * np, s), dbase(sizeof(uint64_t) * (np + 1), s);
    wg::check_cuda(cudaMemcpyAsync(dmasks.get(), masks.data(), dmasks.size(), cudaMemcpyHostToDevice, s),
                   "upload batch masks");
    wg::check_cuda(cudaMemcpyAsync(dbase.get(), item_base.data(), dbase.size(), cudaMemcpyHostToDevice, s),
                   "upload batch bases");
    wg::Scratch keys(sizeof(uint64_t) * K * N, s), idx(sizeof(uint32_t) * N, s), raw(sizeof(uint32_t) * N, s);
    const unsigned g = wg::grid_for(N, kThreads, device, 8);
    WG_TIMED("pbatch_keys_kernel", s,
      pbatch_keys_kernel<<<g, kThreads, 0, s>>>(dmasks.as<PairMasks>(), dbase.as<uint64_t>(),
                                                static_cast<uint32_t>(np), N, W, keys.as<uint64_t>(),
                                                idx.as<uint32_t>(), raw.as<uint32_t>()));
    wg::check_launch("launch batch keys");
    wg::radix_sort_keys(device, N, K, keys, idx, s, true);  // stable: nested-loop order within equal keys
    b.code.reset(sizeof(uint32_t) * N, s);
    pbatch_gather_kernel<<<g, kThreads, 0, s>>>(idx.as<uint32_t>(), raw.as<uint32_t>(), N, b.code.as<uint32_t>());
    wg::check_launch("launch batch gather");
    raw.release();
    idx.release();
    wg::Scratch flags(sizeof(uint32_t) * N, s), segid(sizeof(uint32_t) * N, s), total(sizeof(uint32_t), s);
    pbatch_head_kernel<<<g, kThreads, 0, s>>>(keys.as<uint64_t>(), N, K, flags.as<uint32_t>());
    wg::check_launch("launch batch segment heads");
    wgs::exclusive_scan<uint32_t>(flags.as<uint32_t>(), segid.as<uint32_t>(), N, total.as<uint32_t>(), s);
    uint32_t S = 0;
    wg::check_cuda(cudaMemcpyAsync(&S, total.get(), sizeof(S), cudaMemcpyDeviceToHost, s), "read segment count");
    wg::check_cuda(cudaStreamSynchronize(s), "read segment count");
    b.S = S;
    b.seg_start.reset(sizeof(uint32_t) * (size_t(S) + 1), s);
    b.seg_pair.reset(sizeof(uint32_t) * S, s);
    b.seg_keys.reset(sizeof(uint64_t) * std::max<size_t>(1, size_t(S) * 2 * W), s);
    pbatch_segments_kernel<<<g, kThreads, 0, s>>>(flags.as<uint32_t>(), segid.as<uint32_t>(), keys.as<uint64_t>(), N,
                                                  W, b.seg_start.as<uint32_t>(), b.seg_pair.as<uint32_t>(),
                                                  b.seg_keys.as<uint64_t>());
    wg::check_launch("launch batch segments");
    const uint32_t n32 = static_cast<uint32_t>(N);
    wg::check_cuda(cudaMemcpyAsync(b.seg_start.as<uint32_t>() + S, &n32, sizeof(n32), cudaMemcpyHostToDevice, s),
                   "write segment end");
    b.tiles = (N + kTile - 1) / kTile;
    b.tile_seg.reset(sizeof(uint32_t) * (b.tiles + 1), s);
    // the heads before a tile's first position: every kTile-th entry of the scan
    wg::check_cuda(cudaMemcpy2DAsync(b.tile_seg.get(), sizeof(uint32_t), segid.get(), sizeof(uint32_t) * kTile,
                                     sizeof(uint32_t), b.tiles, cudaMemcpyDeviceToDevice, s),
                   "gather tile segments");
    wg::check_cuda(cudaMemcpyAsync(b.tile_seg.as<uint32_t>() + b.tiles, &S, sizeof(S), cudaMemcpyHostToDevice, s),
                   "write tile segment end");
    wg::Scratch cnt(sizeof(unsigned) * np, s);
    wg::check_cuda(cudaMemsetAsync(cnt.get(), 0, cnt.size(), s), "clear segment counts");
    pbatch_count_kernel<<<wg::grid_for(S, kThreads, device, 8), kThreads, 0, s>>>(b.seg_pair.as<uint32_t>(), S,
                                                                                 cnt.as<unsigned>());
    wg::check_launch("launch batch segment counts");
    std::vector<unsigned> hcnt(np);
    wg::check_cuda(cudaMemcpyAsync(hcnt.data(), cnt.get(), cnt.size(), cudaMemcpyDeviceToHost, s),
                   "read segment counts");
    wg::check_cuda(cudaStreamSynchronize(s), "read segment counts");
    uint64_t run = 0;
    for (size_t p = 0; p < np; ++p) {
      b.seg_base[p] = run;
      b.n_seg[p] = hcnt[p];
      nums[p].seg_base = run;
      nums[p].n_seg = hcnt[p];
      run += hcnt[p];
    }
    if (run != S) wg::throw_invalid("product batch segment count mismatch");
  }
  const size_t S = b.S;
  b.pairs.reset(sizeof(PairNum) * std::max<size_t>(np, 1), s);
  wg::check_cuda(cudaMemcpyAsync(b.pairs.get(), nums.data(), sizeof(PairNum) * np, cudaMemcpyHostToDevice, s),
                 "upload batch pairs");
  {
    // the tile in which each pair's first segment starts (its first product's)
    std::vector<uint32_t> tile_of(std::max<size_t>(np, 1), 0);
    for (size_t p = 0; p < np; ++p) tile_of[p] = static_cast<uint32_t>(item_base[p] / kTile);
    b.tile_of.reset(sizeof(uint32_t) * tile_of.size(), s);
    wg::check_cuda(cudaMemcpyAsync(b.tile_of.get(), tile_of.data(), b.tile_of.size(), cudaMemcpyHostToDevice, s),
                   "upload pair tiles");
    wg::check_cuda(cudaStreamSynchronize(s), "upload pair tiles");
  }
  b.run.reset(sizeof(PairRun) * np + 16, s);
  b.kept.reset(sizeof(uint32_t) * (b.tiles + 1), s);
  b.sums.reset(sizeof(double2) * S, s);
  b.saved.reset(sizeof(uint32_t) * b.tiles, s);
  b.out_x.reset(sizeof(uint64_t) * S * W, s);
  b.out_z.reset(sizeof(uint64_t) * S * W, s);
  b.out_c.reset(sizeof(double) * 2 * S, s);
  b.counts.reset(sizeof(uint64_t) * std::max<size_t>(np, 1), s);
  wg::check_cuda(cudaMemsetAsync(b.counts.get(), 0, b.counts.size(), s), "clear batch counts");
  wg::check_cuda(cudaDeviceSynchronize(), "prepare product batch");
}

void run_batch(wg_products_batch_s& b, cudaStream_t s) {
  const int device = b.device;
  const size_t S = b.S;
  if (b.n_pairs == 0) return;
  if (S == 0) {
    wg::check_cuda(cudaMemsetAsync(b.counts.get(), 0, sizeof(uint64_t) * b.n_pairs, s), "clear batch counts");
    return;
  }
  const bool fused = b.mode == WG_PRODUCTS_FUSED;
  const int max_mode = fused ? kMaxNone : b.rtol > 0.0 ? kMaxFull : kMaxInf;
  wg::check_cuda(cudaMemsetAsync(b.run.get(), 0, b.run.size(), s), "clear batch state");
  auto* run = b.run.as<PairRun>();
  auto* any = reinterpret_cast<uint32_t*>(run + b.n_pairs);
  auto* pairs = b.pairs.as<PairNum>();
  auto* code = b.code.as<uint32_t>();
  if (max_mode == kMaxFull) {
    auto maxima = [&](auto* kernel, int items, int ctas) {  // resident CTAs an SM
      const unsigned g = wg::grid_for(b.N, kThreads / 32 * items, device, ctas);
      WG_TIMED("pbatch_max_kernel", s,
        kernel<<<g, kThreads, 0, s>>>(pairs, b.tile_seg.as<uint32_t>(), b.seg_pair.as<uint32_t>(), code, b.N, run));
    };
    if (b.N < (size_t{1} << 20)) maxima(pbatch_max_kernel<1>, kMaxItems<1>, 8);
    else maxima(pbatch_max_kernel<4>, kMaxItems<4>, 4);
    wg::check_launch("launch batch maxima");
  }
  auto pass = [&](auto* kernel, const char* name) {
    WG_TIMED(name, s,
      kernel<<<static_cast<unsigned>(b.tiles), kThreads, 0, s>>>(
          pairs, static_cast<uint32_t>(b.n_pairs), b.tile_seg.as<uint32_t>(), b.seg_start.as<uint32_t>(), b.seg_pair.as<uint32_t>(),
          b.seg_keys.as<uint64_t>(), code, b.W, b.atol, b.rtol, run, any, b.kept.as<uint32_t>(),
          b.tile_of.as<uint32_t>(), b.out_x.as<uint64_t>(), b.out_z.as<uint64_t>(), b.out_c.as<double2>(),
          b.counts.as<uint64_t>(), SavedSums{b.sums.as<double2>(), b.saved.as<uint32_t>()}));
    wg::check_launch("launch batch pass");
  };
  auto both = [&](auto* first, auto* again) {
    pass(first, "pbatch_pass_kernel");
    WG_TIMED("pbatch_scan_kernel", s, pbatch_scan_kernel<<<1, 1024, 0, s>>>(any, b.kept.as<uint32_t>(), b.tiles));
    wg::check_launch("launch batch scan");
    pass(again, "pbatch_redo_kernel");
  };
  auto width = [&](auto w) {
    constexpr int WT = decltype(w)::value;
    if (max_mode == kMaxNone) both(pbatch_pass_kernel<WT, kMaxNone, false>, pbatch_pass_kernel<WT, kMaxNone, true>);
    else if (max_mode == kMaxInf) both(pbatch_pass_kernel<WT, kMaxInf, false>, pbatch_pass_kernel<WT, kMaxInf, true>);
    else both(pbatch_pass_kernel<WT, kMaxFull, false>, pbatch_pass_kernel<WT, kMaxFull, true>);
  };
  if (b.W == 1) width(std::integral_constant<int, 1>{});
  else if (b.W == 2) width(std::integral_constant<int, 2>{});
  else width(std::integral_constant<int, 0>{});
}

}  // namespace

extern "C" {

int wg_products_batch_create(int device, size_t words, size_t n_pairs, const uint64_t* const* lhs_x,
                             const uint64_t* const* lhs_z, const double* const* lhs_c, const size_t* n_lhs,
                             const uint64_t* const* rhs_x, const uint64_t* const* rhs_z,
                             const double* const* rhs_c, const size_t* n_rhs, int mode, double atol, double rtol,
                             wg_products_batch_t* batch, wg_stream_t stream) {
  return wg::guarded([&] {
    if (!batch) wg::throw_invalid("product batch output handle is null");
    *batch = nullptr;
    if (mode != WG_PRODUCTS_SIMPLIFY && mode != WG_PRODUCTS_FUSED)
      wg::throw_invalid("a product batch runs in simplify or fused mode");
    if (mode == WG_PRODUCTS_SIMPLIFY &&
        (atol < 0.0 || rtol < 0.0 || !std::isfinite(atol) || !std::isfinite(rtol)))
      wg::throw_invalid("simplify tolerances must be non-negative finite values");
    if (n_pairs > 0xfffffffeull) wg::throw_invalid("too many pairs in one product batch");
    if (n_pairs > 0 && (!n_lhs || !n_rhs || !lhs_c || !rhs_c || !lhs_x || !lhs_z || !rhs_x || !rhs_z))
      wg::throw_invalid("product batch pointer arrays must not be null");
    wg::DeviceGuard g(device);
    // the caller's operands may still be in flight on its stream
    wg::check_cuda(cudaStreamSynchronize(stream), "synchronize before a product batch");
    std::unique_ptr<wg_products_batch_s> b(new wg_products_batch_s());
    b->device = device;
    b->W = static_cast<int>(words);
    b->mode = mode;
    b->atol = atol;
    b->rtol = rtol;
    b->n_pairs = n_pairs;
    build_batch(*b, lhs_x, lhs_z, lhs_c, n_lhs, rhs_x, rhs_z, rhs_c, n_rhs);
    *batch = b.release();
  });
}

int wg_products_batch_run(wg_products_batch_t batch, wg_stream_t stream) {
  return wg::guarded([&] {
    if (!batch) wg::throw_invalid("product batch is null");
    wg::DeviceGuard g(batch->device);
    run_batch(*batch, stream);
  });
}

int wg_products_batch_result(wg_products_batch_t batch, size_t pair, uint64_t** x, uint64_t** z, double** coeffs,
                             size_t* capacity) {
  return wg::guarded([&] {
    if (!batch) wg::throw_invalid("product batch is null");
    if (pair >= batch->n_pairs) wg::throw_invalid("product batch pair index is out of range");
    const size_t base = batch->seg_base[pair];
    const size_t W = static_cast<size_t>(batch->W);
    if (x) *x = batch->n_seg[pair] && W ? batch->out_x.as<uint64_t>() + base * W : nullptr;
    if (z) *z = batch->n_seg[pair] && W ? batch->out_z.as<uint64_t>() + base * W : nullptr;
    if (coeffs) *coeffs = batch->n_seg[pair] ? batch->out_c.as<double>() + 2 * base : nullptr;
    if (capacity) *capacity = batch->n_seg[pair];
  });
}

int wg_products_batch_counts(wg_products_batch_t batch, uint64_t** counts) {
  return wg::guarded([&] {
    if (!batch) wg::throw_invalid("product batch is null");
    if (!counts) wg::throw_invalid("product batch counts output is null");
    *counts = batch->counts.as<uint64_t>();
  });
}

int wg_products_batch_info(wg_products_batch_t batch, size_t* n_products, size_t* n_keys) {
  return wg::guarded([&] {
    if (!batch) wg::throw_invalid("product batch is null");
    if (n_products) *n_products = batch->N;
    if (n_keys) *n_keys = batch->S;
  });
}

int wg_products_batch_destroy(wg_products_batch_t batch) {
  return wg::guarded([&] {
    if (!batch) return;
    wg::DeviceGuard g(batch->device);
    wg::check_cuda(cudaDeviceSynchronize(), "finish product batch runs");
    delete batch;
  });
}

}  // extern "C"
