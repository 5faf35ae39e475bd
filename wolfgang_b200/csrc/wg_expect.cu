// wg_expect.cu -- x-grouped statevector expectation, its adjoint, and the
// batched persistent form.
//
// Convention (reference src/expectation.cpp:121-150):
//   P|b> = i^y (-1)^{popc(z&b)} |b^x>,  y = popc(x&z),
//   e_k = <psi|P_k|psi> = sum_b conj(psi[b^x]) i^y (-1)^{popc(z&b)} psi[b]  (real),
//   E = sum_k c_k e_k.
// Terms sharing an x-mask form a group: with t_b = conj(psi[b^x]) psi[b] and
// s_k(b) = (-1)^{popc(z_k&b)},
//   e_k = sum_b s_k(b) {Re, -Im, -Re, Im}[y mod 4] t_b.
// b and b^x give the same summand, so half of the b's do where they are known
// apart by a bit above the tile.
//
// Tiles.  The amplitudes are cut into tiles of 2^12 (the low 12 bits of b; of
// 2^n, at least 2^9, for fewer qubits).  Groups whose x agree above the tile
// bits form a class: every group of a class pairs tile J with tile J ^ (x >> 12).
// A CTA keeps tile J in registers, brings the other one into shared memory
// once for all groups of the class, and the next one while it computes
// (before, every group read both from L2).  A group is cut into sub-groups of
// at most 8 terms of even y (which take Re t) and 8 of odd y (Im t).
//
// Forward.  A warp holds 32 x 16 amplitudes of the tile.  The sums of 8 terms
// over them are matrix products: signs (8 terms x 4 amplitudes) times t (4
// amplitudes x 8), FP64 m8n8k4, 16 of them a component whatever the number of
// terms; what is left of the columns is added up with the terms' signs.  A
// sub-group's even and odd terms are taken together, from the same loads.
//
// Adjoint.  (H psi)[j] = sum_g F_g(j^x) psi[j^x].  F's real part at j is an entry
// of a table of the 2^8 sign patterns of the sub-group's even terms, its
// imaginary part one of the odd terms': two 8-byte shared-memory reads an
// amplitude.  The patterns are a linear function of j, the XOR of a word for the
// tile, the warp, the lane and the thread's own amplitudes.
//
// Every partial sum is stored and reduced in a fixed order: results are
// deterministic run to run.

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <numeric>
#include <vector>

#include "wg_common.cuh"

namespace {

using wgd::c128;

constexpr int kThreads = 256;
constexpr int kTotalThreads = 1024;      // of the block that sums up a pair
constexpr uint64_t kJoinSums = 8192;     // partial sums
constexpr size_t kJoinTerms = 512;       // and terms of a pair up to which that block also sums its terms
constexpr int kTileBits = 12;            // amplitudes per tile: 2^12 at most
constexpr int kTileMin = 9;              // and 2^9 at least (zeros above 2^n)
constexpr int kTileMax = 1 << kTileBits;
constexpr int kPiece = 8;                // terms per sub-group of either parity of y
constexpr int kSegSubs = 16;             // sub-groups of one class staged at a time (adjoint)
constexpr int kSegEntries = 2048;        // and their table entries
constexpr int kChunkPieces = 128;        // pieces of one forward item
constexpr int kFwdThreads = 512;         // two sets of 256 x 16 amplitudes = a tile
constexpr int kFwdInner = 8;             // warps of a set
constexpr int kAdjThreads = 512;         // x 8 amplitudes = a tile
// Least work of a split, in the costs of make_plan (a sub-group 90): its sums are written
// and read again.  Half of it where these are less than a whole tile's.
constexpr uint32_t kSplitCost = 400;
constexpr uint32_t kDiagFlag = 4;        // ty bit: the term's group has x == 0
constexpr uint32_t kTwiceFlag = 8;       // ty bit: the forward pass meets every pair of the group twice

// A piece of a sub-group: terms [t0, t0 + nk), all of even or all of odd y.
struct __align__(16) FwdPiece {
  uint32_t xlo;              // x within the tile
  uint32_t xhi;              // and above it
  uint32_t t0;
  uint8_t nk, odd;
  uint8_t pair;              // even terms, and the next piece has the sub-group's odd ones: taken together
  uint8_t turn;              // the set of threads that takes it
  uint32_t zlo[kPiece];      // z within the tile
  uint32_t zhi[kPiece];      // and above it
};
static_assert(sizeof(FwdPiece) == 80, "copied in 16-byte pieces");
constexpr uint32_t kReads = 0x80000000u;  // chunk bit: its pieces read psi themselves

// A sub-group: terms [t0, t0 + nre) of even y, then nim of odd y.  A sign word has the even terms' signs in bits
// 3-10, the odd ones' in bits 19-26: byte offsets into the tables.
struct __align__(16) AdjSub {
  uint32_t xlo;
  uint32_t tab;              // first entry of its tables: 2^nre, then 2^nim
  uint32_t t0;
  uint16_t nre, nim;
  uint32_t mixed;            // some coefficient is neither real nor imaginary (set with the coefficients)
  uint32_t pad[3];
  uint32_t zhi[2 * kPiece];  // z above the tile
  uint32_t own[8];           // signs for the thread's amplitudes (tile bits m-3 to m-1)
  uint32_t warp[16];         // for tile bits 5 to m-4
  uint32_t lane[32];         // for tile bits 0-4
};
static_assert(sizeof(AdjSub) == 320, "copied in 16-byte pieces");

// Consecutive sub-groups of one class.
struct __align__(16) SegDev {
  uint32_t xhi;          // x above the tile
  uint32_t s0, subs;     // sub-groups [s0, s0 + subs)
  uint32_t tab, entries; // their table entries
  uint32_t pad[3];
};

// Device-side description of one operator (kernel parameter, by value).
struct PlanDev {
  int n, m;                  // qubits, tile bits
  uint32_t T, G, S, NP, NS;  // terms, groups, sub-groups, pieces, segments
  uint32_t tiles;            // 2^(n - m)
  uint32_t chunks, ranges;   // forward items: chunks of pieces x ranges of tiles
  uint32_t splits;           // parts of the segments that an adjoint tile is split into
  uint32_t joined;           // one block sums the partial sums of all terms and E
  const FwdPiece* piece;     // [NP]
  AdjSub* asub;              // [S]
  const SegDev* seg;         // [NS]
  const uint32_t* chunk;     // [chunks + 1] first piece of a chunk | kReads
  const uint32_t* bounds;    // [splits + 1] segments of the splits
  const uint32_t* ty;        // [T] y mod 4 | flags
  const uint32_t* torig;     // [T] original index of sorted term
  double* coeffs;            // [2T] original-order coefficients
  double* table;             // adjoint tables of the part of c_k (-i)^y that its y makes it
                             // (real where y is even)
  double* other;             // and of the other part (read where AdjSub::mixed)
  double* partial;           // [T][ranges] forward partial sums
};

struct wg_plan_host {
  int device;
  PlanDev dev;
  size_t n_groups = 0;
  uint32_t chunk_most = 0;   // pieces of the largest chunk
  uint64_t tile_cost = 0;    // the adjoint's work on a tile, in SegDev's costs
  wg::Scratch mem;  // all of the above
};

}  // namespace

struct wg_expect_plan_s {
  wg_plan_host h;
};

namespace {

template <typename Amp>
__device__ __forceinline__ c128 load_amp(const void* psi, uint64_t i);

template <>
__device__ __forceinline__ c128 load_amp<double2>(const void* psi, uint64_t i) {
  const double2 v = __ldg(static_cast<const double2*>(psi) + i);
  return {v.x, v.y};
}

template <>
__device__ __forceinline__ c128 load_amp<float2>(const void* psi, uint64_t i) {
  const float2 v = __ldg(static_cast<const float2*>(psi) + i);
  return {static_cast<double>(v.x), static_cast<double>(v.y)};
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// One (operator, statevector) pair of a launch.
struct PairDev {
  PlanDev plan;
  const void* psi;
  double* evals;    // e_k outputs (original order); null where the plan joins its sums and nobody asked
  double* result;   // E output or null
  double* hpsi;     // H psi output or null
  double2* part;    // splits x 2^n partial H psi, or null
  uint32_t group;   // chunks of a forward item
  uint32_t per_range;  // forward items of a range of tiles
  uint64_t fold;    // an adjoint item takes all splits of its tile, one after another
};

// A launch over one or several pairs (kernel parameter).  A single pair travels in
// the parameter itself: nothing to allocate, copy or free for a call.
struct BatchDev {
  const PairDev* pairs;       // [np], null for a single one
  const uint64_t* item_base;  // [np+1] forward items per pair
  const uint64_t* term_base;  // [np+1] flat term offsets (0 for pairs whose sums are joined)
  const uint64_t* tile_base;  // [np+1] adjoint items (0 for pairs without H psi): tiles x splits
  const uint64_t* amp_base;   // [np+1] amplitudes of the pairs whose adjoint is split
  unsigned long long* counters;  // [2] forward / adjoint work queues; null: an item for every CTA
  uint32_t np;
  uint64_t n_items, n_terms, n_tiles, n_amps;
  PairDev one;
  __device__ __forceinline__ const PairDev& pair(uint32_t p) const { return pairs ? pairs[p] : one; }
};

template <typename T>
__device__ __forceinline__ uint32_t upper_index(const T* base, uint32_t n, T v) {
  // last i in [0, n) with base[i] <= v (base[0] <= v assumed)
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (base[mid] <= v) lo = mid;
    else hi = mid;
  }
  return lo;
}

// The pair that flat index v belongs to; v becomes the index within the pair.
__device__ __forceinline__ uint32_t find_pair(const BatchDev& B, const uint64_t* base, uint64_t& v) {
  if (!B.pairs) return 0;
  const uint32_t p = upper_index<uint64_t>(base, B.np + 1, v);
  v -= base[p];
  return p;
}

__device__ __forceinline__ void copy_pair(PairDev& to, const PairDev& from) {
  static_assert(sizeof(PairDev) % 8 == 0, "copied in 8-byte pieces");
  if (threadIdx.x < sizeof(PairDev) / 8)
    reinterpret_cast<uint64_t*>(&to)[threadIdx.x] = reinterpret_cast<const uint64_t*>(&from)[threadIdx.x];
}

// ------------------------------------------------------------- tiles

template <int BYTES>
__device__ __forceinline__ void copy_async(void* to, const void* from) {
  const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(to));
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(from) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(a), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// Two tile buffers.  complex128 amplitudes are copied as they are, the next
// tile into the other buffer; complex64 ones are copied into the halves of the
// second buffer by turns and widened from there into the first (once for all
// groups of a class: the conversions would cost as much as the products).
template <typename Amp>
struct TileBuffers {
  static constexpr bool kWide = sizeof(Amp) == 16;
  double2* b0;
  double2* b1;
  int cur = 0;

  // starts the copy of tile J (2^m amplitudes from J << m on, of 2^n); the
  // caller commits
  __device__ __forceinline__ void fetch(const void* psi, uint64_t J, int m, int n, int slot) {
    const uint64_t base = J << m;
    const int size = 1 << m, have = n < m ? 1 << n : size;
    const Amp* from = static_cast<const Amp*>(psi) + base;
    if constexpr (kWide) {
      double2* to = slot ? b1 : b0;
      for (int i = threadIdx.x; i < size; i += blockDim.x) {
        if (i < have) copy_async<16>(to + i, from + i);
        else to[i] = make_double2(0.0, 0.0);
      }
    } else {
      float2* to = reinterpret_cast<float2*>(b1) + slot * kTileMax;
      for (int i = threadIdx.x; i < size; i += blockDim.x) {
        if (i < have) copy_async<8>(to + i, from + i);
        else to[i] = make_float2(0.0f, 0.0f);
      }
    }
  }
  // complex64: the fetched tile, widened (all copies of this thread are done;
  // each thread widens what it fetched)
  __device__ __forceinline__ void widen(int m, int slot) {
    const float2* from = reinterpret_cast<const float2*>(b1) + slot * kTileMax;
    for (int i = threadIdx.x; i < (1 << m); i += blockDim.x) {
      const float2 v = from[i];
      b0[i] = make_double2(static_cast<double>(v.x), static_cast<double>(v.y));
    }
  }
};

// v with its sign flipped where bit 31 of `sign` is set
__device__ __forceinline__ double flip(double v, uint32_t sign) {
  return __hiloint2double(__double2hiint(v) ^ static_cast<int>(sign & 0x80000000u), __double2loint(v));
}
// ------------------------------------------------------------- forward

struct FwdShared {
  double2 tile[2][kTileMax];
  double acc[kFwdInner][kChunkPieces * kPiece];  // by warp, piece and term
  FwdPiece piece[kChunkPieces];
  uint32_t seg_xhi[kChunkPieces];
  uint32_t seg_at[kChunkPieces + 1];
  uint32_t segs, reads;
  unsigned long long item;
  PairDev pair;
};
static_assert(sizeof(FwdShared) <= 227 * 1024, "shared memory of an SM");

// C (8 x 8) += A (8 x 4) B (4 x 8) in FP64.  Lane l holds A[l / 4][l % 4],
// B[l % 4][l / 4] and C[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double& c0, double& c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// Where a thread's amplitudes lie in a tile of 2^m: M is m where it is known
// at compile time (12 bits: the shifts become constants), else 0.
template <int M>
struct Layout {
  int m_;
  __device__ __forceinline__ int m() const { return M ? M : m_; }
  __device__ __forceinline__ uint32_t off16(int r) const { return static_cast<uint32_t>(r) << (m() - 4); }
  __device__ __forceinline__ uint32_t off8(int r) const { return static_cast<uint32_t>(r) << (m() - 3); }
};

// Signs of a piece's terms for the products: the lane's term is lane / 4.
struct TermSigns {
  uint32_t zlo, one, e0, e1, e2;
  __device__ __forceinline__ TermSigns(const FwdPiece& pd, uint32_t J, uint32_t where, int m, int lane) {
    constexpr uint32_t kSign = 0x80000000u;
    zlo = pd.zlo[lane >> 2];
    one = 0x3ff00000u ^ (static_cast<uint32_t>(__popc((zlo & where) ^ (pd.zhi[lane >> 2] & J))) << 31);
    e0 = (zlo << (35 - m)) & kSign;
    e1 = (zlo << (34 - m)) & kSign;
    e2 = (zlo << (33 - m)) & kSign;
  }
  // +-1 for step k of the inner bits
  __device__ __forceinline__ double at(int k) const {
    uint32_t hi = one;
    if (k & 1) hi ^= e0;
    if (k & 2) hi ^= e1;
    if (k & 4) hi ^= e2;
    return __hiloint2double(static_cast<int>(hi), 0);
  }
};

// Adds a piece's sums over tile J to acc[0..7] (kParts 1: even terms, 2: odd ones), or a pair's to those and the
// next eight (3): a is the thread's part of tile J, load the tile that x pairs it with.  Amplitude bits of the
// tile: 0-1 lane % 4 (the products' inner index, with t's bits m-4 to m-2), 2-4 lane / 4 (the columns, with t's
// bit m-1), 5 to m-5 the warp.  An amplitude's products follow its load at once: four independent chains of a
// pair keep the pipe busy while the next loads are under way.
template <int M, int kParts, class Load>
__device__ __forceinline__ void forward_unit(const Layout<M>& lay, const FwdPiece* pd, const Load& load,
                                             const c128 (&a)[16], uint32_t J, int tt, int lane, double* acc) {
  const int m = lay.m();
  const uint32_t at = static_cast<uint32_t>(tt) ^ pd->xlo, where = static_cast<uint32_t>(tt) & ~28u;
  constexpr int kCount = kParts == 3 ? 2 : 1;
  const TermSigns first(pd[0], J, where, m, lane), second(pd[kCount - 1], J, where, m, lane);
  double c[kCount][4] = {};
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double s0 = first.at(k), s1 = kCount == 2 ? second.at(k) : 0.0;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int q = k + 8 * half;
      const double2 v = load(at ^ lay.off16(q));
      const double re = fma(v.x, a[q].re, v.y * a[q].im), im = fma(v.x, a[q].im, -(v.y * a[q].re));
      mma_f64(c[0][2 * half], c[0][2 * half + 1], s0, kParts == 2 ? im : re);
      if constexpr (kCount == 2) mma_f64(c[1][2 * half], c[1][2 * half + 1], s1, im);
    }
  }
#pragma unroll
  for (int i = 0; i < kCount; ++i) {
    const uint32_t zlo = i ? second.zlo : first.zlo, bit2 = zlo << 29;
    double v = (c[i][0] + flip(c[i][1], bit2)) + flip(c[i][2] + flip(c[i][3], bit2), zlo << (32 - m));
    v = flip(v, static_cast<uint32_t>(__popc((zlo >> 3) & (lane & 3))) << 31);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    if ((lane & 3) == 0) acc[kPiece * i + (lane >> 2)] += v;
  }
}

template <int M, class Load>
__device__ __forceinline__ void forward_any(const Layout<M>& lay, const FwdPiece* pd, const Load& load,
                                            const c128 (&a)[16], uint32_t J, int tt, int lane, double* acc) {
  if (pd->pair) forward_unit<M, 3>(lay, pd, load, a, J, tt, lane, acc);
  else if (pd->odd) forward_unit<M, 2>(lay, pd, load, a, J, tt, lane, acc);
  else forward_unit<M, 1>(lay, pd, load, a, J, tt, lane, acc);
}

// A CTA takes (chunk of pieces, range of tiles) items.  24 qubits, 20,000 terms
// in 1,699 groups: 40 ms (87 ms with 16 masked sums a pair; 50 ms with a piece's
// loads before its products, the parities apart and 32 pieces a chunk); 20
// qubits, 4,096 terms in 2,526 groups: 2.0 ms (4.5).  Bound by the FP64 pipe, 61 %
// busy (47 % products, 14 % the t's): four warps a scheduler (tile J takes half of
// the registers) do not cover all of the chains' latency.
template <typename Amp>
__global__ void __launch_bounds__(kFwdThreads, 1) expect_forward_kernel(const __grid_constant__ BatchDev B) {
  extern __shared__ __align__(16) unsigned char raw[];
  FwdShared& sh = *reinterpret_cast<FwdShared*>(raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (uint64_t turn = blockIdx.x;; turn += gridDim.x) {
    __syncthreads();
    uint64_t item = turn;
    if (B.counters) {
      if (tid == 0) sh.item = atomicAdd(B.counters, 1ull);
      __syncthreads();
      item = sh.item;
    }
    if (item >= B.n_items) break;
    copy_pair(sh.pair, B.pair(find_pair(B, B.item_base, item)));
    __syncthreads();
    const PairDev& Q = sh.pair;
    const PlanDev& P = Q.plan;
    const void* psi = Q.psi;
    const uint32_t r = static_cast<uint32_t>(item);
    // ranges outermost: the CTAs that run together meet the same tiles in L2
    const uint32_t range = r / Q.per_range, chunk = (r - range * Q.per_range) * Q.group;
    const uint32_t taken = min(Q.group, P.chunks - chunk);
    const uint32_t piece0 = P.chunk[chunk] & ~kReads, pieces = (P.chunk[chunk + taken] & ~kReads) - piece0;
    const int m = P.m, n = P.n;
    const uint32_t J0 = static_cast<uint32_t>(static_cast<uint64_t>(P.tiles) * range / P.ranges);
    const uint32_t J1 = static_cast<uint32_t>(static_cast<uint64_t>(P.tiles) * (range + 1) / P.ranges);
    // the chunk's pieces, and its runs of equal xhi
    {
      const uint4* from = reinterpret_cast<const uint4*>(P.piece + piece0);
      uint4* to = reinterpret_cast<uint4*>(sh.piece);
      for (uint32_t i = tid; i < pieces * (sizeof(FwdPiece) / 16); i += kFwdThreads) to[i] = from[i];
      for (uint32_t i = lane; i < pieces * kPiece; i += 32)
        if (warp < kFwdInner) sh.acc[warp][i] = 0.0;
      if (warp == kFwdInner) {
        uint32_t segs = 0, reads = kReads;  // of all of the item's chunks
#pragma unroll 1  // unrolled it cost the whole kernel 1 to 2 % (code placement)
        for (uint32_t c = lane; c < taken; c += 32) reads &= P.chunk[chunk + c];
        for (uint32_t at = 0; at < pieces; at += 32) {
          const uint32_t i = at + lane;
          const bool in = i < pieces;
          const uint32_t xhi = in ? P.piece[piece0 + i].xhi : 0;
          const bool head = in && (i == 0 || xhi != P.piece[piece0 + i - 1].xhi);
          const uint32_t heads = __ballot_sync(0xffffffffu, head);
          if (head) {
            const uint32_t to = segs + __popc(heads & ((1u << lane) - 1u));
            sh.seg_xhi[to] = xhi;
            sh.seg_at[to] = i;
          }
          segs += __popc(heads);
        }
        const bool all = __all_sync(0xffffffffu, (reads & kReads) != 0);
        if (lane == 0) {
          sh.reads = all;
          sh.segs = segs;
          sh.seg_at[segs] = pieces;
        }
      }
    }
    __syncthreads();
    const uint32_t segs = sh.segs;
    // thread tt of the tile holds amplitudes tt + (q << m-4); the sets of
    // threads (two for tiles of 2^12, more for smaller ones) take a piece each
    const int tt = tid & ((1 << (m - 4)) - 1);
    const uint32_t slice = tid >> (m - 4);
    c128 a[16];
    auto load_own = [&](uint32_t J) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const uint64_t b = (static_cast<uint64_t>(J) << m) + tt + (static_cast<uint32_t>(q) << (m - 4));
        a[q] = (b >> n) == 0 ? load_amp<Amp>(psi, b) : c128{0.0, 0.0};
      }
    };
    double* const acc = sh.acc[tt >> 5];
    // a segment with x above the tile pairs J with J ^ xhi once, from the side
    // whose lowest bit of xhi is clear
    auto this_side = [](uint32_t J, uint32_t xhi) { return xhi == 0 || !((J >> (__ffs(static_cast<int>(xhi)) - 1)) & 1u); };
    if (sh.reads) {
      // hardly two pieces of a class: each reads the paired tile itself, and
      // nothing waits for the others
      for (uint32_t J = J0; J < J1; ++J) {
        load_own(J);
        for (uint32_t i = 0; i < pieces; i += sh.piece[i].pair ? 2 : 1) {
          const FwdPiece* pd = sh.piece + i;
          if (pd->turn != slice || !this_side(J, pd->xhi)) continue;
          const Amp* from = static_cast<const Amp*>(psi) + (static_cast<uint64_t>(J ^ pd->xhi) << kTileBits);
          auto load = [&](uint32_t i) {
            const c128 v = load_amp<Amp>(from, i);
            return make_double2(v.re, v.im);
          };
          forward_any(Layout<kTileBits>{kTileBits}, pd, load, a, J, tt, lane, acc + kPiece * i);
        }
      }
    } else {
      // (tile, segment) steps
      auto next_step = [&](uint32_t& J, uint32_t& g) {
        while (J < J1) {
          for (; g < segs; ++g)
            if (this_side(J, sh.seg_xhi[g])) return true;
          g = 0;
          ++J;
        }
        return false;
      };
      TileBuffers<Amp> buf{sh.tile[0], sh.tile[1]};
      constexpr bool kWide = TileBuffers<Amp>::kWide;
      uint32_t J = J0, g = 0, have = 0xffffffffu;
      bool more = next_step(J, g);
      int slot = 0;
      if (more) buf.fetch(psi, J ^ sh.seg_xhi[g], m, n, 0);
      copy_commit();
      while (more) {
        uint32_t Jn = J, gn = g + 1;
        const bool more_n = next_step(Jn, gn);
        if (more_n) buf.fetch(psi, Jn ^ sh.seg_xhi[gn], m, n, slot ^ 1);
        copy_commit();
        if (have != J) {
          have = J;
          load_own(J);
        }
        copy_wait<1>();
        if (!kWide) buf.widen(m, slot);
        __syncthreads();
        const double2* src = kWide && slot ? buf.b1 : buf.b0;
        auto load = [&](uint32_t i) { return src[i]; };
        const uint32_t i1 = sh.seg_at[g + 1];
        for (uint32_t i = sh.seg_at[g]; i < i1; i += sh.piece[i].pair ? 2 : 1) {
          const FwdPiece* pd = sh.piece + i;
          if (pd->turn != slice) continue;
          if (m == kTileBits) forward_any(Layout<kTileBits>{m}, pd, load, a, J, tt, lane, acc + kPiece * i);
          else forward_any(Layout<0>{m}, pd, load, a, J, tt, lane, acc + kPiece * i);
        }
        __syncthreads();
        J = Jn;
        g = gn;
        more = more_n;
        slot ^= 1;
      }
    }
    copy_wait<0>();
    __syncthreads();
    for (uint32_t k = tid; k < pieces * kPiece; k += kFwdThreads) {
      const FwdPiece& pd = sh.piece[k / kPiece];
      if (k % kPiece >= pd.nk) continue;
      double s = 0.0;
#pragma unroll
      for (int v = 0; v < kFwdInner; ++v) s += sh.acc[v][k];
      P.partial[static_cast<uint64_t>(pd.t0 + k % kPiece) * P.ranges + range] = s;
    }
  }
}

// e_k from the sum over all pairs
__device__ __forceinline__ double scaled(double s, uint32_t ty) {
  const double e = ((ty & 3u) == 1 || (ty & 3u) == 2) ? -s : s;
  return ty & (kDiagFlag | kTwiceFlag) ? e : 2.0 * e;
}

// e_k from the ranges' partial sums, scaled by the pairing factor, by eight lanes
// in a fixed order (one thread took 17 us for 256 ranges); every lane gets it.
__device__ __forceinline__ double term_value(const PlanDev& P, uint32_t k, uint32_t lane8) {
  const double* part = P.partial + static_cast<uint64_t>(k) * P.ranges;
  double s = 0.0;
#pragma unroll 8
  for (uint32_t c = lane8; c < P.ranges; c += 8) s += part[c];
#pragma unroll
  for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return scaled(s, P.ty[k]);
}

// The term values in original order; flat over the terms of the pairs whose sums
// are not joined.
__global__ void __launch_bounds__(kThreads) expect_finish_terms_kernel(const __grid_constant__ BatchDev B) {
  const uint32_t lane8 = threadIdx.x & 7;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x / 8;
  const uint64_t first = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) / 8;
  for (uint64_t f0 = first; f0 - (threadIdx.x & 31) / 8 < B.n_terms; f0 += stride) {  // a warp leaves together
    uint64_t k = min(f0, B.n_terms - 1);
    const PairDev& Q = B.pair(find_pair(B, B.term_base, k));
    const double e = term_value(Q.plan, static_cast<uint32_t>(k), lane8);
    if (lane8 == 0 && f0 < B.n_terms) Q.evals[Q.plan.torig[k]] = e;
  }
}

// E_p = sum_k c_k e_k, one block per pair, tree reduction in a fixed order; where
// the plan says so, the term values too.
__global__ void __launch_bounds__(kTotalThreads) expect_total_kernel(const __grid_constant__ BatchDev B) {
  __shared__ double sre[kTotalThreads / 32], sim[kTotalThreads / 32];
  for (uint32_t p = blockIdx.x; p < B.np; p += gridDim.x) {
    const PairDev& Q = B.pair(p);
    const PlanDev& P = Q.plan;
    if (!Q.result && !P.joined) continue;
    double re = 0.0, im = 0.0;
    if (P.joined && P.ranges < 8) {
      for (uint32_t k = threadIdx.x; k < P.T; k += kTotalThreads) {
        double s = 0.0;
        for (uint32_t c = 0; c < P.ranges; ++c) s += P.partial[static_cast<uint64_t>(k) * P.ranges + c];
        const double e = scaled(s, P.ty[k]);
        const uint32_t o = P.torig[k];
        if (Q.evals) Q.evals[o] = e;
        re += P.coeffs[2 * o] * e;
        im += P.coeffs[2 * o + 1] * e;
      }
    } else if (P.joined) {
      const uint32_t lane8 = threadIdx.x & 7;
      for (uint32_t k0 = threadIdx.x / 8; k0 - (threadIdx.x & 31) / 8 < P.T; k0 += kTotalThreads / 8) {
        const uint32_t k = min(k0, P.T - 1);
        const double e = term_value(P, k, lane8);
        if (lane8 != 0 || k0 >= P.T) continue;
        const uint32_t o = P.torig[k];
        if (Q.evals) Q.evals[o] = e;
        re += P.coeffs[2 * o] * e;
        im += P.coeffs[2 * o + 1] * e;
      }
    } else {
      for (uint32_t k = threadIdx.x; k < P.T; k += kTotalThreads) {
        re += P.coeffs[2 * k] * Q.evals[k];
        im += P.coeffs[2 * k + 1] * Q.evals[k];
      }
    }
    __syncwarp();
    re = warp_sum(re);
    im = warp_sum(im);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
      sre[warp] = re;
      sim[warp] = im;
    }
    __syncthreads();
    if (warp == 0) {
      re = lane < kTotalThreads / 32 ? sre[lane] : 0.0;
      im = lane < kTotalThreads / 32 ? sim[lane] : 0.0;
      re = warp_sum(re);
      im = warp_sum(im);
      if (lane == 0 && Q.result) {
        Q.result[0] = re;
        Q.result[1] = im;
      }
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------- adjoint

struct AdjStage {
  AdjSub sub[kSegSubs];
  double table[kSegEntries];
};

struct AdjShared {
  double2 tile[2][kTileMax];
  AdjStage stage[2];
  unsigned long long item;
  PairDev pair;
};
static_assert(sizeof(AdjShared) <= 227 * 1024, "shared memory of an SM");

__device__ __forceinline__ double entry(const double* table, uint32_t bytes) {
  return *reinterpret_cast<const double*>(reinterpret_cast<const char*>(table) + bytes);
}

// Adds one sub-group's share of H psi in tile J to the thread's 8 amplitudes.
// table: its staged tables; other: its tables of the other parts, in memory.
template <int M>
__device__ __forceinline__ void adjoint_sub(const Layout<M>& lay, const AdjSub& sd, const double* table,
                                            const double* other, const double2* src, c128 (&acc)[8], uint32_t J,
                                            int tt, int lane) {
  constexpr uint32_t kOffsets = 8 * 255u;
  // lanes 0-7 and 16-23 give the signs of the terms in the tile
  const uint32_t mine = lane & 8 ? 0u : sd.zhi[(lane & 7) | ((lane & 16) >> 1)];
  const uint32_t S = (__ballot_sync(0xffffffffu, __popc(mine & J) & 1) << 3) ^ sd.lane[lane] ^ sd.warp[tt >> 5];
  const uint32_t nre = sd.nre, nim = sd.nim;
  const uint32_t at = static_cast<uint32_t>(tt) ^ sd.xlo;
  const double* tim = table + (1u << nre);
  const uint4 o0 = reinterpret_cast<const uint4*>(sd.own)[0], o1 = reinterpret_cast<const uint4*>(sd.own)[1];
  const uint32_t own[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
  if (sd.mixed) {
    // complex coefficients: both tables add to both parts of F
    const double* oim = other + (1u << nre);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t q = S ^ own[r], qr = q & kOffsets, qi = (q >> 16) & kOffsets;
      const double fre = entry(table, qr) + entry(oim, qi), fim = entry(tim, qi) + entry(other, qr);
      const double2 v = src[at ^ lay.off8(r)];
      acc[r].re = fma(-v.y, fim, fma(v.x, fre, acc[r].re));
      acc[r].im = fma(v.y, fre, fma(v.x, fim, acc[r].im));
    }
  } else if (nim == 0) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const double fre = entry(table, (S ^ own[r]) & kOffsets);
      const double2 v = src[at ^ lay.off8(r)];
      acc[r].re = fma(v.x, fre, acc[r].re);
      acc[r].im = fma(v.y, fre, acc[r].im);
    }
  } else if (nre == 0) {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const double fim = entry(tim, ((S ^ own[r]) >> 16) & kOffsets);
      const double2 v = src[at ^ lay.off8(r)];
      acc[r].re = fma(-v.y, fim, acc[r].re);
      acc[r].im = fma(v.x, fim, acc[r].im);
    }
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t q = S ^ own[r];
      const double fre = entry(table, q & kOffsets), fim = entry(tim, (q >> 16) & kOffsets);
      const double2 v = src[at ^ lay.off8(r)];
      acc[r].re = fma(-v.y, fim, fma(v.x, fre, acc[r].re));
      acc[r].im = fma(v.y, fre, fma(v.x, fim, acc[r].im));
    }
  }
}

// Output-stationary: a CTA owns tile J of H psi, 8 amplitudes a thread, and
// walks the segments of its split.  Bound by shared-memory wavefronts (78 % of
// the cycles; 8 an amplitude and sub-group at least: 4 for psi, 2 for either
// table): 44 ms on 24 qubits with 20,000 terms (80 ms with tables of complex
// entries and psi read through L1).
template <typename Amp>
__global__ void __launch_bounds__(kAdjThreads, 1) expect_adjoint_kernel(const __grid_constant__ BatchDev B) {
  extern __shared__ __align__(16) unsigned char raw[];
  AdjShared& sh = *reinterpret_cast<AdjShared*>(raw);
  const int tid = threadIdx.x, lane = tid & 31;
  constexpr bool kWide = TileBuffers<Amp>::kWide;
  for (uint64_t turn = blockIdx.x;; turn += gridDim.x) {
    __syncthreads();
    uint64_t item = turn;
    if (B.counters) {
      if (tid == 0) sh.item = atomicAdd(B.counters + 1, 1ull);
      __syncthreads();
      item = sh.item;
    }
    if (item >= B.n_tiles) break;
    copy_pair(sh.pair, B.pair(find_pair(B, B.tile_base, item)));
    __syncthreads();
    const PairDev& Q = sh.pair;
    const PlanDev& P = Q.plan;
    const void* psi = Q.psi;
    const uint32_t splits = P.splits, parts = Q.fold ? 1 : splits;  // items of a tile
    // tiles outermost: the CTAs that run together share tiles and segments
    const uint32_t J = static_cast<uint32_t>(item / parts);
    uint32_t split = static_cast<uint32_t>(item - static_cast<uint64_t>(J) * parts);
    const uint32_t g0 = P.bounds[split], g1 = P.bounds[Q.fold ? splits : split + 1];
    uint32_t split_end = P.bounds[split + 1];
    const int m = P.m, n = P.n;
    const int tt = tid & ((1 << (m - 3)) - 1);
    const uint32_t slice = tid >> (m - 3), slices = kAdjThreads >> (m - 3);
    TileBuffers<Amp> buf{sh.tile[0], sh.tile[1]};
    auto fetch_stage = [&](const SegDev& sg, int slot) {
      AdjStage& st = sh.stage[slot];
      const char* from = reinterpret_cast<const char*>(P.asub + sg.s0);
      char* to = reinterpret_cast<char*>(st.sub);
      for (uint32_t i = tid; i < sg.subs * (sizeof(AdjSub) / 16); i += kAdjThreads)
        copy_async<16>(to + 16 * i, from + 16 * i);
      for (uint32_t i = tid; i < sg.entries / 2; i += kAdjThreads)
        copy_async<16>(st.table + 2 * i, P.table + sg.tab + 2 * i);
    };
    c128 acc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = {0.0, 0.0};
    int slot = 0, stage = 0;
    SegDev sg = P.seg[g0], nx = P.seg[min(g0 + 1, g1 - 1)];
    buf.fetch(psi, J ^ sg.xhi, m, n, 0);
    fetch_stage(sg, 0);
    copy_commit();
    bool fresh = true;  // the segment's tile is not the one before's
    for (uint32_t g = g0; g < g1; ++g) {
      const bool last = g + 1 == g1;
      const SegDev after = P.seg[min(g + 2, g1 - 1)];  // a step ahead of its use
      const bool fresh_n = !last && nx.xhi != sg.xhi;
      if (fresh_n) buf.fetch(psi, J ^ nx.xhi, m, n, slot ^ 1);
      if (!last) fetch_stage(nx, stage ^ 1);
      copy_commit();
      copy_wait<1>();
      if (!kWide && fresh) buf.widen(m, slot);
      __syncthreads();
      const double2* src = kWide && slot ? buf.b1 : buf.b0;
      const AdjStage& st = sh.stage[stage];
      if (m == kTileBits) {
        const Layout<kTileBits> lay{m};
        for (uint32_t i = 0; i < sg.subs; ++i) {
          const AdjSub& sd = st.sub[i];
          adjoint_sub(lay, sd, st.table + (sd.tab - sg.tab), P.other + sd.tab, src, acc, J, tt, lane);
        }
      } else {
        const Layout<0> lay{m};
        for (uint32_t i = 0; i < sg.subs; ++i) {
          if ((i & (slices - 1)) != slice) continue;
          const AdjSub& sd = st.sub[i];
          adjoint_sub(lay, sd, st.table + (sd.tab - sg.tab), P.other + sd.tab, src, acc, J, tt, lane);
        }
      }
      __syncthreads();
      if (g + 1 == split_end) {
        // the split's sums: stored, or added to those of the splits before (the order of expect_join_kernel)
        if (slices > 1) {
          // the slices' sums, slice by slice, behind the tile (what is fetched meanwhile lies in front)
          if (slice > 0) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const uint32_t j = tt + (static_cast<uint32_t>(r) << (m - 3));
              sh.tile[0][(slice << m) + j] = make_double2(acc[r].re, acc[r].im);
            }
          }
          __syncthreads();
          if (slice == 0) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const uint32_t j = tt + (static_cast<uint32_t>(r) << (m - 3));
              for (uint32_t v = 1; v < slices; ++v) {
                const double2 o = sh.tile[0][(v << m) + j];
                acc[r].re += o.x;
                acc[r].im += o.y;
              }
            }
          }
        }
        if (slice == 0) {
          double2* out = parts > 1 ? Q.part + (static_cast<uint64_t>(split) << n) : reinterpret_cast<double2*>(Q.hpsi);
          const bool add = parts == 1 && split > 0;
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            const uint64_t j = (static_cast<uint64_t>(J) << m) + tt + (static_cast<uint32_t>(r) << (m - 3));
            if ((j >> n) != 0) continue;
            double2 v = make_double2(acc[r].re, acc[r].im);
            if (add) {
              const double2 before = out[j];
              v.x += before.x;
              v.y += before.y;
            }
            out[j] = v;
          }
        }
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r] = {0.0, 0.0};
        ++split;
        if (!last) split_end = P.bounds[split + 1];
      }
      if (fresh_n) slot ^= 1;
      fresh = fresh_n;
      stage ^= 1;
      sg = nx;
      nx = after;
    }
    copy_wait<0>();
  }
}

// H psi of the pairs whose segments were split, summed over the splits in order.
__global__ void __launch_bounds__(kThreads) expect_join_kernel(const __grid_constant__ BatchDev B) {
  for (uint64_t f = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; f < B.n_amps;
       f += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    uint64_t j = f;
    const PairDev& Q = B.pair(find_pair(B, B.amp_base, j));
    const double2* part = Q.part + j;
    const uint32_t splits = Q.plan.splits;
    const int n = Q.plan.n;
    double2 s = part[0];
#pragma unroll 8
    for (uint32_t k = 1; k < splits; ++k) {
      const double2 v = part[static_cast<uint64_t>(k) << n];
      s.x += v.x;
      s.y += v.y;
    }
    reinterpret_cast<double2*>(Q.hpsi)[j] = s;
  }
}

// ------------------------------------------------------------- plan build

// The adjoint's tables from the coefficients, a warp per sub-group: entry q of
// a piece is the sum of its terms' c_k (-i)^y_k (i^y, and (-1)^y for the signs,
// which are those at j where the adjoint needs them at j ^ x), with the sign of
// bit kk of q, in order.  The coefficients come from `from` (original order,
// `reals` doubles each) and go to the plan too: every term lies in one sub-group.
__global__ void plan_tables_kernel(PlanDev P, const double* __restrict__ from, int reals) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < P.S; i += (gridDim.x * blockDim.x) >> 5) {
    AdjSub& sd = P.asub[i];
    // lane kk holds term kk of the sub-group
    double own = 0.0, other = 0.0;
    if (lane < static_cast<uint32_t>(sd.nre) + sd.nim) {
      const uint32_t k = sd.t0 + lane, o = P.torig[k];
      const c128 c = reals == 2 ? c128{from[2 * static_cast<size_t>(o)], from[2 * static_cast<size_t>(o) + 1]}
                                : c128{from[o], 0.0};
      P.coeffs[2 * static_cast<size_t>(o)] = c.re;
      P.coeffs[2 * static_cast<size_t>(o) + 1] = c.im;
      const c128 d = wgd::rotate(c, (4u - (P.ty[k] & 3u)) & 3u);
      const bool odd = P.ty[k] & 1u;
      own = odd ? d.im : d.re;
      other = odd ? d.re : d.im;
    }
    const bool mixed = __any_sync(0xffffffffu, other != 0.0);  // true for a NaN
    if (lane == 0) sd.mixed = mixed;
    uint32_t first = 0, tab = sd.tab;
    for (int half = 0; half < 2; ++half) {
      const uint32_t nk = half ? sd.nim : sd.nre;
      for (uint32_t q0 = 0; q0 < (1u << nk); q0 += 32) {
        const uint32_t q = q0 + lane;
        double a = 0.0, b = 0.0;
        for (uint32_t kk = 0; kk < nk; ++kk) {
          const double x = __shfl_sync(0xffffffffu, own, first + kk), y = __shfl_sync(0xffffffffu, other, first + kk);
          a += (q >> kk) & 1u ? -x : x;
          b += (q >> kk) & 1u ? -y : y;
        }
        if (q < (1u << nk)) {
          P.table[tab + q] = a;
          if (mixed) P.other[tab + q] = b;
        }
      }
      tab += 1u << nk;
      first += nk;
    }
  }
}

void refresh_coeffs(const wg_plan_host& h, const double* from, int reals, cudaStream_t s) {
  const PlanDev& P = h.dev;
  if (P.T == 0) return;
  plan_tables_kernel<<<wg::grid_for(32 * static_cast<size_t>(P.S), kThreads, h.device, 8), kThreads, 0, s>>>(P, from,
                                                                                                             reals);
  wg::check_launch("launch adjoint tables");
}

// Appends raw bytes to the host image of the plan, 16-byte aligned.
struct Blob {
  std::vector<unsigned char> bytes;
  template <typename T>
  size_t put(const std::vector<T>& v) {
    const size_t at = (bytes.size() + 15) & ~size_t{15};
    bytes.resize(at + sizeof(T) * v.size());
    if (!v.empty()) std::memcpy(bytes.data() + at, v.data(), sizeof(T) * v.size());
    return at;
  }
};

// adjoint = false: for E alone, on this stream only (no sub-groups, segments or
// tables, no wait).
wg_plan_host* make_plan(int device, size_t n, size_t T, const uint64_t* x, const uint64_t* z, const double* c,
                        bool adjoint, cudaStream_t s) {
  if (n > 63) wg::throw_invalid("expectation_statevector requires num_qubits <= 63");
  if (T > 0xffffffffull) wg::throw_invalid("expectation supports at most 2^32-1 terms");
  std::unique_ptr<wg_plan_host> p(new wg_plan_host());
  p->device = device;
  PlanDev& d = p->dev;
  std::memset(&d, 0, sizeof(d));
  d.n = static_cast<int>(n);
  d.T = static_cast<uint32_t>(T);
  d.m = std::max(kTileMin, std::min(static_cast<int>(n), kTileBits));
  d.tiles = static_cast<int>(n) > d.m ? 1u << std::min<int>(31, static_cast<int>(n) - d.m) : 1u;
  if (T == 0) return p.release();
  // masks to the host; the plan's tables are built there
  const int words = n == 0 ? 0 : 1;
  std::vector<uint64_t> hx(T, 0), hz(T, 0);
  if (words) {
    wg::check_cuda(cudaMemcpyAsync(hx.data(), x, 8 * T, cudaMemcpyDeviceToHost, s), "read x masks");
    wg::check_cuda(cudaMemcpyAsync(hz.data(), z, 8 * T, cudaMemcpyDeviceToHost, s), "read z masks");
  }
  wg::check_cuda(cudaStreamSynchronize(s), "read masks");
  if (words && n < 64) {
    uint64_t bits = 0;
    for (size_t i = 0; i < T; ++i) bits |= hx[i] | hz[i];
    // the kernels index psi[b ^ x]: masks must stay below 2^n
    if ((bits >> n) != 0) wg::throw_invalid("Pauli masks set bits at or above num_qubits");
  }
  // terms sorted by x (stable): groups; by (x >> m, x) at once, since x sorts that way
  std::vector<uint32_t> order(T);
  std::iota(order.begin(), order.end(), 0u);
  std::stable_sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return hx[a] < hx[b]; });
  const int m = d.m;
  std::vector<uint32_t> ty(T), torig(T), seg_cost, chunk{0}, bounds;
  std::vector<FwdPiece> piece;
  std::vector<AdjSub> asub;
  std::vector<SegDev> seg;
  // room for terms of hardly equal x (grown step by step, these two were a tenth of a plan of 1,000,000)
  piece.reserve(std::min<size_t>(T, size_t{1} << 20));
  if (adjoint) asub.reserve(std::min<size_t>(T, size_t{1} << 20));
  // the order of a piece's terms: those whose z are linearly independent on the
  // lane bits first, so that the lanes' entries spread over the banks
  auto spread = [&](uint32_t* first, uint32_t count) {
    uint32_t basis[5] = {}, at = 0;
    for (uint32_t i = 0; i < count; ++i) {
      uint32_t v = static_cast<uint32_t>(hz[first[i]]) & 31u;
      for (int b = 4; b >= 0 && v; --b) {
        if (!((v >> b) & 1u)) continue;
        if (basis[b]) {
          v ^= basis[b];
          continue;
        }
        basis[b] = v;
        std::rotate(first + at, first + i, first + i + 1);
        ++at;
        break;
      }
    }
  };
  size_t groups = 0;
  uint64_t entries = 0;
  std::vector<uint32_t> even, odd;
  for (size_t g0 = 0, t0 = 0; g0 < T;) {
    const uint64_t gx = hx[order[g0]];
    size_t ge = g0;
    even.clear();
    odd.clear();
    for (; ge < T && hx[order[ge]] == gx; ++ge) {
      const uint32_t o = order[ge];
      (__builtin_popcountll(gx & hz[o]) & 1 ? odd : even).push_back(o);
    }
    ++groups;
    const size_t subs = std::max((even.size() + kPiece - 1) / kPiece, (odd.size() + kPiece - 1) / kPiece);
    for (size_t i = 0; i < subs; ++i) {
      AdjSub ad{};
      ad.xlo = static_cast<uint32_t>(gx & ((uint64_t{1} << m) - 1));
      ad.t0 = static_cast<uint32_t>(t0);
      ad.tab = static_cast<uint32_t>(entries);
      uint32_t plane[kTileBits] = {};  // sign word of tile bit q
      for (int half = 0; half < 2; ++half) {
        std::vector<uint32_t>& all = half ? odd : even;
        const size_t from = std::min(all.size(), i * kPiece);
        const uint32_t nk = static_cast<uint32_t>(std::min<size_t>(kPiece, all.size() - from));
        (half ? ad.nim : ad.nre) = static_cast<uint16_t>(nk);
        spread(all.data() + from, nk);
        FwdPiece pd{};
        pd.xlo = ad.xlo;
        pd.xhi = static_cast<uint32_t>(gx >> m);
        pd.t0 = static_cast<uint32_t>(t0);
        pd.nk = static_cast<uint8_t>(nk);
        pd.odd = static_cast<uint8_t>(half);
        if (half && nk && ad.nre) piece.back().pair = 1;
        for (uint32_t kk = 0; kk < nk; ++kk, ++t0) {
          const uint32_t o = all[from + kk];
          torig[t0] = o;
          ty[t0] = static_cast<uint32_t>(__builtin_popcountll(gx & hz[o]) & 3) |
                   (gx == 0 ? kDiagFlag : (gx >> m) == 0 ? kTwiceFlag : 0u);
          pd.zlo[kk] = static_cast<uint32_t>(hz[o] & ((uint64_t{1} << m) - 1));
          pd.zhi[kk] = ad.zhi[half * kPiece + kk] = static_cast<uint32_t>(hz[o] >> m);
          for (int q = 0; adjoint && q < m; ++q) plane[q] |= static_cast<uint32_t>((hz[o] >> q) & 1u) << (3 + 16 * half + kk);
        }
        if (nk) piece.push_back(pd);
        entries += uint64_t{1} << nk;
      }
      entries += entries & 1u;  // staged in 16-byte pieces
      if (!adjoint) continue;
      for (int q = 0; q < 5; ++q)
        for (int l = 0; l < (1 << q); ++l) ad.lane[l | 1 << q] = ad.lane[l] ^ plane[q];
      for (int q = 5; q < m - 3; ++q)
        for (int l = 0; l < (1 << (q - 5)); ++l) ad.warp[l | 1 << (q - 5)] = ad.warp[l] ^ plane[q];
      for (int q = 0; q < 3; ++q)
        for (int l = 0; l < (1 << q); ++l) ad.own[l | 1 << q] = ad.own[l] ^ plane[m - 3 + q];
      asub.push_back(ad);
    }
    g0 = ge;
  }
  if (entries > 0xffffffffull) wg::throw_invalid("expectation plan: too many terms for its tables");
  const size_t S = asub.size(), NP = piece.size();
  auto xhi_of = [&](size_t i) { return static_cast<uint32_t>(hx[torig[asub[i].t0]] >> m); };
  auto tab_end = [&](size_t i) { return i + 1 < S ? asub[i + 1].tab : static_cast<uint32_t>(entries); };
  const auto& props = wg::device_props(device);
  const size_t sms = static_cast<size_t>(props.sm_count);
  // Segments: sub-groups of one class, at most kSegSubs; fewer where a few
  // tiles could not occupy the device otherwise (the adjoint splits at segments).
  const size_t slices = static_cast<size_t>(kTileMax) >> m;
  const size_t seg_subs = std::min<size_t>(
      kSegSubs, std::max<size_t>(slices, (S * d.tiles + 2 * sms - 1) / (2 * sms)));
  for (size_t i = 0; i < S;) {  // none without the adjoint
    size_t e = i + 1;
    while (e < S && e - i < seg_subs && xhi_of(e) == xhi_of(i) && tab_end(e) - asub[i].tab <= kSegEntries) ++e;
    // work of a segment, in hundredths of a tile's fetch: the tile, and its
    // sub-groups (in as many turns as the slices leave)
    const bool same = !seg.empty() && seg.back().xhi == xhi_of(i);
    seg.push_back(SegDev{xhi_of(i), static_cast<uint32_t>(i), static_cast<uint32_t>(e - i), asub[i].tab,
                         tab_end(e - 1) - asub[i].tab, {}});
    const uint32_t cost = (same ? 20u : 100u) + static_cast<uint32_t>((e - i + slices - 1) / slices) * 90u;
    seg_cost.push_back((seg_cost.empty() ? 0u : seg_cost.back()) + cost);
    i = e;
  }
  // The adjoint's tiles are split by segments until there are about four items
  // an SM.  The plan alone sets the splits and with them the order of the sums, so
  // that a pair's H psi has the same bits in every batch, however that runs them.
  if (adjoint) {
    const size_t NS = seg.size();
    const size_t splits = std::max<size_t>(
        1, std::min<size_t>({(4 * sms + d.tiles / 2) / d.tiles, NS, 64, seg_cost.back() / (m < kTileBits ? kSplitCost / 2 : kSplitCost)}));
    bounds.push_back(0);
    for (size_t k = 1; k < splits; ++k) {
      // the segment at which k / splits of the work is done; each split takes one at least
      const uint32_t to = static_cast<uint32_t>(static_cast<uint64_t>(seg_cost.back()) * k / splits);
      size_t at = static_cast<size_t>(std::lower_bound(seg_cost.begin(), seg_cost.end(), to) - seg_cost.begin()) + 1;
      at = std::min(std::max<size_t>(at, bounds.back() + 1), NS - (splits - k));
      bounds.push_back(static_cast<uint32_t>(at));
    }
    bounds.push_back(static_cast<uint32_t>(NS));
    p->tile_cost = seg_cost.back();
    d.splits = static_cast<uint32_t>(splits);
  }
  // Forward items: chunks of pieces (their sums stay in shared memory) times
  // ranges of tiles; about eight items an SM where there is the work.
  const size_t sets = (static_cast<size_t>(kFwdThreads) * 16) >> m;
  const size_t chunk_pieces = std::min<size_t>(
      kChunkPieces, std::max<size_t>(sets, (NP * d.tiles + 4 * sms - 1) / (4 * sms)));
  std::vector<uint32_t> load(sets);
  bool was_direct = false;
  for (size_t i = 0; i < NP;) {
    size_t e = i, units = 0, segs = 0;
    while (e < NP && e - i + 1 + piece[e].pair <= chunk_pieces) {
      segs += e == i || piece[e].xhi != piece[e - 1].xhi;
      ++units;
      e += 1 + piece[e].pair;
    }
    // Staging a class's tile pays where more than a piece or two of it follow: 21
    // qubits, 16 terms of as many classes, complex64, 105 us staged and 60 direct.
    const bool direct = m == kTileBits && static_cast<int>(n) > m && 4 * units <= 5 * segs;
    // the sets' turns: the least loaded one of the segment's (of the chunk's
    // where nothing is staged); a last pair is shared by two equally loaded ones
    // A class that goes on from the chunk before goes on with its loads: an item may
    // take several chunks together.
    const bool goes_on = !direct && i > 0 && !was_direct && piece[i].xhi == piece[i - 1].xhi;
    if (!goes_on) std::fill(load.begin(), load.end(), 0u);
    was_direct = direct;
    for (size_t k = i; k < e;) {
      if (!direct && k > i && piece[k].xhi != piece[k - 1].xhi) std::fill(load.begin(), load.end(), 0u);
      const size_t next = k + 1 + piece[k].pair;
      const size_t to = static_cast<size_t>(std::min_element(load.begin(), load.end()) - load.begin());
      const bool last = !direct && (next >= e || piece[next].xhi != piece[k].xhi);
      if (piece[k].pair && last && std::count(load.begin(), load.end(), load[to]) > 1) piece[k].pair = 0;
      load[to] += 1u + piece[k].pair;
      piece[k].turn = static_cast<uint8_t>(to);
      k += 1 + piece[k].pair;
    }
    if (direct) chunk.back() |= kReads;
    p->chunk_most = std::max(p->chunk_most, static_cast<uint32_t>(e - i));
    chunk.push_back(static_cast<uint32_t>(e));
    i = e;
  }
  d.chunks = static_cast<uint32_t>(chunk.size() - 1);
  d.ranges = static_cast<uint32_t>(
      std::max<size_t>(1, std::min<size_t>({d.tiles, 256, (8 * sms + d.chunks - 1) / d.chunks})));
  d.S = static_cast<uint32_t>(S);
  d.NP = static_cast<uint32_t>(NP);
  d.NS = static_cast<uint32_t>(seg.size());
  d.G = static_cast<uint32_t>(groups);
  p->n_groups = groups;
  d.joined = T <= kJoinTerms && static_cast<uint64_t>(T) * d.ranges <= kJoinSums;
  Blob blob;
  blob.bytes.reserve(sizeof(FwdPiece) * NP + sizeof(AdjSub) * S + sizeof(SegDev) * seg.size() +
                     4 * (chunk.size() + bounds.size() + 2 * T) + 7 * 16);
  const size_t o_piece = blob.put(piece), o_asub = blob.put(asub), o_seg = blob.put(seg), o_chunk = blob.put(chunk),
               o_bounds = blob.put(bounds), o_ty = blob.put(ty), o_torig = blob.put(torig);
  const size_t o_coeffs = (blob.bytes.size() + 15) & ~size_t{15}, o_partial = o_coeffs + 16 * T;
  const size_t o_table = (o_partial + 8 * static_cast<uint64_t>(T) * d.ranges + 15) & ~size_t{15};
  p->mem.reset(o_table + (adjoint ? 16 * entries : 0), s);
  wg::check_cuda(cudaMemcpyAsync(p->mem.get(), blob.bytes.data(), blob.bytes.size(), cudaMemcpyHostToDevice, s),
                 "upload plan");
  auto* base = static_cast<unsigned char*>(p->mem.get());
  d.piece = reinterpret_cast<const FwdPiece*>(base + o_piece);
  d.asub = reinterpret_cast<AdjSub*>(base + o_asub);
  d.seg = reinterpret_cast<const SegDev*>(base + o_seg);
  d.chunk = reinterpret_cast<const uint32_t*>(base + o_chunk);
  d.bounds = reinterpret_cast<const uint32_t*>(base + o_bounds);
  d.ty = reinterpret_cast<const uint32_t*>(base + o_ty);
  d.torig = reinterpret_cast<const uint32_t*>(base + o_torig);
  d.coeffs = reinterpret_cast<double*>(base + o_coeffs);
  d.partial = reinterpret_cast<double*>(base + o_partial);
  d.table = reinterpret_cast<double*>(base + o_table);
  d.other = d.table + entries;
  if (!adjoint) {
    // the caller's coefficients outlive the call; the upload's source is staged
    d.coeffs = const_cast<double*>(c);
    return p.release();
  }
  refresh_coeffs(*p, c, 2, s);
  // pageable source above: wait until the plan image is on the device
  wg::check_cuda(cudaStreamSynchronize(s), "build plan");
  // The plan outlives the caller's stream: release its memory on the legacy
  // default stream.
  p->mem.rebind(nullptr);
  return p.release();
}

struct RunSpec {
  wg_plan_host* plan;
  const void* psi;
  double* result;
  double* term_values;
  double* hpsi;
};

}  // namespace

// A prepared batch: device work tables for fixed (plan, psi, outputs) pairs.
// Running it only enqueues kernels (no host synchronisation, no host copies),
// so a run can be captured in a CUDA graph and replayed.
struct wg_expect_batch_s {
  int device = 0;
  int dtype = WG_DTYPE_C128;
  int sms = 0;
  BatchDev dev{};
  wg::Scratch table;  // the pairs and the work queues
  wg::Scratch parts;  // partial H psi of the pairs whose adjoint is split, term values that nobody asked for
};

namespace {

constexpr int kMaxDevices = 64;

// The kernels' shared memory, set once per device.
void allow_smem(int device) {
  static std::once_flag done[kMaxDevices];
  if (device < 0 || device >= kMaxDevices) wg::throw_invalid("CUDA device ordinal is out of range");
  std::call_once(done[device], [] {  // a throw leaves the flag unset: the next call retries
    auto allow = [](auto* kernel, size_t bytes) {
      wg::check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)),
                     "set expectation shared memory");
    };
    allow(expect_forward_kernel<double2>, sizeof(FwdShared));
    allow(expect_forward_kernel<float2>, sizeof(FwdShared));
    allow(expect_adjoint_kernel<double2>, sizeof(AdjShared));
    allow(expect_adjoint_kernel<float2>, sizeof(AdjShared));
  });
}

// How a batch divides its pairs.  A plan is divided as if it had the device for itself;
// among others a pair takes several of its chunks in one forward item, and the splits
// of a tile one after another in one adjoint item: what an item fetches, and the sums
// that a split writes and reads, then serve more terms.  Neither changes a bit.  64
// pairs of 14 qubits and 1,000 terms with H psi 2.47 -> 1.05 ms, 400 of 100 terms 6.5
// -> 1.63; 30 pairs of 8 to 18 qubits 2.02 -> 1.77; and no partial H psi for most pairs
// (up to 37 MB each, now 2 GB at most in all: the tiles that are still split are at most
// three an SM, of 64 splits and 64 KB each).
struct Division {
  double forward = 0.0;  // pieces x tiles of a forward item, at most
  double adjoint = 0.0;  // tiles of at most this cost are one adjoint item
};

// Forward items: four for every SM, and at least eight pieces x tiles.  Adjoint items:
// a tile that is no more than 1.35 of an SM's share of the batch, as long as the SMs'
// last turn at such tiles is not mostly empty, else of a third.
Division divide_batch(const std::vector<RunSpec>& specs, int sms) {
  Division d;
  if (specs.size() <= 1) return d;
  double fwd = 0.0, adj = 0.0;
  for (const RunSpec& r : specs) {
    fwd += static_cast<double>(r.plan->dev.NP) * r.plan->dev.tiles;
    if (r.hpsi) adj += static_cast<double>(r.plan->tile_cost) * r.plan->dev.tiles;
  }
  d.forward = std::max(8.0, fwd / (4.0 * sms));
  const double share = adj / sms;
  d.adjoint = 1.35 * share;
  uint64_t large = 0;  // items above a third of the share
  for (const RunSpec& r : specs) {
    const double cost = static_cast<double>(r.plan->tile_cost);
    if (r.hpsi && cost > share / 3.0 && cost <= d.adjoint) large += r.plan->dev.tiles;
  }
  const uint64_t turns = (large + sms - 1) / sms;
  if (3 * large < 2 * turns * sms) d.adjoint = share / 3.0;
  return d;
}

// The pairs in order of their adjoint items' work, largest first: the queue ends with
// the small ones.
std::vector<RunSpec> by_work(const std::vector<RunSpec>& specs) {
  std::vector<RunSpec> out(specs);
  std::stable_sort(out.begin(), out.end(), [](const RunSpec& a, const RunSpec& b) {
    return a.plan->tile_cost * (a.hpsi ? 1 : 0) > b.plan->tile_cost * (b.hpsi ? 1 : 0);
  });
  return out;
}

wg_expect_batch_s* make_batch(int device, const std::vector<RunSpec>& given, int dtype, cudaStream_t s) {
  if (dtype != WG_DTYPE_C128 && dtype != WG_DTYPE_C64) wg::throw_invalid("psi dtype must be complex64 or complex128");
  std::unique_ptr<wg_expect_batch_s> b(new wg_expect_batch_s());
  b->device = device;
  b->dtype = dtype;
  b->sms = wg::device_props(device).sm_count;
  allow_smem(device);
  const std::vector<RunSpec> specs = by_work(given);
  const size_t np = specs.size();
  if (np > 0xffffffffull) wg::throw_invalid("too many pairs in one batch");
  std::vector<PairDev> pairs(np);
  std::vector<uint64_t> item_base(np + 1, 0), term_base(np + 1, 0), tile_base(np + 1, 0), amp_base(np + 1, 0);
  const Division division = divide_batch(specs, b->sms);
  uint64_t bytes = 0;  // of the partial H psi and the term values, then where they lie
  std::vector<uint64_t> part_at(np, 0), ev_at(np, 0);
  for (size_t i = 0; i < np; ++i) {
    const PlanDev& P = specs[i].plan->dev;
    // tile numbers are 32 bits; no device holds a larger state
    if (P.n > kTileBits + 31) wg::throw_invalid("expectation_statevector: the statevector exceeds device memory");
    const wg_plan_host& h = *specs[i].plan;
    uint32_t group = 1;
    if (np > 1 && P.T) {
      const double chunk_work = static_cast<double>(P.NP) / P.chunks * P.tiles / P.ranges;  // of an item of one chunk
      group = static_cast<uint32_t>(
          std::max(1.0, std::min<double>(division.forward / chunk_work, kChunkPieces / h.chunk_most)));
    }
    const bool fold = P.splits > 1 && static_cast<double>(h.tile_cost) <= division.adjoint;
    const uint32_t parts = fold ? 1 : P.splits;
    pairs[i] = PairDev{P, specs[i].psi, specs[i].term_values, specs[i].result, specs[i].hpsi, nullptr, group,
                       (P.chunks + group - 1) / group, fold};
    item_base[i + 1] = item_base[i] + (P.T ? static_cast<uint64_t>(pairs[i].per_range) * P.ranges : 0);
    term_base[i + 1] = term_base[i] + (P.joined ? 0 : P.T);
    tile_base[i + 1] = tile_base[i];
    amp_base[i + 1] = amp_base[i];
    if (specs[i].hpsi && P.T) {
      tile_base[i + 1] += static_cast<uint64_t>(P.tiles) * parts;
      if (parts > 1) {
        amp_base[i + 1] += uint64_t{1} << P.n;
        part_at[i] = bytes;
        bytes += static_cast<uint64_t>(parts) << (P.n + 4);
      }
    }
    if (!specs[i].term_values && !P.joined && P.T) {
      ev_at[i] = bytes;
      bytes += (8 * static_cast<uint64_t>(P.T) + 15) & ~uint64_t{15};
    }
  }
  if (bytes) {
    b->parts.reset(bytes, s);
    b->parts.rebind(nullptr);
    auto* base = b->parts.as<unsigned char>();
    for (size_t i = 0; i < np; ++i) {
      const PlanDev& P = pairs[i].plan;
      if (pairs[i].hpsi && P.T && P.splits > 1 && !pairs[i].fold) pairs[i].part = reinterpret_cast<double2*>(base + part_at[i]);
      if (!pairs[i].evals && !P.joined && P.T) pairs[i].evals = reinterpret_cast<double*>(base + ev_at[i]);
    }
  }
  BatchDev& d = b->dev;
  d.np = static_cast<uint32_t>(np);
  d.n_items = item_base[np];
  d.n_terms = term_base[np];
  d.n_tiles = tile_base[np];
  d.n_amps = amp_base[np];
  // A queue where some CTA takes several items: which side of a pairing a tile is
  // on makes them uneven (21 qubits, 16 terms: 112 us taking turns, 60 queued).
  const bool queue = np > 1 || std::max(d.n_items, d.n_tiles) > static_cast<uint64_t>(b->sms);
  if (np == 1) d.one = pairs[0];
  if (!queue) return b.release();
  std::vector<unsigned char> host;
  auto put = [&](const void* src, size_t n) {
    const size_t at = (host.size() + 15) & ~size_t{15};
    host.resize(at + n);
    std::memcpy(host.data() + at, src, n);
    return at;
  };
  const unsigned long long zero[2] = {0, 0};
  const size_t o_cnt = put(zero, sizeof(zero));
  size_t o_pairs = 0, o_item = 0, o_term = 0, o_tile = 0, o_amp = 0;
  if (np > 1) {
    o_pairs = put(pairs.data(), sizeof(PairDev) * np);
    o_item = put(item_base.data(), 8 * (np + 1));
    o_term = put(term_base.data(), 8 * (np + 1));
    o_tile = put(tile_base.data(), 8 * (np + 1));
    o_amp = put(amp_base.data(), 8 * (np + 1));
  }
  b->table.reset(host.size(), s);
  b->table.rebind(nullptr);
  auto* base = static_cast<unsigned char*>(b->table.get());
  d.counters = reinterpret_cast<unsigned long long*>(base + o_cnt);
  if (np == 1) return b.release();
  // pageable source: the call returns once the bytes are staged
  wg::check_cuda(cudaMemcpyAsync(b->table.get(), host.data(), host.size(), cudaMemcpyHostToDevice, s),
                 "upload work table");
  d.pairs = reinterpret_cast<const PairDev*>(base + o_pairs);
  d.item_base = reinterpret_cast<const uint64_t*>(base + o_item);
  d.term_base = reinterpret_cast<const uint64_t*>(base + o_term);
  d.tile_base = reinterpret_cast<const uint64_t*>(base + o_tile);
  d.amp_base = reinterpret_cast<const uint64_t*>(base + o_amp);
  return b.release();
}

// Enqueues forward, finish, totals and adjoint; no host synchronisation.
void run_batch(const wg_expect_batch_s& b, cudaStream_t s) {
  const BatchDev& d = b.dev;
  if (d.np == 0) return;
  if (d.counters) wg::check_cuda(cudaMemsetAsync(d.counters, 0, 16, s), "reset work queues");
  const unsigned persistent = static_cast<unsigned>(b.sms);  // one CTA an SM: its tiles fill the shared memory
  if (d.n_items) {
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(d.n_items, persistent));
    auto* kernel = b.dtype == WG_DTYPE_C128 ? expect_forward_kernel<double2> : expect_forward_kernel<float2>;
    WG_TIMED("expect_forward_kernel", s, kernel<<<grid, kFwdThreads, sizeof(FwdShared), s>>>(d));
    wg::check_launch("launch expectation forward");
  }
  const unsigned wave = static_cast<unsigned>(b.sms) * 8;
  if (d.n_terms) {
    const unsigned grid =
        static_cast<unsigned>(std::min<uint64_t>((8 * d.n_terms + kThreads - 1) / kThreads, wave));
    WG_TIMED("expect_finish_terms_kernel", s, expect_finish_terms_kernel<<<grid, kThreads, 0, s>>>(d));
    wg::check_launch("launch expectation finish");
  }
  WG_TIMED("expect_total_kernel", s,
           expect_total_kernel<<<std::min<uint32_t>(d.np, 65535u), kTotalThreads, 0, s>>>(d));
  wg::check_launch("launch expectation total");
  if (d.n_tiles) {
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>(d.n_tiles, persistent));
    auto* kernel = b.dtype == WG_DTYPE_C128 ? expect_adjoint_kernel<double2> : expect_adjoint_kernel<float2>;
    WG_TIMED("expect_adjoint_kernel", s, kernel<<<grid, kAdjThreads, sizeof(AdjShared), s>>>(d));
    wg::check_launch("launch expectation adjoint");
  }
  if (d.n_amps) {
    const unsigned grid = static_cast<unsigned>(std::min<uint64_t>((d.n_amps + kThreads - 1) / kThreads, wave));
    WG_TIMED("expect_join_kernel", s, expect_join_kernel<<<grid, kThreads, 0, s>>>(d));
    wg::check_launch("launch expectation join");
  }
}

// Pairs whose operator has no terms: E = 0, e = {}, H psi = 0.
void clear_empty(const std::vector<RunSpec>& specs, cudaStream_t s) {
  for (const RunSpec& r : specs) {
    if (r.plan->dev.T != 0) continue;
    if (r.result) wg::check_cuda(cudaMemsetAsync(r.result, 0, 16, s), "clear expectation");
    if (r.hpsi) wg::check_cuda(cudaMemsetAsync(r.hpsi, 0, 16ull << r.plan->dev.n, s), "clear H psi");
  }
}

void run_specs(int device, const std::vector<RunSpec>& specs, int dtype, cudaStream_t s) {
  std::unique_ptr<wg_expect_batch_s> b(make_batch(device, specs, dtype, s));
  clear_empty(specs, s);
  run_batch(*b, s);
  // stream-ordered release after the kernels that read the tables
  b->table.rebind(s);
  b->parts.rebind(s);
}

std::vector<RunSpec> batch_specs(int device, size_t n_pairs, const wg_expect_plan_t* plans, const void* const* psis,
                                 double* const* results, double* const* term_values, double* const* hpsis) {
  std::vector<RunSpec> specs(n_pairs);
  for (size_t i = 0; i < n_pairs; ++i) {
    if (!plans[i]) wg::throw_invalid("expectation plan is null");
    if (plans[i]->h.device != device) wg::throw_invalid("expectation plan belongs to another device");
    if (!psis[i]) wg::throw_invalid("CUDA statevector data pointer must be non-null");
    for (size_t j = 0; j < i; ++j)
      if (plans[j] == plans[i]) wg::throw_invalid("a plan may appear at most once per batched launch");
    specs[i] = RunSpec{&plans[i]->h, psis[i], results ? results[i] : nullptr, term_values ? term_values[i] : nullptr,
                       hpsis ? hpsis[i] : nullptr};
  }
  return specs;
}

}  // namespace

extern "C" {

int wg_expect_plan_create(int device, size_t n_qubits, size_t n_terms, const uint64_t* x, const uint64_t* z,
                          const double* coeffs, wg_expect_plan_t* plan, wg_stream_t stream) {
  return wg::guarded([&] {
    *plan = nullptr;
    if (n_qubits > 63) wg::throw_invalid("expectation_statevector requires num_qubits <= 63");
    wg::DeviceGuard g(device);
    std::unique_ptr<wg_plan_host> p(make_plan(device, n_qubits, n_terms, x, z, coeffs, true, stream));
    *plan = reinterpret_cast<wg_expect_plan_t>(new wg_expect_plan_s{std::move(*p)});
  });
}

int wg_expect_plan_destroy(wg_expect_plan_t plan) {
  return wg::guarded([&] {
    if (!plan) return;
    wg::DeviceGuard g(plan->h.device);
    delete plan;
  });
}

int wg_expect_plan_set_coeffs(wg_expect_plan_t plan, const double* coeffs, wg_stream_t stream) {
  return wg::guarded([&] {
    if (!plan) wg::throw_invalid("expectation plan is null");
    wg::DeviceGuard g(plan->h.device);
    refresh_coeffs(plan->h, coeffs, 2, stream);
  });
}

int wg_expect_plan_set_real_coeffs(wg_expect_plan_t plan, const double* coeffs, wg_stream_t stream) {
  return wg::guarded([&] {
    if (!plan) wg::throw_invalid("expectation plan is null");
    wg::DeviceGuard g(plan->h.device);
    refresh_coeffs(plan->h, coeffs, 1, stream);
  });
}

int wg_expect_plan_info(wg_expect_plan_t plan, size_t* n_groups, size_t* n_terms) {
  return wg::guarded([&] {
    if (!plan) wg::throw_invalid("expectation plan is null");
    *n_groups = plan->h.n_groups;
    *n_terms = plan->h.dev.T;
  });
}

int wg_expect_plan_run(wg_expect_plan_t plan, const void* psi, int psi_dtype, double* result, double* term_values,
                       double* hpsi, wg_stream_t stream) {
  return wg::guarded([&] {
    if (!plan) wg::throw_invalid("expectation plan is null");
    if (!psi) wg::throw_invalid("CUDA statevector data pointer must be non-null");
    wg::DeviceGuard g(plan->h.device);
    run_specs(plan->h.device, {RunSpec{&plan->h, psi, result, term_values, hpsi}}, psi_dtype, stream);
  });
}

int wg_expectation(int device, size_t n_qubits, size_t n_terms, const uint64_t* x, const uint64_t* z,
                   const double* coeffs, const void* psi, int psi_dtype, double* result_host, wg_stream_t stream) {
  return wg::guarded([&] {
    if (n_qubits > 63) wg::throw_invalid("expectation_statevector requires num_qubits <= 63");
    if (psi_dtype != WG_DTYPE_C128 && psi_dtype != WG_DTYPE_C64)
      wg::throw_invalid("psi dtype must be complex64 or complex128");
    result_host[0] = result_host[1] = 0.0;
    if (n_terms == 0) return;
    if (!psi) wg::throw_invalid("CUDA statevector data pointer must be non-null");
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    std::unique_ptr<wg_plan_host> p(make_plan(device, n_qubits, n_terms, x, z, coeffs, false, s));
    wg::Scratch res(16, s);
    run_specs(device, {RunSpec{p.get(), psi, res.as<double>(), nullptr, nullptr}}, psi_dtype, s);
    wg::check_cuda(cudaMemcpyAsync(result_host, res.get(), 16, cudaMemcpyDeviceToHost, s), "read expectation");
    wg::check_cuda(cudaStreamSynchronize(s), "read expectation");
  });
}

int wg_expect_batched(int device, size_t n_pairs, const wg_expect_plan_t* plans, const void* const* psis,
                      int psi_dtype, double* const* results, double* const* term_values, double* const* hpsis,
                      wg_stream_t stream) {
  return wg::guarded([&] {
    if (n_pairs == 0) return;
    wg::DeviceGuard g(device);
    run_specs(device, batch_specs(device, n_pairs, plans, psis, results, term_values, hpsis), psi_dtype, stream);
  });
}

int wg_expect_batch_create(int device, size_t n_pairs, const wg_expect_plan_t* plans, const void* const* psis,
                           int psi_dtype, double* const* results, double* const* term_values,
                           double* const* hpsis, wg_expect_batch_t* batch, wg_stream_t stream) {
  return wg::guarded([&] {
    *batch = nullptr;
    wg::DeviceGuard g(device);
    const auto specs = batch_specs(device, n_pairs, plans, psis, results, term_values, hpsis);
    for (const RunSpec& r : specs)
      if (r.plan->dev.T == 0) wg::throw_invalid("a prepared batch needs operators with at least one term");
    *batch = make_batch(device, specs, psi_dtype, stream);
    wg::check_cuda(cudaStreamSynchronize(stream), "prepare batch");
  });
}

int wg_expect_batch_run(wg_expect_batch_t batch, wg_stream_t stream) {
  return wg::guarded([&] {
    if (!batch) wg::throw_invalid("expectation batch is null");
    wg::DeviceGuard g(batch->device);
    run_batch(*batch, stream);
  });
}

int wg_expect_batch_destroy(wg_expect_batch_t batch) {
  return wg::guarded([&] {
    if (!batch) return;
    wg::DeviceGuard g(batch->device);
    delete batch;
  });
}

}  // extern "C"
