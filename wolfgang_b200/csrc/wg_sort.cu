// wg_sort.cu -- stable radix sort of (64-bit code, 32-bit index) pairs, and of
// multi-word keys by way of it.
//
// One pass per 8 code bits, least significant first.  The digit counts of all
// passes are taken in one reading of the codes; a pass then reads each pair
// once and writes it once (24 bytes of traffic an item).  A tile of 4,096
// pairs learns where its digits go by decoupled look-back (D. Merrill and
// M. Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back",
// NVIDIA NVR-2016-002): it publishes its own counts, adds up its
// predecessors' until it meets one that knows its total, and publishes its
// total.  Tiles are numbered by a ticket taken when a CTA starts, so that all
// a tile waits for is already running; the wait is bounded all the same.

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "wg_common.cuh"
#include "wg_sort.cuh"
#include "wg_sort_block.cuh"

namespace wgo {

namespace passes {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;
constexpr uint32_t kSpinLimit = 1u << 24;  // unless wg_set_wait_limit says otherwise
constexpr int kLook = 8;

// A status word: value (56 bits) | pass + 1 (6 bits) | state (2 bits).  The
// pass number tells this pass's words from the previous ones', so the array
// is cleared once per sort.
constexpr unsigned long long kCounted = 1ull << 62;  // the tile's own count
constexpr unsigned long long kTotal = 2ull << 62;    // all tiles' up to this one
constexpr unsigned long long kValue = (1ull << 56) - 1;

struct PassSmem {
  uint64_t keys[kTile];   // the tile in output order; before that, warp_count
  uint32_t idx[kTile];
  uint32_t to[kDigits];   // output place of the tile's place 0, per digit
  uint32_t warp_sum[kDigits / 32];
  uint32_t tile;
};

// What bounds a pass: 24 bytes of HBM traffic an item, in runs of the items of
// one digit in a tile, and the instructions that rank an item (eight ballots
// give the lanes of equal digit; __match_any_sync and masks built by shared
// atomics measured 5 % either way).  16,777,216 pairs take 0.143 ms, 2.8 TB/s, at
// three CTAs of 512 threads and 8 items a thread (two CTAs: 0.18 ms; 256 threads
// of 16 items: 0.21 ms); the pass before, a histogram, a scan and a scatter of
// whole keys, took 0.46 ms.  A digit is one byte of one half of the code: 67,108,864
// pairs 0.53 ms shifting 64 bits, 0.51 with a byte permute.
template <bool kHigh>  // the digit lies in the code's upper half
static __global__ void __launch_bounds__(kThreads, 3) radix_pass_kernel(
    const uint64_t* __restrict__ kin, uint64_t* __restrict__ kout, const uint32_t* __restrict__ iin,
    uint32_t* __restrict__ iout, uint32_t n, int pass, const uint32_t* __restrict__ base,
    unsigned long long* status, SortControl* ctl, uint32_t limit) {
  extern __shared__ __align__(16) unsigned char raw[];
  PassSmem& sm = *reinterpret_cast<PassSmem*>(raw);
  uint32_t* warp_count = reinterpret_cast<uint32_t*>(sm.keys);  // [kWarps][kDigits]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) sm.tile = atomicAdd(&ctl->ticket[pass], 1u);
  for (int i = tid; i < kWarps * kDigits; i += kThreads) warp_count[i] = 0;
  __syncthreads();
  const uint32_t tile = sm.tile;
  const size_t t0 = static_cast<size_t>(tile) * kTile;
  const uint32_t valid = static_cast<uint32_t>(min(static_cast<size_t>(kTile), n - t0));
  const uint32_t byte = 0x4440u | (static_cast<uint32_t>(pass) & 3u);
  // a warp's items are consecutive: place warp * 256 + 32 j + lane
  uint64_t key[kItems];
  uint32_t pos[kItems / 2];  // places of two items each
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const uint32_t p = warp * (32 * kItems) + 32 * j + lane;
    key[j] = p < valid ? kin[t0 + p] : ~0ull;  // absent items come last, behind the tile's digit 255
  }
  uint32_t* mine = warp_count + warp * kDigits;
  const uint32_t below = (1u << lane) - 1u;
  auto digit = [&](uint64_t k) {
    return __byte_perm(static_cast<uint32_t>(kHigh ? k >> 32 : k), 0u, byte);
  };
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const uint32_t d = digit(key[j]);
    uint32_t same = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 8; ++b) {
      const bool on = (d >> b) & 1u;
      const uint32_t v = __ballot_sync(0xffffffffu, on);
      same &= on ? v : ~v;
    }
    const uint32_t before = mine[d];
    __syncwarp();
    const uint32_t rank = __popc(same & below);
    if (rank == 0) mine[d] = before + __popc(same);
    __syncwarp();
    if (j & 1) pos[j >> 1] |= (before + rank) << 16;
    else pos[j >> 1] = before + rank;
  }
  __syncthreads();
  // thread d < 256 owns digit d: its items in the tile, by warp
  const bool owner = tid < kDigits;
  const unsigned long long tag = static_cast<unsigned long long>(pass + 1) << 56;
  volatile unsigned long long* st = status + static_cast<size_t>(tile) * kDigits + tid;
  uint32_t count = 0, start = 0;
  if (owner) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = warp_count[w * kDigits + tid];
      warp_count[w * kDigits + tid] = count;
      count += c;
    }
    // where each digit starts within the tile, absent items included
    uint32_t incl = count;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) sm.warp_sum[warp] = incl;
    start = incl - count;
    if (tid == kDigits - 1) count -= kTile - valid;
    *st = (tile == 0 ? kTotal : kCounted) | tag | count;
  }
  __syncthreads();
  if (owner) {
    for (int w = 0; w < warp; ++w) start += sm.warp_sum[w];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) warp_count[w * kDigits + tid] += start;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j) pos[j >> 1] += mine[digit(key[j])] << (16 * (j & 1));
  __syncthreads();  // the counts are read: the tile takes their place
#pragma unroll
  for (int j = 0; j < kItems; ++j) sm.keys[(pos[j >> 1] >> (16 * (j & 1))) & 0xffffu] = key[j];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const uint32_t p = warp * (32 * kItems) + 32 * j + lane;
    if (p < valid) sm.idx[(pos[j >> 1] >> (16 * (j & 1))) & 0xffffu] = iin ? iin[t0 + p] : static_cast<uint32_t>(t0 + p);
  }
  // look back
  unsigned long long prefix = 0;
  if (owner && tile > 0) {
    // kLook predecessors are read at a time: one after another their latency
    // is what a pass spends (5,000,000 pairs: 70 us a pass one by one)
    const volatile unsigned long long* look = st;
    uint32_t spins = 0;
    for (uint32_t t = tile; t > 0;) {
      unsigned long long v[kLook];
#pragma unroll
      for (int e = 0; e < kLook; ++e)
        v[e] = static_cast<uint32_t>(e) < t ? look[-static_cast<ptrdiff_t>((e + 1) * kDigits)] : 0ull;
      int used = 0;
      bool total = false;
#pragma unroll
      for (int e = 0; e < kLook; ++e) {
        if (total || used != e) continue;  // found, or one before is not there yet
        if (((v[e] ^ tag) & (63ull << 56)) != 0 || (v[e] >> 62) == 0) continue;
        prefix += v[e] & kValue;
        total = (v[e] >> 62) == 2;
        used = e + 1;
      }
      if (total) break;
      if (used == 0 && ++spins >= limit) {
        ctl->timeout = 1;
        break;
      }
      look -= static_cast<ptrdiff_t>(used) * kDigits;
      t -= used;
    }
    *st = kTotal | tag | (prefix + count);
  }
  if (owner) sm.to[tid] = base[pass * kDigits + tid] + static_cast<uint32_t>(prefix) - start;
  __syncthreads();
#pragma unroll 4
  for (uint32_t p = tid; p < valid; p += kThreads) {
    const uint64_t k = sm.keys[p];
    const uint32_t o = sm.to[digit(k)] + p;
    if (o < n) {  // always, unless a look-back gave up
      kout[o] = k;
      iout[o] = sm.idx[p];
    }
  }
}

// hist[pass][digit] -> places where the digits start, one block per pass.
static __global__ void __launch_bounds__(kDigits) radix_base_kernel(uint32_t* hist, uint32_t n) {
  __shared__ uint32_t sums[kDigits / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t c = hist[blockIdx.x * kDigits + threadIdx.x];
  {
    // the zeros, which are not counted, are the rest
    const uint32_t s = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) sums[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      c = n;
      for (int w = 0; w < kDigits / 32; ++w) c -= sums[w];
    }
    __syncthreads();
  }
  uint32_t incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) sums[warp] = incl;
  __syncthreads();
  uint32_t start = incl - c;
  for (int w = 0; w < warp; ++w) start += sums[w];
  hist[blockIdx.x * kDigits + threadIdx.x] = start;
}

}  // namespace passes

size_t pair_tiles(size_t n) { return (n + passes::kTile - 1) / passes::kTile; }

void sort_pairs(size_t n, PairBuffers& b, int count, bool implied, cudaStream_t s) {
  using namespace passes;
  if (n == 0 || count == 0) return;
  wg::allow_smem(radix_pass_kernel<false>, sizeof(PassSmem));
  wg::allow_smem(radix_pass_kernel<true>, sizeof(PassSmem));
  radix_base_kernel<<<count, kDigits, 0, s>>>(b.hist, static_cast<uint32_t>(n));
  wg::check_launch("launch radix bases");
  const unsigned tiles = static_cast<unsigned>(pair_tiles(n));
  for (int p = 0; p < count; ++p) {
    auto* kernel = p < 4 ? radix_pass_kernel<false> : radix_pass_kernel<true>;
    WG_TIMED("radix_pass_kernel", s,
      kernel<<<tiles, kThreads, sizeof(PassSmem), s>>>(b.k0, b.k1, implied && p == 0 ? nullptr : b.i0, b.i1,
                                                       static_cast<uint32_t>(n), p, b.hist, b.status, b.control,
                                                       wg::wait_limit(kSpinLimit)));
    wg::check_launch("launch radix pass");
    std::swap(b.k0, b.k1);
    std::swap(b.i0, b.i1);
  }
}

CodeSpec choose_code(const KeyBits& kb, size_t n) {
  CodeSpec c{};
  c.B = kb.B;
  c.words = std::max(1, (kb.B + 63) / 64);
  c.exact = kb.B <= 64;
  // A pass costs more than the ties that its bits would tell apart as long as
  // some 28 bits more than log2 n are there: on 67,108,864 products of
  // 100-qubit local terms passes and reduction take 6.17 ms with 64 bits, 5.75
  // with 56 and 6.50 with 48; on 536,870,912 the whole call 70.6 with 64, 67.6
  // with 56.
  c.nb = c.exact ? std::max(1, kb.B) : n <= (size_t{1} << 20) ? 48 : n <= (size_t{1} << 30) ? 56 : 64;
  c.k = 0;
  if (!c.exact && kb.density > 0.0 && kb.density < 0.45) {
    // the remainder's width that suits a mean gap of 1 / density
    const double k = std::round(std::log2(0.69 / kb.density));
    c.k = static_cast<int>(std::min(16.0, std::max(0.0, k)));
  }
  return c;
}

}  // namespace wgo

namespace {

using namespace wgo;

// Codes of structure-of-arrays keys (word k of item i at keys[k * n + i]) and
// their digit counts.
struct SoaWords {
  const uint64_t* keys;
  size_t n;
  __device__ __forceinline__ uint64_t operator()(size_t i, int k) const { return keys[static_cast<size_t>(k) * n + i]; }
};

__global__ void __launch_bounds__(256) soa_code_kernel(SoaWords src, int K, const unsigned long long* __restrict__ bits,
                                                       CodeSpec spec, int passes, uint64_t* __restrict__ code,
                                                       uint32_t* hist) {
  extern __shared__ uint32_t sh[];
  clear_digits(sh, passes);
  __syncthreads();
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < src.n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    // the packed key's words as the code asks for them, one after another
    int k = 0, base = 0;  // next key word, varying bits before it
    uint64_t rest = 0;    // of that word, what belongs to the next packed one
    bool whole;
    const uint64_t c = key_code(spec, [&](int w) {
      uint64_t cur = rest;
      rest = 0;
      while (k < K && base < 64 * (w + 1)) {
        const uint64_t m = bits[k];
        uint64_t v = src(i, k) & m;
        while (v) {
          const int b = 63 - __clzll(static_cast<long long>(v));
          v ^= uint64_t{1} << b;
          const int r = base + __popcll(m & ~((uint64_t{2} << b) - 1));
          (r < 64 * (w + 1) ? cur : rest) |= 0x8000000000000000ull >> (r & 63);
        }
        base += __popcll(m);
        ++k;
      }
      return cur;
    }, &whole);
    code[i] = c;
    count_digits(sh, c, passes);
  }
  __syncthreads();
  store_digits(sh, passes, hist);
}

// The varying bits of key word k as code, read through the order so far.
__global__ void __launch_bounds__(256) soa_word_kernel(SoaWords src, int k, const unsigned long long* __restrict__ bits,
                                                       int passes, const uint32_t* __restrict__ order,
                                                       uint64_t* __restrict__ code, uint32_t* hist) {
  extern __shared__ uint32_t sh[];
  clear_digits(sh, passes);
  __syncthreads();
  const uint64_t m = bits[k];
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < src.n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    uint64_t c = 0;
    for (uint64_t v = src(order ? order[i] : i, k) & m; v; v &= v - 1)
      c |= uint64_t{1} << __popcll(m & ((v & (0 - v)) - 1));
    code[i] = c;
    count_digits(sh, c, passes);
  }
  __syncthreads();
  store_digits(sh, passes, hist);
}

// Equal neighbouring codes of unequal keys: the codes did not sort the keys.
__global__ void __launch_bounds__(256) soa_check_kernel(const uint64_t* __restrict__ code,
                                                        const uint32_t* __restrict__ order, SoaWords src, int K,
                                                        SortControl* ctl) {
  const size_t n = src.n;
  if (ctl->timeout) return;  // the order is not whole
  bool mixed = false;
  for (size_t i = 1 + blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    if (code[i] != code[i - 1]) continue;
    const size_t a = order[i], b = order[i - 1];
    for (int k = 0; k < K; ++k) mixed |= src(a, k) != src(b, k);
  }
  if (mixed) ctl->mixed = 1;
}

// The runs of equal codes in stable key order, a thread per run; ctl->mixed
// where a run of more than kTieRun items holds several keys.
constexpr uint32_t kTieRun = 64;

__global__ void __launch_bounds__(256) soa_ties_kernel(const uint64_t* __restrict__ code, uint32_t* order,
                                                       SoaWords src, int K, SortControl* ctl) {
  const size_t n = src.n;
  auto compare = [&](uint32_t a, uint32_t b) {
    for (int k = 0; k < K; ++k) {
      const uint64_t u = src(a, k), v = src(b, k);
      if (u != v) return u < v ? -1 : 1;
    }
    return 0;
  };
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i + 1 < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    if (code[i + 1] != code[i] || (i > 0 && code[i - 1] == code[i])) continue;
    size_t e = i + 2;
    while (e < n && e - i <= kTieRun && code[e] == code[i]) ++e;
    if (e - i > kTieRun) {
      // a long run of one key is in order as it is; of several, or too long to see: the words
      bool same = true;
      for (e = i + 1; e < n && code[e] == code[i] && same; ++e) same = e - i < 4096 && compare(order[i], order[e]) == 0;
      if (!same) ctl->mixed = 1;
      continue;
    }
    for (size_t q = i + 1; q < e; ++q) {
      const uint32_t o = order[q];
      size_t r = q;
      for (; r > i && compare(order[r - 1], o) > 0; --r) order[r] = order[r - 1];
      order[r] = o;
    }
  }
}

__global__ void __launch_bounds__(256) soa_gather_kernel(SoaWords src, int K, const uint32_t* __restrict__ order,
                                                         uint64_t* __restrict__ keys) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < src.n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const uint32_t o = order[i];
    for (int k = 0; k < K; ++k) keys[static_cast<size_t>(k) * src.n + i] = src(o, k);
  }
}

__global__ void __launch_bounds__(256) soa_index_kernel(size_t n, const uint32_t* __restrict__ order,
                                                        const uint32_t* __restrict__ idx, uint32_t* __restrict__ out) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    out[i] = idx[order[i]];
}

__global__ void __launch_bounds__(kBlockSortThreads) soa_block_kernel(SoaWords src, int K,
                                                                     const uint32_t* __restrict__ idx,
                                                                     uint64_t* __restrict__ keys,
                                                                     uint32_t* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char raw[];
  BlockSort& sm = *reinterpret_cast<BlockSort*>(raw);
  const int n = static_cast<int>(src.n);
  const uint16_t* order = block_sort(sm, n, K, [&](int k, int i) { return src(i, k); });
  for (int i = threadIdx.x; i < n; i += kBlockSortThreads) {
    const int o = order[i];
    for (int k = 0; k < K; ++k) keys[static_cast<size_t>(k) * n + i] = src(o, k);
    out[i] = idx[o];
  }
}

}  // namespace

namespace wg {

// Keys varying in at most 64 bits are sorted by those bits; wider ones by
// their codes, and only if some equal codes turn out to stand for different
// keys by all their words.  `alike`: the keys are known to agree in long
// stretches, so that codes would tie: the words at once.
// Device memory beside the keys and indices: 24 bytes an item while the pairs are
// sorted, then 4 and a second copy of the indices, then of the keys.
void radix_sort_keys(int device, size_t n, int K, Scratch& keys, Scratch& idx, cudaStream_t s, bool alike) {
  if (n <= 1 || K == 0) return;
  if (n > 0xffffffffull) throw_invalid("sort item count exceeds the index range");
  const SoaWords src{keys.as<uint64_t>(), n};
  if (n <= static_cast<size_t>(kBlockSortItems)) {
    Scratch keys2(sizeof(uint64_t) * K * n, s), idx2(sizeof(uint32_t) * n, s);
    allow_smem(soa_block_kernel, sizeof(BlockSort));
    WG_TIMED("soa_block_kernel", s,
      soa_block_kernel<<<1, kBlockSortThreads, sizeof(BlockSort), s>>>(src, K, idx.as<uint32_t>(),
                                                                     keys2.as<uint64_t>(), idx2.as<uint32_t>()));
    check_launch("launch block sort");
    std::swap(keys, keys2);
    std::swap(idx, idx2);
    return;
  }
  KeyBits kb = key_bits(device, K, n, src, size_t{0}, src, s);
  CodeSpec spec = choose_code(kb, n);
  if (!spec.exact) spec.nb = 64;  // ties cost more here than in a reduction
  const int passes = kb.B == 0 ? 0 : (spec.nb + 7) / 8;
  if (passes == 0) return;  // every key is the same
  const auto* bits = kb.masks.as<unsigned long long>();
  const size_t tiles = pair_tiles(n);
  // the codes and one of the item arrays go when the order, in the other, is known
  Scratch pairs((2 * sizeof(uint64_t) + sizeof(uint32_t)) * n, s), order(sizeof(uint32_t) * n, s);
  const size_t zero_bytes = sizeof(uint64_t) * kDigits * tiles + sizeof(uint32_t) * kDigits * kMaxPasses + sizeof(SortControl);
  Scratch zero(zero_bytes, s);
  check_cuda(cudaMemsetAsync(zero.get(), 0, zero_bytes, s), "clear sort state");
  PairBuffers b{};
  b.k0 = pairs.as<uint64_t>();
  b.k1 = b.k0 + n;
  b.i0 = order.as<uint32_t>();
  b.i1 = reinterpret_cast<uint32_t*>(b.k1 + n);
  if (passes % 2) std::swap(b.i0, b.i1);
  b.status = zero.as<unsigned long long>();
  b.hist = reinterpret_cast<uint32_t*>(b.status + kDigits * tiles);
  b.control = reinterpret_cast<SortControl*>(b.hist + kDigits * kMaxPasses);
  const unsigned g = grid_for(n, 256, device, 4);
  SortControl h{};
  auto outcome = [&] {  // of the look-backs too, which is known only now
    check_cuda(cudaMemcpyAsync(&h, b.control, sizeof(h), cudaMemcpyDeviceToHost, s), "read sort state");
    check_cuda(cudaStreamSynchronize(s), "read sort state");
    if (h.timeout) throw Error(WG_ERR_TIMEOUT, "radix sort: a tile waited too long for its predecessors");
  };
  bool by_words = alike && !spec.exact;
  if (!by_words) {
    allow_smem(soa_code_kernel, digit_smem(kMaxPasses));
    WG_TIMED("soa_code_kernel", s,
      soa_code_kernel<<<g, 256, digit_smem(passes), s>>>(src, K, bits, spec, passes, b.k0, b.hist));
    check_launch("launch sort codes");
    sort_pairs(n, b, passes, true, s);
    if (!spec.exact) {
      soa_check_kernel<<<g, 256, 0, s>>>(b.k0, b.i0, src, K, b.control);
      check_launch("launch sort check");
    }
    outcome();
    if (h.mixed) {
      check_cuda(cudaMemsetAsync(b.control, 0, sizeof(SortControl), s), "clear sort state");
      WG_TIMED("soa_ties_kernel", s, soa_ties_kernel<<<g, 256, 0, s>>>(b.k0, b.i0, src, K, b.control));
      check_launch("launch sort ties");
      outcome();
    }
    by_words = h.mixed != 0;
  }
  if (by_words) {
    allow_smem(soa_word_kernel, digit_smem(kMaxPasses));
    bool first = true;
    for (int k = K - 1; k >= 0; --k) {
      const int count = (kb.vary[k] + 7) / 8;
      if (count == 0) continue;
      check_cuda(cudaMemsetAsync(zero.get(), 0, zero_bytes, s), "clear sort state");
      WG_TIMED("soa_word_kernel", s,
        soa_word_kernel<<<g, 256, digit_smem(count), s>>>(src, k, bits, count, first ? nullptr : b.i0, b.k0, b.hist));
      check_launch("launch sort word");
      sort_pairs(n, b, count, first, s);
      first = false;
      outcome();
    }
  }
  if (b.i0 != order.as<uint32_t>())
    check_cuda(cudaMemcpyAsync(order.get(), b.i0, order.size(), cudaMemcpyDeviceToDevice, s), "copy sort order");
  pairs.release();
  zero.release();
  {
    Scratch idx2(sizeof(uint32_t) * n, s);
    soa_index_kernel<<<g, 256, 0, s>>>(n, order.as<uint32_t>(), idx.as<uint32_t>(), idx2.as<uint32_t>());
    check_launch("launch sort index");
    std::swap(idx, idx2);
  }
  Scratch keys2(sizeof(uint64_t) * K * n, s);
  WG_TIMED("soa_gather_kernel", s,
    soa_gather_kernel<<<g, 256, 0, s>>>(src, K, order.as<uint32_t>(), keys2.as<uint64_t>()));
  check_launch("launch sort gather");
  std::swap(keys, keys2);
}

}  // namespace wg
