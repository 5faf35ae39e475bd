// wg_sort_block.cuh -- key packing, and a stable sort of a few thousand
// multi-word keys by one CTA.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "wg_common.cuh"
#include "wg_sort.cuh"

namespace wg {

// Dynamic shared memory above 48 KB must be allowed per kernel and device; the
// call is cheap and idempotent.
template <class K>
void allow_smem(K kernel, size_t bytes) {
  check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)),
             "set kernel shared memory");
}

}  // namespace wg

namespace wgo {

// The bits of a key (word(k), K words) under the masks `bits`, packed to the
// front of `words` words, handed out in order as put(w, value).
template <class Word, class Put>
__device__ __forceinline__ void pack_key(const unsigned long long* __restrict__ bits, int K, Word&& word, Put&& put,
                                         int words) {
  uint64_t cur = 0;
  int at = 0, base = 0;
  for (int k = 0; k < K; ++k) {
    const uint64_t m = bits[k];
    uint64_t v = word(k) & m;
    while (v) {
      const int b = 63 - __clzll(static_cast<long long>(v));
      v ^= uint64_t{1} << b;
      const int r = base + __popcll(m & ~((uint64_t{2} << b) - 1));
      while (r >= 64 * (at + 1)) {
        put(at++, cur);
        cur = 0;
      }
      cur |= 0x8000000000000000ull >> (r & 63);
    }
    base += __popcll(m);
  }
  while (at < words) {
    put(at++, cur);
    cur = 0;
  }
}

// Per list y: found[y][0][k] = OR of key word k, found[y][1][k] = OR of its
// complement, pop[y] = set bits in all.
template <class A, class C>
__global__ void __launch_bounds__(256) key_bits_kernel(A a, size_t na, C c, size_t nc, int K,
                                                       unsigned long long* __restrict__ found,
                                                       unsigned long long* __restrict__ pop) {
  const int y = blockIdx.y;
  const size_t n = y == 0 ? na : nc;
  unsigned long long set = 0;
  for (int k = 0; k < K; ++k) {
    uint64_t one = 0, none = 0;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
      const uint64_t v = y == 0 ? a(i, k) : c(i, k);
      one |= v;
      none |= ~v;
      set += __popcll(v);
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      one |= __shfl_xor_sync(0xffffffffu, one, o);
      none |= __shfl_xor_sync(0xffffffffu, none, o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (one) atomicOr(found + (2 * y) * K + k, static_cast<unsigned long long>(one));
      if (none) atomicOr(found + (2 * y + 1) * K + k, static_cast<unsigned long long>(none));
    }
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) set += __shfl_xor_sync(0xffffffffu, set, o);
  if ((threadIdx.x & 31) == 0 && set) atomicAdd(pop + y, set);
}

// masks[k] = bits of word k that vary in either list
static __global__ void key_masks_kernel(const unsigned long long* __restrict__ found, int K, int lists,
                                        unsigned long long* __restrict__ masks) {
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    unsigned long long m = 0;
    for (int y = 0; y < lists; ++y) m |= found[2 * y * K + k] & found[(2 * y + 1) * K + k];
    masks[k] = m;
  }
}

// Which key bits vary over one list (nc == 0), or over the XORs of the keys of
// two.  Word(i, k) of a list gives its item i's key word k.  Synchronises s.
template <class A, class C>
KeyBits key_bits(int device, int K, size_t na, const A& a, size_t nc, const C& c, cudaStream_t s) {
  KeyBits kb{};
  kb.side_by_side = nc > 0;
  kb.K = K;
  const int lists = nc > 0 ? 2 : 1;
  const size_t words = 4 * static_cast<size_t>(K) + 2;
  wg::Scratch found(sizeof(uint64_t) * words, s);
  kb.masks.reset(sizeof(uint64_t) * K, s);
  wg::check_cuda(cudaMemsetAsync(found.get(), 0, sizeof(uint64_t) * words, s), "clear key bits");
  auto* f = found.as<unsigned long long>();
  const dim3 grid(wg::grid_for(std::max(na, nc), 256, device, 4), lists);
  WG_TIMED("key_bits_kernel", s, (key_bits_kernel<A, C><<<grid, 256, 0, s>>>(a, na, c, nc, K, f, f + 4 * K)));
  wg::check_launch("launch key bits");
  key_masks_kernel<<<1, 256, 0, s>>>(f, K, lists, kb.masks.as<unsigned long long>());
  wg::check_launch("launch key masks");
  std::vector<unsigned long long> h(words);
  wg::check_cuda(cudaMemcpyAsync(h.data(), f, sizeof(uint64_t) * words, cudaMemcpyDeviceToHost, s), "read key bits");
  wg::check_cuda(cudaStreamSynchronize(s), "read key bits");
  unsigned long long constant[2] = {0, 0};  // set bits that every key of a list has
  for (int k = 0; k < K; ++k) {
    unsigned long long vary = 0;
    for (int y = 0; y < lists; ++y) {
      constant[y] += __builtin_popcountll(~h[(2 * y + 1) * K + k]);
      vary |= h[2 * y * K + k] & h[(2 * y + 1) * K + k];
    }
    kb.vary.push_back(__builtin_popcountll(vary));
    kb.B += kb.vary.back();
  }
  const double B = std::max(1, kb.B);
  const double p = std::min(1.0, static_cast<double>(h[4 * K] - constant[0] * na) / (B * static_cast<double>(na)));
  const double q = nc > 0 ? std::min(1.0, static_cast<double>(h[4 * K + 1] - constant[1] * nc) / (B * static_cast<double>(nc))) : 0.0;
  kb.density = p * (1.0 - q) + q * (1.0 - p);
  return kb;
}

// ------------------------------------------------------- sort by one CTA

constexpr int kBlockSortThreads = 1024;
constexpr int kBlockSortItems = 8192;
constexpr int kBlockSortWarps = kBlockSortThreads / 32;
constexpr int kBlockSortRounds = kBlockSortItems / kBlockSortThreads;

struct __align__(16) BlockSort {
  uint16_t order[2][kBlockSortItems];
  uint32_t count[kDigits * (kBlockSortWarps + 1)];  // [digit][warp], padded against bank conflicts
  uint32_t total[kDigits];
  unsigned long long one, none;
  unsigned long long ones[4], nones[4];
};

// block_sort for up to kWindowItems items whose words (4 at most) vary within
// windows of kWindowBits bits together: false where they do not.  Window bits and
// item number make one 64-bit value, and a bitonic network sorts those (unlike
// one another, so its order is the stable one): a warp's 64 of them by shuffles, the
// others through shared memory, a barrier a step.  1,920 products of 16 qubits took
// 18 us in four 8-bit passes of five barriers and 8,448 counters each; a call 61 us
// with those and 55 with the network.
constexpr int kWindowItems = 2 * kBlockSortThreads, kIndexBits = 11, kWindowBits = 64 - kIndexBits;
static_assert(kWindowItems == 1 << kIndexBits && sizeof(BlockSort::count) >= 2 * 8 * kWindowItems, "two buffers");

template <class Word>
__device__ bool window_sort(BlockSort& sm, int n, int K, Word&& word) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (n > kWindowItems || K > 4) return false;
  if (tid < 4) sm.ones[tid] = sm.nones[tid] = 0;
  __syncthreads();
  const int i0 = 2 * tid;  // the thread's items are i0 and i0 + 1
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (k >= K) break;
    uint64_t one = 0, none = 0;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      if (i0 + e < n) {
        const uint64_t v = word(k, i0 + e);
        one |= v;
        none |= ~v;
      }
    }
    const uint32_t o0 = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(one));
    const uint32_t o1 = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(one >> 32));
    const uint32_t z0 = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(none));
    const uint32_t z1 = __reduce_or_sync(0xffffffffu, static_cast<uint32_t>(none >> 32));
    if (lane == 0) {
      if (o0 | o1) atomicOr(&sm.ones[k], static_cast<unsigned long long>(o1) << 32 | o0);
      if (z0 | z1) atomicOr(&sm.nones[k], static_cast<unsigned long long>(z1) << 32 | z0);
    }
  }
  __syncthreads();
  int low[4], width[4], bits = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const unsigned long long vary = k < K ? sm.ones[k] & sm.nones[k] : 0ull;
    low[k] = vary ? __ffsll(static_cast<long long>(vary)) - 1 : 0;
    width[k] = vary ? 64 - __clzll(static_cast<long long>(vary)) - low[k] : 0;
    bits += width[k];
  }
  if (bits > kWindowBits) return false;  // for all threads alike
  uint64_t a[2];
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    a[e] = ~0ull;  // absent items come last
    if (i0 + e < n) {
      uint64_t c = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (width[k]) c = c << width[k] | ((word(k, i0 + e) >> low[k]) & ((uint64_t{1} << width[k]) - 1));
      a[e] = c << kIndexBits | static_cast<uint64_t>(i0 + e);
    }
  }
  int size = 64;
  while (size < n) size <<= 1;
  ulonglong2* buffer = reinterpret_cast<ulonglong2*>(sm.count);  // [2][kWindowItems / 2]
  int side = 0;
  for (int k = 2; k <= size; k <<= 1) {
    const bool up = (i0 & k) == 0;  // i0 and i0 + 1 alike
    for (int j = k >> 1; j >= 2; j >>= 1) {
      uint64_t b[2];
      if (j >= 64) {
        buffer[side * (kWindowItems / 2) + tid] = make_ulonglong2(a[0], a[1]);
        __syncthreads();
        const ulonglong2 v = buffer[side * (kWindowItems / 2) + (tid ^ (j >> 1))];
        b[0] = v.x;
        b[1] = v.y;
        side ^= 1;  // the next step's buffer was read before this step's barrier
      } else {
        b[0] = __shfl_xor_sync(0xffffffffu, a[0], j >> 1);
        b[1] = __shfl_xor_sync(0xffffffffu, a[1], j >> 1);
      }
      const bool small = ((i0 & j) == 0) == up;
      a[0] = (a[0] < b[0]) == small ? a[0] : b[0];
      a[1] = (a[1] < b[1]) == small ? a[1] : b[1];
    }
    // j = 1: within the thread; for k = 2 its direction is bit 1 of i0
    const uint64_t x = a[0] < a[1] ? a[0] : a[1], y = a[0] < a[1] ? a[1] : a[0];
    a[0] = up ? x : y;
    a[1] = up ? y : x;
  }
#pragma unroll
  for (int e = 0; e < 2; ++e)
    if (i0 + e < n) sm.order[0][i0 + e] = static_cast<uint16_t>(a[e] & (kWindowItems - 1));
  __syncthreads();
  return true;
}

// The items 0..n-1 (n <= kBlockSortItems) in stable ascending order of their
// keys (word(k, item), word 0 most significant), by LSD passes over 8-bit
// windows of the bits that vary.  Returns a shared array; ends with a barrier.
// A pass's time is that of its five barriers and the keys' loads (L1 or L2).
template <class Word>
__device__ const uint16_t* block_sort(BlockSort& sm, int n, int K, Word&& word) {
  if (window_sort(sm, n, K, word)) return sm.order[0];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rounds = (n + kBlockSortThreads - 1) / kBlockSortThreads;
  const int w0 = warp * 32 * rounds;  // a warp's places are consecutive
  const uint32_t below = (1u << lane) - 1u;
  int cur = 0;
  for (int i = tid; i < n; i += kBlockSortThreads) sm.order[0][i] = static_cast<uint16_t>(i);
  for (int k = K - 1; k >= 0; --k) {
    if (tid == 0) sm.one = sm.none = 0;
    __syncthreads();
    {
      uint64_t one = 0, none = 0;
      for (int i = tid; i < n; i += kBlockSortThreads) {
        const uint64_t v = word(k, i);
        one |= v;
        none |= ~v;
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        one |= __shfl_xor_sync(0xffffffffu, one, o);
        none |= __shfl_xor_sync(0xffffffffu, none, o);
      }
      if (lane == 0) {
        if (one) atomicOr(&sm.one, static_cast<unsigned long long>(one));
        if (none) atomicOr(&sm.none, static_cast<unsigned long long>(none));
      }
    }
    __syncthreads();
    uint64_t vary = sm.one & sm.none;
    while (vary) {
      const int shift = __ffsll(static_cast<long long>(vary)) - 1;
      vary &= ~(uint64_t{255} << shift);
      const uint16_t* from = sm.order[cur];
      uint16_t* to = sm.order[cur ^ 1];
      for (int i = tid; i < kDigits * (kBlockSortWarps + 1); i += kBlockSortThreads) sm.count[i] = 0;
      __syncthreads();
      uint32_t digit[kBlockSortRounds], rank[kBlockSortRounds];
#pragma unroll
      for (int r = 0; r < kBlockSortRounds; ++r) {
        const int p = w0 + 32 * r + lane;
        digit[r] = r < rounds && p < n ? static_cast<uint32_t>(word(k, from[p]) >> shift) & 255u : kDigits;
      }
#pragma unroll
      for (int r = 0; r < kBlockSortRounds; ++r) {
        if (r < rounds) {
          const uint32_t same = __match_any_sync(0xffffffffu, digit[r]);
          const uint32_t at = digit[r] * (kBlockSortWarps + 1) + warp;
          const uint32_t before = digit[r] < kDigits ? sm.count[at] : 0;
          __syncwarp();
          const uint32_t mine = __popc(same & below);
          if (mine == 0 && digit[r] < kDigits) sm.count[at] = before + __popc(same);
          __syncwarp();
          rank[r] = before + mine;
        }
      }
      __syncthreads();
      // per digit: the warps' first places; a warp takes 8 digits, a lane a warp's count
#pragma unroll
      for (int e = 0; e < kDigits / kBlockSortWarps; ++e) {
        const int d = warp * (kDigits / kBlockSortWarps) + e;
        const uint32_t c = sm.count[d * (kBlockSortWarps + 1) + lane];
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        sm.count[d * (kBlockSortWarps + 1) + lane] = incl - c;
        if (lane == 31) sm.total[d] = incl;
      }
      __syncthreads();
      if (warp == 0) {
        uint32_t c[kDigits / 32], sum = 0;
#pragma unroll
        for (int e = 0; e < kDigits / 32; ++e) {
          c[e] = sm.total[lane * (kDigits / 32) + e];
          sum += c[e];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        uint32_t at = incl - sum;
#pragma unroll
        for (int e = 0; e < kDigits / 32; ++e) {
          sm.total[lane * (kDigits / 32) + e] = at;
          at += c[e];
        }
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kBlockSortRounds; ++r) {
        const int p = w0 + 32 * r + lane;
        if (r < rounds && p < n)
          to[sm.total[digit[r]] + sm.count[digit[r] * (kBlockSortWarps + 1) + warp] + rank[r]] = from[p];
      }
      cur ^= 1;
      __syncthreads();
    }
  }
  __syncthreads();
  return sm.order[cur];
}

}  // namespace wgo
