// wg_commute.cu -- bit-packed all-pairs commutation matrix and its consumers.
//
// Semantics (reference src/detail/commutation.hpp:10-46, src/commute.cpp:27-93):
// terms l and r commute iff parity(sum_w popc((lx_w & rz_w) ^ (lz_w & rx_w))) == 0.
// Because parity is additive over XOR, all words fold into one 64-bit value
// before a single population count.
//
// Output: bits[row*pitch + c/32] bit (c%32) = 1 iff (row, c) commute.  The
// reference writes one byte per entry (src/cuda/commutation_cuda.cu:123-151);
// the bit matrix is 8x smaller, which is what bounds the kernel at large sizes.

#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

#include "wg_common.cuh"

namespace {

constexpr int kColsPerLane = 8;                    // rhs columns held in registers per lane
constexpr int kWarpCols = 32 * kColsPerLane;       // 256 columns = 8 output words per warp
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsPerWarpIter = 64;               // rows a warp sweeps per column tile

// ---------------------------------------------------------------------------
// algo 1: popcount / LOP3 with warp-ballot packing.
// CTA = one 256-column tile x (kWarps * kRowsPerWarpIter) rows.  Every lane
// keeps the masks of its 8 columns in registers; each row's masks are a
// broadcast load; the 8 ballots of a row give 8 consecutive output words,
// stored by lanes 0..7 as one 32-byte sector.
template <int W>
__global__ void __launch_bounds__(kThreads) commute_ballot_kernel(
    const uint64_t* __restrict__ lx, const uint64_t* __restrict__ lz, size_t n_l,
    const uint64_t* __restrict__ rx, const uint64_t* __restrict__ rz, size_t n_r,
    uint32_t* __restrict__ bits, size_t pitch) {
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const size_t col_tile = blockIdx.x;
  const size_t col0 = col_tile * kWarpCols;
  const size_t words_needed = (n_r + 31) / 32;

  uint64_t cx[kColsPerLane][W], cz[kColsPerLane][W];
  uint32_t valid = 0;  // bit k: column k of this lane exists
#pragma unroll
  for (int k = 0; k < kColsPerLane; ++k) {
    const size_t c = col0 + 32 * k + lane;
    const bool ok = c < n_r;
    valid |= ok ? (1u << k) : 0u;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      cx[k][w] = ok ? __ldg(rx + c * W + w) : 0;
      cz[k][w] = ok ? __ldg(rz + c * W + w) : 0;
    }
  }
  // Word k of this tile holds columns col0 + 32k + lane; mask off absent ones.
  uint32_t word_valid[kColsPerLane];
#pragma unroll
  for (int k = 0; k < kColsPerLane; ++k) word_valid[k] = __ballot_sync(0xffffffffu, (valid >> k) & 1u);

  const size_t row_begin = static_cast<size_t>(blockIdx.y) * (kWarps * kRowsPerWarpIter) + warp;
  const size_t row_end = min(n_l, static_cast<size_t>(blockIdx.y + 1) * (kWarps * kRowsPerWarpIter));
  for (size_t row = row_begin; row < row_end; row += kWarps) {
    uint64_t ax[W], az[W];
#pragma unroll
    for (int w = 0; w < W; ++w) {
      ax[w] = __ldg(lx + row * W + w);
      az[w] = __ldg(lz + row * W + w);
    }
    uint32_t mine = 0;
#pragma unroll
    for (int k = 0; k < kColsPerLane; ++k) {
      uint64_t acc = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) acc ^= (ax[w] & cz[k][w]) ^ (az[w] & cx[k][w]);
      const uint32_t folded = static_cast<uint32_t>(acc) ^ static_cast<uint32_t>(acc >> 32);
      const bool commute = (__popc(folded) & 1u) == 0;
      const uint32_t word = __ballot_sync(0xffffffffu, commute) & word_valid[k];
      if (lane == k) mine = word;
    }
    const size_t wi = col_tile * kColsPerLane + lane;
    if (lane < kColsPerLane && wi < words_needed) bits[row * pitch + wi] = mine;
  }
}

// Generic word count (W > 4): masks read per pair from global/L1.
__global__ void __launch_bounds__(kThreads) commute_generic_kernel(
    const uint64_t* __restrict__ lx, const uint64_t* __restrict__ lz, size_t n_l,
    const uint64_t* __restrict__ rx, const uint64_t* __restrict__ rz, size_t n_r, size_t W,
    uint32_t* __restrict__ bits, size_t pitch) {
  const int lane = threadIdx.x & 31;
  const size_t words_needed = (n_r + 31) / 32;
  const size_t total = n_l * words_needed;
  const size_t warp_global = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  for (size_t item = warp_global; item < total; item += nwarps) {
    const size_t row = item / words_needed;
    const size_t wi = item - row * words_needed;
    const size_t c = wi * 32 + lane;
    bool commute = false;
    if (c < n_r) {
      uint64_t acc = 0;
      for (size_t w = 0; w < W; ++w)
        acc ^= (lx[row * W + w] & rz[c * W + w]) ^ (lz[row * W + w] & rx[c * W + w]);
      commute = (__popcll(acc) & 1u) == 0;
    }
    const uint32_t word = __ballot_sync(0xffffffffu, commute);
    if (lane == 0) bits[row * pitch + wi] = word;
  }
}

// ---------------------------------------------------------------------------
// Dense uint8 flags straight from the masks, without the bit matrix.  A warp
// holds the masks of 32 COLS columns (a lane's columns are 32 apart, so that each
// of its stores is 32 consecutive bytes of the warp) and sweeps rows.  Per pair: 4
// LOP3 per mask word, a population count (a quarter of the issue rate of a LOP3), a
// byte store.  One wave of CTAs, each warp with as many rows as that leaves it, and
// the next row's masks loaded ahead: 4,099^2 flags of 20 qubits 28 us a call (36 with
// 1.4 waves and no loads ahead; 88 through the bit matrix, 36 + 27 us of kernels).
template <int W>
constexpr int kFlagCols = W <= 2 ? 8 : 4;  // columns of a lane
template <int W>
constexpr int kFlagCtas = W == 1 ? 4 : 2;  // CTAs per SM that the registers are held down to

template <int W>
__global__ void __launch_bounds__(kThreads, kFlagCtas<W>) commute_flags_kernel(
    const uint64_t* __restrict__ lx, const uint64_t* __restrict__ lz, size_t n_l, const uint64_t* __restrict__ rx,
    const uint64_t* __restrict__ rz, size_t n_r, uint8_t* __restrict__ out, uint32_t rows_per_warp) {
  constexpr int COLS = kFlagCols<W>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t tile = static_cast<size_t>(blockIdx.x) * (32 * COLS), col0 = tile + lane;
  uint64_t cx[COLS][W], cz[COLS][W];
#pragma unroll
  for (int k = 0; k < COLS; ++k) {
    const size_t c = col0 + 32 * k;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      cx[k][w] = c < n_r ? __ldg(rx + c * W + w) : 0;
      cz[k][w] = c < n_r ? __ldg(rz + c * W + w) : 0;
    }
  }
  const size_t row0 = (static_cast<size_t>(blockIdx.y) * kWarps + warp) * rows_per_warp;
  if (row0 >= n_l) return;
  const int rows = static_cast<int>(min(n_l - row0, static_cast<size_t>(rows_per_warp)));
  uint8_t* o = out + row0 * n_r + col0;
  lx += row0 * W;
  lz += row0 * W;
  auto flag = [&](const uint64_t(&ax)[W], const uint64_t(&az)[W], int k) {
    uint32_t acc = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      acc ^= static_cast<uint32_t>(ax[w]) & static_cast<uint32_t>(cz[k][w]);
      acc ^= static_cast<uint32_t>(az[w]) & static_cast<uint32_t>(cx[k][w]);
      acc ^= static_cast<uint32_t>(ax[w] >> 32) & static_cast<uint32_t>(cz[k][w] >> 32);
      acc ^= static_cast<uint32_t>(az[w] >> 32) & static_cast<uint32_t>(cx[k][w] >> 32);
    }
    return static_cast<uint8_t>(~__popc(acc) & 1);
  };
  // the next row's masks are in flight while a row is worked on
  uint64_t nx[W], nz[W];
#pragma unroll
  for (int w = 0; w < W; ++w) nx[w] = __ldg(lx + w), nz[w] = __ldg(lz + w);
  const int mine = static_cast<int>(min(static_cast<size_t>(COLS), (max(n_r, col0) - col0 + 31) / 32));
  const bool whole = tile + 32 * COLS <= n_r;
  for (int r = 0; r < rows; ++r, o += n_r) {
    uint64_t ax[W], az[W];
    const size_t next = static_cast<size_t>(min(r + 1, rows - 1)) * W;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      ax[w] = nx[w];
      az[w] = nz[w];
      nx[w] = __ldg(lx + next + w);
      nz[w] = __ldg(lz + next + w);
    }
    if (whole) {
#pragma unroll
      for (int k = 0; k < COLS; ++k) o[32 * k] = flag(ax, az, k);
    } else {
#pragma unroll
      for (int k = 0; k < COLS; ++k)
        if (k < mine) o[32 * k] = flag(ax, az, k);
    }
  }
}

// n_qubits == 0: every pair commutes.
__global__ void fill_ones_kernel(uint32_t* bits, size_t rows, size_t cols, size_t pitch) {
  const size_t words_needed = (cols + 31) / 32;
  const size_t total = rows * words_needed;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = i / words_needed;
    const size_t wi = i - row * words_needed;
    const size_t rem = cols - wi * 32;
    bits[row * pitch + wi] = rem >= 32 ? 0xffffffffu : ((1u << rem) - 1u);
  }
}

// ---------------------------------------------------------------------------
// algo 2: bit-plane XOR.  For a block of 1024 LW rhs columns, the planes of qubit
// q are the bit-vectors over the block of the columns that anticommute there with
// an X (their z bits), a Z (their x bits) and a Y (x ^ z).  Row l's output word j
// is the complement of the XOR, over l's support, of word j of the plane of l's
// letter: weight(l) shared-memory reads of LW words per lane instead of 32
// (4 W LOP3 + POPC) per word.
//
// Bound by the shared-memory data path (88 % of its wavefronts used): LW wavefronts
// per set qubit, row and 32 LW words, beside LW for the output and about 3 for the
// row's list.  131,072^2 terms of 128 qubits, weight 6.4, 2.15 GB of output: 0.64 ms
// (with X and Z planes, 256 equal CTAs and planes built by ballots 1.07 ms).
//   - Three planes per qubit, not two with a Y reading both.
//   - A warp takes up to 32 rows; lane r lists row r's planes (16-bit vector
//     indexes, kRowList of them, 24-byte rows: 2-way bank conflicts), which the
//     warp then reads four at a time as a broadcast.  A longer row is listed mask
//     word by mask word by the whole warp when its turn comes.
//   - The launch holds as many CTAs as the device runs at once, and each takes an
//     equal run of (column block, row) pairs: a block's planes are built once or
//     twice per CTA, and no last wave runs part empty.
//   - The planes are built by 32x32 bit transposes; plane vector v of qubit q lies
//     at v ^ (q & 31), so that the 32 qubits that a warp writes at a time fall
//     into different banks.
//   - A lane's LW words are consecutive where the output can be written as
//     vectors, else 32 apart, so that each store is 32 consecutive words.
constexpr int kMaxConfiguredDevices = 64;
constexpr int kRowList = 12;   // planes listed per row beforehand
constexpr int kListBytes = 32 * kRowList * 2 + 64 * 2 + 32;  // per warp: lists, one long row's word, counts

constexpr size_t plane_smem(int W, int LW, int threads) {
  return static_cast<size_t>(64 * W) * 3 * 32 * LW * 4 + static_cast<size_t>(threads / 32) * kListBytes;
}

// Bit i of lane t's result: bit t of lane i's v.
__device__ __forceinline__ uint32_t transpose32(uint32_t v, int lane) {
#pragma unroll
  for (int s = 16, k = 0; s >= 1; s >>= 1, ++k) {
    constexpr uint32_t kLow[5] = {0x0000ffffu, 0x00ff00ffu, 0x0f0f0f0fu, 0x33333333u, 0x55555555u};
    const uint32_t m = kLow[k];  // columns with bit s clear
    const uint32_t y = __shfl_xor_sync(0xffffffffu, v, s);
    v = (lane & s) ? ((v & ~m) | ((y & ~m) >> s)) : ((v & m) | ((y & m) << s));
  }
  return v;
}

template <int LW>
struct WordVec;
template <>
struct WordVec<2> {
  using type = uint2;
};
template <>
struct WordVec<4> {
  using type = uint4;
};

template <int LW>
__device__ __forceinline__ void load_words(uint32_t (&w)[LW], const typename WordVec<LW>::type& v) {
  w[0] = v.x;
  w[1] = v.y;
  if constexpr (LW == 4) {
    w[2] = v.z;
    w[3] = v.w;
  }
}

template <int LW>
__device__ __forceinline__ typename WordVec<LW>::type make_words(const uint32_t (&w)[LW]) {
  if constexpr (LW == 4)
    return make_uint4(w[0], w[1], w[2], w[3]);
  else
    return make_uint2(w[0], w[1]);
}

// acc ^= the cnt planes of a list (8-byte aligned).
template <int LW>
__device__ __forceinline__ void xor_list(uint32_t (&acc)[LW], const typename WordVec<LW>::type* planes,
                                         const uint16_t* list, int cnt, int lane) {
  const uint2* l4 = reinterpret_cast<const uint2*>(list);
  auto plane = [&](uint32_t (&w)[LW], uint32_t entry) { load_words<LW>(w, planes[entry ^ static_cast<uint32_t>(lane)]); };
  int k = 0;
  for (; k + 4 <= cnt; k += 4) {
    const uint2 e = l4[k >> 2];
    uint32_t a[LW], b[LW], c[LW], d[LW];
    plane(a, e.x & 0xffffu);
    plane(b, e.x >> 16);
    plane(c, e.y & 0xffffu);
    plane(d, e.y >> 16);
#pragma unroll
    for (int h = 0; h < LW; ++h) acc[h] ^= a[h] ^ b[h] ^ c[h] ^ d[h];
  }
  if (k < cnt) {
    const uint2 e = l4[k >> 2];
    uint32_t a[LW];
    plane(a, e.x & 0xffffu);
    if (k + 1 < cnt) {
      uint32_t b[LW];
      plane(b, e.x >> 16);
#pragma unroll
      for (int h = 0; h < LW; ++h) a[h] ^= b[h];
    }
    if (k + 2 < cnt) {
      uint32_t c[LW];
      plane(c, e.y & 0xffffu);
#pragma unroll
      for (int h = 0; h < LW; ++h) a[h] ^= c[h];
    }
#pragma unroll
    for (int h = 0; h < LW; ++h) acc[h] ^= a[h];
  }
}

// List entry of qubit q for a letter with bits (x, z): the plane's vector 0 is at
// its index 32 (3 q + letter) + (q & 31).
__device__ __forceinline__ uint16_t plane_entry(int q, uint32_t x, uint32_t z) {
  return static_cast<uint16_t>(((q * 3 + static_cast<int>(x + 2 * z) - 1) << 5) | (q & 31));
}

template <int W, int LW, int THREADS>
__global__ void __launch_bounds__(THREADS) commute_plane_kernel(
    const uint64_t* __restrict__ lx, const uint64_t* __restrict__ lz, size_t n_l,
    const uint64_t* __restrict__ rx, const uint64_t* __restrict__ rz, size_t n_r,
    uint32_t* __restrict__ bits, size_t pitch, size_t total, size_t per_cta) {
  using Vec = typename WordVec<LW>::type;
  constexpr int kWordsCta = 32 * LW;  // output words per row and column block
  constexpr int kWarpsCta = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  Vec* planes = reinterpret_cast<Vec*>(smem);
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  unsigned char* mine = smem + static_cast<size_t>(64 * W) * 3 * kWordsCta * 4 + warp * kListBytes;
  uint16_t* lists = reinterpret_cast<uint16_t*>(mine);                  // [32][kRowList]
  uint16_t* longs = reinterpret_cast<uint16_t*>(mine + 32 * kRowList * 2);  // [64]
  uint8_t* counts = mine + 32 * kRowList * 2 + 128;                     // [32]
  const size_t words_needed = (n_r + 31) / 32;
  const bool vectors = pitch % LW == 0 && (reinterpret_cast<uintptr_t>(bits) & (4 * LW - 1)) == 0;
  const int jstep = vectors ? 1 : 32, jmul = vectors ? LW : 1;  // lane's word h of a block: jmul lane + jstep h

  // per_cta <= total, and the pairs run block by block
  size_t at = min(total, static_cast<size_t>(blockIdx.x) * per_cta);
  const size_t end = min(total, at + per_cta);
  while (at < end) {
    const size_t block = at / n_l, row0 = at - block * n_l;
    const size_t row1 = min(n_l, row0 + (end - at));
    at += row1 - row0;
    const size_t col0 = block * (32 * kWordsCta);
    __syncthreads();  // the planes of the block before are read
    for (int v = warp; v < 32; v += kWarpsCta) {
#pragma unroll
      for (int w = 0; w < W; ++w) {
        uint64_t vx[LW], vz[LW];
#pragma unroll
        for (int h = 0; h < LW; ++h) {
          const size_t c = col0 + 32 * static_cast<size_t>(jmul * v + jstep * h) + lane;
          vx[h] = c < n_r ? __ldg(rx + c * W + w) : 0;
          vz[h] = c < n_r ? __ldg(rz + c * W + w) : 0;
        }
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t x[LW], z[LW], y[LW];
#pragma unroll
          for (int h = 0; h < LW; ++h) {
            x[h] = transpose32(static_cast<uint32_t>(vx[h] >> (32 * half)), lane);
            z[h] = transpose32(static_cast<uint32_t>(vz[h] >> (32 * half)), lane);
            y[h] = x[h] ^ z[h];
          }
          const int q = w * 64 + half * 32 + lane;
          Vec* p = planes + static_cast<size_t>(q) * 96 + (v ^ lane);  // q & 31 == lane
          p[0] = make_words<LW>(z);   // X on the left
          p[32] = make_words<LW>(x);  // Z
          p[64] = make_words<LW>(y);  // Y
        }
      }
    }
    __syncthreads();
    uint32_t valid[LW];
    bool write_ok[LW];
    const size_t wi0 = block * kWordsCta + static_cast<size_t>(jmul * lane);
#pragma unroll
    for (int h = 0; h < LW; ++h) {
      const size_t wi = wi0 + static_cast<size_t>(jstep * h);
      write_ok[h] = wi < words_needed;
      valid[h] = !write_ok[h] ? 0u : (n_r - 32 * wi < 32 ? (1u << (n_r - 32 * wi)) - 1u : 0xffffffffu);
    }
    // up to 32 rows to a warp at a time, fewer where the CTA's run is short
    const size_t batch = min(static_cast<size_t>(32), (row1 - row0 + kWarpsCta - 1) / kWarpsCta);
    for (size_t rbase = row0 + batch * warp; rbase < row1; rbase += batch * kWarpsCta) {
      const int nrows = static_cast<int>(min(batch, row1 - rbase));
      const size_t my = rbase + lane;
      uint64_t mx[W], mz[W];
      int cnt = 0;
#pragma unroll
      for (int w = 0; w < W; ++w) {
        mx[w] = lane < nrows ? __ldg(lx + my * W + w) : 0;
        mz[w] = lane < nrows ? __ldg(lz + my * W + w) : 0;
        cnt += __popcll(mx[w] | mz[w]);
      }
      counts[lane] = static_cast<uint8_t>(cnt <= kRowList ? cnt : 255);
      if (cnt <= kRowList) {
        uint16_t* l = lists + lane * kRowList;
#pragma unroll
        for (int w = 0; w < W; ++w)
          for (uint64_t m = mx[w] | mz[w]; m; m &= m - 1) {
            const int b = __ffsll(static_cast<long long>(m)) - 1;
            *l++ = plane_entry(w * 64 + b, static_cast<uint32_t>(mx[w] >> b) & 1u, static_cast<uint32_t>(mz[w] >> b) & 1u);
          }
      }
      __syncwarp();
      uint32_t* out = bits + rbase * pitch + wi0;
      for (int rr = 0; rr < nrows; ++rr, out += pitch) {
        uint32_t acc[LW];
#pragma unroll
        for (int h = 0; h < LW; ++h) acc[h] = 0xffffffffu;
        const int n = counts[rr];
        if (n != 255) {
          xor_list<LW>(acc, planes, lists + rr * kRowList, n, lane);
        } else {
#pragma unroll
          for (int w = 0; w < W; ++w) {
            const uint64_t ax = __shfl_sync(0xffffffffu, mx[w], rr), az = __shfl_sync(0xffffffffu, mz[w], rr);
            const uint64_t m = ax | az;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
              const int b = 32 * half + lane;
              if ((m >> b) & 1u)
                longs[__popcll(m & ((1ull << b) - 1))] =
                    plane_entry(w * 64 + b, static_cast<uint32_t>(ax >> b) & 1u, static_cast<uint32_t>(az >> b) & 1u);
            }
            __syncwarp();
            xor_list<LW>(acc, planes, longs, __popcll(m), lane);
            __syncwarp();  // before the next word's list
          }
        }
#pragma unroll
        for (int h = 0; h < LW; ++h) acc[h] &= valid[h];
        if (vectors && write_ok[LW - 1]) {
          *reinterpret_cast<Vec*>(out) = make_words<LW>(acc);
        } else {
#pragma unroll
          for (int h = 0; h < LW; ++h)
            if (write_ok[h]) out[jstep * h] = acc[h];
        }
      }
      __syncwarp();  // every lane is done with this batch's lists
    }
  }
}

template <int W>
void launch_ballot(const uint64_t* lx, const uint64_t* lz, size_t n_l, const uint64_t* rx,
                   const uint64_t* rz, size_t n_r, uint32_t* bits, size_t pitch, cudaStream_t s) {
  const size_t col_tiles = (n_r + kWarpCols - 1) / kWarpCols;
  const size_t row_chunks = (n_l + kWarps * kRowsPerWarpIter - 1) / (kWarps * kRowsPerWarpIter);
  if (row_chunks > 65535) {
    // Split the launch along rows to respect gridDim.y.
    const size_t rows_per_launch = 65535ull * kWarps * kRowsPerWarpIter;
    for (size_t r0 = 0; r0 < n_l; r0 += rows_per_launch) {
      const size_t nrows = min(rows_per_launch, n_l - r0);
      launch_ballot<W>(lx + r0 * W, lz + r0 * W, nrows, rx, rz, n_r, bits + r0 * pitch, pitch, s);
    }
    return;
  }
  dim3 grid(static_cast<unsigned>(col_tiles), static_cast<unsigned>(row_chunks));
  WG_TIMED("commute_ballot_kernel", s,
    commute_ballot_kernel<W><<<grid, kThreads, 0, s>>>(lx, lz, n_l, rx, rz, n_r, bits, pitch));
  wg::check_launch("launch commutation (ballot)");
}

template <int W, int LW, int THREADS>
void launch_plane_as(const uint64_t* lx, const uint64_t* lz, size_t n_l, const uint64_t* rx, const uint64_t* rz,
                     size_t n_r, uint32_t* bits, size_t pitch, int device, cudaStream_t s, size_t max_rows) {
  constexpr size_t kColsCta = 1024 * LW;
  constexpr size_t smem = plane_smem(W, LW, THREADS);
  static_assert(smem <= 227 * 1024, "planes and lists of one CTA");
  auto* kernel = commute_plane_kernel<W, LW, THREADS>;
  // The shared-memory opt-in is per device and per kernel; set once per device
  // (std::call_once also orders host threads that launch concurrently).
  static std::once_flag configured[kMaxConfiguredDevices];
  static int resident[kMaxConfiguredDevices];  // CTAs that an SM runs at once
  if (device < 0 || device >= kMaxConfiguredDevices) wg::throw_invalid("CUDA device ordinal is out of range");
  std::call_once(configured[device], [&] {  // a throw leaves the flag unset: the next call retries
    wg::check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)),
                   "configure bit-plane commutation");
    int ctas = 0;
    wg::check_cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ctas, kernel, THREADS, smem),
                   "configure bit-plane commutation");
    resident[device] = std::max(1, ctas);
  });
  const size_t blocks = (n_r + kColsCta - 1) / kColsCta;
  const size_t total = wg::checked_mul(blocks, n_l, "commutation bit matrix");
  // A CTA for each one that the device runs at once, while it has kMinRows rows to
  // build a block's planes for; more of them with max_rows.
  constexpr size_t kMinRows = 64;
  const size_t most = static_cast<size_t>(wg::device_props(device).sm_count) * static_cast<size_t>(resident[device]);
  size_t ctas = std::min(most, (total + kMinRows - 1) / kMinRows);
  if (max_rows) ctas = std::max(ctas, std::min<size_t>(1u << 20, (total + max_rows - 1) / max_rows));
  const size_t per_cta = (total + ctas - 1) / ctas;
  WG_TIMED("commute_plane_kernel", s,
    (kernel<<<static_cast<unsigned>(ctas), THREADS, smem, s>>>(lx, lz, n_l, rx, rz, n_r, bits, pitch, total,
                                                               per_cta)));
  wg::check_launch("launch commutation (bit-plane)");
}

// Candidates of the commutation autotuner (wg_tune.cu) on 1-4 mask words:
//   0 ballot kernel;
//   1 bit-plane, two output words per lane (2,048-column blocks);
//   2 bit-plane, four output words per lane (4,096-column blocks; 1-2 mask words
//     only: the planes of 4,096 columns take 96 KB of shared memory per word);
//   3, 4 as 1, 2 with at most 2,048 rows per CTA (more CTAs than run at once).
// Returns false when the candidate does not serve this width.
// Two words per lane: as many threads as let an SM hold 32 warps beside the planes.
template <int W>
bool launch_candidate_w(int c, const uint64_t* lx, const uint64_t* lz, size_t n_l, const uint64_t* rx,
                        const uint64_t* rz, size_t n_r, uint32_t* bits, size_t pitch, int device, cudaStream_t s) {
  switch (c) {
    case 0: launch_ballot<W>(lx, lz, n_l, rx, rz, n_r, bits, pitch, s); return true;
    case 1:
    case 3:
      launch_plane_as<W, 2, W == 1 ? 256 : W == 2 ? 512 : 1024>(lx, lz, n_l, rx, rz, n_r, bits, pitch, device, s,
                                                                c == 1 ? 0 : 2048);
      return true;
    case 2:
    case 4:
      if constexpr (W <= 2) {
        launch_plane_as<W, 4, 1024>(lx, lz, n_l, rx, rz, n_r, bits, pitch, device, s, c == 2 ? 0 : 2048);
        return true;
      }
      return false;
    default: return false;
  }
}

bool launch_candidate(int c, size_t words, const uint64_t* lx, const uint64_t* lz, size_t n_l, const uint64_t* rx,
                      const uint64_t* rz, size_t n_r, uint32_t* bits, size_t pitch, int device, cudaStream_t s) {
  switch (words) {
    case 1: return launch_candidate_w<1>(c, lx, lz, n_l, rx, rz, n_r, bits, pitch, device, s);
    case 2: return launch_candidate_w<2>(c, lx, lz, n_l, rx, rz, n_r, bits, pitch, device, s);
    case 3: return launch_candidate_w<3>(c, lx, lz, n_l, rx, rz, n_r, bits, pitch, device, s);
    case 4: return launch_candidate_w<4>(c, lx, lz, n_l, rx, rz, n_r, bits, pitch, device, s);
    default: return false;
  }
}

// The measured default block of the bit-plane kernel.  With 4,096 columns (1-2 mask
// words) a row's list and loop are paid half as often as with 2,048: 131,072^2 terms
// of 128 qubits, weight 12.5, 1.24 against 2.24 ms; 16,384^2 46 against 64 us;
// 4,099^2 27.5 both, and smaller products 10-20 % behind.  Up to 2,048 columns the
// wider block would be half empty.
int default_plane_candidate(size_t W, size_t n_l, size_t n_r) {
  return (W <= 2 && n_r > 2048 && n_l >= (size_t{1} << 26) / n_r) ? 2 : 1;
}

// Default choice between the two algorithms, from the sizes and the word
// count alone: it reads no term data, so it costs no device-to-host copy and
// no synchronisation, and a call that uses it can be captured in a CUDA graph.
// Cost model per output word:
//   ballot: 32 pairs * (4W LOP3 + 1 POPC + pack)  ~ 32 * (4W + 2) instructions
//   plane : one 16-byte shared load (4 wavefronts a warp) per set qubit of the
//           lhs row and four words, plus the planes built once per CTA.
// Measured on 131,072^2 terms with a quarter of the bits set (weight 9 of 20, 56
// of 128, 109 of 250): 0.72, 3.9 and 9.9 ms against the ballot kernel's 12.9, 16.7
// and 35.9.  Small products keep the ballot kernel (no planes to build): 256^2 and
// 20 qubits 14 us by ballots, 10 by planes, 64^2 8 and 10.  Callers
// that know the weight pass algo 1 or 2 themselves, and the autotuner's cached
// measurement replaces this rule for shape classes it has searched.
int default_algo(size_t W, size_t n_l, size_t n_r) {
  if (W > 4 || n_r < 512 || n_l < 64) return 1;
  return 2;
}

template <int W>
void launch_flags(const uint64_t* lx, const uint64_t* lz, size_t n_l, const uint64_t* rx, const uint64_t* rz,
                  size_t n_r, uint8_t* out, int device, cudaStream_t s) {
  constexpr int kCols = 32 * kFlagCols<W>;
  const size_t tiles = (n_r + kCols - 1) / kCols;
  // One wave of CTAs while a warp has no more than 64 rows: it reads its columns
  // once for them all.
  const size_t ctas = static_cast<size_t>(wg::device_props(device).sm_count) * kFlagCtas<W>;
  const size_t chunks = std::max<size_t>(1, ctas / tiles);  // along the rows
  size_t rows = std::min<size_t>(64, (n_l + chunks * kWarps - 1) / (chunks * kWarps));
  while ((n_l + rows * kWarps - 1) / (rows * kWarps) > 65535) rows *= 2;
  if (rows > 0x7fffffffu || tiles > 0x7fffffffu) wg::throw_invalid("commutation matrix exceeds the launch grid");
  const dim3 grid(static_cast<unsigned>(tiles), static_cast<unsigned>((n_l + rows * kWarps - 1) / (rows * kWarps)));
  WG_TIMED("commute_flags_kernel", s,
    commute_flags_kernel<W><<<grid, kThreads, 0, s>>>(lx, lz, n_l, rx, rz, n_r, out, static_cast<uint32_t>(rows)));
  wg::check_launch("launch commutation flags");
}

// uint8 flags by commute_flags_kernel: false above 4 mask words and for none.
bool commutation_flags(int device, size_t words, const uint64_t* lx, const uint64_t* lz, size_t n_l,
                       const uint64_t* rx, const uint64_t* rz, size_t n_r, uint8_t* out, cudaStream_t s) {
  switch (words) {
    case 1: launch_flags<1>(lx, lz, n_l, rx, rz, n_r, out, device, s); return true;
    case 2: launch_flags<2>(lx, lz, n_l, rx, rz, n_r, out, device, s); return true;
    case 3: launch_flags<3>(lx, lz, n_l, rx, rz, n_r, out, device, s); return true;
    case 4: launch_flags<4>(lx, lz, n_l, rx, rz, n_r, out, device, s); return true;
    default: return false;
  }
}

// wg_commutation_bits' work.  allow_search = false never measures (the
// no-allocation entry point): cached autotuner choices or the defaults only.
void commutation_bits(int device, size_t words, const uint64_t* lhs_x, const uint64_t* lhs_z, size_t n_lhs,
                      const uint64_t* rhs_x, const uint64_t* rhs_z, size_t n_rhs, uint32_t* bits,
                      size_t pitch_words, int algo, bool allow_search, cudaStream_t stream) {
    if (pitch_words < (n_rhs + 31) / 32) wg::throw_invalid("commutation bit matrix pitch is too small");
    if (algo < 0 || algo > 2) wg::throw_invalid("commutation algo must be 0, 1 or 2");
    if (n_lhs == 0 || n_rhs == 0) return;
    wg::DeviceGuard g(device);
    (void)wg::checked_mul(n_lhs, pitch_words, "commutation bit matrix");
    cudaStream_t s = stream;
    if (words == 0) {
      fill_ones_kernel<<<wg::grid_for(n_lhs * pitch_words, 256, device, 8), 256, 0, s>>>(bits, n_lhs, n_rhs,
                                                                                          pitch_words);
      wg::check_launch("launch commutation fill");
      return;
    }
    if (words <= 4) {
      const int plane = default_plane_candidate(words, n_lhs, n_rhs);
      const int fallback = algo == 1 ? 0 : algo == 2 ? plane : (default_algo(words, n_lhs, n_rhs) == 1 ? 0 : plane);
      int choice = fallback;
      bool done = false;
      if (algo == 0)
        choice = wg::tune_choose(
            wg::kTuneCommute, static_cast<int>(words), wg::ceil_log2(n_lhs), wg::ceil_log2(n_rhs), fallback,
            allow_search, s,
            [&](int c) {
              return launch_candidate(c, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, bits, pitch_words, device,
                                      s);
            },
            &done);
      if (!done && !launch_candidate(choice, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, bits, pitch_words,
                                     device, s))
        launch_candidate(fallback, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, bits, pitch_words, device, s);
      return;
    }
    const size_t items = n_lhs * ((n_rhs + 31) / 32);
    WG_TIMED("commute_generic_kernel", s,
      commute_generic_kernel<<<wg::grid_for(items * 32, 256, device, 8), 256, 0, s>>>(
          lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, words, bits, pitch_words));
    wg::check_launch("launch commutation (generic)");
}

}  // namespace

extern "C" {

int wg_commutation_bits(int device, size_t words, const uint64_t* lhs_x, const uint64_t* lhs_z,
                        size_t n_lhs, const uint64_t* rhs_x, const uint64_t* rhs_z, size_t n_rhs,
                        uint32_t* bits, size_t pitch_words, int algo, wg_stream_t stream) {
  return wg::guarded([&] {
    commutation_bits(device, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, bits, pitch_words, algo, true,
                     stream);
  });
}

}  // extern "C"

namespace {

// One thread per output byte group of 4 (uint32 store of four 0/1 flags).
__global__ void bits_to_u8_kernel(const uint32_t* __restrict__ bits, size_t rows, size_t cols,
                                  size_t pitch, uint8_t* __restrict__ out) {
  const size_t quads = (cols + 3) / 4;
  const size_t total = rows * quads;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t row = i / quads;
    const size_t q = i - row * quads;
    const size_t c0 = q * 4;
    const uint32_t word = bits[row * pitch + c0 / 32];
    const uint32_t nib = (word >> (c0 % 32)) & 0xFu;
    const size_t base = row * cols + c0;
    if (c0 + 4 <= cols && ((reinterpret_cast<uintptr_t>(out) + base) & 3) == 0) {
      const uint32_t v = (nib & 1u) | ((nib >> 1) & 1u) << 8 | ((nib >> 2) & 1u) << 16 | ((nib >> 3) & 1u) << 24;
      *reinterpret_cast<uint32_t*>(out + base) = v;
    } else {
      for (size_t k = 0; k < 4 && c0 + k < cols; ++k) out[base + k] = (nib >> k) & 1u;
    }
  }
}

// Row counts: one warp per row.
__global__ void bits_row_count_kernel(const uint32_t* __restrict__ bits, size_t rows, size_t cols,
                                      size_t pitch, uint64_t* __restrict__ row_counts,
                                      unsigned long long* __restrict__ total) {
  const int lane = threadIdx.x & 31;
  const size_t words = (cols + 31) / 32;
  const size_t warp = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
  const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  unsigned long long mine = 0;
  for (size_t row = warp; row < rows; row += nwarps) {
    unsigned long long cnt = 0;
    for (size_t j = lane; j < words; j += 32) cnt += __popc(bits[row * pitch + j]);
#pragma unroll
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && row_counts) row_counts[row] = cnt;
    mine += cnt;
  }
  if (lane == 0 && total) atomicAdd(total, mine);
}

// Column counts: thread per column, rows in chunks (blockIdx.y), atomics per chunk.
__global__ void bits_col_count_kernel(const uint32_t* __restrict__ bits, size_t rows, size_t cols,
                                      size_t pitch, size_t rows_per_chunk,
                                      unsigned long long* __restrict__ col_counts) {
  const size_t c = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (c >= cols) return;
  const size_t r0 = blockIdx.y * rows_per_chunk;
  const size_t r1 = min(rows, r0 + rows_per_chunk);
  unsigned long long cnt = 0;
  for (size_t r = r0; r < r1; ++r) cnt += (bits[r * pitch + c / 32] >> (c % 32)) & 1u;
  atomicAdd(col_counts + c, cnt);
}

__global__ void u8_row_count_kernel(const uint8_t* __restrict__ f, size_t rows, size_t cols,
                                    uint64_t* __restrict__ row_counts, unsigned long long* __restrict__ total) {
  const int lane = threadIdx.x & 31;
  const size_t warp = (blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x) >> 5;
  const size_t nwarps = (static_cast<size_t>(gridDim.x) * blockDim.x) >> 5;
  unsigned long long mine = 0;
  for (size_t row = warp; row < rows; row += nwarps) {
    unsigned long long cnt = 0;
    for (size_t j = lane; j < cols; j += 32) cnt += f[row * cols + j] != 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    if (lane == 0 && row_counts) row_counts[row] = cnt;
    mine += cnt;
  }
  if (lane == 0 && total) atomicAdd(total, mine);
}

__global__ void u8_col_count_kernel(const uint8_t* __restrict__ f, size_t rows, size_t cols,
                                    size_t rows_per_chunk, unsigned long long* __restrict__ col_counts) {
  const size_t c = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x;
  if (c >= cols) return;
  const size_t r0 = blockIdx.y * rows_per_chunk;
  const size_t r1 = min(rows, r0 + rows_per_chunk);
  unsigned long long cnt = 0;
  for (size_t r = r0; r < r1; ++r) cnt += f[r * cols + c] != 0;
  atomicAdd(col_counts + c, cnt);
}

template <typename RowK, typename ColK>
void run_counts(int device, size_t rows, size_t cols, uint64_t* row_counts, uint64_t* col_counts,
                uint64_t* total, cudaStream_t s, RowK row_launch, ColK col_launch) {
  wg::Scratch tot(sizeof(unsigned long long), s);
  wg::check_cuda(cudaMemsetAsync(tot.get(), 0, sizeof(unsigned long long), s), "clear count");
  if (rows > 0 && cols > 0) {
    row_launch(tot.as<unsigned long long>());
    if (col_counts) {
      wg::check_cuda(cudaMemsetAsync(col_counts, 0, cols * sizeof(uint64_t), s), "clear column counts");
      col_launch(reinterpret_cast<unsigned long long*>(col_counts));
    }
  } else {
    if (row_counts && rows) wg::check_cuda(cudaMemsetAsync(row_counts, 0, rows * 8, s), "clear row counts");
    if (col_counts && cols) wg::check_cuda(cudaMemsetAsync(col_counts, 0, cols * 8, s), "clear column counts");
  }
  if (total) {
    unsigned long long h = 0;
    wg::check_cuda(cudaMemcpyAsync(&h, tot.get(), sizeof(h), cudaMemcpyDeviceToHost, s), "read count");
    wg::check_cuda(cudaStreamSynchronize(s), "read count");
    *total = h;
  }
}

}  // namespace

extern "C" {

int wg_bits_to_u8(int device, const uint32_t* bits, size_t rows, size_t cols, size_t pitch_words,
                  uint8_t* out, wg_stream_t stream) {
  return wg::guarded([&] {
    if (rows == 0 || cols == 0) return;
    wg::DeviceGuard g(device);
    const size_t total = rows * ((cols + 3) / 4);
    WG_TIMED("bits_to_u8_kernel", stream,
      bits_to_u8_kernel<<<wg::grid_for(total, 256, device, 8), 256, 0, stream>>>(bits, rows, cols, pitch_words, out));
    wg::check_launch("launch bits to u8");
  });
}

int wg_bits_count(int device, const uint32_t* bits, size_t rows, size_t cols, size_t pitch_words,
                  uint64_t* row_counts, uint64_t* col_counts, uint64_t* total, wg_stream_t stream) {
  return wg::guarded([&] {
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    run_counts(
        device, rows, cols, row_counts, col_counts, total, s,
        [&](unsigned long long* tot) {
          bits_row_count_kernel<<<wg::grid_for(rows * 32, 256, device, 8), 256, 0, s>>>(bits, rows, cols, pitch_words,
                                                                                       row_counts, tot);
          wg::check_launch("launch row counts");
        },
        [&](unsigned long long* cc) {
          const size_t chunk = 4096;
          dim3 grid(static_cast<unsigned>((cols + 255) / 256), static_cast<unsigned>((rows + chunk - 1) / chunk));
          bits_col_count_kernel<<<grid, 256, 0, s>>>(bits, rows, cols, pitch_words, chunk, cc);
          wg::check_launch("launch column counts");
        });
  });
}

int wg_u8_count(int device, const uint8_t* flags, size_t rows, size_t cols, uint64_t* row_counts,
                uint64_t* col_counts, uint64_t* total, wg_stream_t stream) {
  return wg::guarded([&] {
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    run_counts(
        device, rows, cols, row_counts, col_counts, total, s,
        [&](unsigned long long* tot) {
          u8_row_count_kernel<<<wg::grid_for(rows * 32, 256, device, 8), 256, 0, s>>>(flags, rows, cols, row_counts,
                                                                                     tot);
          wg::check_launch("launch row counts");
        },
        [&](unsigned long long* cc) {
          const size_t chunk = 4096;
          dim3 grid(static_cast<unsigned>((cols + 255) / 256), static_cast<unsigned>((rows + chunk - 1) / chunk));
          u8_col_count_kernel<<<grid, 256, 0, s>>>(flags, rows, cols, chunk, cc);
          wg::check_launch("launch column counts");
        });
  });
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Commutation flags without any device allocation.
//
// Some callers cannot allocate device memory while they use this library: a
// host framework that owns the whole device budget and accounts for every byte
// itself, a caller that must not call cudaMalloc/cudaFree in a latency-critical
// loop (those calls synchronise the device), or a caller that has to keep its
// memory footprint fixed after start-up.  For them the bit-packed matrix that
// the ordinary path keeps in a caller or pool buffer lives here instead, in one
// static device array of kNoAllocScratchBytes.  Every GPU that loads this
// library holds that array until the process exits.
constexpr size_t kNoAllocScratchBytes = size_t{32} << 20;  // 32 MiB
static __device__ __align__(256) uint32_t g_noalloc_bits[kNoAllocScratchBytes / sizeof(uint32_t)];

namespace {

// Device address of g_noalloc_bits on `device`, resolved once per device with
// that device current.  (Host code cannot use the symbol's name as an address.)
uint32_t* noalloc_scratch(int device) {
  static std::mutex mu;
  static std::vector<uint32_t*> addr;
  std::lock_guard<std::mutex> lk(mu);
  if (addr.size() <= static_cast<size_t>(device)) addr.resize(device + 1, nullptr);
  if (!addr[device]) {
    void* p = nullptr;
    wg::check_cuda(cudaGetSymbolAddress(&p, g_noalloc_bits), "resolve the no-allocation scratch address");
    addr[device] = static_cast<uint32_t*>(p);
  }
  return addr[device];
}

}  // namespace

extern "C" int wg_commutation_flags(int device, size_t words, const uint64_t* lhs_x, const uint64_t* lhs_z,
                                    size_t n_lhs, const uint64_t* rhs_x, const uint64_t* rhs_z, size_t n_rhs,
                                    uint8_t* out, wg_stream_t stream) {
  return wg::guarded([&] {
    if (n_lhs == 0 || n_rhs == 0) return;
    wg::DeviceGuard g(device);
    (void)wg::checked_mul(n_lhs, n_rhs, "commutation matrix");
    if (commutation_flags(device, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, out, stream)) return;
    const size_t pitch = (n_rhs + 31) / 32;
    wg::Scratch bits(wg::checked_mul(n_lhs, pitch * 4, "commutation bit matrix"), stream);
    commutation_bits(device, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, bits.as<uint32_t>(), pitch, 0, true,
                     stream);
    const int rc = wg_bits_to_u8(device, bits.as<uint32_t>(), n_lhs, n_rhs, pitch, out, stream);
    if (rc != WG_OK) throw wg::Error(rc, wg_last_error());
  });
}

extern "C" int wg_commutation_u8_noalloc(int device, size_t words, const uint64_t* lhs_x, const uint64_t* lhs_z,
                                         size_t n_lhs, const uint64_t* rhs_x, const uint64_t* rhs_z, size_t n_rhs,
                                         uint8_t* out, wg_stream_t stream) {
  int status = wg::guarded([&] {
    if (n_lhs == 0 || n_rhs == 0) return;
    const size_t pitch = (n_rhs + 31) / 32;
    const size_t bytes = wg::checked_mul(wg::checked_mul(n_lhs, pitch, "commutation bit matrix"), 4,
                                         "commutation bit matrix");
    if (bytes > kNoAllocScratchBytes)
      wg::throw_invalid("commutation matrix too large for the no-allocation path: n_lhs * ceil(n_rhs/32) * 4 = " +
                        std::to_string(bytes) + " bytes exceeds the 32 MiB static scratch");
    wg::DeviceGuard g(device);
    if (commutation_flags(device, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, out, stream)) return;
    uint32_t* bits = noalloc_scratch(device);
    // More than 4 mask words: the ordinary path's kernels do the work; they
    // allocate nothing themselves.  The kernel choice reads no term data and never measures
    // (the autotuner's cached choice or the size rule), so a call after the
    // first synchronises nothing.
    commutation_bits(device, words, lhs_x, lhs_z, n_lhs, rhs_x, rhs_z, n_rhs, bits, pitch, 0, false, stream);
    const int rc = wg_bits_to_u8(device, bits, n_lhs, n_rhs, pitch, out, stream);
    if (rc != WG_OK) throw wg::Error(rc, wg_last_error());
  });
  return status;
}
