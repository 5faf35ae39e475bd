// wg_group.cu -- greedy commuting groups and the Z-count expectation.
//
// group_commuting (reference src/grouping.cpp:197-290):
//   order = terms sorted by (weight desc, canonical key, index)   (:36-62)
//   qwc : a term joins the first group whose OR-basis has no conflict
//         ((tx & gz) ^ (tz & gx)) == 0 in every word               (:64-84)
//   full: a term joins the first group all of whose members commute with it
//                                                                  (:96-126)
//   otherwise it opens a new group.  Groups list members in placement order.
// A term's fate at a group depends only on the earlier terms that reached that
// group, so the first-fit can be run group by group as well as term by term: the
// terms stream, in order, through stages of 32 groups each.  A stage places the
// terms that one of its groups accepts and passes the rest on, in order, and all
// stages work at once on different parts of the stream (see Pipe below).  More
// than 256 qubits: chunks of terms instead, a lower bound for each term over the
// whole GPU and a warp that places them in order (group_bound_n_kernel).

#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <vector>

#include "wg_common.cuh"
#include "wg_scan.cuh"

namespace {

constexpr int kThreads = 256;

// Sort keys for the deterministic order: word 0 = (64 W - weight) so that an
// ascending sort puts heavier terms first, then the canonical key words.
__global__ void order_keys_kernel(const uint64_t* __restrict__ x, const uint64_t* __restrict__ z, size_t T, int W,
                                  uint64_t* __restrict__ keys, uint32_t* __restrict__ idx) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < T;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    uint64_t wgt = 0;
    for (int w = 0; w < W; ++w) {
      const uint64_t a = x[i * W + w], b = z[i * W + w];
      wgt += __popcll(a | b);
      keys[static_cast<size_t>(1 + 2 * w) * T + i] = a;
      keys[static_cast<size_t>(2 + 2 * w) * T + i] = b;
    }
    keys[i] = static_cast<uint64_t>(64 * W) - wgt;  // larger weight -> smaller key
    idx[i] = static_cast<uint32_t>(i);
  }
}

__global__ void gather_terms_kernel(const uint64_t* __restrict__ x, const uint64_t* __restrict__ z,
                                    const uint32_t* __restrict__ order, size_t T, int W, uint64_t* __restrict__ ox,
                                    uint64_t* __restrict__ oz) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < T;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t t = order[i];
    for (int w = 0; w < W; ++w) {
      ox[i * W + w] = x[t * W + w];
      oz[i * W + w] = z[t * W + w];
    }
  }
}

constexpr int kChunk = 1024;     // terms per chunk (qwc), more than 256 qubits
constexpr int kChunkFull = 96;   // terms per chunk in full mode
constexpr int kBoundThreads = 256;
constexpr int kResolveThreads = 256;
// warps that search one term's bound in full mode, warp s every kBoundSplit-th
// round of 32 groups from round s
constexpr int kBoundSplit = 8;

// ------------------------------------------------------------- pipeline
//
// Stage s holds groups 32 s to 32 s + 31, one per lane.  An empty group accepts
// every term, so a stage with room takes the first term it sees that none of its
// groups accepts, which is the sequential first-fit's new group.  The terms that
// a stage passes on lie in one list for all stages: stage s writes its k-th after
// it has read k or more of its predecessor's, so the predecessor's unread ones
// are further on.  status[s] tells how many there are (and kDone when there will
// be no more), and in its upper half how far the stage has read.  Stages take their number by a ticket, so that whoever a stage
// waits for is already running.  A stage may see no term for as long as an earlier
// one takes them all, so a wait gives up only when no earlier stage has read on for
// kPollLimit polls (the upper halves tell; a count of batches that all stages add to
// by atomics made the first stage 3 % slower).
constexpr int kStageGroups = 32;
constexpr unsigned long long kDone = 1ull << 63;
constexpr uint32_t kPollLimit = 1u << 26;  // unless wg_set_wait_limit says otherwise

struct Pipe {
  const uint64_t* ox;            // terms in processing order
  const uint64_t* oz;
  uint32_t n;                    // terms that reach the first stage
  int fresh;                     // they are the positions 0..n-1; else the list's first n entries
  uint32_t* list;
  unsigned long long* status;    // [stages], zeroed
  uint32_t base;                 // first group of the first stage
  uint32_t batch;                // terms taken at a time
  uint32_t limit;                // polls without progress before a wait gives up
  uint32_t* group_of;
  // full mode: members that do not fit in shared memory, in blocks of kBlock
  uint64_t* more;                // [blocks][2 W][kBlock] their words
  uint32_t* next;                // [blocks] a group's next block
};

struct PipeControl {
  uint32_t ticket;
  uint32_t timeout;
  uint32_t groups;  // groups opened so far
  uint32_t blocks;  // blocks of members taken so far (full mode)
};

// Terms passed on, and half of those read above them.
__device__ __forceinline__ unsigned long long stage_status(uint32_t read, uint32_t written) {
  return static_cast<unsigned long long>(read >> 1) << 32 | written;
}

// Terms that stage s can read, and whether more may come; waits until `want`
// are there or the predecessor is done.
__device__ __forceinline__ uint32_t wait_terms(const Pipe& p, uint32_t s, uint32_t have, uint32_t want,
                                               PipeControl* ctl) {
  if (s == 0) return min(want, p.n - have);
  const volatile unsigned long long* st = p.status + s - 1;
  unsigned long long seen = 0;
  bool watched = false;
  for (uint32_t spins = 1;; ++spins) {
    const unsigned long long v = *st;
    const uint32_t there = static_cast<uint32_t>(v & ~kDone) - have;
    if (there >= want || (v & kDone)) {
      __threadfence();
      return min(there, want);
    }
    if (spins >= p.limit) {
      unsigned long long now = 0;
#pragma unroll 1
      for (uint32_t e = 1; e <= s; ++e) now += st[1 - static_cast<int>(e)];
      if (watched && now == seen) {
        ctl->timeout = 1;
        return 0;
      }
      watched = true;
      seen = now;
      spins = 0;
    }
    __nanosleep(64);
  }
}

__device__ __forceinline__ uint32_t stream_term(const Pipe& p, uint32_t s, uint32_t k) {
  return s == 0 && p.fresh ? k : __ldcg(p.list + k);
}

template <int W>
__device__ __forceinline__ void load_term(const uint64_t* t, uint64_t (&r)[2 * W]) {
  const ulonglong2* q = reinterpret_cast<const ulonglong2*>(t);
#pragma unroll
  for (int j = 0; j < W; ++j) {
    const ulonglong2 v = q[j];
    r[2 * j] = v.x;
    r[2 * j + 1] = v.y;
  }
}

// qwc: no qubit on which the term and the basis hold different non-identity
// Paulis.  Rows are [x words | z words].
template <int W>
__device__ __forceinline__ bool row_accepts(const uint64_t (&t)[2 * W], const uint64_t (&b)[2 * W]) {
  uint64_t d = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) d |= (t[w] & b[W + w]) ^ (t[W + w] & b[w]);
  return d == 0;
}

template <int W>
__device__ __forceinline__ bool anticommutes(const uint64_t (&t)[2 * W], const uint64_t (&r)[2 * W]) {
  uint64_t acc = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) acc ^= (t[w] & r[W + w]) ^ (t[W + w] & r[w]);
  return (__popcll(acc) & 1u) != 0;
}

// Places up to 32 terms in order, by one warp: lane j has the groups that accept
// term j (accepts) and the earlier ones of the 32 that it conflicts with
// (against).  A group still accepts a term unless one of the 32 that it conflicts
// with joined the group.  Terms that conflict with none that may be placed go
// where they would go alone, all at once; the others one by one.  Returns the
// lane's term's group, UINT_MAX for none; *joined: terms that joined the lane's
// group.  sm: 32 words of the warp's own.
__device__ __forceinline__ uint32_t place_terms(uint32_t accepts, uint32_t against, uint32_t* sm, uint32_t* joined) {
  const int lane = threadIdx.x & 31;
  const uint32_t some = __ballot_sync(0xffffffffu, accepts != 0);
  *joined = 0;
  if (!some) return UINT_MAX;
  uint32_t mine = UINT_MAX;
  const bool alone = accepts != 0 && !(against & some);
  sm[lane] = 0;
  __syncwarp();
  if (alone) {
    mine = __ffs(accepts) - 1;
    atomicOr(&sm[mine], 1u << lane);
  }
  __syncwarp();
  uint32_t in = sm[lane];
  for (uint32_t rest = some & ~__ballot_sync(0xffffffffu, alone); rest; rest &= rest - 1) {
    const int j = __ffs(rest) - 1;
    const uint32_t a = __shfl_sync(0xffffffffu, accepts, j), c = __shfl_sync(0xffffffffu, against, j);
    const uint32_t ok = __ballot_sync(0xffffffffu, ((a >> lane) & 1u) && !(c & in));
    const int g = __ffs(ok) - 1;  // -1: none
    if (lane == j) mine = static_cast<uint32_t>(g);
    if (lane == g) in |= 1u << j;
  }
  __syncwarp();
  *joined = in;
  return mine;
}

constexpr int kPlaceWarps = 4;    // qwc: warps that check and place
constexpr int kBringWarps = 4;    // and that bring the next batch
constexpr int kQwcThreads = 32 * (kPlaceWarps + kBringWarps);
constexpr int kQwcMost = 512;     // most terms of a batch

// qwc: the placing warps hold the stage's 32 bases, a group per lane, each the
// same.  They take the batch's terms 32 at a time: each checks a quarter against
// the bases as they are (independent checks, one ballot each), then all place
// the 32 (place_terms), each for itself, and update their bases.  The other warps
// bring the next batch in meanwhile, and for each 32 the table of which conflict.
// What bounds the whole is the first stage, which sees every term, at about
// 72 cycles each; one warp that read the groups' bases from shared memory,
// 32 groups at a time, took 510.  65,536 terms on 128 qubits in 1,216 groups:
// 2.5 ms (before: 17.6 and 1.0 ms for the bounds).
template <int W>
__global__ void __launch_bounds__(kQwcThreads) group_qwc_kernel(Pipe pipe, PipeControl* ctl) {
  extern __shared__ __align__(16) unsigned char raw[];
  const uint32_t batch = pipe.batch;
  uint64_t* rows = reinterpret_cast<uint64_t*>(raw);  // [2][batch][2W]
  uint32_t* ids = reinterpret_cast<uint32_t*>(rows + 2 * static_cast<size_t>(batch) * (2 * W));  // [2][batch]
  uint32_t* conflicts = ids + 2 * batch;  // [2][batch] earlier terms of its 32 that a term conflicts with
  uint32_t* got = conflicts + 2 * batch;  // [batch] group in the stage, or UINT_MAX
  __shared__ uint32_t s_stage, s_n[2], s_left[kQwcThreads / 32], s_accepts[2][32], s_in[kPlaceWarps][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kBring = 32 * kBringWarps, kPer = kQwcMost / kBring, kFirst = 32 * kPlaceWarps;
  if (tid == 0) s_stage = atomicAdd(&ctl->ticket, 1u);
  __syncthreads();
  const uint32_t stage = s_stage;
  uint32_t read = 0, written = 0;  // terms taken from the stream, passed on
  // the bringing warps: the next batch into buffer b
  auto bring = [&](int b) {
    if (tid == kFirst) s_n[b] = wait_terms(pipe, stage, read, batch, ctl);
    asm volatile("bar.sync 1, %0;" ::"n"(kBring) : "memory");
    const uint32_t n = s_n[b];
    uint32_t id[kPer];
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const uint32_t k = tid - kFirst + e * kBring;
      id[e] = k < n ? stream_term(pipe, stage, read + k) : 0;
    }
#pragma unroll
    for (int e = 0; e < kPer; ++e) {
      const uint32_t k = tid - kFirst + e * kBring;
      if (k >= n) continue;
      ids[b * batch + k] = id[e];
      uint64_t* row = rows + (b * batch + k) * (2 * W);
#pragma unroll
      for (int w = 0; w < W; ++w) {
        row[w] = __ldg(pipe.ox + static_cast<size_t>(id[e]) * W + w);
        row[W + w] = __ldg(pipe.oz + static_cast<size_t>(id[e]) * W + w);
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kBring) : "memory");
    for (uint32_t t0 = 32 * (warp - kPlaceWarps); t0 < n; t0 += kBring) {
      const uint64_t* block = rows + (b * batch + t0) * (2 * W);
      const uint32_t m = min(32u, n - t0);
      uint64_t t[2 * W], r[2 * W];
      load_term<W>(block + min(static_cast<uint32_t>(lane), m - 1) * (2 * W), t);
      uint32_t mine = 0;
#pragma unroll 4
      for (uint32_t j = 0; j < m; ++j) {
        load_term<W>(block + j * (2 * W), r);
        const uint32_t c = __ballot_sync(0xffffffffu, !row_accepts<W>(t, r));
        if (lane == static_cast<int>(j)) mine = c & ((1u << j) - 1u);
      }
      if (lane < static_cast<int>(m)) conflicts[b * batch + t0 + lane] = mine;
    }
  };
  uint64_t basis[2 * W];
#pragma unroll
  for (int e = 0; e < 2 * W; ++e) basis[e] = 0;
  bool used = false;
  if (warp >= kPlaceWarps) bring(0);
  __syncthreads();
  int cur = 0;
  while (true) {
    const uint32_t n = s_n[cur];
    if (n == 0) break;
    read += n;
    if (warp >= kPlaceWarps) {
      bring(cur ^ 1);
    } else {
      constexpr int kShare = 32 / kPlaceWarps;
      for (uint32_t t0 = 0; t0 < n; t0 += 32) {
        const uint64_t* block = rows + (cur * batch + t0) * (2 * W);
        const uint32_t m = min(32u, n - t0);
        bool ok[kShare];
#pragma unroll
        for (int i = 0; i < kShare; ++i) {
          const uint32_t j = warp * kShare + i;
          uint64_t t[2 * W];
          load_term<W>(block + min(j, m - 1) * (2 * W), t);
          ok[i] = row_accepts<W>(t, basis) && j < m;
        }
        uint32_t mask = 0;
#pragma unroll
        for (int i = 0; i < kShare; ++i) {
          const uint32_t a = __ballot_sync(0xffffffffu, ok[i]);
          if (lane == i) mask = a;
        }
        uint32_t* all = s_accepts[(t0 >> 5) & 1];
        if (lane < kShare) all[warp * kShare + lane] = mask;
        asm volatile("bar.sync 2, %0;" ::"n"(32 * kPlaceWarps) : "memory");
        uint32_t joined;
        const uint32_t mine = place_terms(all[lane], lane < static_cast<int>(m) ? conflicts[cur * batch + t0 + lane] : 0,
                                          s_in[warp], &joined);
        if (warp == 0 && lane < static_cast<int>(m)) got[t0 + lane] = mine;
        used |= joined != 0;
        for (; joined; joined &= joined - 1) {
          uint64_t t[2 * W];
          load_term<W>(block + (__ffs(joined) - 1) * (2 * W), t);
#pragma unroll
          for (int e = 0; e < 2 * W; ++e) basis[e] |= t[e];
        }
        __syncwarp();
      }
    }
    __syncthreads();
    // the placed terms' groups, and the others to the next stage, in order
    for (uint32_t k0 = 0; k0 < n; k0 += kQwcThreads) {
      const uint32_t k = k0 + tid;
      const uint32_t id = k < n ? ids[cur * batch + k] : 0, g = k < n ? got[k] : 0;
      const bool left = k < n && g == UINT_MAX;
      if (k < n && !left) pipe.group_of[id] = pipe.base + stage * kStageGroups + g;
      const uint32_t b = __ballot_sync(0xffffffffu, left);
      if (lane == 0) s_left[warp] = __popc(b);
      __syncthreads();
      uint32_t at = written + __popc(b & ((1u << lane) - 1u));
      uint32_t sum = 0;
      for (int w = 0; w < kQwcThreads / 32; ++w) {
        if (w < warp) at += s_left[w];
        sum += s_left[w];
      }
      if (left) __stcg(pipe.list + at, id);
      written += sum;
      __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) *const_cast<volatile unsigned long long*>(pipe.status + stage) = stage_status(read, written);
    cur ^= 1;
  }
  if (tid == 0) {
    __threadfence();
    *const_cast<volatile unsigned long long*>(pipe.status + stage) = kDone | written;
  }
  if (warp == 0) {
    const uint32_t u = __ballot_sync(0xffffffffu, used);
    if (lane == 0 && u) atomicMax(&ctl->groups, pipe.base + stage * kStageGroups + __popc(u));
  }
}

constexpr int kFullMost = 31;   // most terms of a batch: a warp each, and one that brings the next batch
constexpr uint32_t kScan = 8;   // members checked with a group per lane

// members of each group that a full-mode stage keeps in shared memory
template <int W>
constexpr int kKept = 320 / W;
// words of the m-th members of the 32 groups, and one against bank conflicts
template <int W>
constexpr int kMemberRow = 2 * W * 32 + 1;
// members of a block beyond those (of 32 at 4 words, 2 KB: 8,192 Z strings on 250
// qubits 36 against 13 ms, 16,384 random terms on 200 3.65 against 3.3 ms)
constexpr uint32_t kBlock = 128;

// Blocks that T terms can need: full ones, and a last one for each group with
// more than kKept members.
template <int W>
constexpr size_t member_blocks(size_t T) {
  return T / kBlock + T / (kKept<W> + 1) + 1;
}

// Full mode: a batch of up to 31 terms, a warp each.  A warp checks its term
// against the first 8 members of all groups, a group per lane: of most groups
// one of them anticommutes.  The groups that are left are checked one after
// another, a member per lane, also behind those in shared memory: the words of
// the members beyond lie in blocks of 128, word by word, that all the batch's
// warps read at about the same time (through L1; one lane that followed a linked
// list of members took 811 ms for 16,384 Z strings on 40 qubits, 1,207 ms on
// 128: this takes 25.5 and 35 ms).  Warp 0 then places the batch in order
// (place_terms), while one more warp brings the next batch and the table of
// which of its terms anticommute.  32,768 terms on 128 qubits in 708 groups: 5.0
// ms (before: 60 ms; with a group per lane for all members, which 32 warps load
// again and again: 7.8 ms).
template <int W>
__global__ void __launch_bounds__(1024) group_full_kernel(Pipe pipe, PipeControl* ctl) {
  extern __shared__ __align__(16) unsigned char raw[];
  uint64_t* members = reinterpret_cast<uint64_t*>(raw);  // [kKept][kMemberRow]
  __shared__ __align__(16) uint64_t term[2][kFullMost + 1][2 * W];
  __shared__ uint32_t ids[2][kFullMost + 1], against[2][kFullMost + 1];
  __shared__ uint32_t accepts[32], place[32], slot[32], block[32], s_in[32];
  __shared__ uint32_t count[kStageGroups], first[kStageGroups], last[kStageGroups];  // members, first and last block
  __shared__ uint32_t s_stage, s_n[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int bringer = static_cast<int>(pipe.batch);
  constexpr uint32_t kIn = kKept<W>;
  if (tid == 0) s_stage = atomicAdd(&ctl->ticket, 1u);
  if (tid < kStageGroups) count[tid] = 0;
  __syncthreads();
  const uint32_t stage = s_stage;
  uint32_t read = 0, written = 0;
  auto bring = [&](int b) {
    uint32_t n = 0;
    if (lane == 0) n = wait_terms(pipe, stage, read, pipe.batch, ctl);
    n = __shfl_sync(0xffffffffu, n, 0);
    __threadfence();  // lane 0 saw the count: the others read what lies below it
    uint64_t t[2 * W], r[2 * W];
    const bool has = lane < static_cast<int>(n);
    const uint32_t id = has ? stream_term(pipe, stage, read + lane) : 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
      t[w] = has ? __ldg(pipe.ox + static_cast<size_t>(id) * W + w) : 0;
      t[W + w] = has ? __ldg(pipe.oz + static_cast<size_t>(id) * W + w) : 0;
    }
    if (has) {
      ids[b][lane] = id;
#pragma unroll
      for (int e = 0; e < 2 * W; ++e) term[b][lane][e] = t[e];
    }
    __syncwarp();
    uint32_t mine = 0;
    for (uint32_t j = 0; j < n; ++j) {
      load_term<W>(term[b][j], r);
      const uint32_t c = __ballot_sync(0xffffffffu, anticommutes<W>(t, r));
      if (lane == static_cast<int>(j)) mine = c & ((1u << j) - 1u);
    }
    if (has) against[b][lane] = mine;
    if (lane == 0) s_n[b] = n;
  };
  if (warp == bringer) bring(0);
  __syncthreads();
  int cur = 0;
  while (true) {
    const uint32_t n = s_n[cur];
    if (n == 0) break;
    read += n;
    if (warp == bringer) {
      bring(cur ^ 1);
    } else if (warp < static_cast<int>(n)) {
      uint64_t t[2 * W], r[2 * W];
      load_term<W>(term[cur][warp], t);
      const uint32_t c = count[lane], in = min(c, kIn);
      bool ok = true;
      const uint32_t scan = min(in, kScan);
#pragma unroll 4
      for (uint32_t k = 0; k < kScan; ++k) {
        if (k < scan) {
          const uint64_t* row = members + k * kMemberRow<W> + lane;
#pragma unroll
          for (int e = 0; e < 2 * W; ++e) r[e] = row[32 * e];
          ok = ok && !anticommutes<W>(t, r);
        }
      }
      uint32_t a = __ballot_sync(0xffffffffu, ok);
      for (uint32_t rest = a & __ballot_sync(0xffffffffu, in > kScan); rest; rest &= rest - 1) {
        const int g = __ffs(rest) - 1;
        const uint32_t all = __shfl_sync(0xffffffffu, in, g);
        bool bad = false;
        for (uint32_t k0 = kScan; k0 < all; k0 += 32) {
          const uint32_t k = k0 + lane;
          if (k < all) {
            const uint64_t* row = members + k * kMemberRow<W> + g;
#pragma unroll
            for (int e = 0; e < 2 * W; ++e) r[e] = row[32 * e];
            bad = anticommutes<W>(t, r);
          }
          if (__any_sync(0xffffffffu, bad)) {
            a &= ~(1u << g);
            break;
          }
        }
      }
      // this CTA wrote the blocks before its last barrier: plain loads see them
      for (uint32_t rest = a & __ballot_sync(0xffffffffu, c > kIn); rest; rest &= rest - 1) {
        const int g = __ffs(rest) - 1;
        uint32_t left = __shfl_sync(0xffffffffu, c, g) - kIn;
        for (uint32_t blk = first[g], after;; blk = after) {
          after = pipe.next[blk];  // on its way meanwhile; not set for a last block, nor used
          const uint64_t* words = pipe.more + static_cast<size_t>(blk) * (2 * W * kBlock);
          bool bad = false;
#pragma unroll
          for (uint32_t k0 = 0; k0 < kBlock; k0 += 32) {
            if (k0 + lane < left) {
#pragma unroll
              for (int e = 0; e < 2 * W; ++e) r[e] = words[e * kBlock + k0 + lane];
              bad |= anticommutes<W>(t, r);
            }
          }
          if (__any_sync(0xffffffffu, bad)) {
            a &= ~(1u << g);
            break;
          }
          if (left <= kBlock) break;
          left -= kBlock;
        }
      }
      if (lane == 0) accepts[warp] = a;
    }
    __syncthreads();
    if (warp == 0) {
      const bool has = lane < static_cast<int>(n);
      uint32_t joined;
      const uint32_t mine = place_terms(has ? accepts[lane] : 0, has ? against[cur][lane] : 0, s_in, &joined);
      uint32_t c = count[lane];
      s_in[lane] = joined;
      place[lane] = mine;
      __syncwarp();
      // a term's place in its group: behind the members and the batch's earlier terms
      const uint32_t before = mine == UINT_MAX ? 0 : count[mine] + __popc(s_in[mine] & ((1u << lane) - 1u));
      slot[lane] = before;
      __syncwarp();
      for (uint32_t rest = joined; rest; rest &= rest - 1, ++c) {
        if (c < kIn) continue;
        if ((c - kIn) % kBlock == 0) {
          const uint32_t fresh = atomicAdd(&ctl->blocks, 1u);  // below member_blocks(terms)
          if (c == kIn) first[lane] = fresh;
          else pipe.next[last[lane]] = fresh;
          last[lane] = fresh;
        }
        block[__ffs(rest) - 1] = last[lane];
      }
      count[lane] = c;
      const bool left = has && mine == UINT_MAX;
      const uint32_t b = __ballot_sync(0xffffffffu, left);
      if (left) __stcg(pipe.list + written + __popc(b & ((1u << lane) - 1u)), ids[cur][lane]);
      else if (has) pipe.group_of[ids[cur][lane]] = pipe.base + stage * kStageGroups + mine;
      written += __popc(b);
      __threadfence();
      __syncwarp();
      if (lane == 0) *const_cast<volatile unsigned long long*>(pipe.status + stage) = stage_status(read, written);
    }
    __syncthreads();
    if (warp < static_cast<int>(n) && place[warp] != UINT_MAX && lane < 2 * W) {
      const uint32_t k = slot[warp];
      if (k < kIn) members[k * kMemberRow<W> + 32 * lane + place[warp]] = term[cur][warp][lane];
      else pipe.more[(static_cast<size_t>(block[warp]) * (2 * W) + lane) * kBlock + (k - kIn) % kBlock] = term[cur][warp][lane];
    }
    cur ^= 1;
    __syncthreads();
  }
  if (warp == 0) {
    if (lane == 0) {
      __threadfence();
      *const_cast<volatile unsigned long long*>(pipe.status + stage) = kDone | written;
    }
    const uint32_t u = __ballot_sync(0xffffffffu, count[lane] > 0);
    if (lane == 0 && u) atomicMax(&ctl->groups, pipe.base + stage * kStageGroups + __popc(u));
  }
}

// 64-bit sort keys from group ids; carried index = processing position.
__global__ void widen_ids_kernel(const uint32_t* __restrict__ gid, size_t T, uint64_t* __restrict__ keys,
                                 uint32_t* __restrict__ pos) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < T;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    keys[i] = gid[i];
    pos[i] = static_cast<uint32_t>(i);
  }
}

__global__ void group_head_kernel(const uint64_t* __restrict__ sorted_gid, size_t T, uint32_t* __restrict__ flags) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < T;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    flags[i] = (i == 0 || sorted_gid[i] != sorted_gid[i - 1]) ? 1u : 0u;
}

__global__ void group_out_kernel(const uint32_t* __restrict__ order, const uint32_t* __restrict__ pos_sorted,
                                 const uint32_t* __restrict__ flags, const uint32_t* __restrict__ fpos, size_t T,
                                 uint64_t* __restrict__ order_out, uint64_t* __restrict__ starts) {
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < T;
       i += static_cast<size_t>(gridDim.x) * blockDim.x) {
    order_out[i] = order[pos_sorted[i]];
    if (flags[i]) starts[fpos[i]] = i;
  }
}

// Terms per batch that the autotuner chooses among (candidates 1 and 3 are the
// defaults); every batch gives the same groups.
constexpr uint32_t kQwcBatches[] = {128, 256, 512};
constexpr uint32_t kFullBatches[] = {8, 16, 24, 31};
static_assert(kQwcBatches[2] <= kQwcMost && kFullBatches[3] <= kFullMost, "staging holds a batch");

// Runs the stages, as many as the device holds at once; where terms are left
// behind the last of them, those through as many again.
template <int W>
uint32_t run_pipeline(int device, bool full, Pipe pipe, uint32_t T, cudaStream_t s) {
  const uint32_t stages = static_cast<uint32_t>(wg::device_props(device).sm_count);
  const size_t zero_bytes = sizeof(unsigned long long) * stages + sizeof(PipeControl);
  wg::Scratch zero(zero_bytes, s);
  pipe.status = zero.as<unsigned long long>();
  auto* ctl = reinterpret_cast<PipeControl*>(pipe.status + stages);
  const size_t smem = full ? sizeof(uint64_t) * kKept<W> * kMemberRow<W>
                           : 2 * static_cast<size_t>(pipe.batch) * (16 * W + 8) + 4 * static_cast<size_t>(pipe.batch);
  if (full) {
    wg::check_cuda(cudaFuncSetAttribute(group_full_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(smem)),
                   "set grouping shared memory");
  } else {
    wg::check_cuda(cudaFuncSetAttribute(group_qwc_kernel<W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(smem)),
                   "set grouping shared memory");
  }
  wg::Scratch more, next;
  if (full) {
    const size_t blocks = member_blocks<W>(T);
    more.reset(sizeof(uint64_t) * 2 * W * kBlock * blocks, s);
    next.reset(sizeof(uint32_t) * blocks, s);
    pipe.more = more.as<uint64_t>();
    pipe.next = next.as<uint32_t>();
  }
  pipe.n = T;
  pipe.fresh = 1;
  pipe.base = 0;
  std::vector<unsigned char> host(zero_bytes);
  while (true) {
    wg::check_cuda(cudaMemsetAsync(zero.get(), 0, zero_bytes, s), "clear grouping state");
    const uint32_t need = std::min<uint32_t>(stages, (pipe.n + kStageGroups - 1) / kStageGroups);
    if (full) {
      WG_TIMED("group_full_kernel", s,
        group_full_kernel<W><<<need, 32 * (pipe.batch + 1), smem, s>>>(pipe, ctl));
    } else {
      WG_TIMED("group_qwc_kernel", s, group_qwc_kernel<W><<<need, kQwcThreads, smem, s>>>(pipe, ctl));
    }
    wg::check_launch("launch grouping");
    wg::check_cuda(cudaMemcpyAsync(host.data(), zero.get(), zero_bytes, cudaMemcpyDeviceToHost, s), "read grouping state");
    wg::check_cuda(cudaStreamSynchronize(s), "grouping");
    const auto* st = reinterpret_cast<const unsigned long long*>(host.data());
    const auto* c = reinterpret_cast<const PipeControl*>(st + stages);
    if (c->timeout) throw wg::Error(WG_ERR_TIMEOUT, "grouping: a stage waited too long for its predecessor");
    const uint32_t left = static_cast<uint32_t>(st[need - 1] & ~kDone);
    if (left == 0) return c->groups;
    pipe.n = left;
    pipe.fresh = 0;
    pipe.base += need * kStageGroups;
  }
}

// ------------------------------------------------ any number of mask words
// More than 4 mask words (over 256 qubits): the first-fit by chunks of terms.  The
// whole GPU finds for every term of a chunk the first group that accepts it among
// those that the earlier chunks left (a lower bound: a group only ever accepts
// less), then one warp places the chunk's terms in order from their bounds on.
// Term rows are interleaved once as trows[i] = [x words | z words] (processing
// order) and read word by word; a chunk's are staged in shared memory, the qwc
// basis rows and the full-mode member lists (linked) stay in global memory.  The
// chunk is shortened when its staged rows would not fit in shared memory.

__device__ __forceinline__ bool row_accepts_n(const uint64_t* t, const uint64_t* b, int W) {
  uint64_t d = 0;
  for (int w = 0; w < W; ++w) d |= (t[w] & b[W + w]) ^ (t[W + w] & b[w]);
  return d == 0;
}

// parity of the symplectic product of two [x | z] rows
__device__ __forceinline__ bool anticommutes_n(const uint64_t* t, const uint64_t* row, int W) {
  uint64_t acc = 0;
  for (int w = 0; w < W; ++w) acc ^= (t[w] & row[W + w]) ^ (t[W + w] & row[w]);
  return (__popcll(acc) & 1u) != 0;
}

__device__ __forceinline__ bool members_commute_n(const uint64_t* t, const uint64_t* __restrict__ trows,
                                                  const uint32_t* next, uint32_t m, int W) {
  for (; m != UINT_MAX; m = next[m])
    if (anticommutes_n(t, trows + static_cast<size_t>(m) * (2 * W), W)) return false;
  return true;
}

__global__ void interleave_rows_kernel(const uint64_t* __restrict__ ox, const uint64_t* __restrict__ oz, size_t T,
                                       int W, uint64_t* __restrict__ trows) {
  const size_t n = T * static_cast<size_t>(W);
  for (size_t k = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; k < n;
       k += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const size_t i = k / W, w = k - i * W;
    trows[i * (2 * W) + w] = ox[k];
    trows[i * (2 * W) + W + w] = oz[k];
  }
}

// Full mode: lb[i] = the first group of whose members none anticommutes with term i,
// by kBoundSplit warps a term.
__global__ void __launch_bounds__(kBoundThreads) group_search_full_n_kernel(
    const uint64_t* __restrict__ trows, int W, uint32_t c0, uint32_t c1, const uint32_t* __restrict__ first,
    const uint32_t* __restrict__ next, const uint32_t* __restrict__ n_groups, uint32_t* lb) {
  const uint32_t G0 = *n_groups;
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const uint32_t units = (c1 - c0) * kBoundSplit;
  for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < units; u += nw) {
    const uint32_t i = c0 + u / kBoundSplit, sub = u % kBoundSplit;
    const uint64_t* t = trows + static_cast<size_t>(i) * (2 * W);
    for (uint32_t g0 = sub * 32; g0 < G0; g0 += 32 * kBoundSplit) {
      uint32_t best = 0;
      if (lane == 0) best = *static_cast<volatile uint32_t*>(&lb[i]);
      best = __shfl_sync(0xffffffffu, best, 0);
      if (g0 >= best) break;
      const uint32_t g = g0 + lane;
      const bool ok = g < G0 && members_commute_n(t, trows, next, first[g], W);
      const unsigned b = __ballot_sync(0xffffffffu, ok);
      if (b) {
        if (lane == 0) atomicMin(&lb[i], g0 + __ffs(b) - 1);
        break;
      }
    }
  }
}

// lb[i] = the first group that accepts term i (full mode: as found by the search);
// full mode: lbm[i] = which of the 32 groups from there on do.
__global__ void __launch_bounds__(kBoundThreads) group_bound_n_kernel(
    const uint64_t* __restrict__ trows, int W, uint32_t c0, uint32_t c1, const uint64_t* __restrict__ rows,
    const uint32_t* __restrict__ first, const uint32_t* __restrict__ next, const uint32_t* __restrict__ n_groups,
    uint32_t* __restrict__ lb, uint32_t* __restrict__ lbm, int full) {
  const uint32_t G0 = *n_groups;
  const int lane = threadIdx.x & 31;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  for (uint32_t i = c0 + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); i < c1; i += nw) {
    const uint64_t* t = trows + static_cast<size_t>(i) * (2 * W);
    uint32_t found = G0;
    if (full) {
      found = min(lb[i], G0);
    } else {
      for (uint32_t g0 = 0; g0 < G0; g0 += 32) {
        const uint32_t g = g0 + lane;
        const bool ok = g < G0 && row_accepts_n(t, rows + static_cast<size_t>(g) * (2 * W), W);
        const unsigned b = __ballot_sync(0xffffffffu, ok);
        if (b) {
          found = g0 + __ffs(b) - 1;
          break;
        }
      }
    }
    __syncwarp();
    if (lane == 0) lb[i] = found;
    if (full) {
      const uint32_t g = found + lane;
      const bool ok = g < G0 && members_commute_n(t, trows, next, first[g], W);
      const unsigned m = __ballot_sync(0xffffffffu, ok);
      if (lane == 0) lbm[i] = m;
    }
  }
}

// Places a chunk's n terms in order, qwc, by one warp: lane g % 32 owns basis row g in
// global memory.  Returns the number of groups.
__device__ uint32_t place_qwc_n(const uint64_t* st, const uint32_t* slb, uint32_t* sgid, uint32_t n, uint32_t G,
                                uint64_t* B, int W) {
  const uint32_t lane = threadIdx.x & 31;
  const size_t rw = 2 * static_cast<size_t>(W);
  uint32_t k = 0;
  while (k < n) {
    uint32_t l = 0;
    for (; k < n; ++k) {
      const uint64_t* t = st + k * rw;
      l = slb[k];
      const uint32_t g = l + ((lane - l) & 31u);
      const bool ok = g < G && row_accepts_n(t, B + g * rw, W);
      const uint32_t best = __reduce_min_sync(0xffffffffu, ok ? g : UINT_MAX);
      if (best == UINT_MAX) break;
      if (best % 32 == lane)
        for (size_t e = 0; e < rw; ++e) B[best * rw + e] |= t[e];
      if (lane == 0) sgid[k] = best;
    }
    if (k >= n) break;
    const uint64_t* t = st + k * rw;
    uint32_t best = UINT_MAX;
    for (uint32_t g0 = l + 32; best == UINT_MAX && g0 < G; g0 += 32) {
      const uint32_t g = g0 + ((lane - g0) & 31u);
      const bool ok = g < G && row_accepts_n(t, B + g * rw, W);
      best = __reduce_min_sync(0xffffffffu, ok ? g : UINT_MAX);
    }
    const bool fresh = best == UINT_MAX;
    if (fresh) best = G;
    if (best % 32 == lane)
      for (size_t e = 0; e < rw; ++e) B[best * rw + e] = fresh ? t[e] : (B[best * rw + e] | t[e]);
    if (fresh) ++G;
    if (lane == 0) sgid[k] = best;
    ++k;
  }
  return G;
}

// The same in full mode: members that joined in this chunk are checked from its staged
// rows, the others were by the bound.
__device__ uint32_t place_full_n(const uint64_t* __restrict__ trows, const uint64_t* st, const uint32_t* slb,
                                 const uint32_t* smask, uint32_t* sgid, uint32_t n, uint32_t c0, uint32_t G0,
                                 uint32_t* first, uint32_t* last, uint32_t* next, int W) {
  const uint32_t lane = threadIdx.x & 31;
  const size_t rw = 2 * static_cast<size_t>(W);
  uint32_t G = G0;
  auto chunk_members_commute = [&](const uint64_t* t, uint32_t g, uint32_t k) {
    for (uint32_t q = 0; q < k; ++q)
      if (sgid[q] == g && anticommutes_n(t, st + q * rw, W)) return false;
    return true;
  };
  auto place = [&](uint32_t k, uint32_t best, bool fresh) {
    if ((k & 31u) == lane) sgid[k] = best;
    if (lane == 0) {
      const uint32_t i = c0 + k;
      next[i] = UINT_MAX;
      if (fresh) first[best] = i;
      else next[last[best]] = i;
      last[best] = i;
    }
  };
  uint32_t k = 0;
  while (k < n) {
    uint32_t l = 0;
    for (; k < n; ++k) {
      const uint64_t* t = st + k * rw;
      l = slb[k];
      if (l >= G0) break;
      bool bad = false;
      for (uint32_t q = lane; q < k; q += 32)
        if (sgid[q] == l && anticommutes_n(t, st + q * rw, W)) bad = true;
      if (__any_sync(0xffffffffu, bad)) break;
      place(k, l, false);
    }
    if (k >= n) break;
    __syncwarp();
    const uint64_t* t = st + k * rw;
    const uint32_t m = smask[k];
    uint32_t best = UINT_MAX;
    {
      const uint32_t g = l + lane;
      const bool ok = l < G0 && lane > 0 && g < G0 && ((m >> lane) & 1u) && chunk_members_commute(t, g, k);
      best = __reduce_min_sync(0xffffffffu, ok ? g : UINT_MAX);
    }
    for (uint32_t g0 = l + 32; best == UINT_MAX && g0 < G0; g0 += 32) {
      const uint32_t g = g0 + lane;
      const bool ok = g < G0 && members_commute_n(t, trows, next, first[g], W);
      best = __reduce_min_sync(0xffffffffu, ok ? g : UINT_MAX);
    }
    for (uint32_t g0 = G0; best == UINT_MAX && g0 < G; g0 += 32) {
      const uint32_t g = g0 + lane;
      const bool ok = g < G && chunk_members_commute(t, g, k);
      best = __reduce_min_sync(0xffffffffu, ok ? g : UINT_MAX);
    }
    const bool fresh = best == UINT_MAX;
    if (fresh) best = G;
    place(k, best, fresh);
    if (fresh) ++G;
    __syncwarp();
    ++k;
  }
  return G;
}

// One CTA: stages the chunk's rows, up to cap_terms, and its first warp places them.
__global__ void __launch_bounds__(kResolveThreads) group_resolve_n_kernel(
    const uint64_t* __restrict__ trows, int W, uint32_t c0, uint32_t c1, uint32_t cap_terms, uint64_t* rows,
    uint32_t* first, uint32_t* last, uint32_t* next, const uint32_t* __restrict__ lb,
    const uint32_t* __restrict__ lbm, uint32_t* __restrict__ group_of, uint32_t* __restrict__ n_groups, int full) {
  extern __shared__ __align__(16) unsigned char nraw[];
  const size_t rw = 2 * static_cast<size_t>(W);
  const uint32_t n = c1 - c0;
  uint64_t* st = reinterpret_cast<uint64_t*>(nraw);
  uint32_t* slb = reinterpret_cast<uint32_t*>(st + static_cast<size_t>(cap_terms) * rw);
  uint32_t* sgid = slb + cap_terms;
  uint32_t* smask = sgid + cap_terms;
  const uint32_t G0 = *n_groups;
  for (size_t k = threadIdx.x; k < n * rw; k += blockDim.x) st[k] = trows[static_cast<size_t>(c0) * rw + k];
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    slb[k] = lb[c0 + k];
    if (full) smask[k] = lbm[c0 + k];
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const uint32_t G = full ? place_full_n(trows, st, slb, smask, sgid, n, c0, G0, first, last, next, W)
                            : place_qwc_n(st, slb, sgid, n, G0, rows, W);
    if (threadIdx.x == 0) *n_groups = G;
  }
  __syncthreads();
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) group_of[c0 + k] = sgid[k];
}

void run_greedy_n(int device, bool full, int W, const uint64_t* trows, uint32_t T, uint64_t* rows, uint32_t* first,
                  uint32_t* last, uint32_t* next, uint32_t* lb, uint32_t* lbm, uint32_t* gid, uint32_t* ng,
                  cudaStream_t s) {
  const auto& props = wg::device_props(device);
  const size_t per_term = 16 * static_cast<size_t>(W) + 12;  // staged row, bound, group id, bound mask
  const size_t smem_max = static_cast<size_t>(props.max_smem_optin);
  const uint32_t want = full ? kChunkFull : kChunk;
  const uint32_t chunk = static_cast<uint32_t>(std::min<size_t>(want, smem_max / per_term));
  if (chunk == 0) wg::throw_invalid("group_commuting: a term row does not fit in shared memory");
  const size_t smem = static_cast<size_t>(chunk) * per_term;
  wg::check_cuda(cudaFuncSetAttribute(group_resolve_n_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(smem)),
                 "set group resolve shared memory");
  wg::check_cuda(cudaMemsetAsync(ng, 0, 4, s), "clear group count");
  const unsigned max_blocks = static_cast<unsigned>(props.sm_count) * 8;
  for (uint32_t c0 = 0; c0 < T; c0 += chunk) {
    const uint32_t c1 = T - c0 > chunk ? c0 + chunk : T;
    const unsigned blocks = std::min<unsigned>(max_blocks, (c1 - c0 + kBoundThreads / 32 - 1) / (kBoundThreads / 32));
    if (full) {
      wg::check_cuda(cudaMemsetAsync(lb + c0, 0xff, 4 * static_cast<size_t>(c1 - c0), s), "clear bounds");
      const unsigned sblocks = std::min<unsigned>(
          max_blocks, ((c1 - c0) * kBoundSplit + kBoundThreads / 32 - 1) / (kBoundThreads / 32));
      WG_TIMED("group_search_full_n_kernel", s,
        group_search_full_n_kernel<<<sblocks, kBoundThreads, 0, s>>>(trows, W, c0, c1, first, next, ng, lb));
      wg::check_launch("launch group bound search");
    }
    WG_TIMED("group_bound_n_kernel", s,
      group_bound_n_kernel<<<blocks, kBoundThreads, 0, s>>>(trows, W, c0, c1, rows, first, next, ng, lb, lbm,
                                                            full ? 1 : 0));
    wg::check_launch("launch group bounds");
    WG_TIMED("group_resolve_n_kernel", s,
      group_resolve_n_kernel<<<1, kResolveThreads, smem, s>>>(trows, W, c0, c1, chunk, rows, first, last, next, lb,
                                                              lbm, gid, ng, full ? 1 : 0));
    wg::check_launch("launch group resolve");
  }
}

// ---------------------------------------------------------------- Z counts

__global__ void or_reduce_kernel(const uint64_t* __restrict__ v, size_t n, unsigned long long* __restrict__ out) {
  uint64_t acc = 0;
  for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
       i += static_cast<size_t>(gridDim.x) * blockDim.x)
    acc |= v[i];
#pragma unroll
  for (int o = 16; o; o >>= 1) acc |= __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0 && acc) atomicOr(out, static_cast<unsigned long long>(acc));
}

// Block per term: weighted parity sum over rows, then c_k * (sum / total).
__global__ void __launch_bounds__(kThreads) zcount_terms_kernel(const uint64_t* __restrict__ z, size_t T, int W,
                                                               const uint64_t* __restrict__ packed,
                                                               const double* __restrict__ counts, size_t rows,
                                                               double* __restrict__ weighted) {
  __shared__ double red[kThreads / 32];
  for (size_t t = blockIdx.x; t < T; t += gridDim.x) {
    double acc = 0.0;
    for (size_t r = threadIdx.x; r < rows; r += kThreads) {
      unsigned odd = 0;
      for (int w = 0; w < W; ++w) odd ^= __popcll(z[t * W + w] & packed[r * W + w]) & 1u;
      acc += odd ? -counts[r] : counts[r];
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      double s = 0.0;
      for (int w = 0; w < kThreads / 32; ++w) s += red[w];
      weighted[t] = s;
    }
    __syncthreads();
  }
}

__global__ void zcount_total_kernel(const double* __restrict__ c, const double* __restrict__ weighted, size_t T,
                                    const double* __restrict__ counts, size_t rows, double* __restrict__ out) {
  // single thread: sums in the reference's order (total over rows, then terms)
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double total = 0.0;
  for (size_t r = 0; r < rows; ++r) total += counts[r];
  double re = 0.0, im = 0.0;
  for (size_t t = 0; t < T; ++t) {
    const double f = weighted[t] / total;
    re += c[2 * t] * f;
    im += c[2 * t + 1] * f;
  }
  out[0] = re;
  out[1] = im;
}

}  // namespace

extern "C" {

int wg_group_commuting(int device, size_t words, size_t n_terms, const uint64_t* x, const uint64_t* z, int mode_full,
                       size_t* order_out, size_t* sizes_out, size_t* n_groups, wg_stream_t stream) {
  return wg::guarded([&] {
    *n_groups = 0;
    if (n_terms == 0) return;
    if (n_terms >= 0xffffffffull) wg::throw_invalid("group_commuting supports fewer than 2^32-1 terms");
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    const size_t T = n_terms;
    const int W = static_cast<int>(words);
    const int K = 1 + 2 * W;
    wg::Scratch keys(8 * K * T, s), idx(4 * T, s);
    order_keys_kernel<<<wg::grid_for(T, kThreads, device, 4), kThreads, 0, s>>>(x, z, T, W, keys.as<uint64_t>(),
                                                                                idx.as<uint32_t>());
    wg::check_launch("launch order keys");
    wg::radix_sort_keys(device, T, K, keys, idx, s);
    keys.release();
    const uint32_t* order = idx.as<uint32_t>();
    const size_t Wa = W > 0 ? W : 1;
    wg::Scratch ox(8 * Wa * T, s), oz(8 * Wa * T, s);
    if (W > 0) {
      gather_terms_kernel<<<wg::grid_for(T, kThreads, device, 4), kThreads, 0, s>>>(x, z, order, T, W,
                                                                                   ox.as<uint64_t>(), oz.as<uint64_t>());
      wg::check_launch("launch gather terms");
    } else {
      wg::check_cuda(cudaMemsetAsync(ox.get(), 0, 8 * T, s), "clear masks");
      wg::check_cuda(cudaMemsetAsync(oz.get(), 0, 8 * T, s), "clear masks");
    }
    const bool full = mode_full != 0;
    const uint32_t T32 = static_cast<uint32_t>(T);
    wg::Scratch gid(4 * T, s);
    uint32_t G = 0;
    if (W <= 4) {
      wg::Scratch list(4 * T, s);
      auto place = [&](uint32_t batch) {
        Pipe pipe{};
        pipe.ox = ox.as<uint64_t>();
        pipe.oz = oz.as<uint64_t>();
        pipe.list = list.as<uint32_t>();
        pipe.group_of = gid.as<uint32_t>();
        pipe.batch = batch;
        pipe.limit = wg::wait_limit(kPollLimit);
        switch (W) {
          case 0:
          case 1: G = run_pipeline<1>(device, full, pipe, T32, s); break;
          case 2: G = run_pipeline<2>(device, full, pipe, T32, s); break;
          case 3: G = run_pipeline<3>(device, full, pipe, T32, s); break;
          default: G = run_pipeline<4>(device, full, pipe, T32, s); break;
        }
      };
      // terms per batch: the autotuner's choice for (mode, words, log2 terms)
      const uint32_t* cands = full ? kFullBatches : kQwcBatches;
      bool done = false;
      const int choice = wg::tune_choose(
          full ? wg::kTuneGroupFull : wg::kTuneGroupQwc, W, wg::ceil_log2(T), 0, full ? 3 : 1, true, s,
          [&](int c) {
            place(cands[c]);
            return true;
          },
          &done);
      if (!done) place(cands[choice]);
    } else {
      wg::Scratch rows(16 * Wa * T, s), first(4 * T, s), last(4 * T, s), next(4 * T, s), lb(4 * T, s), lbm(4 * T, s), ng(4, s),
          trows(16 * Wa * T, s);
      WG_TIMED("interleave_rows_kernel", s,
        interleave_rows_kernel<<<wg::grid_for(T * W, kThreads, device, 4), kThreads, 0, s>>>(
            ox.as<uint64_t>(), oz.as<uint64_t>(), T, W, trows.as<uint64_t>()));
      wg::check_launch("launch interleave rows");
      run_greedy_n(device, full, W, trows.as<uint64_t>(), T32, rows.as<uint64_t>(), first.as<uint32_t>(),
                   last.as<uint32_t>(), next.as<uint32_t>(), lb.as<uint32_t>(), lbm.as<uint32_t>(),
                   gid.as<uint32_t>(), ng.as<uint32_t>(), s);
      wg::check_cuda(cudaMemcpyAsync(&G, ng.get(), 4, cudaMemcpyDeviceToHost, s), "read group count");
      wg::check_cuda(cudaStreamSynchronize(s), "group greedy");
    }
    // Stable partition of processing positions by group id.
    wg::Scratch gkeys(8 * T, s), pos(4 * T, s);
    widen_ids_kernel<<<wg::grid_for(T, kThreads, device, 4), kThreads, 0, s>>>(gid.as<uint32_t>(), T,
                                                                             gkeys.as<uint64_t>(), pos.as<uint32_t>());
    wg::check_launch("launch group id widen");
    wg::radix_sort_keys(device, T, 1, gkeys, pos, s);
    wg::Scratch flags(4 * T, s), fpos(4 * T, s), out_order(8 * T, s), starts(8 * (size_t(G) + 1), s);
    const unsigned gr = wg::grid_for(T, kThreads, device, 4);
    group_head_kernel<<<gr, kThreads, 0, s>>>(gkeys.as<uint64_t>(), T, flags.as<uint32_t>());
    wg::check_launch("launch group heads");
    wgs::exclusive_scan<uint32_t>(flags.as<uint32_t>(), fpos.as<uint32_t>(), T, nullptr, s);
    group_out_kernel<<<gr, kThreads, 0, s>>>(order, pos.as<uint32_t>(), flags.as<uint32_t>(), fpos.as<uint32_t>(), T,
                                             out_order.as<uint64_t>(), starts.as<uint64_t>());
    wg::check_launch("launch group output");
    std::vector<uint64_t> hs(static_cast<size_t>(G) + 1);
    static_assert(sizeof(size_t) == sizeof(uint64_t), "size_t must be 64-bit");
    wg::check_cuda(cudaMemcpyAsync(order_out, out_order.get(), 8 * T, cudaMemcpyDeviceToHost, s), "read groups");
    wg::check_cuda(cudaMemcpyAsync(hs.data(), starts.get(), 8 * G, cudaMemcpyDeviceToHost, s), "read groups");
    wg::check_cuda(cudaStreamSynchronize(s), "read groups");
    hs[G] = T;
    for (uint32_t k = 0; k < G; ++k) sizes_out[k] = hs[k + 1] - hs[k];
    *n_groups = G;
  });
}

int wg_expectation_z_counts(int device, size_t words, size_t n_terms, const uint64_t* x, const uint64_t* z,
                            const double* coeffs, size_t rows, const uint64_t* packed, const double* counts,
                            double* result_host, wg_stream_t stream) {
  return wg::guarded([&] {
    result_host[0] = result_host[1] = 0.0;
    wg::DeviceGuard g(device);
    cudaStream_t s = stream;
    if (n_terms > 0 && words > 0) {
      wg::Scratch o(8, s);
      wg::check_cuda(cudaMemsetAsync(o.get(), 0, 8, s), "clear");
      or_reduce_kernel<<<wg::grid_for(n_terms * words, kThreads, device, 4), kThreads, 0, s>>>(
          x, n_terms * words, o.as<unsigned long long>());
      wg::check_launch("launch diagonal check");
      unsigned long long h = 0;
      wg::check_cuda(cudaMemcpyAsync(&h, o.get(), 8, cudaMemcpyDeviceToHost, s), "read diagonal check");
      wg::check_cuda(cudaStreamSynchronize(s), "read diagonal check");
      if (h != 0) wg::throw_invalid("expectation_z_counts requires diagonal Pauli terms");
    }
    if (n_terms == 0) return;
    wg::Scratch weighted(8 * n_terms, s), res(16, s);
    const unsigned grid = static_cast<unsigned>(std::min<size_t>(n_terms, 65535));
    WG_TIMED("zcount_terms_kernel", s,
      zcount_terms_kernel<<<grid, kThreads, 0, s>>>(z, n_terms, static_cast<int>(words), packed, counts, rows,
                                                    weighted.as<double>()));
    wg::check_launch("launch z-count terms");
    zcount_total_kernel<<<1, 32, 0, s>>>(coeffs, weighted.as<double>(), n_terms, counts, rows, res.as<double>());
    wg::check_launch("launch z-count total");
    wg::check_cuda(cudaMemcpyAsync(result_host, res.get(), 16, cudaMemcpyDeviceToHost, s), "read z-count result");
    wg::check_cuda(cudaStreamSynchronize(s), "read z-count result");
  });
}

}  // extern "C"
