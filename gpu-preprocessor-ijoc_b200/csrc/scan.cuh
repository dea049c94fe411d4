// Single-pass prefix sums and stream selections over any per-item function.
//
// One launch does what took a flag kernel, two scan kernels and a gather: a
// tile evaluates its items, publishes its sums, finds the sums of the tiles
// before it by a decoupled look-back and hands every item its prefix.  Tiles
// are taken from a ticket counter, so every tile that a look-back waits for is
// running; a wait still gives up after kScanPolls polls and sets the context's
// error word, which the host checks at its next wait.  The published words
// come from a workspace of the context that every launch leaves zeroed (the
// last block to finish clears what the launch used), so nothing is cleared
// beforehand.
#pragma once

#include "common.cuh"

namespace gpp {

constexpr int kScanItems = 8;
constexpr int kScanTile = kThreads * kScanItems;
constexpr int kScanPolls = 1 << 22;
// A published word: two flag bits (1 the tile's own sum, 2 the sum of all
// tiles up to it) over a 62-bit value.
constexpr unsigned long long kScanOwn = 1ull << 62, kScanAll = 2ull << 62, kScanValue = (1ull << 62) - 1;

// Zeroed words for one launch: `words` published words and two counters.
// Launches on the context's own stream share its workspace; on another stream
// the words belong to this object.
struct LookbackSpace {
  unsigned long long* words = nullptr;
  unsigned int* counters = nullptr;   // ticket, blocks done
  DBuf<unsigned long long> own;
  LookbackSpace(size_t count, cudaStream_t s);
};

__device__ __forceinline__ unsigned long long ld_published(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_published(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Sum of the tiles before tile t, by one warp: 32 predecessors per round,
// their own sums added back to the nearest sum of all (before tile 0: zero).
__device__ __forceinline__ long long scan_lookback(const unsigned long long* words, int64_t t, int32_t* error) {
  const int lane = threadIdx.x & 31;
  unsigned long long before = 0;
  for (int64_t end = t - 1;; end -= 32) {
    const int64_t j = end - lane;
    unsigned long long w = kScanAll;
    if (j >= 0) {
      w = ld_published(words + j);
      for (int polls = 1; (w >> 62) == 0; ++polls) {
        if (polls == kScanPolls) {
          *reinterpret_cast<volatile int32_t*>(error) = 1;
          __threadfence_system();   // before any answer
          w = kScanAll;
          break;
        }
        w = ld_published(words + j);
      }
    }
    const unsigned all = __ballot_sync(0xffffffffu, (w >> 62) == 2);
    const int first = all ? __ffs(all) - 1 : 32;
    unsigned long long v = lane <= first ? (w & kScanValue) : 0ull;
#pragma unroll
    for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    before += v;
    if (all) return (long long)before;
  }
}

// Publishes the tile's sum and returns the sum of the tiles before it; called
// by one warp.
__device__ __forceinline__ long long publish_and_look_back(unsigned long long* words, int64_t t, int64_t tiles,
                                                           long long sum, int32_t* error) {
  const int lane = threadIdx.x & 31;
  if (lane == 0 && tiles > 1) st_published(words + t, (t == 0 ? kScanAll : kScanOwn) | (unsigned long long)sum);
  if (t == 0) return 0;
  const long long before = scan_lookback(words, t, error);
  if (lane == 0) st_published(words + t, kScanAll | (unsigned long long)(before + sum));
  return before;
}

// The last block to get here zeroes the launch's words and counters; every
// thread of every block calls it once its block's look-backs are over.
__device__ __forceinline__ void leave_zeroed(unsigned long long* words, int64_t count, unsigned int* counters) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(counters + 1, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  for (int64_t i = threadIdx.x; i < count; i += blockDim.x) words[i] = 0;
  if (threadIdx.x < 2) counters[threadIdx.x] = 0;
}

// Exclusive prefix sums of K nonnegative per-item values at once.
// in(i, v) fills v[K]; out(i, before, v) gets the sums before item i;
// total(sums) is called once.  in and out may work on the same array: a thread
// reads its items before it writes them, and no other thread touches them.
template <class T, int K, class In, class Out, class Total>
__global__ void __launch_bounds__(kThreads)
scan_tiles(int64_t n, int64_t tiles, In in, Out out, Total total, unsigned long long* words, unsigned int* counters,
           int32_t* error) {
  after_previous_kernel();
  __shared__ T warp_sums[K][kThreads / 32];
  __shared__ long long tile_before[K];
  __shared__ unsigned int ticket;
  if (threadIdx.x == 0) ticket = tiles > 1 ? atomicAdd(counters, 1u) : 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t = ticket;
  const int64_t base = t * kScanTile + int64_t(threadIdx.x) * kScanItems;
  T v[kScanItems][K], local[K];
#pragma unroll
  for (int c = 0; c < K; ++c) local[c] = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
#pragma unroll
    for (int c = 0; c < K; ++c) v[k][c] = 0;
    if (base + k < n) in(base + k, v[k]);
#pragma unroll
    for (int c = 0; c < K; ++c) local[c] += v[k][c];
  }
  T incl[K];
#pragma unroll
  for (int c = 0; c < K; ++c) {
    incl[c] = local[c];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const T peer = __shfl_up_sync(0xffffffffu, incl[c], off);
      if (lane >= off) incl[c] += peer;
    }
    if (lane == 31) warp_sums[c][warp] = incl[c];
  }
  __syncthreads();
  if (warp < K) {
    T sum = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) sum += warp_sums[warp][w];
    const long long before = publish_and_look_back(words + int64_t(warp) * tiles, t, tiles, (long long)sum, error);
    if (lane == 0) tile_before[warp] = before;
  }
  __syncthreads();
  T run[K];
#pragma unroll
  for (int c = 0; c < K; ++c) {
    T before = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) before += w < warp ? warp_sums[c][w] : T(0);
    run[c] = T(tile_before[c]) + before + incl[c] - local[c];
  }
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k < n) out(base + k, run, v[k]);
#pragma unroll
    for (int c = 0; c < K; ++c) run[c] += v[k][c];
  }
  if (t == tiles - 1 && threadIdx.x == kThreads - 1) total(run);
  if (tiles > 1) leave_zeroed(words, tiles * K, counters);
}

template <class T, int K, class In, class Out, class Total>
void scan_items(int64_t n, In in, Out out, Total total, cudaStream_t s) {
  const int64_t tiles = n > 0 ? (n + kScanTile - 1) / kScanTile : 1;   // no items: the total alone
  LookbackSpace w(size_t(tiles) * K, s);
  GPP_LAUNCH((scan_tiles<T, K, In, Out, Total>), int(tiles), kThreads, 0, s, n, tiles, in, out, total, w.words,
             w.counters, ctx().host_error);
}

// Selection in order: pred(i) says whether item i is taken (called once per
// item), emit(i, rank, taken) gets its rank among the taken ones (for an item
// not taken: the number taken before it); the number taken goes to *count or,
// in the waiting form, to the host.
// A warp reads 32 consecutive items at a time, and ranks come from ballots.
template <class Pred, class Emit>
__global__ void __launch_bounds__(kThreads)
select_tiles(int64_t n, int64_t tiles, Pred pred, Emit emit, int32_t* count, Mailbox* mail, uint32_t seq,
             unsigned long long* words, unsigned int* counters, int32_t* error) {
  after_previous_kernel();
  __shared__ int warp_sums[kThreads / 32];
  __shared__ long long tile_before;
  __shared__ unsigned int ticket;
  if (threadIdx.x == 0) ticket = tiles > 1 ? atomicAdd(counters, 1u) : 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t t = ticket;
  const int64_t base = t * kScanTile + warp * 32 * kScanItems + lane;
  unsigned taken[kScanItems];
  int sum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + k * 32;
    const bool take = i < n && pred(i);
    taken[k] = __ballot_sync(0xffffffffu, take);
    sum += __popc(taken[k]);
  }
  if (lane == 0) warp_sums[warp] = sum;
  __syncthreads();
  if (warp == 0) {
    int all = 0;
#pragma unroll
    for (int w = 0; w < kThreads / 32; ++w) all += warp_sums[w];
    const long long before = publish_and_look_back(words, t, tiles, all, error);
    if (lane == 0) {
      tile_before = before;
      if (t == tiles - 1) {
        if (count) *count = int32_t(before + all);
        if (mail) post_values(mail, seq, before + all);
      }
    }
  }
  __syncthreads();
  int rank = int(tile_before);
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) rank += w < warp ? warp_sums[w] : 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int64_t i = base + k * 32;
    if (i < n) emit(i, rank + __popc(taken[k] & ((1u << lane) - 1u)), (taken[k] >> lane & 1u) != 0);
    rank += __popc(taken[k]);
  }
  if (tiles > 1) leave_zeroed(words, tiles, counters);
}

template <class Pred, class Emit>
void select_items(int64_t n, Pred pred, Emit emit, int32_t* count, cudaStream_t s) {
  const int64_t tiles = n > 0 ? (n + kScanTile - 1) / kScanTile : 1;   // no items: a count of 0
  LookbackSpace w(size_t(tiles), s);
  GPP_LAUNCH((select_tiles<Pred, Emit>), int(tiles), kThreads, 0, s, n, tiles, pred, emit, count, nullptr, 0u, w.words,
             w.counters, ctx().host_error);
}

// The same, the number taken being posted to `mail`.
template <class Pred, class Emit>
void select_and_post(int64_t n, Pred pred, Emit emit, Mailbox* mail, uint32_t seq, cudaStream_t s) {
  const int64_t tiles = n > 0 ? (n + kScanTile - 1) / kScanTile : 1;
  LookbackSpace w(size_t(tiles), s);
  GPP_LAUNCH((select_tiles<Pred, Emit>), int(tiles), kThreads, 0, s, n, tiles, pred, emit, nullptr, mail, seq, w.words,
             w.counters, ctx().host_error);
}

// The same, waiting for the number taken.
template <class Pred, class Emit>
int32_t select_and_count(int64_t n, Pred pred, Emit emit, cudaStream_t s, const char* where = __builtin_FUNCTION()) {
  if (n <= 0) return 0;
  auto& c = ctx();
  const uint32_t seq = c.open_mail();
  select_and_post(n, pred, emit, c.box(seq), seq, s);
  return int32_t(c.await(c.box(seq), seq, where)[0]);
}

}  // namespace gpp
