// Stable LSD radix sort of (uint64 key, int32 value) pairs.
//
// Replaces the reference's thrust::sort of (hash, id) tuples
// (rule_parallel_rows.cu:742-770, rule_parallel_columns.cu:958-975): with the
// input in ascending id order, a stable sort by key yields (key, id) order.
//
// The caller names the key bits that can differ; every window of eight such
// bits is one pass.  Inputs of at most kBlockSortMax pairs are sorted by one
// block in shared memory; larger ones take one histogram launch for all
// passes and one launch per pass, which reads and writes every pair once: a
// tile ranks its keys, publishes its digit counts and finds its output
// offsets by a decoupled look-back over its predecessors.  A digit that turns
// out constant makes its pass return at once (decided on the device, so the
// sort waits for nothing unless it is told to).
#include "sort.hpp"

#include <atomic>
#include <mutex>
#include <vector>

namespace gpp {

namespace {

constexpr int kDigits = 256;
// Windows are eight bits wide, of a 64-bit key; they start at their lowest varying bit, but
// at bit 56 at most, where the last may cover bits of the one before it (harmless, as a
// pass is stable).
constexpr int kMaxPasses = 8;

struct SortPasses {
  int count = 0;
  int shift[kMaxPasses] = {};
};
SortPasses passes_of(uint64_t varying) {
  SortPasses p;
  while (varying) {
    const int shift = std::min(56, __builtin_ctzll(varying));
    p.shift[p.count++] = shift;
    varying &= ~(0xffull << shift);
  }
  return p;
}

__device__ __forceinline__ int digit_of(uint64_t key, int shift) { return int((key >> shift) & 0xff); }

// Exclusive scan over the first 256 threads of a block, one digit each; all
// threads of the block must call it.  `warp_sums` holds 8 ints.
__device__ __forceinline__ int scan_digits(int v, int* warp_sums) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const int peer = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += peer;
  }
  if (warp < 8 && lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  int before = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) before += w < warp ? warp_sums[w] : 0;
  __syncthreads();
  return before + incl - v;
}

// Rank of a warp's key among the warp's earlier keys of the same digit:
// `counts` is the warp's own row of 256 running counts, so no other warp is
// waited for.  `d` is 256 for a position past the end.  The lanes of one digit
// come from nine ballots: __match_any_sync took 389 us where they take 299 (a
// sort of 2,000,003 random pairs), and 1,051 against 878 (8 million).
__device__ __forceinline__ int warp_rank(int* counts, int d) {
  const int lane = threadIdx.x & 31;
  unsigned peers = 0xffffffffu;
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const bool bit = (d >> b) & 1;
    const unsigned m = __ballot_sync(0xffffffffu, bit);
    peers &= bit ? m : ~m;
  }
  const int leader = __ffs(peers) - 1;
  int before = 0;
  if (lane == leader && d < kDigits) {
    before = counts[d];
    counts[d] = before + __popc(peers);
  }
  __syncwarp();
  before = __shfl_sync(0xffffffffu, before, leader);
  return before + __popc(peers & ((1u << lane) - 1u));
}

// ---- one block --------------------------------------------------------------
//
// Most sorts of a presolve round are small (the winners of one rule, the
// hashes of the rows that may be shared).  One block holds the keys in shared
// memory and moves 16-bit positions through the passes, so a pass is a rank,
// two barriers and a scatter in shared memory.  Only the windows that vary are
// sorted by.  Against the bitonic network over (key, position) this replaced
// (78 barriered rounds at 4,096 pairs, 34 us on average over a presolve's
// sorts) it takes 8-12 us for the two to four windows those sorts have.
//
// Few pairs are ranked by comparing each with all, a thread to a pair: 8 to 10 us for up
// to 100 pairs, 13 for 256 and 18 for 384, where the passes take 8.4 us and 1.65 for each
// window that varies, whatever the number of pairs (the bitonic network: 8 to 18 us for
// 2 to 256 pairs).
constexpr int kCountSort = 48;   // pairs for each byte that varies
constexpr int kBlockSortMax = 8192;
constexpr int kBlockSortThreads = 1024;
constexpr int kBlockSortWarps = kBlockSortThreads / 32;
constexpr int kBlockSortItems = kBlockSortMax / kBlockSortThreads;
constexpr size_t kBlockSortCounts = sizeof(int) * kBlockSortWarps * kDigits;

// Bytes that vary: about the passes.
__host__ __device__ __forceinline__ int varying_bytes(uint64_t varying) {
  int count = 0;
#pragma unroll
  for (int k = 0; k < 64; k += 8) count += (varying >> k & 0xff) != 0;
  return count;
}
static_assert(kCountSort * 8 <= kBlockSortThreads, "a thread for each pair");

size_t block_sort_smem(int n) {
  const size_t padded = size_t(n + 7) / 8 * 8;
  return kBlockSortCounts + padded * (sizeof(uint64_t) + 2 * sizeof(uint16_t));
}

template <bool kMayCount>
__global__ void __launch_bounds__(kBlockSortThreads)
block_sort_pairs(uint64_t* keys, int32_t* vals, int n, uint64_t may_vary) {
  after_previous_kernel();
  extern __shared__ __align__(16) unsigned char block_sort_mem[];
  __shared__ int digit_start[kDigits];
  __shared__ int warp_sums[8];
  __shared__ unsigned long long varies;
  const int padded = (n + 7) / 8 * 8;
  int* counts = reinterpret_cast<int*>(block_sort_mem);
  auto* k = reinterpret_cast<uint64_t*>(block_sort_mem + kBlockSortCounts);
  auto* from = reinterpret_cast<uint16_t*>(k + padded);
  auto* to = from + padded;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int items = (n + kBlockSortThreads - 1) / kBlockSortThreads;
  if (threadIdx.x == 0) varies = 0;
  __syncthreads();
  const uint64_t first = keys[0];
  uint64_t acc = 0;
  for (int i = threadIdx.x; i < n; i += kBlockSortThreads) {
    const uint64_t key = keys[i];
    k[i] = key;
    from[i] = uint16_t(i);
    acc |= key ^ first;
  }
  const uint32_t lo = __reduce_or_sync(0xffffffffu, uint32_t(acc));
  const uint32_t hi = __reduce_or_sync(0xffffffffu, uint32_t(acc >> 32));
  if (lane == 0 && (lo | hi)) atomicOr(&varies, (uint64_t(hi) << 32) | lo);
  __syncthreads();
  uint64_t left = varies & may_vary;
  if (kMayCount && n <= kCountSort * varying_bytes(left)) {
    const int i = threadIdx.x;
    if (i < n) {
      const uint64_t mine = k[i] & may_vary;
      int rank = 0;
#pragma unroll 8
      for (int j = 0; j < n; ++j) {
        const uint64_t other = k[j] & may_vary;
        rank += other < mine || (other == mine && j < i) ? 1 : 0;
      }
      to[rank] = uint16_t(i);
    }
    __syncthreads();
    auto* t = from;
    from = to;
    to = t;
    left = 0;
  }
  int* own = counts + warp * kDigits;
  const int base = warp * 32 * items + lane;   // a warp owns consecutive positions
  while (left) {
    const int shift = min(56, __ffsll((long long)left) - 1);
    left &= ~(0xffull << shift);
    for (int d = lane; d < kDigits; d += 32) own[d] = 0;
    __syncwarp();
    int rank[kBlockSortItems], at[kBlockSortItems];
#pragma unroll
    for (int q = 0; q < kBlockSortItems; ++q) {
      if (q >= items) break;
      const int i = base + q * 32;
      at[q] = i < n ? from[i] : 0;
      rank[q] = warp_rank(own, i < n ? digit_of(k[at[q]], shift) : kDigits);
    }
    __syncthreads();
    // Digit d's count per warp becomes its start within the digit.
    int total = 0;
    if (threadIdx.x < kDigits)
      for (int w = 0; w < kBlockSortWarps; ++w) {
        const int c = counts[w * kDigits + threadIdx.x];
        counts[w * kDigits + threadIdx.x] = total;
        total += c;
      }
    const int start = scan_digits(total, warp_sums);
    if (threadIdx.x < kDigits) digit_start[threadIdx.x] = start;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kBlockSortItems; ++q) {
      if (q >= items) break;
      if (base + q * 32 >= n) continue;
      const int d = digit_of(k[at[q]], shift);
      to[digit_start[d] + own[d] + rank[q]] = uint16_t(at[q]);
    }
    __syncthreads();
    auto* t = from;
    from = to;
    to = t;
  }
  int32_t v[kBlockSortItems];
#pragma unroll
  for (int q = 0; q < kBlockSortItems; ++q) {
    const int i = q * kBlockSortThreads + int(threadIdx.x);
    v[q] = i < n ? vals[from[i]] : 0;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kBlockSortItems; ++q) {
    const int i = q * kBlockSortThreads + int(threadIdx.x);
    if (i < n) {
      keys[i] = k[from[i]];
      vals[i] = v[q];
    }
  }
}

// ---- tiles ------------------------------------------------------------------

// What the histogram launch leaves for the passes: per pass the digit counts,
// then (written by its last block) the digits' first output positions, whether
// the digit is constant, and which buffer holds the pairs before the pass.
struct SortPlan {
  unsigned long long counts[kMaxPasses][kDigits];
  long long start[kMaxPasses][kDigits];
  int constant[kMaxPasses];
  int source[kMaxPasses + 1];   // 0 the caller's arrays, 1 the scratch copy; the last entry after all passes
  unsigned int tickets[kMaxPasses];
  unsigned int blocks_done;
  int failed;   // a look-back's wait ran out
};

// Digit counts of all passes.  Bound by the eight shared-memory atomics of a key, and
// before that, with one key of a thread in flight and every shared digit added by itself,
// by the load's latency and the conflicts on one counter: 154 us for 8 million random
// keys, 66 now; 8 million equal ones 154 and 33.
constexpr int kHistogramKeys = 4;   // a thread's keys in flight
__global__ void __launch_bounds__(kThreads)
sort_histogram(const uint64_t* __restrict__ keys, int64_t n, SortPasses passes, SortPlan* plan, Mailbox* mail,
               uint32_t seq) {
  after_previous_kernel();
  __shared__ int h[kMaxPasses][kDigits];
  __shared__ bool last;
  __shared__ int warp_sums[8];
  for (int p = 0; p < passes.count; ++p) h[p][threadIdx.x] = 0;
  __syncthreads();
  // A digit that all lanes share (high digits of small keys) is counted for the warp, as
  // long as it stays the same, and added when it changes; so is a whole key.
  uint64_t run_key = 0;
  int run_keys = 0;
  int run_digit[kMaxPasses], run_count[kMaxPasses];
#pragma unroll
  for (int p = 0; p < kMaxPasses; ++p) run_digit[p] = run_count[p] = 0;
  const int lane = threadIdx.x & 31;
  const auto add_run = [&] {
    if (run_keys && lane < passes.count) atomicAdd(&h[lane][digit_of(run_key, passes.shift[lane])], run_keys);
  };
  const int64_t stride = int64_t(gridDim.x) * kThreads * kHistogramKeys;
  for (int64_t base = (int64_t(blockIdx.x) * kThreads + threadIdx.x - lane) * kHistogramKeys; base < n; base += stride) {
    uint64_t key[kHistogramKeys];
#pragma unroll
    for (int q = 0; q < kHistogramKeys; ++q) {
      const int64_t i = base + q * 32 + lane;
      key[q] = i < n ? keys[i] : 0;
    }
#pragma unroll
    for (int q = 0; q < kHistogramKeys; ++q) {
      const int64_t first = base + q * 32;
      if (first >= n) break;   // warp-uniform
      const bool in = first + lane < n;
      const uint64_t lead = __shfl_sync(0xffffffffu, key[q], 0);
      const uint64_t diff = in ? key[q] ^ lead : ~0ull;
      const uint64_t varies = (uint64_t(__reduce_or_sync(0xffffffffu, uint32_t(diff >> 32))) << 32) |
                              __reduce_or_sync(0xffffffffu, uint32_t(diff));
      if (varies == 0) {
        if (lead == run_key) {
          run_keys += 32;
          continue;
        }
        add_run();
        run_key = lead;
        run_keys = 32;
        continue;
      }
#pragma unroll
      for (int p = 0; p < kMaxPasses; ++p) {
        if (p >= passes.count) break;
        const int d = digit_of(key[q], passes.shift[p]);
        if (digit_of(varies, passes.shift[p]) == 0) {
          if (d != run_digit[p]) {
            if (lane == 0 && run_count[p]) atomicAdd(&h[p][run_digit[p]], run_count[p]);
            run_digit[p] = d;
            run_count[p] = 0;
          }
          run_count[p] += 32;
        } else if (in) {
          atomicAdd(&h[p][d], 1);
        }
      }
    }
  }
  add_run();
#pragma unroll
  for (int p = 0; p < kMaxPasses; ++p)
    if (lane == 0 && run_count[p]) atomicAdd(&h[p][run_digit[p]], run_count[p]);
  __syncthreads();
  for (int p = 0; p < passes.count; ++p) {
    const int c = h[p][threadIdx.x];
    if (c) atomicAdd(&plan->counts[p][threadIdx.x], (unsigned long long)c);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&plan->blocks_done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  int source = 0;
  uint32_t constants = 0;
  for (int p = 0; p < passes.count; ++p) {
    const unsigned long long c = __ldcg(&plan->counts[p][threadIdx.x]);
    // 64-bit scan of the counts as two halves split at bit 22 (256 low halves stay below
    // 2^30, the high ones' sum is at most n / 2^22).
    const int low = scan_digits(int(c & 0x3fffff), warp_sums), high = scan_digits(int(c >> 22), warp_sums);
    plan->start[p][threadIdx.x] = (long long)low + ((long long)high << 22);
    const int constant = __syncthreads_or(c == (unsigned long long)n);
    if (threadIdx.x == 0) {
      plan->constant[p] = constant;
      plan->source[p] = source;
    }
    if (constant) constants |= 1u << p;
    else source ^= 1;
  }
  if (threadIdx.x == 0) {
    plan->source[passes.count] = source;
    if (mail) post_values(mail, seq, constants);
  }
}

// A tile's published word per digit: two flag bits (0 nothing yet, 1 the
// tile's own count, 2 the count of all tiles up to it) over the count.
template <class Word>
struct TileWord {
  static constexpr int kShift = sizeof(Word) * 8 - 2;
  static constexpr Word kValue = (Word(1) << kShift) - 1;
  static constexpr Word kOwn = Word(1) << kShift, kAll = Word(2) << kShift;
};
__device__ __forceinline__ uint32_t ld_word(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_word(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_word(uint32_t* p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_word(unsigned long long* p, unsigned long long v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// One pass over one tile.  Tiles are taken in ticket order, so every tile that
// a look-back waits for is running; a wait still gives up after `max_polls` polls
// and sets the error word that the host checks at its next wait.  The tile goes on
// with a count that is too small: its pairs stay within their digits' ranges, but
// some positions of the pass are then never written.  The later passes, whose digit
// counts would no longer hold, are marked constant and so do not run (a flag of its
// own, looked at as each pass starts, took 9 us of a sort of 2 million pairs), and
// the last launch gives every pair key and value 0, which the kernels between here
// and the host's check can use as an index.
// Bound by the memory traffic (24 bytes a pair) and the ranking; tiles of
// kItems x 256 pairs: sixteen items keep the look-back short against the
// tile's work on large inputs, eight spread mid-size inputs over the SMs.
// 2,000,003 random pairs: 506 us before (four launches a pass: histogram, two
// of scan, scatter), 294 now; the look-back by one tile a round trip took 10 us more
// (and 129 against 113 for 250,000 pairs).
constexpr int kPolls = 1 << 22;
std::atomic<int> g_max_polls{kPolls};

template <int kItems>
struct SortTile {
  static constexpr int kPairs = kThreads * kItems;
  static constexpr size_t kBytes = size_t(kPairs) * (sizeof(uint64_t) + sizeof(int32_t));
};

constexpr int kAhead = 4;

template <int kItems, class Word>
__global__ void __launch_bounds__(kThreads, kItems == 8 ? 4 : 3)   // as shared memory allows
sort_pass(uint64_t* keys0, int32_t* vals0, uint64_t* keys1, int32_t* vals1, int64_t n, int pass, int shift,
          SortPlan* plan, Word* words, int max_polls, int32_t* error) {
  after_previous_kernel();
  constexpr int kPairs = SortTile<kItems>::kPairs;
  using W = TileWord<Word>;
  extern __shared__ __align__(16) unsigned char sort_tile_mem[];
  __shared__ int counts[8][kDigits];
  __shared__ int local_start[kDigits];
  __shared__ long long out_base[kDigits];
  __shared__ int warp_sums[8];
  __shared__ unsigned int ticket;
  if (plan->constant[pass]) return;
  auto* tile_keys = reinterpret_cast<uint64_t*>(sort_tile_mem);
  auto* tile_vals = reinterpret_cast<int32_t*>(tile_keys + kPairs);
  const bool swapped = plan->source[pass] != 0;
  const uint64_t* in_keys = swapped ? keys1 : keys0;
  const int32_t* in_vals = swapped ? vals1 : vals0;
  uint64_t* out_keys = swapped ? keys0 : keys1;
  int32_t* out_vals = swapped ? vals0 : vals1;
  if (threadIdx.x == 0) ticket = atomicAdd(&plan->tickets[pass], 1u);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int d = lane; d < kDigits; d += 32) counts[warp][d] = 0;
  __syncthreads();
  const int64_t tile = ticket;
  const int64_t first = tile * kPairs;
  const int tile_n = int(min(int64_t(kPairs), n - first));
  uint64_t key[kItems];
  int32_t val[kItems];
  int rank[kItems];
  const int p0 = warp * 32 * kItems + lane;
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int i = p0 + q * 32;
    key[q] = i < tile_n ? in_keys[first + i] : 0;
  }
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    const int i = p0 + q * 32;
    val[q] = i < tile_n ? in_vals[first + i] : 0;
  }
#pragma unroll
  for (int q = 0; q < kItems; ++q)
    rank[q] = warp_rank(counts[warp], p0 + q * 32 < tile_n ? digit_of(key[q], shift) : kDigits);
  __syncthreads();
  int tile_total;
  {
    const int d = threadIdx.x;   // one digit per thread
    int total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int c = counts[w][d];
      counts[w][d] = total;
      total += c;
    }
    Word* own = words + size_t(tile) * kDigits + d;
    st_word(own, (tile == 0 ? W::kAll : W::kOwn) | Word(total));
    local_start[d] = scan_digits(total, warp_sums);
    tile_total = total;
  }
  __syncthreads();
  // The tile's own order first, so that the registers are free and the published
  // counts have arrived when the look-back starts.
#pragma unroll
  for (int q = 0; q < kItems; ++q) {
    if (p0 + q * 32 >= tile_n) continue;
    const int d = digit_of(key[q], shift);
    const int slot = local_start[d] + counts[warp][d] + rank[q];
    tile_keys[slot] = key[q];
    tile_vals[slot] = val[q];
  }
  {
    // One digit per thread goes back kAhead tiles per round trip: tiles that run
    // at the same time publish their own counts at about the same time, and one
    // word at a time kept the last of many tiles waiting.
    const int d = threadIdx.x;
    Word before = 0;
    bool done = tile == 0;
    for (int64_t t = tile - 1; !done; t -= kAhead) {
      Word w[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) w[q] = t >= q ? ld_word(words + size_t(t - q) * kDigits + d) : W::kAll;
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (done) continue;
        for (int polls = 1; (w[q] >> W::kShift) == 0; ++polls) {
          if (polls >= max_polls) {
            plan->failed = 1;
            for (int p = pass + 1; p < kMaxPasses; ++p) plan->constant[p] = 1;
            *reinterpret_cast<volatile int32_t*>(error) = 1;
            __threadfence_system();   // before any answer
            w[q] = W::kAll;
            break;
          }
          w[q] = ld_word(words + size_t(t - q) * kDigits + d);
        }
        before += w[q] & W::kValue;
        done = (w[q] >> W::kShift) == 2;
      }
    }
    if (tile > 0) st_word(words + size_t(tile) * kDigits + d, W::kAll | (before + Word(tile_total)));
    out_base[d] = plan->start[pass][d] + (long long)before - local_start[d];
  }
  __syncthreads();
  for (int q = threadIdx.x; q < tile_n; q += kThreads) {
    const uint64_t k = tile_keys[q];
    const int64_t dst = out_base[digit_of(k, shift)] + q;
    out_keys[dst] = k;
    out_vals[dst] = tile_vals[q];
  }
}

// The pairs back into the caller's arrays when the passes left them in the
// scratch copy; zeros after a failed pass.
__global__ void sort_copy_back(int64_t n, int passes, const SortPlan* __restrict__ plan, uint64_t* __restrict__ keys,
                               int32_t* __restrict__ vals, const uint64_t* __restrict__ from_keys,
                               const int32_t* __restrict__ from_vals) {
  after_previous_kernel();
  const bool failed = plan->failed != 0;
  if (plan->source[passes] == 0 && !failed) return;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    keys[i] = failed ? 0 : from_keys[i];
    vals[i] = failed ? 0 : from_vals[i];
  }
}

// The opt-in shared-memory limits are per-device function attributes: set
// once per device, with that device current.
void allow_shared_memory() {
  static std::mutex mu;
  static std::vector<bool> configured;
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  std::lock_guard<std::mutex> lock(mu);
  if (size_t(dev) >= configured.size()) configured.resize(size_t(dev) + 1, false);
  if (configured[size_t(dev)]) return;
  const auto set = [](auto kernel, size_t bytes) {
    check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)), "sort smem");
  };
  set(block_sort_pairs<false>, block_sort_smem(kBlockSortMax));
  set(block_sort_pairs<true>, block_sort_smem(kCountSort * 8));
  set(sort_pass<8, uint32_t>, SortTile<8>::kBytes);
  set(sort_pass<16, uint32_t>, SortTile<16>::kBytes);
  set(sort_pass<16, unsigned long long>, SortTile<16>::kBytes);
  configured[size_t(dev)] = true;
}

// With `ask` the host learns from the histogram which digits are constant and leaves
// their passes out.  It waits for that behind the first kAskBehind passes, so the device
// has work meanwhile.  A pass that returns at once costs 2 to 5 us: 20,000 equal keys
// took 42 us, 24 so, and 8 million with one byte that varies 292, 201 so with the
// histogram's share of that.
constexpr int kAskBehind = 2;

template <int kItems, class Word>
void sort_tiles(uint64_t* keys, int32_t* vals, int64_t n, const SortPasses& passes, cudaStream_t s, bool ask) {
  const int64_t tiles = (n + SortTile<kItems>::kPairs - 1) / SortTile<kItems>::kPairs;
  const size_t words = size_t(tiles) * kDigits;
  DBuf<uint64_t> k2(size_t(n), s);
  DBuf<int32_t> v2(size_t(n), s);
  DBuf<unsigned char> scratch(sizeof(SortPlan) + sizeof(Word) * words * size_t(passes.count), s);
  scratch.zero();
  auto* plan = reinterpret_cast<SortPlan*>(scratch.p);
  auto* tile_words = reinterpret_cast<Word*>(scratch.p + sizeof(SortPlan));
  auto& c = ctx();
  ask = ask && passes.count > kAskBehind;
  const uint32_t seq = ask ? c.open_mail() : 0;
  Mailbox* const mail = ask ? c.box(seq) : nullptr;
  GPP_LAUNCH_BYTES(sort_histogram, 8.0 * n, grid_stride_blocks((n + kHistogramKeys - 1) / kHistogramKeys, kThreads, 4),
                   kThreads, 0, s, keys, n, passes, plan, mail, seq);
  uint64_t constants = 0;
  for (int p = 0; p < passes.count; ++p) {
    if (ask && p == kAskBehind) {
      c.poll(mail, seq, 4, "constant digits", false);   // an expired wait still needs the last launch
      constants = mail->words[0] & 0xffffffffu;
    }
    if (constants >> p & 1u) continue;
    GPP_LAUNCH_BYTES((sort_pass<kItems, Word>), 24.0 * n, int(tiles), kThreads, SortTile<kItems>::kBytes, s, keys, vals,
                     k2.p, v2.p, n, p, passes.shift[p], plan, tile_words + words * size_t(p),
                     g_max_polls.load(std::memory_order_relaxed), c.host_error);
  }
  if (constants + 1 == uint64_t(1) << passes.count) return;   // nothing moved
  GPP_LAUNCH(sort_copy_back, grid_stride_blocks(n), kThreads, 0, s, n, passes.count, plan, keys, vals, k2.p, v2.p);
}

}  // namespace

void inject_sort_wait_limit(int polls) { g_max_polls.store(polls > 0 ? polls : kPolls); }

void radix_sort_pairs(uint64_t* keys, int32_t* vals, int64_t n, cudaStream_t s, uint64_t may_vary, bool ask) {
  if (n <= 1 || may_vary == 0) return;
  allow_shared_memory();
  if (n <= kBlockSortMax) {
    if (n <= kCountSort * varying_bytes(may_vary))   // few enough for the counting, as far as the host knows
      GPP_LAUNCH(block_sort_pairs<true>, 1, kBlockSortThreads, block_sort_smem(int(n)), s, keys, vals, int(n), may_vary);
    else
      GPP_LAUNCH(block_sort_pairs<false>, 1, kBlockSortThreads, block_sort_smem(int(n)), s, keys, vals, int(n), may_vary);
    return;
  }
  const SortPasses passes = passes_of(may_vary);
  if (n < (int64_t(1) << 20)) sort_tiles<8, uint32_t>(keys, vals, n, passes, s, ask);
  else if (n < (int64_t(1) << 30)) sort_tiles<16, uint32_t>(keys, vals, n, passes, s, ask);
  else sort_tiles<16, unsigned long long>(keys, vals, n, passes, s, ask);   // counts past 30 bits
}

}  // namespace gpp
