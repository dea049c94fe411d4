// Engine context, status block, scans and the canonical deterministic sum.
#include "scan.cuh"

#include <atomic>
#include <cstdlib>
#include <thread>

#include <algorithm>
#include <chrono>
#include <string>
#include <memory>

namespace gpp {

uint64_t& launch_counter() {
  static thread_local uint64_t count = 0;
  return count;
}
uint64_t& sync_counter() {
  static thread_local uint64_t n = 0;
  return n;
}

Context::Context() {
  check(cudaGetDevice(&device), "cudaGetDevice");
  // Blocking stream: implicitly ordered after work the caller queued on the
  // legacy default stream, as the reference's synchronous API assumes.
  check(cudaStreamCreateWithFlags(&stream, cudaStreamDefault), "cudaStreamCreate");
  // A pool of this context alone: with one pool per host thread, the batched
  // form's workers neither share a pool lock nor get ordered after each other
  // by block reuse across their streams.
  cudaMemPoolProps props{};
  props.allocType = cudaMemAllocationTypePinned;
  props.location.type = cudaMemLocationTypeDevice;
  props.location.id = device;
  check(cudaMemPoolCreate(&pool, &props), "cudaMemPoolCreate");
  uint64_t keep = UINT64_MAX;  // keep freed blocks in the pool between presolve calls
  check(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep), "pool threshold");
  check(cudaMallocHost(reinterpret_cast<void**>(&host_status), sizeof(int32_t) * kStatusWords),
        "cudaMallocHost status");
  check(cudaMallocHost(reinterpret_cast<void**>(&host_scalar), 16), "cudaMallocHost scalar");
  check(cudaMallocHost(reinterpret_cast<void**>(&host_error), sizeof(int32_t)), "cudaMallocHost error");
  *host_error = 0;
  check(cudaMallocHost(reinterpret_cast<void**>(&mail), sizeof(Mailbox) * (kMailBoxes + kNnzBoxes + kLateBoxes + 1)), "cudaMallocHost mail");
  std::memset(static_cast<void*>(mail), 0, sizeof(Mailbox) * (kMailBoxes + kNnzBoxes + kLateBoxes + 1));
  nnz_mail = mail + kMailBoxes;
  late_mail = nnz_mail + kNnzBoxes;
  fixed_mail = late_mail + kLateBoxes;
  check(cudaMalloc(reinterpret_cast<void**>(&report_words), sizeof(int32_t) * 16), "cudaMalloc report");
  check(cudaMemsetAsync(report_words, 0, sizeof(int32_t) * 16, stream), "report words");
}

void Context::sync(const char* label) {
  ++sync_counter();
  if (!profiling()) {
    check(cudaStreamSynchronize(stream), label);
  } else {
    const auto t0 = std::chrono::steady_clock::now();
    check(cudaStreamSynchronize(stream), label);
    profile_sync(label, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
  }
  raise_device_error(label);
}

Report Context::open_report(int count) {
  const uint32_t seq = open_mail();
  return Report{report_words, reinterpret_cast<unsigned int*>(report_words + 15), box(seq), seq, count, false};
}
Report Context::open_report(int count, int32_t* words) {
  const uint32_t seq = open_mail();
  return Report{words, reinterpret_cast<unsigned int*>(report_words + 15), box(seq), seq, count, true};
}

void Context::poll(const Mailbox* box, uint32_t seq, int words, const char* where, bool raise) {
  int k = 0;   // words seen
  auto posted = [&] {
    while (k < words && uint32_t(box->words[k] >> 32) == seq) ++k;
    return k == words;
  };
  if (!posted()) ++sync_counter();
  const auto t0 = profiling() ? std::chrono::steady_clock::now() : std::chrono::steady_clock::time_point();
  for (uint64_t polls = 1; !posted(); ++polls) {
    if (polls % 4096 == 0) {
      const cudaError_t e = cudaStreamQuery(stream);
      if (e == cudaSuccess && !posted()) throw CudaError(std::string(where) + ": the kernel posted no answer");
      if (e != cudaSuccess && e != cudaErrorNotReady) check(e, where);
    }
    if (polls > 4096 && polls % 64 == 0) std::this_thread::yield();
    __builtin_ia32_pause();
  }
  std::atomic_thread_fence(std::memory_order_acquire);
  if (profiling())
    profile_sync(where, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count());
  if (raise) raise_device_error(where);
}

void Context::raise_device_error(const char* where) {
  if (!*static_cast<volatile int32_t*>(host_error)) return;
  *host_error = 0;
  throw CudaError(std::string(where) + ": a block's bounded wait for its predecessors ran out");
}

Context::~Context() {
  if (mail) cudaFreeHost(mail);
  if (report_words) cudaFree(report_words);
  if (host_status) cudaFreeHost(host_status);
  if (host_scalar) cudaFreeHost(host_scalar);
  if (host_error) cudaFreeHost(host_error);
  if (side) cudaStreamDestroy(side);
  if (stream) cudaStreamDestroy(stream);
}

cudaStream_t Context::side_stream() {
  if (!side) check(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking), "cudaStreamCreate side");
  return side;
}

Context& ctx() {
  // One context per host thread and device (the reference's contract is one
  // presolve per host thread on the current device).
  // Never destroyed: the stream and pinned block stay valid until process
  // exit, so buffers released during thread-exit destruction can still be
  // returned to the stream-ordered pool.
  static thread_local std::vector<Context*>* per_device = new std::vector<Context*>();
  int dev = 0;
  check(cudaGetDevice(&dev), "cudaGetDevice");
  if (size_t(dev) >= per_device->size()) per_device->resize(size_t(dev) + 1, nullptr);
  if (!(*per_device)[size_t(dev)]) (*per_device)[size_t(dev)] = new Context();
  return *(*per_device)[size_t(dev)];
}

namespace {
std::atomic<int64_t> g_alloc_countdown{-1};   // < 0: no failure armed
}  // namespace

void inject_alloc_failure(int64_t after) { g_alloc_countdown.store(after < 0 ? -1 : after); }

// Host-side reuse of scratch blocks.  A presolve allocates and frees a few
// thousand scratch buffers, each a cudaMallocFromPoolAsync / cudaFreeAsync
// pair of driver calls on the host's critical path between launches.  Blocks
// are rounded up to a size class (at most 25% over) and a block its own
// context frees on that context's stream goes to the context's book
// (block_book.hpp); the next request of that class on that stream takes it back
// with no driver call.  Reuse is safe without events: everything on one stream
// runs in issue order, so a kernel that gets the block runs after every kernel
// that used it.  A block freed by another thread or on another stream goes back
// to the pool, and out of the book of the context that had handed it out: the
// address may come back from any pool, as a block of another size.
// At most BlockBook::kCap bytes are held this way across all contexts; past that
// a freed block goes back to the pool.  The batched form's threads share nothing
// here but that cap.  GPP_ALLOC_CACHE=0 turns the reuse off.
namespace {
bool alloc_cache_on() {
  static const bool on = [] {
    const char* e = std::getenv("GPP_ALLOC_CACHE");
    return !(e && e[0] == '0');
  }();
  return on;
}
}  // namespace

cudaError_t pool_alloc(void** p, size_t bytes, cudaStream_t s) {
  if (g_alloc_countdown.load(std::memory_order_relaxed) >= 0) {
    int64_t left = g_alloc_countdown.load();
    while (left >= 0 && !g_alloc_countdown.compare_exchange_weak(left, left - 1)) {
    }
    if (left == 0) {
      *p = nullptr;
      return cudaErrorMemoryAllocation;
    }
  }
  Context& c = ctx();
  if (!alloc_cache_on()) return cudaMallocFromPoolAsync(p, bytes, c.pool, s);
  const size_t cls = BlockBook::size_class(bytes);
  if (s == c.stream && (*p = c.blocks.take(cls))) return cudaSuccess;
  const cudaError_t e = cudaMallocFromPoolAsync(p, cls, c.pool, s);
  if (e == cudaSuccess) c.blocks.lend(*p, cls);
  return e;
}

void pool_free(void* p, cudaStream_t s) {
  if (!p) return;
  if (alloc_cache_on()) {
    Context& c = ctx();
    const size_t cls = c.blocks.give_back(p);
    if (cls == 0) BlockBook::forget(p);   // another context's
    else if (s == c.stream && c.blocks.hold(p, cls)) return;
  }
  cudaFreeAsync(p, s);
}

void release_to_driver(void* p, cudaStream_t s) {
  if (alloc_cache_on()) BlockBook::forget(p);
  cudaFreeAsync(p, s);
}

Status::Status() {
  check(pool_alloc(reinterpret_cast<void**>(&d), sizeof(int32_t) * Context::kStatusWords, ctx().stream),
        "status alloc");
}
Status::~Status() { if (d) pool_free(d, ctx().stream); }
void Status::clear(int words) {
  check(cudaMemsetAsync(d, 0, sizeof(int32_t) * size_t(words), ctx().stream), "status clear");
}
const int32_t* Status::read(int words, const char* where) {
  auto& c = ctx();
  check(cudaMemcpyAsync(c.host_status, d, sizeof(int32_t) * size_t(words), cudaMemcpyDeviceToHost, c.stream),
        "status read");
  c.sync(where);
  return c.host_status;
}

LookbackSpace::LookbackSpace(size_t count, cudaStream_t s) {
  auto& c = ctx();
  const size_t need = count + 1;   // the counters take the first word
  unsigned long long* base;
  if (s == c.stream) {
    if (c.lookback_words < need) {
      const size_t grown = std::max({need, 2 * c.lookback_words, size_t(4096)});
      unsigned long long* p = dalloc<unsigned long long>(grown);
      dfree(std::exchange(c.lookback, p));
      c.lookback_words = grown;
      check(cudaMemsetAsync(p, 0, sizeof(unsigned long long) * grown, s), "look-back words");
    }
    base = c.lookback;
  } else {
    own.alloc(need, s);
    own.zero();
    base = own.p;
  }
  counters = reinterpret_cast<unsigned int*>(base);
  words = base + 1;
}

namespace {
// Chunk totals, then (the last block to finish) their sum in chunk order,
// posted to the host.
__global__ void __launch_bounds__(kThreads)
det_sum_kernel(const double* __restrict__ v, const uint8_t* __restrict__ mask, int64_t n, double* chunk_totals,
               unsigned int* done, Mailbox* mail, uint32_t seq) {
  after_previous_kernel();
  __shared__ double sm[kThreads];
  __shared__ bool last;
  const int64_t base = int64_t(blockIdx.x) * 2048;
  double acc = 0.0;
  for (int64_t k = base + threadIdx.x; k < n && k < base + 2048; k += kThreads) acc += mask && !mask[k] ? 0.0 : v[k];
  sm[threadIdx.x] = acc;
  __syncthreads();
  for (int h = kThreads / 2; h > 0; h >>= 1) {
    if (threadIdx.x < unsigned(h)) sm[threadIdx.x] = sm[threadIdx.x] + sm[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    chunk_totals[blockIdx.x] = sm[0];
    __threadfence();
    last = atomicAdd(done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double total = 0.0;
  for (int first = 0; first < int(gridDim.x); first += kThreads) {
    const int c = first + int(threadIdx.x);
    sm[threadIdx.x] = c < int(gridDim.x) ? __ldcg(chunk_totals + c) : 0.0;
    __syncthreads();
    if (threadIdx.x == 0) {   // zeros past the last chunk change nothing
#pragma unroll 16
      for (int k = 0; k < kThreads; ++k) total += sm[k];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *done = 0;
    post_values(mail, seq, __double_as_longlong(total));
  }
}
}  // namespace

void exclusive_scan_i32(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s) {
  scan_items<int32_t, 1>(
      n, [in] __device__(int64_t i, int32_t(&v)[1]) { v[0] = in[i]; },
      [out] __device__(int64_t i, const int32_t(&before)[1], const int32_t(&)[1]) { out[i] = before[0]; },
      [out, n] __device__(const int32_t(&sum)[1]) { out[n] = sum[0]; }, s);
}
int32_t exclusive_scan_total(const int32_t* in, int32_t* out, int64_t n, cudaStream_t s, const char* where) {
  auto& c = ctx();
  const uint32_t seq = c.open_mail();
  Mailbox* mail = c.box(seq);
  scan_items<int32_t, 1>(
      n, [in] __device__(int64_t i, int32_t(&v)[1]) { v[0] = in[i]; },
      [out] __device__(int64_t i, const int32_t(&before)[1], const int32_t(&)[1]) { out[i] = before[0]; },
      [=] __device__(const int32_t(&sum)[1]) {
        out[n] = sum[0];
        post_values(mail, seq, sum[0]);
      },
      s);
  return int32_t(c.await(mail, seq, where)[0]);
}
std::pair<int64_t, int64_t> exclusive_scan_pair_i64(const int64_t* a, int64_t* a_out, const int64_t* b, int64_t* b_out,
                                                    int64_t n, cudaStream_t s, const char* where) {
  auto& c = ctx();
  const uint32_t seq = c.open_mail();
  Mailbox* mail = c.box(seq);
  scan_items<int64_t, 2>(
      n,
      [=] __device__(int64_t i, int64_t(&v)[2]) {
        v[0] = a[i];
        v[1] = b[i];
      },
      [=] __device__(int64_t i, const int64_t(&before)[2], const int64_t(&)[2]) {
        a_out[i] = before[0];
        b_out[i] = before[1];
      },
      [=] __device__(const int64_t(&sum)[2]) {
        a_out[n] = sum[0];
        b_out[n] = sum[1];
        post_values(mail, seq, sum[0], sum[1]);
      },
      s);
  const int64_t* t = c.await(mail, seq, where);
  return {t[0], t[1]};
}

LateValue det_sum_later(const double* v, const uint8_t* mask, int64_t n, cudaStream_t s) {
  if (n <= 0) return LateValue{};
  auto& c = ctx();
  const int64_t chunks = (n + 2047) / 2048;
  DBuf<double> part(size_t(chunks), s);
  if (++c.late_seq == 0) ++c.late_seq;
  const uint32_t seq = c.late_seq;
  const Report r = c.open_report(0);   // its block counter
  GPP_LAUNCH(det_sum_kernel, int(chunks), kThreads, 0, s, v, mask, n, part.p, r.done,
             c.late_mail + seq % Context::kLateBoxes, seq);
  return LateValue{0.0, seq};
}
double LateValue::get() const {
  if (seq == 0) return known;
  auto& c = ctx();
  const int64_t bits = c.await(c.late_mail + seq % Context::kLateBoxes, seq, "det_sum")[0];
  double total;
  std::memcpy(&total, &bits, sizeof(total));
  return total;
}
double det_sum(const double* v, const uint8_t* mask, int64_t n, cudaStream_t s) {
  return det_sum_later(v, mask, n, s).get();
}

namespace {
thread_local std::string g_last_error;

struct ProfileRecord {
  std::string name;
  double bytes;
  cudaEvent_t begin, end;   // null for a host wait, whose host time is host_ms
  double host_ms;
};
struct ProfileState {
  bool on = false;
  std::vector<ProfileRecord> records;
  std::vector<cudaEvent_t> pool;
  size_t next = 0;
};
ProfileState& profile_state() {
  static thread_local ProfileState* p = new ProfileState;  // never destroyed (see ctx())
  return *p;
}
}  // namespace

bool profiling() { return profile_state().on; }
cudaEvent_t profile_event() {
  auto& p = profile_state();
  if (p.next == p.pool.size()) {
    cudaEvent_t e;
    check(cudaEventCreate(&e), "cudaEventCreate");
    p.pool.push_back(e);
  }
  return p.pool[p.next++];
}
void profile_record(const char* name, double bytes, cudaEvent_t begin, cudaEvent_t end) {
  profile_state().records.push_back({name, bytes, begin, end, 0.0});
}
int64_t profile_last() {
  auto& p = profile_state();
  return p.on && !p.records.empty() ? int64_t(p.records.size()) - 1 : -1;
}
void profile_add_bytes(int64_t record, double bytes) {
  auto& p = profile_state();
  if (record >= 0 && size_t(record) < p.records.size()) p.records[size_t(record)].bytes += bytes;
}
void profile_sync(const char* label, double ms) {
  profile_state().records.push_back({std::string("sync: ") + label, 0.0, nullptr, nullptr, ms});
}
void profile_enable(bool on) {
  auto& p = profile_state();
  p.on = on;
  p.records.clear();
  p.next = 0;
}
// Aggregates recorded launches by kernel name: launches, total ms, total bytes.
std::vector<ProfileSummary> profile_summary() {
  auto& p = profile_state();
  check(cudaDeviceSynchronize(), "profile sync");
  std::vector<ProfileSummary> out;
  for (const auto& r : p.records) {
    float ms = float(r.host_ms);
    if (r.begin) check(cudaEventElapsedTime(&ms, r.begin, r.end), "cudaEventElapsedTime");
    ProfileSummary* s = nullptr;
    for (auto& o : out)
      if (o.name == r.name) s = &o;
    if (!s) {
      out.push_back({r.name, 0, 0.0, 0.0});
      s = &out.back();
    }
    s->launches += 1;
    s->ms += ms;
    s->bytes += r.bytes;
  }
  return out;
}
void set_last_error(const std::string& s) { g_last_error = s; }
const char* last_error() { return g_last_error.c_str(); }

}  // namespace gpp
