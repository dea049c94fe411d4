// The host-side book of one engine context's device blocks: the blocks it has
// handed out, with their size classes, and the freed ones it holds for reuse.
// Plain C++ (tests/cpp/block_book.cpp runs it without a device).
#pragma once

#include <atomic>
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <thread>
#include <unordered_map>
#include <vector>

namespace gpp {

class BlockBook {
 public:
  static constexpr int64_t kCap = int64_t(8) << 30;          // bytes held by all books
  static constexpr int64_t kCreditStep = int64_t(64) << 20;  // a book draws on the cap, and returns, in these steps

  BlockBook() {
    std::lock_guard<std::mutex> lock(registry().mu);
    registry().books.push_back(this);   // for good: contexts are never destroyed
  }
  BlockBook(const BlockBook&) = delete;
  BlockBook& operator=(const BlockBook&) = delete;

  // At most 25% over the request.
  static size_t size_class(size_t bytes) {
    if (bytes <= 256) return 256;
    const int high = 63 - __builtin_clzll(uint64_t(bytes));
    const size_t grain = size_t(1) << (high - 2 > 8 ? high - 2 : 8);
    return (bytes + grain - 1) / grain * grain;
  }

  // A held block of the class, from now on handed out; null when none is held.
  void* take(size_t cls) {
    auto& list = free_[class_index(cls)];
    if (list.empty()) return nullptr;
    void* p = list.back();
    list.pop_back();
    held_ -= int64_t(cls);
    lend(p, cls);
    return_credit();
    return p;
  }
  // The pool has handed out a block.
  void lend(void* p, size_t cls) {
    Locked lock(busy_);
    lent_[p] = cls;
  }
  // The context frees a block: its class, or 0 for a block that this book did
  // not hand out.
  size_t give_back(void* p) {
    Locked lock(busy_);
    const auto it = lent_.find(p);
    if (it == lent_.end()) return 0;
    const size_t cls = it->second;
    lent_.erase(it);
    return cls;
  }
  // Holds a block that came back; false when the cap leaves no room for it.
  bool hold(void* p, size_t cls) {
    if (!may_hold(int64_t(cls))) return false;
    held_ += int64_t(cls);
    free_[class_index(cls)].push_back(p);
    return true;
  }
  // A block that goes back to a pool without its own book: out of every book, so
  // that no later block at the address is taken for it.  Before the pool gets it.
  static void forget(void* p) {
    std::lock_guard<std::mutex> lock(registry().mu);
    for (BlockBook* b : registry().books)
      if (b->give_back(p)) return;   // a block is in one book at most
  }

  int64_t held() const { return held_; }
  int64_t credit() const { return credit_; }

 private:
  struct Registry {
    std::mutex mu;
    std::vector<BlockBook*> books;
  };
  static Registry& registry() {
    static Registry* r = new Registry;   // never destroyed
    return *r;
  }
  static std::atomic<int64_t>& drawn() {
    static std::atomic<int64_t> bytes{0};
    return bytes;
  }
  // Index of a size class: its power of two and its quarter.
  static int class_index(size_t cls) {
    const int high = 63 - __builtin_clzll(uint64_t(cls));
    return high * 4 + int((cls >> (high - 2)) & 3);
  }
  bool may_hold(int64_t bytes) {
    const int64_t over = held_ + bytes - credit_;
    if (over <= 0) return true;
    const int64_t draw = (over + kCreditStep - 1) / kCreditStep * kCreditStep;
    if (drawn().fetch_add(draw, std::memory_order_relaxed) + draw > kCap) {
      drawn().fetch_sub(draw, std::memory_order_relaxed);
      return false;
    }
    credit_ += draw;
    return true;
  }

  // Credit past what is held goes back in whole steps, but for one: blocks that
  // come and go within a step draw and return nothing.
  void return_credit() {
    const int64_t spare = (credit_ - held_) / kCreditStep - 1;
    if (spare <= 0) return;
    credit_ -= spare * kCreditStep;
    drawn().fetch_sub(spare * kCreditStep, std::memory_order_relaxed);
  }

  // The record of blocks in use is the one part that other threads reach (forget),
  // for a lookup at a time, so a flag does: 64 LPs presolved one after the other took
  // 165.7 ms with it, 167.9 with a mutex, 165.4 with neither.
  struct Locked {
    std::atomic<bool>& busy;
    explicit Locked(std::atomic<bool>& flag) : busy(flag) {
      while (busy.exchange(true, std::memory_order_acquire)) std::this_thread::yield();
    }
    ~Locked() { busy.store(false, std::memory_order_release); }
  };
  std::atomic<bool> busy_{false};
  std::unordered_map<void*, size_t> lent_;
  static constexpr int kClasses = 256;
  std::vector<void*> free_[kClasses];
  int64_t held_ = 0, credit_ = 0;
};

}  // namespace gpp
