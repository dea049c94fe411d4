// Runs the engine's book of device blocks (csrc/block_book.hpp) on made-up
// addresses: argv[1] names the check.
#include <cstdio>
#include <cstring>
#include <thread>

#include "block_book.hpp"

using gpp::BlockBook;

#define CHECK(what)                                                  \
  do {                                                               \
    if (!(what)) {                                                   \
      std::printf("line %d: %s does not hold\n", __LINE__, #what);   \
      return 1;                                                      \
    }                                                                \
  } while (0)

static void* address(int64_t k) { return reinterpret_cast<void*>(k << 20); }

// A block that another context's thread frees, or the caller by gpp_device_free, is
// no longer in its own book when the address comes back from another pool.
static int freed_elsewhere() {
  BlockBook* a = new BlockBook;
  BlockBook* b = new BlockBook;
  const size_t large = BlockBook::size_class(1 << 20), small = BlockBook::size_class(300);
  a->lend(address(1), large);
  size_t known = 1;
  std::thread([&] {
    known = b->give_back(address(1));
    BlockBook::forget(address(1));
  }).join();
  CHECK(known == 0);
  b->lend(address(1), small);                  // the other pool hands the address out
  CHECK(a->give_back(address(1)) == 0);        // and the first context frees the block
  BlockBook::forget(address(1));
  CHECK(b->give_back(address(1)) == 0);
  a->lend(address(2), large);                  // the ordinary way round
  CHECK(a->give_back(address(2)) == large);
  CHECK(a->hold(address(2), large) && a->held() == int64_t(large));
  CHECK(a->take(small) == nullptr && a->take(large) == address(2) && a->held() == 0);
  CHECK(a->give_back(address(2)) == large);
  BlockBook::forget(address(3));               // memory of no book
  return 0;
}

// What one context held does not stay taken from the others once its blocks are in
// use again, and all together hold no more than the cap.
static int credit_returns() {
  BlockBook* a = new BlockBook;
  BlockBook* b = new BlockBook;
  const size_t cls = BlockBook::size_class(size_t(64) << 20);
  const int64_t most = BlockBook::kCap / int64_t(cls);
  for (int64_t k = 1; k <= most; ++k) CHECK(a->hold(address(k), cls));
  CHECK(!a->hold(address(most + 1), cls) && !b->hold(address(most + 1), cls));
  for (int64_t k = 1; k <= most; ++k) CHECK(a->take(cls) != nullptr);
  CHECK(a->held() == 0 && a->credit() <= 2 * BlockBook::kCreditStep);
  int64_t held = 0;
  while (b->hold(address(1000 + held), cls)) ++held;
  CHECK(held >= most - 2 && held <= most);
  CHECK(b->held() + a->credit() <= BlockBook::kCap && b->credit() >= b->held());
  // Small blocks that come and go within a step return nothing.
  const size_t small = BlockBook::size_class(4096);
  CHECK(a->hold(address(5), small));
  const int64_t credit = a->credit();
  CHECK(a->take(small) == address(5) && a->credit() == credit && a->hold(address(5), small) && a->credit() == credit);
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "freed_elsewhere")) return freed_elsewhere();
  if (argc == 2 && !std::strcmp(argv[1], "credit_returns")) return credit_returns();
  std::printf("unknown check\n");
  return 2;
}
