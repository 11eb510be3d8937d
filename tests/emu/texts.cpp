// Formatting gathered normal forms on a thread with a small stack -- TESTS ONLY.
#include <pthread.h>

#include <cstring>
#include <utility>
#include <vector>

#include "host.hpp"

using namespace hvm;

namespace {
struct Args {
  int shape;
  unsigned size;
  std::string text;
};
// A right-nested list (shape 0) or an even tree (1) of `size` nodes, as a
// gather gives it: the words in readback's order.
void* format(void* p) {
  Args& a = *static_cast<Args*>(p);
  std::vector<uint64_t> pairs;
  const uint64_t root = 16 * (a.size + 1ull);
  auto child = [&](uint64_t k) { return k <= a.size ? port_new(T_CTR, 0, 16 * k) : port_new(T_NUM, 0, 0); };
  std::vector<std::pair<uint64_t, uint64_t>> todo = {{root, child(1)}};  // address, word
  while (!todo.empty()) {
    auto [addr, word] = todo.back();
    todo.pop_back();
    pairs.push_back(addr);
    pairs.push_back(word);
    if ((word & 7) != T_CTR) continue;
    const uint64_t k = (word & ADDR_MASK) / 16;
    todo.push_back({16 * k + 8, a.shape ? child(2 * k + 1) : child(k + 1)});
    todo.push_back({16 * k, a.shape ? child(2 * k) : port_new(T_NUM, 0, 0)});
  }
  Book book;
  const uint64_t offset = 0;
  const unsigned count = unsigned(pairs.size() / 2);
  auto out = readback_pairs_many(book, pairs.data(), &offset, &count, &root, 1, 2 * (a.size + 2ull), 4);
  a.text = out[0].ok ? out[0].text : "error: " + out[0].error;
  return nullptr;
}
}  // namespace

// Formats on a thread with `stack` bytes of stack; returns the text's length.
extern "C" size_t hvm64emu_text(int shape, unsigned size, size_t stack, char* buf, size_t cap) {
  Args a{shape, size, {}};
  pthread_attr_t attr;
  pthread_attr_init(&attr);
  if (pthread_attr_setstacksize(&attr, stack)) return 0;
  pthread_t th;
  if (pthread_create(&th, &attr, format, &a)) return 0;
  pthread_join(th, nullptr);
  pthread_attr_destroy(&attr);
  strncpy(buf, a.text.c_str(), cap - 1);
  return a.text.size();
}
