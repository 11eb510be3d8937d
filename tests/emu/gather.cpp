// gather_walk's limit on the host build of the device runtime -- TESTS ONLY.
#include "emu.cpp"

// Walks a normal form of `size` binary nodes with a limit of `limit` pairs: a
// list nested on the right (shape 0), or a tree as even as `size` allows
// (shape 1).  Returns the pairs walked, negative when the walk stopped early.
extern "C" long long hvm64emu_limited_walk(int shape, unsigned size, unsigned limit) {
  std::vector<ull> heap(2 * (size_t(size) + 2), 0);
  const ull root = 16 * (size + 1ull);
  auto set = [&](ull w, ull v) { heap[w >> 3] = v; };
  auto node = [](unsigned k) { return mkport(T_CTR, 0, 16ull * k); };
  auto child = [&](unsigned k) { return k <= size ? node(k) : mkport(T_NUM, 0, 0); };
  set(root, child(1));
  for (unsigned k = 1; k <= size; k++) {
    set(16ull * k, shape ? child(2 * k) : mkport(T_NUM, 0, 0));
    set(16ull * k + 8, shape ? child(2 * k + 1) : child(k + 1));
  }
  Params P{};
  P.heap = heap.data();
  P.heap_bytes = heap.size() * 8;
  Ctrl C{};
  P.ctrl = &C;
  g_P = P;
  std::vector<ull> stk(256);
  bool deep = false, stopped = false;
  const unsigned n = gather_walk(0, root, nullptr, 0, stk.data(), 256, &deep, limit, &stopped);
  return deep || C.error ? -1000000000ll : stopped ? -(long long)n : (long long)n;
}
