// The redex queue's tickets over many runs of one ring -- TESTS ONLY.
#include "emu.cpp"

// `runs` runs with capacities and uses in turn; the largest sequence word a
// run can have left is its last ticket plus its capacity.  Returns the first
// run whose tickets do not start on a multiple of its capacity above all words
// earlier runs left, or whose own would wrap, or 0.
extern "C" unsigned long long hvm64emu_tickets(unsigned long long runs) {
  Ctrl c{};
  uint64_t next = 0;
  ull word = 0;
  for (ull r = 1; r <= runs; r++) {
    const unsigned qlog2 = unsigned(4 + r % 21);
    queue_begin(c, qlog2, 1776, next);
    if (c.q_mask != (1ull << qlog2) - 1 || (c.q_base & c.q_mask) || c.q_base <= word || c.q_head != c.q_base ||
        c.q_tail != c.q_base || c.q_base + (1ull << 36) < c.q_base)
      return r;
    c.q_tail += r % 5 ? r % 977 : 1u << 21;  // pushed; some warps left waiting
    c.q_head = c.q_tail + (r % 3 ? 1776 : 0);
    word = c.q_tail + c.q_mask + 1;
    if (r % 1024) queue_end(c, next);  // (else: a run whose control block could not be read)
  }
  return 0;
}
