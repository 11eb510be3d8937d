// Node accounting of one interaction on the host build of the device runtime
// -- TESTS ONLY.  An interaction consumes up to four nodes, both wires of each,
// and any of the wires' CASes may lose (the wire's other end was taken: it
// holds LOCK); the redirect left behind is freed by another lane, either at
// once or after the interaction.  Every node must be reclaimed exactly once.
#include "emu.cpp"

namespace {
struct Lane {
  std::unique_ptr<WarpSmem> W = new_warp();
  Ctx c{W.get(), 0, 0};
};
}  // namespace

// For every pair of outcomes (bit 2 * node + word: that wire's CAS loses) of
// two interactions in a row on one lane and the same `nodes` nodes.  `order`
// 0: a node's two wires after each other, 1: all first wires, then all second
// ones.  `chase` 1: a redirect is freed right after it was left.  Returns how
// often a node was lost, plus how often one was reclaimed twice.
extern "C" unsigned long long hvm64emu_pairs(unsigned nodes, int order, int chase) {
  constexpr ull HEAP = 1 << 20;
  Emu E;
  std::vector<std::atomic<unsigned>> out(HEAP / 16);
  g_node_out = out.data();
  g_alloc_faults = 0;
  E.heap.assign(HEAP / 8, 0);
  E.nets.assign(1, NetState{});
  E.C.bump = 1;
  E.C.heap_nodes = HEAP / 16;
  E.C.heap_bytes = HEAP;
  E.C.chunk_nodes = 32;
  E.C.reuse_mark = HEAP;  // (never: free nodes stay with their lane)
  E.C.spin_limit = 1 << 20;
  E.P.heap = E.heap.data();
  E.P.heap_bytes = HEAP;
  E.P.ctrl = &E.C;
  E.P.nets = E.nets.data();
  E.P.nnets = 1;
  E.P.ovf_flush = OVF_FLUSH;
  g_P = E.P;
  g_emu = &E;
  Lane me, other;
  unsigned long long lost = 0;
  auto word = [&](unsigned base, unsigned w) { return 16ull * (base + w / 2) + 8 * (w & 1); };
  const unsigned words = 2 * nodes, consumed = 100, ends = 200, targets = 300;
  for (unsigned first = 0; first < (1u << words); first++)
    for (unsigned second = 0; second < (1u << words); second++)
      for (unsigned lose : {first, second}) {
        for (unsigned w = 0; w < words; w++) {
          const bool l = (lose >> w) & 1;
          E.heap[word(consumed, w) / 8] = pvar(word(ends, w));
          E.heap[word(ends, w) / 8] = l ? P_LOCK : pvar(word(consumed, w));
          E.heap[word(targets, w) / 8] = P_LOCK;
          if (!(w & 1)) check_handed_out(word(consumed, w));
        }
        Exec x;
        for (unsigned k = 0; k < words; k++) {
          const unsigned w = order ? 2 * (k % nodes) + k / nodes : k;
          ull R[2] = {word(consumed, w), pvar(word(targets, w))};
          exec_ins<1>(me.c, x, DevInstr{I_LINK, 0, 0, 0, 1, 0, uint8_t(w & 1 ? INS_A_LAST : 0), 0}, R);
          if (chase && ((lose >> w) & 1)) {
            half_free(other.c, word(consumed, w));
            settle(other.c);
          }
        }
        settle(me.c);
        if (!chase)
          for (unsigned w = 0; w < words; w++)
            if ((lose >> w) & 1) {
              half_free(other.c, word(consumed, w));
              settle(other.c);
            }
        for (unsigned k = 0; k < nodes; k++) lost += out[consumed + k].exchange(0) & 1u;
        for (Lane* l : {&me, &other}) l->W->freed_n = 0;  // (this test hands the same nodes out again)
      }
  return E.C.error ? ~0ull : lost + g_alloc_faults.load();
}
