// Device runtime of the B200 interaction-net reducer.
//
// Heap: one HBM arena of 16-byte nodes (two 8-byte port words), addressed by
// byte offset, so a node's other half is `addr ^ 8` exactly as in the
// reference (runtime/src/addr.rs:36-50).  Node 0 is reserved (the free-list
// terminator and a scratch target for guarded accesses).
//
// Every heap access is a strong GPU-scope operation (ld/st.relaxed.gpu or an
// atomic), so no SM reads a stale L1 copy of a word another SM changed.  A
// freshly allocated node is filled with LOCK and fenced before its address
// can escape; readers treat LOCK as "not ready yet" and wait, which is the
// reference's own protocol (runtime/src/wire.rs:67-75).
//
// Every wait is bounded: after `spin_limit` polls, or when another lane has
// already failed, the wait gives up, the run's error word is set and all
// warps drain and exit.  An address is bounds-checked where it is read from the
// heap to be followed (heap_at, a constructor match, a free list's link); one
// outside the arena sets HVM64_ERR_BAD_ADDR and is redirected to node 0.  The
// words of a lane's own nodes and of nodes checked that way are accessed
// without another check, so a protocol fault cannot become a memory fault.
#pragma once
#include <stdint.h>
#include <stddef.h>

#ifndef __CUDACC__
#include <atomic>
#include <chrono>
#include <thread>
#endif

#include "host.hpp"
#include "hvm64.h"
#include "num.h"

namespace hvm {
namespace dev {

typedef unsigned long long ull;

#ifndef HVM_SCAP
#define HVM_SCAP 512
#endif
#ifndef HVM_HEADROOM
#define HVM_HEADROOM 192
#endif
constexpr int WARPS = 2;            // warps per reducer block
constexpr int THREADS = WARPS * 32;
constexpr int SCAP = HVM_SCAP;      // per-warp shared-memory redex stack (power of two)
constexpr int HEADROOM = HVM_HEADROOM;  // stack slots kept free for the redexes of one step
static_assert((SCAP & (SCAP - 1)) == 0 && SCAP >= 64, "SCAP is a power of two, at least 64");
static_assert(HEADROOM >= 0 && SCAP - HEADROOM >= 32, "a step's window needs SCAP - HEADROOM >= 32");
constexpr int CHUNK = 32;           // redexes per global-queue slot
// Per-warp pool of free nodes ready for reuse.  (With 64 a sort of 2^15 keys takes
// 92 ms on the device instead of 87, a batch of 451 nets 296 instead of 267.)
constexpr int POOL = 160;
constexpr int POOL_BUDGETED = 64;   // and where what a warp holds back comes off a budget or a fixed heap
constexpr int FREED_ALONE = 2;      // words an interaction may have freed alone before it looks at their siblings
constexpr int FAILS = 2;            // wires of an interaction, left as redirects, that it remembers
constexpr unsigned ICACHE = 32;     // instructions of the step's Def staged in shared memory
constexpr unsigned SMALL_REGS = 10; // Defs with at most this many registers use shared memory

constexpr ull P_ERA = 2;
constexpr ull P_FREE = 0x8000000000000000ull;
constexpr ull P_LOCK = 0xFFFFFFFFFFFFFFF0ull;
constexpr ull P_GONE = 0xFFFFFFFFFFFFFFFFull;
constexpr ull P_CLAIM = 0xFFFFFFFFFFFFFFF8ull;  // a freed word whose node a lane is about to reclaim (see claim)
constexpr ull A_MASK = 0x0000FFFFFFFFFFF8ull;
constexpr ull X_BIT = 1ull << 47;  // expansion-agent Ref ports

enum : int { RW_ANNI = 0, RW_COMM, RW_ERAS, RW_DREF, RW_OPER };

// Global control block.  Hot counters sit on their own 128-byte lines.
struct Ctrl {
  ull bump;        // next never-used node index
  ull heap_nodes;
  ull heap_bytes;
  ull chunk_nodes;
  ull spin_limit;
  ull deadline;    // %globaltimer ns (the host emulation's; reducer warps keep their own, from timeout_ns)
  ull donate_min;
  ull max_warps;   // holders (warps + queued slots) per net beyond which no work is donated; 0: no cap
  ull q_mask;      // queue capacity - 1
  ull q_base;      // the run's first ticket
  ull q_warps;     // reducer warps
  int error;
  int error_net;
  ull error_info;
  ull pad0[4];
  long long nets_left;
  ull pad1[31];
  ull q_head;      // pop tickets taken: ahead of q_tail by the warps that wait
  ull pad3[15];
  ull q_tail;
  ull pad4[15];
  ull stat_donated, stat_spilled, stat_overflow, pad10;
  ull stat_steps, stat_lanes, stat_busy_cycles, stat_idle_cycles;
  ull timeout_ns;  // per launch: each warp's deadline is its start + timeout_ns
  ull pad5[7];
  ull req_head;       // serving: requests admitted so far
  ull pad6[15];
  ull req_tail;       // serving: requests the host has written (host copies, device reads)
  int stop;           // serving: the host asks the reducer to end once idle
  int pad7;
  ull pad8[14];
  ull free_top;       // shared stack of free-node batches: batch head address | push count << 44
  ull reuse_mark;     // bump position from which free nodes are shared between warps
  ull captured;       // pre-reduce: redexes recorded by inert Defs (see capture)
  ull rw_done;        // interactions folded so far, when the run has an interaction limit
  ull pad9[12];
};

constexpr int NCOUNT = 8;  // rw[5] then comm22, dref_nodes, dref_links
enum : int { EX_COMM22 = 5, EX_DNODES, EX_DLINKS };

struct NetState {  // 112 bytes
  ull root;            // byte offset of the root wire
  long long pending;   // warps holding this net's work + queued chunks
  ull rw[NCOUNT];
  int prog;            // DevDef index of the boot program
  int status;
  ull ticket, t_admit; // serving: the request running in this slot
};

struct Slot {  // 544 bytes: one chunk of up to 32 redexes of one net
  ull seq;
  unsigned net;
  unsigned count;
  ull pad[2];
  ull r[2 * CHUNK];
};

// Host side: the queue's part of a run's control block.  `next` is kept beside
// the ring: the first ticket of the run to come, above every sequence word that
// earlier runs left in it (all zero before the first) and a multiple of every
// capacity.  It moves on by what a run used (queue_end; by more than any run
// uses until then), so it does not wrap in 2^39 runs.
constexpr unsigned MAX_QLOG2 = 24;  // the largest capacity
constexpr unsigned Q_RUN_BITS = 36;
inline void queue_begin(Ctrl& c, unsigned qlog2, unsigned warps, uint64_t& next) {
  if (next == 0) next = 1ull << MAX_QLOG2;
  c.q_mask = (1ull << qlog2) - 1;
  c.q_warps = warps;
  c.q_base = c.q_head = c.q_tail = next;
  next += 1ull << Q_RUN_BITS;
}
// `c`: the control block after the run.  Its last words lie at most one lap
// above its tickets.
inline void queue_end(const Ctrl& c, uint64_t& next) {
  const uint64_t used = (c.q_head > c.q_tail ? c.q_head : c.q_tail) + c.q_mask + 1;
  next = ((used >> MAX_QLOG2) + 1) << MAX_QLOG2;
}

// Serving: one request (host -> device) and one completion record (device ->
// host).  Both live in page-locked host memory mapped into the device.
struct ServeReq {  // 16 bytes
  ull ticket;       // nonzero
  unsigned slot;    // net slot the request runs in
  unsigned prog;    // DevDef index of the Def to boot
};
struct ServeDone {  // 128 bytes; `ticket` is written last
  ull ticket;
  int status;
  unsigned pairs;   // (address, word) pairs gathered into the slot's output
  ull root;
  ull rw[NCOUNT];
  ull t_admit, t_done;  // %globaltimer, ns
  ull pad[2];
};

struct Params {
  ull* heap;
  ull heap_bytes;
  Ctrl* ctrl;
  NetState* nets;
  unsigned nnets;
  Slot* q;
  const DevDef* __restrict__ defs;
  const DevInstr* __restrict__ instrs;
  const ull* __restrict__ labbits;
  unsigned ndefs;
  // per-warp overflow stacks: warp g of the reducer grid owns
  // spill[2 * spill_cap * g ...] (spill_cap redexes); null: none
  unsigned spill_cap;
  ull* spill;
  unsigned ovf_flush;           // free-list length at which a lane publishes it (see free_list_push)
  // register files of Def calls needing more than LOCAL_REGS registers:
  // warp g owns bigregs[32 * MAX_REGS * g ...], [register][lane]; null: none
  ull* bigregs;
  // pre-reduce (all zero otherwise): boot without the expansion agent
  // (Net::reduce after Net::boot, transform/src/pre_reduce.rs:145-147); the
  // buffer for redexes inert Defs capture; an interaction limit
  unsigned no_expand, capture_cap;
  ull* capture;
  ull rw_limit;
  // work sharing (see Ctrl, which holds the queue's counters): copies here are
  // constant-bank operands, where a load would miss L1 after every fence
  ull q_base, q_mask;
  unsigned q_warps, donate_min, max_warps;
  unsigned max_pushes;  // redexes one interaction may push, over all Defs
  unsigned pool_cap;    // a warp's pool of free nodes: POOL or POOL_BUDGETED
  unsigned chunk_shift; // a lane takes at most this fraction (2^-chunk_shift) of the fresh nodes left at once
  unsigned gen;  // 1: the compiled Def functions match the loaded Book (HVM_GEN_INCLUDE builds)
  // serving (all zero for a batch run)
  unsigned serve;
  const ServeReq* req;         // device ring of req_cap requests
  ServeDone* done;             // per slot (mapped host memory)
  ull* out;                    // per slot: out_cap (address, word) pairs (mapped host memory)
  unsigned req_cap, out_cap;
};

// The run's parameters: one constant-memory block per device, uploaded on
// the launching stream before the run's kernels (constant-bank operands cost
// no instruction; a per-block shared-memory copy measured 11 % slower).  A
// run owns the block until its kernels finish: the host runner gives runs on
// one device turns (hvm64.cu, DeviceTurn).  The host emulation uses a plain
// global.
#ifdef __CUDACC__
__constant__ Params g_P;
#else
inline Params g_P;
#endif

// ---- platform layer ------------------------------------------------------------
// The runtime below is written against these few operations.  Under nvcc
// they are strong GPU-scope PTX accesses and CUDA atomics; under a host
// compiler (the CPU emulation harness the tests build from this same file)
// they are std::atomic_ref operations, so the protocol logic can be exercised
// with many host threads.
#ifdef __CUDACC__
#define HVM_DEV __device__
#define HVM_INL __device__ __forceinline__
// Rare paths stay out of line so the hot loop stays small (instruction cache)
// and needs fewer registers.
#define HVM_COLD __device__ __noinline__
__device__ __forceinline__ ull ld_gpu(const ull* p) {
  ull v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_gpu(ull* p, ull v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ int ld_gpu32(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ ull globaltimer() {
  ull t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ ull atom_exch(ull* p, ull v) { return atomicExch(p, v); }
__device__ __forceinline__ ull atom_cas(ull* p, ull e, ull v) { return atomicCAS(p, e, v); }
__device__ __forceinline__ ull atom_add(ull* p, ull v) { return atomicAdd(p, v); }
__device__ __forceinline__ int atom_cas32(int* p, int e, int v) { return atomicCAS(p, e, v); }
__device__ __forceinline__ unsigned atom_add_u32(unsigned* p, unsigned v) { return atomicAdd(p, v); }
__device__ __forceinline__ int atom_add_i32(int* p, int v) { return atomicAdd(p, v); }
// Fetch-and-add on a word of a warp's shared-memory state (`p` is a generic
// pointer into shared memory).  A plain shared-memory atomic per lane:
// aggregating the converged lanes first (match, leader, shuffle) measured
// 8 % slower overall -- its extra instructions cost more than the few lanes
// that serialise on the word.
__device__ __forceinline__ int smem_add_i32(int* p, int v) {
  int old;
  unsigned a = unsigned(__cvta_generic_to_shared(p));
  asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(old) : "r"(a), "r"(v) : "memory");
  return old;
}
__device__ __forceinline__ unsigned smem_add_u32(unsigned* p, unsigned v) {
  return unsigned(smem_add_i32(reinterpret_cast<int*>(p), int(v)));
}
// A release fence: the node fills and links before it are visible to any
// lane that later reaches the node through a port published after it.
__device__ __forceinline__ void mem_fence() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void mem_fence_sc() { asm volatile("fence.sc.gpu;" ::: "memory"); }
__device__ __forceinline__ void pause_brief() { __nanosleep(64); }
// LOCK-fill nodes [s, s+n) with 16-byte stores.
__device__ __forceinline__ void lock_fill(ull* H, ull s, ull n) {
  ulonglong2* c = reinterpret_cast<ulonglong2*>(H) + s;
  for (ull k = 0; k < n; k++) c[k] = make_ulonglong2(P_LOCK, P_LOCK);
}
#else
#define HVM_DEV
#define HVM_INL inline
#define HVM_COLD __attribute__((noinline))
#ifdef HVM_EMU_STRESS
// Test builds only: yield at random inside memory operations to widen race
// windows.
inline void emu_jitter() {
  thread_local unsigned x = 0x9E3779B9u ^ unsigned(std::hash<std::thread::id>{}(std::this_thread::get_id()));
  x ^= x << 13; x ^= x >> 17; x ^= x << 5;
  if ((x & 31) == 0) std::this_thread::yield();
}
#else
inline void emu_jitter() {}
#endif
inline ull ld_gpu(const ull* p) {
  emu_jitter();
  return std::atomic_ref<ull>(*const_cast<ull*>(p)).load(std::memory_order_acquire);
}
inline void st_gpu(ull* p, ull v) {
  emu_jitter();
  std::atomic_ref<ull>(*p).store(v, std::memory_order_release);
}
inline int ld_gpu32(const int* p) {
  return std::atomic_ref<int>(*const_cast<int*>(p)).load(std::memory_order_acquire);
}
inline ull globaltimer() {
  return ull(std::chrono::duration_cast<std::chrono::nanoseconds>(
                 std::chrono::steady_clock::now().time_since_epoch()).count());
}
inline ull atom_exch(ull* p, ull v) {
  emu_jitter();
  return std::atomic_ref<ull>(*p).exchange(v);
}
inline ull atom_cas(ull* p, ull e, ull v) {
  emu_jitter();
  std::atomic_ref<ull>(*p).compare_exchange_strong(e, v);
  return e;
}
inline ull atom_add(ull* p, ull v) { return std::atomic_ref<ull>(*p).fetch_add(v); }
inline int atom_cas32(int* p, int e, int v) {
  std::atomic_ref<int>(*p).compare_exchange_strong(e, v);
  return e;
}
inline unsigned atom_add_u32(unsigned* p, unsigned v) { return std::atomic_ref<unsigned>(*p).fetch_add(v); }
inline int atom_add_i32(int* p, int v) { return std::atomic_ref<int>(*p).fetch_add(v); }
inline int smem_add_i32(int* p, int v) { return atom_add_i32(p, v); }
inline unsigned smem_add_u32(unsigned* p, unsigned v) { return atom_add_u32(p, v); }
inline void mem_fence() { std::atomic_thread_fence(std::memory_order_seq_cst); }
inline void mem_fence_sc() { std::atomic_thread_fence(std::memory_order_seq_cst); }
inline void pause_brief() { std::this_thread::yield(); }
inline void lock_fill(ull* H, ull s, ull n) {
  for (ull k = 0; k < 2 * n; k++) st_gpu(H + 2 * s + k, P_LOCK);
}
#endif
#ifdef HVM_EMU_CHECK_ALLOC
// Host test builds only: per node, whether it is handed out (top bit); a node
// handed out while out, or reclaimed while not out, is counted here.
inline std::atomic<unsigned>* g_node_out = nullptr;
inline std::atomic<unsigned long long> g_alloc_faults{0};
inline void check_handed_out(ull node) {
  if (node && (g_node_out[node >> 4].fetch_or(1u) & 1u)) g_alloc_faults++;
}
inline void check_reclaimed(ull node) {
  if (!(g_node_out[node >> 4].fetch_and(~1u) & 1u)) g_alloc_faults++;
}
#endif
HVM_INL long long ld_gpu64s(const long long* p) {
  return (long long)ld_gpu(reinterpret_cast<const ull*>(p));
}

// ---- ports (runtime/src/port.rs) ---------------------------------------------
HVM_INL unsigned ptag(ull p) { return unsigned(p & 7); }
HVM_INL unsigned plab(ull p) { return unsigned(p >> 48); }
HVM_INL ull paddr(ull p) { return p & A_MASK; }
HVM_INL ull mkport(unsigned tag, unsigned lab, ull addr) { return (ull(lab) << 48) | addr | tag; }
HVM_INL ull pvar(ull a) { return a | T_VAR; }
HVM_INL ull pred(ull a) { return a | T_RED; }
HVM_INL bool principal(ull p) { return ptag(p) >= T_REF; }
HVM_INL bool skippable(ull p) {  // port.rs:205-207
  return ptag(p) == T_NUM || (ptag(p) == T_REF && plab(p) != 0xFFFF);
}
HVM_INL bool is_expand(ull p) { return ptag(p) == T_REF && (p & X_BIT) != 0; }
// Trg (runtime/src/linker.rs:228-281): a wire is its address with the Red tag.
HVM_INL bool trg_is_wire(ull t) { return ptag(t) == T_RED; }

// The rules other than Def calls run as short instruction lists of the same
// VM (see exec_ins), on registers their set-up fills (see classify):
//   two links of consumed wires   registers 0, 1 (one node's words) with 2, 3
//   four links                    registers 0 - 3 (two nodes' words) with 4 - 7
//   a binary operator and a number: register 0 (rhs wire), 1 (result wire), 2 (number and operator)
constexpr unsigned RULE_LINK2 = 0, RULE_LINK2_LEN = 2;
constexpr unsigned RULE_LINK4 = 2, RULE_LINK4_LEN = 4;
constexpr unsigned RULE_OP = 6, RULE_OP_LEN = 2;
constexpr unsigned RULE_INS = 8;
// (I_OPRED: do_op_num on a T_OP node's two wires)
#ifdef __CUDACC__
__constant__
#else
inline
#endif
const DevInstr RULES[RULE_INS] = {
    {I_LINK, 0, 0, 0, 2, 0, 0, 0}, {I_LINK, 0, 0, 1, 3, 0, INS_A_LAST | INS_B_LAST, 0},
    {I_LINK, 0, 0, 0, 4, 0, 0, 0}, {I_LINK, 0, 0, 1, 5, 0, INS_A_LAST, 0},
    {I_LINK, 0, 0, 2, 6, 0, 0, 0}, {I_LINK, 0, 0, 3, 7, 0, INS_A_LAST, 0},
    {I_OPRED, 0, 0, 0, 2, 2, 0, 0}, {I_LINK, 0, 0, 1, 2, 0, INS_A_LAST, 0},
};

// Rule class of a redex, following interact()'s dispatch: the Def index for
// a Def call (calls of one Def run the same instruction stream), else a small
// code per rule.  Warps pick redexes of one class per step to stay convergent.
HVM_INL unsigned redex_class(ull a, ull b) {
  unsigned at = unsigned(a & 7), bt = unsigned(b & 7);
  if (at == T_REF && !(a & X_BIT) && a != P_ERA) return 63 + unsigned((a & A_MASK) >> 3);  // 64 + Def index
  if (bt == T_REF && !(b & X_BIT) && b != P_ERA) return 63 + unsigned((b & A_MASK) >> 3);
  if ((a & X_BIT) || (b & X_BIT)) return 1;
  if (at == bt) return 2 + at;  // annihilation (or nilary pair)
  return 16 + at * 8 + bt;      // commutation / native ops
}

// Per-warp shared state of the reducer (one per warp; the CPU emulation
// harness gives each host thread one too).  Warps' states lie back to back in
// shared memory and `icache` is filled with 16-byte stores, so the size is
// kept a multiple of 16.
struct alignas(16) WarpSmem {
  ull stk[2 * SCAP];          // redex stack (ring of SCAP pairs)
  ull regs[SMALL_REGS * 32];  // VM registers, [register][lane]
  ull pool[POOL];             // free nodes ready for reuse
  ull freed[POOL];            // nodes reclaimed during the current step
  DevInstr icache[ICACHE];    // the instructions of `icache_def`, staged for this step
  DevInstr rules[RULE_INS];   // the rules' own instructions (RULES)
  DevDef idef;                // that Def's header
  unsigned icache_def;        // Def index staged in icache (~0u: none)
  ull rw[NCOUNT];             // counters of the warp's current net
  unsigned cnt[NCOUNT * 32];  // per lane: counts of this step, [counter][lane] (folded into rw)
  ull ovf[32];                // per lane: free list head | pushes since published << 48 (see free_list_push)
  ull fw[FREED_ALONE * 32];   // per lane: words freed alone by the current interaction
  ull fails[FAILS * 32];      // per lane: the first consumed wires the current interaction left as redirects
  ull bnext[32], bend[32];    // per lane: pre-LOCKed bump chunk [bnext, bend), node indices
#ifdef HVM_GEN_INCLUDE
  unsigned allocs[32];        // per lane: nodes allocated (for the DREF statistics)
#endif
  unsigned ring_base;         // this step's pushes go to stack slots ring_base + k ...
  unsigned ring_cap;          // ... for k < ring_cap; push k >= ring_cap goes to the overflow stack
  ull* sp;                    // this warp's overflow stack in HBM (null: none; pushes go to the queue)
  ull* bigregs;               // this warp's register files for Defs above LOCAL_REGS (null: none)
  unsigned sp_n, sp_cap;      // redexes in it between steps, and its capacity
  int pool_cap;               // 0: no reuse pool (reclaimed nodes go to `ovf`)
  ull st_steps, st_lanes, st_busy, st_idle, st_donated, st_spilled;
  unsigned ring_cnt;
  int pool_n;
  int freed_n;
  unsigned pad;
};
static_assert(sizeof(WarpSmem) % 16 == 0 && offsetof(WarpSmem, icache) % 16 == 0 &&
                  offsetof(WarpSmem, rules) % 16 == 0 && offsetof(WarpSmem, stk) % 16 == 0,
              "the 16-byte accesses to every warp's state must be aligned");

// Initial per-lane / per-warp runtime state (lane `ln` of warp state `W`).
HVM_INL void lane_init(WarpSmem* W, unsigned ln) {
  for (int k = 0; k < NCOUNT; k++) W->cnt[k * 32 + ln] = 0;
  W->ovf[ln] = 0;
  for (int k = 0; k < FREED_ALONE; k++) W->fw[k * 32 + ln] = 0;
  W->bnext[ln] = W->bend[ln] = 0;
#ifdef HVM_GEN_INCLUDE
  W->allocs[ln] = 0;
#endif
}

// ---- cold paths as free functions over scalars -------------------------------
// (A Lane never has its address taken, so its state stays in registers.)
HVM_COLD void run_fail(unsigned net, int code, ull info) {
  if (atom_cas32(&g_P.ctrl->error, 0, code) == 0) {
    g_P.ctrl->error_info = info;
    g_P.ctrl->error_net = int(net);
  }
}
HVM_INL bool run_failed() { return ld_gpu32(&g_P.ctrl->error) != 0; }
// run_fail for the failure branches of code that is inlined at many sites
// (heap accesses, bounded waits): a call there, even one never taken, makes
// every such site keep its live registers across the call, which costs the
// reducer about a tenth of its throughput.
// (Only the code is recorded: storing the net and detail too measured 4 %
// slower.)
HVM_INL void run_fail_here(int code) { atom_cas32(&g_P.ctrl->error, 0, code); }
// One poll of a bounded wait; false = abandon the wait.
HVM_INL bool run_spin(unsigned net, unsigned& it) {
  ++it;
  if ((it & 63) == 0) {
    if (run_failed()) return false;
    if (it > g_P.ctrl->spin_limit) {
      run_fail_here(HVM64_ERR_TIMEOUT);
      return false;
    }
    pause_brief();
  }
  return true;
}
HVM_INL ull* heap_at(unsigned net, ull a) {
  if (a >= g_P.heap_bytes) {
    run_fail_here(HVM64_ERR_BAD_ADDR);
    a = 0;
  }
  return g_P.heap + (a >> 3);
}
// wire.rs:342-350: wait until the word is not LOCK and take it.
HVM_COLD ull relock(unsigned net, ull w) {
  unsigned it = 0;
  for (;;) {
    ull got = atom_exch(heap_at(net, w), P_LOCK);
    if (got != P_LOCK) return got;
    if (!run_spin(net, it)) return P_ERA;
  }
}
HVM_COLD uint32_t binary_op(unsigned net, uint32_t a, uint32_t op, uint32_t b) {
  int e = 0;
  uint32_t r = num_binary(a, op, b, &e);
  if (e) run_fail(net, HVM64_ERR_DIV0, net);
  return r;
}
// Neither the warp's stack nor its overflow stack had room: the platform
// driver ships the redex to shared work (the CUDA driver: a one-redex queue
// slot, or HVM64_ERR_QUEUE when the queue is full -- it never waits).
HVM_COLD void push_overflow(unsigned net, ull a, ull b);
// A lane's free list of reclaimed nodes is linked through their left words
// (right words LOCK); the lane's head word holds the first node's address in
// bits 0-47 and the number of nodes pushed since the list was last
// published in bits 48-63.
//
// Free nodes move between warps through one shared stack of batches, once
// the heap is past its reuse mark (Ctrl::reuse_mark: half the heap): a lane's
// list is published whole once it holds Params::ovf_flush nodes (OVF_FLUSH for
// a batch, 32 for a server, which keeps fewer nodes stranded per lane), the
// batch's head node linking the next batch through its right word, and a lane
// whose list is empty takes a batch before it takes fresh nodes from the bump
// pointer.  Below the mark, allocation stays
// on the bump pointer and the lanes' own lists (no shared traffic).  The top
// word carries a push/pop count above the address bits, so a pop whose
// batch was taken and republished meanwhile fails its CAS (ABA).
#ifndef HVM_OVF_FLUSH
#define HVM_OVF_FLUSH 128
#endif
constexpr unsigned OVF_FLUSH = HVM_OVF_FLUSH;  // batch runs (a server publishes after 32)
constexpr ull FT_ADDR = (1ull << 44) - 1;
constexpr ull FT_TAG = 1ull << 44;
constexpr ull OVF_ADDR = (1ull << 48) - 1;
HVM_INL bool past_reuse_mark() { return ld_gpu(&g_P.ctrl->bump) >= g_P.ctrl->reuse_mark; }
HVM_COLD void free_publish(unsigned net, ull* ovf) {
  ull head = *ovf & OVF_ADDR;
  if (!head) return;
  ull* top = &g_P.ctrl->free_top;
  unsigned it = 0;
  for (;;) {
    ull t = ld_gpu(top);
    st_gpu(heap_at(net, head | 8), t & FT_ADDR);
    mem_fence();  // the batch's links are visible before its head is
    if (atom_cas(top, t, (head & FT_ADDR) | ((t & ~FT_ADDR) + FT_TAG)) == t) break;
    if (!run_spin(net, it)) return;  // lost CASes are other lanes' progress; still bounded
  }
  *ovf = 0;
}
// Take one batch from the shared stack as the lane's list; false when empty.
// (The lanes of a step run out together and contend for the top: each lost
// CAS is another lane's success, so a lane tries long enough for many of
// them before it falls back to fresh nodes.)
HVM_COLD bool free_take(unsigned net, ull* ovf) {
  ull* top = &g_P.ctrl->free_top;
  for (int tries = 0; tries < 2048; tries++) {
    if ((tries & 7) == 7) pause_brief();
    ull t = ld_gpu(top);
    ull a = t & FT_ADDR;
    if (a == 0) return false;
    // Stale when the batch was taken meanwhile; then the CAS below fails.
    ull next = ld_gpu(heap_at(net, a | 8));
    if (atom_cas(top, t, (next & FT_ADDR) | ((t & ~FT_ADDR) + FT_TAG)) == t) {
      mem_fence();
      st_gpu(heap_at(net, a | 8), P_LOCK);
      *ovf = a;
      return true;
    }
  }
  return false;
}
constexpr ull CHUNK_LEAST = 8;
// Pop the lane's free list (or, past the reuse mark, a shared batch) / take
// a new pre-LOCKed bump chunk.
struct Refill {
  ull node, bnext, bend;
};
HVM_COLD Refill alloc_refill(unsigned net, ull* ovf) {
  const bool own = (*ovf & OVF_ADDR) != 0;
  const ull used = own ? 0 : ld_gpu(&g_P.ctrl->bump);
  if (own || (used >= g_P.ctrl->reuse_mark && free_take(net, ovf))) {
    ull a = *ovf & OVF_ADDR, n = *ovf >> 48;
    if (a >= g_P.heap_bytes) {  // links are heap words: checked before the node is handed out
      run_fail(net, HVM64_ERR_BAD_ADDR, a);
      *ovf = 0;
      return {0, 0, 0};
    }
    *ovf = (ld_gpu(heap_at(net, a)) & OVF_ADDR) | ((n ? n - 1 : 0) << 48);
    st_gpu(heap_at(net, a), P_LOCK);
    mem_fence();
    return {a, 0, 0};
  }
  // At most the lane's share of what is left (an eighth of it over all lanes,
  // see sharing_params): work is shared out to every warp from a few waiting
  // redexes on, and a full chunk a lane took a tree sum of 2^10 leaves 18 MB of
  // heap, a sort of 2^9 keys 69 MB.  Not below CHUNK_LEAST, where the counter
  // itself is what a narrow net waits for (a Church tower in 8 MB: 93 ms with
  // single nodes, 77 ms with full chunks).
  ull n = g_P.ctrl->chunk_nodes;
  const ull share = (g_P.ctrl->heap_nodes - (used < g_P.ctrl->heap_nodes ? used : g_P.ctrl->heap_nodes)) >> g_P.chunk_shift;
  if (share < n && n > CHUNK_LEAST) n = share > CHUNK_LEAST ? share : CHUNK_LEAST;
  ull s = atom_add(&g_P.ctrl->bump, n);
  if (s + n > g_P.ctrl->heap_nodes) {
    run_fail(net, HVM64_ERR_OOM, s);
    return {0, 0, 0};
  }
  lock_fill(g_P.heap, s, n);
  mem_fence();  // LOCK is visible before any of these nodes escapes
  return {s << 4, s + 1, s + n};
}
// A reclaimed node (both words LOCK) onto a lane's free list.
HVM_INL void free_list_push(unsigned net, ull* ovf, ull node) {
  ull n = (*ovf >> 48) + 1;
  st_gpu(heap_at(net, node), *ovf & OVF_ADDR);
  *ovf = node | (n < 0xFFFF ? n << 48 : 0xFFFFull << 48);
  if (n >= g_P.ovf_flush && past_reuse_mark()) free_publish(net, ovf);
}

// ---- the runtime proper ------------------------------------------------------
// Everything works on a three-word context (warp state, lane, net).  A lane's
// mutable state (freed-word slots, bump chunk) lives in its warp's shared
// memory.  The usual paths are inlined once into the reducer's step (exec_ins);
// the others are out-of-line functions.
struct Ctx {
  WarpSmem* W;
  unsigned lane;
  unsigned net;
};

#define LS(field) (c.W->field[c.lane])             // a lane's slot
#define FW(k) (c.W->fw[(k) * 32 + c.lane])          // freed-word slot k

HVM_INL ull hload(const Ctx c, ull a) { return ld_gpu(heap_at(c.net, a)); }
HVM_INL void hstore(const Ctx c, ull a, ull v) { st_gpu(heap_at(c.net, a), v); }
HVM_INL ull hswap(const Ctx c, ull a, ull v) { return atom_exch(heap_at(c.net, a), v); }
HVM_INL ull hcas(const Ctx c, ull a, ull e, ull v) { return atom_cas(heap_at(c.net, a), e, v); }
HVM_INL void count(const Ctx c, int k, ull v = 1) { c.W->cnt[k * 32 + c.lane] += unsigned(v); }

// wire.rs:342-350
HVM_INL ull lock_target(const Ctx c, ull w) {
  ull got = hswap(c, w, P_LOCK);
  return got != P_LOCK ? got : relock(c.net, w);
}

// ---- allocator -------------------------------------------------------------
// The reference's allocator (runtime/src/allocator.rs:73-110) writes LOCK
// into both words of every node it hands out and links a node into a free
// list once both halves are FREE.  Here a free node always holds LOCK in both
// words, so alloc() itself touches no heap memory:
//  - a bump chunk is LOCK-filled and fenced when it is taken;
//  - a node an interaction consumes has both its words taken by exchanges
//    with LOCK.  Once both wires are linked nothing refers to the node, it
//    already holds what a free node must hold, and it is reclaimed without
//    touching memory (recycle; see wire_done);
//  - a word freed alone follows the reference's store-FREE / read-other-half /
//    CAS sequence, which decides which lane reclaims the node (half_free,
//    settle, claim); the lane that does writes LOCK and fences.
// Every address alloc() returns lies in the heap: it comes from the bump
// pointer, from recycle() (called with checked addresses), or from a list
// whose links are checked as they are followed (alloc_refill).  Stores to a
// new node's words therefore need no check of their own, even in the steps
// that still run after an allocation failed (alloc() then returns node 0, a
// scratch node).
HVM_COLD void recycle_spill(const Ctx c, ull node) { free_list_push(c.net, &LS(ovf), node); }
HVM_INL void recycle(const Ctx c, ull node) {
#ifdef HVM_EMU_CHECK_ALLOC
  check_reclaimed(node);
#endif
  int k = c.W->pool_cap ? smem_add_i32(&c.W->freed_n, 1) : POOL;
  if (k < c.W->pool_cap) c.W->freed[k] = node;
  else recycle_spill(c, node);
}
// A node whose words this lane has just LOCKed with stores.
HVM_COLD void recycle_stored(const Ctx c, ull node) {
  if (node >= g_P.heap_bytes) return run_fail(c.net, HVM64_ERR_BAD_ADDR, node);
  mem_fence();  // the LOCKs are visible before the node is handed out again
  recycle(c, node);
}
HVM_COLD ull alloc_slow(const Ctx c) {
  Refill r = alloc_refill(c.net, &LS(ovf));
  if (r.bend) {
    LS(bnext) = r.bnext;
    LS(bend) = r.bend;
  }
  return r.node;
}
#ifdef HVM_EMU_CHECK_ALLOC
HVM_INL ull alloc_unchecked(const Ctx c);
HVM_INL ull alloc(const Ctx c) {
  ull n = alloc_unchecked(c);
  check_handed_out(n);
  return n;
}
HVM_INL ull alloc_unchecked(const Ctx c) {
#else
HVM_INL ull alloc(const Ctx c) {
#endif
#ifdef HVM_GEN_INCLUDE
  LS(allocs)++;
#endif
  int k = smem_add_i32(&c.W->pool_n, -1) - 1;
  if (k >= 0) return c.W->pool[k];
  ull b = LS(bnext);
  if (b != LS(bend)) {
    LS(bnext) = b + 1;
    return b << 4;
  }
  return alloc_slow(c);
}
HVM_COLD ull alloc_cold(const Ctx c) { return alloc(c); }
// A word freed alone: a node found fully free is claimed by CAS on its left
// word, then kept only if its right word is still free -- between the load
// and the CAS the node may have been reclaimed by the other half's owner,
// reused, and half-freed again (ABA); then the left word is handed back.
// (Not LOCK in between: the owner of the other half would take that for a
// word it linked, see was_linked.)
HVM_COLD void claim(const Ctx c, ull w, ull other) {
  if (!w || other != P_FREE) return;
  ull l = w & ~8ull;
  if (hcas(c, l, P_FREE, P_CLAIM) != P_FREE) return;
  if (hload(c, l | 8) == P_FREE) {
    hstore(c, l, P_LOCK);
    hstore(c, l | 8, P_LOCK);
    recycle_stored(c, l);
  } else {
    hstore(c, l, P_FREE);
  }
}
// End of an interaction: look at the other half of every word freed alone
// (the loads are in flight together).
HVM_COLD void settle(const Ctx c) {
  ull w0 = FW(0), w1 = FW(1);
  if (!(w0 | w1)) return;
  mem_fence_sc();  // the FREEs are visible before the loads: of two lanes freeing one node's halves, one sees both
  ull o0 = w0 ? hload(c, w0 ^ 8) : 0, o1 = w1 ? hload(c, w1 ^ 8) : 0;
  FW(0) = FW(1) = 0;
  claim(c, w0, o0);
  claim(c, w1, o1);
}
HVM_COLD void half_free(const Ctx c, ull a) {
  ull x = a ^ 8;
  int k = -1;
  if (a != 0) {
    if (FW(0) == x) k = 0;
    else if (FW(1) == x) k = 1;
  }
  if (k >= 0) {  // both halves freed by this interaction: no one else can claim the node
    FW(k) = 0;
    ull l = a & ~8ull;
    hstore(c, l, P_LOCK);
    hstore(c, l | 8, P_LOCK);
    recycle_stored(c, l);
    return;
  }
  hstore(c, a, P_FREE);
  if (FW(0) == 0) FW(0) = a;
  else if (FW(1) == 0) FW(1) = a;
  else {
    settle(c);
    FW(0) = a;
  }
}
static_assert(FREED_ALONE == 2, "settle and half_free name their slots");

// ---- redex pushes (linker.rs:70-85) -----------------------------------------
// The reference's queue is an unbounded vector (linker.rs:308-344); here a
// step's k-th push goes to the warp's shared-memory stack while it has room,
// then to the warp's private overflow stack in HBM (slot sp_n + k - ring_cap),
// then to the global queue.  None of these waits for anyone.
HVM_COLD void push_spill(const Ctx c, ull a, ull b, unsigned j) {
  unsigned i = c.W->sp_n + j;
  if (c.W->sp && i < c.W->sp_cap) {
    c.W->sp[2 * ull(i)] = a;
    c.W->sp[2 * ull(i) + 1] = b;
    return;
  }
  push_overflow(c.net, a, b);
}
HVM_INL void push(const Ctx c, ull a, ull b) {
  unsigned cap = c.W->ring_cap;
  unsigned k = smem_add_u32(&c.W->ring_cnt, 1u);
  if (k < cap) {
    unsigned i = (c.W->ring_base + k) & unsigned(SCAP - 1);
    c.W->stk[2 * i] = a;
    c.W->stk[2 * i + 1] = b;
  } else {
    push_spill(c, a, b, k - cap);
  }
}
// After a step that pushed `cnt` redexes (the value of ring_cnt): how many of
// them went to the overflow stack (the rest of those past ring_cap went to
// the queue).
HVM_INL unsigned spilled_of(const WarpSmem* W, unsigned cnt) {
  if (cnt <= W->ring_cap || !W->sp) return 0;
  unsigned over = cnt - W->ring_cap, room = W->sp_cap - W->sp_n;
  return over < room ? over : room;
}
// Upper bound on the redexes one interaction of rule class `cls` pushes
// (redex_class codes): an instruction of a Def pushes at most one (each
// link resolves to at most one active pair); a Def call that commutes
// instead (def.rs:182-184) pushes two, comm22 four, the other rules fewer.
HVM_INL unsigned pushes_bound(unsigned cls) {
  if (cls >= 64 && cls - 64 < g_P.ndefs) {
    unsigned r = g_P.defs[cls - 64].redexes;
    return r > 4 ? r : 4;
  }
  return 4;
}
HVM_INL void redux(const Ctx c, ull a, ull b) {
  if (skippable(a) && skippable(b)) count(c, RW_ERAS);
  else push(c, a, b);
}

// ---- linker (runtime/src/linker.rs:25-203) ----------------------------------
HVM_INL void half_link_port_port(const Ctx c, ull a, ull b) {
  if (ptag(a) == T_VAR) hstore(c, paddr(a), b);
}
HVM_INL void link_port_port(const Ctx c, ull a, ull b) {
  if (principal(a) && principal(b)) {
    redux(c, a, b);
  } else {
    half_link_port_port(c, a, b);
    half_link_port_port(c, b, a);
  }
}
HVM_COLD void resolve_redirect_pri(const Ctx c, ull ap, ull aw, ull bp);
// The CAS lost against another lane linking the same wire: leave a redirect
// (linker.rs:109-123).
HVM_COLD void half_link_failed(const Ctx c, ull ap, ull aw, ull bp) {
  if (ptag(bp) == T_VAR) {
    hstore(c, aw, pred(paddr(bp)));
  } else if (principal(bp)) {
    hstore(c, aw, bp);
    resolve_redirect_pri(c, ap, aw, bp);
  } else {
    run_fail(c.net, HVM64_ERR_BAD_PAIR, bp);
  }
}
HVM_COLD void half_link_wire_port(const Ctx c, ull ap, ull aw, ull bp) {
  if (ptag(ap) == T_VAR) {
    if (hcas(c, paddr(ap), pvar(aw), bp) == pvar(aw)) half_free(c, aw);
    else half_link_failed(c, ap, aw, bp);
  } else {
    half_free(c, aw);
  }
}
// link_wire_port for a wire whose target `ap` was already taken (locked).
HVM_COLD void link_locked_wire_port(const Ctx c, ull aw, ull ap, ull bp) {
  if (principal(ap) && principal(bp)) {
    half_free(c, aw);
    redux(c, ap, bp);
  } else {
    half_link_wire_port(c, ap, aw, bp);
    half_link_port_port(c, bp, ap);
  }
}
HVM_INL void link_wire_port(const Ctx c, ull aw, ull bp) { link_locked_wire_port(c, aw, lock_target(c, aw), bp); }
HVM_COLD void resolve_redirect_pri(const Ctx c, ull ap, ull aw, ull bp) {
  unsigned it = 0;
  for (;;) {
    ull tw = paddr(ap);
    ull tp = hload(c, tw);
    if (tp == P_LOCK) {
      if (!run_spin(c.net, it)) return;
      continue;
    }
    if (ptag(tp) == T_RED) {
      if (!run_spin(c.net, it)) return;  // (a chain of redirects is finite, but after a failure it may be a cycle)
      half_free(c, tw);
      ap = tp;
      continue;
    }
    if (ptag(tp) == T_VAR) {
      if (hcas(c, tw, tp, bp) == tp) {
        tw = paddr(tp);
        tp = hload(c, tw);
        unsigned it2 = 0;
        while (tp != P_LOCK && ptag(tp) == T_RED) {
          half_free(c, tw);
          tw = paddr(tp);
          tp = hload(c, tw);
          if (!run_spin(c.net, it2)) return;
        }
        // The other end's way here is cut (its word holds bp now) and every
        // redirect on it is freed: when it led back to aw, nothing names aw
        // any more.  (Lanes of one step often take both ends of a wire at
        // the same time; without this each such meeting lost a node.)
        if (tw == aw) half_free(c, aw);
        return;
      }
      if (!run_spin(c.net, it)) return;
      continue;
    }
    if (principal(tp) || tp == P_GONE) {
      ull xw = aw < tw ? aw : tw;
      ull yw = aw < tw ? tw : aw;
      ull xp = hswap(c, xw, P_GONE);
      if (xp != P_GONE) {
        ull yp = hswap(c, yw, P_GONE);
        redux(c, xp, yp);
      } else {
        half_free(c, xw);
        unsigned it3 = 0;
        while (hload(c, yw) != P_GONE)  // (never LOCK meanwhile: see was_linked)
          if (!run_spin(c.net, it3)) return;
        half_free(c, yw);
      }
      return;
    }
    run_fail(c.net, HVM64_ERR_BAD_PAIR, tp);
    return;
  }
}
// ---- compiled Defs (HVM_GEN_INCLUDE) -----------------------------------------
// The primitives generated Def functions call: each instruction as one
// function, freeing consumed wires word by word (half_free).
#ifdef HVM_GEN_INCLUDE
HVM_INL void link_trg_port(const Ctx c, ull a, ull b) {
  if (trg_is_wire(a)) link_wire_port(c, a, b);
  else link_port_port(c, a, b);
}
HVM_COLD void link_wire_wire(const Ctx c, ull aw, ull bw) {
  // Both words belong to nodes this interaction consumes, so no other lane
  // takes them: the two exchanges go out together (one round trip instead of
  // two) and give the values the reference's take-one-then-the-other does; a
  // word its creator has not written yet (LOCK) is waited for after both.
  ull ap = hswap(c, aw, P_LOCK);
  ull bp = hswap(c, bw, P_LOCK);
  if (ap == P_LOCK) ap = relock(c.net, aw);
  if (bp == P_LOCK) bp = relock(c.net, bw);
  if (principal(ap) && principal(bp)) {
    half_free(c, aw);
    half_free(c, bw);
    redux(c, ap, bp);
  } else {
    half_link_wire_port(c, ap, aw, bp);
    half_link_wire_port(c, bp, bw, ap);
  }
}
HVM_COLD void link_trg(const Ctx c, ull a, ull b) {
  bool aw = trg_is_wire(a), bw = trg_is_wire(b);
  if (aw && bw) link_wire_wire(c, a, b);
  else if (aw) link_wire_port(c, a, b);
  else if (bw) link_wire_port(c, b, a);
  else link_port_port(c, a, b);
}
HVM_INL void free_trg(const Ctx c, ull t) {
  if (trg_is_wire(t)) half_free(c, t);
}
// The target of a Trg about to be consumed by a VM instruction.  A wire is
// locked rather than read: every path of the instruction then either frees
// that wire or links it at once (which would lock it first), so taking the
// lock up front saves a round trip and changes nothing observable.
HVM_INL ull trg_take(const Ctx c, ull t) { return trg_is_wire(t) ? lock_target(c, t) : t; }
// link_trg_port for a Trg taken with trg_take.
HVM_INL void link_taken(const Ctx c, ull t, ull target, ull b) {
  if (trg_is_wire(t)) link_locked_wire_port(c, t, target, b);
  else link_port_port(c, t, b);
}

HVM_COLD void do_ctr(const Ctx c, unsigned lab, ull trg, ull& o1, ull& o2) {
  ull port = trg_take(c, trg);
  if (ptag(port) == T_CTR && plab(port) == lab) {
    free_trg(c, trg);
    count(c, RW_ANNI);
    o1 = paddr(port);  // Trg::wire
    o2 = paddr(port) ^ 8;
    return;
  }
  ull n = alloc(c);
  link_taken(c, trg, port, mkport(T_CTR, lab, n));
  o1 = pvar(n);
  o2 = pvar(n ^ 8);
}
HVM_COLD void do_op(const Ctx c, unsigned op, ull trg, ull& o1, ull& o2) {
  ull port = trg_take(c, trg);
  if (ptag(port) == T_NUM) {
    free_trg(c, trg);
    ull n = alloc(c);
    hstore(c, n, ull(num_unary(op, uint32_t(port))));
    o1 = mkport(T_OP, NT_SYM, n);
    o2 = pvar(n ^ 8);
    return;
  }
  if (port == P_ERA) {
    free_trg(c, trg);
    o1 = o2 = P_ERA;
    return;
  }
  ull n = alloc(c);
  link_taken(c, trg, port, mkport(T_OP, op, n));
  o1 = pvar(n);
  o2 = pvar(n ^ 8);
}
HVM_COLD ull do_op_num(const Ctx c, unsigned op, ull trg, uint32_t rhs) {
  ull port = trg_take(c, trg);
  if (ptag(port) == T_NUM) {
    count(c, RW_OPER);
    free_trg(c, trg);
    return ull(binary_op(c.net, uint32_t(port), op, rhs));
  }
  if (port == P_ERA) {
    free_trg(c, trg);
    return P_ERA;
  }
  ull n = alloc(c);
  link_taken(c, trg, port, mkport(T_OP, op, n));
  hstore(c, n, ull(rhs));
  return pvar(n ^ 8);
}
HVM_COLD ull create_wire_to(const Ctx c, ull port) {  // node.rs:176-182
  ull a = alloc(c);
  half_free(c, a ^ 8);
  link_port_port(c, port, pvar(a));
  return a;
}
HVM_COLD void do_switch(const Ctx c, ull trg, ull& o1, ull& o2) {
  ull port = trg_take(c, trg);
  if (ptag(port) == T_NUM) {
    count(c, RW_OPER);
    free_trg(c, trg);
    uint32_t num = uint32_t(port);
    uint32_t n = num_tag(num) == NT_U24 ? num_payload(num) : 0;
    ull c1 = alloc(c);
    if (n == 0) {
      link_port_port(c, pvar(c1 ^ 8), P_ERA);
      o1 = mkport(T_CTR, 0, c1);
      o2 = create_wire_to(c, pvar(c1));
    } else {
      ull c2 = alloc(c);
      link_port_port(c, pvar(c1), P_ERA);
      link_port_port(c, pvar(c1 ^ 8), mkport(T_CTR, 0, c2));
      link_port_port(c, pvar(c2), ull(num_u24(n - 1)));
      o1 = mkport(T_CTR, 0, c1);
      o2 = create_wire_to(c, pvar(c2 ^ 8));
    }
    return;
  }
  if (port == P_ERA) {
    count(c, RW_ERAS);
    free_trg(c, trg);
    o1 = o2 = P_ERA;
    return;
  }
  ull m = alloc(c);
  link_taken(c, trg, port, mkport(T_SWITCH, 0, m));
  o1 = pvar(m);
  o2 = pvar(m ^ 8);
}
#endif

HVM_COLD void comm02(const Ctx c, ull a, ull b) {  // interact.rs:162-168
  count(c, RW_COMM);
  ull b1 = paddr(b);
  link_wire_port(c, b1, a);
  link_wire_port(c, b1 ^ 8, a);
}
// An inert Def's call (transform/src/pre_reduce.rs:96-101): the redex is
// recorded for the host, which puts it back into the net's redexes.
HVM_COLD void capture(const Ctx c, ull port, ull trg) {
  ull k = atom_add(&g_P.ctrl->captured, 1ull);
  if (k >= g_P.capture_cap) return run_fail(c.net, HVM64_ERR_OUTPUT, k);
  g_P.capture[2 * k] = port;
  g_P.capture[2 * k + 1] = trg;
}
// ---- instruction VM (runtime/src/instruction.rs:400-500, def.rs:217-289) -----
// One function runs every instruction kind and, through the RULES lists, every
// rule that rewires two binary nodes.  What bounds it is not memory bandwidth
// but instruction supply and the chain of dependent L2 round trips, so it is
// written to be inlined once into the reducer's step, without calls on its
// usual paths (an out-of-line function per primitive spent most of its
// instructions saving and restoring registers), and all kinds share one code
// path for taking a wire, allocating, and linking: the lanes of a step stay
// together and their memory operations go out together.  Against the
// out-of-line form, on one B200: a sort of 2^15 keys 620 -> 228 ms, a batch of
// 451 nets 1273 -> 694 ms, 90 -> 63 warp instructions an interaction.
//
// Every instruction has the same shape:
//   take    its operands that are wires, with one exchange each (both in
//           flight together).  Every path then links or frees them at once,
//           which would lock them first, so taking them up front changes
//           nothing observable;
//   rule    constructor match, operator, switch: what the operand meets;
//   link    the operand's target with the other side (linker.rs:25-203).
//
// More than half of a Def's instructions build its own nodes, and the encoder
// knows which (specialise_fresh, host.cpp): those need no take, no match and
// no general link.  They have kinds of their own (I_CALL to I_FCONST) with a
// few operations each (340-690 cycles instead of 1300-2000; a sort of 2^9 keys
// 20.1 -> 17.9 ms, a batch of 451 nets 369 -> 343 ms).
//
// Wires an interaction consumes come in pairs, the two words of one consumed
// node.  The encoder marks the operand that consumes the later one of a pair
// (INS_A_LAST, INS_B_LAST); the node is reclaimed there, when neither of its
// words was left as a redirect (wire_done, wire_failed).
struct Exec {
  unsigned nf = 0;  // wires left as redirects so far (the first FAILS of them are in WarpSmem::fails)
  unsigned anni = 0, oper = 0, eras = 0, nodes = 0;
};
#define FAIL(k) (c.W->fails[(k) * 32 + c.lane])
// Whether this interaction, which has left `nf` wires as redirects, linked the
// wire `w`.  Past the wires it remembers the word tells: a linked wire's still
// holds the LOCK it was taken with, which nobody else touches any more; a
// redirect, what it resolves to (P_GONE) and a word freed by whoever followed
// it are all something else.  Asked while the node's other word is this
// lane's: nobody reclaims the node, so the word cannot be another's.  (Always
// reading the word: a tree sum of 2^18 leaves 3.39 -> 3.47 ms.)
HVM_INL bool was_linked(const Ctx c, ull w, unsigned nf) {
  for (unsigned k = 0; k < unsigned(FAILS) && k < nf; k++)
    if (FAIL(k) == w) return false;
  return nf <= unsigned(FAILS) || hload(c, w) == P_LOCK;
}
// The later wire `w` of a pair was linked, and some wire of this interaction
// was left as a redirect.
HVM_COLD void pair_done(const Ctx c, ull w, unsigned nf) {
  if (was_linked(c, w ^ 8, nf)) recycle(c, w & ~8ull);
  else half_free(c, w);  // freed alone; whoever follows the redirect frees the other half
}
HVM_INL void wire_done(const Ctx c, const Exec& x, ull w, bool last) {
  if (last) {
    if (x.nf == 0) recycle(c, w & ~8ull);
    else pair_done(c, w, x.nf);
  }
}
// The CAS on wire `w`'s other end lost: leave a redirect in `w`, the
// interaction's `nf`-th.  When the earlier wire of its pair was linked, that
// one's word is freed alone.
HVM_COLD void wire_failed(const Ctx c, ull xp, ull w, ull yp, unsigned nf, bool last) {
  const bool linked = last && was_linked(c, w ^ 8, nf);
  if (nf < unsigned(FAILS)) FAIL(nf) = w;
  half_link_failed(c, xp, w, yp);
  if (linked) half_free(c, w ^ 8);
}
#undef FAIL

// Instruction `I` on registers R[i * S].
template <unsigned S> HVM_INL void exec_ins(const Ctx c, Exec& x, const DevInstr I, ull* R) {
  const unsigned kind = I.k;
  if (kind == I_CONST) {
    R[I.a * S] = I.port;
    return;
  }
  if (kind == I_WIRES) {
    ull n = alloc_cold(c);
    x.nodes++;
    R[I.a * S] = pvar(n);
    R[I.b * S] = n;
    R[I.c * S] = pvar(n ^ 8);
    R[I.d * S] = n ^ 8;
    return;
  }
  if (kind == I_CAPTURE) return capture(c, I.port, R[I.a * S]);
  if (kind >= I_CALL) {  // register b (I_CALL, I_FCTR: none) and, but for I_FLINK, register a hold ports of own nodes
    if (kind <= I_FCTR) {
      const ull n = alloc(c);
      const ull p = mkport(T_CTR, I.lab, n);
      x.nodes++;
      if (kind == I_CALL) push(c, I.port, p);
      else st_gpu(g_P.heap + (paddr(R[I.a * S]) >> 3), p);
      R[I.b * S] = pvar(n);
      R[I.c * S] = pvar(n ^ 8);
      return;
    }
    const ull A = R[I.a * S];
    if (kind == I_FCONST) {
      st_gpu(g_P.heap + (paddr(A) >> 3), I.port);
      return;
    }
    const ull B = R[I.b * S];
    ull ap = A;
    if (ptag(A) == T_RED) {
      ap = atom_exch(g_P.heap + (A >> 3), P_LOCK);
      if (ap == P_LOCK) ap = relock(c.net, A);
      ull ra = pvar(A);
      if (ptag(ap) == T_VAR) ra = atom_cas(heap_at(c.net, paddr(ap)), pvar(A), B);
      st_gpu(g_P.heap + (paddr(B) >> 3), ap);
      if (ra == pvar(A)) wire_done(c, x, A, (I.d & INS_A_LAST) != 0);
      else wire_failed(c, ap, A, B, x.nf++, (I.d & INS_A_LAST) != 0);
      return;
    }
    if (ptag(A) == T_VAR) st_gpu(g_P.heap + (paddr(A) >> 3), B);
    st_gpu(g_P.heap + (paddr(B) >> 3), A);
    return;
  }
  // take
  const bool isl = kind == I_LINK;
  const ull A = R[I.a * S];
  const ull B = isl || kind == I_OPRED ? R[I.b * S] : I.port;
  const bool aw = ptag(A) == T_RED, bw = isl && ptag(B) == T_RED;
  ull ap = A, bp = B;
  // (wires hold checked addresses: a constructor match checks its node's)
  if (aw) ap = atom_exch(g_P.heap + (A >> 3), P_LOCK);
  if (bw) bp = atom_exch(g_P.heap + (B >> 3), P_LOCK);
  if (aw && ap == P_LOCK) ap = relock(c.net, A);
  if (bw && bp == P_LOCK) bp = relock(c.net, B);
  // rule
  bool link = true;
  if (kind >= I_CTR) {
    const unsigned t = ptag(ap);
    const bool num = t == T_NUM, match = kind == I_CTR && t == T_CTR && plab(ap) == I.lab;
    const bool era = ap == P_ERA && kind != I_CTR && kind != I_OPRED;
    ull n = 0, o1, o2;
    // (an operator's result on numbers needs no node, nor does an erased one)
    const bool fast = match || era || (num && (kind == I_OPNUM || kind == I_OPRED));
    if (!fast) {
      n = alloc(c);
      x.nodes++;
    }
    o1 = pvar(n);
    o2 = pvar(n ^ 8);
    link = !fast;
    if (kind == I_CTR) {
      if (match) {
        x.anni++;
        o1 = paddr(ap);  // Trg::wire
        if (o1 >= g_P.heap_bytes) {
          run_fail_here(HVM64_ERR_BAD_ADDR);
          o1 = 0;
        }
        o2 = o1 ^ 8;
      }
      bp = mkport(T_CTR, I.lab, n);
    } else if (kind == I_SWITCH) {
      bp = mkport(T_SWITCH, 0, n);
      if (num) {
        x.oper++;
        link = false;
        const uint32_t v = uint32_t(ap);
        const uint32_t k = num_tag(v) == NT_U24 ? num_payload(v) : 0;
        o1 = mkport(T_CTR, 0, n);
        // The arms' node may be matched by the next instruction, so the
        // word behind the result is filled now: with a wire of a node of its
        // own (node.rs:176-182), whose other word counts as consumed.
        ull tgt = n, w = alloc_cold(c);
        x.nodes++;
        if (k == 0) {
          st_gpu(g_P.heap + ((n ^ 8) >> 3), P_ERA);
        } else {
          ull n2 = alloc_cold(c);
          x.nodes++;
          st_gpu(g_P.heap + (n >> 3), P_ERA);
          st_gpu(g_P.heap + ((n ^ 8) >> 3), mkport(T_CTR, 0, n2));
          st_gpu(g_P.heap + (n2 >> 3), ull(num_u24(k - 1)));
          tgt = n2 ^ 8;
        }
        st_gpu(g_P.heap + (tgt >> 3), pvar(w));
        st_gpu(g_P.heap + (w >> 3), pvar(tgt));
        o2 = w;
      } else if (era) {
        x.eras++;
        o1 = o2 = P_ERA;
      }
    } else if (kind == I_OP) {
      bp = mkport(T_OP, I.op, n);
      if (num) {
        link = false;
        st_gpu(g_P.heap + (n >> 3), ull(num_unary(I.op, uint32_t(ap))));
        o1 = mkport(T_OP, NT_SYM, n);
      } else if (era) {
        o1 = o2 = P_ERA;
      }
    } else {  // I_OPNUM: operator and right operand in the instruction; I_OPRED: number and operator in B
      const bool red = kind == I_OPRED;
      const uint32_t op = red ? uint32_t(B >> 32) : I.op;
      if (num) {
        x.oper++;
        o2 = red ? binary_op(c.net, uint32_t(B), op, uint32_t(ap)) : binary_op(c.net, uint32_t(ap), op, uint32_t(I.port));
      } else if (era) {
        o2 = P_ERA;
      } else {
        bp = mkport(T_OP, red ? unsigned(NT_SYM) : op, n);
        st_gpu(g_P.heap + (n >> 3), red ? ull(num_unary(op, uint32_t(B))) : ull(uint32_t(I.port)));
      }
    }
    if (kind < I_OPNUM || kind == I_SWITCH) R[I.b * S] = o1;
    R[I.c * S] = o2;
  }
  const bool alast = (I.d & INS_A_LAST) != 0, blast = (I.d & INS_B_LAST) != 0;
  // link
  const bool both = principal(ap) && principal(bp);
  const bool acas = link && aw && !both && ptag(ap) == T_VAR, bcas = link && bw && !both && ptag(bp) == T_VAR;
  ull ra = pvar(A), rb = pvar(B);
  if (acas) ra = atom_cas(heap_at(c.net, paddr(ap)), pvar(A), bp);
  if (bcas) rb = atom_cas(heap_at(c.net, paddr(bp)), pvar(B), ap);
  if (link) {
    if (both) {
      if (skippable(ap) && skippable(bp)) x.eras++;
      else push(c, ap, bp);
    } else {
      // ports that are not behind wires name words of nodes this lane made
      if (!aw && ptag(ap) == T_VAR) st_gpu(g_P.heap + (paddr(ap) >> 3), bp);
      if (!bw && ptag(bp) == T_VAR) st_gpu(g_P.heap + (paddr(bp) >> 3), ap);
    }
  }
  if (aw) {
    if (ra == pvar(A)) wire_done(c, x, A, alast);
    else wire_failed(c, ap, A, bp, x.nf++, alast);
  }
  if (bw) {
    if (rb == pvar(B)) wire_done(c, x, B, blast);
    else wire_failed(c, bp, B, ap, x.nf++, blast);
  }
}
// The counters of an interaction that ran instructions.
HVM_INL void exec_counts(const Ctx c, const Exec& x, bool def, unsigned links) {
  if (x.anni) count(c, RW_ANNI, x.anni);
  if (x.oper) count(c, RW_OPER, x.oper);
  if (x.eras) count(c, RW_ERAS, x.eras);
  if (def) {
    count(c, EX_DNODES, x.nodes);
    count(c, EX_DLINKS, links);
  }
}
template <unsigned S> HVM_INL void exec_def(const Ctx c, const DevDef& d, ull t0, ull* R) {
  Exec x;
  R[0] = t0;
  const DevInstr* ins = g_P.instrs + d.ins_off;
  for (unsigned k = 0; k < d.ins_len; k++) exec_ins<S>(c, x, ins[k], R);
  exec_counts(c, x, true, d.links);
}
// The instructions of Def `id` past those a step stages, for one lane.
HVM_COLD unsigned exec_rest(const Ctx c, unsigned nf, unsigned id, ull* R) {
  Exec x;
  x.nf = nf;
  const DevInstr* ins = g_P.instrs + g_P.defs[id].ins_off;
  const unsigned len = g_P.defs[id].ins_len;
  for (unsigned k = ICACHE; k < len; k++) exec_ins<32>(c, x, ins[k], R);
  exec_counts(c, x, true, 0);
  return x.nf;
}
// A Def call outside a step's shared instruction stream, or one that needs
// more registers than the warp's shared memory holds for a lane.
HVM_COLD void exec_large(const Ctx c, const DevDef& d, ull t0) {
  if (d.nregs <= LOCAL_REGS) {
    ull R[LOCAL_REGS];
    return exec_def<1>(c, d, t0, R);
  }
  // (the reference grows its register scratch to any Def, runtime/src/def.rs:221-223)
  if (!c.W->bigregs || d.nregs > MAX_REGS) return run_fail(c.net, HVM64_ERR_BAD_INPUT, d.nregs);
  exec_def<32>(c, d, t0, c.W->bigregs + c.lane);
}
// A compiled build (hvm64 compile) includes the Book's Defs as functions;
// they run when the loaded Book is the one they were generated from.
#ifdef HVM_GEN_INCLUDE
#include HVM_GEN_INCLUDE
HVM_COLD bool gen_run(const Ctx c, unsigned id, ull t0) {
  unsigned before = LS(allocs);
  bool done = gen_call(c, id, t0);
  count(c, EX_DNODES, LS(allocs) - before);
  return done;
}
#endif
HVM_COLD void run_def(const Ctx c, unsigned id, ull t0) {
  if (id >= g_P.ndefs) return run_fail(c.net, HVM64_ERR_BAD_INPUT, id);
#ifdef HVM_GEN_INCLUDE
  if (g_P.gen && gen_run(c, id, t0)) return;
#endif
  const DevDef d = g_P.defs[id];
  exec_large(c, d, t0);
}

// def.rs:30-37 (LabSet::has); the expansion agent's set is LabSet::ALL.
HVM_INL bool def_has(const Ctx c, ull ref, unsigned lab) {
  if (ref & X_BIT) return lab < 0xFFFF;
  unsigned id = unsigned((paddr(ref) >> 3) - 1);
  if (id >= g_P.ndefs) {
    run_fail(c.net, HVM64_ERR_BAD_INPUT, ref);
    return true;
  }
  const DevDef& d = g_P.defs[id];
  if (lab >= d.min_safe) return false;
  unsigned w = lab >> 6;
  if (w >= d.lab_len) return false;
  return (g_P.labbits[d.lab_off + w] >> (lab & 63)) & 1;
}

// ---- expansion agent (runtime/src/net.rs:63-108) ----------------------------
// An agent is a Ref port with X_BIT whose address names a heap word holding
// its output port (the reference boxes an `ExpandDef { out }`).
HVM_COLD ull new_expand(const Ctx c, ull out) {
  ull w = alloc(c);
  half_free(c, w ^ 8);
  hstore(c, w, out);
  return mkport(T_REF, 0xFFFF, X_BIT | w);
}
HVM_COLD ull take_expand(const Ctx c, ull port) {
  ull w = paddr(port) & ~X_BIT;
  unsigned it = 0;
  ull out;
  while ((out = hload(c, w)) == P_LOCK)
    if (!run_spin(c.net, it)) break;
  half_free(c, w);
  return out;
}
HVM_COLD void expand_call(const Ctx c, ull self, ull port) {
  if (ptag(port) == T_REF && port != P_ERA) {
    if (port & X_BIT) {
      ull a = take_expand(c, self), b = take_expand(c, port);
      return link_port_port(c, a, b);
    }
    // (what call() does for a nilary argument; calling it would make the
    // call graph recursive, and its stack depth unknown to the compiler)
    count(c, RW_DREF);
    return run_def(c, unsigned((paddr(port) >> 3) - 1), self);
  }
  ull out = take_expand(c, self);
  unsigned t = ptag(port);
  if (t == T_RED) return run_fail(c.net, HVM64_ERR_BAD_PAIR, port);
  if (t == T_REF || t == T_NUM || t == T_VAR) return link_port_port(c, out, port);
  ull o1 = paddr(port);
  ull n = alloc(c);
  link_port_port(c, out, mkport(t, plab(port), n));
  link_wire_port(c, o1, new_expand(c, pvar(n)));
  link_wire_port(c, o1 ^ 8, new_expand(c, pvar(n ^ 8)));
}
// net.rs:65-69
HVM_COLD ull expand(const Ctx c, ull root) {
  ull a = alloc(c);
  half_free(c, a ^ 8);
  link_wire_port(c, root, new_expand(c, pvar(a)));
  return a;
}
// def.rs:177-189
HVM_COLD void call(const Ctx c, ull port, ull trg) {
  if (ptag(trg) == T_CTR && !def_has(c, port, plab(trg))) return comm02(c, port, trg);
  count(c, RW_DREF);
  if (port & X_BIT) return expand_call(c, port, trg);
  run_def(c, unsigned((paddr(port) >> 3) - 1), trg);
}

// ---- interact.rs:6-44 ----------------------------------------------------------
// The pairs no instruction list covers: a nilary pair, a call whose argument
// is nilary, the expansion agent, and pairs without a rule.
HVM_COLD void interact_other(const Ctx c, ull a, ull b) {
  unsigned at = ptag(a), bt = ptag(b);
  if (at <= T_VAR || bt <= T_VAR) return run_fail(c.net, HVM64_ERR_BAD_PAIR, a);
  bool an = at == T_REF || at == T_NUM, bn = bt == T_REF || bt == T_NUM;
  if (at == T_REF && bn && !skippable(a)) return call(c, a, b);
  if (an && bt == T_REF && !skippable(b)) return call(c, b, a);
  if (an && bn) return count(c, RW_ERAS);
  if (at == T_REF && bt == T_CTR && plab(b) >= plab(a)) return comm02(c, a, b);
  if (bt == T_REF && at == T_CTR && plab(a) >= plab(b)) return comm02(c, b, a);
  if (at == T_REF) return call(c, a, b);
  if (bt == T_REF) return call(c, b, a);
  run_fail(c.net, HVM64_ERR_BAD_PAIR, a);
}

// Sets up registers R[i * S] for redex (a, b) and counts its rule.  Returns the
// RULES list to run (offset | length << 8), or one of these.
enum : unsigned { RUN_DEF = 1u << 16, RUN_OTHER = 2u << 16 };
template <unsigned S> HVM_INL unsigned classify(const Ctx c, Exec& x, ull a, ull b, ull* R, unsigned& id) {
  // by tag: Ref < Num < Op < Switch < Ctr
  if (ptag(a) > ptag(b)) {
    ull t = a;
    a = b;
    b = t;
  }
  const unsigned at = ptag(a), bt = ptag(b);
  // nilary pairs, pairs without a rule, expansion agents
  if (bt <= T_NUM || at <= T_VAR || at == 4 || (at == T_OP && bt == T_SWITCH) ||
      (at == T_SWITCH && bt == T_CTR && plab(b) == 0) || is_expand(a))
    return RUN_OTHER;
  ull b1 = paddr(b);
  if (b1 >= g_P.heap_bytes) {
    run_fail_here(HVM64_ERR_BAD_ADDR);
    b1 = 0;
  }
  if (at == T_REF && a != P_ERA) {  // def.rs:177-189
    if (bt != T_CTR || (plab(b) < plab(a) && def_has(c, a, plab(b)))) {
      id = unsigned((paddr(a) >> 3) - 1);
      count(c, RW_DREF);
      R[0] = b;
      return RUN_DEF;
    }
  }
  R[0] = b1;
  R[S] = b1 ^ 8;
  if (at == T_REF || (at == T_NUM && bt == T_CTR)) {  // comm02, interact.rs:162-168
    count(c, RW_COMM);
    R[2 * S] = R[3 * S] = a;
    return RULE_LINK2 | RULE_LINK2_LEN << 8;
  }
  if (at == T_NUM) {
    if (bt == T_OP) {  // op_num, interact.rs:251-270
      R[2 * S] = ull(uint32_t(a)) | ull(plab(b)) << 32;
      return RULE_OP | RULE_OP_LEN << 8;
    }
    // switch_num, interact.rs:201-223
    x.oper++;
    const uint32_t num = uint32_t(a);
    const uint32_t n = num_tag(num) == NT_U24 ? num_payload(num) : 0;
    ull y = alloc_cold(c);
    R[2 * S] = mkport(T_CTR, 0, y);
    if (n == 0) {
      st_gpu(g_P.heap + ((y ^ 8) >> 3), P_ERA);
      R[3 * S] = pvar(y);
    } else {
      ull z = alloc_cold(c);
      st_gpu(g_P.heap + (y >> 3), P_ERA);
      st_gpu(g_P.heap + ((y ^ 8) >> 3), mkport(T_CTR, 0, z));
      st_gpu(g_P.heap + (z >> 3), ull(num_u24(n - 1)));
      R[3 * S] = pvar(z ^ 8);
    }
    return RULE_LINK2 | RULE_LINK2_LEN << 8;
  }
  ull a1 = paddr(a);
  if (a1 >= g_P.heap_bytes) {
    run_fail_here(HVM64_ERR_BAD_ADDR);
    a1 = 0;
  }
  R[2 * S] = a1;
  R[3 * S] = a1 ^ 8;
  if (at == bt && (at != T_CTR || plab(a) == plab(b))) {  // anni2, interact.rs:72-79
    x.anni++;
    return RULE_LINK2 | RULE_LINK2_LEN << 8;
  }
  // comm22, interact.rs:118-141
  count(c, RW_COMM);
  count(c, EX_COMM22);
  ull n[4];
  for (int k = 0; k < 4; k++) n[k] = alloc_cold(c);  // two copies of a, two of b
  st_gpu(g_P.heap + (n[0] >> 3), pvar(n[2]));
  st_gpu(g_P.heap + (n[2] >> 3), pvar(n[0]));
  st_gpu(g_P.heap + ((n[0] ^ 8) >> 3), pvar(n[3]));
  st_gpu(g_P.heap + (n[3] >> 3), pvar(n[0] ^ 8));
  st_gpu(g_P.heap + (n[1] >> 3), pvar(n[2] ^ 8));
  st_gpu(g_P.heap + ((n[2] ^ 8) >> 3), pvar(n[1]));
  st_gpu(g_P.heap + ((n[1] ^ 8) >> 3), pvar(n[3] ^ 8));
  st_gpu(g_P.heap + ((n[3] ^ 8) >> 3), pvar(n[1] ^ 8));
  // b's wires get copies of a, a's wires copies of b
  R[4 * S] = mkport(at, plab(a), n[0]);
  R[5 * S] = mkport(at, plab(a), n[1]);
  R[6 * S] = mkport(bt, plab(b), n[2]);
  R[7 * S] = mkport(bt, plab(b), n[3]);
  return RULE_LINK4 | RULE_LINK4_LEN << 8;
}
static_assert(SMALL_REGS >= 8, "comm22's registers");

// One interaction of one lane (the reducer's warps run the same steps with
// their instructions staged, see reduce_kernel).
HVM_COLD void interact(const Ctx c, ull a, ull b) {
  Exec x;
  ull* R = c.W->regs + c.lane;
  unsigned id = 0, p = classify<32>(c, x, a, b, R, id);
  if (p == RUN_OTHER) return interact_other(c, a, b);
  if (p == RUN_DEF) return run_def(c, id, R[0]);
  for (unsigned k = 0; k < p >> 8; k++) exec_ins<32>(c, x, RULES[(p & 0xFF) + k], R);
  exec_counts(c, x, false, 0);
}

// ---- normal-form gather (device-side readback) -------------------------------
// Walks net `net`'s normal form from word `root` the way host readback does
// (host/src/readback.rs:23-87): the root word, both words of every node it
// reaches, each redirect chain a Var goes through.  Writes the first `cap`
// (address, word) pairs to `out` and returns how many there are; `stk` (scap
// entries) is the depth-first stack.  *deep is set when the stack overflowed
// (the count is then incomplete).  A walk of more than `limit` pairs stops once
// it has passed GATHER_SHARE subtrees it still has to come back to, and sets
// *stopped: a walk with fewer (a list's) has nothing to share.
constexpr unsigned GATHER_SHARE = 4;
HVM_COLD unsigned gather_walk(unsigned net, ull root, ull* out, unsigned cap, ull* stk,
                                             unsigned scap, bool* deep, unsigned limit = ~0u,
                                             bool* stopped = nullptr) {
  const ull hb = g_P.heap_bytes;
  unsigned sp = 0, n = 0;
  auto emit = [&](ull w, ull v) {
    if (n < cap) {
      out[2 * n] = w;
      out[2 * n + 1] = v;
    }
    n++;
  };
  auto live = [&](ull p) {
    ull a = p & A_MASK;
    return (p >> 48) == 0 && a != 0 && a < hb;
  };
  stk[sp++] = root;
  while (sp) {
    if (n > limit && sp >= GATHER_SHARE) {
      *stopped = true;
      break;
    }
    ull w = stk[--sp];
    ull v = ld_gpu(heap_at(net, w));
    emit(w, v);
    unsigned t = unsigned(v & 7);
    if (t == T_VAR || t == T_RED) {
      if (live(v)) {
        ull e = paddr(v);
        for (unsigned g = 0; g < (1u << 20); g++) {
          ull x = ld_gpu(heap_at(net, e));
          emit(e, x);
          if ((x & 7) != T_RED || !live(x)) break;
          e = paddr(x);
        }
      }
    } else if (t == T_OP || t == T_CTR || t == T_SWITCH) {
      if (sp + 2 > scap) {
        *deep = true;
        break;
      }
      ull a = paddr(v);
      stk[sp++] = a ^ 8;
      stk[sp++] = a;
    }
  }
  return n;
}

// A normal form split for a parallel gather.  A single walk is a chain of
// dependent loads, so one thread first expands the top of the tree breadth
// first (at most GTOP words, until a level holds 32 items or more); the items
// left at the edge, and every word that starts a redirect chain, become
// subtrees that other threads walk with gather_walk.  Every subtree's pairs
// form one contiguous run of gather_walk's depth-first order, so sizes summed
// bottom-up over the expanded top give every run's offset.
constexpr unsigned GTOP = 512, GTASKS = 256;
enum : unsigned char { GATHER_LEAF = 0, GATHER_NODE = 1, GATHER_SUB = 2 };
struct GatherTop {
  ull* w;              // the item's word address
  ull* v;              // its word (leaf and node items)
  ull* sz;             // size in pairs, then (gather_place) offset
  unsigned* ref;       // node: index of its first child (the second follows); subtree: its number
  unsigned char* kind;
  unsigned nt, nk;     // items, subtrees
};
HVM_DEV void gather_top(unsigned net, ull root, GatherTop& T) {
  const ull hb = g_P.heap_bytes;
  auto live = [&](ull p) {
    ull a = p & A_MASK;
    return (p >> 48) == 0 && a != 0 && a < hb;
  };
  unsigned nt = 1, nk = 0, lo = 0, hi = 1, depth = 0;
  T.w[0] = root;
  while (lo < hi) {
    const unsigned width = hi - lo;
    // (expanding a level adds at most `width` chain subtrees and 2 * width
    // items to the next level, which may all become subtrees: checked here so
    // that the numbers of items and subtrees stay within the arrays)
    if (width >= 32u || nt + 2 * width > GTOP || nk + 3 * width > GTASKS || depth >= 48) {
      for (unsigned k = lo; k < hi; k++) {  // the edge: subtrees
        T.kind[k] = GATHER_SUB;
        T.ref[k] = nk++;
      }
      break;
    }
    for (unsigned k = lo; k < hi; k++) {
      ull v = ld_gpu(heap_at(net, T.w[k]));
      T.v[k] = v;
      unsigned t = unsigned(v & 7);
      if (t == T_OP || t == T_CTR || t == T_SWITCH) {
        T.kind[k] = GATHER_NODE;
        T.ref[k] = nt;
        T.w[nt++] = paddr(v);
        T.w[nt++] = paddr(v) ^ 8;
      } else if ((t == T_VAR || t == T_RED) && live(v)) {
        T.kind[k] = GATHER_SUB;  // a redirect chain: walked as a subtree
        T.ref[k] = nk++;
      } else {
        T.kind[k] = GATHER_LEAF;
      }
    }
    lo = hi;
    hi = nt;
    depth++;
  }
  T.nt = nt;
  T.nk = nk;
}
// Sizes bottom-up from the subtrees' counts (tc, by subtree number); returns
// the whole walk's pair count.  (Children follow their parent in T.)
HVM_DEV ull gather_sizes(GatherTop& T, const unsigned* tc) {
  for (unsigned k = T.nt; k-- > 0;)
    T.sz[k] = T.kind[k] == GATHER_LEAF ? 1
              : T.kind[k] == GATHER_SUB ? ull(tc[T.ref[k]])
                                        : 1 + T.sz[T.ref[k]] + T.sz[T.ref[k] + 1];
  return T.sz[0];
}
// After gather_sizes: turns sizes into offsets (a node reads its first child's
// size before overwriting it with the child's offset) and writes the top's
// own words at theirs; the subtrees then go at T.sz[k].
HVM_DEV void gather_place(GatherTop& T, const unsigned* tc, ull* dst) {
  (void)tc;
  T.sz[0] = 0;
  for (unsigned k = 0; k < T.nt; k++) {
    const ull at = T.sz[k];
    if (T.kind[k] == GATHER_SUB) continue;
    dst[2 * at] = T.w[k];
    dst[2 * at + 1] = T.v[k];
    if (T.kind[k] == GATHER_NODE) {
      unsigned c = T.ref[k];
      ull s0 = T.sz[c];
      T.sz[c] = at + 1;
      T.sz[c + 1] = at + 1 + s0;
    }
  }
}

#undef LS
#undef FW

}  // namespace dev
}  // namespace hvm
