// Host build of the synchronisation protocols (CPU ranks over POSIX shared
// memory, C++ acquire/release atomics in place of the PTX ones): the epoch
// barrier and the pipelined double-tree all-reduce, with the same flag layout
// (tccl_b200.h), the same bounded waits and the same status words as the
// device kernels, plus switches that inject faults — a rank that never sends
// one signal, a rank that stalls, a rank that stops half way.  Failure handling
// is tested here, on the host, because a GPU must never be hung or faulted on
// purpose.  The reference has neither timeouts nor fault tests: all its spins
// are unbounded (triton_barrier.py:108-118).
#include <atomic>
#include <chrono>
#include <cstdint>
#include <cstring>
#include <thread>
#include <vector>

#include "../tccl_b200.h"

namespace {

using clk = std::chrono::steady_clock;

struct HostComm {
  int world, rank;
  uint32_t* flags[TCCL_MAX_WORLD];  // every rank's flag region (shared memory)
  uint32_t* local;                  // this rank's private words
  uint64_t timeout_ns;
};

inline std::atomic<uint32_t>& A(uint32_t* p) { return *reinterpret_cast<std::atomic<uint32_t>*>(p); }

void record_failure(const HostComm& c, int code, int block, int peer, int where, uint32_t seen, uint32_t want) {
  uint32_t* st = c.local + TCCL_LOCAL_STATUS;
  uint32_t expected = 0;
  if (A(st + TCCL_ST_CODE).compare_exchange_strong(expected, (uint32_t)code)) {
    st[TCCL_ST_BLOCK] = (uint32_t)block;
    st[TCCL_ST_PEER] = (uint32_t)peer;
    st[TCCL_ST_WHERE] = (uint32_t)where;
    st[TCCL_ST_SEEN] = seen;
    st[TCCL_ST_WANT] = want;
  }
  A(st + TCCL_ST_ABORT).store(1u, std::memory_order_release);
}
inline bool aborted(const HostComm& c) {
  return A(c.local + TCCL_LOCAL_STATUS + TCCL_ST_ABORT).load(std::memory_order_relaxed) != 0;
}

// same contract as the device wait_reach(): acquire-poll until the flag reaches `want`
// (wrap-around order), give up at the deadline or as soon as this rank has aborted
bool wait_reach(uint32_t* flag, uint32_t want, const HostComm& c, clk::time_point deadline, int block, int peer,
                int where) {
  uint32_t spins = 0;
  for (;;) {
    const uint32_t v = A(flag).load(std::memory_order_acquire);
    if ((int32_t)(v - want) >= 0) return true;
    if ((++spins & 63u) == 0u) {
      if (aborted(c)) return false;
      if (clk::now() > deadline) {
        record_failure(c, TCCL_TIMEOUT, block, peer, where, v, want);
        return false;
      }
      std::this_thread::yield();
    }
  }
}

struct Faults {
  int drop_signal_to;   // barrier: never signal this peer (-1 = none)
  int stall_ms;         // sleep this long before signalling
  int stop_after_chunk; // tree: stop taking part after this many chunks (-1 = never)
};

bool barrier(const HostComm& c, int bid, clk::time_point deadline, const Faults& f) {
  const uint32_t e = c.local[TCCL_LOCAL_EPOCH + bid] + 1u;
  if (f.stall_ms > 0) std::this_thread::sleep_for(std::chrono::milliseconds(f.stall_ms));
  for (int p = 0; p < c.world; ++p) {
    if (p == f.drop_signal_to) continue;  // injected fault: the signal is lost
    A(c.flags[p] + TCCL_FLAG_BAR + bid * TCCL_MAX_WORLD + c.rank).store(e, std::memory_order_release);
  }
  bool ok = true;
  for (int p = 0; p < c.world && ok; ++p)
    ok = wait_reach(c.flags[c.rank] + TCCL_FLAG_BAR + bid * TCCL_MAX_WORLD + p, e, c, deadline, bid, p, TCCL_W_BARRIER);
  c.local[TCCL_LOCAL_EPOCH + bid] = e;
  return ok;
}

uint32_t* up_flag(const HostComm& c, int rank, int tree, int k, int slot) {
  return c.flags[rank] + TCCL_FLAG_TREE_UP + ((tree * TCCL_TREE_MAX_CTAS + k) * 2 + slot);
}
uint32_t* down_flag(const HostComm& c, int rank, int tree, int k) {
  return c.flags[rank] + TCCL_FLAG_TREE_DOWN + (tree * TCCL_TREE_MAX_CTAS + k);
}
uint32_t* ack_flag(const HostComm& c, int rank, int tree, int k) {
  return c.flags[rank] + TCCL_FLAG_TREE_ACK + (tree * TCCL_TREE_MAX_CTAS + k);
}
uint32_t* dack_flag(const HostComm& c, int rank, int tree, int k, int slot) {
  return c.flags[rank] + TCCL_FLAG_TREE_DACK + ((tree * TCCL_TREE_MAX_CTAS + k) * 2 + slot);
}

struct TreeJob {
  const float* in;              // this rank's input (read by nobody else)
  float* buf[TCCL_MAX_WORLD];   // every rank's result buffer; parents store the sum into their children's
  float* ring[TCCL_MAX_WORLD];  // every rank's ring: [tree][child slot][chunk % depth][chunk elements]
  uint64_t numel, chunk;
  uint64_t ring_stride;         // elements per ring slot: fixed for the communicator, >= any chunk
  int parent[2], left[2], right[2], child_slot[2];
  bool pull_down;               // way down: children copy the sum out of their parent's buffer and acknowledge
  bool early_post;              // see tree_worker
};
constexpr int kDepth = TCCL_TREE_RING_DEPTH;

float* ring_slot(const TreeJob& j, int rank, int tree, int cslot, uint32_t seq) {
  return j.ring[rank] + ((size_t)((tree * 2 + cslot) * kDepth) + seq % kDepth) * j.ring_stride;
}

constexpr int kAhead = 4;      // slices between polling and posting, as in tree_allreduce.cu
constexpr int kDataWarps = 2;

// an mbarrier: an arrival count and a phase
struct Mbar {
  std::atomic<int> pending{0};
  std::atomic<uint32_t> phase{0};
  int count = 0;
  void init(int n) {
    count = n;
    pending.store(n, std::memory_order_relaxed);
    phase.store(0, std::memory_order_relaxed);
  }
  void arrive() {
    if (pending.fetch_sub(1, std::memory_order_acq_rel) == 1) {
      pending.store(count, std::memory_order_relaxed);
      phase.fetch_add(1, std::memory_order_release);
    }
  }
  // like mbarrier.try_wait.parity in a loop: returns once the phase with this parity has completed
  void wait(uint32_t parity) const {
    while ((phase.load(std::memory_order_acquire) & 1u) == parity) std::this_thread::yield();
  }
  // bounded form: false once `give_up` says so
  template <class F> bool wait(uint32_t parity, const F& give_up) const {
    while ((phase.load(std::memory_order_acquire) & 1u) == parity) {
      if (give_up()) return false;
      std::this_thread::yield();
    }
    return true;
  }
};

// One (tree, direction) worker = what one CTA does on the device (K = 1 slice): the protocol of tree_allreduce.cu with
// the same counters, running totals and ring reuse rule, and the same split inside the CTA — a polling warp that waits
// for the counters up to kAhead slices ahead of the data, data warps that only load, add and store, and a posting warp
// that raises the counters behind them — with the three rings of mbarriers that hand a slice over: `ready` (inputs
// there, destination free), `done` (every data warp has issued its stores), `sent` (counters raised).
// `early_post` is a mistake kept so that the sanitizer can be seen to catch it: the posting warp goes by the FIRST data
// warp that is done with a slice.
void tree_worker(const HostComm& c, const TreeJob& j, int tree, bool is_up, clk::time_point deadline, const Faults& f) {
  const int me = c.rank, parent = j.parent[tree], left = j.left[tree], right = j.right[tree];
  const int cslot = j.child_slot[tree];
  const uint64_t nchunks = (j.numel + j.chunk - 1) / j.chunk;
  const uint64_t mine = nchunks > (uint64_t)tree ? (nchunks - tree + 1) / 2 : 0;
  const int role = (is_up ? 0 : 2) + tree;
  uint32_t* seq_word = c.local + TCCL_LOCAL_TREE_SEQ + role * TCCL_TREE_MAX_CTAS;
  const uint32_t base = *seq_word;
  uint64_t slices = is_up || parent >= 0 ? mine : 0;  // the root has no way down
  bool stopped = false;                               // injected: this rank stops here
  if (f.stop_after_chunk >= 0 && slices > (uint64_t)f.stop_after_chunk) {
    slices = (uint64_t)f.stop_after_chunk;
    stopped = true;
  }
  Mbar ready[kAhead], done[kAhead], sent[kAhead];
  for (int i = 0; i < kAhead; ++i) {
    ready[i].init(1);
    done[i].init(j.early_post ? 1 : kDataWarps);
    sent[i].init(1);
  }
  std::atomic<int> abort_cta{0};
  const auto late = deadline + std::chrono::nanoseconds(c.timeout_ns / 4) + std::chrono::milliseconds(1);
  auto give_up = [&] { return abort_cta.load(std::memory_order_relaxed) != 0 || clk::now() > late; };
  auto fail = [&] { abort_cta.store(1, std::memory_order_relaxed); };

  auto post = [&] {
    for (uint64_t n = 0; n < slices; ++n) {
      const uint32_t g = base + (uint32_t)n;
      if (!done[n % kAhead].wait((uint32_t)(n / kAhead) & 1u, give_up)) return fail();
      if (is_up && parent >= 0) {
        A(up_flag(c, parent, tree, 0, cslot)).store(g + 1u, std::memory_order_release);
      } else {
        if (left >= 0) A(down_flag(c, left, tree, 0)).store(g + 1u, std::memory_order_release);
        if (right >= 0) A(down_flag(c, right, tree, 0)).store(g + 1u, std::memory_order_release);
      }
      if (is_up) {
        if (left >= 0) A(ack_flag(c, left, tree, 0)).store(g + 1u, std::memory_order_release);
        if (right >= 0) A(ack_flag(c, right, tree, 0)).store(g + 1u, std::memory_order_release);
      } else if (j.pull_down) {  // this slice of the parent's buffer is no longer needed
        A(dack_flag(c, parent, tree, 0, cslot)).store(g + 1u, std::memory_order_release);
      }
      sent[n % kAhead].arrive();
    }
  };
  auto poll = [&] {
    for (uint64_t n = 0; n < slices; ++n) {
      const uint32_t g = base + (uint32_t)n;
      if (n >= (uint64_t)kAhead && !sent[n % kAhead].wait((uint32_t)(n / kAhead - 1) & 1u, give_up)) return fail();
      if (is_up) {
        // the children's partials are in my ring; the slot to be filled at the parent is free
        if (left >= 0 && !wait_reach(up_flag(c, me, tree, 0, 0), g + 1u, c, deadline, tree, left, TCCL_W_TREE_UP)) return fail();
        if (right >= 0 && !wait_reach(up_flag(c, me, tree, 0, 1), g + 1u, c, deadline, tree, right, TCCL_W_TREE_UP)) return fail();
        if (parent >= 0 &&
            !wait_reach(ack_flag(c, me, tree, 0), g + 1u - (uint32_t)kDepth, c, deadline, tree, parent, TCCL_W_TREE_UP))
          return fail();
      } else if (!wait_reach(down_flag(c, me, tree, 0), g + 1u, c, deadline, 2 + tree, parent, TCCL_W_TREE_DOWN)) {
        return fail();
      }
      ready[n % kAhead].arrive();
    }
    if (j.pull_down && !is_up && mine && !stopped) {
      // the caller may overwrite this rank's buffer once the call returns: wait until the children have copied it
      const uint32_t want = base + (uint32_t)mine;
      if (left >= 0 && !wait_reach(dack_flag(c, me, tree, 0, 0), want, c, deadline, 2 + tree, left, TCCL_W_TREE_DOWN)) return fail();
      if (right >= 0 && !wait_reach(dack_flag(c, me, tree, 0, 1), want, c, deadline, 2 + tree, right, TCCL_W_TREE_DOWN)) return fail();
    }
  };
  auto data = [&](int warp) {
    for (uint64_t n = 0; n < slices; ++n) {
      const uint32_t g = base + (uint32_t)n;
      if (!ready[n % kAhead].wait((uint32_t)(n / kAhead) & 1u, give_up)) return fail();
      const uint64_t clo = (2 * n + tree) * j.chunk, chi = std::min(clo + j.chunk, j.numel);
      const uint64_t per = (chi - clo + kDataWarps - 1) / kDataWarps;  // the warps share the slice
      const uint64_t lo = std::min(clo + per * warp, chi), hi = std::min(lo + per, chi);
      if (is_up) {
        const float* lr = left >= 0 ? ring_slot(j, me, tree, 0, g) : nullptr;
        const float* rr = right >= 0 ? ring_slot(j, me, tree, 1, g) : nullptr;
        float* pr = parent >= 0 ? ring_slot(j, parent, tree, cslot, g) : nullptr;
        for (uint64_t i = lo; i < hi; ++i) {
          const float v = j.in[i] + (lr ? lr[i - clo] : 0.f) + (rr ? rr[i - clo] : 0.f);
          if (pr) {
            pr[i - clo] = v;
          } else {  // the root: the final value goes to its own and its children's result buffers
            j.buf[me][i] = v;
            if (!j.pull_down) {
              if (left >= 0) j.buf[left][i] = v;
              if (right >= 0) j.buf[right][i] = v;
            }
          }
        }
      } else if (j.pull_down) {
        std::memcpy(j.buf[me] + lo, j.buf[parent] + lo, (hi - lo) * sizeof(float));
      } else {
        if (left >= 0) std::memcpy(j.buf[left] + lo, j.buf[me] + lo, (hi - lo) * sizeof(float));
        if (right >= 0) std::memcpy(j.buf[right] + lo, j.buf[me] + lo, (hi - lo) * sizeof(float));
      }
      if (j.early_post && warp) continue;
      done[n % kAhead].arrive();
    }
  };
  std::vector<std::thread> th;
  th.emplace_back(post);
  th.emplace_back(poll);
  for (int w = 0; w < kDataWarps; ++w) th.emplace_back(data, w);
  for (auto& x : th) x.join();
  if (!stopped && !abort_cta.load()) *seq_word = base + (uint32_t)mine;
}

}  // namespace

extern "C" {

struct hp_comm {
  int32_t world, rank;
  uint64_t flags[TCCL_MAX_WORLD];
  uint64_t local;
  uint64_t timeout_ns;
};
struct hp_faults {
  int32_t drop_signal_to, stall_ms, stop_after_chunk;
};
struct hp_tree {
  uint64_t in;                    // this rank's input
  uint64_t buf[TCCL_MAX_WORLD];   // result buffers (the inputs themselves when reducing in place)
  uint64_t ring[TCCL_MAX_WORLD];  // 4 * TCCL_TREE_RING_DEPTH * ring_stride floats per rank
  uint64_t numel, chunk, ring_stride;
  int32_t parent[2], left[2], right[2], child_slot[2];
  int32_t pull_down;              // 1: children copy the sum out of their parent's buffer (the large-message form)
  int32_t early_post;             // 1: the mistake that tree_worker keeps
};

static HostComm to_comm(const hp_comm* h) {
  HostComm c;
  c.world = h->world;
  c.rank = h->rank;
  for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = reinterpret_cast<uint32_t*>(h->flags[p]);
  c.local = reinterpret_cast<uint32_t*>(h->local);
  c.timeout_ns = h->timeout_ns;
  return c;
}

// returns 1 on success, 0 if a wait gave up (see the status words)
int hp_barrier(const hp_comm* h, int bid, int rounds, const hp_faults* f) {
  HostComm c = to_comm(h);
  Faults ft{f ? f->drop_signal_to : -1, f ? f->stall_ms : 0, -1};
  const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
  for (int i = 0; i < rounds; ++i)
    if (!barrier(c, bid, deadline, ft)) return 0;
  return 1;
}

// pipelined double-tree all-reduce over float buffers in shared memory; like the kernel it has
// neither an entry nor an exit barrier (counters are running totals, the ring has a fixed layout)
int hp_tree_allreduce(const hp_comm* h, const hp_tree* t, const hp_faults* f) {
  HostComm c = to_comm(h);
  Faults ft{-1, f ? f->stall_ms : 0, f ? f->stop_after_chunk : -1};
  TreeJob j;
  j.in = reinterpret_cast<const float*>(t->in);
  for (int p = 0; p < TCCL_MAX_WORLD; ++p) {
    j.buf[p] = reinterpret_cast<float*>(t->buf[p]);
    j.ring[p] = reinterpret_cast<float*>(t->ring[p]);
  }
  j.numel = t->numel;
  j.chunk = t->chunk;
  j.ring_stride = t->ring_stride;
  j.pull_down = t->pull_down != 0;
  j.early_post = t->early_post != 0;
  if (j.chunk > j.ring_stride) return 0;
  for (int i = 0; i < 2; ++i) {
    j.parent[i] = t->parent[i];
    j.left[i] = t->left[i];
    j.right[i] = t->right[i];
    j.child_slot[i] = t->child_slot[i];
  }
  const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
  if (ft.stall_ms > 0) std::this_thread::sleep_for(std::chrono::milliseconds(ft.stall_ms));
  std::vector<std::thread> th;
  for (int tree = 0; tree < 2; ++tree)
    for (int up = 0; up < 2; ++up) th.emplace_back([&, tree, up] { tree_worker(c, j, tree, up != 0, deadline, ft); });
  for (auto& x : th) x.join();
  return !aborted(c) ? 1 : 0;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// In-process self-test: `world` ranks as threads of one process.  Built with
// -fsanitize=thread this checks that every plain (non-atomic) access of the data
// buffers is ordered by the release/acquire flag protocol — the race detector the
// GPU side cannot have.  Returns 0 on success, a positive code otherwise.
static int tree_selftest(int world, int numel, int chunk, int rounds, bool early_post) {
  if (world < 1 || world > TCCL_MAX_WORLD) return 100;
  constexpr int kCalls = 6;  // back to back, no barrier in between, alternating chunk sizes and forms of the way down
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> data(world, std::vector<float>(numel));
  std::vector<std::vector<float>> rings(world, std::vector<float>((size_t)4 * TCCL_TREE_RING_DEPTH * chunk, 0.f));
  std::atomic<int> bad{0};
  // neighbours: the same low-bit rule as parallel/tree.py
  auto nbr_a = [&](int N, int r, int* parent, int* left, int* right) {
    *parent = *left = *right = -1;
    if (N == 1) return;
    if (r == 0) {
      int top = 1;
      while (top * 2 <= N - 1) top *= 2;
      *left = top;
      return;
    }
    const int s = r & -r;
    int up = (r ^ s) | (s << 1);
    if (up >= N) up = r ^ s;
    *parent = up;
    if (s == 1) return;
    *left = r - (s >> 1);
    int step = s >> 1, rt = r + step;
    while (rt >= N && step > 1) {
      step >>= 1;
      rt = r + step;
    }
    *right = rt >= N ? -1 : rt;
  };
  auto nbr = [&](int N, int r, int tree, int* parent, int* left, int* right) {
    if (tree == 0) return nbr_a(N, r, parent, left, right);
    nbr_a(N, (r + 1) % N, parent, left, right);
    auto back = [&](int x) { return x < 0 ? -1 : (x - 1 + N) % N; };
    *parent = back(*parent);
    *left = back(*left);
    *right = back(*right);
  };
  std::vector<int> results(world, 0);
  std::vector<std::thread> ranks;
  for (int r = 0; r < world; ++r) {
    ranks.emplace_back([&, r] {
      hp_comm h{};
      h.world = world;
      h.rank = r;
      for (int p = 0; p < world; ++p) h.flags[p] = reinterpret_cast<uint64_t>(flags[p].data());
      h.local = reinterpret_cast<uint64_t>(local[r].data());
      h.timeout_ns = (early_post ? 1ull : 20ull) * 1000 * 1000 * 1000;  // the mistake may also end in a wait that runs out
      hp_faults none{-1, 0, -1};
      int ok = hp_barrier(&h, 1, rounds, &none);
      for (int call = 0; call < kCalls && ok; ++call) {
        // this rank's own data only: written here, read by its up workers, overwritten with the
        // sum by its parent (after this rank has contributed the chunk) — the in-place form
        for (int i = 0; i < numel; ++i) data[r][i] = (float)((r + 1) * ((i % 7) + 1) + call);
        hp_tree t{};
        t.in = reinterpret_cast<uint64_t>(data[r].data());
        for (int p = 0; p < world; ++p) {
          t.buf[p] = reinterpret_cast<uint64_t>(data[p].data());
          t.ring[p] = reinterpret_cast<uint64_t>(rings[p].data());
        }
        t.numel = (uint64_t)numel;
        t.chunk = (uint64_t)((call & 1) ? std::max(1, chunk / 2) : chunk);
        t.ring_stride = (uint64_t)chunk;
        t.early_post = early_post;
        t.pull_down = (call >> 1) & 1;  // push, push, pull, pull: both forms and the change between them
        for (int tr = 0; tr < 2; ++tr) {
          int parent, left, right;
          nbr(world, r, tr, &parent, &left, &right);
          t.parent[tr] = parent;
          t.left[tr] = left;
          t.right[tr] = right;
          t.child_slot[tr] = 0;
          if (parent >= 0) {
            int pp, pl, pr;
            nbr(world, parent, tr, &pp, &pl, &pr);
            t.child_slot[tr] = pl == r ? 0 : 1;
          }
        }
        ok = ok && hp_tree_allreduce(&h, &t, &none);
        const float tot = (float)(world * (world + 1) / 2);
        for (int i = 0; i < numel && ok; ++i)
          if (data[r][i] != tot * (float)((i % 7) + 1) + (float)(world * call)) bad.store(2);
      }
      results[r] = ok;
    });
  }
  for (auto& th : ranks) th.join();
  for (int r = 0; r < world; ++r)
    if (!results[r]) return 1;
  return bad.load();
}
extern "C" int hp_selftest_threads(int world, int numel, int chunk, int rounds) {
  return tree_selftest(world, numel, chunk, rounds, false);
}
// the posting warp of every CTA goes by the first data warp that is done: must be caught
extern "C" int hp_selftest_tree_early_post(int world, int numel, int chunk) {
  return tree_selftest(world, numel, chunk, 1, true);
}

// ---------------------------------------------------------------------------
// Model of the fused GEMM -> reduce-scatter flag protocol (gemm_rs.cu), ranks and
// CTAs as threads: entry barrier per CTA index; every "CTA" walks its tiles in owner
// order (own rows first), writes a partial into slot [src][tile] of the OWNER's
// staging area with plain stores and raises that tile's epoch flag one tile later
// (the deferred release of the copy-engine epilogue); the final phase shares the
// rank's tiles out over all CTAs, acquires the W flags of a tile and sums the slots;
// the last CTA of a rank to finish advances the epoch.  Two calls run back to back
// so that slot reuse across calls (protected by the entry barrier) is covered too.
// Under ThreadSanitizer this verifies that every plain slot access is ordered.
extern "C" int hp_selftest_gemm_rs(int world, int ctas, int tiles_per_owner, int calls) {
  if (world < 1 || world > TCCL_MAX_WORLD || ctas < 1 || ctas > 64 || tiles_per_owner > 64) return 100;
  constexpr int kElems = 16;  // one "tile" of the model
  const int tpo = tiles_per_owner;
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> stage(world, std::vector<float>((size_t)world * tpo * kElems, 0.f));
  std::vector<std::vector<float>> out(world, std::vector<float>((size_t)tpo * kElems, 0.f));
  std::atomic<int> bad{0};
  auto partial = [](int call, int src, int owner, int lt, int e) {
    return (float)((call + 1) * 1000 + src * 100 + owner * 10 + lt) + 0.25f * e;
  };
  for (int call = 0; call < calls; ++call) {
    std::vector<std::thread> th;
    for (int r = 0; r < world; ++r)
      for (int b = 0; b < ctas; ++b)
        th.emplace_back([&, r, b, call] {
          HostComm c;
          c.world = world;
          c.rank = r;
          for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = p < world ? flags[p].data() : nullptr;
          c.local = local[r].data();
          c.timeout_ns = 20ull * 1000 * 1000 * 1000;
          const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
          Faults none{-1, 0, -1};
          const uint32_t epoch = A(c.local + TCCL_LOCAL_TILE_EPOCH).load(std::memory_order_relaxed) + 1u;
          // per-CTA barrier row: the model keeps one epoch word per (rank, bid) like the device
          {
            // barrier() updates c.local[EPOCH + bid]; rows are private to this CTA index
            if (!barrier(c, b, deadline, none)) bad.store(1);
          }
          uint32_t* pending = nullptr;
          for (int t = b; t < world * tpo; t += ctas) {
            const int j = t / tpo, lt = t - j * tpo;
            const int owner = (r + j) % world;
            if (pending) {  // flush the previous tile's flag (its "copies" are complete)
              A(pending).store(epoch, std::memory_order_release);
              pending = nullptr;
            }
            float* slot = stage[owner].data() + ((size_t)r * tpo + lt) * kElems;
            for (int e = 0; e < kElems; ++e) slot[e] = partial(call, r, owner, lt, e);
            pending = c.flags[owner] + TCCL_FLAG_TILE + r * TCCL_MAX_TILES + lt;
          }
          if (pending) A(pending).store(epoch, std::memory_order_release);
          // final phase: tiles of this rank shared out over its CTAs
          for (int lt = b; lt < tpo; lt += ctas) {
            bool ok = true;
            for (int src = 0; src < world && ok; ++src)
              ok = wait_reach(c.flags[r] + TCCL_FLAG_TILE + src * TCCL_MAX_TILES + lt, epoch, c, deadline, b, src,
                              TCCL_W_TILE);
            if (!ok) {
              bad.store(2);
              return;
            }
            for (int e = 0; e < kElems; ++e) {
              float s = 0.f;
              for (int src = 0; src < world; ++src) s += stage[r][((size_t)src * tpo + lt) * kElems + e];
              out[r][(size_t)lt * kElems + e] = s;
            }
          }
          // the last CTA of the rank publishes the epoch for the next call
          const uint32_t done = A(c.local + TCCL_LOCAL_SCHED).fetch_add(1u, std::memory_order_acq_rel);
          if (done == (uint32_t)ctas - 1u) {
            A(c.local + TCCL_LOCAL_SCHED).store(0u, std::memory_order_relaxed);
            A(c.local + TCCL_LOCAL_TILE_EPOCH).store(epoch, std::memory_order_release);
          }
        });
    for (auto& x : th) x.join();  // = stream order: a rank's next kernel starts after this one ended
    if (bad.load()) return bad.load();
    for (int r = 0; r < world; ++r)
      for (int lt = 0; lt < tpo; ++lt)
        for (int e = 0; e < kElems; ++e) {
          float s = 0.f;
          for (int src = 0; src < world; ++src) s += partial(call, src, r, lt, e);
          if (out[r][(size_t)lt * kElems + e] != s) return 3;
        }
  }
  return 0;
}

// ---------------------------------------------------------------------------
// Model of the all-gather -> GEMM arrival protocol (ag_gemm.cu): `movers` threads per
// rank copy their share of every row tile of the rank's shard into slot [rank] of every
// rank's gathered buffer (plain stores), count themselves done per row tile, and the
// last one raises the row tile's epoch flag on every rank; `consumers` threads per rank
// wait for a remote row tile's flag before reading its rows.  Movers start with their
// own barrier row (the previous call's readers are done); the last thread of a rank to
// finish advances the epoch.
extern "C" int hp_selftest_ag(int world, int movers, int consumers, int row_tiles, int calls) {
  if (world < 1 || world > TCCL_MAX_WORLD || movers < 1 || movers > 32 || consumers < 1 || consumers > 32) return 100;
  constexpr int kRow = 24;  // elements per row tile in the model
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> full(world, std::vector<float>((size_t)world * row_tiles * kRow, 0.f));
  std::atomic<int> bad{0};
  auto val = [](int call, int src, int rt, int e) { return (float)(call * 10000 + src * 1000 + rt * 50 + e); };
  const int nthreads = movers + consumers;
  for (int call = 0; call < calls; ++call) {
    std::vector<std::thread> th;
    for (int r = 0; r < world; ++r)
      for (int b = 0; b < nthreads; ++b)
        th.emplace_back([&, r, b, call] {
          HostComm c;
          c.world = world;
          c.rank = r;
          for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = p < world ? flags[p].data() : nullptr;
          c.local = local[r].data();
          c.timeout_ns = 20ull * 1000 * 1000 * 1000;
          const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
          Faults none{-1, 0, -1};
          const uint32_t epoch = A(c.local + TCCL_LOCAL_TILE_EPOCH).load(std::memory_order_relaxed) + 1u;
          if (b < movers) {
            if (!barrier(c, b, deadline, none)) bad.store(1);
            for (int rt = 0; rt < row_tiles; ++rt) {
              for (int e = b; e < kRow; e += movers)
                for (int q = 0; q < world; ++q) full[q][((size_t)r * row_tiles + rt) * kRow + e] = val(call, r, rt, e);
              const uint32_t done = A(c.local + TCCL_LOCAL_AGCNT + rt).fetch_add(1u, std::memory_order_acq_rel);
              if (done == (uint32_t)movers - 1u) {
                A(c.local + TCCL_LOCAL_AGCNT + rt).store(0u, std::memory_order_relaxed);
                for (int q = 0; q < world; ++q)
                  A(c.flags[q] + TCCL_FLAG_AG + r * TCCL_MAX_ROW_TILES + rt).store(epoch, std::memory_order_release);
              }
            }
          } else {
            const int cb = b - movers;
            for (int t = cb; t < world * row_tiles; t += consumers) {
              const int src = t / row_tiles, rt = t - src * row_tiles;
              if (src != r &&
                  !wait_reach(c.flags[r] + TCCL_FLAG_AG + src * TCCL_MAX_ROW_TILES + rt, epoch, c, deadline, b, src,
                              TCCL_W_TILE)) {
                bad.store(2);
                return;
              }
              if (src == r) continue;  // own rows come straight from the shard
              for (int e = 0; e < kRow; ++e)
                if (full[r][((size_t)src * row_tiles + rt) * kRow + e] != val(call, src, rt, e)) bad.store(3);
            }
          }
          const uint32_t done = A(c.local + TCCL_LOCAL_SCHED).fetch_add(1u, std::memory_order_acq_rel);
          if (done == (uint32_t)nthreads - 1u) {
            A(c.local + TCCL_LOCAL_SCHED).store(0u, std::memory_order_relaxed);
            A(c.local + TCCL_LOCAL_TILE_EPOCH).store(epoch, std::memory_order_release);
          }
        });
    for (auto& x : th) x.join();
    if (bad.load()) return bad.load();
  }
  return 0;
}

// ---------------------------------------------------------------------------
// Model of the small-message push all-reduce (AllReduceOneShotPush): every rank stores its
// input into slot [half][rank] of every rank, ONE barrier, local sum, and no exit barrier.
// A rank is `kCtas` threads (the CTAs of its launch) that meet at a kernel boundary between
// calls, as kernels of one stream do; the ranks run free of each other, so a rank may be a
// call ahead of a peer.  Consecutive calls differ in message size and in grid.  All slot
// accesses are plain loads and stores: ThreadSanitizer checks that the bytes being
// overwritten are never still being read.
//   scheme 0 (the kernel): fixed slot layout — half h at h * region / 2, rank r's slot at
//            r * slot_elems — and the half taken from a per-rank count of completed push calls
//            that the last CTA of a launch advances.
//   scheme 1 (a broken variant kept to show that the check has teeth): slot size = message size
//            and the half = low bit of the CTA's own barrier epoch.  With mixed sizes and grids
//            a fast rank overwrites bytes a slow peer is still summing: a data race (and often
//            a wrong sum).
namespace {
struct KernelBoundary {  // sense-reversing barrier among the CTA threads of one rank
  std::atomic<int> count{0};
  std::atomic<int> sense{0};
  // `stop`: once it is non-zero (a check failed somewhere) nobody waits any more — a thread that has left its
  // call loop must not leave the others stuck here
  void arrive_and_wait(int n, int& my_sense, const std::atomic<int>* stop = nullptr) {
    my_sense ^= 1;
    if (count.fetch_add(1, std::memory_order_acq_rel) == n - 1) {
      count.store(0, std::memory_order_relaxed);
      sense.store(my_sense, std::memory_order_release);
    } else {
      while (sense.load(std::memory_order_acquire) != my_sense) {
        if (stop && stop->load(std::memory_order_relaxed)) return;
        std::this_thread::yield();
      }
    }
  }
};
}  // namespace

extern "C" int hp_selftest_push(int world, int calls, int scheme) {
  if (world < 1 || world > TCCL_MAX_WORLD) return 100;
  constexpr int kCtas = 4;
  constexpr int kSlotElems = 64;                 // capacity of one fixed slot
  static const int kSizes[3] = {64, 32, 8};      // message elements of call n: kSizes[n % 3] ...
  static const int kGrids[3] = {4, 2, 1};        // ... and its grid
  const size_t region = (size_t)2 * world * kSlotElems;
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> slots(world, std::vector<float>(region, 0.f));
  std::vector<KernelBoundary> boundary(world);
  std::atomic<int> bad{0};
  std::vector<std::thread> th;
  auto val = [](int call, int r, int i) { return (float)(call * 100 + r * 10 + i % 3); };
  for (int r = 0; r < world; ++r)
    for (int bid = 0; bid < kCtas; ++bid)
      th.emplace_back([&, r, bid] {
        HostComm c;
        c.world = world;
        c.rank = r;
        for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = p < world ? flags[p].data() : nullptr;
        c.local = local[r].data();
        c.timeout_ns = 20ull * 1000 * 1000 * 1000;
        Faults none{-1, 0, -1};
        int my_sense = 0;
        for (int call = 0; call < calls; ++call) {
          const int n = kSizes[call % 3], grid = kGrids[call % 3];
          if (bid < grid && !bad.load(std::memory_order_relaxed)) {
            const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
            size_t base, slot;
            uint32_t seq = 0;
            if (scheme == 0) {
              seq = A(c.local + TCCL_LOCAL_PUSH_SEQ).load(std::memory_order_relaxed);
              slot = kSlotElems;
              base = (size_t)(seq & 1u) * (region / 2);
            } else {
              const uint32_t e = c.local[TCCL_LOCAL_EPOCH + bid] + 1u;
              slot = (size_t)n;
              base = (size_t)(e & 1u) * world * slot;
            }
            const int lo = n * bid / grid, hi = n * (bid + 1) / grid;  // this CTA's slab
            for (int q = 0; q < world; ++q)
              for (int i = lo; i < hi; ++i) slots[q][base + (size_t)r * slot + i] = val(call, r, i);
            if (!barrier(c, bid, deadline, none)) {
              bad.store(1);
            } else {
              for (int i = lo; i < hi; ++i) {
                float s = 0.f, want = 0.f;
                for (int p = 0; p < world; ++p) {
                  s += slots[r][base + (size_t)p * slot + i];
                  want += val(call, p, i);
                }
                if (s != want) bad.store(2);
              }
              if (scheme == 0) {
                const uint32_t done = A(c.local + TCCL_LOCAL_PUSH_DONE).fetch_add(1u, std::memory_order_acq_rel);
                if (done == (uint32_t)grid - 1u) {
                  A(c.local + TCCL_LOCAL_PUSH_DONE).store(0u, std::memory_order_relaxed);
                  A(c.local + TCCL_LOCAL_PUSH_SEQ).store(seq + 1u, std::memory_order_relaxed);
                }
              }
            }
            if ((call & 3) == (r + bid) % 4) std::this_thread::yield();  // let ranks and CTAs drift apart
          }
          boundary[r].arrive_and_wait(kCtas, my_sense);  // the next kernel starts when this one is done
        }
      });
  for (auto& x : th) x.join();
  return bad.load();
}

// ---------------------------------------------------------------------------
// Model of the bulk-copy two-shot all-reduce (allreduce_bulk.cu).  Per rank and CTA: a loader, a
// few reducers and a storer around 3 input stages and 2 output stages guarded by mbarriers
// (modelled with an arrival count and a phase), and a COPY ENGINE thread that runs the bulk
// copies later than they are issued — a load arrives on the stage's barrier when its bytes have
// landed, a store group counts as "read" only once the engine has copied it — so a stage that is
// released or refilled too early shows up as a data race.  Ranks meet at the epoch barrier on
// entry and on exit; two calls run back to back, in place.
namespace {
struct CopyJob {
  float* dst;
  const float* src;
  size_t n;
  Mbar* arrive_on;  // loads: the stage's "full" barrier; stores: null
  int group;        // stores: bulk group number (-1 for loads)
};
struct CopyEngine {
  std::vector<CopyJob> jobs;             // written by the issuing threads under `lock`, read by the engine
  std::atomic<int> issued{0}, taken{0};
  std::atomic<int> groups_read{0};       // store groups whose source stage has been read
  std::atomic<bool> stop{false};
  std::atomic_flag lock = ATOMIC_FLAG_INIT;
  explicit CopyEngine(size_t cap) : jobs(cap) {}
  void submit(const CopyJob& j) {
    while (lock.test_and_set(std::memory_order_acquire)) std::this_thread::yield();
    jobs[(size_t)issued.load(std::memory_order_relaxed)] = j;
    issued.fetch_add(1, std::memory_order_release);
    lock.clear(std::memory_order_release);
  }
  void run() {
    for (;;) {
      const int t = taken.load(std::memory_order_relaxed);
      if (t < issued.load(std::memory_order_acquire)) {
        const CopyJob j = jobs[(size_t)t];
        std::memcpy(j.dst, j.src, j.n * sizeof(float));
        if (j.arrive_on) j.arrive_on->arrive();
        if (j.group >= 0) groups_read.store(j.group + 1, std::memory_order_release);
        taken.store(t + 1, std::memory_order_release);
      } else if (stop.load(std::memory_order_acquire)) {
        return;
      } else {
        std::this_thread::yield();
      }
    }
  }
};
}  // namespace

// `early_release` != 0 is the mistake the output stages guard against, kept so that the sanitizer can be seen to
// catch it: the storer frees a stage as soon as its copies are ISSUED instead of when they have read it.
extern "C" int hp_selftest_bulk(int world, int ctas, int chunk, int chunks_per_cta, int calls, int early_release) {
  if (world < 1 || world > TCCL_MAX_WORLD || ctas < 1 || ctas > 8) return 100;
  constexpr int kIn = 3, kOut = 2, kReducers = 3;
  const size_t per = (size_t)ctas * chunks_per_cta * chunk - (size_t)chunk / 3;  // a ragged last chunk
  const size_t numel = per * world;
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> data(world, std::vector<float>(numel));
  std::atomic<int> bad{0};
  std::vector<KernelBoundary> boundary(world);
  std::vector<std::thread> th;
  for (int r = 0; r < world; ++r)
    for (int bid = 0; bid < ctas; ++bid)
      th.emplace_back([&, r, bid] {
        // one "CTA": its shared memory, barriers and copy engine live here; its roles are threads
        HostComm c;
        c.world = world;
        c.rank = r;
        for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = p < world ? flags[p].data() : nullptr;
        c.local = local[r].data();
        c.timeout_ns = 60ull * 1000 * 1000 * 1000;
        Faults none{-1, 0, -1};
        std::vector<float> in_st((size_t)kIn * world * chunk), out_st((size_t)kOut * chunk);
        int my_sense = 0;
        for (int call = 0; call < calls; ++call) {
          if (bid == 0)  // the "host" of rank r fills its input between two kernels
            for (size_t i = 0; i < numel; ++i) data[r][i] = (float)((r + 1) * (int)(i % 5 + 1) + call);
          boundary[r].arrive_and_wait(ctas, my_sense);
          const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
          Mbar full_in[kIn], empty_in[kIn], full_out[kOut], empty_out[kOut];
          for (int s = 0; s < kIn; ++s) {
            full_in[s].init(world);  // one arrival per landed copy (the kernel counts bytes instead)
            empty_in[s].init(kReducers);
          }
          for (int s = 0; s < kOut; ++s) {
            full_out[s].init(kReducers);
            empty_out[s].init(1);
          }
          if (!barrier(c, bid, deadline, none)) bad.store(1);  // entry: every rank's input is written
          const size_t lo = per * r;
          const size_t nchunks = (per + chunk - 1) / chunk;
          CopyEngine eng((size_t)(2 * world) * (nchunks / ctas + 2));
          std::thread engine([&] { eng.run(); });
          std::thread loader([&] {
            uint32_t q = 0;
            for (size_t ci = bid; ci < nchunks; ci += ctas, ++q) {
              const int s = q % kIn;
              empty_in[s].wait(((q / kIn) & 1u) ^ 1u);
              const size_t v0 = lo + ci * chunk, cnt = std::min((size_t)chunk, lo + per - v0);
              for (int p = 0; p < world; ++p)
                eng.submit({in_st.data() + ((size_t)s * world + p) * chunk, data[p].data() + v0, cnt, &full_in[s], -1});
            }
          });
          std::vector<std::thread> reducers;
          for (int j = 0; j < kReducers; ++j)
            reducers.emplace_back([&, j] {
              uint32_t q = 0;
              for (size_t ci = bid; ci < nchunks; ci += ctas, ++q) {
                const int s = q % kIn, so = q % kOut;
                full_in[s].wait((q / kIn) & 1u);
                empty_out[so].wait(((q / kOut) & 1u) ^ 1u);
                const size_t v0 = lo + ci * chunk, cnt = std::min((size_t)chunk, lo + per - v0);
                for (size_t k = j; k < cnt; k += kReducers) {
                  float sum = 0.f;
                  for (int p = 0; p < world; ++p) sum += in_st[((size_t)s * world + p) * chunk + k];
                  out_st[(size_t)so * chunk + k] = sum;
                }
                full_out[so].arrive();
                empty_in[s].arrive();
              }
            });
          std::thread storer([&] {
            uint32_t q = 0;
            for (size_t ci = bid; ci < nchunks; ci += ctas, ++q) {
              const int so = q % kOut;
              full_out[so].wait((q / kOut) & 1u);
              const size_t v0 = lo + ci * chunk, cnt = std::min((size_t)chunk, lo + per - v0);
              for (int p = 0; p < world; ++p)  // one bulk group: the copies into every rank's destination
                eng.submit({data[p].data() + v0, out_st.data() + (size_t)so * chunk, cnt, nullptr,
                            p == world - 1 ? (int)q : -1});
              if (early_release) {
                empty_out[so].arrive();
              } else if (q >= 1) {  // cp.async.bulk.wait_group.read 1: the previous group has read its stage
                while (eng.groups_read.load(std::memory_order_acquire) < (int)q) std::this_thread::yield();
                empty_out[(q - 1) % kOut].arrive();
              }
            }
            // cp.async.bulk.wait_group 0: every copy this CTA issued has landed
            while (eng.taken.load(std::memory_order_acquire) < eng.issued.load(std::memory_order_acquire))
              std::this_thread::yield();
          });
          loader.join();
          for (auto& x : reducers) x.join();
          storer.join();
          eng.stop.store(true, std::memory_order_release);
          engine.join();
          if (!barrier(c, bid, deadline, none)) bad.store(1);  // exit: all results have landed everywhere
          boundary[r].arrive_and_wait(ctas, my_sense);
          if (bid == 0) {
            const float tot = (float)(world * (world + 1) / 2);
            for (size_t i = 0; i < numel; ++i)
              if (data[r][i] != tot * (float)(i % 5 + 1) + (float)(world * call)) bad.store(2);
          }
          boundary[r].arrive_and_wait(ctas, my_sense);
        }
      });
  for (auto& x : th) x.join();
  return bad.load();
}

// ---------------------------------------------------------------------------
// Model of the barrier-free all-gather -> GEMM on CTA pairs (ag_gemm_pair.cu).  Every CTA of a
// rank is a mover thread (the epilogue warps: stores its share of the rank's shard into the
// gathered buffer of the peers, in batches to all ranks or — `ring` — destination by destination,
// and the CTA that completes a batch raises the row tiles' flags) and a consumer thread (the
// producer warp: waits for a remote row tile's flag, then reads the rows from the LOCAL gathered
// buffer).  There is NO entry barrier: the gathered buffer has two halves that alternate on a
// per-rank count of completed calls, and the ranks run free of each other — a rank may be a call
// ahead of a peer — while the CTAs of one rank meet at a kernel boundary between calls, as kernels
// of one stream do.  All buffer accesses are plain: ThreadSanitizer checks the claim that a rank
// reaches call n+2 (and overwrites the half of call n) only after every peer has finished call n.
// `mode`: bit 0 = ring-ordered movers; bit 1 = ONE buffer instead of two halves and still no barrier —
// the mistake the halves are there to prevent, kept so that the sanitizer can be seen to catch it.
extern "C" int hp_selftest_ag_pair(int world, int ctas, int row_tiles, int calls, int mode) {
  if (world < 1 || world > TCCL_MAX_WORLD || ctas < 1 || ctas > 16 || row_tiles < 1 || row_tiles > 8) return 100;
  const int ring = mode & 1;
  const bool one_buffer = (mode & 2) != 0;
  constexpr int kRow = 24;
  const size_t half_elems = (size_t)world * row_tiles * kRow;
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> full(world, std::vector<float>(2 * half_elems, 0.f));
  std::vector<KernelBoundary> boundary(world);
  std::atomic<int> bad{0};
  auto val = [](int call, int src, int rt, int e) { return (float)(call * 10000 + src * 1000 + rt * 50 + e); };
  std::vector<std::thread> th;
  for (int r = 0; r < world; ++r)
    for (int b = 0; b < ctas; ++b)
      th.emplace_back([&, r, b] {
        HostComm c;
        c.world = world;
        c.rank = r;
        for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = p < world ? flags[p].data() : nullptr;
        c.local = local[r].data();
        c.timeout_ns = 8ull * 1000 * 1000 * 1000;
        int my_sense = 0;
        for (int call = 0; call < calls && !bad.load(std::memory_order_relaxed); ++call) {
          const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
          const uint32_t epoch = A(c.local + TCCL_LOCAL_TILE_EPOCH).load(std::memory_order_relaxed) + 1u;
          const size_t hoff =
              one_buffer ? 0 : (size_t)(A(c.local + TCCL_LOCAL_AG_SEQ).load(std::memory_order_relaxed) & 1u) * half_elems;
          std::thread mover([&] {
            // groups of (destinations, row tiles) that end in one count + flag raise
            const int ngroups = ring ? world - 1 : std::min(2, row_tiles);
            for (int g = 0; g < ngroups; ++g) {
              const int rt0 = ring ? 0 : g * row_tiles / ngroups, rt1 = ring ? row_tiles : (g + 1) * row_tiles / ngroups;
              for (int q = 0; q < world; ++q) {
                if (q == r) continue;  // the own rows are read from the shard
                if (ring && q != (r + 1 + g) % world) continue;
                for (int rt = rt0; rt < rt1; ++rt)
                  for (int e = b; e < kRow; e += ctas)
                    full[q][hoff + ((size_t)r * row_tiles + rt) * kRow + e] = val(call, r, rt, e);
              }
              const uint32_t done = A(c.local + TCCL_LOCAL_AGCNT + g).fetch_add(1u, std::memory_order_acq_rel);
              if (done == (uint32_t)ctas - 1u) {
                A(c.local + TCCL_LOCAL_AGCNT + g).store(0u, std::memory_order_relaxed);
                for (int q = 0; q < world; ++q) {
                  if (q == r || (ring && q != (r + 1 + g) % world)) continue;
                  for (int rt = rt0; rt < rt1; ++rt)
                    A(c.flags[q] + TCCL_FLAG_AG + r * TCCL_MAX_ROW_TILES + rt).store(epoch, std::memory_order_release);
                }
              }
            }
          });
          // consumer: this CTA's tiles, the previous rank's rows first (they arrive first in ring order)
          for (int t = b; t < (world - 1) * row_tiles; t += ctas) {
            const int j = t / row_tiles, rt = t - j * row_tiles;
            const int src = ((r - 1 - j) % world + world) % world;
            if (!wait_reach(c.flags[r] + TCCL_FLAG_AG + src * TCCL_MAX_ROW_TILES + rt, epoch, c, deadline, b, src,
                            TCCL_W_TILE)) {
              bad.store(2);
              break;
            }
            for (int e = 0; e < kRow; ++e)
              if (full[r][hoff + ((size_t)src * row_tiles + rt) * kRow + e] != val(call, src, rt, e)) bad.store(3);
          }
          mover.join();
          const uint32_t done = A(c.local + TCCL_LOCAL_SCHED).fetch_add(1u, std::memory_order_acq_rel);
          if (done == (uint32_t)ctas - 1u) {
            A(c.local + TCCL_LOCAL_SCHED).store(0u, std::memory_order_relaxed);
            A(c.local + TCCL_LOCAL_AG_SEQ).fetch_add(1u, std::memory_order_relaxed);
            A(c.local + TCCL_LOCAL_TILE_EPOCH).store(epoch, std::memory_order_relaxed);
          }
          if ((call & 3) == (r + b) % 4) std::this_thread::yield();  // let the ranks drift apart
          boundary[r].arrive_and_wait(ctas, my_sense, &bad);          // the next kernel of this rank's stream
        }
      });
  for (auto& x : th) x.join();
  return bad.load();
}

// ---------------------------------------------------------------------------
// Model of the barrier-free GEMM -> reduce-scatter on CTA pairs (gemm_rs_pair.cu): every CTA of a
// rank writes its partial tiles into slot [source][tile] of the OWNER's staging area and raises
// the tile's flag there; then the CTAs of a rank share out the rank's own tiles (a cursor), wait
// for the W flags of a tile and sum the W staged partials.  NO entry barrier: the staging area
// has two halves that alternate on a per-rank count of completed calls; ranks run free of each
// other, the CTAs of one rank meet at a kernel boundary between calls.  ThreadSanitizer checks the
// claim that a rank reaches call n+2 (and overwrites the half of call n) only after its call n+1
// got every peer's partials of call n+1, i.e. after every peer has finished reading call n.
// `mode` bit 1: ONE half only and still no barrier — the mistake, kept to show the check has teeth.
extern "C" int hp_selftest_rs_pair(int world, int ctas, int tiles_per_owner, int calls, int mode) {
  if (world < 1 || world > TCCL_MAX_WORLD || ctas < 1 || ctas > 16 || tiles_per_owner < 1 || tiles_per_owner > 64) return 100;
  constexpr int kElems = 16;
  const bool one_half = (mode & 2) != 0;
  const int tpo = tiles_per_owner;
  const size_t half_elems = (size_t)world * tpo * kElems;
  std::vector<std::vector<uint32_t>> flags(world, std::vector<uint32_t>(TCCL_FLAG_WORDS, 0u));
  std::vector<std::vector<uint32_t>> local(world, std::vector<uint32_t>(TCCL_LOCAL_WORDS, 0u));
  std::vector<std::vector<float>> stage(world, std::vector<float>(2 * half_elems, 0.f));
  std::vector<std::vector<float>> out(world, std::vector<float>((size_t)tpo * kElems, 0.f));
  std::vector<KernelBoundary> boundary(world);
  std::atomic<int> bad{0};
  auto partial = [](int call, int src, int owner, int lt, int e) {
    return (float)(call * 1000 + src * 100 + owner * 10 + (lt * 3 + e) % 7);
  };
  std::vector<std::thread> th;
  for (int r = 0; r < world; ++r)
    for (int b = 0; b < ctas; ++b)
      th.emplace_back([&, r, b] {
        HostComm c;
        c.world = world;
        c.rank = r;
        for (int p = 0; p < TCCL_MAX_WORLD; ++p) c.flags[p] = p < world ? flags[p].data() : nullptr;
        c.local = local[r].data();
        c.timeout_ns = 8ull * 1000 * 1000 * 1000;
        int my_sense = 0;
        for (int call = 0; call < calls && !bad.load(std::memory_order_relaxed); ++call) {
          const auto deadline = clk::now() + std::chrono::nanoseconds(c.timeout_ns);
          const uint32_t epoch = A(c.local + TCCL_LOCAL_TILE_EPOCH).load(std::memory_order_relaxed) + 1u;
          const size_t hoff =
              one_half ? 0 : (size_t)(A(c.local + TCCL_LOCAL_RS_SEQ).load(std::memory_order_relaxed) & 1u) * half_elems;
          // mainloop + epilogue: this CTA's tiles, owners in turn (peers first, own rows last)
          for (int t = b; t < world * tpo; t += ctas) {
            const int lt = t / world, owner = (r + 1 + t % world) % world;
            float* slot = stage[owner].data() + hoff + ((size_t)r * tpo + lt) * kElems;
            for (int e = 0; e < kElems; ++e) slot[e] = partial(call, r, owner, lt, e);
            A(c.flags[owner] + TCCL_FLAG_TILE + r * TCCL_MAX_TILES + lt).store(epoch, std::memory_order_release);
          }
          // final reduction of the rank's own tiles, shared out over its CTAs
          for (;;) {
            const uint32_t u = A(c.local + TCCL_LOCAL_RS_NEXT).fetch_add(1u, std::memory_order_acq_rel);
            if (u >= (uint32_t)tpo) break;
            bool ok = true;
            for (int src = 0; src < world && ok; ++src)
              ok = wait_reach(c.flags[r] + TCCL_FLAG_TILE + src * TCCL_MAX_TILES + u, epoch, c, deadline, b, src, TCCL_W_TILE);
            if (!ok) {
              bad.store(2);
              break;
            }
            for (int e = 0; e < kElems; ++e) {
              float s = 0.f, want = 0.f;
              for (int src = 0; src < world; ++src) {
                s += stage[r][hoff + ((size_t)src * tpo + u) * kElems + e];
                want += partial(call, src, r, (int)u, e);
              }
              out[r][(size_t)u * kElems + e] = s;
              if (s != want) bad.store(3);
            }
          }
          boundary[r].arrive_and_wait(ctas, my_sense, &bad);  // every CTA of the rank has left its final loop
          if (bad.load(std::memory_order_relaxed)) break;
          if (b == 0) {  // what the last CTA of the kernel does
            A(c.local + TCCL_LOCAL_RS_NEXT).store(0u, std::memory_order_relaxed);
            A(c.local + TCCL_LOCAL_RS_SEQ).fetch_add(1u, std::memory_order_relaxed);
            A(c.local + TCCL_LOCAL_TILE_EPOCH).store(epoch, std::memory_order_relaxed);
          }
          if ((call & 3) == (r + b) % 4) std::this_thread::yield();  // let the ranks drift apart
          boundary[r].arrive_and_wait(ctas, my_sense, &bad);  // the next kernel of this rank's stream
        }
      });
  for (auto& x : th) x.join();
  return bad.load();
}

// ---------------------------------------------------------------------------
// Model of the flag-in-line double tree (tree_allreduce_ll.cu): every line on the wire is
// {payload, call number} twice, written and polled as two 8-byte halves (the unit that arrives
// whole); there are no counters and no acknowledgements, only slots [tree][left | right |
// down][call mod depth] per rank.  Ranks run free of each other over many calls (the four role
// threads of a rank meet between calls, as the CTAs of consecutive kernels do); the sums are
// checked after every call.  What this exercises is the numbering: a rank that is a call ahead
// writes the NEXT slot, and a slot comes round again only when its lines have long been read —
// `depth` = 1 is accepted too and must still give the right sums, because a rank cannot finish
// call n before every rank has contributed to call n.
extern "C" int hp_selftest_tree_ll(int world, int numel, int calls, int depth) {
  if (world < 1 || world > TCCL_MAX_WORLD || numel < 2 || (numel & 1) || depth < 1 || depth > 8) return 100;
  const int lines = numel / 2;                  // two floats of payload per line
  const int half0 = (lines + 1) / 2;            // tree 0 takes the first half of the lines, tree 1 the rest
  using Half = std::atomic<uint64_t>;
  // slot(rank, tree, which, seq) -> 2 * lines halves
  const size_t slot_halves = (size_t)2 * lines;
  std::vector<std::vector<Half>> ll(world);
  for (auto& v : ll) v = std::vector<Half>((size_t)2 * 3 * depth * slot_halves);
  for (auto& v : ll)
    for (auto& h : v) h.store(0, std::memory_order_relaxed);
  auto slot = [&](int rank, int tree, int which, uint32_t seq) {
    return ll[rank].data() + ((size_t)(tree * 3 + which) * depth + seq % depth) * slot_halves;
  };
  std::vector<std::vector<float>> in(world, std::vector<float>(numel)), out(world, std::vector<float>(numel, 0.f));
  std::vector<KernelBoundary> boundary(world);
  std::atomic<int> bad{0};
  auto nbr = [&](int N, int r, int tree, int* parent, int* left, int* right) {
    auto a = [&](int rr, int* p, int* l, int* rt) {
      *p = *l = *rt = -1;
      if (N == 1) return;
      if (rr == 0) {
        int top = 1;
        while (top * 2 <= N - 1) top *= 2;
        *l = top;
        return;
      }
      const int s = rr & -rr;
      int up = (rr ^ s) | (s << 1);
      if (up >= N) up = rr ^ s;
      *p = up;
      if (s == 1) return;
      *l = rr - (s >> 1);
      int step = s >> 1, x = rr + step;
      while (x >= N && step > 1) {
        step >>= 1;
        x = rr + step;
      }
      *rt = x >= N ? -1 : x;
    };
    if (tree == 0) return a(r, parent, left, right);
    a((r + 1) % N, parent, left, right);
    auto back = [&](int x) { return x < 0 ? -1 : (x - 1 + N) % N; };
    *parent = back(*parent);
    *left = back(*left);
    *right = back(*right);
  };
  auto pack = [](float d, uint32_t flag) {
    uint32_t u;
    std::memcpy(&u, &d, 4);
    return (uint64_t)u | ((uint64_t)flag << 32);
  };
  const auto t_end = clk::now() + std::chrono::seconds(60);
  // polls one line until both halves carry `flag`; false when the time is up or a check failed elsewhere
  auto get = [&](Half* line, uint32_t flag, float* d0, float* d1) {
    for (;;) {
      const uint64_t a = line[0].load(std::memory_order_relaxed), b = line[1].load(std::memory_order_relaxed);
      if ((uint32_t)(a >> 32) == flag && (uint32_t)(b >> 32) == flag) {
        const uint32_t ua = (uint32_t)a, ub = (uint32_t)b;
        std::memcpy(d0, &ua, 4);
        std::memcpy(d1, &ub, 4);
        return true;
      }
      if (bad.load(std::memory_order_relaxed) || clk::now() > t_end) return false;
      std::this_thread::yield();
    }
  };
  auto put = [&](Half* line, float d0, float d1, uint32_t flag) {
    line[0].store(pack(d0, flag), std::memory_order_relaxed);
    line[1].store(pack(d1, flag), std::memory_order_relaxed);
  };
  std::vector<std::thread> th;
  for (int r = 0; r < world; ++r)
    for (int role = 0; role < 4; ++role)
      th.emplace_back([&, r, role] {
        const int tree = role & 1;
        const bool is_up = role < 2;
        int parent, left, right;
        nbr(world, r, tree, &parent, &left, &right);
        int cslot = 0;
        if (parent >= 0) {
          int pp, pl, pr;
          nbr(world, parent, tree, &pp, &pl, &pr);
          cslot = pl == r ? 0 : 1;
        }
        const int lo = tree ? half0 : 0, n = tree ? lines - half0 : half0;
        int my_sense = 0;
        for (int call = 0; call < calls && !bad.load(std::memory_order_relaxed); ++call) {
          if (role == 0)  // the rank's "host" writes the input between two kernels
            for (int i = 0; i < numel; ++i) in[r][i] = (float)((r + 1) * (i % 5 + 1) + call);
          boundary[r].arrive_and_wait(4, my_sense, &bad);
          const uint32_t g = (uint32_t)call, flag = g + 1u;  // every pipeline counts its own calls: here they agree
          bool ok = true;
          if (is_up) {
            for (int i = 0; i < n && ok; ++i) {
              float d0 = in[r][2 * (lo + i)], d1 = in[r][2 * (lo + i) + 1], x0, x1;
              if (left >= 0) {
                ok = get(slot(r, tree, 0, g) + 2 * i, flag, &x0, &x1);
                d0 += x0;
                d1 += x1;
                if (ok && right >= 0) {
                  ok = get(slot(r, tree, 1, g) + 2 * i, flag, &x0, &x1);
                  d0 += x0;
                  d1 += x1;
                }
              }
              if (!ok) break;
              if (parent >= 0) {
                put(slot(parent, tree, cslot, g) + 2 * i, d0, d1, flag);
              } else {
                if (left >= 0) put(slot(left, tree, 2, g) + 2 * i, d0, d1, flag);
                if (right >= 0) put(slot(right, tree, 2, g) + 2 * i, d0, d1, flag);
                out[r][2 * (lo + i)] = d0;
                out[r][2 * (lo + i) + 1] = d1;
              }
            }
          } else if (parent >= 0) {
            for (int i = 0; i < n && ok; ++i) {
              float d0, d1;
              ok = get(slot(r, tree, 2, g) + 2 * i, flag, &d0, &d1);
              if (!ok) break;
              if (left >= 0) put(slot(left, tree, 2, g) + 2 * i, d0, d1, flag);
              if (right >= 0) put(slot(right, tree, 2, g) + 2 * i, d0, d1, flag);
              out[r][2 * (lo + i)] = d0;
              out[r][2 * (lo + i) + 1] = d1;
            }
          }
          if (!ok) bad.store(1);
          if ((call & 3) == (r + role) % 4) std::this_thread::yield();  // let the ranks drift apart
          boundary[r].arrive_and_wait(4, my_sense, &bad);
          if (role == 0 && !bad.load(std::memory_order_relaxed)) {
            const float tot = (float)(world * (world + 1) / 2);
            for (int i = 0; i < numel; ++i)
              if (out[r][i] != tot * (float)(i % 5 + 1) + (float)(world * call)) bad.store(2);
          }
          boundary[r].arrive_and_wait(4, my_sense, &bad);
        }
      });
  for (auto& x : th) x.join();
  return bad.load();
}

// ---------------------------------------------------------------------------
// Model of how a CTA pair ends (gemm_tcgen05_2cta.cuh, gemm_skinny.cu).  The epilogue of the second CTA arrives on the
// leader's tmem_empty barriers and the leader's MMA thread commits to the second CTA's empty barriers; such remote
// arrivals travel through an INTERCONNECT thread that delivers them later than they are issued.  Both CTAs meet at a
// split cluster barrier whose arrival is relaxed, and what a CTA leaves behind is taken over by the next one (`rounds`
// pairs run one after the other on the same two shared memories).  The accumulators and stages used last are reused by
// nobody, so nothing in the mainloop waits for the arrivals that free them: `drain` = 1 (the kernels) waits for their
// last phases between the barrier's halves; `drain` = 0 is the mistake, kept so that the sanitizer can be seen to catch
// it: a late arrival hits the shared memory of the next CTA.
namespace {
struct PairSmem {
  Mbar full[2], empty[2], tmem_full[2], tmem_empty[2];
  uint32_t owner = 0;  // plain: which CTA's shared memory this is; every delivery looks at it
};
struct Interconnect {
  struct Arrival {
    PairSmem* at;
    Mbar* bar;
    uint32_t owner;
  };
  std::vector<Arrival> sent;
  std::atomic<int> issued{0};
  std::atomic<bool> stop{false};
  std::atomic<int> strays{0};  // arrivals that found another CTA's shared memory
  std::atomic_flag lock = ATOMIC_FLAG_INIT;
  explicit Interconnect(size_t cap) : sent(cap) {}
  void arrive(PairSmem* at, Mbar* bar, uint32_t owner) {
    while (lock.test_and_set(std::memory_order_acquire)) std::this_thread::yield();
    sent[(size_t)issued.load(std::memory_order_relaxed)] = Arrival{at, bar, owner};
    issued.fetch_add(1, std::memory_order_release);
    lock.clear(std::memory_order_release);
  }
  void run() {
    for (int t = 0;;) {
      if (t < issued.load(std::memory_order_acquire)) {
        std::this_thread::sleep_for(std::chrono::microseconds(20));  // on its way
        const Arrival a = sent[(size_t)t++];
        if (a.at->owner != a.owner) strays.fetch_add(1);
        a.bar->arrive();
      } else if (stop.load(std::memory_order_acquire)) {
        return;
      } else {
        std::this_thread::yield();
      }
    }
  }
};
}  // namespace

extern "C" int hp_selftest_pair_exit(int tiles, int rounds, int drain) {
  if (tiles < 0 || tiles > 64 || rounds < 1 || rounds > 1000) return 100;
  PairSmem sm[2];
  Interconnect net((size_t)rounds * tiles * 4 + 4);
  std::thread wire([&] { net.run(); });
  KernelBoundary start, own_cta[2];
  std::atomic<int> at_end{0};  // relaxed arrivals at the pair's last barrier
  // a stray arrival leaves a barrier out of step: nobody waits on after one (or after ten seconds)
  const auto give_up = clk::now() + std::chrono::seconds(10);
  auto lost = [&] {
    if (clk::now() > give_up) net.strays.fetch_add(1);
    return net.strays.load(std::memory_order_relaxed) != 0;
  };
  auto await = [&](const Mbar& b, uint32_t parity) { b.wait(parity, lost); };
  auto cta = [&](int c, int role) {
    int sense = 0, cta_sense = 0;
    for (int round = 1; round <= rounds && !net.strays.load(); ++round) {
      if (role == 0) {  // the next CTA sets up the shared memory it was given
        PairSmem& s = sm[c];
        s.owner = (uint32_t)round;
        for (int i = 0; i < 2; ++i) {
          s.full[i].init(2);
          s.empty[i].init(1);
          s.tmem_full[i].init(1);
          s.tmem_empty[i].init(2);
        }
      }
      start.arrive_and_wait(6, sense, &net.strays);  // producer, MMA (or idle) and epilogue threads of both CTAs
      const uint32_t own = (uint32_t)round;
      auto parity = [](int use) { return ((uint32_t)use & 1u) ^ 1u; };  // of a ring of two, before its use / 2-th filling
      if (role == 0) {  // producer: one stage per tile; the bytes of both CTAs are counted on the leader's barrier
        for (int t = 0; t < tiles; ++t) {
          await(sm[c].empty[t & 1], parity(t >> 1));
          if (c == 0) sm[0].full[t & 1].arrive();
          else net.arrive(&sm[0], &sm[0].full[t & 1], own);
        }
      } else if (role == 1 && c == 0) {  // the leader's MMA thread
        for (int t = 0; t < tiles; ++t) {
          await(sm[0].tmem_empty[t & 1], parity(t >> 1));
          await(sm[0].full[t & 1], (uint32_t)(t >> 1) & 1u);
          sm[0].empty[t & 1].arrive();
          net.arrive(&sm[1], &sm[1].empty[t & 1], own);
          sm[0].tmem_full[t & 1].arrive();
          net.arrive(&sm[1], &sm[1].tmem_full[t & 1], own);
        }
      } else if (role == 2) {  // epilogue
        for (int t = 0; t < tiles; ++t) {
          await(sm[c].tmem_full[t & 1], (uint32_t)(t >> 1) & 1u);
          if (c == 0) sm[0].tmem_empty[t & 1].arrive();
          else net.arrive(&sm[0], &sm[0].tmem_empty[t & 1], own);
        }
      }
      own_cta[c].arrive_and_wait(3, cta_sense, &net.strays);  // __syncthreads
      at_end.fetch_add(1, std::memory_order_relaxed);
      for (int t = tiles; drain && t < tiles + 2; ++t) {
        if (role == 0) await(sm[c].empty[t & 1], parity(t >> 1));
        if (role == 1 && c == 0) await(sm[0].tmem_empty[t & 1], parity(t >> 1));
      }
      while (at_end.load(std::memory_order_acquire) < 6 * round && !lost()) std::this_thread::yield();
      own_cta[c].arrive_and_wait(3, cta_sense, &net.strays);  // the CTA is gone, its SM is free
    }
  };
  std::vector<std::thread> th;
  for (int c = 0; c < 2; ++c)
    for (int role = 0; role < 3; ++role) th.emplace_back(cta, c, role);
  for (auto& x : th) x.join();
  net.stop.store(true);
  wire.join();
  return net.strays.load() ? 1 : 0;
}

// ---------------------------------------------------------------------------
// Model of a wait whose lanes go on to something they do together (`agree` in gemm_tcgen05.cuh: the data warps of
// tree_allreduce.cu, the epilogue warps of the GEMMs).  Every lane polls the mbarrier by itself, and while the wait is being given up elsewhere in the CTA one lane may see that just before the phase completes and the
// others just after: here lane 0 looks first.  `uniform` = 1 (the kernel): the lanes vote and leave or go on together.
// `uniform` = 0 is the mistake, kept to show that it is caught: the lanes that go on wait for lane 0 at their next
// __syncwarp or named barrier, lane 0 waits for them at the CTA's last __syncthreads, and the CTA never returns.  Returns 1 where a
// barrier of the model is still short of a lane after a second.
extern "C" int hp_selftest_warp_verdict(int uniform) {
  constexpr int kLanes = 4;
  Mbar ready;
  ready.init(1);
  std::atomic<int> abort_cta{1}, looked{0}, at_vote{0}, no{0}, at_sync{0}, at_end{0}, stuck{0};
  auto meet = [&](std::atomic<int>& count) {
    count.fetch_add(1);
    const auto late = clk::now() + std::chrono::seconds(1);
    while (count.load() < kLanes) {
      if (clk::now() > late) {
        stuck.store(1);
        return;
      }
      std::this_thread::yield();
    }
  };
  auto lane = [&](int l) {
    if (l > 0) while (!looked.load()) std::this_thread::yield();
    bool ok = ready.wait(0u, [&] { return abort_cta.load() != 0; });  // the phase first, then the flag
    if (l == 0) {
      ready.arrive();
      looked.store(1);
    }
    if (uniform) {  // __all_sync
      if (!ok) no.fetch_add(1);
      meet(at_vote);
      ok = no.load() == 0;
    }
    if (ok) meet(at_sync);  // the __syncwarp behind the slice's stores
    meet(at_end);
  };
  std::vector<std::thread> th;
  for (int l = 0; l < kLanes; ++l) th.emplace_back(lane, l);
  for (auto& x : th) x.join();
  return stuck.load();
}
