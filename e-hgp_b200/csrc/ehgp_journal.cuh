// Forest journal of the direct Morse hierarchy on the device (ehgp_journal.cu): inputs, the
// records it leaves in HBM, and the memory it works in.
#pragma once

#include "ehgp_internal.cuh"

namespace ehgp {

// Device memory handed out in order from one kept block; what does not fit goes to further
// blocks, which the next reset folds into one of the total size.  Records that the device has no
// room for go to pinned host memory, which the kernels write over the bus.
class DeviceArena {
 public:
  explicit DeviceArena(std::atomic<uint64_t>& held) : held_(held) {}  // counts the bytes of its blocks there
  DeviceArena(const DeviceArena&) = delete;
  DeviceArena& operator=(const DeviceArena&) = delete;
  ~DeviceArena() { release(); }
  // Forgets every piece handed out (nothing on the device may still use them) and makes room for `want`
  // bytes in one block; 0: no block.
  cudaError_t reset(uint64_t want);
  cudaError_t take(void** p, uint64_t bytes);
  template <class T>
  cudaError_t take(T** p, uint64_t count) {
    return take(reinterpret_cast<void**>(p), count * sizeof(T));
  }
  // A record array: on the device, or in host memory (always with `spilled`).
  template <class T>
  cudaError_t take_record(T** p, uint64_t count) {
    if (!spilled) {
      const cudaError_t e = take(p, count);
      if (e != cudaErrorMemoryAllocation) return e;
      cudaGetLastError();
    }
    return take_host(reinterpret_cast<void**>(p), count * sizeof(T));
  }
  bool on_host(const void* p) const;
  void release_host();
  void release();
  bool spilled = false;
  uint64_t largest = ~uint64_t{0};  // larger blocks are refused (tests)

 private:
  cudaError_t add(uint64_t size, uint64_t used, void** p);
  cudaError_t take_host(void** p, uint64_t bytes);
  void release_device();
  struct Block {
    char* p;
    uint64_t size, used;
  };
  std::vector<Block> blocks_, host_;
  std::atomic<uint64_t>& held_;
};

// Rounds of the forest journal over all families, and as many by its last block (12 to 21 and 1 to 47 on uniform,
// lattice, mixture and graded clouds of 256 to 50,653 points).
constexpr uint32_t kForestRounds = 64;
constexpr int kJournalOrders = 18;  // orders 1..10 and the ends of their ranges

// The resolved arms of every order.  Families (saddles) and birth handles of orders >= 2 are
// both numbered by rank-partition position: family f is the event at rb2 + f, and handle n + i
// the event at rb2 + i, so family f of order k and handle n + f of order k + 1 are one event.
struct JournalIn {
  uint32_t n = 0, keff = 0;
  uint32_t handles = 0, families = 0, arms = 0;
  uint32_t rounds = kForestRounds;      // at most that
  uint32_t fam0[kJournalOrders] = {};   // first family of order k (k = 1..keff + 1)
  uint32_t han0[kJournalOrders] = {};   // first handle of order k
  const uint32_t* ev = nullptr;         // [families] facade index (ascending within an order)
  const uint32_t* cls = nullptr;        // [families] level class (ascending within an order)
  const uint32_t* armoff = nullptr;     // [families + 1]
  const uint32_t* term = nullptr;       // [arms] birth handle that ends the arm's descent
};

// Records in the reference's arena order with global indices (device pointers into the arena).
struct JournalOut {
  ehgp_journal_batch* jb = nullptr;
  ehgp_role_record* roles = nullptr;
  ehgp_family_record* fam = nullptr;
  ehgp_forest_node* nodes = nullptr;
  uint32_t* children = nullptr;
  ehgp_forest_birth* births = nullptr;
  ehgp_forest_binding* bindings = nullptr;
  ehgp_forest_saddle* saddles = nullptr;
  ehgp_forest_group* groups = nullptr;
  ehgp_forest_batch* fb = nullptr;
  ehgp_vertical_assignment* vert = nullptr;
  std::vector<ehgp_forest_root> roots;  // on the host (one per surviving component)
  uint64_t n_batches = 0, n_roles = 0, n_nodes = 0, n_children = 0, n_groups = 0, n_vert = 0;
  uint32_t rest = 0;  // families that the rounds left to the host
};

// Device bytes the journal takes from its arena for these counts (nodes and children, which
// it counts itself, not included).
uint64_t journal_bytes(const JournalIn& in);
int journal_run(Ctx& ctx, const JournalIn& in, DeviceArena& mem, JournalOut& out, uint64_t* launches);

}  // namespace ehgp
