// Forest journal of the direct Morse hierarchy on the device: event journal and family
// records, frozen-root quotient, batched hyper-Kruskal forest and vertical maps of every order.
//
// Reference semantics (Ludwig-H/E-HGP, morsehgp3d/):
//  journal  src/cpu/hierarchy/direct_morse_event_journal.cpp:260-400 (roles, batches of equal
//           (order, exact level));
//  forest   src/cpu/hierarchy/direct_morse_forest_journal.cpp:1042-2150: per batch, strict arms
//           resolved against the components before the batch, transitive carrier classes, no
//           prior reduced root = reduced birth, one = continuation, two or more = multifusion,
//           then unions (the least handle survives) and births.
//
// The reference applies the batches one after another.  Here every record comes from one
// structure that is built in parallel, the death tree of the handles:
//  * A handle dies in the batch that merges its component with one that holds an older (lesser)
//    handle.  parent(x) is a handle of that older component and death(x) the level class, so the
//    carrier of x before class c is reached from x by climbing while death < c (after class c:
//    while death <= c).
//  * Boruvka rounds find the deaths.  Every component looks for its first family (hyperedge of the
//    arms' handles; families are numbered by time) that leads outside.  If one of the
//    components it meets there is older, its oldest handle dies at that family and the component
//    hooks onto the older one; otherwise it waits.  A hooked chain climbs to older handles and to
//    earlier families, so at that family the chain is already one component, and the root's
//    oldest handle is the component's.  Of two components whose first family is the same, the
//    younger hooks, so every round makes progress; the number of rounds is the longest chain of
//    ever older partners: 10-60 on random clouds, but as many as points where
//    the spacing shrinks along a curve.  What a bounded number of rounds leaves is applied family by
//    family on the host (the contracted components and families are the same problem again).
//  * Counts of carriers, reduced roots, nodes, children and groups before a batch are prefix
//    sums over the families; the reduced root of a component at a level is the last node created
//    under its oldest handle, found by binary search in the nodes sorted by handle.
// Batches with one saddle (almost all, off exact ties) form one group; the saddles of larger
// batches are sorted by the carrier their group merges into.
//
// Bound: random reads of the handles' arrays (L2) in the tree and the carriers, then HBM writes
// of the records (8.3 GB at 50,653 points, K = 10).  16.9 ms there (24.8 M families, 84 M arms);
// one union-find thread per order and a record pool on 16 host cores took 343 ms.
#include "ehgp_journal.cuh"

#include <algorithm>
#include <cstdlib>
#include <memory>
#include <new>

namespace ehgp {

cudaError_t DeviceArena::reset(uint64_t want) {
  spilled = false;
  for (Block& b : host_) b.used = 0;
  uint64_t have = 0;
  for (const Block& b : blocks_) have += b.size;
  if (want && blocks_.size() == 1 && blocks_[0].size >= want && blocks_[0].size <= largest) {
    blocks_[0].used = 0;
    return cudaSuccess;
  }
  release_device();
  if (want == 0) return cudaSuccess;
  void* p = nullptr;
  if (add(std::max(have, want + want / 16) + 4096, 0, &p) == cudaSuccess) return cudaSuccess;
  cudaGetLastError();
  return add(want, 0, &p);
}

cudaError_t DeviceArena::take(void** p, uint64_t bytes) {
  bytes = (bytes + 255) / 256 * 256;
  for (Block& b : blocks_)
    if (b.used + bytes <= b.size) {
      *p = b.p + b.used;
      b.used += bytes;
      return cudaSuccess;
    }
  return add(bytes + bytes / 8 + 4096, bytes, p);
}

cudaError_t DeviceArena::add(uint64_t size, uint64_t used, void** p) {
  if (size > largest) return cudaErrorMemoryAllocation;
  blocks_.reserve(blocks_.size() + 1);
  const cudaError_t e = cudaMalloc(p, size);
  if (e != cudaSuccess) return e;
  blocks_.push_back({static_cast<char*>(*p), size, used});
  held_ += size;
  return cudaSuccess;
}

cudaError_t DeviceArena::take_host(void** p, uint64_t bytes) {
  bytes = (bytes + 255) / 256 * 256;
  for (Block& b : host_)
    if (b.used + bytes <= b.size) {
      *p = b.p + b.used;
      b.used += bytes;
      return cudaSuccess;
    }
  host_.reserve(host_.size() + 1);
  const uint64_t size = bytes + bytes / 8 + 4096;
  const cudaError_t e = cudaHostAlloc(p, size, cudaHostAllocPortable | cudaHostAllocMapped);
  if (e == cudaSuccess) host_.push_back({static_cast<char*>(*p), size, bytes});
  return e;
}

bool DeviceArena::on_host(const void* p) const {
  for (const Block& b : host_)
    if (p >= b.p && p < b.p + b.size) return true;
  return false;
}

void DeviceArena::release_device() {
  for (const Block& b : blocks_) {
    cudaFree(b.p);
    held_ -= b.size;
  }
  blocks_.clear();
}

void DeviceArena::release_host() {
  for (const Block& b : host_) cudaFreeHost(b.p);
  host_.clear();
}

void DeviceArena::release() {
  release_device();
  release_host();
}

namespace {

constexpr int kT = 256;
constexpr uint32_t kNone = 0xffffffffu;
constexpr uint32_t kSaddle = 0x80000000u;    // role source: family index with this bit, else a handle
constexpr uint32_t kTailFamilies = 1u << 13;  // active families that one block takes on alone

inline uint32_t nblk(uint64_t m, int t = kT) { return m ? (uint32_t)((m + t - 1) / t) : 1u; }

// Journal error bits (device word).
constexpr uint32_t kErrUnborn = 1u, kErrNoRoot = 4u;

struct J {  // kernel view of the input
  uint32_t n, keff, handles, families, arms;
  uint32_t fam0[kJournalOrders], han0[kJournalOrders], role0[kJournalOrders];
  const uint32_t* __restrict__ ev;
  const uint32_t* __restrict__ cls;
  const uint32_t* __restrict__ armoff;
  const uint32_t* __restrict__ term;
};

__device__ __forceinline__ uint32_t family_order(const J& j, uint32_t f) {
  uint32_t k = 1;
  while (k < j.keff && f >= j.fam0[k + 1]) ++k;
  return k;
}

// Death tree and touch state of the handles.
struct Tree {
  uint2* dead;      // [handles] (parent, death class or kNone while alive)
  uint32_t* touch;  // [handles] class of the first family that has the handle as a carrier
  uint32_t* from;   // [handles] the carrier whose reduced root it took over at its first touch
  uint2* range;     // [handles] its nodes in sorted order
  const uint32_t* node_cls;  // [nodes] level class of the sorted nodes
  const uint32_t* node_idx;  // [nodes] their index among the created nodes
  uint32_t n;
  uint2* skip;      // [handles] (the handle kSkip climbs up, the last death on the way), where climbs are long
};
constexpr int kSkip = 64;

__device__ __forceinline__ uint32_t carrier_before(const Tree& t, uint32_t x, uint32_t cls) {
  if (t.skip)
    for (uint2 k = t.skip[x]; k.y < cls; k = t.skip[x]) x = k.x;
  for (uint2 d = t.dead[x]; d.y < cls; d = t.dead[x]) x = d.x;
  return x;
}
__device__ __forceinline__ uint32_t carrier_after(const Tree& t, uint32_t x, uint32_t cls) {
  if (t.skip)
    for (uint2 k = t.skip[x]; k.y <= cls && k.y != kNone; k = t.skip[x]) x = k.x;
  for (uint2 d = t.dead[x]; d.y <= cls && d.y != kNone; d = t.dead[x]) x = d.x;
  return x;
}
__device__ __forceinline__ bool touched_before(const Tree& t, uint32_t c, uint32_t cls) {
  return c < t.n || t.touch[c] < cls;
}

// Reduced root (global node index) of the component whose oldest handle is c: the last node
// created under c at a class below `lim`, else the root c took over when it was first touched.
__device__ uint32_t reduced_root(const Tree& t, uint32_t c, uint64_t lim) {
  for (;;) {
    const uint2 r = t.range[c];
    uint32_t lo = r.x, hi = r.y;
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if ((uint64_t)t.node_cls[mid] < lim) lo = mid + 1;
      else hi = mid;
    }
    if (lo > r.x) return t.n + t.node_idx[lo - 1];
    if (c < t.n) return c;
    lim = t.touch[c];  // strictly earlier at every step
    c = t.from[c];
    if (c == kNone) return kNone;
  }
}

// Distinct carriers of family f in ascending order.
__device__ __forceinline__ int distinct_carriers(const uint32_t* __restrict__ car, uint32_t a0, uint32_t a1,
                                                 uint32_t d[4]) {
  int m = 0;
  for (uint32_t a = a0; a < a1; ++a) {
    const uint32_t c = car[a];
    int i = 0;
    while (i < m && d[i] < c) ++i;
    if (i < m && d[i] == c) continue;
    for (int q = m; q > i; --q) d[q] = d[q - 1];
    d[i] = c;
    ++m;
  }
  return m;
}

// ---- prefix sums ----------------------------------------------------------------------
// Exclusive sums of C words per item in item order: per-block totals, their scan by one block,
// then each block's own scan with the items' sums handed to `out`.  A warp owns 8 rows of 32
// consecutive items, so every load is coalesced and a block synchronises once.
template <int C>
struct Sums {
  uint32_t v[C];
};
constexpr int kScanTile = kT * 8;

template <int C, class In>
__device__ __forceinline__ Sums<C> warp_total(uint32_t m, uint32_t base, uint32_t lane, const In& in) {
  Sums<C> s{};
  for (int r = 0; r < 8; ++r) {
    const uint32_t i = base + r * 32 + lane;
    if (i < m) {
      const Sums<C> x = in(i);
#pragma unroll
      for (int c = 0; c < C; ++c) s.v[c] += x.v[c];
    }
  }
#pragma unroll
  for (int c = 0; c < C; ++c)
    for (int o = 16; o > 0; o >>= 1) s.v[c] += __shfl_xor_sync(0xffffffffu, s.v[c], o);
  return s;
}

template <int C, class In>
__global__ void __launch_bounds__(kT) k_sum_tiles(uint32_t m, In in, uint32_t* __restrict__ tot, uint32_t nb) {
  __shared__ uint32_t w[C][kT / 32];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const Sums<C> s = warp_total<C>(m, blockIdx.x * kScanTile + warp * 256, lane, in);
  if (lane == 0)
    for (int c = 0; c < C; ++c) w[c][warp] = s.v[c];
  __syncthreads();
  if (threadIdx.x < C) {
    uint32_t t = 0;
    for (int q = 0; q < kT / 32; ++q) t += w[threadIdx.x][q];
    tot[(uint64_t)threadIdx.x * (nb + 1) + blockIdx.x] = t;
  }
}

// One block per channel: exclusive scan of the nb tile totals, the grand total in slot nb.
__global__ void __launch_bounds__(1024) k_sum_top(uint32_t nb, uint32_t* __restrict__ tot_all) {
  __shared__ uint32_t w[32];
  __shared__ uint32_t carry;
  uint32_t* tot = tot_all + (uint64_t)blockIdx.x * (nb + 1);
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t b = 0; b < nb; b += 1024) {
    const uint32_t i = b + threadIdx.x;
    const uint32_t v = i < nb ? tot[i] : 0u;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)lane >= o) x += y;
    }
    if (lane == 31) w[warp] = x;
    __syncthreads();
    if (warp == 0) {
      uint32_t y = w[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
        if ((int)lane >= o) y += z;
      }
      w[lane] = y;
    }
    __syncthreads();
    const uint32_t before = carry + (warp ? w[warp - 1] : 0u);
    if (i < nb) tot[i] = before + x - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) tot[nb] = carry;
}

template <int C, class In, class Out>
__global__ void __launch_bounds__(kT) k_sum_apply(uint32_t m, In in, const uint32_t* __restrict__ tot, uint32_t nb,
                                                  Out out) {
  __shared__ uint32_t w[C][kT / 32];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t base = blockIdx.x * kScanTile + warp * 256;
  const Sums<C> mine = warp_total<C>(m, base, lane, in);
  if (lane == 0)
    for (int c = 0; c < C; ++c) w[c][warp] = mine.v[c];
  __syncthreads();
  Sums<C> run;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    run.v[c] = tot[(uint64_t)c * (nb + 1) + blockIdx.x];
    for (uint32_t q = 0; q < warp; ++q) run.v[c] += w[c][q];
  }
  for (int r = 0; r < 8; ++r) {
    const uint32_t i = base + r * 32 + lane;
    const Sums<C> x = i < m ? in(i) : Sums<C>{};
    Sums<C> ex;
#pragma unroll
    for (int c = 0; c < C; ++c) {
      uint32_t s = x.v[c];
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
        if ((int)lane >= o) s += y;
      }
      ex.v[c] = run.v[c] + s - x.v[c];
      run.v[c] += __shfl_sync(0xffffffffu, s, 31);
    }
    if (i < m) out(i, x, ex);
  }
}

// tot: C * (tiles + 1) words; the totals are at tot[c * (tiles + 1) + tiles].
template <int C, class In, class Out>
void prefix_sums(cudaStream_t st, uint32_t m, const In& in, uint32_t* tot, const Out& out, uint64_t* launches) {
  const uint32_t nb = nblk(m, kScanTile);
  k_sum_tiles<C><<<nb, kT, 0, st>>>(m, in, tot, nb);
  k_sum_top<<<C, 1024, 0, st>>>(nb, tot);
  k_sum_apply<C><<<nb, kT, 0, st>>>(m, in, tot, nb, out);
  *launches += 3;
}

// ---- 1. death tree ----------------------------------------------------------------------
__global__ void __launch_bounds__(kT) k_fj_init(uint32_t handles, Tree t, uint32_t* __restrict__ lab,
                                                uint32_t* __restrict__ best0, uint32_t* __restrict__ best1) {
  const uint32_t h = blockIdx.x * kT + threadIdx.x;
  if (h >= handles) return;
  t.dead[h] = make_uint2(h, kNone);
  t.touch[h] = kNone;
  t.from[h] = kNone;
  t.range[h] = make_uint2(0u, 0u);
  lab[h] = h;
  best0[h] = kNone;
  best1[h] = kNone;
}

// The active families: distinct components of the arms (absent = the first one again).
struct Active {
  uint4* comp;
  uint32_t* fam;
};

__device__ __forceinline__ void offer(uint32_t* best, uint32_t c, uint32_t f) {
  if (__ldcg(best + c) > f) atomicMin(best + c, f);
}

constexpr int kRows = 4;  // entries per thread and step

// Appends a block's kept entries to `to` and offers their families to their components.  Loads,
// stores and atomics on one address run one after another, so the block takes its slots with one
// atomic and sends one offer to the least component it meets (in late rounds one that almost
// every entry touches).  All rounds on 12,289 uniform points (4.9 M families): 20.2 ms with an
// append and an offer per warp and a label store per entry, 1.4 ms like this.
__device__ __forceinline__ void append_and_offer(const bool (&keep)[kRows], const uint4 (&c)[kRows],
                                                 const uint32_t (&f)[kRows], const Active& to, uint32_t* count,
                                                 uint32_t* best) {
  __shared__ uint32_t warp_n[32], s_hot, s_first;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  if (threadIdx.x == 0) s_hot = s_first = kNone;
  uint32_t least[kRows], low = kNone, bal[kRows], n = 0;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    least[r] = keep[r] ? min(min(c[r].x, c[r].y), min(c[r].z, c[r].w)) : kNone;
    low = min(low, least[r]);
    bal[r] = __ballot_sync(0xffffffffu, keep[r]);
    n += __popc(bal[r]);
  }
  low = __reduce_min_sync(0xffffffffu, low);
  __syncthreads();
  if (lane == 0) {
    warp_n[warp] = n;
    atomicMin(&s_hot, low);
  }
  __syncthreads();
  const uint32_t hot = s_hot;
  if (hot == kNone) {  // nothing kept: uniform over the block
    __syncthreads();
    return;
  }
  uint32_t first = kNone;
#pragma unroll
  for (int r = 0; r < kRows; ++r)
    if (least[r] == hot) first = min(first, f[r]);
  first = __reduce_min_sync(0xffffffffu, first);
  if (lane == 0 && first != kNone) atomicMin(&s_first, first);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t total = 0;
    for (uint32_t w = 0; w < warps; ++w) {
      const uint32_t x = warp_n[w];
      warp_n[w] = total;
      total += x;
    }
    s_first = (offer(best, hot, s_first), atomicAdd(count, total));
  }
  __syncthreads();
  uint32_t at = s_first + warp_n[warp];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    if (keep[r]) {
      const uint32_t slot = at + __popc(bal[r] & ((1u << lane) - 1u));
      to.comp[slot] = c[r];
      to.fam[slot] = f[r];
      if (c[r].x != hot) offer(best, c[r].x, f[r]);
      if (c[r].y != hot && c[r].y != c[r].x) offer(best, c[r].y, f[r]);
      if (c[r].z != hot && c[r].z != c[r].x && c[r].z != c[r].y) offer(best, c[r].z, f[r]);
      if (c[r].w != hot && c[r].w != c[r].x && c[r].w != c[r].y && c[r].w != c[r].z) offer(best, c[r].w, f[r]);
    }
    at += __popc(bal[r]);
  }
  __syncthreads();
}

// Checks every arm's handle (of the family's order, born at an earlier level) and starts the
// first round: every handle is its own component.
__global__ void __launch_bounds__(kT) k_fj_first(J j, Active to, uint32_t* __restrict__ count,
                                                 uint32_t* __restrict__ best, uint32_t* __restrict__ err) {
  bool keep[kRows];
  uint4 c[kRows];
  uint32_t fs[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t f = (blockIdx.x * kRows + r) * kT + threadIdx.x;
    keep[r] = false;
    c[r] = make_uint4(0, 0, 0, 0);
    fs[r] = f;
    if (f >= j.families) continue;
    const uint32_t k = family_order(j, f), a0 = j.armoff[f], a1 = j.armoff[f + 1], fc = j.cls[f];
    uint32_t v[4];
    bool ok = true;
    for (int i = 0; i < 4; ++i) {
      v[i] = a0 + i < a1 ? j.term[a0 + i] : v[0];
      ok &= v[i] >= j.han0[k] && v[i] < j.han0[k + 1] && (v[i] < j.n || j.cls[v[i] - j.n] < fc);
    }
    if (!ok) atomicOr(err, kErrUnborn);
    c[r] = make_uint4(v[0], v[1], v[2], v[3]);
    keep[r] = ok && !(v[1] == v[0] && v[2] == v[0] && v[3] == v[0]);
  }
  append_and_offer(keep, c, fs, to, count, best);
}

// A component whose first family is this one hooks onto the oldest component that it meets
// there, when that one is older.
// kShared: hooks and rounds share one launch (the tail), so nothing may come from a stale L1 line;
// in the launches of their own, the words that every entry reads stay in L1.
template <bool kShared>
__device__ __forceinline__ uint32_t word(const uint32_t* p) {
  return kShared ? __ldcg(p) : *p;
}
template <bool kShared>
__device__ __forceinline__ void hook_entry(const uint32_t* cls, uint4 c, uint32_t f, const uint32_t* best,
                                           uint32_t* best_next, const Tree& t, uint32_t* lab) {
  const uint32_t least = min(min(c.x, c.y), min(c.z, c.w));
  const uint32_t v[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (word<kShared>(best + v[i]) != f) continue;
    best_next[v[i]] = kNone;  // by the one entry that won v[i]: a store per entry queues on a large component
    if (v[i] == least) continue;
    t.dead[v[i]] = make_uint2(least, cls[f]);
    lab[v[i]] = least;
  }
}

// The entry's components after the hooks (whole hooked chains are followed; the label of a hooked
// component is shortened to the root for the entries that come later).
template <bool kShared>
__device__ __forceinline__ uint32_t current_component(uint32_t* lab, uint32_t x) {
  const uint32_t up = word<kShared>(lab + x);
  uint32_t r = up;
  for (uint32_t p = word<kShared>(lab + r); p != r; p = word<kShared>(lab + r)) r = p;
  if (r != up) lab[x] = r;  // (a store per entry of a large component would queue on its label)
  return r;
}
template <bool kShared>
__device__ __forceinline__ bool advance_entry(uint4& c, uint32_t* lab) {
  const uint4 o = c;
  c.x = current_component<kShared>(lab, o.x);
  c.y = o.y == o.x ? c.x : current_component<kShared>(lab, o.y);
  c.z = o.z == o.x ? c.x : (o.z == o.y ? c.y : current_component<kShared>(lab, o.z));
  c.w = o.w == o.x ? c.x : (o.w == o.y ? c.y : (o.w == o.z ? c.z : current_component<kShared>(lab, o.w)));
  return !(c.y == c.x && c.z == c.x && c.w == c.x);
}

__global__ void __launch_bounds__(kT) k_fj_hook(const uint32_t* __restrict__ cls, Active in,
                                                const uint32_t* __restrict__ count, const uint32_t* best,
                                                uint32_t* best_next, Tree t, uint32_t* lab) {
  const uint32_t m = *count;
  for (uint32_t i = blockIdx.x * kT + threadIdx.x; i < m; i += gridDim.x * kT)
    hook_entry<false>(cls, in.comp[i], in.fam[i], best, best_next, t, lab);
}

// One step of the advance: the block's entries b .. b + kRows * blockDim.x - 1.
template <bool kShared>
__device__ __forceinline__ void advance_block(uint32_t b, uint32_t m, const Active& in, const Active& to,
                                              uint32_t* count_next, uint32_t* best_next, uint32_t* lab) {
  bool keep[kRows];
  uint4 c[kRows];
  uint32_t f[kRows];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t i = b + r * blockDim.x + threadIdx.x;
    keep[r] = false;
    c[r] = make_uint4(0, 0, 0, 0);
    f[r] = 0;
    if (i >= m) continue;
    c[r] = in.comp[i];
    f[r] = in.fam[i];
    keep[r] = advance_entry<kShared>(c[r], lab);
  }
  append_and_offer(keep, c, f, to, count_next, best_next);
}

__global__ void __launch_bounds__(kT) k_fj_advance(Active in, const uint32_t* __restrict__ count, Active to,
                                                   uint32_t* count_next, uint32_t* best_next, uint32_t* lab) {
  const uint32_t m = *count;
  for (uint32_t b = blockIdx.x * kRows * kT; b < m; b += gridDim.x * kRows * kT)
    advance_block<false>(b, m, in, to, count_next, best_next, lab);
}

// The last active families: one block runs up to `rounds` rounds without returning to the host.
// left[0]: the families still active then, left[1]: 1 when they are in `next`.
__global__ void __launch_bounds__(1024) k_fj_tail(const uint32_t* __restrict__ cls, Active cur, Active next,
                                                  const uint32_t* __restrict__ count, uint32_t* best,
                                                  uint32_t* best_next, Tree t, uint32_t* lab, uint32_t rounds,
                                                  uint32_t* __restrict__ left_over) {
  __shared__ uint32_t left;
  uint32_t m = *count, round = 0;
  for (; m > 0 && round < rounds; ++round) {
    if (threadIdx.x == 0) left = 0;
    for (uint32_t i = threadIdx.x; i < m; i += 1024)
      hook_entry<true>(cls, cur.comp[i], cur.fam[i], best, best_next, t, lab);
    __threadfence();
    __syncthreads();
    for (uint32_t b = 0; b < m; b += kRows * 1024) advance_block<true>(b, m, cur, next, &left, best_next, lab);
    __threadfence();
    __syncthreads();
    m = left;
    __syncthreads();
    const Active a = cur;
    cur = next;
    next = a;
    uint32_t* q = best;
    best = best_next;
    best_next = q;
  }
  if (threadIdx.x == 0) {
    left_over[0] = m;
    left_over[1] = round & 1u;
  }
}

__global__ void __launch_bounds__(kT) k_fj_rest_keys(uint32_t m, const uint32_t* __restrict__ fam,
                                                     uint64_t* __restrict__ key, uint32_t* __restrict__ val) {
  const uint32_t i = blockIdx.x * kT + threadIdx.x;
  if (i >= m) return;
  key[i] = fam[i];
  val[i] = i;
}

// Deaths found on the host: (handle, older handle, family).
__global__ void __launch_bounds__(kT) k_fj_deaths(uint32_t m, const uint32_t* __restrict__ cls,
                                                  const uint4* __restrict__ deaths, Tree t) {
  const uint32_t i = blockIdx.x * kT + threadIdx.x;
  if (i >= m) return;
  const uint4 d = deaths[i];
  t.dead[d.x] = make_uint2(d.y, cls[d.z]);
}

// Kruskal's algorithm over families in ascending order: the deaths of the components' oldest handles.
// val: the families' places in `comp`; key: the families.
void deaths_in_order(uint32_t handles, const std::vector<uint4>& comp, const std::vector<uint64_t>& key,
                     const std::vector<uint32_t>& val, std::vector<uint4>& deaths) {
  // parent + 1, 0 = a root: zero pages that are never touched are never made
  const std::unique_ptr<uint32_t, void (*)(void*)> hold(static_cast<uint32_t*>(std::calloc(handles, sizeof(uint32_t))), std::free);
  uint32_t* up = hold.get();
  if (!up) throw std::bad_alloc();
  auto find = [up](uint32_t x) {
    while (up[x]) {
      const uint32_t p = up[x] - 1;
      if (up[p]) up[x] = up[p];
      x = p;
    }
    return x;
  };
  for (size_t i = 0; i < key.size(); ++i) {
    const uint4 c = comp[val[i]];
    uint32_t r[4] = {find(c.x), find(c.y), find(c.z), find(c.w)};
    const uint32_t least = std::min(std::min(r[0], r[1]), std::min(r[2], r[3]));
    for (uint32_t x : r) {
      if (x == least || up[x]) continue;
      up[x] = least + 1;
      deaths.push_back(make_uint4(x, least, (uint32_t)key[i], 0u));
    }
  }
}

// parent(x) becomes the oldest handle of the component that x dies into, so deaths increase
// along every climb (a parent read before or after its own shortening is valid).
__global__ void __launch_bounds__(kT) k_fj_normalise(uint32_t handles, Tree t) {
  const uint32_t h = blockIdx.x * kT + threadIdx.x;
  if (h >= handles) return;
  const uint2 d = t.dead[h];
  if (d.y == kNone) return;
  const uint32_t p = carrier_after(t, d.x, d.y);
  if (p != d.x) t.dead[h].x = p;
}

// Deaths increase along a climb, so kSkip steps of it can be taken at once when the last one can.
__global__ void __launch_bounds__(kT) k_fj_skips(uint32_t handles, Tree t, uint2* __restrict__ skip) {
  const uint32_t h = blockIdx.x * kT + threadIdx.x;
  if (h >= handles) return;
  uint2 k = make_uint2(h, 0u);
  for (int i = 0; i < kSkip; ++i) {
    const uint2 d = t.dead[k.x];
    if (d.y == kNone) {
      k.y = kNone;
      break;
    }
    k = d;
  }
  skip[h] = k;
}

// ---- 2. carriers and groups ----------------------------------------------------------------
__device__ __forceinline__ bool in_shared_batch(const J& j, uint32_t f) {  // another saddle at its level
  const uint32_t k = family_order(j, f), c = j.cls[f];
  return (f > j.fam0[k] && j.cls[f - 1] == c) || (f + 1 < j.fam0[k + 1] && j.cls[f + 1] == c);
}

__global__ void __launch_bounds__(kT) k_fj_carriers(J j, Tree t, uint32_t* __restrict__ car,
                                                    uint32_t* __restrict__ shared_count) {
  const uint32_t f = blockIdx.x * kT + threadIdx.x;
  if (f >= j.families) return;
  const uint32_t c = j.cls[f], a0 = j.armoff[f], a1 = j.armoff[f + 1];
  for (uint32_t a = a0; a < a1; ++a) {
    const uint32_t r = carrier_before(t, j.term[a], c);
    car[a] = r;
    if (r >= j.n && __ldcg(t.touch + r) > c) atomicMin(t.touch + r, c);
  }
  if (in_shared_batch(j, f)) atomicAdd(shared_count, 1u);
}

// Groups of the saddles alone in their batch: distinct carriers and those with a reduced root; an
// untouched oldest carrier takes over the one reduced root there is.  (Slot = family.)
__global__ void __launch_bounds__(kT) k_fj_groups(J j, Tree t, const uint32_t* __restrict__ car,
                                                  const uint32_t* __restrict__ slot_q, uint32_t* __restrict__ gc,
                                                  uint32_t* __restrict__ gp) {
  const uint32_t f = blockIdx.x * kT + threadIdx.x;
  if (f >= j.families || (slot_q && slot_q[f] != kNone)) return;
  const uint32_t c = j.cls[f];
  uint32_t d[4];
  const int m = distinct_carriers(car, j.armoff[f], j.armoff[f + 1], d);
  uint32_t np = 0, one = kNone;
  for (int i = 0; i < m; ++i)
    if (touched_before(t, d[i], c)) {
      ++np;
      one = d[i];
    }
  if (np == 1 && one != d[0]) t.from[d[0]] = one;
  gc[f] = (uint32_t)m;
  gp[f] = np;
}

// Channels over the slots: groups, created nodes, children, carriers merged away, reduced roots
// merged away (np - 1, modulo 2^32).
struct GroupIn {
  const uint32_t* gc;
  const uint32_t* gp;
  __device__ Sums<5> operator()(uint32_t s) const {
    const uint32_t c = gc[s], p = gp[s];
    if (c == 0) return Sums<5>{};
    return Sums<5>{{1u, p != 1u ? 1u : 0u, p >= 2u ? p : 0u, c - 1u, p - 1u}};
  }
};
struct GroupSums {  // exclusive sums over the slots, [families + 1]
  uint32_t *g, *node, *child, *dc, *dp;
};
struct GroupOut {
  GroupSums s;
  uint32_t last;
  __device__ void operator()(uint32_t i, const Sums<5>& x, const Sums<5>& e) const {
    s.g[i] = e.v[0];
    s.node[i] = e.v[1];
    s.child[i] = e.v[2];
    s.dc[i] = e.v[3];
    s.dp[i] = e.v[4];
    if (i == last) {
      s.g[i + 1] = e.v[0] + x.v[0];
      s.node[i + 1] = e.v[1] + x.v[1];
      s.child[i + 1] = e.v[2] + x.v[2];
      s.dc[i + 1] = e.v[3] + x.v[3];
      s.dp[i + 1] = e.v[4] + x.v[4];
    }
  }
};

// ---- 2b. batches with several saddles ---------------------------------------------------
// Their saddles keep the batch's slots, ordered by (oldest carrier of the group, family); the
// group's carriers are the distinct carriers of its saddles.
struct Shared {          // q: position among these saddles; empty when there are none
  uint32_t m = 0;
  uint32_t* fam = nullptr;      // [m] family, in family order
  uint32_t* slot_q = nullptr;   // [families] q of a slot, or kNone
  uint32_t* sorted = nullptr;   // [m] family at slot position q
  uint32_t* gid = nullptr;      // [m] group of slot position q
  uint32_t* armoff = nullptr;   // [m] first binding of slot position q
  uint32_t* oldest = nullptr;   // per group: oldest carrier
  uint32_t* cars = nullptr;     // per group: distinct carriers
  uint32_t* priors = nullptr;   // per group: those with a reduced root
  uint32_t* one = nullptr;      // per group: one of them
  uint32_t* saddles = nullptr;  // per group: saddles
  uint32_t* head = nullptr;     // per group: its first q
};

struct SharedFlagIn {
  J j;
  __device__ Sums<1> operator()(uint32_t f) const { return Sums<1>{{in_shared_batch(j, f) ? 1u : 0u}}; }
};
struct SharedFlagOut {
  uint32_t* fam;
  uint32_t* slot_q;
  __device__ void operator()(uint32_t f, const Sums<1>& x, const Sums<1>& e) const {
    slot_q[f] = x.v[0] ? e.v[0] : kNone;
    if (x.v[0]) fam[e.v[0]] = f;
  }
};
struct RunIn {  // first saddle of its batch
  J j;
  const uint32_t* fam;
  __device__ Sums<1> operator()(uint32_t q) const {
    const uint32_t f = fam[q];
    return Sums<1>{{q == 0 || fam[q - 1] + 1 != f || j.cls[f - 1] != j.cls[f] || f == j.fam0[family_order(j, f)] ? 1u : 0u}};
  }
};
struct RunOut {
  J j;
  Tree t;
  const uint32_t* fam;
  uint64_t* key;
  uint32_t* val;
  __device__ void operator()(uint32_t q, const Sums<1>& x, const Sums<1>& e) const {
    const uint32_t f = fam[q];
    key[q] = (uint64_t)(e.v[0] + x.v[0]) << 32 | carrier_after(t, j.term[j.armoff[f]], j.cls[f]);
    val[q] = q;
  }
};
struct SharedGroupIn {  // (first of its group, arms) in slot order
  J j;
  const uint32_t* fam;
  const uint64_t* key;  // sorted
  const uint32_t* val;
  __device__ Sums<2> operator()(uint32_t q) const {
    const uint32_t f = fam[val[q]];
    return Sums<2>{{q == 0 || key[q] != key[q - 1] ? 1u : 0u, j.armoff[f + 1] - j.armoff[f]}};
  }
};
struct SharedGroupOut {
  J j;
  Shared s;
  const uint64_t* key;
  const uint32_t* val;
  uint32_t* prefix;
  __device__ void operator()(uint32_t q, const Sums<2>& x, const Sums<2>& e) const {
    const uint32_t g = e.v[0] + x.v[0] - 1u;
    s.sorted[q] = s.fam[val[q]];
    s.gid[q] = g;
    prefix[q] = e.v[1];
    if (x.v[0]) {
      s.head[g] = q;
      s.oldest[g] = (uint32_t)key[q];
      s.cars[g] = s.priors[g] = s.saddles[g] = 0u;
      s.one[g] = kNone;
    }
  }
};

// Bindings of a batch start at its first family's arms; (group, carrier) keys of every saddle.
__global__ void __launch_bounds__(kT) k_fj_shared_arms(J j, Shared s, const uint64_t* __restrict__ key,
                                                       const uint32_t* __restrict__ prefix,
                                                       const uint32_t* __restrict__ car, uint64_t* __restrict__ ckey,
                                                       uint32_t* __restrict__ cval) {
  const uint32_t q = blockIdx.x * kT + threadIdx.x;
  if (q >= s.m) return;
  uint32_t lo = 0, hi = q;  // first position of the run (keys ascend by run)
  while (lo < hi) {
    const uint32_t mid = (lo + hi) / 2;
    if (key[mid] >> 32 < key[q] >> 32) lo = mid + 1;
    else hi = mid;
  }
  s.armoff[q] = j.armoff[s.fam[lo]] + (prefix[q] - prefix[lo]);
  const uint32_t f = s.sorted[q], g = s.gid[q];
  atomicAdd(s.saddles + g, 1u);
  uint32_t d[4];
  const int m = distinct_carriers(car, j.armoff[f], j.armoff[f + 1], d);
  for (int i = 0; i < 4; ++i) {
    ckey[4ull * q + i] = i < m ? (uint64_t)g << 32 | d[i] : ~uint64_t{0};
    cval[4ull * q + i] = 4 * q + i;
  }
}

__global__ void __launch_bounds__(kT) k_fj_shared_carriers(J j, Tree t, Shared s, const uint64_t* __restrict__ ckey) {
  const uint32_t i = blockIdx.x * kT + threadIdx.x;
  if (i >= 4 * s.m) return;
  const uint64_t key = ckey[i];
  if (key == ~uint64_t{0} || (i > 0 && ckey[i - 1] == key)) return;
  const uint32_t g = (uint32_t)(key >> 32), c = (uint32_t)key;
  atomicAdd(s.cars + g, 1u);
  if (touched_before(t, c, j.cls[s.sorted[s.head[g]]])) {
    atomicAdd(s.priors + g, 1u);
    s.one[g] = c;
  }
}

__global__ void __launch_bounds__(kT) k_fj_shared_groups(J j, Tree t, Shared s, uint32_t* __restrict__ gc,
                                                         uint32_t* __restrict__ gp) {
  const uint32_t q = blockIdx.x * kT + threadIdx.x;
  if (q >= s.m) return;
  const uint32_t g = s.gid[q], slot = s.fam[q];
  const bool head = s.head[g] == q;
  gc[slot] = head ? s.cars[g] : 0u;
  gp[slot] = head ? s.priors[g] : 0u;
  if (head && s.priors[g] == 1 && s.one[g] != s.oldest[g]) t.from[s.oldest[g]] = s.one[g];
}

// (group, reduced root) keys of the multifusions' distinct carriers.
__global__ void __launch_bounds__(kT) k_fj_shared_prior_keys(J j, Tree t, Shared s, const uint64_t* __restrict__ ckey,
                                                             uint64_t* __restrict__ pkey, uint32_t* __restrict__ pval) {
  const uint32_t i = blockIdx.x * kT + threadIdx.x;
  if (i >= 4 * s.m) return;
  const uint64_t key = ckey[i];
  uint64_t out = ~uint64_t{0};
  if (key != ~uint64_t{0} && !(i > 0 && ckey[i - 1] == key)) {
    const uint32_t g = (uint32_t)(key >> 32), c = (uint32_t)key, cls = j.cls[s.sorted[s.head[g]]];
    if (s.priors[g] >= 2 && touched_before(t, c, cls)) out = (uint64_t)g << 32 | reduced_root(t, c, cls);
  }
  pkey[i] = out;
  pval[i] = i;
}

__global__ void __launch_bounds__(kT) k_fj_shared_children(Shared s, GroupSums gs, const uint64_t* __restrict__ pkey,
                                                           uint32_t* __restrict__ children) {
  const uint32_t i = blockIdx.x * kT + threadIdx.x;
  if (i >= 4 * s.m || pkey[i] == ~uint64_t{0}) return;
  const uint32_t g = (uint32_t)(pkey[i] >> 32);
  uint32_t lo = 0, hi = i;  // first entry of the group
  while (lo < hi) {
    const uint32_t mid = (lo + hi) / 2;
    if (pkey[mid] >> 32 < g) lo = mid + 1;
    else hi = mid;
  }
  children[gs.child[s.fam[s.head[g]]] + (i - lo)] = (uint32_t)pkey[i];
}

// ---- 3. roles and batches --------------------------------------------------------------
// Roles of an order are its births and saddles merged in facade order.
__device__ __forceinline__ uint32_t lower_bound_ev(const uint32_t* __restrict__ ev, uint32_t lo, uint32_t hi, uint32_t x) {
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if (ev[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Event e (rank-partition position) is the birth of order k + 1 and the saddle of order k, for
// k = family_order(e): its role in each, at (own position) + (events of the other kind before it).
// A block's events are consecutive, so the bounds of its first and last event bracket the searches.
__global__ void __launch_bounds__(kT) k_fj_roles(J j, uint32_t nbirths, uint32_t* __restrict__ src,
                                                 uint32_t* __restrict__ rcls) {
  __shared__ uint32_t br[4];  // brackets: births after, saddles before
  const uint32_t e0 = blockIdx.x * kT, e = e0 + threadIdx.x, e1 = min(e0 + kT, j.families) - 1;
  if (e0 >= j.families) return;
  const uint32_t k0 = family_order(j, e0), k1 = family_order(j, e1);
  if (k0 == k1) {
    const uint32_t t = threadIdx.x;
    if (t == 0 || t == 32) {  // as a birth of order k0 + 1: among the saddles of that order
      const uint32_t kb = k0 + 1;
      if (kb <= j.keff) br[t ? 1 : 0] = lower_bound_ev(j.ev, j.fam0[kb], j.fam0[kb + 1], j.ev[t ? e1 : e0]);
    } else if (t == 64 || t == 96) {  // as a saddle of order k0: among the births of that order
      if (k0 > 1) br[t == 64 ? 2 : 3] = lower_bound_ev(j.ev, j.fam0[k0 - 1], j.fam0[k0], j.ev[t == 64 ? e0 : e1]);
    }
  }
  __syncthreads();
  if (e >= j.families) return;
  const uint32_t k = family_order(j, e), x = j.ev[e], c = j.cls[e];
  const bool one = k0 == k1;
  if (e < nbirths) {
    const uint32_t kb = k + 1;
    const uint32_t lo = one ? br[0] : j.fam0[kb], hi = one ? br[1] : j.fam0[kb + 1];
    const uint32_t r = j.role0[kb] + (e - j.fam0[k]) + (lower_bound_ev(j.ev, lo, hi, x) - j.fam0[kb]);
    src[r] = j.n + e;
    rcls[r] = c;
  }
  uint32_t before = j.n;  // order one: every birth is at level 0
  if (k > 1) {
    const uint32_t lo = one ? br[2] : j.fam0[k - 1], hi = one ? br[3] : j.fam0[k];
    before = lower_bound_ev(j.ev, lo, hi, x) - j.fam0[k - 1];
  }
  const uint32_t r = j.role0[k] + (e - j.fam0[k]) + before;
  src[r] = e | kSaddle;
  rcls[r] = c;
}

__global__ void __launch_bounds__(kT) k_fj_singletons(uint32_t n, uint32_t* __restrict__ src, uint32_t* __restrict__ rcls,
                                                      ehgp_forest_node* __restrict__ nodes) {
  const uint32_t p = blockIdx.x * kT + threadIdx.x;
  if (p >= n) return;
  src[p] = p;
  rcls[p] = kNone;  // level 0
  nodes[p] = ehgp_forest_node{1u, kNone, 0u, 0u, 0u, p, kNone};
}

__device__ __forceinline__ uint32_t role_order(const J& j, uint32_t r) {
  uint32_t k = 1;
  while (k < j.keff && r >= j.role0[k + 1]) ++k;
  return k;
}

struct BatchIn {  // first role of its batch
  J j;
  const uint32_t* rcls;
  __device__ Sums<1> operator()(uint32_t r) const {
    return Sums<1>{{r == j.role0[role_order(j, r)] || rcls[r] != rcls[r - 1] ? 1u : 0u}};
  }
};
struct BatchOut {
  J j;
  const uint32_t* src;
  uint32_t* first;      // [batches] first role
  uint32_t* fam_batch;  // [families]
  ehgp_role_record* roles;
  ehgp_forest_birth* births;
  ehgp_family_record* fam;
  __device__ void operator()(uint32_t r, const Sums<1>& x, const Sums<1>& e) const {
    const uint32_t b = e.v[0] + x.v[0] - 1u, s = src[r], k = role_order(j, r);
    if (x.v[0]) first[b] = r;
    if (s & kSaddle) {
      const uint32_t f = s & ~kSaddle, fi = j.ev[f], a0 = j.armoff[f];
      roles[r] = ehgp_role_record{b, j.n + fi, 1u};
      fam[f] = ehgp_family_record{fi, j.n + fi, r, b, k, a0, j.armoff[f + 1] - a0};
      fam_batch[f] = b;
    } else {
      const uint32_t proj = s < j.n ? s : j.n + j.ev[s - j.n];
      roles[r] = ehgp_role_record{b, proj, 0u};
      births[s] = ehgp_forest_birth{proj, b, k, s, s < j.n ? s : kNone};
    }
  }
};

__global__ void __launch_bounds__(kT) k_fj_batches(J j, uint32_t nbatch, uint32_t nrole, GroupSums gs,
                                                   const uint32_t* __restrict__ src, const uint32_t* __restrict__ first,
                                                   ehgp_journal_batch* __restrict__ jb, ehgp_forest_batch* __restrict__ fb) {
  __shared__ uint32_t sj[kT * 7], sf[kT * 13];  // odd strides: no bank conflicts
  const uint32_t b0 = blockIdx.x * kT, b = b0 + threadIdx.x;
  if (b < nbatch) {
    const uint32_t r0 = first[b], r1 = b + 1 < nbatch ? first[b + 1] : nrole;
    const uint32_t k = role_order(j, r0), hk = j.han0[k], fk = j.fam0[k], R = j.role0[k];
    // births and saddles of the order before role r
    auto split = [&](uint32_t r, uint32_t& bl, uint32_t& sl) {
      if (r == j.role0[k + 1]) {
        bl = j.han0[k + 1] - hk;
        sl = j.fam0[k + 1] - fk;
        return;
      }
      const uint32_t s = src[r];
      if (s & kSaddle) {
        sl = (s & ~kSaddle) - fk;
        bl = r - R - sl;
      } else {
        bl = s - hk;
        sl = r - R - bl;
      }
    };
    uint32_t bl0, sl0, bl1, sl1;
    split(r0, bl0, sl0);
    split(r1, bl1, sl1);
    const uint32_t nb = bl1 - bl0, ns = sl1 - sl0, s0 = fk + sl0, s1 = fk + sl1;
    const uint32_t lev = hk + bl0 < j.n && nb ? kNone : nb ? j.ev[hk + bl0 - j.n] : j.ev[s0];
    const uint32_t q0 = k == 1 ? bl0 : 0u, q1 = k == 1 ? bl1 : 0u;  // reduced roots of the order-one births
    const uint32_t wj[6] = {k, lev, r0, r1 - r0, nb, ns};
    const uint32_t wf[12] = {k, lev, hk + bl0, nb, s0, ns, gs.g[s0], gs.g[s1] - gs.g[s0],
                             bl0 - (gs.dc[s0] - gs.dc[fk]), q0 - (gs.dp[s0] - gs.dp[fk]),
                             bl1 - (gs.dc[s1] - gs.dc[fk]), q1 - (gs.dp[s1] - gs.dp[fk])};
    for (int w = 0; w < 6; ++w) sj[threadIdx.x * 7 + w] = wj[w];
    for (int w = 0; w < 12; ++w) sf[threadIdx.x * 13 + w] = wf[w];
  }
  __syncthreads();
  const uint32_t cnt = min(nbatch - b0, (uint32_t)kT);
  uint32_t* oj = reinterpret_cast<uint32_t*>(jb + b0);
  uint32_t* of = reinterpret_cast<uint32_t*>(fb + b0);
  for (uint32_t i = threadIdx.x; i < cnt * 6; i += kT) oj[i] = sj[i / 6 * 7 + i % 6];
  for (uint32_t i = threadIdx.x; i < cnt * 12; i += kT) of[i] = sf[i / 12 * 13 + i % 12];
}

// ---- 4. nodes ----------------------------------------------------------------------------
// Created nodes in slot order: their slot, and the sort key (the group's oldest carrier).
__global__ void __launch_bounds__(kT) k_fj_node_keys(J j, Shared s, GroupSums gs, const uint32_t* __restrict__ car,
                                                     const uint32_t* __restrict__ gc, const uint32_t* __restrict__ gp,
                                                     uint32_t* __restrict__ node_slot, uint64_t* __restrict__ key,
                                                     uint32_t* __restrict__ val) {
  const uint32_t slot = blockIdx.x * kT + threadIdx.x;
  if (slot >= j.families || gc[slot] == 0 || gp[slot] == 1) return;
  const uint32_t q = s.m ? s.slot_q[slot] : kNone, i = gs.node[slot];
  uint32_t oldest;
  if (q != kNone) {
    oldest = s.oldest[s.gid[q]];
  } else {
    oldest = kNone;
    for (uint32_t a = j.armoff[slot]; a < j.armoff[slot + 1]; ++a) oldest = min(oldest, car[a]);
  }
  node_slot[i] = slot;
  key[i] = oldest;
  val[i] = i;
}

__global__ void __launch_bounds__(kT) k_fj_node_ranges(uint32_t m, const uint32_t* __restrict__ v0,
                                                       const uint32_t* __restrict__ v1, const uint64_t* __restrict__ k0,
                                                       const uint64_t* __restrict__ k1, const uint32_t* __restrict__ state,
                                                       int passes, const uint32_t* __restrict__ cls,
                                                       const uint32_t* __restrict__ node_slot, uint2* range,
                                                       uint32_t* __restrict__ node_cls, uint32_t* __restrict__ node_idx) {
  const uint32_t i = blockIdx.x * kT + threadIdx.x;
  if (i >= m) return;
  const bool second = state[2 * passes] != 0;
  const uint64_t* key = second ? k1 : k0;
  const uint32_t v = (second ? v1 : v0)[i], h = (uint32_t)key[i];
  node_idx[i] = v;
  node_cls[i] = cls[node_slot[v]];  // a batch's slots share its class
  if (i == 0 || (uint32_t)key[i - 1] != h) range[h].x = i;
  if (i + 1 == m || (uint32_t)key[i + 1] != h) range[h].y = i + 1;
}

// ---- 5. saddle, group, node and binding records ----------------------------------------------
__global__ void __launch_bounds__(kT) k_fj_records(J j, Tree t, Shared s, GroupSums gs, const uint32_t* __restrict__ car,
                                                   const uint32_t* __restrict__ gc, const uint32_t* __restrict__ gp,
                                                   const uint32_t* __restrict__ fam_batch,
                                                   const ehgp_journal_batch* __restrict__ jb,
                                                   ehgp_forest_binding* __restrict__ bindings,
                                                   ehgp_forest_saddle* __restrict__ saddles,
                                                   ehgp_forest_group* __restrict__ groups,
                                                   ehgp_forest_node* __restrict__ nodes, uint32_t* __restrict__ children,
                                                   uint32_t* __restrict__ err) {
  // the records are written through shared memory: 36- and 44-byte rows leave as whole lines
  __shared__ uint32_t ss[kT * 9], sg[kT * 11];
  const uint32_t s0 = blockIdx.x * kT, slot = s0 + threadIdx.x;
  const uint32_t send = min(s0 + kT, j.families);
  const uint32_t g0 = gs.g[s0], gend = gs.g[send];
  if (slot < j.families) {
    const uint32_t q = s.m ? s.slot_q[slot] : kNone;
    const uint32_t f = q != kNone ? s.sorted[q] : slot;
    const uint32_t cls = j.cls[f], a0 = j.armoff[f], a1 = j.armoff[f + 1], b = fam_batch[f];
    const uint32_t out0 = q != kNone ? s.armoff[q] : a0;
    uint32_t d[4], prior[4];
    const int m = distinct_carriers(car, a0, a1, d);
    uint32_t np = 0;
    for (int i = 0; i < m; ++i) {
      prior[i] = kNone;
      if (touched_before(t, d[i], cls)) {
        prior[i] = reduced_root(t, d[i], cls);
        ++np;
        if (prior[i] == kNone) atomicOr(err, kErrNoRoot);
      }
    }
    for (uint32_t a = a0; a < a1; ++a) {
      const uint32_t c = car[a];
      uint32_t p = kNone;
      for (int i = 0; i < m; ++i)
        if (d[i] == c) p = prior[i];
      reinterpret_cast<uint4*>(bindings)[out0 + (a - a0)] = make_uint4(a, f, c, p);
    }
    const uint32_t grp = gs.g[slot] - (gc[slot] == 0 ? 1u : 0u);
    const uint32_t ws[9] = {f, j.ev[f], b, out0, a1 - a0, (uint32_t)m, (uint32_t)m - np, np, grp};
    for (int w = 0; w < 9; ++w) ss[threadIdx.x * 9 + w] = ws[w];
    if (gc[slot]) {  // first saddle of its group
      const uint32_t fc = gc[slot], fp = gp[slot], kind = fp == 1 ? 1u : fp == 0 ? 0u : 2u;
      const uint32_t child = gs.child[slot], nchild = kind == 2 ? fp : 0u;
      const uint32_t created = kind == 1 ? kNone : j.n + gs.node[slot];
      uint32_t result = created, count = 1;
      if (q != kNone) {
        count = s.saddles[s.gid[q]];
        if (kind == 1) result = reduced_root(t, s.one[s.gid[q]], cls);
      } else {
        // ascending reduced roots
        for (int i = 1; i < m; ++i) {
          const uint32_t x = prior[i];
          int p = i;
          while (p > 0 && prior[p - 1] > x) {
            prior[p] = prior[p - 1];
            --p;
          }
          prior[p] = x;
        }
        if (kind == 1) result = prior[0];
        for (uint32_t i = 0; i < nchild; ++i) children[child + i] = prior[i];
      }
      const uint32_t wg[11] = {b, slot, count, fc, fc - fp, fp, child, nchild, created, result, kind};
      for (int w = 0; w < 11; ++w) sg[(grp - g0) * 11 + w] = wg[w];
      if (kind != 1)
        nodes[created] = ehgp_forest_node{family_order(j, f), jb[b].level_event, kind == 0 ? 1u : 2u, child, nchild,
                                          kNone, grp};
    }
  }
  __syncthreads();
  uint32_t* os = reinterpret_cast<uint32_t*>(saddles + s0);
  for (uint32_t i = threadIdx.x; i < (send - s0) * 9; i += kT) os[i] = ss[i];
  uint32_t* og = reinterpret_cast<uint32_t*>(groups + g0);
  for (uint32_t i = threadIdx.x; i < (gend - g0) * 11; i += kT) og[i] = sg[i];
}

// ---- 6. vertical maps and final roots ----------------------------------------------------------
// The first carrier of a node's group is a birth of its order, and the same event is a saddle one
// order down; the image is the reduced root, on the closed cut at the node's level, of the
// component that saddle's arms lie in.
__global__ void __launch_bounds__(kT) k_fj_vertical(J j, Tree t, Shared s, uint32_t first, uint32_t total,
                                                    const uint32_t* __restrict__ node_slot,
                                                    const uint32_t* __restrict__ car,
                                                    const ehgp_forest_node* __restrict__ nodes,
                                                    ehgp_vertical_assignment* __restrict__ vert,
                                                    uint32_t* __restrict__ err) {
  const uint32_t i = first + blockIdx.x * kT + threadIdx.x;
  if (i >= total) return;
  const uint32_t slot = node_slot[i], q = s.m ? s.slot_q[slot] : kNone, f = q != kNone ? s.sorted[q] : slot;
  const uint32_t cls = j.cls[f], below = car[j.armoff[f]] - j.n;
  const uint32_t c = carrier_after(t, j.term[j.armoff[below]], cls);
  const uint32_t root = reduced_root(t, c, (uint64_t)cls + 1);
  if (root == kNone) atomicOr(err, kErrNoRoot);
  reinterpret_cast<uint4*>(vert)[i - first] =
      make_uint4(j.n + i, root, family_order(j, f), nodes[j.n + i].level_event);
}

__global__ void __launch_bounds__(kT) k_fj_roots(J j, Tree t, ehgp_forest_root* __restrict__ roots, uint32_t cap,
                                                 uint32_t* __restrict__ count) {
  const uint32_t h = blockIdx.x * kT + threadIdx.x;
  if (h >= j.handles || t.dead[h].y != kNone || !(h < j.n || t.touch[h] != kNone)) return;
  const uint32_t at = atomicAdd(count, 1u);
  if (at < cap)
    roots[at] = ehgp_forest_root{h < j.n ? 1u : family_order(j, h - j.n) + 1u, h, reduced_root(t, h, uint64_t{1} << 32)};
}

}  // namespace

uint64_t journal_bytes(const JournalIn& in) {
  const uint64_t F = in.families, H = in.handles, A = in.arms, R = H + F;
  return H * (8 + 4 + 4 + 8 + 4 + 4 + 4 + sizeof(ehgp_forest_birth)) + F * (2 * 20 + 8 + 20 + 4) + A * (4 + 16) +
         F * (sizeof(ehgp_family_record) + sizeof(ehgp_forest_saddle) + sizeof(ehgp_forest_group)) +
         R * (12 + sizeof(ehgp_role_record) + sizeof(ehgp_journal_batch) + sizeof(ehgp_forest_batch)) + (1u << 20);
}

int journal_run(Ctx& ctx, const JournalIn& in, DeviceArena& mem, JournalOut& out, uint64_t* launches) {
  cudaStream_t st = ctx.stream;
  const uint32_t F = in.families, H = in.handles, A = in.arms, R = H + F;
  out = JournalOut{};
  cudaError_t e = cudaSuccess;
  auto no_memory = [&] {
    cudaGetLastError();
    return abi_fail(&ctx, EHGP_ERR_OUT_OF_MEMORY, "the forest journal does not fit the device");
  };
#define TAKE(p, c) \
  if ((e = mem.take(&(p), (c))) != cudaSuccess) return no_memory()
#define TAKE_RECORD(p, c) \
  if ((e = mem.take_record(&(p), (c))) != cudaSuccess) return no_memory()
  if ((uint64_t)H + F >= kSaddle)
    return abi_fail(&ctx, EHGP_ERR_CAPACITY, "the forest journal exceeds 32-bit record indices");
  J j{};
  j.n = in.n;
  j.keff = in.keff;
  j.handles = H;
  j.families = F;
  j.arms = A;
  for (int k = 0; k < kJournalOrders; ++k) {
    j.fam0[k] = in.fam0[k];
    j.han0[k] = in.han0[k];
  }
  j.role0[1] = 0;
  for (uint32_t k = 1; k <= in.keff; ++k)
    j.role0[k + 1] = j.role0[k] + (in.han0[k + 1] - in.han0[k]) + (in.fam0[k + 1] - in.fam0[k]);
  j.ev = in.ev;
  j.cls = in.cls;
  j.armoff = in.armoff;
  j.term = in.term;
  // ---- death tree ----
  Tree t{};
  t.n = in.n;
  uint32_t *lab, *best[2], *cnt, *tot, *car, *gc, *gp;
  Active act[2];
  TAKE(t.dead, H);
  TAKE(t.touch, H);
  TAKE(t.from, H);
  TAKE(t.range, H);
  TAKE(lab, H);
  TAKE(best[0], H);
  TAKE(best[1], H);
  TAKE(cnt, 8);  // [0], [1] active families (ping-pong), [2] errors, [3] saddles sharing a batch, [4] roots,
                 // [5], [6] what the tail left
  TAKE(tot, 5ull * (nblk(R, kScanTile) + 1));
  for (Active& a : act) {
    TAKE(a.comp, F);
    TAKE(a.fam, F);
  }
  TAKE(car, A);
  TAKE(gc, F);
  TAKE(gp, F);
  uint32_t hc[8] = {0};
  auto read = [&](const char* where) -> int {
    if ((e = cudaMemcpyAsync(hc, cnt, sizeof hc, cudaMemcpyDeviceToHost, st)) == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return abi_cuda_fail(&ctx, e, where);
    if (hc[2] & kErrUnborn)
      return abi_fail(&ctx, EHGP_ERR_DEGENERATE, "a strict arm descended to a minimum that is not yet born");
    if (hc[2] & kErrNoRoot)
      return abi_fail(&ctx, EHGP_ERR_DEGENERATE, "a reduced node has no lower-order image through its carrier saddle");
    return EHGP_OK;
  };
  cudaMemsetAsync(cnt, 0, 8 * sizeof(uint32_t), st);
  k_fj_init<<<nblk(H), kT, 0, st>>>(H, t, lab, best[0], best[1]);
  ++*launches;
  uint64_t *ckey[2] = {nullptr, nullptr}, *pkey[2] = {nullptr, nullptr};
  uint32_t *cval[2] = {nullptr, nullptr}, *rcounts = nullptr;
  // sorts m keys; returns the buffers that hold the result
  auto sort = [&](uint64_t m, uint64_t** key, uint32_t** val, int bits, uint64_t** rk, uint32_t** rv, int* passes) -> int {
    RadixScratch rs{rcounts, ctx.radix.state, ctx.radix.wait};
    *passes = radix_sort_kv(st, (uint32_t)m, val[0], val[1], key[0], key[1], bits, rs, launches);
    uint32_t which = 0;
    if ((e = cudaMemcpyAsync(&which, ctx.radix.state + 2 * *passes, 4, cudaMemcpyDeviceToHost, st)) == cudaSuccess)
      e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return abi_cuda_fail(&ctx, e, "forest journal sort");
    *rk = key[which ? 1 : 0];
    *rv = val[which ? 1 : 0];
    return EHGP_OK;
  };
  Shared sh;
  int s;
  if (F) {
    k_fj_first<<<nblk(F, kT * kRows), kT, 0, st>>>(j, act[0], cnt, best[0], cnt + 2);
    ++*launches;
    if ((s = read("forest journal")) != EHGP_OK) return s;
    uint32_t live = hc[0], cur = 0;
    // Three rounds between looks at the count (on most clouds each shrinks it to a half or less).
    for (uint32_t round = 0; live > kTailFamilies && round < in.rounds; round += 3) {
      for (int r = 0; r < 3; ++r) {
        const uint32_t grid = std::min(nblk(live, kT * kRows), 148u * 8);
        k_fj_hook<<<grid, kT, 0, st>>>(j.cls, act[cur], cnt + cur, best[cur], best[1 - cur], t, lab);
        cudaMemsetAsync(cnt + (1 - cur), 0, sizeof(uint32_t), st);
        k_fj_advance<<<grid, kT, 0, st>>>(act[cur], cnt + cur, act[1 - cur], cnt + (1 - cur), best[1 - cur], lab);
        *launches += 2;
        cur = 1 - cur;
      }
      if ((s = read("forest journal rounds")) != EHGP_OK) return s;
      live = hc[cur];
    }
    const bool tail = live <= kTailFamilies;
    if (tail && live) {
      k_fj_tail<<<1, 1024, 0, st>>>(j.cls, act[cur], act[1 - cur], cnt + cur, best[cur], best[1 - cur], t, lab, in.rounds, cnt + 5);
      ++*launches;
    }
    uint2* skip = nullptr;
    auto carriers = [&] {
      t.skip = nullptr;
      k_fj_normalise<<<nblk(H), kT, 0, st>>>(H, t);
      if (skip) {
        k_fj_skips<<<nblk(H), kT, 0, st>>>(H, t, skip);
        ++*launches;
      }
      t.skip = skip;
      k_fj_carriers<<<nblk(F), kT, 0, st>>>(j, t, car, cnt + 3);
      *launches += 2;
      return read("forest journal carriers");
    };
    // (as if the rounds had ended: one look at the counts tells)
    if (tail && (s = carriers()) != EHGP_OK) return s;
    const uint32_t rest = tail && live ? hc[5] : live;
    out.rest = rest;
    if (rest) {
      const Active& a = act[tail ? cur ^ hc[6] : cur];
      for (int i = 0; i < 2; ++i) {
        TAKE(ckey[i], rest);
        TAKE(cval[i], rest);
      }
      TAKE(rcounts, radix_counts_words(rest));
      k_fj_rest_keys<<<nblk(rest), kT, 0, st>>>(rest, a.fam, ckey[0], cval[0]);
      uint64_t* key;
      uint32_t* val;
      int passes;
      if ((s = sort(rest, ckey, cval, 32, &key, &val, &passes)) != EHGP_OK) return s;
      std::vector<uint4> deaths;
      uint4* d_deaths;
      try {
        std::vector<uint4> comp(rest);
        std::vector<uint64_t> keys(rest);
        std::vector<uint32_t> vals(rest);
        cudaMemcpyAsync(comp.data(), a.comp, rest * sizeof(uint4), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(keys.data(), key, rest * sizeof(uint64_t), cudaMemcpyDeviceToHost, st);
        cudaMemcpyAsync(vals.data(), val, rest * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
        if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "forest journal rest");
        deaths_in_order(H, comp, keys, vals, deaths);
      } catch (const std::bad_alloc&) {
        return no_memory();
      }
      const uint32_t m = (uint32_t)deaths.size();
      TAKE(d_deaths, m);
      cudaMemcpyAsync(d_deaths, deaths.data(), m * sizeof(uint4), cudaMemcpyHostToDevice, st);
      k_fj_deaths<<<nblk(m), kT, 0, st>>>(m, j.cls, d_deaths, t);
      *launches += 2;
      TAKE(skip, H);  // a chain of deaths is as long as its components
      // the carriers of the unfinished tree are made again
      cudaMemsetAsync(t.touch, 0xff, H * sizeof(uint32_t), st);
      cudaMemsetAsync(cnt + 3, 0, sizeof(uint32_t), st);
      if ((s = carriers()) != EHGP_OK) return s;
    }
    sh.m = hc[3];
  }
  // ---- batches with several saddles ----
  const uint64_t M = sh.m;
  uint64_t* ck = nullptr;
  if (M) {
    uint32_t* prefix;
    TAKE(sh.fam, M);
    TAKE(sh.slot_q, F);
    TAKE(sh.sorted, M);
    TAKE(sh.gid, M);
    TAKE(sh.armoff, M);
    TAKE(sh.oldest, M);
    TAKE(sh.cars, M);
    TAKE(sh.priors, M);
    TAKE(sh.one, M);
    TAKE(sh.saddles, M);
    TAKE(sh.head, M);
    TAKE(prefix, M);
    for (int i = 0; i < 2; ++i) {
      TAKE(ckey[i], 4 * M);
      TAKE(cval[i], 4 * M);
      TAKE(pkey[i], 4 * M);
    }
    TAKE(rcounts, radix_counts_words(4 * M));
    prefix_sums<1>(st, F, SharedFlagIn{j}, tot, SharedFlagOut{sh.fam, sh.slot_q}, launches);
    prefix_sums<1>(st, (uint32_t)M, RunIn{j, sh.fam}, tot, RunOut{j, t, sh.fam, pkey[0], cval[0]}, launches);
    uint64_t* key;
    uint32_t* val;
    int passes;
    if ((s = sort(M, pkey, cval, 64, &key, &val, &passes)) != EHGP_OK) return s;
    prefix_sums<2>(st, (uint32_t)M, SharedGroupIn{j, sh.fam, key, val}, tot, SharedGroupOut{j, sh, key, val, prefix},
                   launches);
    // the sorted values are in sh.sorted now: cval is free
    k_fj_shared_arms<<<nblk(M), kT, 0, st>>>(j, sh, key, prefix, car, ckey[0], cval[0]);
    ++*launches;
    if ((s = sort(4 * M, ckey, cval, 64, &ck, &val, &passes)) != EHGP_OK) return s;
    k_fj_shared_carriers<<<nblk(4 * M), kT, 0, st>>>(j, t, sh, ck);
    k_fj_shared_groups<<<nblk(M), kT, 0, st>>>(j, t, sh, gc, gp);
    *launches += 2;
  }
  GroupSums gs{};
  TAKE(gs.g, F + 1ull);
  TAKE(gs.node, F + 1ull);
  TAKE(gs.child, F + 1ull);
  TAKE(gs.dc, F + 1ull);
  TAKE(gs.dp, F + 1ull);
  const uint32_t nbt = nblk(F, kScanTile);
  uint32_t ht[5] = {0, 0, 0, 0, 0}, node1 = 0;
  if (F) {
    k_fj_groups<<<nblk(F), kT, 0, st>>>(j, t, car, sh.slot_q, gc, gp);
    ++*launches;
    prefix_sums<5>(st, F, GroupIn{gc, gp}, tot, GroupOut{gs, F - 1}, launches);
    for (int c = 0; c < 5; ++c)
      cudaMemcpyAsync(ht + c, tot + (uint64_t)c * (nbt + 1) + nbt, 4, cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(&node1, gs.node + in.fam0[2], 4, cudaMemcpyDeviceToHost, st);  // nodes of order one
  } else {
    for (uint32_t* p : {gs.g, gs.node, gs.child, gs.dc, gs.dp}) cudaMemsetAsync(p, 0, 4, st);
  }
  // ---- roles and batches ----
  uint32_t *src, *rcls, *first, *fam_batch;
  TAKE(src, R);
  TAKE(rcls, R);
  TAKE(first, R);
  TAKE(fam_batch, F);
  TAKE_RECORD(out.roles, R);
  TAKE_RECORD(out.births, H);
  TAKE_RECORD(out.fam, F);
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "forest journal groups");
  const uint32_t Nn = ht[1];
  out.n_groups = ht[0];
  out.n_nodes = in.n + (uint64_t)Nn;
  out.n_children = ht[2];
  out.n_roles = R;
  out.n_vert = Nn - node1;
  TAKE_RECORD(out.nodes, out.n_nodes);
  TAKE_RECORD(out.children, out.n_children);
  TAKE_RECORD(out.vert, out.n_vert);
  k_fj_singletons<<<nblk(in.n), kT, 0, st>>>(in.n, src, rcls, out.nodes);
  if (F) k_fj_roles<<<nblk(F), kT, 0, st>>>(j, H - in.n, src, rcls);
  *launches += 1 + (F ? 1 : 0);
  prefix_sums<1>(st, R, BatchIn{j, rcls}, tot, BatchOut{j, src, first, fam_batch, out.roles, out.births, out.fam},
                 launches);
  uint32_t nbatch = 0;
  {
    const uint32_t nbr = nblk(R, kScanTile);
    cudaMemcpyAsync(&nbatch, tot + nbr, 4, cudaMemcpyDeviceToHost, st);
  }
  // ---- nodes by oldest handle ----
  uint32_t* node_slot = nullptr;
  TAKE(node_slot, Nn);
  if (Nn) {
    uint64_t* key[2];
    uint32_t *val[2], *ncls, *nidx;
    for (int i = 0; i < 2; ++i) {
      TAKE(key[i], Nn);
      TAKE(val[i], Nn);
    }
    TAKE(ncls, Nn);
    TAKE(nidx, Nn);
    uint32_t* ncounts;
    TAKE(ncounts, radix_counts_words(Nn));
    k_fj_node_keys<<<nblk(F), kT, 0, st>>>(j, sh, gs, car, gc, gp, node_slot, key[0], val[0]);
    int bits = 8;
    while (bits < 32 && (H >> bits)) bits += 8;
    RadixScratch rs{ncounts, ctx.radix.state, ctx.radix.wait};
    const int passes = radix_sort_kv(st, Nn, val[0], val[1], key[0], key[1], bits, rs, launches);
    k_fj_node_ranges<<<nblk(Nn), kT, 0, st>>>(Nn, val[0], val[1], key[0], key[1], ctx.radix.state, passes, j.cls, node_slot,
                                              t.range, ncls, nidx);
    *launches += 2;
    t.node_cls = ncls;
    t.node_idx = nidx;
  }
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "forest journal batches");
  out.n_batches = nbatch;
  TAKE_RECORD(out.jb, out.n_batches);
  TAKE_RECORD(out.fb, out.n_batches);
  TAKE_RECORD(out.bindings, A);
  TAKE_RECORD(out.saddles, F);
  TAKE_RECORD(out.groups, out.n_groups);
  k_fj_batches<<<nblk(nbatch), kT, 0, st>>>(j, nbatch, R, gs, src, first, out.jb, out.fb);
  ++*launches;
  if (F) {
    k_fj_records<<<nblk(F), kT, 0, st>>>(j, t, sh, gs, car, gc, gp, fam_batch, out.jb, out.bindings, out.saddles,
                                         out.groups, out.nodes, out.children, cnt + 2);
    ++*launches;
  }
  if (M) {
    uint64_t* pk;
    uint32_t* val;
    int passes;
    k_fj_shared_prior_keys<<<nblk(4 * M), kT, 0, st>>>(j, t, sh, ck, pkey[0], cval[0]);
    if ((s = sort(4 * M, pkey, cval, 64, &pk, &val, &passes)) != EHGP_OK) return s;
    k_fj_shared_children<<<nblk(4 * M), kT, 0, st>>>(sh, gs, pk, out.children);
    *launches += 2;
  }
  if (out.n_vert) {
    k_fj_vertical<<<nblk(out.n_vert), kT, 0, st>>>(j, t, sh, node1, Nn, node_slot, car, out.nodes, out.vert, cnt + 2);
    ++*launches;
  }
  // ---- final roots (one per surviving component; sorted by node on the host) ----
  for (uint32_t cap = 4096;;) {
    ehgp_forest_root* roots;
    TAKE(roots, cap);
    cudaMemsetAsync(cnt + 4, 0, sizeof(uint32_t), st);
    k_fj_roots<<<nblk(H), kT, 0, st>>>(j, t, roots, cap, cnt + 4);
    ++*launches;
    if ((s = read("forest journal roots")) != EHGP_OK) return s;
    if (hc[4] <= cap) {
      out.roots.resize(hc[4]);
      if (hc[4] && (e = cudaMemcpy(out.roots.data(), roots, hc[4] * sizeof(ehgp_forest_root), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return abi_cuda_fail(&ctx, e, "forest journal roots");
      break;
    }
    cap = hc[4];
  }
#undef TAKE
#undef TAKE_RECORD
  std::sort(out.roots.begin(), out.roots.end(),
            [](const ehgp_forest_root& x, const ehgp_forest_root& y) { return x.node < y.node; });
  return EHGP_OK;
}

}  // namespace ehgp
