// Pair critical-sphere supports (rank <= s_max) on sm_100a.
//
// Reference semantics (Ludwig-H/E-HGP, morsehgp3d/):
//  build_exact_pair_support_stream (include/morsehgp3d/hierarchy/pair_support_stream.hpp:415)
//  with its leaf rule classify_leaf_pair / classify_sparse_closed_ball
//  (src/cpu/hierarchy/pair_support_stream.cpp:1781-2094):
//   * the sphere of a pair (u, v) is its diametral sphere: centre (u + v) / 2,
//     squared level |u - v|^2 / 4;
//   * w is strictly inside iff (w - u).(w - v) < 0, on the sphere iff = 0;
//   * the pair is relevant iff its strict interior count I <= s_max - 2, where
//     s_max = min(min(K, n) + 1, n);
//   * a shell of exactly {u, v} gives an event (closed rank I + 2), a larger
//     shell gives an extra-shell diagnostic with the complete shell count and
//     the least extra shell PointId;
//   * records are in (u, v) order (event_less, pair_support_stream.cpp:120-130).
//
// B200 design (replacing the reference's CPU frontier of node pairs with BigInt
// bounds, pair_support_stream.cpp:1518-2249):
//  * every point u owns a witness list W_u = its 64 nearest other points
//    (FP64 order); R_u^2 is the 64th squared distance;
//  * one warp per u, in Morton order, walks the LBVH over partners v that
//    follow u in Morton order (each unordered pair is visited once), 32 nodes a
//    step, one per lane; a walk that grows long hands the rest of its stack to
//    further warps (points at the rim of a cluster have walks hundreds of times
//    the usual length);
//  * a subtree B of partners is pruned when at least s_max - 1 witnesses w of
//    u satisfy max_{v in B} (w - u).(w - v) < 0 with certainty (binary32
//    bound with a conservative margin): every pair (u, v in B) then has more
//    than s_max - 2 strict interior points;
//  * a leaf pair whose sphere lies in the strict 64-NN ball of u or of v
//    (|u - v| < R_u: every point of the closed diametral ball is within |u - v|
//    of u) is classified from that witness list alone; any other leaf pair is
//    dropped when enough witnesses of u or of v lie inside its sphere for
//    certain, and else runs an exact closed-ball query over the LBVH with early
//    rejection;
//  * every side decision is FP64 with a rigorous error bound, then exact
//    integers at the cloud scale inside the bound.
#include "ehgp_internal.cuh"
#include "ehgp_exact.cuh"

#include <cstring>

namespace ehgp {
namespace {

constexpr int kThreads = 128;
constexpr int kPairsBlocks = 5;  // resident blocks of k_pairs that the registers are shared out for (see there)
constexpr uint32_t kStack = 512; // warp traversal stack
// While the stack holds more than this, one node is taken per step: depth first, a walk adds at
// most the tree's depth (63 + log2 n + 1) to it.
constexpr uint32_t kStackWide = kStack - 64 - 128;
constexpr int kW = 64;           // witnesses per point (two per lane)
constexpr int kMaxInterior = 9;  // s_max - 2 for K >= 10

__host__ __device__ inline uint32_t nblocks(uint64_t n, int t = kThreads) {
  const uint64_t b = (n + t - 1) / t;
  return b == 0 ? 1u : (uint32_t)b;
}

__device__ __forceinline__ uint64_t dbits(double v) { return (uint64_t)__double_as_longlong(v); }

__device__ __forceinline__ TNode load_node(const TNode* __restrict__ tn, uint32_t i) {
  const float4* p = reinterpret_cast<const float4*>(tn + i);
  const float4 a = __ldg(p), b = __ldg(p + 1);
  TNode t;
  t.lo[0] = a.x; t.lo[1] = a.y; t.lo[2] = a.z; t.left = __float_as_uint(a.w);
  t.hi[0] = b.x; t.hi[1] = b.y; t.hi[2] = b.z; t.right = __float_as_uint(b.w);
  return t;
}

__device__ __forceinline__ double d2fp(double ax, double ay, double az, double bx, double by, double bz) {
  const double dx = ax - bx, dy = ay - by, dz = az - bz;
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ double box_lb(const TNode& t, double qx, double qy, double qz) {
  const double dx = fmax(fmax((double)t.lo[0] - qx, qx - (double)t.hi[0]), 0.0);
  const double dy = fmax(fmax((double)t.lo[1] - qy, qy - (double)t.hi[1]), 0.0);
  const double dz = fmax(fmax((double)t.lo[2] - qz, qz - (double)t.hi[2]), 0.0);
  return (dx * dx + dy * dy + dz * dz) * (1.0 - 4.0 * kDistRelErr);
}

__device__ __forceinline__ double box_ub(const TNode& t, double qx, double qy, double qz) {
  const double dx = fmax(fabs((double)t.lo[0] - qx), fabs((double)t.hi[0] - qx));
  const double dy = fmax(fabs((double)t.lo[1] - qy), fabs((double)t.hi[1] - qy));
  const double dz = fmax(fabs((double)t.lo[2] - qz), fabs((double)t.hi[2] - qz));
  return (dx * dx + dy * dy + dz * dz) * (1.0 + 4.0 * kDistRelErr);
}

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

constexpr int kWarpsPerBlock = kThreads / 32;

// ---- 64 nearest neighbours (FP64 order; witnesses, no exactness needed) --------
// One warp per point.  The 64 nearest points so far are kept sorted across the warp (lane l holds
// the l-th and the (32 + l)-th); candidates are collected 32 at a time and merged in.  The walk takes
// 32 nodes of a shared stack per step, and is pruned from the start at the largest distance to
// 64 points next to u in Morton order.
// Bound: latency of the walk's dependent node loads.  A thread per point with its list in local
// memory took 5.69 ms on 29,791 lattice points and 2.40 on 8,009 clustered ones; this 0.51 and 0.17.
struct DistId {
  double d;
  uint32_t id;
};
__device__ __forceinline__ DistId shfl_xor(const DistId& x, int o) {
  return DistId{__shfl_xor_sync(0xffffffffu, x.d, o), __shfl_xor_sync(0xffffffffu, x.id, o)};
}
__device__ __forceinline__ DistId lesser(const DistId& a, const DistId& b) { return b.d < a.d ? b : a; }
__device__ __forceinline__ DistId greater_of(const DistId& a, const DistId& b) { return b.d < a.d ? a : b; }

// Ascending order of a bitonic sequence (one element per lane).
__device__ __forceinline__ DistId bitonic_merge(DistId x, uint32_t lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const DistId o = shfl_xor(x, j);
    const bool take = ((lane & j) == 0) ? o.d < x.d : x.d < o.d;
    if (take) x = o;
  }
  return x;
}
__device__ __forceinline__ DistId bitonic_sort(DistId x, uint32_t lane) {
#pragma unroll
  for (uint32_t k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      const DistId o = shfl_xor(x, j);
      const bool up = ((lane & j) == 0) == ((lane & k) == 0 || k == 32);
      if (up ? o.d < x.d : x.d < o.d) x = o;
    }
  return x;
}

struct KnnShared {
  uint32_t stack[kStack];
  double cd[64];
  uint32_t cid[64];
};

__global__ void __launch_bounds__(kThreads)
k_witness_knn(uint32_t n, uint32_t kw, uint32_t root, const TNode* __restrict__ tn,
              const uint32_t* __restrict__ leaf_pid, const double* __restrict__ px, const double* __restrict__ py,
              const double* __restrict__ pz, uint32_t* __restrict__ W, double* __restrict__ R2,
              uint32_t* __restrict__ err) {
  __shared__ KnnShared shared[kWarpsPerBlock];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t pos = blockIdx.x * kWarpsPerBlock + warp;
  if (pos >= n) return;
  KnnShared& sh = shared[warp];
  const uint32_t p = leaf_pid[pos];
  const double qx = px[p], qy = py[p], qz = pz[p];
  if (n - 1 <= (uint32_t)kW) {  // every other point is a witness (kw = n - 1)
    for (uint32_t j = lane; j < (uint32_t)kW; j += 32)
      W[(uint64_t)p * kW + j] = j < n - 1 ? leaf_pid[j < pos ? j : j + 1] : kInvalid32;
    if (lane == 0) R2[p] = INFINITY;
    return;
  }
  double seed = 0.0;  // at least 64 points lie within it
  const uint32_t w0 = min(pos > 32u ? pos - 32u : 0u, n - 65u);
  for (uint32_t j = lane; j <= 64; j += 32) {
    const uint32_t q = leaf_pid[w0 + j];
    seed = fmax(seed, d2fp(qx, qy, qz, px[q], py[q], pz[q]));
  }
  for (int o = 16; o > 0; o >>= 1) seed = fmax(seed, __shfl_xor_sync(0xffffffffu, seed, o));
  DistId lo{INFINITY, kInvalid32}, hi{INFINITY, kInvalid32};
  double thr = seed;
  uint32_t top = 1, cnt = 0;
  if (lane == 0) sh.stack[0] = root;
  __syncwarp();
  auto merge = [&](uint32_t m) {  // the first m <= 32 collected candidates
    DistId x{INFINITY, kInvalid32};
    if (lane < m) x = DistId{sh.cd[lane], sh.cid[lane]};
    x = bitonic_sort(x, lane);
    x = shfl_xor(x, 31);                            // descending
    hi = bitonic_merge(lesser(hi, x), lane);        // the 32 least of the upper half and the new ones
    const DistId r = shfl_xor(hi, 31);
    const DistId l2 = lesser(lo, r);
    hi = bitonic_merge(greater_of(lo, r), lane);
    lo = bitonic_merge(l2, lane);
    thr = fmin(seed, __shfl_sync(0xffffffffu, hi.d, 31));
  };
  while (top > 0) {
    const uint32_t batch = top > kStackWide ? 1u : min(top, 32u);
    uint32_t node = kInvalid32;
    if (lane < batch) node = sh.stack[top - 1 - lane];
    __syncwarp();
    top -= batch;
    bool take = false, expand = false;
    double d = 0.0;
    TNode t;
    if (node != kInvalid32) {
      t = load_node(tn, node);
      if (t.left == kInvalid32) {
        if (t.right != p) {
          d = d2fp(qx, qy, qz, px[t.right], py[t.right], pz[t.right]);
          take = d <= thr;
        }
      } else {
        expand = box_lb(t, qx, qy, qz) <= thr;
      }
    }
    const uint32_t tb = __ballot_sync(0xffffffffu, take), eb = __ballot_sync(0xffffffffu, expand);
    if (take) {
      const uint32_t at = cnt + __popc(tb & lanemask_lt());
      sh.cd[at] = d;
      sh.cid[at] = t.right;
    }
    if (expand) {
      const uint32_t at = top + 2 * __popc(eb & lanemask_lt());
      sh.stack[at] = t.right;
      sh.stack[at + 1] = t.left;
    }
    top += 2 * __popc(eb);
    cnt += __popc(tb);
    if (top + 64 > kStack) {  // deeper than an LBVH can be
      if (lane == 0) atomicOr(err, kErrCapacity);
      return;
    }
    __syncwarp();
    if (cnt >= 32) {
      merge(32);
      cnt -= 32;
      __syncwarp();
      if (lane < cnt) {
        sh.cd[lane] = sh.cd[32 + lane];
        sh.cid[lane] = sh.cid[32 + lane];
      }
      __syncwarp();
    }
  }
  if (cnt) merge(cnt);
  W[(uint64_t)p * kW + lane] = lo.id;
  W[(uint64_t)p * kW + 32 + lane] = hi.id;
  // witness radius: every point strictly closer than R2 is in W
  if (lane == 31) R2[p] = hi.d;
}

// ---- exact side of w relative to the diametral sphere of (u, v) ---------------------
struct Pt {
  double x, y, z;
};
__device__ __forceinline__ Pt point(const double* px, const double* py, const double* pz, uint32_t i) {
  return Pt{px[i], py[i], pz[i]};
}

// sign((w - u).(w - v)): -1 strictly inside, 0 on the sphere, +1 outside.
__device__ int diametral_side(const Pt& w, const Pt& u, const Pt& v, uint32_t iw, uint32_t iu, uint32_t iv,
                              const double* px, const double* py, const double* pz, int S) {
  const double t0 = (w.x - u.x) * (w.x - v.x), t1 = (w.y - u.y) * (w.y - v.y), t2 = (w.z - u.z) * (w.z - v.z);
  const double acc = t0 + t1 + t2;
  const double bound = 16.0 * 1.1102230246251565e-16 * (fabs(t0) + fabs(t1) + fabs(t2)) + 1e-300;
  if (acc > bound) return 1;
  if (acc < -bound) return -1;
  const double* P[3] = {px, py, pz};
  WInt<4> s = WInt<4>::zero();
  for (int a = 0; a < 3; ++a) {
    const __int128 xw = fixed_of(dbits(P[a][iw]), S), xu = fixed_of(dbits(P[a][iu]), S),
                   xv = fixed_of(dbits(P[a][iv]), S);
    s = wadd(s, wmul(WInt<4>::from_i128(xw - xu), WInt<4>::from_i128(xw - xv)));
  }
  return s.sign();
}

struct PairRec {
  uint32_t u, v, interior, shell, witness;
  uint32_t ids[kMaxInterior];
  uint32_t pad[2];
};
static_assert(sizeof(PairRec) == 64, "pair record is one 64-byte line");

// ---- warp-per-point enumeration ---------------------------------------------------
// One warp owns one point u; lane l holds witnesses l and l + 32 of W_u.
constexpr int kQueue = 256;       // warp-cooperative ball-query frontier (power of two)
constexpr uint32_t kLeaves = 64;  // partners waiting for their classification
constexpr uint32_t kRecs = 16;    // records waiting to leave with one atomic
// Work a warp does before it hands its stack over: a step looks at 32 nodes or at one partner.
// 8,009 clustered points, K = 10: 29.9 ms with every walk in one warp, one node a step (the longest
// walks ran alone at the end, with a global query for most partners), 7.1 ms like this; lattices,
// whose walks are short, 4.7 ms both ways (29,791 points).
constexpr uint32_t kPairSteps = 128;
// A handed-over walk: Morton position of u, node count, nodes.
constexpr uint32_t kTaskNodes = 6;
struct PairTask {
  uint32_t pos, count, node[kTaskNodes];
};

struct WarpShared {
  float4 wit[kW];                 // scaled w - u (binary32), |w - u|^2
  uint32_t stack[kStack];
  uint32_t queue[kQueue];
  uint32_t ids[kMaxInterior + 64];
  uint32_t leaf[kLeaves + 32];
  PairRec rec[kRecs];
  double su[4];                   // -u and 1, scaled
};

// Appends the ids of flagged lanes (two flags per lane) to sh.ids[base...];
// returns the number appended.  Writes only while the total stays <= cap.
__device__ __forceinline__ uint32_t warp_append(WarpShared& sh, uint32_t base, bool f0, uint32_t id0, bool f1,
                                                uint32_t id1, uint32_t cap) {
  const uint32_t b0 = __ballot_sync(0xffffffffu, f0), b1 = __ballot_sync(0xffffffffu, f1);
  const uint32_t c0 = __popc(b0), total = c0 + __popc(b1);
  if (base + total <= cap) {
    const uint32_t lt = lanemask_lt();
    if (f0) sh.ids[base + __popc(b0 & lt)] = id0;
    if (f1) sh.ids[base + c0 + __popc(b1 & lt)] = id1;
  }
  return total;
}

struct WarpBall {
  uint32_t interior;
  uint32_t shell;    // extra shell points
  uint32_t witness;  // least extra shell id
  bool rejected;
};

// Classifies the two candidates of every lane (w0, w1; kInvalid32 = none).
__device__ __forceinline__ void warp_classify(WarpBall& b, WarpShared& sh, uint32_t w0, uint32_t w1, uint32_t iu,
                                              uint32_t iv, const Pt& u, const Pt& v, const double* px,
                                              const double* py, const double* pz, int S, uint32_t cap) {
  int s0 = 1, s1 = 1;
  if (w0 != kInvalid32 && w0 != iu && w0 != iv)
    s0 = diametral_side(point(px, py, pz, w0), u, v, w0, iu, iv, px, py, pz, S);
  if (w1 != kInvalid32 && w1 != iu && w1 != iv)
    s1 = diametral_side(point(px, py, pz, w1), u, v, w1, iu, iv, px, py, pz, S);
  const uint32_t added = warp_append(sh, b.interior, s0 < 0, w0, s1 < 0, w1, cap);
  b.interior += added;
  if (b.interior > cap) b.rejected = true;
  const uint32_t sb0 = __ballot_sync(0xffffffffu, s0 == 0), sb1 = __ballot_sync(0xffffffffu, s1 == 0);
  b.shell += __popc(sb0) + __popc(sb1);
  const uint32_t mw = min(s0 == 0 ? w0 : kInvalid32, s1 == 0 ? w1 : kInvalid32);
  b.witness = min(b.witness, __reduce_min_sync(0xffffffffu, mw));
}

// Warp-cooperative exact closed-ball query over the LBVH (breadth-first over
// the subtrees that straddle the sphere, 32 nodes per step), early rejection.
__device__ void warp_ball_query(WarpBall& b, WarpShared& sh, uint32_t iu, uint32_t iv, const Pt& u, const Pt& v,
                                uint32_t root, const TNode* tn, const uint32_t* leaf_pid, const uint32_t* n_begin,
                                const uint32_t* n_end, const double* px, const double* py, const double* pz, int S,
                                uint32_t cap, uint32_t* err, unsigned long long& nodes_seen) {
  const uint32_t lane = threadIdx.x & 31u;
  const double mx = 0.5 * (u.x + v.x), my = 0.5 * (u.y + v.y), mz = 0.5 * (u.z + v.z);
  const double r2 = 0.25 * d2fp(u.x, u.y, u.z, v.x, v.y, v.z);
  const double r2_hi = r2 * (1.0 + 8.0 * kDistRelErr) + 1e-300, r2_lo = r2 * (1.0 - 8.0 * kDistRelErr);
  uint32_t head = 0, tail = 1;
  if (lane == 0) sh.queue[0] = root;
  __syncwarp();
  while (head < tail && !b.rejected) {
    const uint32_t batch = min(tail - head, 32u);
    nodes_seen += batch;
    uint32_t node = kInvalid32;
    if (lane < batch) node = sh.queue[(head + lane) & (kQueue - 1)];
    __syncwarp();
    uint32_t leafw = kInvalid32, bulk_b = 0, bulk_e = 0;
    bool expand = false;
    TNode t;
    if (node != kInvalid32) {
      t = load_node(tn, node);
      if (t.left == kInvalid32) {
        leafw = t.right;
      } else if (box_lb(t, mx, my, mz) <= r2_hi) {
        if (box_ub(t, mx, my, mz) < r2_lo) {
          bulk_b = n_begin[node];
          bulk_e = n_end[node];
        } else {
          expand = true;
        }
      }
    }
    warp_classify(b, sh, leafw, kInvalid32, iu, iv, u, v, px, py, pz, S, cap);
    // whole subtrees strictly inside
    uint32_t bulk_total = bulk_e - bulk_b;
    for (int off = 16; off > 0; off >>= 1) bulk_total += __shfl_xor_sync(0xffffffffu, bulk_total, off);
    if (bulk_total) {
      if (b.interior + bulk_total > cap) {
        b.rejected = true;
      } else {
        // append the ids lane by lane (at most cap of them in total)
        uint32_t before = bulk_e - bulk_b;
        for (int off = 1; off < 32; off <<= 1) {
          const uint32_t t2 = __shfl_up_sync(0xffffffffu, before, off);
          if ((int)lane >= off) before += t2;
        }
        before -= (bulk_e - bulk_b);
        for (uint32_t q = bulk_b; q < bulk_e; ++q) sh.ids[b.interior + before + (q - bulk_b)] = leaf_pid[q];
        b.interior += bulk_total;
      }
    }
    // children of straddling subtrees
    const uint32_t eb = __ballot_sync(0xffffffffu, expand);
    const uint32_t pushes = 2 * __popc(eb);
    if (tail - head - batch + pushes > kQueue) {
      if (lane == 0) atomicOr(err, kErrCapacity);
      b.rejected = true;
      break;
    }
    if (expand) {
      const uint32_t at = tail + 2 * __popc(eb & lanemask_lt());
      sh.queue[at & (kQueue - 1)] = t.left;
      sh.queue[(at + 1) & (kQueue - 1)] = t.right;
    }
    __syncwarp();
    head += batch;
    tail += pushes;
  }
  __syncwarp();
}

// Writes the warp's finished records: one atomic for all of them (every record of the cloud takes
// its place on one address), whole lines.
__device__ __forceinline__ void flush_records(const WarpShared& sh, uint32_t& kept, PairRec* __restrict__ out,
                                              uint32_t out_cap, uint32_t* __restrict__ counters, uint32_t lane) {
  __syncwarp();
  uint32_t slot = 0;
  if (lane == 0 && kept) slot = atomicAdd(counters, kept);
  slot = __shfl_sync(0xffffffffu, slot, 0);
  const uint32_t room = slot < out_cap ? min(kept, out_cap - slot) : 0u;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(sh.rec);
  uint32_t* dst = reinterpret_cast<uint32_t*>(out + slot);
  for (uint32_t w = lane; w < room * 16; w += 32) dst[w] = src[w];
  kept = 0;
  __syncwarp();
}

// tasks == nullptr: warp i starts the walk of Morton position i at the root; else it goes on with
// tasks[i].  Walks longer than kPairSteps leave the rest of their stack in next[0 .. next_cap).  A
// reservation is never given back (*next_count may end above next_cap): the ranges that warps are
// given are disjoint and leave no slot below min(*next_count, next_cap) unwritten.  What does not fit is
// walked on in place, by a warp that asks no more.
// Bound by the latency of the walk's dependent loads, so the registers are held to five blocks per SM
// (96, against 147 and three): 29,791 lattice points 4.81 -> 3.86 ms, 50,653 at K = 4 3.46 -> 2.55,
// 15,000 mixture points 8.82 -> 7.86; at six blocks 4.02 / 2.67 / 9.00 (the spills cost more); all of these
// with a box per lane in the pruning test.  Now 3.01 / 1.20 ms, and 5.03 on another 15,000-point mixture.
__global__ void __launch_bounds__(kThreads, kPairsBlocks)
k_pairs(uint32_t n, uint32_t cap, uint32_t root, const TNode* __restrict__ tn, const uint32_t* __restrict__ leaf_pid,
        const uint32_t* __restrict__ n_begin, const uint32_t* __restrict__ n_end, const double* __restrict__ px,
        const double* __restrict__ py, const double* __restrict__ pz, const int* __restrict__ scale,
        const uint32_t* __restrict__ W, const double* __restrict__ R2, PairRec* __restrict__ out,
        uint32_t out_cap, uint32_t* __restrict__ counters, unsigned long long* __restrict__ stats,
        uint32_t* __restrict__ err, const PairTask* __restrict__ tasks, uint32_t ntask, PairTask* __restrict__ next,
        uint32_t next_cap, uint32_t* __restrict__ next_count) {
  __shared__ WarpShared shared[kWarpsPerBlock];
  __shared__ unsigned long long s_stats[6];
  if (threadIdx.x < 6) s_stats[threadIdx.x] = 0;
  __syncthreads();
  // work counters (identical in every lane; lane 0 publishes them)
  unsigned long long visits = 0, local_pairs = 0, ball_queries = 0, ball_nodes = 0, emitted = 0;
  uint32_t refused = 0;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t wi = blockIdx.x * kWarpsPerBlock + warp;
  if (wi < (tasks ? ntask : n)) {  // uniform per warp
    WarpShared& sh = shared[warp];
    const uint32_t pos = tasks ? tasks[wi].pos : wi;
    const uint32_t iu = leaf_pid[pos];
    const Pt u = point(px, py, pz, iu);
    const int S = scale[0];
    const double r2u = R2[iu];
    // The binary32 tests work on differences scaled by a power of two that brings the cloud's largest
    // coordinate to 2^30, so that their products neither overflow nor lose their margins to underflow
    // (conversions of denormals and products add up to 2^-117; a witness closer than 2^-48 decides nothing).
    const double f = __hiloint2double((1023 + min(30 - scale[1], 1000)) << 20, 0);
    if (lane < 4) sh.su[lane] = lane == 0 ? -u.x * f : lane == 1 ? -u.y * f : lane == 2 ? -u.z * f : f;
    // this lane's two witnesses of u
    const uint32_t w0 = W[(uint64_t)iu * kW + lane], w1 = W[(uint64_t)iu * kW + 32 + lane];
    float4 a0 = make_float4(0.f, 0.f, 0.f, 0.f), a1 = a0;
    if (w0 != kInvalid32) { a0.x = (float)((px[w0] - u.x) * f); a0.y = (float)((py[w0] - u.y) * f); a0.z = (float)((pz[w0] - u.z) * f); }
    if (w1 != kInvalid32) { a1.x = (float)((px[w1] - u.x) * f); a1.y = (float)((py[w1] - u.y) * f); a1.z = (float)((pz[w1] - u.z) * f); }
    a0.w = a0.x * a0.x + a0.y * a0.y + a0.z * a0.z;
    a1.w = a1.x * a1.x + a1.y * a1.y + a1.z * a1.z;
    if (!(a0.w >= 0x1p-96f)) a0 = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!(a1.w >= 0x1p-96f)) a1 = make_float4(0.f, 0.f, 0.f, 0.f);
    sh.wit[lane] = a0;
    sh.wit[32 + lane] = a1;
    const uint32_t nw = __popc(__ballot_sync(0xffffffffu, w0 != kInvalid32)) +
                        __popc(__ballot_sync(0xffffffffu, w1 != kInvalid32));  // the first nw slots
    const uint32_t need = cap + 1;
    uint32_t top = 1, nleaf = 0, kept = 0, steps = 0;
    bool list_full = false;
    if (tasks) {
      top = min(tasks[wi].count, kTaskNodes);
      if (lane < top) sh.stack[lane] = tasks[wi].node[lane];
    } else if (lane == 0) {
      sh.stack[0] = root;
    }
    __syncwarp();
    const double lo = 1.0 - 4.0 * kDistRelErr, hi = 1.0 + 4.0 * kDistRelErr;
    // Classifies the pair (u, v) with the whole warp and keeps its record when it is relevant.
    auto pair = [&](uint32_t iv) {
      const Pt v = point(px, py, pz, iv);
      const double d2 = d2fp(u.x, u.y, u.z, v.x, v.y, v.z);
      WarpBall b{0u, 0u, kInvalid32, false};
      if (d2 * hi < r2u * lo) {
        ++local_pairs;
        warp_classify(b, sh, w0, w1, iu, iv, u, v, px, py, pz, S, cap);
      } else {
        const uint32_t v0 = W[(uint64_t)iv * kW + lane], v1 = W[(uint64_t)iv * kW + 32 + lane];
        if (d2 * hi < R2[iv] * lo) {
          ++local_pairs;
          warp_classify(b, sh, v0, v1, iu, iv, u, v, px, py, pz, S, cap);
        } else {
          // witnesses of u, or of v, strictly inside this one sphere for certain: enough of them
          // reject the pair without a global query.  (w - u).(w - v) = |e|^2 - e.(q - p) with
          // e = w - p for the end p the witness belongs to and q the other end; the margin
          // covers binary32 differences.
          const double sf = sh.su[3], vx = (v.x - u.x) * sf, vy = (v.y - u.y) * sf, vz = (v.z - u.z) * sf;
          auto inside = [&](double ex, double ey, double ez, double sx, double sy, double sz) {
            const double ee = ex * ex + ey * ey + ez * ez, tx = ex * sx, ty = ey * sy, tz = ez * sz;
            return ee - (tx + ty + tz) < -1e-5 * (ee + fabs(tx) + fabs(ty) + fabs(tz));
          };
          auto of_u = [&](uint32_t w, const float4& a) {
            return w != kInvalid32 && w != iv && inside(a.x, a.y, a.z, vx, vy, vz);
          };
          auto of_v = [&](uint32_t w) {
            return w != kInvalid32 && w != iu && inside((px[w] - v.x) * sf, (py[w] - v.y) * sf, (pz[w] - v.z) * sf, -vx, -vy, -vz);
          };
          const uint32_t cu = __popc(__ballot_sync(0xffffffffu, of_u(w0, a0))) +
                              __popc(__ballot_sync(0xffffffffu, of_u(w1, a1)));
          if (cu >= need) return;
          const uint32_t cv = __popc(__ballot_sync(0xffffffffu, of_v(v0))) + __popc(__ballot_sync(0xffffffffu, of_v(v1)));
          if (cv >= need) return;
          ++ball_queries;
          steps += 8;
          warp_ball_query(b, sh, iu, iv, u, v, root, tn, leaf_pid, n_begin, n_end, px, py, pz, S, cap, err, ball_nodes);
        }
      }
      __syncwarp();
      if (b.rejected || b.interior > cap) return;
      ++emitted;
      // interior ids ascending: lane i holds the i-th, its rank is the number of lesser ids
      const uint32_t mine = lane < b.interior ? sh.ids[lane] : kInvalid32;
      uint32_t rank = 0;
      for (uint32_t i = 0; i < b.interior; ++i) rank += __shfl_sync(0xffffffffu, mine, i) < mine ? 1u : 0u;
      PairRec& r = sh.rec[kept];
      if (lane == 0) {
        r.u = min(iu, iv);
        r.v = max(iu, iv);
        r.interior = b.interior;
        r.shell = b.shell + 2;
        r.witness = b.witness;
        r.pad[0] = r.pad[1] = 0;
      }
      if (lane < b.interior) r.ids[rank] = mine;
      else if (lane < (uint32_t)kMaxInterior) r.ids[lane] = kInvalid32;
      if (++kept == kRecs) flush_records(sh, kept, out, out_cap, counters, lane);
      __syncwarp();
    };
    while (top > 0 || nleaf > 0) {
      if (nleaf >= kLeaves || top == 0) {
        for (uint32_t i = 0; i < nleaf; ++i) pair(sh.leaf[i]);
        steps += nleaf;
        nleaf = 0;
        __syncwarp();
        continue;
      }
      if (steps >= kPairSteps && top > 1 && !list_full) {  // hand the rest over, from the top
        const uint32_t made = (top + kTaskNodes - 1) / kTaskNodes;
        uint32_t at = next_cap;
        if (lane == 0 && *(volatile const uint32_t*)next_count < next_cap) at = atomicAdd(next_count, made);
        at = __shfl_sync(0xffffffffu, at, 0);
        const uint32_t fit = at < next_cap ? min(made, next_cap - at) : 0u;
        for (uint32_t i = lane; i < fit; i += 32) {
          const uint32_t end = top - i * kTaskNodes, begin = end > kTaskNodes ? end - kTaskNodes : 0u;
          PairTask t;
          t.pos = pos;
          t.count = end - begin;
          for (uint32_t j = 0; j < kTaskNodes; ++j) t.node[j] = j < t.count ? sh.stack[begin + j] : 0u;
          next[at + i] = t;
        }
        list_full = fit < made;
        refused = list_full ? 1u : 0u;
        top -= min(top, fit * kTaskNodes);
        __syncwarp();
        continue;
      }
      const uint32_t batch = top > kStackWide ? 1u : min(top, 32u);
      uint32_t node = kInvalid32;
      if (lane < batch) node = sh.stack[top - 1 - lane];
      __syncwarp();
      top -= batch;
      visits += batch;
      ++steps;
      bool open = false;
      TNode t;
      t.left = t.right = kInvalid32;
      float lx = 0.f, ly = 0.f, lz = 0.f, hx = 0.f, hy = 0.f, hz = 0.f;
      if (node != kInvalid32 && n_end[node] > pos + 1) {  // every partner follows u in Morton order
        t = load_node(tn, node);
        open = true;
        const double sx = sh.su[0], sy = sh.su[1], sz = sh.su[2], sf = sh.su[3];
        lx = (float)__fma_rn((double)t.lo[0], sf, sx), ly = (float)__fma_rn((double)t.lo[1], sf, sy);
        lz = (float)__fma_rn((double)t.lo[2], sf, sz), hx = (float)__fma_rn((double)t.hi[0], sf, sx);
        hy = (float)__fma_rn((double)t.hi[1], sf, sy), hz = (float)__fma_rn((double)t.hi[2], sf, sz);
      }
      if (nw >= need) {
        // max over v in box of (w-u).(w-v) = sum_i a_i (a_i - (a_i >= 0 ? lo_i : hi_i)), a = w - u: below 0
        // with certainty for `need` witnesses, no pair of u with the box is relevant.  Two witnesses per lane
        // and one box after another: with a box per lane and one witness after another, the few boxes of a
        // sparse walk cost 64 steps (50,000 points on a line, K = 2: 2.06 ms against 0.38; 50,653 lattice points,
        // K = 4 2.57 against 1.20, 29,791 at K = 10 3.77 against 3.01).
        const float4 w_lo = sh.wit[lane], w_hi = sh.wit[lane + 32];
        for (uint32_t todo = __ballot_sync(0xffffffffu, open); todo; todo &= todo - 1) {
          const uint32_t q = (uint32_t)__ffs((int)todo) - 1;
          const float bx = __shfl_sync(0xffffffffu, lx, q), by = __shfl_sync(0xffffffffu, ly, q),
                      bz = __shfl_sync(0xffffffffu, lz, q), cx = __shfl_sync(0xffffffffu, hx, q),
                      cy = __shfl_sync(0xffffffffu, hy, q), cz = __shfl_sync(0xffffffffu, hz, q);
          auto certain = [&](const float4& a) {
            const float tx = a.x * (a.x - (a.x >= 0.f ? bx : cx));
            const float ty = a.y * (a.y - (a.y >= 0.f ? by : cy));
            const float tz = a.z * (a.z - (a.z >= 0.f ? bz : cz));
            return tx + ty + tz < -1e-5f * (fabsf(tx) + fabsf(ty) + fabsf(tz) + a.w);
          };
          const uint32_t in = __popc(__ballot_sync(0xffffffffu, certain(w_lo))) + __popc(__ballot_sync(0xffffffffu, certain(w_hi)));
          if (lane == q) open = in < need;
        }
      }
      const bool is_leaf = open && t.left == kInvalid32, expand = open && !is_leaf;
      const uint32_t lb = __ballot_sync(0xffffffffu, is_leaf), eb = __ballot_sync(0xffffffffu, expand);
      if (is_leaf) sh.leaf[nleaf + __popc(lb & lanemask_lt())] = t.right;
      nleaf += __popc(lb);
      if (expand) {
        const uint32_t at = top + 2 * __popc(eb & lanemask_lt());
        sh.stack[at] = t.right;
        sh.stack[at + 1] = t.left;
      }
      top += 2 * __popc(eb);
      if (top + 64 > kStack) {  // deeper than an LBVH can be
        if (lane == 0) atomicOr(err, kErrCapacity);
        top = nleaf = 0;
      }
      __syncwarp();
    }
    flush_records(sh, kept, out, out_cap, counters, lane);
  }
  if (lane == 0) {
    atomicAdd(s_stats + 0, visits);
    atomicAdd(s_stats + 1, local_pairs);
    atomicAdd(s_stats + 2, ball_queries);
    atomicAdd(s_stats + 3, ball_nodes);
    atomicAdd(s_stats + 4, emitted);
    if (refused) atomicAdd(s_stats + 5, 1ull);
  }
  __syncthreads();
  if (threadIdx.x < 6 && s_stats[threadIdx.x]) atomicAdd(stats + threadIdx.x, s_stats[threadIdx.x]);
}

__global__ void __launch_bounds__(256)
k_pair_keys(uint32_t m, const PairRec* __restrict__ recs, uint64_t* __restrict__ key, uint32_t* __restrict__ order) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  key[i] = ((uint64_t)recs[i].u << 32) | recs[i].v;
  order[i] = i;
}

__global__ void __launch_bounds__(256)
k_pair_gather(uint32_t m, const uint32_t* __restrict__ vals0, const uint32_t* __restrict__ vals1,
              const uint32_t* __restrict__ state, int passes, const PairRec* __restrict__ recs,
              PairRec* __restrict__ sorted, const double* __restrict__ px, const double* __restrict__ py,
              const double* __restrict__ pz, const int* __restrict__ scale, uint64_t* __restrict__ levelD) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const PairRec r = recs[radix_result(state, passes, vals0, vals1)[i]];
  sorted[i] = r;
  const int S = scale[0];
  __int128 a[3], b[3];
  const double* P[3] = {px, py, pz};
  for (int k = 0; k < 3; ++k) {
    a[k] = fixed_of(dbits(P[k][r.u]), S);
    b[k] = fixed_of(dbits(P[k][r.v]), S);
  }
  const WInt<4> D = exact_dist2(a, b);
  for (int w = 0; w < 4; ++w) levelD[4ull * i + w] = D.w[w];
}

}  // namespace

// Bytes of each record buffer for `c` records: raw, sorted, key, order0, order1, levelD, radix counts.
static void pair_record_bytes(uint64_t c, uint64_t* b) {
  b[0] = c * sizeof(PairRec);
  b[1] = c * sizeof(PairRec);
  b[2] = c * sizeof(uint64_t);
  b[3] = c * sizeof(uint32_t);
  b[4] = c * sizeof(uint32_t);
  b[5] = c * 4 * sizeof(uint64_t);
  b[6] = radix_counts_words(c) * sizeof(uint32_t);
}

cudaError_t pairs_records_alloc(Ctx& ctx, uint64_t capacity) {
  PairBuffers& p = ctx.pb;
  void** bufs[7] = {&p.raw, &p.sorted, (void**)&p.key, (void**)&p.order0, (void**)&p.order1, (void**)&p.levelD,
                    (void**)&p.radix_counts};
  uint64_t old_b[7], new_b[7];
  pair_record_bytes(p.capacity, old_b);
  pair_record_bytes(capacity, new_b);
  for (int i = 0; i < 7; ++i) {
    ctx_free(ctx, *bufs[i], old_b[i]);
    *bufs[i] = nullptr;
  }
  p.capacity = 0;
  for (int i = 0; i < 7; ++i) {
    const cudaError_t e = ctx_alloc(ctx, bufs[i], new_b[i]);
    if (e != cudaSuccess) {
      for (int j = 0; j < i; ++j) {
        ctx_free(ctx, *bufs[j], new_b[j]);
        *bufs[j] = nullptr;
      }
      return e;
    }
  }
  p.capacity = (uint32_t)capacity;
  return cudaSuccess;
}

cudaError_t pairs_alloc(Ctx& ctx) {
  const uint64_t n = ctx.max_points;
  PairBuffers& p = ctx.pb;
  cudaError_t e = cudaSuccess;
#define EHGP_ALLOC(ptr, bytes) \
  if ((e = ctx_alloc(ctx, (void**)&(ptr), (bytes))) != cudaSuccess) return e
  EHGP_ALLOC(p.W, n * kW * sizeof(uint32_t));
  EHGP_ALLOC(p.R2, n * sizeof(double));
  EHGP_ALLOC(p.counters, 8 * sizeof(uint32_t));
  EHGP_ALLOC(p.stats, 8 * sizeof(unsigned long long));
  p.task_cap = p.task_limit = (uint32_t)(2 * n + 4096);  // handed-over walks per round (what does not fit goes on in place)
  EHGP_ALLOC(p.tasks, 2ull * p.task_cap * sizeof(PairTask));
#undef EHGP_ALLOC
  // records: about 38 per point in lattices and uniform clouds; grown on demand
  return pairs_records_alloc(ctx, 48 * n + 1024);
}

// Witness lists + pair enumeration + (u, v) sort.  Returns the record count
// (or a status through ctx on failure).
int pairs_run(Ctx& ctx, uint32_t K, uint32_t* out_count) {
  const uint32_t n = (uint32_t)ctx.built_n;
  PairBuffers& p = ctx.pb;
  LbvhBuffers& b = ctx.lb;
  GeomBuffers& g = ctx.gb;
  cudaStream_t st = ctx.stream;
  const uint32_t keff = K < n ? K : n;
  const uint32_t smax = (keff + 1 < n) ? keff + 1 : n;
  *out_count = 0;
  p.count = 0;
  p.resident = false;
  ++ctx.pair_runs;
  if (smax < 2 || n < 2) {
    p.K = K;
    p.resident = true;
    return EHGP_OK;
  }
  const uint32_t cap = smax - 2;
  if (cap > (uint32_t)kMaxInterior) return abi_fail(&ctx, EHGP_ERR_INVALID_ARGUMENT, "K above 10 is not supported");
  const uint32_t root = 2 * n - 2;
  const uint32_t kw = (n - 1 < (uint32_t)kW) ? n - 1 : (uint32_t)kW;
  uint64_t launches = 0;
  cudaEventRecord(ctx.ev0, st);
  k_witness_knn<<<nblocks(n, kWarpsPerBlock), kThreads, 0, st>>>(n, kw, root, g.tnodes, b.leaf_pid, b.px, b.py, b.pz, p.W, p.R2,
                                                  ctx.d_err);
  ++launches;
  uint32_t hc[2] = {0, 0};
  cudaError_t e = cudaSuccess;
  // count -> allocate -> emit: the enumeration counts every record and writes those that fit;
  // when the count exceeds the buffer, the buffer grows to it and the enumeration runs again
  for (int attempt = 0; attempt < 2; ++attempt) {
    cudaMemsetAsync(p.counters, 0, 8 * sizeof(uint32_t), st);
    cudaMemsetAsync(p.stats, 0, 8 * sizeof(unsigned long long), st);
    cudaEventRecord(ctx.evk0, st);
    unsigned long long hs[8];
    PairTask* task[2] = {(PairTask*)p.tasks, (PairTask*)p.tasks + p.task_cap};
    uint64_t handed = 0;
    uint32_t ntask = 0;  // 0: the walks from the root; then those that were handed over, while there are any
    for (int round = 0;; ++round) {
      const uint32_t warps = round ? ntask : n;
      k_pairs<<<nblocks(warps, kWarpsPerBlock), kThreads, 0, st>>>(
          n, cap, root, g.tnodes, b.leaf_pid, b.n_begin, b.n_end, b.px, b.py, b.pz, g.scale, p.W, p.R2, (PairRec*)p.raw,
          p.capacity, p.counters, p.stats, ctx.d_err, round ? task[round & 1] : nullptr, ntask, task[(round + 1) & 1],
          p.task_limit, p.counters + 1);
      ++launches;
      uint32_t hn[2];
      cudaEventRecord(ctx.evk1, st);
      cudaMemcpyAsync(hn, p.counters, sizeof(hn), cudaMemcpyDeviceToHost, st);
      cudaMemcpyAsync(hc + 1, ctx.d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
      cudaMemcpyAsync(hs, p.stats, sizeof(hs), cudaMemcpyDeviceToHost, st);
      e = cudaStreamSynchronize(st);
      if (e != cudaSuccess) return abi_cuda_fail(&ctx, e, "pair enumeration");
      hc[0] = hn[0];
      ntask = hn[1] < p.task_limit ? hn[1] : p.task_limit;
      handed += ntask;
      if (ntask == 0 || hc[1]) break;
      cudaMemsetAsync(p.counters + 1, 0, sizeof(uint32_t), st);
    }
    {
      float kms = 0.f;
      cudaEventElapsedTime(&kms, ctx.evk0, ctx.evk1);
      ctx.kernel_ms = kms;
      for (int i = 0; i < 8; ++i) ctx.kernel_stats[i] = hs[i];
      ctx.kernel_stats[6] = handed;
    }
    if (hc[1]) return abi_device_status(&ctx, hc[1]);
    if (hc[0] <= p.capacity) break;
    if (attempt == 1 || (uint64_t)hc[0] >= 0xffff0000ull)
      return abi_fail(&ctx, EHGP_ERR_CAPACITY, "pair-support records exceed 32-bit record indices");
    if ((e = pairs_records_alloc(ctx, grown_capacity(hc[0]))) != cudaSuccess) {
      cudaGetLastError();
      return abi_fail(&ctx, EHGP_ERR_OUT_OF_MEMORY, "the pair-support records do not fit the device");
    }
    ++ctx.regrowths;
  }
  const uint32_t m = hc[0];
  if (m) {
    k_pair_keys<<<(m + 255) / 256, 256, 0, st>>>(m, (const PairRec*)p.raw, p.key, p.order0);
    RadixScratch rs{p.radix_counts, ctx.radix.state, ctx.radix.wait};
    const IndirectKey stage[1] = {{p.key, 0}};
    const int bits[1] = {64};
    const int passes = radix_sort_indirect(st, m, p.order0, p.order1, stage, bits, 1, rs, &launches);
    k_pair_gather<<<(m + 255) / 256, 256, 0, st>>>(m, p.order0, p.order1, ctx.radix.state, passes,
                                                    (const PairRec*)p.raw, (PairRec*)p.sorted, b.px, b.py, b.pz,
                                                    g.scale, p.levelD);
    launches += 2;
  }
  cudaEventRecord(ctx.ev1, st);
  cudaMemcpyAsync(hc + 1, ctx.d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "pair sort");
  if (hc[1]) return abi_device_status(&ctx, hc[1]);
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1);
  ctx.last_ms = ms;
  ctx.last_launches = launches;
  p.count = m;
  p.K = K;
  p.witness_ready = true;
  p.resident = true;
  *out_count = m;
  return EHGP_OK;
}

}  // namespace ehgp

extern "C" {

int ehgp_pairs(ehgp_ctx* ctx, uint32_t K, const ehgp_pairs_out* out) try {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  ctx->last_error.clear();
  if (ctx->poisoned) return ehgp::abi_fail(ctx, EHGP_ERR_POISONED, "the context is poisoned by an earlier CUDA failure");
  if (ctx->built_n == 0) return ehgp::abi_fail(ctx, EHGP_ERR_NOT_BUILT, "ehgp_pairs needs a resident LBVH");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "cudaSetDevice");
  if (!ctx->geom_ready) {
    ehgp::geom_prepare(*ctx, (uint32_t)ctx->built_n);
    if ((e = cudaGetLastError()) != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "traversal preparation");
  }
  if (!ctx->scale_valid)
    return ehgp::abi_fail(ctx, EHGP_ERR_NUMERIC_RANGE, "the cloud exceeds the exact fixed-point range");
  cudaMemsetAsync(ctx->d_err, 0, sizeof(uint32_t), ctx->stream);
  uint32_t m = 0;
  const int s = ehgp::pairs_run(*ctx, K, &m);
  if (s != EHGP_OK) return s;
  if (out && out->count) *out->count = m;
  if (out && out->records && m) {
    if (out->capacity < m) return ehgp::abi_fail(ctx, EHGP_ERR_CAPACITY, "the output capacity is below the record count");
    std::vector<ehgp::CopyOut> list{{(char*)out->records, (const char*)ctx->pb.sorted, (uint64_t)m * 64}};
    if (out->level_num) list.push_back({(char*)out->level_num, (const char*)ctx->pb.levelD, (uint64_t)m * 32});
    e = ehgp::copy_out(*ctx, list);
    if (e != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "pair copy");
  }
  return EHGP_OK;
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

}  // extern "C"
