// Direct Morse hierarchy on sm_100a: terminal facade, Morse event journal,
// saddle arm seeds, strict-arm descent, frozen-root quotient and the batched
// hyper-Kruskal forest journal.
//
// Reference semantics (Ludwig-H/E-HGP, morsehgp3d/):
//  facade   src/cpu/hierarchy/direct_support_terminal.cpp:68-300 — accepted events of
//           arity 2-4 ordered by (exact level, closed rank, interior ids, support ids);
//           birth_order = rank if rank <= K_eff, saddle_order = rank - 1 if 2 <= rank <= K_eff + 1;
//  journal  src/cpu/hierarchy/direct_morse_event_journal.cpp:260-400 — n singleton births
//           (order 1, level 0) plus one role per order, batches of equal (order, exact level);
//  seeds    src/cpu/hierarchy/direct_saddle_arm_seed_journal.cpp:380-420 — one family per
//           saddle role, one arm F_u = (I u U) \ {u} per support point u;
//  forest   src/cpu/hierarchy/direct_morse_forest_journal.cpp:1042-2150 — per batch, strict
//           arms resolved against the pre-batch locator, transitive carrier quotient,
//           q_R = 0 reduced birth, 1 continuation, >= 2 multifusion, then unions and births.
//
// B200 design:
//  * events are assembled, given a rigorous FP64 level interval and sorted on the device
//    (LSD radix over the level bits); only runs whose intervals overlap are settled exactly
//    on the device (2304-bit level comparisons), so the facade order is exact;
//  * a stable partition by closed rank gives every order's births and saddle families in
//    facade order at once; births are hashed by facet on the device;
//  * all strict arms descend in rounds of one step per queued facet: miniball support, LBVH ball
//    query at its centre, the k nearest, the strict level decrease certified, until the facet
//    hits a birth; what binary64 leaves open takes the exact step (miniball by exhaustive exact
//    enumeration, cutoff shell by 832-bit distance comparisons).  The terminal facet does not
//    depend on the locator state (a descent chain only reaches a minimum, and minima of lower
//    level are bound before the arm's batch), so the arms of all batches descend together;
//  * the forest journal over the resolved arms is built on the device (ehgp_journal.cu).
#include "ehgp_internal.cuh"
#include "ehgp_exact.cuh"
#include "ehgp_journal.cuh"
#include "ehgp_sphere.cuh"

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <functional>
#include <map>
#include <memory>
#include <numeric>
#include <vector>


namespace ehgp {

struct HierState;

namespace {

constexpr double kU = 1.1102230246251565e-16;
constexpr double kFilt = 64.0 * kU;
constexpr double kTiny = 1e-300;
constexpr int kMaxFacet = 10;
constexpr int kT = 256;              // threads per block of the elementwise kernels
constexpr int kCandCap = 64;         // ball-query candidates per descent step
constexpr int kDStack = 96;          // LBVH traversal stack per descent thread (depth <= 63 + log2 n + 1)
constexpr uint32_t kSortQueueMin = 1u << 15;  // descent queues at least this long are sorted spatially
constexpr int kDescentSteps = 512;   // descent steps per arm

// Slow-path counters of the descent (read back per call): [0] exhaustive miniball
// enumerations, [1] exact hull signs, [2] exact closed-ball sides, [3] exact level
// conversions, [4] exact band orders, [5] exact cutoff comparisons, [6] strictness
// checks on a cutoff equal to the level.
__device__ unsigned long long g_descent_slow[8];
// LBVH nodes visited by the descent's ball queries, striped over 64 counters by block
// (one atomic per step, spread to keep a single address from serialising them).
constexpr int kVisitStripes = 64;
__device__ unsigned long long g_descent_visits[kVisitStripes];
__device__ __forceinline__ void slow(int i) { atomicAdd(&g_descent_slow[i], 1ull); }

// Descent status of an arm.
enum ArmStatus : uint8_t {
  kArmOk = 0,
  kArmUnresolved = 1,   // canonical top-k choice equals the facet
  kArmPlateau = 2,      // no strict level decrease
  kArmCapacity = 3,     // ball query or traversal capacity
  kArmSteps = 4,        // step budget
  kArmInternal = 5,     // no miniball or inconsistent top-k
};

__host__ __device__ inline uint32_t nblk(uint64_t n, int t) {
  const uint64_t b = (n + t - 1) / t;
  return b == 0 ? 1u : (uint32_t)b;
}

// Device layouts of the support records (ehgp_pairs.cu, ehgp_higher.cu).
struct alignas(16) PairRecD {
  uint32_t u, v, interior, shell, witness;
  uint32_t ids[9];
  uint32_t pad[2];
};
struct alignas(16) HigherRecD {
  uint32_t size;
  uint32_t ids[4];
  uint32_t interior, shell, witness;
  uint32_t iids[8];
};
struct alignas(16) EvRec {
  uint32_t size, ids[4], nint, rank, iids[9];
};
static_assert(sizeof(EvRec) == 64 && sizeof(PairRecD) == 64 && sizeof(HigherRecD) == 64, "64-byte records");

__device__ __forceinline__ TNode load_node(const TNode* __restrict__ tn, uint32_t i) {
  const float4* p = reinterpret_cast<const float4*>(tn + i);
  const float4 a = __ldg(p), b = __ldg(p + 1);
  TNode t;
  t.lo[0] = a.x; t.lo[1] = a.y; t.lo[2] = a.z; t.left = __float_as_uint(a.w);
  t.hi[0] = b.x; t.hi[1] = b.y; t.hi[2] = b.z; t.right = __float_as_uint(b.w);
  return t;
}

__host__ __device__ inline double wdbl(const W& x, int shift) {  // x 2^-shift, relative error ~1e-15
  const bool neg = x.negative();
  const W a = neg ? wneg(x) : x;
  int t = 12;
  while (t > 0 && a.w[t] == 0) --t;
  double v = 0.0;
  for (int i = t; i >= 0 && i >= t - 2; --i) v += ldexp((double)a.w[i], 64 * i - shift);
  return neg ? -v : v;
}

// ---- FP64 circumsphere with uniform error bounds ---------------------------------
// Same bounds as the support kernels: with every difference coordinate bounded by
// M, |computed - exact| <= 64 u m with m of A: 1 (pair), 18 M^4 (triangle), 6 M^3
// (tetrahedron) and of each N coordinate: M (pair), 36 M^5, 18 M^4.
struct FSphere {
  double ax, ay, az;   // ids[0]
  double A, Nx, Ny, Nz;
  double eA, eN;       // error bounds of A and of each N coordinate
  double M;            // difference coordinate bound
};

__device__ void fsphere(const double* __restrict__ px, const double* __restrict__ py, const double* __restrict__ pz,
                        const uint32_t* ids, int size, FSphere& s) {
  s.ax = px[ids[0]];
  s.ay = py[ids[0]];
  s.az = pz[ids[0]];
  double e[3][3];
  double M = 0.0;
#pragma unroll
  for (int j = 1; j < 4; ++j) {
    if (j >= size) continue;
    e[j - 1][0] = px[ids[j]] - s.ax;
    e[j - 1][1] = py[ids[j]] - s.ay;
    e[j - 1][2] = pz[ids[j]] - s.az;
    M = fmax(M, fmax(fabs(e[j - 1][0]), fmax(fabs(e[j - 1][1]), fabs(e[j - 1][2]))));
  }
  M *= (1.0 + 1e-15);
  s.M = M;
  const double M2 = M * M;
  if (size == 1) {
    s.A = 1.0; s.Nx = s.Ny = s.Nz = 0.0; s.eA = 0.0; s.eN = 0.0;
  } else if (size == 2) {
    s.A = 1.0; s.Nx = e[0][0]; s.Ny = e[0][1]; s.Nz = e[0][2];
    s.eA = 0.0; s.eN = 2.0 * kU * M + kTiny;
  } else if (size == 3) {
    const double G11 = (e[0][0] * e[0][0] + e[0][1] * e[0][1]) + e[0][2] * e[0][2];
    const double G22 = (e[1][0] * e[1][0] + e[1][1] * e[1][1]) + e[1][2] * e[1][2];
    const double G12 = (e[0][0] * e[1][0] + e[0][1] * e[1][1]) + e[0][2] * e[1][2];
    const double f1 = G22 * (G11 - G12), f2 = G11 * (G22 - G12);
    s.A = G11 * G22 - G12 * G12;
    s.Nx = f1 * e[0][0] + f2 * e[1][0];
    s.Ny = f1 * e[0][1] + f2 * e[1][1];
    s.Nz = f1 * e[0][2] + f2 * e[1][2];
    s.eA = kFilt * 18.0 * M2 * M2 + kTiny;
    s.eN = kFilt * 36.0 * M2 * M2 * M + kTiny;
  } else {
    const double* e1 = e[0];
    const double* e2 = e[1];
    const double* e3 = e[2];
    const double c23x = e2[1] * e3[2] - e2[2] * e3[1], c23y = e2[2] * e3[0] - e2[0] * e3[2], c23z = e2[0] * e3[1] - e2[1] * e3[0];
    const double c31x = e3[1] * e1[2] - e3[2] * e1[1], c31y = e3[2] * e1[0] - e3[0] * e1[2], c31z = e3[0] * e1[1] - e3[1] * e1[0];
    const double c12x = e1[1] * e2[2] - e1[2] * e2[1], c12y = e1[2] * e2[0] - e1[0] * e2[2], c12z = e1[0] * e2[1] - e1[1] * e2[0];
    const double q1 = (e1[0] * e1[0] + e1[1] * e1[1]) + e1[2] * e1[2];
    const double q2 = (e2[0] * e2[0] + e2[1] * e2[1]) + e2[2] * e2[2];
    const double q3 = (e3[0] * e3[0] + e3[1] * e3[1]) + e3[2] * e3[2];
    s.A = (e1[0] * c23x + e1[1] * c23y) + e1[2] * c23z;
    s.Nx = (q1 * c23x + q2 * c31x) + q3 * c12x;
    s.Ny = (q1 * c23y + q2 * c31y) + q3 * c12y;
    s.Nz = (q1 * c23z + q2 * c31z) + q3 * c12z;
    s.eA = kFilt * 6.0 * M2 * M + kTiny;
    s.eN = kFilt * 18.0 * M2 * M2 + kTiny;
  }
}

// Rigorous interval [lo, hi] of the squared radius |N|^2 / (4 A^2); false when A is not
// bounded away from 0 in FP64.
__device__ bool flevel(const FSphere& s, double& lo, double& hi) {
  const double nn = sqrt(s.Nx * s.Nx + s.Ny * s.Ny + s.Nz * s.Nz);
  const double en = s.eN * 1.7320508075688772;
  const double alo = fabs(s.A) - s.eA, ahi = fabs(s.A) + s.eA;
  if (!(alo > 0.0)) return false;
  const double nlo = fmax(nn - en, 0.0), nhi = nn + en;
  lo = nlo * nlo / (4.0 * ahi * ahi) * (1.0 - 1e-14);
  hi = nhi * nhi / (4.0 * alo * alo) * (1.0 + 1e-14);
  return isfinite(hi);
}

// Exact squared radius converted to FP64 (for ill-conditioned supports): 36-limb free.
__device__ void exact_level_fp(const Cloud& c, const uint32_t* ids, int size, double& lo, double& hi) {
  W A;
  WV N;
  exact_sphere(c, ids, size, A, N);
  // scale both to moderate magnitude: |N|^2 / (4A^2) 2^-2S
  int ta = 12, tn = 12;
  const W aa = A.negative() ? wneg(A) : A;
  while (ta > 0 && aa.w[ta] == 0) --ta;
  const W* comp[3] = {&N.x, &N.y, &N.z};
  int tmax = 0;
  for (int k = 0; k < 3; ++k) {
    const W v = comp[k]->negative() ? wneg(*comp[k]) : *comp[k];
    int t = 12;
    while (t > 0 && v.w[t] == 0) --t;
    tmax = max(tmax, t);
  }
  tn = tmax;
  const int sa = 64 * ta, sn = 64 * tn;
  const double a = wdbl(A, sa);
  const double nx = wdbl(N.x, sn), ny = wdbl(N.y, sn), nz = wdbl(N.z, sn);
  const double r = (nx * nx + ny * ny + nz * nz) / (4.0 * a * a);
  const double L = ldexp(r, 2 * sn - 2 * sa - 2 * c.S);
  lo = L * (1.0 - 1e-13);
  hi = L * (1.0 + 1e-13);
}

// ---- 1. events -------------------------------------------------------------------
__global__ void k_ev_build(uint32_t np, uint32_t nh, const PairRecD* __restrict__ pr, const HigherRecD* __restrict__ hr,
                           const double* __restrict__ px, const double* __restrict__ py,
                           const double* __restrict__ pz, const int* __restrict__ cloud_scale, EvRec* __restrict__ ev,
                           double* __restrict__ lmid, double* __restrict__ lerr, uint64_t* __restrict__ key,
                           uint32_t* __restrict__ diag) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= np + nh) return;
  EvRec r;
  uint32_t shell;
  if (i < np) {
    const PairRecD p = pr[i];
    r.size = 2;
    r.ids[0] = p.u;
    r.ids[1] = p.v;
    r.ids[2] = r.ids[3] = 0;
    r.nint = p.interior;
    for (int j = 0; j < 9; ++j) r.iids[j] = j < (int)p.interior ? p.ids[j] : kInvalid32;
    shell = p.shell;
  } else {
    const HigherRecD h = hr[i - np];
    r.size = h.size;
    for (int j = 0; j < 4; ++j) r.ids[j] = h.ids[j];
    r.nint = h.interior;
    for (int j = 0; j < 9; ++j) r.iids[j] = j < 8 && j < (int)h.interior ? h.iids[j] : kInvalid32;
    shell = h.shell;
  }
  r.rank = r.nint + r.size;
  ev[i] = r;
  if (shell != r.size) {  // relevant extra-shell diagnostic: excluded from the facade
    atomicAdd(diag, 1u);
    key[i] = ~uint64_t{0};
    lmid[i] = INFINITY;
    lerr[i] = 0.0;
    return;
  }
  FSphere s;
  fsphere(px, py, pz, r.ids, (int)r.size, s);
  double lo, hi;
  if (r.size == 2) {
    const double d2 = (s.Nx * s.Nx + s.Ny * s.Ny) + s.Nz * s.Nz;
    lo = 0.25 * d2 * (1.0 - 8.0 * kU);
    hi = 0.25 * d2 * (1.0 + 8.0 * kU);
  } else if (!flevel(s, lo, hi) || hi - lo > 1e-9 * hi) {
    const Cloud c{px, py, pz, cloud_scale[0]};
    exact_level_fp(c, r.ids, (int)r.size, lo, hi);
  }
  const double mid = 0.5 * (lo + hi);
  lmid[i] = mid;
  lerr[i] = 0.5 * (hi - lo) + 1e-15 * mid;
  key[i] = dbits(mid);
}

__global__ void k_ev_gather(uint32_t m, const uint32_t* __restrict__ v0, const uint32_t* __restrict__ v1,
                            const uint32_t* __restrict__ state, int passes, const EvRec* __restrict__ ev,
                            const double* __restrict__ lmid, const double* __restrict__ lerr, EvRec* __restrict__ out,
                            double* __restrict__ omid, double* __restrict__ oerr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint32_t s = radix_result(state, passes, v0, v1)[i];
  out[i] = ev[s];
  omid[i] = lmid[s];
  oerr[i] = lerr[s];
}

// ---- scans (block-local then across blocks) -----------------------------------------
struct OpMax {
  __device__ double operator()(double a, double b) const { return fmax(a, b); }
};
struct OpSum {
  __device__ uint32_t operator()(uint32_t a, uint32_t b) const { return a + b; }
};
struct OpMin {
  __device__ double operator()(double a, double b) const { return fmin(a, b); }
};

// Inclusive prefix max of hi[i] = mid + err (forward) and suffix min of lo = mid - err
// (backward), chunked: one block per 1024 items, then a pass over the blocks' results.
template <class Op>
__global__ void k_scan_blocks(uint32_t m, const double* __restrict__ mid, const double* __restrict__ err, double sgn,
                              int reverse, double* __restrict__ out, double* __restrict__ bsum, Op op, double ident) {
  __shared__ double sh[1024];
  const uint32_t base = blockIdx.x * 1024u;
  for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) {
    const uint32_t j = base + t;
    double v = ident;
    if (j < m) {
      const uint32_t idx = reverse ? m - 1 - j : j;
      v = mid[idx] + sgn * err[idx];
    }
    sh[t] = v;
  }
  __syncthreads();
  for (uint32_t off = 1; off < 1024; off <<= 1) {
    double add[4];
    int c = 0;
    for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) add[c++] = t >= off ? sh[t - off] : ident;
    __syncthreads();
    c = 0;
    for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) {
      sh[t] = op(sh[t], add[c++]);
    }
    __syncthreads();
  }
  for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) {
    const uint32_t j = base + t;
    if (j < m) out[reverse ? m - 1 - j : j] = sh[t];
  }
  if (threadIdx.x == 0) bsum[blockIdx.x] = sh[1023];
}

// Exclusive scan of the block results, in place, by one block: bound by the chain of 1,024-item tiles.
// One thread alone took 0.34 ms for the 4,818 results of 4.9 million events (the four such launches of
// 24.8 million events: 4 ms of the hierarchy call).
template <class T, class Op>
__global__ void __launch_bounds__(1024) k_carry(uint32_t nb, T* __restrict__ bsum, Op op, T ident) {
  __shared__ T w[32];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  T carry = ident;
  for (uint32_t b = 0; b < nb; b += 1024) {
    const uint32_t i = b + threadIdx.x;
    T x = i < nb ? bsum[i] : ident;
    for (int o = 1; o < 32; o <<= 1) {
      const T y = __shfl_up_sync(0xffffffffu, x, o);
      if ((int)lane >= o) x = op(y, x);
    }
    if (lane == 31) w[warp] = x;
    x = __shfl_up_sync(0xffffffffu, x, 1);  // exclusive within the warp
    if (lane == 0) x = ident;
    __syncthreads();
    T y = w[lane];
    for (int o = 1; o < 32; o <<= 1) {  // every warp scans the warps' results
      const T z = __shfl_up_sync(0xffffffffu, y, o);
      if ((int)lane >= o) y = op(z, y);
    }
    const T before = __shfl_sync(0xffffffffu, y, (int)((warp + 31u) & 31u)), all = __shfl_sync(0xffffffffu, y, 31);
    if (i < nb) bsum[i] = op(carry, warp ? op(before, x) : x);
    carry = op(carry, all);
    __syncthreads();
  }
}

template <class Op>
__global__ void k_scan_apply(uint32_t m, int reverse, double* __restrict__ out, const double* __restrict__ bsum,
                             Op op) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t idx = reverse ? m - 1 - j : j;
  out[idx] = op(out[idx], bsum[j / 1024u]);
}

// A boundary between facade positions p - 1 and p is certain when every level
// interval before it lies strictly below every one after it.
__global__ void k_uncertain(uint32_t m, const double* __restrict__ pre_hi, const double* __restrict__ suf_lo,
                            uint32_t* __restrict__ list, uint32_t cap, uint32_t* __restrict__ count) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p == 0 || p >= m) return;
  if (pre_hi[p - 1] < suf_lo[p]) return;
  const uint32_t at = atomicAdd(count, 1u);
  if (at < cap) list[at] = p;
}

__global__ void k_iota(uint32_t m, uint32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) out[i] = i;
}

// ---- exact order inside the runs that the FP64 level intervals leave open ----------
// A run is a maximal range [lo, hi] of facade positions whose intervals overlap.  Each member
// gets its exact level key once (|N|^2 and A^2 of its circumsphere, 2304-bit integers; the
// level is |N|^2 / (4 A^2)), then one thread per run merge-sorts the run's positions by
// (exact level, closed rank, interior ids, support ids) and writes the records back in that
// order with their equal-level flags.
__global__ void k_tie_keys(uint32_t cnt, const uint32_t* __restrict__ pos, const EvRec* __restrict__ ev, Cloud c,
                           WL* __restrict__ knum, WL* __restrict__ ka2) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  const EvRec r = ev[pos[i]];
  W A;
  WV N;
  exact_sphere(c, r.ids, (int)r.size, A, N);
  const WL x = widen<36>(N.x), y = widen<36>(N.y), z = widen<36>(N.z), a = widen<36>(A);
  knum[i] = wadd(wadd(wmul(x, x), wmul(y, y)), wmul(z, z));
  ka2[i] = wmul(a, a);
}

__device__ int tie_level_cmp(const WL* knum, const WL* ka2, uint32_t i, uint32_t j) {
  return wcmp(wmul(knum[i], ka2[j]), wmul(knum[j], ka2[i]));
}

__device__ bool tie_less(const WL* knum, const WL* ka2, const EvRec* rec, uint32_t i, uint32_t j) {
  const int s = tie_level_cmp(knum, ka2, i, j);
  if (s != 0) return s < 0;
  const EvRec& a = rec[i];
  const EvRec& b = rec[j];
  if (a.rank != b.rank) return a.rank < b.rank;
  const uint32_t m = min(a.nint, b.nint);
  for (uint32_t t = 0; t < m; ++t)
    if (a.iids[t] != b.iids[t]) return a.iids[t] < b.iids[t];
  if (a.nint != b.nint) return a.nint < b.nint;
  const uint32_t ms = min(a.size, b.size);
  for (uint32_t t = 0; t < ms; ++t)
    if (a.ids[t] != b.ids[t]) return a.ids[t] < b.ids[t];
  return a.size < b.size;
}

// rec[i], mid[i], err[i]: copies of the member's record and level interval (members of run r are run_off[r] .. run_off[r + 1] - 1,
// at facade positions run_lo[r] ...); idx / tmp: scratch of the member count.
__global__ void k_tie_sort(uint32_t nruns, const uint32_t* __restrict__ run_off, const uint32_t* __restrict__ run_lo,
                           const WL* __restrict__ knum, const WL* __restrict__ ka2, const EvRec* __restrict__ rec,
                           const double* __restrict__ mid, const double* __restrict__ err, uint32_t* __restrict__ idx,
                           uint32_t* __restrict__ tmp, EvRec* __restrict__ ev, double* __restrict__ lmid,
                           double* __restrict__ lerr, uint8_t* __restrict__ eqprev) {
  const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nruns) return;
  const uint32_t b = run_off[r], L = run_off[r + 1] - b;
  for (uint32_t t = 0; t < L; ++t) idx[b + t] = b + t;
  // bottom-up merge sort (stable) of the member indices
  uint32_t* src = idx + b;
  uint32_t* dst = tmp + b;
  for (uint32_t w = 1; w < L; w <<= 1) {
    for (uint32_t lo = 0; lo < L; lo += 2 * w) {
      const uint32_t mid = min(lo + w, L), hi = min(lo + 2 * w, L);
      uint32_t i = lo, j = mid, o = lo;
      while (i < mid && j < hi) dst[o++] = tie_less(knum, ka2, rec, src[j], src[i]) ? src[j++] : src[i++];
      while (i < mid) dst[o++] = src[i++];
      while (j < hi) dst[o++] = src[j++];
    }
    uint32_t* t = src;
    src = dst;
    dst = t;
  }
  const uint32_t p0 = run_lo[r];
  for (uint32_t t = 0; t < L; ++t) {
    ev[p0 + t] = rec[src[t]];
    lmid[p0 + t] = mid[src[t]];  // the level intervals follow their events
    lerr[p0 + t] = err[src[t]];
    if (t > 0) eqprev[p0 + t] = tie_level_cmp(knum, ka2, src[t - 1], src[t]) == 0 ? 1 : 0;
  }
}

// Gathers the facade records of the uncertain runs (the member copies of the tie sort).
__global__ void k_run_gather(uint32_t cnt, const uint32_t* __restrict__ idx, const EvRec* __restrict__ ev,
                             const double* __restrict__ lmid, const double* __restrict__ lerr, EvRec* __restrict__ out,
                             double* __restrict__ omid, double* __restrict__ oerr) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cnt) return;
  out[i] = ev[idx[i]];
  omid[i] = lmid[idx[i]];
  oerr[i] = lerr[idx[i]];
}

// Support records of facade events: out[5i] = size, out[5i + 1..4] = ids (unused 0); an
// index of kInvalid32 (level 0) or past the facade gives size 0.
__global__ void k_event_supports(uint32_t m, const uint32_t* __restrict__ idx, const EvRec* __restrict__ ev,
                                 uint32_t nev, uint32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint32_t e = idx[i];
  const bool ok = e < nev;
  out[5ull * i] = ok ? ev[e].size : 0u;
  for (int j = 0; j < 4; ++j) out[5ull * i + 1 + j] = ok && (uint32_t)j < ev[e].size ? ev[e].ids[j] : 0u;
}

// ---- 2. level classes, rank partition, births -----------------------------------
__global__ void k_level_class(uint32_t m, const uint8_t* __restrict__ eqprev, uint32_t* __restrict__ flag) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < m) flag[p] = (p == 0 || !eqprev[p]) ? 1u : 0u;
}

// Inclusive prefix sum of 32-bit flags (block-local, then carries).
__global__ void k_sum_blocks(uint32_t m, const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                             uint32_t* __restrict__ bsum) {
  __shared__ uint32_t sh[1024];
  const uint32_t base = blockIdx.x * 1024u;
  for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) sh[t] = base + t < m ? in[base + t] : 0u;
  __syncthreads();
  for (uint32_t off = 1; off < 1024; off <<= 1) {
    uint32_t add[4];
    int c = 0;
    for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) add[c++] = t >= off ? sh[t - off] : 0u;
    __syncthreads();
    c = 0;
    for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x) sh[t] += add[c++];
    __syncthreads();
  }
  for (uint32_t t = threadIdx.x; t < 1024; t += blockDim.x)
    if (base + t < m) out[base + t] = sh[t];
  if (threadIdx.x == 0) bsum[blockIdx.x] = sh[1023];
}

__global__ void k_sum_apply(uint32_t m, uint32_t* __restrict__ out, const uint32_t* __restrict__ bsum, int minus1) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) out[j] = out[j] + bsum[j / 1024u] - (minus1 ? 1u : 0u);
}

// Rank keys for the stable partition; the rank histogram is summed per block in shared
// memory (16 bins) before one global add per bin.
__global__ void k_rank_key(uint32_t m, const EvRec* __restrict__ ev, uint64_t* __restrict__ key,
                           uint32_t* __restrict__ iota, uint32_t* __restrict__ hist) {
  __shared__ uint32_t bins[16];
  if (threadIdx.x < 16) bins[threadIdx.x] = 0;
  __syncthreads();
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) {
    const uint32_t r = ev[i].rank;
    key[i] = r;
    iota[i] = i;
    atomicAdd(&bins[r < 15 ? r : 15], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 16 && bins[threadIdx.x]) atomicAdd(&hist[threadIdx.x], bins[threadIdx.x]);
}

__global__ void k_rank_gather(uint32_t m, const uint32_t* __restrict__ v0, const uint32_t* __restrict__ v1,
                              const uint32_t* __restrict__ state, int passes, uint32_t* __restrict__ out) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < m) out[i] = radix_result(state, passes, v0, v1)[i];
}

__device__ __forceinline__ uint32_t facet_hash(const uint32_t* ids, int k) {
  uint64_t h = 0x9E3779B97F4A7C15ull ^ (uint64_t)k;
#pragma unroll
  for (int i = 0; i < kMaxFacet; ++i) {
    if (i >= k) break;
    h ^= ids[i];
    h *= 0xFF51AFD7ED558CCDull;
    h ^= h >> 33;
  }
  h *= 0xC4CEB9FE1A85EC53ull;
  h ^= h >> 33;
  return (uint32_t)h;
}

// I u U, ascending, filled up with kInvalid32: a compare network, so that the words stay in registers.
__device__ __forceinline__ int event_facet(const EvRec& e, uint32_t (&F)[kMaxFacet + 1]) {
#pragma unroll
  for (int j = 0; j <= kMaxFacet; ++j) F[j] = kInvalid32;
  auto put = [&](uint32_t x) {
#pragma unroll
    for (int j = 0; j <= kMaxFacet; ++j) {
      const uint32_t lo = min(F[j], x);
      x = max(F[j], x);
      F[j] = lo;
    }
  };
#pragma unroll
  for (uint32_t j = 0; j < 9; ++j) put(j < e.nint ? e.iids[j] : kInvalid32);
#pragma unroll
  for (uint32_t j = 0; j < 4; ++j) put(j < e.size ? e.ids[j] : kInvalid32);
  return (int)(e.nint + e.size);
}

// Births of orders >= 2: handle = n + position in the rank partition; facets stored
// (10 words, unused = kInvalid32) and hashed (open addressing, handle per slot).
__global__ void k_birth_insert(uint32_t nb, uint32_t n, uint32_t birth_base, const uint32_t* __restrict__ rank_order,
                               const EvRec* __restrict__ ev, uint32_t* __restrict__ bfac, uint32_t* __restrict__ slots,
                               uint32_t mask, uint32_t* __restrict__ err) {
  const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nb) return;
  const uint32_t fi = rank_order[birth_base + b];
  uint32_t F[kMaxFacet + 1];
  const int k = event_facet(ev[fi], F);
  uint2* out = reinterpret_cast<uint2*>(bfac + (uint64_t)b * kMaxFacet);  // 40-byte rows
#pragma unroll
  for (int j = 0; j < kMaxFacet; j += 2) out[j / 2] = make_uint2(F[j], F[j + 1]);
  const uint32_t h = n + b;
  uint32_t s = facet_hash(F, k) & mask;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const uint32_t prev = atomicCAS(&slots[s], kInvalid32, h);
    if (prev == kInvalid32) return;
    s = (s + 1) & mask;
  }
  atomicOr(err, kErrCapacity);
}

// Rank-partition views that the forest journal reads in sequence: level class and support size
// of the event at each rank position.
__global__ void k_rank_info(uint32_t m, const uint32_t* __restrict__ rank_order, const EvRec* __restrict__ ev,
                            const uint32_t* __restrict__ lclass, uint32_t* __restrict__ cls_rp,
                            uint32_t* __restrict__ size_rp) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  const uint32_t fi = rank_order[i];
  cls_rp[i] = lclass[fi];
  size_rp[i] = ev[fi].size;
}

// ---- 3. strict-arm descent ----------------------------------------------------------
struct DescentParams {
  uint32_t n, root;
  const TNode* tn;
  const double* px;
  const double* py;
  const double* pz;
  int S;
  const uint32_t* slots;
  uint32_t mask;
  const uint32_t* bfac;
  uint32_t nbirths;
  const uint32_t* birth_event;  // facade index of the birth of handle n + i
  const double* lmid;           // level intervals of the facade, mid -+ err
  const double* lerr;
};

// A queued facet (64 bytes): its ids, ascending (unused kInvalid32), and what its level must lie
// strictly below: the support of the facet it came from (unused kInvalid32; the first one kInvalid32:
// nothing to check) and the lower end of that one's level interval.
struct __align__(16) QFacet {
  uint32_t F[kMaxFacet];
  uint32_t prev[4];
  double prev_lo;
};
static_assert(sizeof(QFacet) == 64, "four 16-byte words");

__device__ uint32_t probe_facet(const DescentParams& d, const uint32_t* F, int k) {
  if (k == 1) return F[0];  // order-one births are the singletons, handle = PointId
  uint32_t s = facet_hash(F, k) & d.mask;
  for (uint32_t probe = 0; probe <= d.mask; ++probe) {
    const uint32_t h = __ldg(d.slots + s);
    if (h == kInvalid32) return kInvalid32;
    const uint2* f = reinterpret_cast<const uint2*>(d.bfac + (uint64_t)(h - d.n) * kMaxFacet);
    bool eq = true;
#pragma unroll
    for (int j = 0; j < kMaxFacet; j += 2) {
      const uint2 x = __ldg(f + j / 2);
      eq &= x.x == (j < k ? F[j] : kInvalid32) && x.y == (j + 1 < k ? F[j + 1] : kInvalid32);
    }
    if (eq) return h;
    s = (s + 1) & d.mask;
  }
  return kInvalid32;
}

// Exact closed-ball membership of w in the circumsphere of T (side <= 0), FP64 first.
__device__ bool inside_closed(const Cloud& c, const FSphere& fs, const uint32_t* T, int ts, uint32_t w) {
  const double x = c.px[w] - fs.ax, y = c.py[w] - fs.ay, z = c.pz[w] - fs.az;
  const double Mp = fmax(fs.M, fmax(fabs(x), fmax(fabs(y), fabs(z)))) * (1.0 + 1e-15);
  const double q = (x * x + y * y) + z * z;
  const double v = fs.A * q - ((x * fs.Nx + y * fs.Ny) + z * fs.Nz);
  const double M2 = fs.M * fs.M, M4 = M2 * M2;
  const double Am = ts <= 2 ? 1.0 : (ts == 3 ? 18.0 * M4 : 6.0 * M2 * fs.M);
  const double Nm = ts == 1 ? 0.0 : (ts == 2 ? fs.M : (ts == 3 ? 36.0 * M4 * fs.M : 18.0 * M4));
  const double bnd = kFilt * (Am * 3.0 * Mp * Mp + 3.0 * Mp * Nm) + kTiny;
  const int sa = fs.A > fs.eA ? 1 : (fs.A < -fs.eA ? -1 : 0);
  if (sa != 0) {
    if (v * sa < -bnd) return true;
    if (v * sa > bnd) return false;
  }
  slow(2);
  W A;
  WV N;
  exact_sphere(c, T, ts, A, N);
  const WV dq = c.wdiff(w, T[0]);
  const int sd = wsub(wmul(A, wdot(dq, dq)), wdot(dq, N)).sign() * A.sign();
  return sd <= 0;
}

// Exact: the circumcentre of T lies in the closed convex hull of T and T is affinely independent.
__device__ bool hull_centre(const Cloud& c, const uint32_t* T, int ts) {
  if (ts <= 2) return ts == 1 || T[0] != T[1];
  // FP64 signs with the uniform bounds of the support kernels, exact when undecided
  double e[3][3], M = 0.0;
  for (int j = 1; j < ts; ++j) {
    e[j - 1][0] = c.px[T[j]] - c.px[T[0]];
    e[j - 1][1] = c.py[T[j]] - c.py[T[0]];
    e[j - 1][2] = c.pz[T[j]] - c.pz[T[0]];
    M = fmax(M, fmax(fabs(e[j - 1][0]), fmax(fabs(e[j - 1][1]), fabs(e[j - 1][2]))));
  }
  M *= (1.0 + 1e-15);
  const double M2 = M * M;
  int sg[5];
  bool undecided = false;
  auto fs = [&](double v, double b) {
    const int r = v > b ? 1 : (v < -b ? -1 : 2);
    undecided |= r == 2;
    return r;
  };
  if (ts == 3) {
    const double G11 = (e[0][0] * e[0][0] + e[0][1] * e[0][1]) + e[0][2] * e[0][2];
    const double G22 = (e[1][0] * e[1][0] + e[1][1] * e[1][1]) + e[1][2] * e[1][2];
    const double G12 = (e[0][0] * e[1][0] + e[0][1] * e[1][1]) + e[0][2] * e[1][2];
    sg[0] = fs(G12, kFilt * 3.0 * M2 + kTiny);
    sg[1] = fs(G11 - G12, kFilt * 6.0 * M2 + kTiny);
    sg[2] = fs(G22 - G12, kFilt * 6.0 * M2 + kTiny);
    sg[3] = fs(G11 * G22 - G12 * G12, kFilt * 18.0 * M2 * M2 + kTiny);
    if (undecided) { slow(1); tri_signs_exact(c, T, sg); }
    return sg[3] != 0 && sg[0] >= 0 && sg[1] >= 0 && sg[2] >= 0;
  }
  const double* e1 = e[0];
  const double* e2 = e[1];
  const double* e3 = e[2];
  const double c23x = e2[1] * e3[2] - e2[2] * e3[1], c23y = e2[2] * e3[0] - e2[0] * e3[2], c23z = e2[0] * e3[1] - e2[1] * e3[0];
  const double c31x = e3[1] * e1[2] - e3[2] * e1[1], c31y = e3[2] * e1[0] - e3[0] * e1[2], c31z = e3[0] * e1[1] - e3[1] * e1[0];
  const double c12x = e1[1] * e2[2] - e1[2] * e2[1], c12y = e1[2] * e2[0] - e1[0] * e2[2], c12z = e1[0] * e2[1] - e1[1] * e2[0];
  const double q1 = (e1[0] * e1[0] + e1[1] * e1[1]) + e1[2] * e1[2];
  const double q2 = (e2[0] * e2[0] + e2[1] * e2[1]) + e2[2] * e2[2];
  const double q3 = (e3[0] * e3[0] + e3[1] * e3[1]) + e3[2] * e3[2];
  const double detE = (e1[0] * c23x + e1[1] * c23y) + e1[2] * c23z;
  const double Nx = (q1 * c23x + q2 * c31x) + q3 * c12x;
  const double Ny = (q1 * c23y + q2 * c31y) + q3 * c12y;
  const double Nz = (q1 * c23z + q2 * c31z) + q3 * c12z;
  const double l1 = (Nx * c23x + Ny * c23y) + Nz * c23z;
  const double l2 = (Nx * c31x + Ny * c31y) + Nz * c31z;
  const double l3 = (Nx * c12x + Ny * c12y) + Nz * c12z;
  const double l0 = (2.0 * detE) * detE - ((l1 + l2) + l3);
  const double M6 = M2 * M2 * M2;
  sg[0] = fs(detE, kFilt * 6.0 * M2 * M + kTiny);
  sg[1] = fs(l0, kFilt * 396.0 * M6 + kTiny);
  sg[2] = fs(l1, kFilt * 108.0 * M6 + kTiny);
  sg[3] = fs(l2, kFilt * 108.0 * M6 + kTiny);
  sg[4] = fs(l3, kFilt * 108.0 * M6 + kTiny);
  if (undecided) { slow(1); quad_signs_exact(c, T, sg); }
  return sg[0] != 0 && sg[1] >= 0 && sg[2] >= 0 && sg[3] >= 0 && sg[4] >= 0;
}

struct Mini {
  uint32_t T[4];
  int ts;
  FSphere fs;
};

__device__ bool verify_mini(const Cloud& c, const uint32_t* F, int k, Mini& mb) {
  if (!hull_centre(c, mb.T, mb.ts)) return false;
  fsphere(c.px, c.py, c.pz, mb.T, mb.ts, mb.fs);
  for (int i = 0; i < k; ++i) {
    bool sup = false;
    for (int j = 0; j < mb.ts; ++j) sup |= mb.T[j] == F[i];
    if (!sup && !inside_closed(c, mb.fs, mb.T, mb.ts, F[i])) return false;
  }
  return true;
}

// Exact miniball of the facet F (1..10 points): FP64 Welzl proposes the support,
// exact predicates verify it; exhaustive exact enumeration of 1..4-subsets when the
// proposal fails (build_exact_facet_miniball, hierarchy/facet_miniball.hpp:86-102).
__device__ __noinline__ bool facet_miniball(const Cloud& c, const uint32_t* F, int k, Mini& mb) {
  double P[kMaxFacet][3];
  for (int i = 0; i < k; ++i) {
    P[i][0] = c.px[F[i]] - c.px[F[0]];
    P[i][1] = c.py[F[i]] - c.py[F[0]];
    P[i][2] = c.pz[F[i]] - c.pz[F[0]];
  }
  double cx = 0, cy = 0, cz = 0, r2 = 0;
  int T[4] = {0, 0, 0, 0}, ts = 1;
  bool fp_ok = true;
  auto out = [&](int i) {
    const double dx = P[i][0] - cx, dy = P[i][1] - cy, dz = P[i][2] - cz;
    return dx * dx + dy * dy + dz * dz > r2 * (1.0 + 1e-10) + 1e-300;
  };
  auto set_ball = [&](const int* idx, int s) {
    T[0] = idx[0]; T[1] = s > 1 ? idx[1] : 0; T[2] = s > 2 ? idx[2] : 0; T[3] = s > 3 ? idx[3] : 0;
    ts = s;
    const double* a = P[idx[0]];
    if (s == 1) { cx = a[0]; cy = a[1]; cz = a[2]; r2 = 0; return; }
    double e[3][3];
    for (int j = 1; j < s; ++j)
      for (int t = 0; t < 3; ++t) e[j - 1][t] = P[idx[j]][t] - a[t];
    double A, N0, N1, N2;
    if (s == 2) {
      A = 1.0; N0 = e[0][0]; N1 = e[0][1]; N2 = e[0][2];
    } else if (s == 3) {
      const double G11 = e[0][0] * e[0][0] + e[0][1] * e[0][1] + e[0][2] * e[0][2];
      const double G22 = e[1][0] * e[1][0] + e[1][1] * e[1][1] + e[1][2] * e[1][2];
      const double G12 = e[0][0] * e[1][0] + e[0][1] * e[1][1] + e[0][2] * e[1][2];
      A = G11 * G22 - G12 * G12;
      const double f1 = G22 * (G11 - G12), f2 = G11 * (G22 - G12);
      N0 = f1 * e[0][0] + f2 * e[1][0]; N1 = f1 * e[0][1] + f2 * e[1][1]; N2 = f1 * e[0][2] + f2 * e[1][2];
    } else {
      const double* e1 = e[0]; const double* e2 = e[1]; const double* e3 = e[2];
      const double c23[3] = {e2[1] * e3[2] - e2[2] * e3[1], e2[2] * e3[0] - e2[0] * e3[2], e2[0] * e3[1] - e2[1] * e3[0]};
      const double c31[3] = {e3[1] * e1[2] - e3[2] * e1[1], e3[2] * e1[0] - e3[0] * e1[2], e3[0] * e1[1] - e3[1] * e1[0]};
      const double c12[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
      const double q1 = e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2];
      const double q2 = e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2];
      const double q3 = e3[0] * e3[0] + e3[1] * e3[1] + e3[2] * e3[2];
      A = e1[0] * c23[0] + e1[1] * c23[1] + e1[2] * c23[2];
      N0 = q1 * c23[0] + q2 * c31[0] + q3 * c12[0];
      N1 = q1 * c23[1] + q2 * c31[1] + q3 * c12[1];
      N2 = q1 * c23[2] + q2 * c31[2] + q3 * c12[2];
    }
    if (!(fabs(A) > 0.0)) { fp_ok = false; A = 1e-300; }
    const double inv = 0.5 / A;
    cx = a[0] + N0 * inv; cy = a[1] + N1 * inv; cz = a[2] + N2 * inv;
    r2 = (N0 * N0 + N1 * N1 + N2 * N2) * inv * inv;
  };
  int idx[4];
  idx[0] = 0;
  set_ball(idx, 1);
  for (int i = 1; i < k && fp_ok; ++i) {
    if (!out(i)) continue;
    idx[0] = i;
    set_ball(idx, 1);
    for (int j = 0; j < i && fp_ok; ++j) {
      if (!out(j)) continue;
      idx[0] = i; idx[1] = j;
      set_ball(idx, 2);
      for (int l = 0; l < j && fp_ok; ++l) {
        if (!out(l)) continue;
        idx[0] = i; idx[1] = j; idx[2] = l;
        set_ball(idx, 3);
        for (int m = 0; m < l && fp_ok; ++m) {
          if (!out(m)) continue;
          idx[0] = i; idx[1] = j; idx[2] = l; idx[3] = m;
          set_ball(idx, 4);
        }
      }
    }
  }
  if (fp_ok) {
    mb.ts = ts;
    for (int j = 0; j < ts; ++j) mb.T[j] = F[T[j]];
    // canonical support order (ascending ids) for the exact data
    for (int a = 1; a < ts; ++a) {
      const uint32_t x = mb.T[a];
      int b = a;
      while (b > 0 && mb.T[b - 1] > x) { mb.T[b] = mb.T[b - 1]; --b; }
      mb.T[b] = x;
    }
    if (verify_mini(c, F, k, mb)) return true;
  }
  // exhaustive exact enumeration
  slow(0);
  for (int s = (k == 1 ? 1 : 2); s <= 4 && s <= k; ++s) {
    int id[4] = {0, 1, 2, 3};
    while (true) {
      mb.ts = s;
      for (int j = 0; j < s; ++j) mb.T[j] = F[id[j]];
      if (verify_mini(c, F, k, mb)) return true;
      int p = s - 1;
      while (p >= 0 && id[p] == k - s + p) --p;
      if (p < 0) break;
      ++id[p];
      for (int q = p + 1; q < s; ++q) id[q] = id[q - 1] + 1;
    }
  }
  return false;
}

// Exact canonical top-k choice at the miniball centre of F.  Returns the status; on
// success G holds k ascending ids and *cut_below is 1 when the cutoff lies strictly
// below beta(F), 0 when it equals it.
__device__ __noinline__ int topk_choice(const DescentParams& d, const Cloud& c, const Mini& mb, int k, uint32_t* G,
                                        int* cut_below, uint32_t* visits) {
  const FSphere& fs = mb.fs;
  double llo, lhi;
  if (!flevel(fs, llo, lhi)) { slow(3); exact_level_fp(c, mb.T, mb.ts, llo, lhi); }
  // FP64 centre and its error: c~ = a + N / (2A)
  const double inv = 0.5 / fs.A;
  const double ox = fs.Nx * inv, oy = fs.Ny * inv, oz = fs.Nz * inv;
  const double cx = fs.ax + ox, cy = fs.ay + oy, cz = fs.az + oz;
  const double on = sqrt(ox * ox + oy * oy + oz * oz);
  const double nn = sqrt(fs.Nx * fs.Nx + fs.Ny * fs.Ny + fs.Nz * fs.Nz);
  const double relA = fs.eA / fmax(fabs(fs.A) - fs.eA, 1e-300);
  const double relN = fs.eN * 1.7320508075688772 / fmax(nn, 1e-300);
  double dc = on * (relA + relN) * 1.01 + 4.0 * kU * (fabs(cx) + fabs(cy) + fabs(cz)) + kTiny;
  if (!(relA < 0.5) || !isfinite(dc)) dc = 2.0 * sqrt(lhi) + 1e-300;  // centre not trusted: widen the ball
  const double R = sqrt(lhi) * (1.0 + 1e-12) + dc;
  const double R2 = R * R * (1.0 + 1e-12);
  const double ed = 2.0 * R * dc + dc * dc + 8.0 * kU * R2 + kTiny;
  // ball query
  uint32_t cid[kCandCap];
  double cd[kCandCap];
  int cnt = 0;
  uint32_t stack[kDStack];
  int top = 0;
  stack[top++] = d.root;
  // The nearest kCandCap points within R, sorted by FP64 squared distance; a farther point
  // is dropped when the list is full.  Only the points up to the band around the k-th
  // distance matter, so the traversal is pruned at the current k-th distance + 2 ed (it
  // can only decrease), and the dropped points are checked to lie beyond the band below.
  double R2_eff = R2;
  bool dropped = false;
  // The node prune runs in binary32 (the FP64 pipe is the step's tighter unit): qf is the
  // binary32 rounding of the centre and dqf its distance from it, rounded up (exact in binary64).
  // Each axis gap to a node box is lowered by the rounding of the subtraction (a relative
  // 2^-22) and by dqf, clamped at 0; the sum of squares is lowered by a relative 2^-20 and
  // compared with R2_eff rounded up.  The bound never exceeds the exact one, so the prune skips
  // only boxes that hold no point within R2_eff (the FP64 prune skips at least those; the
  // leaves decide membership in FP64 as before).  Far from the origin the FP64 prune stays, and for radii
  // whose squares binary32 does not hold (a gap's square loses the margin to underflow).
  const double qv[3] = {cx, cy, cz};
  const bool f32 = fabs(cx) < 0x1p60 && fabs(cy) < 0x1p60 && fabs(cz) < 0x1p60 && R2 < 0x1p100 && R2 > 0x1p-126;
  float qf[3], dqf[3];
  for (int a = 0; a < 3; ++a) {
    qf[a] = (float)qv[a];
    dqf[a] = __double2float_ru(fabs(qv[a] - (double)qf[a]));
  }
  float R2f = __double2float_ru(R2_eff);
  while (top > 0) {
    const uint32_t node = stack[--top];
    const TNode t = load_node(d.tn, node);
    ++*visits;
    if (t.left == kInvalid32) {
      const uint32_t q = t.right;
      const double dx = c.px[q] - cx, dy = c.py[q] - cy, dz = c.pz[q] - cz;
      const double dd = dx * dx + dy * dy + dz * dz;
      if (dd > R2_eff) continue;
      if (cnt == kCandCap) {
        if (dd >= cd[kCandCap - 1]) { dropped = true; continue; }
        --cnt;
        dropped = true;
      }
      int j = cnt++;
      while (j > 0 && cd[j - 1] > dd) { cd[j] = cd[j - 1]; cid[j] = cid[j - 1]; --j; }
      cd[j] = dd;
      cid[j] = q;
      if (cnt >= k) {
        R2_eff = fmin(R2, (cd[k - 1] + 2.0 * ed) * (1.0 + 1e-12));
        R2f = __double2float_ru(R2_eff);
      }
      continue;
    }
    if (f32) {
      float lbf = 0.f;
      for (int a = 0; a < 3; ++a) {
        const float g0 = fmaxf(fmaxf(t.lo[a] - qf[a], qf[a] - t.hi[a]), 0.f);
        const float g = fmaxf(g0 * (1.f - 0x1p-22f) - dqf[a], 0.f);
        lbf += g * g;
      }
      if (lbf * (1.f - 0x1p-20f) > R2f) continue;
    } else {
      double lb = 0.0;
      for (int a = 0; a < 3; ++a) {
        const double g = fmax(fmax((double)t.lo[a] - qv[a], qv[a] - (double)t.hi[a]), 0.0);
        lb += g * g;
      }
      if (lb * (1.0 - 1e-6) > R2_eff) continue;
    }
    if (top + 2 > kDStack) return kArmCapacity;
    stack[top++] = t.left;
    stack[top++] = t.right;
  }
  if (cnt < k) return kArmInternal;
  // partition around the k-th approximate distance
  const double tk = cd[k - 1];
  // every dropped point is at least as far as the last kept one: it must lie past the band
  if (dropped && !(cd[cnt - 1] > tk + 2.0 * ed)) return kArmCapacity;
  int below = 0, band0 = -1, band1 = -1;
  for (int i = 0; i < cnt; ++i) {
    if (cd[i] < tk - 2.0 * ed) below = i + 1;
    else if (cd[i] <= tk + 2.0 * ed) { if (band0 < 0) band0 = i; band1 = i; }
  }
  int nsel = 0;
  for (int i = 0; i < below; ++i) G[nsel++] = cid[i];
  uint32_t cut_point;
  if (band0 == band1) {  // the k-th is isolated
    G[nsel++] = cid[band0];
    cut_point = cid[band0];
  } else {
    // The band usually holds support points of F's miniball, which lie exactly on
    // its sphere: relate every band member to beta(F) (support points are equal to it
    // by construction; others by FP64, exact when undecided).  When the cutoff is
    // beta(F) the choice needs no mutual order of the members below it.
    const int nb = band1 - band0 + 1;
    uint32_t* B = cid + band0;
    int rel[kCandCap];
    int n_lo = 0, n_eq = 0, n_hi = 0;
    for (int t = 0; t < nb; ++t) {
      bool sup = false;
      for (int j = 0; j < mb.ts; ++j) sup |= mb.T[j] == B[t];
      int r;
      if (sup) r = 0;
      else if (cd[band0 + t] + ed < llo) r = -1;
      else if (cd[band0 + t] - ed > lhi) r = 1;
      else {
        slow(5);
        r = dist_cmp_exact(c, mb.T, mb.ts, B[t], mb.T[0]);
      }
      rel[t] = r;
      n_lo += r < 0;
      n_eq += r == 0;
      n_hi += r > 0;
    }
    const int need = k - below;  // >= 1
    if (need > n_lo && need <= n_lo + n_eq) {
      // cutoff = beta(F): the lower members, then the least ids at beta(F)
      for (int t = 0; t < nb; ++t)
        if (rel[t] < 0) G[nsel++] = B[t];
      uint32_t eq[kCandCap];
      int ne = 0;
      for (int t = 0; t < nb; ++t)
        if (rel[t] == 0) eq[ne++] = B[t];
      for (int a = 1; a < ne; ++a) {
        const uint32_t x = eq[a];
        int b = a;
        while (b > 0 && eq[b - 1] > x) { eq[b] = eq[b - 1]; --b; }
        eq[b] = x;
      }
      for (int t = 0; nsel < k; ++t) G[nsel++] = eq[t];
      cut_point = mb.T[0];
    } else {
      // exact order of the band by (distance, id)
      slow(4);
      for (int a = 1; a < nb; ++a) {
        const uint32_t x = B[a];
        int b = a;
        while (b > 0) {
          const int s = dist_cmp_exact(c, mb.T, mb.ts, B[b - 1], x);
          if (s < 0 || (s == 0 && B[b - 1] < x)) break;
          B[b] = B[b - 1];
          --b;
        }
        B[b] = x;
      }
      cut_point = B[need - 1];
      // strictly below the cutoff, then the least ids of the shell
      int j = 0;
      while (j < nb && dist_cmp_exact(c, mb.T, mb.ts, B[j], cut_point) < 0) G[nsel++] = B[j++];
      while (nsel < k) G[nsel++] = B[j++];  // shell members in id order
    }
  }
  for (int a = 1; a < k; ++a) {
    const uint32_t x = G[a];
    int b = a;
    while (b > 0 && G[b - 1] > x) { G[b] = G[b - 1]; --b; }
    G[b] = x;
  }
  // cutoff versus beta(F) = |T0 - centre|^2
  bool on_sphere = false;
  for (int j = 0; j < mb.ts; ++j) on_sphere |= mb.T[j] == cut_point;
  if (on_sphere) {
    *cut_below = 0;
  } else {
    // FP64 first: the cutoff's approximate distance against the radius interval
    const double dcut = band0 == band1 ? cd[band0] : tk + 2.0 * ed;  // upper bound of the cutoff's FP distance
    if (dcut + ed < llo) {
      *cut_below = 1;
    } else {
      slow(5);
      const int s = dist_cmp_exact(c, mb.T, mb.ts, cut_point, mb.T[0]);
      if (s > 0) return kArmInternal;
      *cut_below = s < 0 ? 1 : 0;
    }
  }
  return kArmOk;
}

// Arm seeds and their first probe, one thread per saddle family: one arm per support point
// (F_u = (I u U) \ {u}); most arms are themselves a birth facet of their order.  Misses are queued
// with their facet for the descent steps while they fit (q_count counts them all).
__global__ void k_arm_probe(DescentParams d, uint32_t f0, uint32_t nfam, const uint32_t* __restrict__ fam_event,
                            const uint32_t* __restrict__ armoff, const EvRec* __restrict__ ev,
                            uint32_t* __restrict__ removed, uint32_t* __restrict__ term, uint32_t* __restrict__ q_arm,
                            QFacet* __restrict__ q_fac, uint32_t q_cap, uint32_t* __restrict__ q_count) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = i < nfam;
  const uint32_t f = f0 + (on ? i : 0u), a0 = armoff[f];
  const EvRec e = ev[fam_event[f]];
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t S[kMaxFacet + 1];
  const int k = event_facet(e, S) - 1;
#pragma unroll
  for (uint32_t t = 0; t < 4; ++t) {  // the whole warp: its misses take their slots with one atomic
    const bool arm = on && t < e.size;
    uint32_t F[kMaxFacet];  // of arm t: (I u U) \ {u}, ascending
#pragma unroll
    for (int j = 0; j < kMaxFacet; ++j) F[j] = S[j] < e.ids[t] ? S[j] : S[j + 1];
    bool miss = false;
    if (arm) {
      const uint32_t h = probe_facet(d, F, k);
      removed[a0 + t] = e.ids[t];
      term[a0 + t] = h;
      miss = h == kInvalid32;
    }
    const uint32_t b = __ballot_sync(0xffffffffu, miss);
    uint32_t base = 0;
    if (lane == 0 && b) base = atomicAdd(q_count, (uint32_t)__popc(b));
    base = __shfl_sync(0xffffffffu, base, 0);
    const uint32_t slot = base + __popc(b & ((1u << lane) - 1u));
    if (!miss || slot >= q_cap) continue;
    q_arm[slot] = a0 + t;
    QFacet q;
#pragma unroll
    for (int j = 0; j < kMaxFacet; ++j) q.F[j] = F[j];
    for (int j = 0; j < 4; ++j) q.prev[j] = kInvalid32;
    q.prev_lo = 0.0;
    q_fac[slot] = q;
  }
}

// Sort keys of a descent queue: the top 24 bits of the Morton code of each facet's least
// point, so that a warp's threads descend from nearby facets (shared traversal paths,
// less divergence).  The order of processing never changes a result.
__global__ void k_queue_keys(uint32_t m, const QFacet* __restrict__ in_fac, const uint64_t* __restrict__ code,
                             uint64_t* __restrict__ key, uint32_t* __restrict__ val) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  key[i] = code[in_fac[i].F[0]] >> 39;
  val[i] = i;
}

// ---- one strict descent step for every queued arm -------------------------------------------------
// Exact miniball of F, exact canonical top-k choice G at its centre, certified beta(G) < beta(F); G is
// probed and either binds the arm or is queued for the next step.  A round is three launches:
//  k_facet_ball  proposes the support of F's miniball in binary32 and certifies it in binary64;
//  k_facet_step  takes the points inside the ball from the LBVH, forms G, checks the level, probes;
//  k_facet_exact runs the arms that either of them left open: the exact fallbacks for every decision.
// The first two make no call (what lives across one goes to local memory) and keep no array in local
// memory; when G is not a birth, the next round's k_facet_ball checks that its level decreased; a birth's
// level interval is known.  Bound: latency of the walk's node loads and its divergence.
// One kernel with the exact fallbacks in its loops, a binary64 miniball of F and one of G per step and a
// sorted candidate list per thread took 104.4 ms over all rounds at 50,653 lattice points (32.2 M
// steps) and 27.6 at 12,289 uniform ones; the three launches take 32.5 and 11.8 ms.

// Counts places of the lanes that have `on` set; `at` of the others is not defined.
__device__ __forceinline__ uint32_t warp_slot(bool on, uint32_t* count) {
  const uint32_t lane = threadIdx.x & 31u, b = __ballot_sync(0xffffffffu, on);
  uint32_t base = 0;
  if (lane == 0 && b) base = atomicAdd(count, (uint32_t)__popc(b));
  base = __shfl_sync(0xffffffffu, base, 0);
  return base + __popc(b & ((1u << lane) - 1u));
}

// Side of the point at offset (x, y, z) from T[0] of the sphere of T: -1 inside, 1 outside, 0 when binary64
// does not decide (the bounds of inside_closed).
__device__ __forceinline__ int side_fp(const FSphere& fs, int ts, double x, double y, double z) {
  const double Mp = fmax(fs.M, fmax(fabs(x), fmax(fabs(y), fabs(z)))) * (1.0 + 1e-15);
  const double q = (x * x + y * y) + z * z;
  const double v = fs.A * q - ((x * fs.Nx + y * fs.Ny) + z * fs.Nz);
  const double M2 = fs.M * fs.M, M4 = M2 * M2;
  const double Am = ts <= 2 ? 1.0 : (ts == 3 ? 18.0 * M4 : 6.0 * M2 * fs.M);
  const double Nm = ts == 1 ? 0.0 : (ts == 2 ? fs.M : (ts == 3 ? 36.0 * M4 * fs.M : 18.0 * M4));
  const double bnd = kFilt * (Am * 3.0 * Mp * Mp + 3.0 * Mp * Nm) + kTiny;
  const double w = fs.A < 0.0 ? -v : v;
  if (!(fabs(fs.A) > fs.eA)) return 0;
  return w < -bnd ? -1 : (w > bnd ? 1 : 0);
}

// The circumcentre of T lies strictly inside its hull for certain (the bounds of hull_centre).
__device__ __forceinline__ bool hull_fp(const Cloud& c, const uint32_t (&T)[4], int ts) {
  if (ts <= 2) return ts == 2;
  double e[3][3], M = 0.0;
#pragma unroll
  for (int j = 1; j < 4; ++j) {
    if (j >= ts) {
      e[j - 1][0] = e[j - 1][1] = e[j - 1][2] = 0.0;
      continue;
    }
    e[j - 1][0] = c.px[T[j]] - c.px[T[0]];
    e[j - 1][1] = c.py[T[j]] - c.py[T[0]];
    e[j - 1][2] = c.pz[T[j]] - c.pz[T[0]];
    M = fmax(M, fmax(fabs(e[j - 1][0]), fmax(fabs(e[j - 1][1]), fabs(e[j - 1][2]))));
  }
  M *= (1.0 + 1e-15);
  const double M2 = M * M;
  if (ts == 3) {
    const double G11 = (e[0][0] * e[0][0] + e[0][1] * e[0][1]) + e[0][2] * e[0][2];
    const double G22 = (e[1][0] * e[1][0] + e[1][1] * e[1][1]) + e[1][2] * e[1][2];
    const double G12 = (e[0][0] * e[1][0] + e[0][1] * e[1][1]) + e[0][2] * e[1][2];
    const double b2 = kFilt * 6.0 * M2 + kTiny;
    return G12 > kFilt * 3.0 * M2 + kTiny && G11 - G12 > b2 && G22 - G12 > b2 &&
           G11 * G22 - G12 * G12 > kFilt * 18.0 * M2 * M2 + kTiny;
  }
  const double* e1 = e[0];
  const double* e2 = e[1];
  const double* e3 = e[2];
  const double c23x = e2[1] * e3[2] - e2[2] * e3[1], c23y = e2[2] * e3[0] - e2[0] * e3[2], c23z = e2[0] * e3[1] - e2[1] * e3[0];
  const double c31x = e3[1] * e1[2] - e3[2] * e1[1], c31y = e3[2] * e1[0] - e3[0] * e1[2], c31z = e3[0] * e1[1] - e3[1] * e1[0];
  const double c12x = e1[1] * e2[2] - e1[2] * e2[1], c12y = e1[2] * e2[0] - e1[0] * e2[2], c12z = e1[0] * e2[1] - e1[1] * e2[0];
  const double q1 = (e1[0] * e1[0] + e1[1] * e1[1]) + e1[2] * e1[2];
  const double q2 = (e2[0] * e2[0] + e2[1] * e2[1]) + e2[2] * e2[2];
  const double q3 = (e3[0] * e3[0] + e3[1] * e3[1]) + e3[2] * e3[2];
  const double detE = (e1[0] * c23x + e1[1] * c23y) + e1[2] * c23z;
  const double Nx = (q1 * c23x + q2 * c31x) + q3 * c12x;
  const double Ny = (q1 * c23y + q2 * c31y) + q3 * c12y;
  const double Nz = (q1 * c23z + q2 * c31z) + q3 * c12z;
  const double l1 = (Nx * c23x + Ny * c23y) + Nz * c23z;
  const double l2 = (Nx * c31x + Ny * c31y) + Nz * c31z;
  const double l3 = (Nx * c12x + Ny * c12y) + Nz * c12z;
  const double l0 = (2.0 * detE) * detE - ((l1 + l2) + l3);
  const double M6 = M2 * M2 * M2, bl = kFilt * 108.0 * M6 + kTiny;
  return fabs(detE) > kFilt * 6.0 * M2 * M + kTiny && l0 > kFilt * 396.0 * M6 + kTiny && l1 > bl && l2 > bl && l3 > bl;
}

constexpr int kFT = 128;           // threads per block of the two fast kernels
constexpr int kBallRounds = 24;    // pivots of the proposal before an arm is left open

// Miniball of every queued facet: T (ascending ids, unused kInvalid32) when it is certified and its level lies
// below the one it must, else the entry goes to `hard` and T.x is kInvalid32.
// The proposal pivots on the farthest point: the ball of the support so far and that point (at most five
// points, Welzl's recursion with the new point on the sphere) until nothing lies outside.  Binary32 on
// differences scaled by a power of two, in shared memory (dynamic indices).
__global__ void __launch_bounds__(kFT, 8)
k_facet_ball(DescentParams d, uint32_t m, const QFacet* __restrict__ in_fac, const uint32_t* __restrict__ rstate, int passes,
             const uint32_t* __restrict__ v0, const uint32_t* __restrict__ v1, uint4* __restrict__ support,
             uint32_t* __restrict__ hard, uint32_t* __restrict__ hard_count) {
  __shared__ float sx[kMaxFacet][kFT], sy[kMaxFacet][kFT], sz[kMaxFacet][kFT];
  const uint32_t t = blockIdx.x * kFT + threadIdx.x, w = threadIdx.x;
  bool open = false;
  uint32_t i = 0;
  if (t < m) {
    i = passes >= 0 ? radix_result(rstate, passes, v0, v1)[t] : t;
    const QFacet& e = in_fac[i];
    const uint32_t f0 = e.F[0];
    const double ax = d.px[f0], ay = d.py[f0], az = d.pz[f0];
    int k = 0;
    float M = 0.f;
    for (int q = 0; q < kMaxFacet; ++q) {
      const uint32_t id = e.F[q];
      if (id == kInvalid32) break;
      const float x = (float)(d.px[id] - ax), y = (float)(d.py[id] - ay), z = (float)(d.pz[id] - az);
      sx[q][w] = x;
      sy[q][w] = y;
      sz[q][w] = z;
      M = fmaxf(M, fmaxf(fabsf(x), fmaxf(fabsf(y), fabsf(z))));
      ++k;
    }
    open = !(M > 1e-30f && M < 1e30f);
    const float scale = open ? 1.f : exp2f((float)-ilogbf(M));
    for (int q = 0; q < k; ++q) {
      sx[q][w] *= scale;
      sy[q][w] *= scale;
      sz[q][w] *= scale;
    }
    float cx = 0.f, cy = 0.f, cz = 0.f, r2 = 0.f;
    uint32_t T = 0;  // positions of the support's points, 8 bits each
    int ts = 1, round = 0;
    auto outside = [&](uint32_t q) {
      const float x = sx[q][w] - cx, y = sy[q][w] - cy, z = sz[q][w] - cz;
      return x * x + y * y + z * z > r2 * (1.f + 1e-5f) + 1e-12f;
    };
    // ball through the points of `idx` (8 bits each), s of them
    auto ball = [&](uint32_t idx, int s) {
      T = idx;
      ts = s;
      const uint32_t a = idx & 255u, p1 = idx >> 8 & 255u;
      const float ox = sx[a][w], oy = sy[a][w], oz = sz[a][w];
      const float x1 = sx[p1][w] - ox, y1 = sy[p1][w] - oy, z1 = sz[p1][w] - oz;
      const float q1 = x1 * x1 + y1 * y1 + z1 * z1;
      float A = 1.f, n0 = x1, n1 = y1, n2 = z1;  // two points
      if (s > 2) {
        const uint32_t p2 = idx >> 16 & 255u;
        const float x2 = sx[p2][w] - ox, y2 = sy[p2][w] - oy, z2 = sz[p2][w] - oz;
        const float q2 = x2 * x2 + y2 * y2 + z2 * z2;
        if (s == 3) {
          const float g = x1 * x2 + y1 * y2 + z1 * z2;
          const float f1 = q2 * (q1 - g), f2 = q1 * (q2 - g);
          A = q1 * q2 - g * g;
          n0 = f1 * x1 + f2 * x2;
          n1 = f1 * y1 + f2 * y2;
          n2 = f1 * z1 + f2 * z2;
        } else {
          const uint32_t p3 = idx >> 24;
          const float x3 = sx[p3][w] - ox, y3 = sy[p3][w] - oy, z3 = sz[p3][w] - oz;
          const float q3 = x3 * x3 + y3 * y3 + z3 * z3;
          const float ax3 = y2 * z3 - z2 * y3, ay3 = z2 * x3 - x2 * z3, az3 = x2 * y3 - y2 * x3;
          const float bx3 = y3 * z1 - z3 * y1, by3 = z3 * x1 - x3 * z1, bz3 = x3 * y1 - y3 * x1;
          const float cx3 = y1 * z2 - z1 * y2, cy3 = z1 * x2 - x1 * z2, cz3 = x1 * y2 - y1 * x2;
          A = x1 * ax3 + y1 * ay3 + z1 * az3;
          n0 = q1 * ax3 + q2 * bx3 + q3 * cx3;
          n1 = q1 * ay3 + q2 * by3 + q3 * cy3;
          n2 = q1 * az3 + q2 * bz3 + q3 * cz3;
        }
      }
      const float inv = __fdividef(0.5f, A);
      n0 *= inv;
      n1 *= inv;
      n2 *= inv;
      cx = ox + n0;
      cy = oy + n1;
      cz = oz + n2;
      r2 = n0 * n0 + n1 * n1 + n2 * n2;
    };
    for (; !open && round < kBallRounds; ++round) {
      float far = r2 * (1.f + 1e-5f) + 1e-12f;
      uint32_t f = 255u;
      for (int q = 0; q < k; ++q) {
        const float x = sx[q][w] - cx, y = sy[q][w] - cy, z = sz[q][w] - cz;
        const float dd = x * x + y * y + z * z;
        if (dd > far) {
          far = dd;
          f = (uint32_t)q;
        }
      }
      if (f == 255u) break;
      const uint32_t old = T;
      const int n_old = ts;
      cx = sx[f][w];
      cy = sy[f][w];
      cz = sz[f][w];
      r2 = 0.f;
      T = f;
      ts = 1;
      for (int j = 0; j < n_old; ++j) {
        const uint32_t pj = old >> (8 * j) & 255u;
        if (!outside(pj)) continue;
        ball(f | pj << 8, 2);
        for (int l = 0; l < j; ++l) {
          const uint32_t pl = old >> (8 * l) & 255u;
          if (!outside(pl)) continue;
          ball(f | pj << 8 | pl << 16, 3);
          for (int n = 0; n < l; ++n) {
            const uint32_t pn = old >> (8 * n) & 255u;
            if (outside(pn)) ball(f | pj << 8 | pl << 16 | pn << 24, 4);
          }
        }
      }
    }
    open = open || round == kBallRounds || ts < 2;
    // certificate in binary64
    uint4 out = make_uint4(kInvalid32, kInvalid32, kInvalid32, kInvalid32);
    if (!open) {
      uint32_t id[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) id[j] = j < ts ? e.F[T >> (8 * j) & 255u] : kInvalid32;
      auto cswap = [](uint32_t& x, uint32_t& y) {
        const uint32_t lo = min(x, y), hi = max(x, y);
        x = lo;
        y = hi;
      };
      cswap(id[0], id[1]);
      cswap(id[2], id[3]);
      cswap(id[0], id[2]);
      cswap(id[1], id[3]);
      cswap(id[1], id[2]);
      const Cloud c{d.px, d.py, d.pz, d.S};
      open = !hull_fp(c, id, ts);
      FSphere fs;
      if (!open) {
        fsphere(d.px, d.py, d.pz, id, ts, fs);
        double lo, hi;
        open = !flevel(fs, lo, hi) || (e.prev[0] != kInvalid32 && !(hi < e.prev_lo));
      }
      for (int q = 0; q < k && !open; ++q) {
        const uint32_t p = e.F[q];
        if (p == id[0] || p == id[1] || p == id[2] || p == id[3]) continue;
        open = side_fp(fs, ts, d.px[p] - fs.ax, d.py[p] - fs.ay, d.pz[p] - fs.az) >= 0;
      }
      if (!open) out = make_uint4(id[0], id[1], id[2], id[3]);
    }
    support[i] = out;
  }
  const uint32_t slot = warp_slot(open, hard_count);
  if (open) hard[slot] = i;
}

constexpr int kStepStack = 32;  // traversal entries per thread (an arm that needs more is left open)
constexpr int kStepIn = 20;     // points inside the ball per thread (likewise; their distances fit in the stack)

// The step of every facet with a certified support: points strictly inside its miniball come from the LBVH;
// with fewer than k of them the choice is those and the least support points (which lie on the sphere),
// with k or more the k nearest.  Any point that binary64 does not place, an order of distances that the
// rounded ones leave open, or an arm that would fail goes to `hard`.
__global__ void __launch_bounds__(kFT, 6)
k_facet_step(DescentParams d, uint32_t m, const uint32_t* __restrict__ in_arm, const QFacet* __restrict__ in_fac,
             const uint4* __restrict__ support, const uint32_t* __restrict__ rstate, int passes,
             const uint32_t* __restrict__ v0, const uint32_t* __restrict__ v1, uint32_t* __restrict__ out_arm,
             QFacet* __restrict__ out_fac, uint32_t* __restrict__ out_count, uint32_t* __restrict__ term,
             unsigned long long* __restrict__ stats, uint32_t* __restrict__ hard, uint32_t* __restrict__ hard_count) {
  __shared__ uint32_t stack[kStepStack][kFT], inside[kStepIn][kFT];
  // Work counters leave through shared memory with the block's last warp (no warp waits for another);
  // a global atomic per arm and counter queues every arm on one address.
  __shared__ unsigned int s_count[3], s_warps;  // node visits, steps, equal cutoffs
  const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x;
  if (w < 3) s_count[w] = 0;
  if (w == 3) s_warps = 0;
  __syncthreads();
  const uint32_t t = blockIdx.x * kFT + w;
  uint32_t i = 0, visits = 0, stepped = 0, equal = 0, G[kMaxFacet];
  bool open = false, go_on = false;
  double llo = 0.0, lhi = 0.0;
  uint32_t T[4] = {kInvalid32, kInvalid32, kInvalid32, kInvalid32};
  if (t < m) {
    i = passes >= 0 ? radix_result(rstate, passes, v0, v1)[t] : t;
    const uint4 sup = support[i];
    T[0] = sup.x;
    T[1] = sup.y;
    T[2] = sup.z;
    T[3] = sup.w;
  }
  if (T[0] != kInvalid32) {
    const int ts = T[2] == kInvalid32 ? 2 : (T[3] == kInvalid32 ? 3 : 4);
    double cx, cy, cz, R2, ed;
    {
      FSphere fs;
      fsphere(d.px, d.py, d.pz, T, ts, fs);
      flevel(fs, llo, lhi);  // certified by k_facet_ball
      // FP64 centre and its error: c~ = a + N / (2A)
      const double inv = 0.5 / fs.A;
      const double ox = fs.Nx * inv, oy = fs.Ny * inv, oz = fs.Nz * inv;
      cx = fs.ax + ox;
      cy = fs.ay + oy;
      cz = fs.az + oz;
      const double on = sqrt(ox * ox + oy * oy + oz * oz);
      const double nn = sqrt(fs.Nx * fs.Nx + fs.Ny * fs.Ny + fs.Nz * fs.Nz);
      const double relA = fs.eA / fmax(fabs(fs.A) - fs.eA, 1e-300);
      const double relN = fs.eN * 1.7320508075688772 / fmax(nn, 1e-300);
      const double dc = on * (relA + relN) * 1.01 + 4.0 * kU * (fabs(cx) + fabs(cy) + fabs(cz)) + kTiny;
      const double R = sqrt(lhi) * (1.0 + 1e-12) + dc;
      R2 = R * R * (1.0 + 1e-12);
      ed = 2.0 * R * dc + dc * dc + 8.0 * kU * R2 + kTiny;
      open = !(relA < 0.5) || !isfinite(dc) ||
             !(fabs(cx) < 0x1p60 && fabs(cy) < 0x1p60 && fabs(cz) < 0x1p60 && R2 < 0x1p100 && R2 > 0x1p-126);
    }
    // binary32 prune as in topk_choice: a lower bound of the distance to a node box, from the rounded centre
    const float qx = (float)cx, qy = (float)cy, qz = (float)cz;
    const float dq = fmaxf(__double2float_ru(fabs(cx - (double)qx)),
                           fmaxf(__double2float_ru(fabs(cy - (double)qy)), __double2float_ru(fabs(cz - (double)qz))));
    const float R2f = __double2float_ru(R2);
    const double in2 = llo - ed, out2 = lhi + ed;  // FP distances below / above them are inside / outside for certain
    uint32_t n_in = 0;
    int top = 0;
    if (!open) stack[top++][w] = d.root;
    while (top > 0) {
      const TNode nd = load_node(d.tn, stack[--top][w]);
      ++visits;
      if (nd.left != kInvalid32) {
        const float g0 = fmaxf(fmaxf(fmaxf(nd.lo[0] - qx, qx - nd.hi[0]), 0.f) * (1.f - 0x1p-22f) - dq, 0.f);
        const float g1 = fmaxf(fmaxf(fmaxf(nd.lo[1] - qy, qy - nd.hi[1]), 0.f) * (1.f - 0x1p-22f) - dq, 0.f);
        const float g2 = fmaxf(fmaxf(fmaxf(nd.lo[2] - qz, qz - nd.hi[2]), 0.f) * (1.f - 0x1p-22f) - dq, 0.f);
        if ((g0 * g0 + g1 * g1 + g2 * g2) * (1.f - 0x1p-20f) > R2f) continue;
        if (top + 2 > kStepStack) {
          open = true;
          break;
        }
        stack[top++][w] = nd.left;
        stack[top++][w] = nd.right;
        continue;
      }
      const uint32_t q = nd.right;
      const double dx = d.px[q] - cx, dy = d.py[q] - cy, dz = d.pz[q] - cz;
      const double dd = dx * dx + dy * dy + dz * dz;
      if (dd > out2 || q == T[0] || q == T[1] || q == T[2] || q == T[3]) continue;
      if (!(dd < in2) || n_in == (uint32_t)kStepIn) {
        open = true;
        break;
      }
      inside[n_in++][w] = q;
    }
    const QFacet& e = in_fac[i];
    uint32_t k = 0;
#pragma unroll
    for (int j = 0; j < kMaxFacet; ++j) k += e.F[j] != kInvalid32 ? 1u : 0u;
    if (!open && n_in > k) {  // drop the farthest; the distances stand in the stack that the walk has left
      for (uint32_t q = 0; q < n_in; ++q) {
        const uint32_t p = inside[q][w];
        const double dx = d.px[p] - cx, dy = d.py[p] - cy, dz = d.pz[p] - cz;
        stack[q][w] = __float_as_uint((float)(dx * dx + dy * dy + dz * dz));  // >= 0: ordered as its bits
      }
      auto farthest = [&]() {
        uint32_t at = 0;
        for (uint32_t q = 1; q < n_in; ++q)
          if (stack[q][w] > stack[at][w]) at = q;
        return at;
      };
      float dropped = 0.f;
      while (n_in > k) {
        const uint32_t at = farthest();
        dropped = __uint_as_float(stack[at][w]);
        --n_in;
        inside[at][w] = inside[n_in][w];
        stack[at][w] = stack[n_in][w];
      }
      // the nearest dropped point is farther than every kept one for certain (both within ed, and rounded)
      open = !(dropped - __uint_as_float(stack[farthest()][w]) > __double2float_ru(2.0 * ed) + 4e-7f * dropped);
    }
    open = open || n_in + (uint32_t)ts < k;
    if (!open) {
      // G ascending: the inside points, then the least support points
#pragma unroll
      for (int j = 0; j < kMaxFacet; ++j) G[j] = kInvalid32;
      auto put = [&](uint32_t x) {
#pragma unroll
        for (int j = 0; j < kMaxFacet; ++j) {
          const uint32_t lo = min(G[j], x);
          x = max(G[j], x);
          G[j] = lo;
        }
      };
      for (uint32_t q = 0; q < n_in; ++q) put(inside[q][w]);
      const bool at_level = n_in < k;  // the cutoff is beta(F): beta(G) must be shown to be less
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n_in + j < k) put(T[j]);
      bool same = true;
#pragma unroll
      for (int j = 0; j < kMaxFacet; ++j) same &= G[j] == e.F[j];
      const uint32_t h = same ? kInvalid32 : probe_facet(d, G, (int)k);
      open = same;
      if (h != kInvalid32) {
        const uint32_t ev = d.birth_event[h - d.n];
        if (at_level && !(d.lmid[ev] + d.lerr[ev] < llo)) open = true;
        else term[in_arm[i]] = h;
      } else {
        go_on = !open;
        if (!at_level) T[0] = kInvalid32;  // a cutoff below the level: nothing to check
      }
      if (!open) {
        stepped = 1;
        equal = at_level ? 1u : 0u;
      }
    }
  }
  __syncwarp();
  const uint32_t slot = warp_slot(go_on, out_count), hslot = warp_slot(open, hard_count);
  if (go_on) {
    out_arm[slot] = in_arm[i];
    QFacet q;
#pragma unroll
    for (int j = 0; j < kMaxFacet; ++j) q.F[j] = G[j];
#pragma unroll
    for (int j = 0; j < 4; ++j) q.prev[j] = T[j];
    q.prev_lo = llo;
    out_fac[slot] = q;
  }
  if (open) hard[hslot] = i;
  visits = __reduce_add_sync(0xffffffffu, visits);
  stepped = __reduce_add_sync(0xffffffffu, stepped);
  equal = __reduce_add_sync(0xffffffffu, equal);
  if (lane != 0) return;
  atomicAdd(s_count + 0, visits);
  atomicAdd(s_count + 1, stepped);
  atomicAdd(s_count + 2, equal);
  __threadfence_block();
  if (atomicAdd(&s_warps, 1u) + 1 < kFT / 32) return;
  __threadfence_block();
  atomicAdd(&g_descent_visits[blockIdx.x % kVisitStripes], (unsigned long long)atomicAdd(s_count + 0, 0u));
  const unsigned int n_step = atomicAdd(s_count + 1, 0u), n_equal = atomicAdd(s_count + 2, 0u);
  atomicAdd(stats, (unsigned long long)n_step);
  atomicAdd(stats + 1, (unsigned long long)n_equal);
  atomicAdd(&g_descent_slow[6], (unsigned long long)n_equal);
}

// The whole step of the queue entries in `hard`, with the exact fallbacks.
__global__ void __launch_bounds__(128)
k_facet_exact(DescentParams d, uint32_t m, const uint32_t* __restrict__ hard, const uint32_t* __restrict__ in_arm,
              const QFacet* __restrict__ in_fac, uint32_t* __restrict__ out_arm, QFacet* __restrict__ out_fac,
              uint32_t* __restrict__ out_count, uint32_t* __restrict__ term, unsigned long long* __restrict__ stats) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t F[kMaxFacet], G[kMaxFacet], a = 0, visits = 0;
  int k = 0;
  bool go_on = false;
  Mini mb;
  int cut_below = 0;
  double flo = 0.0, fhi = 0.0;
  if (t < m) {
    const uint32_t i = hard[t];
    const QFacet e = in_fac[i];
    a = in_arm[i];
    for (int j = 0; j < kMaxFacet; ++j) {
      F[j] = e.F[j];
      k += F[j] != kInvalid32;
    }
    const Cloud c{d.px, d.py, d.pz, d.S};
    // level(lo, hi, S) strictly below the interval or the support it is compared with
    auto below = [&](const Mini& x, const uint32_t* T, int ts, double tlo) {
      double lo, hi;
      if (!flevel(x.fs, lo, hi)) exact_level_fp(c, x.T, x.ts, lo, hi);
      return hi < tlo || level_cmp_exact(c, x.T, x.ts, T, ts) < 0;
    };
    auto step = [&]() -> int {
      if (!facet_miniball(c, F, k, mb)) return kArmInternal;
      if (e.prev[0] != kInvalid32) {
        int ts = 1;
        while (ts < 4 && e.prev[ts] != kInvalid32) ++ts;
        if (!below(mb, e.prev, ts, e.prev_lo)) return kArmPlateau;
      }
      const int s = topk_choice(d, c, mb, k, G, &cut_below, &visits);
      if (s != kArmOk) return s;
      bool same = true;
      for (int j = 0; j < k; ++j) same &= G[j] == F[j];
      return same ? kArmUnresolved : kArmOk;
    };
    int why = step();
    if (why == kArmOk) {
      if (!flevel(mb.fs, flo, fhi)) exact_level_fp(c, mb.T, mb.ts, flo, fhi);
      if (!cut_below) slow(6);
      const uint32_t h = probe_facet(d, G, k);
      go_on = h == kInvalid32;
      if (!go_on) {
        Mini mg;  // beta(G) <= cutoff = beta(F): the decrease must be strict
        if (!cut_below && !facet_miniball(c, G, k, mg)) why = kArmInternal;
        else if (!cut_below && !below(mg, mb.T, mb.ts, flo)) why = kArmPlateau;
        else term[a] = h;
      }
    }
    if (why != kArmOk) {  // failed arms, and the least of them with its status
      atomicAdd(stats + 2, 1ull);
      atomicMin(stats + 3, (unsigned long long)a << 8 | (unsigned long long)why);
    } else {
      atomicAdd(stats, 1ull);
      if (!cut_below) atomicAdd(stats + 1, 1ull);
    }
    atomicAdd(&g_descent_visits[blockIdx.x % kVisitStripes], (unsigned long long)visits);
  }
  __syncwarp();
  const uint32_t slot = warp_slot(go_on, out_count);
  if (!go_on) return;
  out_arm[slot] = a;
  QFacet q;
  for (int j = 0; j < kMaxFacet; ++j) q.F[j] = j < k ? G[j] : kInvalid32;
  for (int j = 0; j < 4; ++j) q.prev[j] = !cut_below && j < mb.ts ? mb.T[j] : kInvalid32;
  q.prev_lo = flo;
  out_fac[slot] = q;
}

}  // namespace

// ---- host state ---------------------------------------------------------------------
struct HierState {
  explicit HierState(Ctx& ctx) : held(ctx.hier_bytes), mem(ctx.hier_bytes) {}
  std::atomic<uint64_t>& held;  // device bytes of everything below
  std::vector<std::pair<void*, uint64_t>> allocs, scratch;  // kept with a result / not used after the descent
  uint64_t cap_events = 0, cap_arms = 0, cap_births = 0, cap_slots = 0;
  // device
  EvRec* ev_raw = nullptr;
  EvRec* ev = nullptr;          // facade order
  double* lmid_raw = nullptr;
  double* lerr_raw = nullptr;
  double* lmid = nullptr;
  double* lerr = nullptr;
  uint64_t* key = nullptr;
  uint64_t* key2 = nullptr;     // key-value sort scratch
  uint32_t* order0 = nullptr;
  uint32_t* order1 = nullptr;
  double* pre_hi = nullptr;
  double* suf_lo = nullptr;
  double* bsum = nullptr;
  uint32_t* ubsum = nullptr;
  uint32_t* uncertain = nullptr;
  uint8_t* eqprev = nullptr;
  uint32_t* lclass = nullptr;   // level class per facade index
  uint32_t* rank_order = nullptr;
  uint32_t* counters = nullptr; // [0] diag, [1] uncertain, [2] err, [3..18] rank histogram
  uint32_t* radix_counts = nullptr;
  uint32_t* bfac = nullptr;
  uint32_t* slots = nullptr;
  uint32_t* term = nullptr;
  unsigned long long* dstats = nullptr;  // [0] descent steps, [1] strictness checks passed, [2] failed arms, [3] least (arm, status)
  uint32_t* qcount = nullptr;   // [0] first-probe misses, [1], [2] step outputs (ping-pong)
  DeviceArena mem;              // (counted in held) the descent's queues, then the forest journal and its records
  uint32_t first_misses = 0, descent_rounds = 0;
  unsigned long long slow[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  unsigned long long visits[kVisitStripes] = {};  // ball-query node visits of the descent steps
  // host results
  uint32_t n = 0, K = 0, keff = 0;
  int S = 0;
  uint64_t events = 0, diagnostics = 0;
  uint32_t* d_cls_rp = nullptr;       // device views (event capacity)
  uint32_t* d_size_rp = nullptr;
  uint32_t* d_armoff = nullptr;
  uint32_t* d_removed = nullptr;
  // exact order of the facade's tie runs on the device (capacities kept across calls)
  WL* tie_num = nullptr;   // [tie_cap] |N|^2 of each run member
  WL* tie_a2 = nullptr;    // [tie_cap] A^2
  uint32_t* tie_idx = nullptr;
  uint32_t* tie_tmp = nullptr;
  uint32_t* tie_pos = nullptr;
  uint32_t* run_off = nullptr;
  uint32_t* run_lo = nullptr;
  uint64_t tie_cap = 0, run_cap = 0;
  bool complete = false;   // `journal` and d_removed hold the result of the last call
  uint64_t families = 0, births = 0, arm_seeds = 0;
  JournalOut journal;
  uint32_t decision = EHGP_ERR_NOT_BUILT;
  double ms_device = 0, ms_forest = 0, ms_descent = 0, ms_ties = 0;
  uint64_t descent_steps = 0, arms = 0, exact_boundaries = 0;
  cudaEvent_t ev_step[2] = {nullptr, nullptr};  // around each descent-step launch
  double ms_steps = 0;                          // summed launch times of the descent rounds
  uint64_t step_launches = 0;
  uint32_t part_arms = 0;  // arms per part of the descent (0: one part); results never depend on it
};

namespace {

template <class T>
cudaError_t halloc(HierState& h, T** p, uint64_t count, std::vector<std::pair<void*, uint64_t>>& list) {
  void* q = nullptr;
  const uint64_t bytes = count * sizeof(T) + 16;
  list.reserve(list.size() + 1);
  const cudaError_t e = cudaMalloc(&q, bytes);
  if (e != cudaSuccess) return e;
  list.push_back({q, bytes});
  h.held += bytes;
  *p = (T*)q;
  return cudaSuccess;
}

void hfree(HierState& h, std::vector<std::pair<void*, uint64_t>>& list) {
  for (const auto& a : list) {
    cudaFree(a.first);
    h.held -= a.second;
  }
  list.clear();
}

// Frees the event arrays; the facade goes with them.
void hfree_all(HierState& h) {
  hfree(h, h.allocs);
  hfree(h, h.scratch);
  h.qcount = nullptr;
  h.events = 0;
  h.complete = false;
  h.decision = EHGP_ERR_NOT_BUILT;
  h.cap_events = h.cap_arms = h.cap_births = h.cap_slots = 0;
}

void free_ties(HierState& h) {
  for (void* q : {(void*)h.tie_num, (void*)h.tie_a2, (void*)h.tie_idx, (void*)h.tie_tmp, (void*)h.tie_pos,
                  (void*)h.run_off, (void*)h.run_lo})
    if (q) cudaFree(q);
  h.tie_num = h.tie_a2 = nullptr;
  h.tie_idx = h.tie_tmp = h.tie_pos = h.run_off = h.run_lo = nullptr;
  h.held -= h.tie_cap * (2 * sizeof(WL) + 12) + h.run_cap * 8;
  h.tie_cap = h.run_cap = 0;
}

cudaError_t ensure_events(HierState& h, uint64_t m) {
  if (m <= h.cap_events && !h.scratch.empty()) return cudaSuccess;
  hfree_all(h);
  const uint64_t cap = m + m / 8 + 1024;
  cudaError_t e;
#define HA(p, c) if ((e = halloc(h, &(p), (c), h.allocs)) != cudaSuccess) return e
#define HS(p, c) if ((e = halloc(h, &(p), (c), h.scratch)) != cudaSuccess) return e
  HA(h.ev_raw, cap);
  HA(h.ev, cap);
  HS(h.lmid_raw, cap);
  HS(h.lerr_raw, cap);
  HS(h.lmid, cap);
  HS(h.lerr, cap);
  HS(h.key, cap);
  HS(h.key2, cap);
  HA(h.order0, cap);
  HS(h.order1, cap);
  HS(h.pre_hi, cap);
  HS(h.suf_lo, cap);
  HA(h.bsum, cap / 1024 + 2);
  HA(h.ubsum, cap / 1024 + 2);
  HS(h.uncertain, 1u << 20);
  HS(h.eqprev, cap);
  HS(h.lclass, cap);
  HA(h.rank_order, cap);
  HA(h.counters, 32);
  HA(h.radix_counts, radix_counts_words(cap));
  HS(h.bfac, cap * kMaxFacet);
  HA(h.d_cls_rp, cap);
  HS(h.d_size_rp, cap);
  HA(h.d_armoff, cap + 1);
  HA(h.dstats, 4);
  const uint64_t arms = 4 * cap;
  HA(h.term, arms);
  HA(h.d_removed, arms);
  uint64_t slots = 1;
  while (slots < 2 * cap + 1024) slots <<= 1;
  HS(h.slots, slots);
#undef HA
#undef HS
  h.cap_events = cap;
  h.cap_arms = arms;
  h.cap_slots = slots;
  return cudaSuccess;
}


void scan_minmax(cudaStream_t st, uint32_t m, const double* mid, const double* err, double* out, double* bsum,
                 bool forward_max, uint64_t* launches) {
  const uint32_t nb = nblk(m, 1024);
  if (forward_max) {
    k_scan_blocks<<<nb, 256, 0, st>>>(m, mid, err, 1.0, 0, out, bsum, OpMax{}, -INFINITY);
    k_carry<<<1, 1024, 0, st>>>(nb, bsum, OpMax{}, -(double)INFINITY);
    k_scan_apply<<<nblk(m, kT), kT, 0, st>>>(m, 0, out, bsum, OpMax{});
  } else {
    k_scan_blocks<<<nb, 256, 0, st>>>(m, mid, err, -1.0, 1, out, bsum, OpMin{}, INFINITY);
    k_carry<<<1, 1024, 0, st>>>(nb, bsum, OpMin{}, (double)INFINITY);
    k_scan_apply<<<nblk(m, kT), kT, 0, st>>>(m, 1, out, bsum, OpMin{});
  }
  *launches += 3;
}

}  // namespace

void hier_trim(Ctx& ctx) {
  if (!ctx.hier) return;
  cudaSetDevice(ctx.device);
  hfree_all(*ctx.hier);
  free_ties(*ctx.hier);
  ctx.hier->mem.release();
}

void hier_free(Ctx& ctx) {
  if (!ctx.hier) return;
  hier_trim(ctx);
  for (cudaEvent_t ev : ctx.hier->ev_step)
    if (ev) cudaEventDestroy(ev);
  delete ctx.hier;
  ctx.hier = nullptr;
}

int hier_run(Ctx& ctx, uint32_t K) {
  if (!ctx.hier) ctx.hier = new HierState(ctx);
  HierState& h = *ctx.hier;
  const uint32_t n = (uint32_t)ctx.built_n;
  cudaStream_t st = ctx.stream;
  LbvhBuffers& b = ctx.lb;
  GeomBuffers& g = ctx.gb;
  uint64_t launches = 0;
  h.decision = EHGP_ERR_NOT_BUILT;
  h.complete = false;
  h.arm_seeds = 0;
  h.n = n;
  h.K = K;
  h.keff = K < n ? K : n;
  if (K == 0 || K > 10) return abi_fail(&ctx, EHGP_ERR_INVALID_ARGUMENT, "K_max must be in [1, 10]");
  // supports for this K
  uint32_t np = 0, nh = 0;
  if (!(ctx.pb.K == K && ctx.pb.resident)) {  // pair supports of this cloud and K
    const int s = pairs_run(ctx, K, &np);
    if (s != EHGP_OK) return s;
  }
  np = ctx.pb.count;
  if (ctx.hb.K != K) {
    const int s = higher_run(ctx, K, &nh);
    if (s != EHGP_OK) return s;
  }
  nh = ctx.hb.count;
  cudaEventRecord(ctx.ev0, st);
  const uint64_t total = (uint64_t)np + nh;
  h.mem.largest = ctx.hier_largest;
  cudaError_t e = ensure_events(h, total + 1);
  if (e == cudaErrorMemoryAllocation) {  // the last call's working memory is made again below
    cudaGetLastError();
    h.mem.reset(0);
    e = ensure_events(h, total + 1);
  }
  if (e != cudaSuccess) return abi_fail(&ctx, EHGP_ERR_OUT_OF_MEMORY, "hierarchy buffers do not fit the device");
  cudaMemsetAsync(h.counters, 0, 32 * sizeof(uint32_t), st);
  cudaMemsetAsync(h.dstats, 0, 4 * sizeof(unsigned long long), st);
  {
    const unsigned long long zero[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    cudaMemcpyToSymbolAsync(g_descent_slow, zero, sizeof(zero), 0, cudaMemcpyHostToDevice, st);
    static const unsigned long long zv[kVisitStripes] = {};
    cudaMemcpyToSymbolAsync(g_descent_visits, zv, sizeof(zv), 0, cudaMemcpyHostToDevice, st);
  }
  if (total)
    k_ev_build<<<nblk(total, kT), kT, 0, st>>>(np, nh, (const PairRecD*)ctx.pb.sorted, (const HigherRecD*)ctx.hb.sorted,
                                                b.px, b.py, b.pz, g.scale, h.ev_raw, h.lmid_raw, h.lerr_raw, h.key,
                                                h.counters);
  ++launches;
  uint32_t hc[2] = {0, 0};
  cudaMemcpyAsync(hc, h.counters, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "hierarchy events");
  h.diagnostics = hc[0];
  const uint32_t m = (uint32_t)(total - hc[0]);
  h.events = m;
  // facade order by the FP64 level midpoints (diagnostics sort last)
  RadixScratch rs{h.radix_counts, ctx.radix.state, ctx.radix.wait};
  if (total) {
    k_iota<<<nblk(total, kT), kT, 0, st>>>((uint32_t)total, h.order0);
    ++launches;
    // facade order: the event keys (FP64 level midpoints, diagnostics last) move with the indices
    const int passes = radix_sort_kv(st, (uint32_t)total, h.order0, h.order1, h.key, h.key2, 64, rs, &launches);
    k_ev_gather<<<nblk(total, kT), kT, 0, st>>>((uint32_t)total, h.order0, h.order1, ctx.radix.state, passes, h.ev_raw,
                                                 h.lmid_raw, h.lerr_raw, h.ev, h.lmid, h.lerr);
    ++launches;
  }
  int scale_h[4];
  cudaMemcpyAsync(scale_h, g.scale, sizeof(scale_h), cudaMemcpyDeviceToHost, st);
  cudaMemsetAsync(h.eqprev, 0, m + 1, st);
  uint32_t unc = 0;
  if (m > 1) {
    scan_minmax(st, m, h.lmid, h.lerr, h.pre_hi, h.bsum, true, &launches);
    scan_minmax(st, m, h.lmid, h.lerr, h.suf_lo, h.bsum, false, &launches);
    k_uncertain<<<nblk(m, kT), kT, 0, st>>>(m, h.pre_hi, h.suf_lo, h.uncertain, 1u << 20, h.counters + 1);
    ++launches;
    cudaMemcpyAsync(&unc, h.counters + 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  }
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "hierarchy facade order");
  h.S = scale_h[0];
  if (unc > (1u << 20)) return abi_fail(&ctx, EHGP_ERR_CAPACITY, "too many uncertain level boundaries in the facade");
  double ms_ties = 0;
  if (unc) {
    const auto tt0 = std::chrono::steady_clock::now();
    std::vector<uint32_t> list(unc);
    cudaMemcpy(list.data(), h.uncertain, unc * sizeof(uint32_t), cudaMemcpyDeviceToHost);
    std::sort(list.begin(), list.end());
    // maximal runs of positions whose order the FP64 intervals leave open: a run starts one
    // before its first uncertain boundary (that boundary before it is certain)
    std::vector<uint32_t> run_off, run_lo, idx;
    for (size_t i = 0; i < list.size();) {
      const uint32_t s0 = list[i] - 1;
      uint32_t s1 = list[i];
      size_t j = i + 1;
      while (j < list.size() && list[j] == s1 + 1) s1 = list[j++];
      run_off.push_back((uint32_t)idx.size());
      run_lo.push_back(s0);
      for (uint32_t t = s0; t <= s1; ++t) idx.push_back(t);
      i = j;
    }
    run_off.push_back((uint32_t)idx.size());
    const uint32_t cnt = (uint32_t)idx.size(), nruns = (uint32_t)run_lo.size();
    // settled on the device: exact level keys per member, then a merge sort per run
    if (h.tie_cap < cnt || h.run_cap < nruns + 1) {
      free_ties(h);
      const uint64_t tc = cnt + cnt / 4 + 64, rc = nruns + nruns / 4 + 64;
      if (cudaMalloc(&h.tie_num, tc * sizeof(WL)) != cudaSuccess || cudaMalloc(&h.tie_a2, tc * sizeof(WL)) != cudaSuccess ||
          cudaMalloc(&h.tie_idx, tc * 4) != cudaSuccess || cudaMalloc(&h.tie_tmp, tc * 4) != cudaSuccess ||
          cudaMalloc(&h.tie_pos, tc * 4) != cudaSuccess || cudaMalloc(&h.run_off, rc * 4) != cudaSuccess ||
          cudaMalloc(&h.run_lo, rc * 4) != cudaSuccess) {
        cudaGetLastError();
        return abi_fail(&ctx, EHGP_ERR_OUT_OF_MEMORY, "the facade tie runs do not fit the device");
      }
      h.tie_cap = tc;
      h.run_cap = rc;
      h.held += tc * (2 * sizeof(WL) + 12) + rc * 8;
    }
    // members' records are copied (ev_raw is free between the facade gather and the level
    // classes) so that the sort writes the facade in place
    cudaMemcpyAsync(h.tie_pos, idx.data(), (uint64_t)cnt * 4, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(h.run_off, run_off.data(), (uint64_t)(nruns + 1) * 4, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(h.run_lo, run_lo.data(), (uint64_t)nruns * 4, cudaMemcpyHostToDevice, st);
    k_run_gather<<<nblk(cnt, kT), kT, 0, st>>>(cnt, h.tie_pos, h.ev, h.lmid, h.lerr, h.ev_raw, h.lmid_raw, h.lerr_raw);
    const Cloud dc{b.px, b.py, b.pz, h.S};
    k_tie_keys<<<nblk(cnt, 128), 128, 0, st>>>(cnt, h.tie_pos, h.ev, dc, h.tie_num, h.tie_a2);
    k_tie_sort<<<nblk(nruns, 64), 64, 0, st>>>(nruns, h.run_off, h.run_lo, h.tie_num, h.tie_a2, h.ev_raw, h.lmid_raw,
                                               h.lerr_raw, h.tie_idx, h.tie_tmp, h.ev, h.lmid, h.lerr, h.eqprev);
    launches += 3;
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "facade tie runs");
    ms_ties = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - tt0).count();
  }
  // level classes
  if (m) {
    uint32_t* flag = h.order1;  // scratch
    k_level_class<<<nblk(m, kT), kT, 0, st>>>(m, h.eqprev, flag);
    const uint32_t nb = nblk(m, 1024);
    k_sum_blocks<<<nb, 256, 0, st>>>(m, flag, h.lclass, h.ubsum);
    k_carry<<<1, 1024, 0, st>>>(nb, h.ubsum, OpSum{}, 0u);
    k_sum_apply<<<nblk(m, kT), kT, 0, st>>>(m, h.lclass, h.ubsum, 1);
    launches += 4;
  }
  // stable partition by closed rank
  uint32_t hist[16] = {0};
  int rpasses = 0;
  if (m) {
    k_rank_key<<<nblk(m, kT), kT, 0, st>>>(m, h.ev, h.key, h.order0, h.counters + 3);
    const IndirectKey stages[1] = {{h.key, 0}};
    const int bits[1] = {8};
    rpasses = radix_sort_indirect(st, m, h.order0, h.order1, stages, bits, 1, rs, &launches);
    k_rank_gather<<<nblk(m, kT), kT, 0, st>>>(m, h.order0, h.order1, ctx.radix.state, rpasses, h.rank_order);
    launches += 2;
    cudaMemcpyAsync(hist, h.counters + 3, 16 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  }
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "hierarchy facade");
  if (h.diagnostics) {
    h.decision = EHGP_ERR_DEGENERATE;
    return abi_fail(&ctx, EHGP_ERR_DEGENERATE,
                    "relevant extra-shell diagnostics: the Morse event journal is not built");
  }
  const uint32_t keff = h.keff;
  // rank segments: rb[r] = first position of rank r in rank_order
  uint64_t rb[18] = {0};
  for (int r = 0; r < 16; ++r) rb[r + 1] = rb[r] + hist[r];
  // births (orders 2..keff): handle n + (position - rb[2])
  const uint64_t nb_higher = rb[keff + 1 > 16 ? 16 : keff + 1] - rb[2];
  if (nb_higher) {
    cudaMemsetAsync(h.slots, 0xff, h.cap_slots * sizeof(uint32_t), st);
    k_birth_insert<<<nblk(nb_higher, kT), kT, 0, st>>>((uint32_t)nb_higher, n, (uint32_t)rb[2], h.rank_order, h.ev,
                                                       h.bfac, h.slots, (uint32_t)(h.cap_slots - 1), h.counters + 2);
    ++launches;
  }
  // families: saddle events of ranks 2..keff+1 in rank-partition order; arms per support point
  const uint64_t fam_lo = rb[2], fam_hi = rb[std::min<uint32_t>(keff + 2, 16)];
  const uint64_t nfam = fam_hi - fam_lo;
  uint64_t narms = 0;
  uint32_t herr = 0;
  if (m) {
    k_rank_info<<<nblk(m, kT), kT, 0, st>>>(m, h.rank_order, h.ev, h.lclass, h.d_cls_rp, h.d_size_rp);
    ++launches;
  }
  if (nfam) {  // arm offsets: inclusive sum of the family sizes into d_armoff + 1
    const uint32_t nb = nblk(nfam, 1024);
    k_sum_blocks<<<nb, 256, 0, st>>>((uint32_t)nfam, h.d_size_rp + fam_lo, h.d_armoff + 1, h.ubsum);
    k_carry<<<1, 1024, 0, st>>>(nb, h.ubsum, OpSum{}, 0u);
    k_sum_apply<<<nblk(nfam, kT), kT, 0, st>>>((uint32_t)nfam, h.d_armoff + 1, h.ubsum, 0);
    cudaMemsetAsync(h.d_armoff, 0, sizeof(uint32_t), st);
    launches += 3;
    uint32_t na = 0;
    cudaMemcpyAsync(&na, h.d_armoff + nfam, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "arm offsets");
    narms = na;
  }
  if (narms > h.cap_arms) return abi_fail(&ctx, EHGP_ERR_CAPACITY, "strict arms exceed the hierarchy buffers");
  h.arms = narms;
  h.exact_boundaries = unc;
  JournalIn in;
  in.n = n;
  in.keff = keff;
  in.handles = (uint32_t)(n + nb_higher);
  in.families = (uint32_t)nfam;
  in.arms = (uint32_t)narms;
  for (uint32_t k = 1; k <= keff + 1; ++k) {
    in.fam0[k] = (uint32_t)(rb[std::min<uint32_t>(k + 1, 16)] - fam_lo);
    in.han0[k] = k == 1 ? 0 : (uint32_t)(n + rb[k] - rb[2]);
  }
  in.rounds = std::min(ctx.forest_rounds, kForestRounds);
  in.ev = h.rank_order + fam_lo;
  in.cls = h.d_cls_rp + fam_lo;
  in.armoff = h.d_armoff;
  in.term = h.term;
  // ---- strict-arm descent ----
  // One part unless a schedule says otherwise: the fewer parts, the fewer rounds, and a round
  // is a few launches and a look at its queue's length.
  uint32_t part_fams = h.part_arms ? std::max(1u, h.part_arms / 4u) : (uint32_t)nfam;
  const uint64_t journal = journal_bytes(in);
  uint64_t q_cap = 0;
  uint32_t *q_arm[2], *q_hard;
  QFacet* q_fac[2];
  uint4* q_sup;
  auto queues = [&]() -> cudaError_t {
    const uint64_t bytes = q_cap * (2 * (4 + sizeof(QFacet)) + 4 + 16) + 4096;
    cudaError_t r = h.mem.reset(std::max(journal, bytes));
    if (r == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      r = h.mem.reset(bytes);
    }
    for (int i = 0; i < 2; ++i) {
      if (r == cudaSuccess) r = h.mem.take(&q_arm[i], q_cap);
      if (r == cudaSuccess) r = h.mem.take(&q_fac[i], q_cap);
    }
    if (r == cudaSuccess) r = h.mem.take(&q_hard, q_cap);
    if (r == cudaSuccess) r = h.mem.take(&q_sup, q_cap);
    return r;
  };
  // Queues for `need` entries (0: a third of a part's arms, what misses the first probe, and some room); parts
  // become smaller while the device has none.
  auto room = [&](uint64_t need) -> bool {
    for (;; need = 0, part_fams = (part_fams + 3) / 4) {
      const uint64_t arms = std::min<uint64_t>(narms, 4ull * part_fams);
      q_cap = need ? need : std::min<uint64_t>(arms, std::max<uint64_t>(arms * 3 / 8, 1u << 16)) + 32;
      if (queues() == cudaSuccess) return true;
      cudaGetLastError();
      if (part_fams <= 1024) return false;
    }
  };
  auto no_queue = [&] {
    cudaGetLastError();
    return abi_fail(&ctx, EHGP_ERR_OUT_OF_MEMORY, "descent queue buffers do not fit the device");
  };
  if (!room(0)) return no_queue();
  if (!h.qcount && (e = halloc(h, &h.qcount, 4, h.allocs)) != cudaSuccess)
    return abi_fail(&ctx, EHGP_ERR_OUT_OF_MEMORY, "descent queue");
  const DescentParams dp{n, 2 * n - 2, g.tnodes, b.px, b.py, b.pz, h.S, h.slots, (uint32_t)(h.cap_slots - 1), h.bfac,
                         (uint32_t)nb_higher, in.ev, h.lmid, h.lerr};
  uint32_t misses = 0, max_rounds = 0;
  h.descent_steps = 0;
  h.ms_steps = 0;
  h.step_launches = 0;
  for (cudaEvent_t& ev : h.ev_step)
    if (!ev && cudaEventCreate(&ev) != cudaSuccess) ev = nullptr;
  cudaEventRecord(ctx.evk0, st);
  cudaMemsetAsync(h.dstats + 3, 0xff, sizeof(unsigned long long), st);
  for (uint32_t f0 = 0, nf = 0; f0 < nfam; f0 += nf) {
    uint32_t pending = 0;
    for (;;) {  // count -> grow (or cut the part) -> queue
      nf = std::min<uint32_t>(part_fams, (uint32_t)nfam - f0);
      cudaMemsetAsync(h.qcount, 0, 4 * sizeof(uint32_t), st);
      k_arm_probe<<<nblk(nf, kT), kT, 0, st>>>(dp, f0, nf, in.ev, h.d_armoff, h.ev, h.d_removed, h.term, q_arm[0],
                                               q_fac[0], (uint32_t)q_cap, h.qcount);
      ++launches;
      cudaMemcpyAsync(&pending, h.qcount, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
      cudaMemcpyAsync(&herr, h.counters + 2, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
      if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "strict-arm seeds");
      if (herr) return abi_fail(&ctx, EHGP_ERR_CAPACITY, "the birth facet table is full");
      if (pending <= q_cap) break;
      if (!room(pending)) return no_queue();
    }
    misses += pending;
    int cur = 0;
    uint32_t rounds = 0;
    while (pending) {
      if (++rounds > (uint32_t)kDescentSteps) {
        h.decision = EHGP_ERR_DEGENERATE;
        return abi_fail(&ctx, EHGP_ERR_DEGENERATE, "a strict arm descent exceeded its step budget");
      }
      uint32_t* oc = h.qcount + 1;  // [1] queued for the next round, [2] left open
      cudaMemsetAsync(oc, 0, 2 * sizeof(uint32_t), st);
      if (h.ev_step[0]) cudaEventRecord(h.ev_step[0], st);
      int spasses = -1;  // large queues run in Morton order of their facets
      if (pending >= kSortQueueMin && pending <= h.cap_events) {
        k_queue_keys<<<nblk(pending, kT), kT, 0, st>>>(pending, q_fac[cur], b.code, h.key, h.order0);
        ++launches;
        spasses = radix_sort_kv(st, pending, h.order0, h.order1, h.key, h.key2, 24, rs, &launches);
      }
      k_facet_ball<<<nblk(pending, kFT), kFT, 0, st>>>(dp, pending, q_fac[cur], ctx.radix.state, spasses, h.order0, h.order1,
                                                       q_sup, q_hard, oc + 1);
      k_facet_step<<<nblk(pending, kFT), kFT, 0, st>>>(dp, pending, q_arm[cur], q_fac[cur], q_sup, ctx.radix.state, spasses,
                                                       h.order0, h.order1, q_arm[1 - cur], q_fac[1 - cur], oc, h.term,
                                                       h.dstats, q_hard, oc + 1);
      launches += 2;
      ++h.step_launches;
      uint32_t hq[2] = {0, 0};
      cudaMemcpyAsync(hq, oc, sizeof(hq), cudaMemcpyDeviceToHost, st);
      if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "strict-arm descent");
      if (hq[1]) {
        k_facet_exact<<<nblk(hq[1], 128), 128, 0, st>>>(dp, hq[1], q_hard, q_arm[cur], q_fac[cur], q_arm[1 - cur],
                                                        q_fac[1 - cur], oc, h.term, h.dstats);
        ++launches;
        cudaMemcpyAsync(hq, oc, sizeof(hq), cudaMemcpyDeviceToHost, st);
      }
      if (h.ev_step[1]) cudaEventRecord(h.ev_step[1], st);
      if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "strict-arm descent");
      pending = hq[0];
      if (h.ev_step[0] && h.ev_step[1]) {
        float sm = 0.f;
        if (cudaEventElapsedTime(&sm, h.ev_step[0], h.ev_step[1]) == cudaSuccess) h.ms_steps += sm;
      }
      cur = 1 - cur;
    }
    max_rounds = std::max(max_rounds, rounds);
  }
  cudaEventRecord(ctx.evk1, st);
  unsigned long long dst[4] = {0, 0, 0, 0};
  cudaMemcpyAsync(dst, h.dstats, sizeof(dst), cudaMemcpyDeviceToHost, st);
  cudaMemcpyFromSymbolAsync(h.slow, g_descent_slow, sizeof(h.slow), 0, cudaMemcpyDeviceToHost, st);
  cudaMemcpyFromSymbolAsync(h.visits, g_descent_visits, sizeof(h.visits), 0, cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&herr, ctx.d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "strict-arm descent");
  if (herr) return abi_device_status(&ctx, herr);
  h.first_misses = misses;
  h.descent_rounds = max_rounds;
  h.descent_steps = dst[0];
  if (dst[2]) {  // report the first failed arm
    static const char* msg[] = {"", "a strict arm descent is unresolved", "a strict arm descent met a plateau",
                                "a strict arm descent exceeded its ball-query capacity",
                                "a strict arm descent exceeded its step budget",
                                "a strict arm descent found no consistent exact miniball or top-k"};
    const uint32_t why = (uint32_t)(dst[3] & 0xff);
    const int status = why == kArmCapacity ? EHGP_ERR_CAPACITY : EHGP_ERR_DEGENERATE;
    h.decision = (uint32_t)status;
    return abi_fail(&ctx, status, msg[why < 6 ? why : 5]);
  }
  // ---- forest journal, in the queues' memory ----
  int js = EHGP_ERR_OUT_OF_MEMORY;
  if (h.mem.reset(journal) == cudaSuccess) {
    h.mem.release_host();
    js = journal_run(ctx, in, h.mem, h.journal, &launches);
  }
  if (js == EHGP_ERR_OUT_OF_MEMORY) {  // no room: what only the descent needed goes, the records leave the device
    cudaGetLastError();
    hfree(h, h.scratch);
    h.mem.reset(0);
    h.mem.spilled = true;
    js = journal_run(ctx, in, h.mem, h.journal, &launches);
  }
  ctx.forest_rest = h.journal.rest;
  if (js != EHGP_OK) return js;
  cudaEventRecord(ctx.ev1, st);
  if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return abi_cuda_fail(&ctx, e, "forest journal");
  {
    float ms = 0;
    cudaEventElapsedTime(&ms, ctx.ev0, ctx.ev1);
    h.ms_device = ms;
    cudaEventElapsedTime(&ms, ctx.evk1, ctx.ev1);
    h.ms_forest = ms;
    if (narms) {
      cudaEventElapsedTime(&ms, ctx.evk0, ctx.evk1);
      ctx.kernel_ms = ms;
      h.ms_descent = ms;
    }
  }
  h.ms_ties = ms_ties;
  ctx.last_launches = launches;
  ctx.last_ms = h.ms_device;
  h.arm_seeds = narms;
  h.families = nfam;
  h.births = in.handles;
  h.complete = true;
  h.decision = EHGP_OK;
  return EHGP_OK;
}

}  // namespace ehgp

extern "C" {

int ehgp_hierarchy(ehgp_ctx* ctx, uint32_t K, ehgp_hier_counts* counts) try {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  ctx->last_error.clear();
  if (ctx->poisoned) return ehgp::abi_fail(ctx, EHGP_ERR_POISONED, "the context is poisoned by an earlier CUDA failure");
  if (ctx->built_n == 0) return ehgp::abi_fail(ctx, EHGP_ERR_NOT_BUILT, "ehgp_hierarchy needs a resident LBVH");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "cudaSetDevice");
  if (!ctx->geom_ready) {
    ehgp::geom_prepare(*ctx, (uint32_t)ctx->built_n);
    if ((e = cudaGetLastError()) != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "traversal preparation");
  }
  if (!ctx->scale_valid)
    return ehgp::abi_fail(ctx, EHGP_ERR_NUMERIC_RANGE, "the cloud exceeds the exact fixed-point range");
  cudaMemsetAsync(ctx->d_err, 0, sizeof(uint32_t), ctx->stream);
  const int s = ehgp::hier_run(*ctx, K);
  if (counts) {
    std::memset(counts, 0, sizeof(*counts));
    if (ctx->hier) {
      const ehgp::HierState& h = *ctx->hier;
      counts->events = h.events;
      counts->diagnostics = h.diagnostics;
      if (h.complete) {
        const ehgp::JournalOut& j = h.journal;
        counts->journal_batches = j.n_batches;
        counts->role_records = j.n_roles;
        counts->families = h.families;
        counts->arm_seeds = h.arm_seeds;
        counts->birth_records = h.births;
        counts->nodes = j.n_nodes;
        counts->children = j.n_children;
        counts->arm_bindings = h.arm_seeds;
        counts->saddle_records = h.families;
        counts->atomic_groups = j.n_groups;
        counts->final_roots = j.roots.size();
        counts->vertical_assignments = j.n_vert;
      }
      counts->k_eff = h.keff;
    }
    counts->decision = (uint32_t)s;
  }
  return s;
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

int ehgp_hier_schedule(ehgp_ctx* ctx, uint32_t chunk_batches, uint32_t part_arms, uint32_t host_threads) try {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  if (!ctx->hier) ctx->hier = new ehgp::HierState(*ctx);
  (void)chunk_batches;  // the forest journal runs on the device
  (void)host_threads;
  ctx->hier->part_arms = part_arms;
  return EHGP_OK;
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

int ehgp_hier_copy(ehgp_ctx* ctx, const ehgp_hier_out* out) try {
  if (!ctx || !out) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  if (ctx->poisoned) return ehgp::abi_fail(ctx, EHGP_ERR_POISONED, "the context is poisoned by an earlier CUDA failure");
  if (!ctx->hier) return ehgp::abi_fail(ctx, EHGP_ERR_NOT_BUILT, "no hierarchy result is resident");
  cudaError_t e = cudaSetDevice(ctx->device);  // the records are on it, and the copies' events belong to it
  if (e != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "cudaSetDevice");
  ehgp::HierState& h = *ctx->hier;
  const ehgp::JournalOut& j = h.journal;
  std::vector<ehgp::CopyOut> list;
  auto add = [&](void* dst, const void* src, uint64_t count, uint64_t size) {
    if (dst && count)
      list.push_back({static_cast<char*>(dst), static_cast<const char*>(src), count * size,
                      h.mem.on_host(src) ? cudaMemcpyHostToHost : cudaMemcpyDeviceToHost});
  };
  add(out->events, h.ev, h.events, sizeof(ehgp::EvRec));
  if (h.complete) {
    add(out->journal_batches, j.jb, j.n_batches, sizeof *j.jb);
    add(out->roles, j.roles, j.n_roles, sizeof *j.roles);
    add(out->families, j.fam, h.families, sizeof *j.fam);
    add(out->arm_removed, h.d_removed, h.arm_seeds, 4);
    add(out->nodes, j.nodes, j.n_nodes, sizeof *j.nodes);
    add(out->children, j.children, j.n_children, 4);
    add(out->births, j.births, h.births, sizeof *j.births);
    add(out->bindings, j.bindings, h.arm_seeds, sizeof *j.bindings);
    add(out->saddles, j.saddles, h.families, sizeof *j.saddles);
    add(out->groups, j.groups, j.n_groups, sizeof *j.groups);
    add(out->batches, j.fb, j.n_batches, sizeof *j.fb);
    add(out->vertical, j.vert, j.n_vert, sizeof *j.vert);
    if (out->roots && !j.roots.empty()) std::memcpy(out->roots, j.roots.data(), j.roots.size() * sizeof j.roots[0]);
  }
  if ((e = ehgp::copy_out(*ctx, list)) != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "hierarchy copy");
  return EHGP_OK;
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

int ehgp_hier_stats(const ehgp_ctx* ctx, double* ms, uint64_t* stats) {
  if (!ctx || !ctx->hier) return EHGP_ERR_INVALID_ARGUMENT;
  const ehgp::HierState& h = *ctx->hier;
  if (ms) {
    ms[0] = h.ms_device;
    ms[1] = h.ms_descent;
    ms[2] = h.ms_forest;
    for (int i = 3; i < 25; ++i) ms[i] = 0.0;
    ms[4] = h.ms_ties;
  }
  if (stats) {
    stats[0] = h.arms;
    stats[1] = h.descent_steps;
    stats[2] = h.exact_boundaries;
    stats[3] = h.events;
    stats[4] = h.first_misses;
    stats[5] = h.descent_rounds;
    for (int i = 0; i < 7; ++i) stats[6 + i] = h.slow[i];
    uint64_t v = 0;
    for (int i = 0; i < ehgp::kVisitStripes; ++i) v += h.visits[i];
    stats[13] = v;
    stats[14] = h.step_launches;
  }
  if (ms) ms[24] = h.ms_steps;
  return EHGP_OK;
}

int ehgp_event_supports(ehgp_ctx* ctx, const uint32_t* events, uint64_t count, uint32_t* out) try {
  if (!ctx || (count && (!events || !out))) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  if (ctx->poisoned) return ehgp::abi_fail(ctx, EHGP_ERR_POISONED, "the context is poisoned by an earlier CUDA failure");
  if (!ctx->hier || ctx->hier->decision != EHGP_OK || !ctx->hier->order0 || !ctx->hier->ev_raw)
    return ehgp::abi_fail(ctx, EHGP_ERR_NOT_BUILT, "ehgp_event_supports needs a hierarchy result");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "cudaSetDevice");
  ehgp::HierState& h = *ctx->hier;
  cudaStream_t st = ctx->stream;
  // chunks through the facade's scratch (index: order0, output: ev_raw), free after the call
  const uint64_t chunk = std::min<uint64_t>(h.cap_events, (h.cap_events * sizeof(ehgp::EvRec)) / 20);
  for (uint64_t b0 = 0; b0 < count; b0 += chunk) {
    const uint32_t m = (uint32_t)std::min<uint64_t>(chunk, count - b0);
    cudaMemcpyAsync(h.order0, events + b0, (uint64_t)m * 4, cudaMemcpyHostToDevice, st);
    ehgp::k_event_supports<<<ehgp::nblk(m, ehgp::kT), ehgp::kT, 0, st>>>(m, h.order0, h.ev, (uint32_t)h.events,
                                                                        (uint32_t*)h.ev_raw);
    e = ehgp::copy_out(*ctx, {{(char*)(out + 5 * b0), (const char*)h.ev_raw, (uint64_t)m * 20}});
    if (e != cudaSuccess) return ehgp::abi_cuda_fail(ctx, e, "facade event supports");
  }
  return EHGP_OK;
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

int ehgp_event_level(ehgp_ctx* ctx, uint64_t event, uint64_t* num, uint64_t* den, int32_t* scale) {
  if (!ctx || !num || !den) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  if (!ctx->hier || event >= ctx->hier->events)
    return ehgp::abi_fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "no such facade event");
  const ehgp::HierState& h = *ctx->hier;
  ehgp::EvRec r;
  cudaError_t ce = cudaMemcpy(&r, h.ev + event, sizeof r, cudaMemcpyDeviceToHost);
  if (ce != cudaSuccess) return ehgp::abi_cuda_fail(ctx, ce, "facade event copy");
  if (r.size < 2 || r.size > 4) return ehgp::abi_fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "no such facade event");
  // the support's coordinates only (the cloud stays on the device)
  double sx[4], sy[4], sz[4];
  uint32_t local[4];
  for (uint32_t j = 0; j < r.size; ++j) {
    if ((ce = cudaMemcpy(sx + j, ctx->lb.px + r.ids[j], 8, cudaMemcpyDeviceToHost)) != cudaSuccess ||
        (ce = cudaMemcpy(sy + j, ctx->lb.py + r.ids[j], 8, cudaMemcpyDeviceToHost)) != cudaSuccess ||
        (ce = cudaMemcpy(sz + j, ctx->lb.pz + r.ids[j], 8, cudaMemcpyDeviceToHost)) != cudaSuccess)
      return ehgp::abi_cuda_fail(ctx, ce, "support coordinates");
    local[j] = j;
  }
  const ehgp::Cloud c{sx, sy, sz, h.S};
  ehgp::W A;
  ehgp::WV N;
  ehgp::exact_sphere(c, local, (int)r.size, A, N);
  using WL = ehgp::WL;
  const WL x = ehgp::widen<36>(N.x), y = ehgp::widen<36>(N.y), z = ehgp::widen<36>(N.z), a = ehgp::widen<36>(A);
  const WL nn = ehgp::wadd(ehgp::wadd(ehgp::wmul(x, x), ehgp::wmul(y, y)), ehgp::wmul(z, z));
  const WL dd = ehgp::wmul(ehgp::wmul(a, a), WL::from_i128(4));
  for (int i = 0; i < 36; ++i) {
    num[i] = nn.w[i];
    den[i] = dd.w[i];
  }
  if (scale) *scale = h.S;
  return EHGP_OK;
}

}  // extern "C"
