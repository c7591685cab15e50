// Stable LSD radix sort of 32-bit indices by 64-bit keys (sm_100a), 8 bits per pass.
//
// Serves every ordered output of the library: the canonical PointId order and the Morton leaf
// order (std::sort of src/cpu/spatial/point_cloud.cpp:58-62 and lbvh.cpp:93-100,512; stability over
// an input in PointId order gives the PointId tie-break), the EMST edge order, the support
// catalogues, the facade and its rank partition, the descent queues.
//
// The digit counts of a pass do not depend on the order of its input, so one kernel counts the digits
// of every pass, a second one turns them into digit bases and marks the passes whose keys share
// one digit (their scatter returns at once and the ping-pong buffer is not flipped), and a pass is one
// kernel: a block ranks a tile in shared memory, publishes its digit counts, sums those of the
// tiles before it while they appear (decoupled look-back: a tile's number is a ticket, so every
// tile it waits for has already started; the wait has a limit all the same), and writes the tile in
// digit order.  A wait that runs out ends with the block counting those tiles itself, so a sort always
// completes.  The host never synchronises inside a sort.  Up to kSmall items one block runs all
// passes in shared memory in one launch.
// Bound: HBM for large inputs, launches for small ones.  With four kernels per pass (tile histogram,
// row scan, digit bases, scatter of 1,024-item tiles) an LBVH build was 144 launches: 0.82 ms for 1,021
// points, 0.32 now.
#include "ehgp_internal.cuh"

namespace ehgp {
namespace {

constexpr int kT = 256, kWarps = kT / 32;
constexpr uint32_t kSmall = 2048;    // items that one block sorts on its own
constexpr int kSmallT = 512, kSmallWarps = kSmallT / 32, kSmallRows = kSmall / kSmallT;
constexpr int kRows = kRadixTile / kT;  // rows of 32 items per warp and tile

// State words: per pass (input buffer, trivial flag), then the digit bases of every pass, then the
// tile tickets.
constexpr int kBases = 2 * (kRadixMaxPasses + 1);
constexpr int kTickets = kBases + 256 * kRadixMaxPasses;
static_assert(kRadixStateWords >= kTickets + kRadixMaxPasses, "state layout");

struct Passes {  // of one sort: key source and shift
  IndirectKey stage[3];
  int first[4];  // first pass of each stage, then their number
  int stages;
};

// Key of item v in pass p (indirect sorts), its digit in place.
__device__ __forceinline__ uint32_t indirect_digit(const Passes& ps, int p, uint32_t v) {
  int s = 0;
  while (s + 1 < ps.stages && p >= ps.first[s + 1]) ++s;
  uint64_t w = __ldg(ps.stage[s].words + v);
  if (ps.stage[s].order) w = order_key(w);
  return (uint32_t)(w >> (8 * (p - ps.first[s]))) & 0xffu;
}

// Digit counts of every pass.  A warp whose lanes share a digit adds once (the high digits of most keys).
__device__ __forceinline__ void count_digit(uint32_t* hist, uint32_t d, bool on) {
  const uint32_t act = __ballot_sync(0xffffffffu, on);
  if (!act) return;
  const uint32_t first = __shfl_sync(0xffffffffu, d, __ffs((int)act) - 1);
  if (__all_sync(0xffffffffu, !on || d == first)) {
    if ((threadIdx.x & 31u) == 0) atomicAdd(hist + first, (uint32_t)__popc(act));
  } else if (on) {
    atomicAdd(hist + d, 1u);
  }
}

template <bool kKv>
__global__ void __launch_bounds__(kT) k_radix_counts(uint32_t n, const uint32_t* __restrict__ vals,
                                                     const uint64_t* __restrict__ keys, Passes ps, int passes,
                                                     uint32_t* __restrict__ state) {
  extern __shared__ uint32_t hist[];  // [passes][256]
  for (int i = threadIdx.x; i < passes * 256; i += kT) hist[i] = 0;
  __syncthreads();
  for (uint32_t b = blockIdx.x * kT; b < n; b += gridDim.x * kT) {
    const uint32_t i = b + threadIdx.x;
    const bool on = i < n;
    if (kKv) {
      const uint64_t key = on ? keys[i] : 0;
      for (int p = 0; p < passes; ++p) count_digit(hist + 256 * p, (uint32_t)(key >> (8 * p)) & 0xffu, on);
    } else {
      const uint32_t v = on ? vals[i] : 0;
      for (int s = 0; s < ps.stages; ++s) {
        uint64_t w = on ? __ldg(ps.stage[s].words + v) : 0;
        if (ps.stage[s].order) w = order_key(w);
        for (int p = ps.first[s]; p < ps.first[s + 1]; ++p)
          count_digit(hist + 256 * p, (uint32_t)(w >> (8 * (p - ps.first[s]))) & 0xffu, on);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += kT)
    if (hist[i]) atomicAdd(state + kBases + i, hist[i]);
}

// Digit bases (a warp per pass) and the buffer every pass starts from.
__global__ void __launch_bounds__(1024) k_radix_plan(uint32_t n, int passes, uint32_t* __restrict__ state) {
  __shared__ uint32_t trivial[32];
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  if ((int)warp < passes) {
    uint32_t* h = state + kBases + 256 * warp;
    uint32_t c[8], sum = 0;
    bool all = false;
    for (int q = 0; q < 8; ++q) {
      c[q] = h[8 * lane + q];
      all |= c[q] == n;
      sum += c[q];
    }
    uint32_t incl = sum;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if ((int)lane >= o) incl += y;
    }
    uint32_t run = incl - sum;
    for (int q = 0; q < 8; ++q) {
      h[8 * lane + q] = run;
      run += c[q];
    }
    const bool any = __any_sync(0xffffffffu, all);
    if (lane == 0) trivial[warp] = any;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  uint32_t cur = 0;
  for (int p = 0; p < passes; ++p) {
    state[2 * p] = cur;
    state[2 * p + 1] = trivial[p];
    cur ^= trivial[p] ? 0u : 1u;
  }
  state[2 * passes] = cur;
}

// Ranks of a warp's rows: rank[r] = items of the same digit before it in this warp; cnt[256] ends as the
// warp's digit counts.  digit 256 marks an absent item.
template <int R>
__device__ __forceinline__ void rank_rows(const uint32_t (&dig)[R], uint32_t (&rank)[R], uint32_t* cnt) {
  const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const uint32_t peers = __match_any_sync(0xffffffffu, dig[r]);
    const int leader = __ffs((int)peers) - 1;
    uint32_t base = 0;
    if ((int)lane == leader && dig[r] < 256u) {
      base = cnt[dig[r]];
      cnt[dig[r]] = base + __popc(peers);
    }
    __syncwarp();
    rank[r] = __shfl_sync(0xffffffffu, base, leader) + __popc(peers & lt);
  }
}

// Exclusive scan of one value per thread over the first 256 threads (all threads call).
__device__ __forceinline__ uint32_t scan256(uint32_t v, uint32_t* tmp) {
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if ((int)lane >= o) x += y;
  }
  if (lane == 31 && warp < 8) tmp[warp] = x;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t w = 0; w < 8 && w < warp; ++w) before += tmp[w];
  __syncthreads();
  return before + x - v;
}

// A tile's published count of a digit: 0 not yet, 1 + its own (at most kRadixTile), or kInclusive + that of
// the tiles up to it.  With two flag bits above the count, sorts of 2^30 items and more overflowed; the
// largest record index is below 2^32 - 2^16.
constexpr uint32_t kInclusive = 2u * kRadixTile;
static_assert(1u + kRadixTile < kInclusive && kInclusive + 0xffff0000u > 0xffff0000u, "published counts are told apart");

// One pass.  look: [2][tiles][256] tile counts; the pass uses the half of its input buffer and clears
// the other half for the next one.
template <bool kKv>
__global__ void __launch_bounds__(kT) k_radix_pass(uint32_t n, uint32_t* __restrict__ vals0, uint32_t* __restrict__ vals1,
                                                   uint64_t* __restrict__ keys0, uint64_t* __restrict__ keys1, Passes ps,
                                                   int pass, uint32_t* __restrict__ state, uint32_t* look, uint32_t tiles,
                                                   uint32_t wait) {
  if (state[2 * pass + 1]) return;  // every key has the same digit: order unchanged
  __shared__ uint32_t cnt[kWarps][256];
  __shared__ uint32_t start[256], gbase[256], tmp[8], s_tile;
  __shared__ uint32_t sval[kRadixTile];
  __shared__ uint64_t skey[kKv ? kRadixTile : 1];
  __shared__ uint8_t sdig[kKv ? 1 : kRadixTile];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  const bool flip = state[2 * pass] != 0;
  const uint32_t* in = flip ? vals1 : vals0;
  uint32_t* out = flip ? vals0 : vals1;
  const uint64_t* kin = flip ? keys1 : keys0;
  uint64_t* kout = flip ? keys0 : keys1;
  if (tid == 0) s_tile = atomicAdd(state + kTickets + pass, 1u);
  for (int w = 0; w < kWarps; ++w) cnt[w][tid] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  uint32_t* mine = look + ((uint64_t)(flip ? tiles : 0) + tile) * 256 + tid;
  look[((uint64_t)(flip ? 0 : tiles) + tile) * 256 + tid] = 0;
  uint32_t v[kRows], dig[kRows], rank[kRows];
  uint64_t key[kKv ? kRows : 1];
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t i = tile * kRadixTile + warp * (kRows * 32) + r * 32 + lane;
    v[r] = i < n ? in[i] : 0u;
    if (kKv) {
      key[r] = i < n ? kin[i] : 0u;
      dig[r] = i < n ? (uint32_t)(key[r] >> (8 * pass)) & 0xffu : 256u;
    } else {
      dig[r] = i < n ? indirect_digit(ps, pass, v[r]) : 256u;
    }
  }
  rank_rows<kRows>(dig, rank, cnt[warp]);
  __syncthreads();
  uint32_t total = 0;  // of digit tid
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const uint32_t c = cnt[w][tid];
    cnt[w][tid] = total;
    total += c;
  }
  atomicExch(mine, total + (tile == 0 ? kInclusive : 1u));
  const uint32_t local = scan256(total, tmp);
  start[tid] = local;
  uint32_t before = 0;
  bool late = false;
  for (uint32_t t = tile, spin = 0; t > 0;) {
    const uint32_t x = *(volatile const uint32_t*)(look + ((uint64_t)(flip ? tiles : 0) + t - 1) * 256 + tid);
    if (x == 0) {
      if (spin++ < wait) continue;
      late = true;
      break;
    }
    if (x >= kInclusive) {
      before += x - kInclusive;
      break;
    }
    before += x - 1u;
    --t;
  }
  if (tile && !late) atomicExch(mine, before + total + kInclusive);
  gbase[tid] = state[kBases + 256 * pass + tid] + before - local;
  if (__syncthreads_or(late)) {  // the pass does not change its input: count the tiles before this one
    sval[tid] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < tile * kRadixTile; i += kT)
      atomicAdd(sval + (kKv ? (uint32_t)(kin[i] >> (8 * pass)) & 0xffu : indirect_digit(ps, pass, in[i])), 1u);
    __syncthreads();
    if (late) {
      atomicExch(mine, sval[tid] + total + kInclusive);
      gbase[tid] += sval[tid] - before;
    }
    __syncthreads();
  }
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    if (dig[r] > 255u) continue;
    const uint32_t at = start[dig[r]] + cnt[warp][dig[r]] + rank[r];
    sval[at] = v[r];
    if (kKv) skey[at] = key[r];
    else sdig[at] = (uint8_t)dig[r];
  }
  __syncthreads();
  const uint32_t items = min((uint32_t)kRadixTile, n - tile * kRadixTile);
  for (uint32_t j = tid; j < items; j += kT) {
    const uint32_t d = kKv ? (uint32_t)(skey[j] >> (8 * pass)) & 0xffu : sdig[j];
    const uint32_t to = gbase[d] + j;
    out[to] = sval[j];
    if (kKv) kout[to] = skey[j];
  }
}

// All passes of a sort of at most kSmall items; the result is in the first buffer.
template <bool kKv>
__global__ void __launch_bounds__(kSmallT) k_radix_small(uint32_t n, uint32_t* __restrict__ vals, uint64_t* __restrict__ keys,
                                                         Passes ps, int passes, uint32_t* __restrict__ state) {
  __shared__ uint32_t cnt[kSmallWarps][256];
  __shared__ uint32_t start[256], tmp[8], s_one;
  __shared__ uint32_t sval[kSmall];
  __shared__ uint64_t skey[kKv ? kSmall : 1];
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t v[kSmallRows], dig[kSmallRows], rank[kSmallRows];
  uint64_t key[kKv ? kSmallRows : 1];
  const uint32_t i0 = warp * (kSmallRows * 32) + lane;
#pragma unroll
  for (int r = 0; r < kSmallRows; ++r) {
    const uint32_t i = i0 + r * 32;
    v[r] = i < n ? vals[i] : 0u;
    if (kKv) key[r] = i < n ? keys[i] : 0u;
  }
  for (int p = 0; p < passes; ++p) {
    for (uint32_t q = tid; q < kSmallWarps * 256u; q += kSmallT) (&cnt[0][0])[q] = 0;
    if (tid == 0) s_one = 0;
#pragma unroll
    for (int r = 0; r < kSmallRows; ++r)
      dig[r] = i0 + r * 32 >= n ? 256u : kKv ? (uint32_t)(key[r] >> (8 * p)) & 0xffu : indirect_digit(ps, p, v[r]);
    __syncthreads();
    rank_rows<kSmallRows>(dig, rank, cnt[warp]);
    __syncthreads();
    uint32_t total = 0;
    if (tid < 256) {
      for (int w = 0; w < kSmallWarps; ++w) {
        const uint32_t c = cnt[w][tid];
        cnt[w][tid] = total;
        total += c;
      }
      if (total == n) s_one = 1;
    }
    const uint32_t local = scan256(total, tmp);
    if (tid < 256) start[tid] = local;
    __syncthreads();
    if (s_one) {  // one digit: order unchanged
      __syncthreads();
      continue;
    }
#pragma unroll
    for (int r = 0; r < kSmallRows; ++r) {
      if (dig[r] > 255u) continue;
      const uint32_t at = start[dig[r]] + cnt[warp][dig[r]] + rank[r];
      sval[at] = v[r];
      if (kKv) skey[at] = key[r];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kSmallRows; ++r) {
      const uint32_t i = i0 + r * 32;
      if (i >= n) continue;
      v[r] = sval[i];
      if (kKv) key[r] = skey[i];
    }
  }
#pragma unroll
  for (int r = 0; r < kSmallRows; ++r) {
    const uint32_t i = i0 + r * 32;
    if (i >= n) continue;
    vals[i] = v[r];
    if (kKv) keys[i] = key[r];
  }
  if (tid == 0) state[2 * passes] = 0;
}

template <bool kKv>
int sort(cudaStream_t st, uint32_t n, uint32_t* vals0, uint32_t* vals1, uint64_t* keys0, uint64_t* keys1, const Passes& ps,
         int passes, RadixScratch& scratch, uint64_t* launches) {
  if (n <= kSmall) {
    k_radix_small<kKv><<<1, kSmallT, 0, st>>>(n, vals0, keys0, ps, passes, scratch.state);
    ++*launches;
    return passes;
  }
  const uint32_t tiles = (n + kRadixTile - 1) / kRadixTile;
  cudaMemsetAsync(scratch.state, 0, kRadixStateWords * sizeof(uint32_t), st);
  cudaMemsetAsync(scratch.counts, 0, (uint64_t)tiles * 256 * sizeof(uint32_t), st);
  const uint32_t blocks = (n + 8 * kT - 1) / (8 * kT);
  k_radix_counts<kKv><<<blocks < 1184 ? blocks : 1184, kT, passes * 256 * sizeof(uint32_t), st>>>(n, vals0, keys0, ps, passes,
                                                                                                  scratch.state);
  k_radix_plan<<<1, 1024, 0, st>>>(n, passes, scratch.state);
  for (int p = 0; p < passes; ++p)
    k_radix_pass<kKv><<<tiles, kT, 0, st>>>(n, vals0, vals1, keys0, keys1, ps, p, scratch.state, scratch.counts, tiles,
                                            scratch.wait);
  *launches += 2 + passes;
  return passes;
}

}  // namespace

int radix_sort_indirect(cudaStream_t stream, uint32_t n, uint32_t* vals0, uint32_t* vals1,
                        const IndirectKey* stages, const int* stage_bits, int stage_count,
                        RadixScratch& scratch, uint64_t* launches) {
  Passes ps{};
  ps.stages = stage_count;
  int pass = 0;
  for (int s = 0; s < stage_count; ++s) {
    ps.stage[s] = stages[s];
    ps.first[s] = pass;
    pass += (stage_bits[s] + 7) / 8;
  }
  ps.first[stage_count] = pass;
  return sort<false>(stream, n, vals0, vals1, nullptr, nullptr, ps, pass, scratch, launches);
}

// Stable LSD sort of (keys0[i], vals0[i]) pairs by the low `bits` bits of the keys; the
// result is in the buffer that radix_result(state, passes, vals0, vals1) selects (the keys
// end beside it, in keys0 or keys1 under the same selection).
int radix_sort_kv(cudaStream_t stream, uint32_t n, uint32_t* vals0, uint32_t* vals1, uint64_t* keys0,
                  uint64_t* keys1, int bits, RadixScratch& scratch, uint64_t* launches) {
  return sort<true>(stream, n, vals0, vals1, keys0, keys1, Passes{}, (bits + 7) / 8, scratch, launches);
}

}  // namespace ehgp
