// C ABI entry points (include/ehgp.h): context lifetime, argument checks,
// device error word -> status code, poisoning, timing.
#include "ehgp_internal.cuh"

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <new>
#include <thread>
#if defined(__x86_64__)
#include <immintrin.h>
#endif
#include <sys/mman.h>

using ehgp::Ctx;

namespace ehgp {

constexpr uint64_t kStageBytes = uint64_t{512} << 10;
constexpr uint64_t kHuge = uint64_t{2} << 20;
// Pageable bytes of one copy from which the pinned ring and its threads are used, and from which a context
// without the ring makes it: the ring saves about 0.02 ms per MB and takes 1.4 ms to make.
constexpr uint64_t kStageFrom = uint64_t{32} << 20, kStageMake = uint64_t{64} << 20;

namespace {

// Streaming copy into memory that is not read back here (the caches keep the staging ring).
void stream_copy(char* dst, const char* src, uint64_t bytes) {
#if defined(__x86_64__)
  const uint64_t lead = std::min<uint64_t>(bytes, (16 - (reinterpret_cast<uintptr_t>(dst) & 15)) & 15);
  std::memcpy(dst, src, lead);
  dst += lead;
  src += lead;
  bytes -= lead;
  uint64_t i = 0;
  for (; i + 64 <= bytes; i += 64)
    for (int q = 0; q < 4; ++q)
      _mm_stream_si128(reinterpret_cast<__m128i*>(dst + i) + q, _mm_loadu_si128(reinterpret_cast<const __m128i*>(src + i) + q));
  std::memcpy(dst + i, src + i, bytes - i);
  _mm_sfence();
#else
  std::memcpy(dst, src, bytes);
#endif
}

// The pinned ring of a context, made by its first large copy: huge pages that are registered take 1.4 ms
// for these 8 MB, cudaMallocHost 7.0 ms.  False (and no ring) when the memory cannot be had.
bool stage_ready(Ctx& ctx) {
  if (ctx.stage) return true;
  constexpr uint64_t bytes = kStageSlots * kStageBytes;
  for (cudaEvent_t& ev : ctx.stage_ev)
    if (!ev && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess) {
      ev = nullptr;
      cudaGetLastError();
      return false;
    }
  void* map = mmap(nullptr, bytes + kHuge, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
  if (map == MAP_FAILED) return false;
  char* at = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(map) + kHuge - 1) & ~(uintptr_t)(kHuge - 1));
  madvise(at, bytes, MADV_HUGEPAGE);
  std::memset(at, 0, bytes);
  if (cudaHostRegister(at, bytes, cudaHostRegisterPortable) != cudaSuccess) {
    cudaGetLastError();
    munmap(map, bytes + kHuge);
    return false;
  }
  ctx.stage = at;
  ctx.stage_map = map;
  return true;
}

void stage_free(Ctx& ctx) {
  if (ctx.stage) {
    cudaHostUnregister(ctx.stage);
    munmap(ctx.stage_map, kStageSlots * kStageBytes + kHuge);
    ctx.stage = nullptr;
  }
  for (cudaEvent_t ev : ctx.stage_ev)
    if (ev) cudaEventDestroy(ev);
}

cudaError_t copy_direct(Ctx& ctx, const std::vector<CopyOut>& list) {
  for (const CopyOut& c : list) {
    const cudaError_t e = cudaMemcpyAsync(c.dst, c.src, c.bytes, c.kind, ctx.stream);
    if (e != cudaSuccess) return e;
  }
  return cudaStreamSynchronize(ctx.stream);
}

}  // namespace

// Copies device ranges to host memory.  Pinned destinations and small ranges go straight there;
// large pageable ones go through a ring of pinned slots that host threads empty while the next
// chunks cross the bus (a pageable cudaMemcpy stages through one thread instead).
cudaError_t copy_out(Ctx& ctx, const std::vector<CopyOut>& list) try {
  cudaStream_t st = ctx.stream;
  cudaError_t e = cudaSuccess;
  std::vector<CopyOut> chunks;
  uint64_t all = 0;
  for (const CopyOut& c : list) all += c.bytes;
  for (const CopyOut& c : list) {
    cudaPointerAttributes at{};
    const bool pageable = cudaPointerGetAttributes(&at, c.dst) == cudaSuccess && at.type == cudaMemoryTypeUnregistered;
    cudaGetLastError();
    if (!pageable || c.bytes <= kStageBytes || all < (ctx.stage ? kStageFrom : kStageMake)) {
      if ((e = cudaMemcpyAsync(c.dst, c.src, c.bytes, c.kind, st)) != cudaSuccess) return e;
      continue;
    }
    for (uint64_t o = 0; o < c.bytes; o += kStageBytes)
      chunks.push_back({c.dst + o, c.src + o, std::min(kStageBytes, c.bytes - o), c.kind});
  }
  if (chunks.empty()) return cudaStreamSynchronize(st);
  if (!stage_ready(ctx)) return copy_direct(ctx, chunks);
  const size_t total = chunks.size();
  std::atomic<size_t> issued{0}, next{0};
  std::atomic<int> failed{0};
  std::vector<std::atomic<uint8_t>> done(total);
  for (auto& d : done) d.store(0, std::memory_order_relaxed);
  auto drain = [&] {
    for (size_t t; (t = next.fetch_add(1)) < total;) {
      while (issued.load(std::memory_order_acquire) <= t && !failed.load(std::memory_order_acquire)) std::this_thread::yield();
      if (failed.load(std::memory_order_acquire)) return;
      const int slot = (int)(t % kStageSlots);
      if (cudaEventSynchronize(ctx.stage_ev[slot]) != cudaSuccess) {
        failed.store(1, std::memory_order_release);
        return;
      }
      stream_copy(chunks[t].dst, ctx.stage + slot * kStageBytes, chunks[t].bytes);
      done[t].store(1, std::memory_order_release);
    }
  };
  const unsigned hw = std::max(2u, std::thread::hardware_concurrency());
  const size_t workers = std::min<size_t>({total, (size_t)8, (size_t)(hw - 1)});
  std::vector<std::thread> pool;
  try {
    for (size_t i = 0; i < workers; ++i) pool.emplace_back([&] {
      cudaSetDevice(ctx.device);
      drain();
    });
  } catch (...) {  // no more threads: the ones that started do the work
  }
  if (pool.empty()) return copy_direct(ctx, chunks);
  for (size_t t = 0; t < total && !failed.load(std::memory_order_acquire); ++t) {
    if (t >= (size_t)kStageSlots)
      while (!done[t - kStageSlots].load(std::memory_order_acquire) && !failed.load(std::memory_order_acquire))
        std::this_thread::yield();
    const int slot = (int)(t % kStageSlots);
    e = cudaMemcpyAsync(ctx.stage + slot * kStageBytes, chunks[t].src, chunks[t].bytes, chunks[t].kind, st);
    if (e == cudaSuccess) e = cudaEventRecord(ctx.stage_ev[slot], st);
    if (e != cudaSuccess) {
      failed.store(1, std::memory_order_release);
      break;
    }
    issued.store(t + 1, std::memory_order_release);
  }
  for (auto& th : pool) th.join();
  const cudaError_t es = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  return es != cudaSuccess ? es : failed.load() ? cudaErrorUnknown : cudaSuccess;
} catch (const std::bad_alloc&) {  // (thrown before the first thread starts)
  return copy_direct(ctx, list);
}

cudaError_t ctx_alloc(Ctx& ctx, void** ptr, size_t bytes) {
  if (bytes == 0) bytes = 16;
  ctx.allocations.reserve(ctx.allocations.size() + 1);  // (what is thrown is thrown before there is memory to lose)
  cudaError_t e = cudaMalloc(ptr, bytes);
  if (e == cudaErrorMemoryAllocation && ctx.hier_bytes) {  // the last hierarchy gives way to this call's buffers
    cudaGetLastError();
    hier_trim(ctx);
    e = cudaMalloc(ptr, bytes);
  }
  if (e == cudaSuccess) {
    ctx.allocations.push_back(*ptr);
    ctx.device_bytes += bytes;
  }
  return e;
}

void ctx_free(Ctx& ctx, void* ptr, size_t bytes) {
  if (!ptr) return;
  for (size_t i = 0; i < ctx.allocations.size(); ++i)
    if (ctx.allocations[i] == ptr) {
      ctx.allocations[i] = ctx.allocations.back();
      ctx.allocations.pop_back();
      cudaFree(ptr);
      ctx.device_bytes -= bytes ? bytes : 16;
      return;
    }
}

}  // namespace ehgp

namespace {

int fail(Ctx* ctx, int status, const char* msg);
int cuda_fail(Ctx* ctx, cudaError_t e, const char* where);
int device_status(Ctx* ctx, uint32_t err);

}  // namespace

namespace ehgp {
int abi_fail(Ctx* ctx, int status, const char* msg) { return fail(ctx, status, msg); }
int abi_cuda_fail(Ctx* ctx, cudaError_t e, const char* where) { return cuda_fail(ctx, e, where); }
int abi_device_status(Ctx* ctx, uint32_t err) { return device_status(ctx, err); }
int abi_no_memory(Ctx* ctx) noexcept {
  try {
    return fail(ctx, EHGP_ERR_OUT_OF_MEMORY, "host memory is exhausted");
  } catch (...) {
    return EHGP_ERR_OUT_OF_MEMORY;
  }
}
}  // namespace ehgp

namespace {

int fail(Ctx* ctx, int status, const char* msg) {
  if (ctx) ctx->last_error = msg;
  return status;
}

int cuda_fail(Ctx* ctx, cudaError_t e, const char* where) {
  if (ctx) {
    ctx->poisoned = true;
    ctx->last_error = std::string(where) + ": " + cudaGetErrorString(e);
  }
  return EHGP_ERR_CUDA;
}

// Maps the device error word to a status code (most specific first).
int device_status(Ctx* ctx, uint32_t err) {
  if (err == 0) return EHGP_OK;
  if (err & ehgp::kErrNonFinite) return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "binary64 coordinates must be finite");
  if (err & ehgp::kErrDuplicate)
    return fail(ctx, EHGP_ERR_DUPLICATE_POINT, "a canonical point cloud cannot contain duplicate geometric points");
  if (err & ehgp::kErrNumericRange)
    return fail(ctx, EHGP_ERR_NUMERIC_RANGE, "an exact evaluation left the supported binary64 range");
  if (err & ehgp::kErrTimeout) return fail(ctx, EHGP_ERR_TIMEOUT, "a bounded device wait ran out");
  if (err & ehgp::kErrCapacity) return fail(ctx, EHGP_ERR_CAPACITY, "a device buffer capacity was exceeded");
  return fail(ctx, EHGP_ERR_CUDA, "internal consistency check failed on the device");
}

// Shared body of the three LBVH build entry points.  `src` is a host or
// device pointer according to `where` (0 host f64, 1 host f32, 2 device f64).
int lbvh_build_common(Ctx* ctx, const void* src, uint64_t n, const ehgp_lbvh_out* out, int where) try {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  ctx->last_error.clear();
  if (ctx->poisoned) return fail(ctx, EHGP_ERR_POISONED, "the context is poisoned by an earlier CUDA failure");
  if (!src || !out) return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "null input or output descriptor");
  if (n == 0) return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "a canonical point cloud cannot be empty");
  if (n > ctx->max_points) return fail(ctx, EHGP_ERR_CAPACITY, "the point count exceeds the context capacity");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaSetDevice");
  ehgp::LbvhBuffers& b = ctx->lb;
  const uint32_t n32 = (uint32_t)n;
  ctx->built_n = 0;
  ctx->geom_ready = false;
  ctx->emst_ready = false;
  ctx->pb.witness_ready = false;
  ctx->pb.resident = false;
  ctx->pb.K = 0;  // supports are resident for one cloud and one K
  ctx->hb.K = 0;
  if (where == 0) {
    e = cudaMemcpyAsync(b.xyz_in, src, 3 * n * sizeof(double), cudaMemcpyHostToDevice, ctx->stream);
  } else if (where == 1) {
    e = cudaMemcpyAsync(b.xyz_in_f32, src, 3 * n * sizeof(float), cudaMemcpyHostToDevice, ctx->stream);
  } else {
    e = cudaMemcpyAsync(b.xyz_in, src, 3 * n * sizeof(double), cudaMemcpyDeviceToDevice, ctx->stream);
  }
  if (e != cudaSuccess) return cuda_fail(ctx, e, "input copy");
  if ((e = cudaMemsetAsync(ctx->d_err, 0, sizeof(uint32_t), ctx->stream)) != cudaSuccess)
    return cuda_fail(ctx, e, "cudaMemsetAsync");
  cudaEventRecord(ctx->ev0, ctx->stream);
  ctx->last_launches = ehgp::lbvh_enqueue(*ctx, n32, where == 1 ? 1 : 0);
  cudaEventRecord(ctx->ev1, ctx->stream);
  if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "LBVH kernel launch");
  cudaMemcpyAsync(ctx->h_status, ctx->d_err, sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream);
  cudaMemcpyAsync(ctx->h_status + 1, b.stats, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream);
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return cuda_fail(ctx, e, "LBVH build");
  float ms = 0.f;
  cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
  ctx->last_ms = ms;
  const int st = device_status(ctx, ctx->h_status[0]);
  if (st != EHGP_OK) return st;
  if ((e = ehgp::lbvh_export(*ctx, n32, out)) != cudaSuccess) return cuda_fail(ctx, e, "LBVH export");
  ctx->built_n = n;
  return EHGP_OK;
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

}  // namespace

extern "C" {

int ehgp_ctx_create(int device, const ehgp_limits* limits, ehgp_ctx** out_ctx) {
  if (!limits || !out_ctx || limits->max_points == 0 || limits->max_points > 0x7fffffffull)
    return EHGP_ERR_INVALID_ARGUMENT;
  *out_ctx = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) return EHGP_ERR_INVALID_ARGUMENT;
  ehgp_ctx* ctx = new (std::nothrow) ehgp_ctx();
  if (!ctx) return EHGP_ERR_OUT_OF_MEMORY;
  ctx->device = device;
  ctx->max_points = limits->max_points;
  cudaError_t e = cudaSetDevice(device);
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev1);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->evk0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->evk1);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->evs0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->evs1);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&ctx->h_status, 64 * sizeof(uint32_t));
  if (e == cudaSuccess) e = ehgp::ctx_alloc(*ctx, (void**)&ctx->d_err, sizeof(uint32_t));
  if (e == cudaSuccess) {
    // admission: the context's resident buffers must fit the HBM fraction
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const double frac = (limits->hbm_fraction > 0.0 && limits->hbm_fraction <= 1.0) ? limits->hbm_fraction : 0.8;
    const double estimate = 900.0 * (double)limits->max_points;  // bytes per point of the resident stages
    if (estimate > frac * (double)total_b || estimate > (double)free_b) e = cudaErrorMemoryAllocation;
  }
  if (e == cudaSuccess) e = ehgp::lbvh_alloc(*ctx);
  if (e == cudaSuccess) e = ehgp::geom_alloc(*ctx);
  if (e == cudaSuccess) e = ehgp::pairs_alloc(*ctx);
  if (e == cudaSuccess) e = ehgp::higher_alloc(*ctx);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    const int st = (e == cudaErrorMemoryAllocation) ? EHGP_ERR_OUT_OF_MEMORY : EHGP_ERR_CUDA;
    cudaGetLastError();
    ehgp_ctx_destroy(ctx);
    return st;
  }
  *out_ctx = ctx;
  return EHGP_OK;
}

int ehgp_ctx_destroy(ehgp_ctx* ctx) {
  if (!ctx) return EHGP_OK;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  ehgp::hier_free(*ctx);
  ehgp::stage_free(*ctx);
  for (void* p : ctx->allocations) cudaFree(p);
  if (ctx->h_status) cudaFreeHost(ctx->h_status);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  for (cudaEvent_t ev : {ctx->evk0, ctx->evk1, ctx->evs0, ctx->evs1})
    if (ev) cudaEventDestroy(ev);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
  return EHGP_OK;
}

const char* ehgp_last_error(const ehgp_ctx* ctx) { return ctx ? ctx->last_error.c_str() : ""; }

const char* ehgp_status_string(int status) {
  switch (status) {
    case EHGP_OK: return "EHGP_OK";
    case EHGP_ERR_INVALID_ARGUMENT: return "EHGP_ERR_INVALID_ARGUMENT";
    case EHGP_ERR_DUPLICATE_POINT: return "EHGP_ERR_DUPLICATE_POINT";
    case EHGP_ERR_CAPACITY: return "EHGP_ERR_CAPACITY";
    case EHGP_ERR_OUT_OF_MEMORY: return "EHGP_ERR_OUT_OF_MEMORY";
    case EHGP_ERR_TIMEOUT: return "EHGP_ERR_TIMEOUT";
    case EHGP_ERR_DEGENERATE: return "EHGP_ERR_DEGENERATE";
    case EHGP_ERR_NUMERIC_RANGE: return "EHGP_ERR_NUMERIC_RANGE";
    case EHGP_ERR_CUDA: return "EHGP_ERR_CUDA";
    case EHGP_ERR_POISONED: return "EHGP_ERR_POISONED";
    case EHGP_ERR_NOT_BUILT: return "EHGP_ERR_NOT_BUILT";
    default: return "EHGP_ERR_UNKNOWN";
  }
}

uint64_t ehgp_ctx_device_bytes(const ehgp_ctx* ctx) { return ctx ? ctx->device_bytes + ctx->hier_bytes : 0; }

int ehgp_ctx_reserve(ehgp_ctx* ctx, uint32_t stage, uint64_t records) {
  if (!ctx || stage > 1 || records == 0 || records >= 0xffff0000ull) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  ctx->last_error.clear();
  if (ctx->poisoned) return fail(ctx, EHGP_ERR_POISONED, "the context is poisoned by an earlier CUDA failure");
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "cudaSetDevice");
  if ((e = cudaStreamSynchronize(ctx->stream)) != cudaSuccess) return cuda_fail(ctx, e, "cudaStreamSynchronize");
  // the resident records (if any) are dropped with the buffers
  if (stage == 0) {
    ctx->pb.K = 0;
    ctx->pb.count = 0;
    ctx->pb.witness_ready = false;
    ctx->pb.resident = false;
    e = ehgp::pairs_records_alloc(*ctx, records);
  } else {
    ctx->hb.K = 0;
    ctx->hb.count = 0;
    e = ehgp::higher_records_alloc(*ctx, records);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(ctx, EHGP_ERR_OUT_OF_MEMORY, "the reserved record buffers do not fit the device");
  }
  return EHGP_OK;
}

uint64_t ehgp_ctx_regrowths(const ehgp_ctx* ctx) { return ctx ? ctx->regrowths : 0; }

int ehgp_ctx_counters(const ehgp_ctx* ctx, uint64_t* out, uint32_t count) {
  if (!ctx || !out) return EHGP_ERR_INVALID_ARGUMENT;
  const uint64_t v[5] = {ehgp_ctx_device_bytes(ctx), ctx->regrowths, ctx->pair_runs, ctx->higher_runs, ctx->forest_rest};
  for (uint32_t i = 0; i < count && i < 5; ++i) out[i] = v[i];
  return EHGP_OK;
}

int ehgp_tune(ehgp_ctx* ctx, uint32_t knob, uint64_t value) {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mutex);
  switch (knob) {
    case EHGP_TUNE_HIGHER_LIST:
      if (value < 1 || value > 1024) return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "list capacity must be in [1, 1024]");
      ctx->hb.list_cap = (uint32_t)value;
      return EHGP_OK;
    case EHGP_TUNE_PAIR_TASKS:
      if (value > ctx->pb.task_cap) return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "handed-over walks are at most 2 * max_points + 4096");
      ctx->pb.task_limit = (uint32_t)value;
      return EHGP_OK;
    case EHGP_TUNE_SORT_WAIT:
      if (value > ehgp::kRadixWait) return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "a sort looks at most 2^20 times");
      ctx->radix.wait = (uint32_t)value;
      return EHGP_OK;
    case EHGP_TUNE_HIERARCHY_BLOCK:
      ctx->hier_largest = value ? value : ~uint64_t{0};
      return EHGP_OK;
    case EHGP_TUNE_FOREST_ROUNDS:
      ctx->forest_rounds = (uint32_t)std::min<uint64_t>(value, 0xffffffffu);
      return EHGP_OK;
    default:
      return fail(ctx, EHGP_ERR_INVALID_ARGUMENT, "unknown tuning knob");
  }
}

int ehgp_lbvh_build(ehgp_ctx* ctx, const double* xyz, uint64_t n, const ehgp_lbvh_out* out) {
  return lbvh_build_common(ctx, xyz, n, out, 0);
}
int ehgp_lbvh_build_f32(ehgp_ctx* ctx, const float* xyz, uint64_t n, const ehgp_lbvh_out* out) {
  return lbvh_build_common(ctx, xyz, n, out, 1);
}
int ehgp_lbvh_build_device(ehgp_ctx* ctx, const double* d_xyz, uint64_t n, const ehgp_lbvh_out* out) {
  return lbvh_build_common(ctx, d_xyz, n, out, 2);
}

int ehgp_step_begin(ehgp_ctx* ctx) {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  return cudaEventRecord(ctx->evs0, ctx->stream) == cudaSuccess ? EHGP_OK : EHGP_ERR_CUDA;
}

int ehgp_step_end(ehgp_ctx* ctx, double* elapsed_ms) {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  cudaSetDevice(ctx->device);
  if (cudaEventRecord(ctx->evs1, ctx->stream) != cudaSuccess || cudaEventSynchronize(ctx->evs1) != cudaSuccess)
    return EHGP_ERR_CUDA;
  float ms = 0.f;
  if (cudaEventElapsedTime(&ms, ctx->evs0, ctx->evs1) != cudaSuccess) return EHGP_ERR_CUDA;
  if (elapsed_ms) *elapsed_ms = ms;
  return EHGP_OK;
}

int ehgp_kernel_stats(const ehgp_ctx* ctx, double* kernel_ms, uint64_t* stats, uint32_t count) {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  if (kernel_ms) *kernel_ms = ctx->kernel_ms;
  for (uint32_t i = 0; stats && i < count && i < 8; ++i) stats[i] = ctx->kernel_stats[i];
  return EHGP_OK;
}

int ehgp_last_timing(const ehgp_ctx* ctx, double* device_ms, uint64_t* kernel_launches) {
  if (!ctx) return EHGP_ERR_INVALID_ARGUMENT;
  if (device_ms) *device_ms = ctx->last_ms;
  if (kernel_launches) *kernel_launches = ctx->last_launches;
  return EHGP_OK;
}

}  // extern "C"
