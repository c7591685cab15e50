// Preloaded into a test's process: host-side failures at the edge of the library, on demand.
//  * hf_watch: counts CUDA calls that need a current device made by this thread before cudaSetDevice;
//  * hf_fail_sync: the next cudaStreamSynchronize of this thread reports a failure (nothing fails);
//  * hf_fail_new: an allocation of this thread throws std::bad_alloc.
#include <dlfcn.h>

#include <atomic>
#include <cstddef>
#include <cstdlib>
#include <new>

namespace {
thread_local bool watching = false, device_set = false, sync_fails = false, new_failed = false;
thread_local long news_left = -1;
std::atomic<int> early{0};

template <class F>
F real(F, const char* name) {
  return reinterpret_cast<F>(dlsym(RTLD_NEXT, name));
}
void note() {
  if (watching && !device_set) ++early;
}
void* allocate(std::size_t n) {
  if (news_left >= 0 && news_left-- == 0) {
    new_failed = true;
    throw std::bad_alloc();
  }
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
}  // namespace

extern "C" {
void hf_watch(int on) {
  watching = on != 0;
  device_set = false;
  early = 0;
}
int hf_early_calls() { return early; }
void hf_fail_sync() { sync_fails = true; }
void hf_fail_new(long after) {
  news_left = after;
  new_failed = false;
}
int hf_new_failed() {
  news_left = -1;
  return new_failed;
}

int cudaSetDevice(int d) {
  device_set = true;
  return real(&cudaSetDevice, "cudaSetDevice")(d);
}
int cudaEventCreateWithFlags(void** e, unsigned flags) {
  note();
  return real(&cudaEventCreateWithFlags, "cudaEventCreateWithFlags")(e, flags);
}
int cudaEventRecord(void* e, void* stream) {
  note();
  return real(&cudaEventRecord, "cudaEventRecord")(e, stream);
}
int cudaMemcpyAsync(void* dst, const void* src, std::size_t n, int kind, void* stream) {
  note();
  return real(&cudaMemcpyAsync, "cudaMemcpyAsync")(dst, src, n, kind, stream);
}
int cudaStreamSynchronize(void* stream) {
  note();
  const int r = real(&cudaStreamSynchronize, "cudaStreamSynchronize")(stream);
  if (!sync_fails) return r;
  sync_fails = false;
  return 719;  // cudaErrorLaunchFailure
}
}

void* operator new(std::size_t n) { return allocate(n); }
void* operator new[](std::size_t n) { return allocate(n); }
void operator delete(void* p) noexcept { std::free(p); }
void operator delete[](void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }
void operator delete[](void* p, std::size_t) noexcept { std::free(p); }
