// Serving engine: many point clouds of uneven sizes on one GPU, continuous batching.
//
// The reference plans this as its Python front end's `fit` and a request loop
// (morsehgp3d/docs/GPU_G4_ARCHITECTURE.md:117-136 memory plan at 80 % of the device,
// :269-294 API); it has no batching or serving code.  Here:
//  * a server owns W workers; each worker owns one context (its own CUDA stream and
//    device buffers) and one host thread, and runs one request at a time through the
//    whole chain: canonical cloud + LBVH, Boruvka EMST, pair and triple/quad supports,
//    direct hierarchy of orders 1..K with vertical maps;
//  * submit copies the request's points and queues it; a worker takes the oldest queued
//    request as soon as it is idle and the request fits the memory budget, so requests
//    that arrive while others run are admitted as workers and memory free up, and their
//    device work and copies overlap with the others' (continuous batching);
//  * admission by memory: every running request reserves an estimate of the device bytes
//    its cloud needs (bytes per point for its K, seeded conservatively and raised to the largest
//    per-point footprint a worker's context has reached); a request is admitted when the
//    reservations stay within hbm_fraction of the device's memory, with what idle workers keep from
//    their last request; where that is in the way, they give it back first;
//  * a request's LBVH, supports and event state stay on the device while it runs; when it
//    completes, its result (forest nodes with the supports of their levels, child arena,
//    forest batches, final roots, vertical maps, EMST edges) is copied to host memory the
//    request owns, and the worker moves on.
// Results are those of running the same cloud alone: each request runs on a context of its
// own with no state shared with the others.
#include "ehgp_internal.cuh"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <memory>
#include <thread>
#include <unordered_map>

#include <sys/mman.h>

namespace {

using Clock = std::chrono::steady_clock;

// Result array of plain records, not initialised: its pages are first touched by the threads that fill
// it (a vector's zeroing touched them all in one thread before).  Large arrays are mapped with huge
// pages advised, so that touching them is a fault per 2 MB.
template <class T>
class ResultArray {
 public:
  ResultArray() = default;
  ResultArray(const ResultArray&) = delete;
  ResultArray& operator=(const ResultArray&) = delete;
  ~ResultArray() { drop(); }
  bool resize(uint64_t n) {
    drop();
    const size_t bytes = n * sizeof(T);
    if (bytes == 0) return true;
    if (bytes >= kMapped) {
      void* p = mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
      if (p == MAP_FAILED) return false;
      madvise(p, bytes, MADV_HUGEPAGE);
      p_ = static_cast<T*>(p);
    } else {
      p_ = static_cast<T*>(std::malloc(bytes));
      if (!p_) return false;
    }
    n_ = n;
    return true;
  }
  T* data() const { return p_; }
  uint64_t bytes() const { return n_ * sizeof(T); }
  T& operator[](uint64_t i) const { return p_[i]; }

 private:
  static constexpr size_t kMapped = size_t{4} << 20;
  void drop() {
    if (p_ && bytes() >= kMapped) munmap(p_, bytes());
    else std::free(p_);
    p_ = nullptr;
    n_ = 0;
  }
  T* p_ = nullptr;
  uint64_t n_ = 0;
};

struct Request {
  uint64_t id = 0;
  int state = EHGP_REQ_QUEUED;
  int status = EHGP_OK;
  std::string error;
  uint64_t n = 0;
  uint32_t K = 10;
  bool f32 = false;
  std::vector<double> xyz64;
  std::vector<float> xyz32;
  uint64_t reserved = 0;
  uint32_t worker = 0;
  Clock::time_point t_submit, t_start, t_end;
  double device_ms = 0;
  // result
  ehgp_hier_counts counts{};
  ResultArray<ehgp_forest_node> nodes;
  ResultArray<uint32_t> children;
  ResultArray<ehgp_forest_batch> batches;
  ResultArray<ehgp_forest_root> roots;
  ResultArray<ehgp_vertical_assignment> vertical;
  ResultArray<uint32_t> node_support;  // 5 words per node
  ResultArray<uint32_t> emst_u, emst_v;
};

struct Worker {
  ehgp_ctx* ctx = nullptr;
  std::thread thread;
  uint64_t max_n_seen = 0;
  uint64_t kept = 0;   // hierarchy memory of the idle context
  bool trim = false;   // asked to give it back
};

}  // namespace

struct ehgp_server {
  int device = 0;
  ehgp_server_limits limits{};
  uint64_t budget = 0;              // bytes the running requests may reserve
  double bytes_per_point[11] = {};  // admission estimate for each K (raised by measurement)
  double records_per_point = 0;     // of them, the index and support buffers: submit refuses by these
  uint64_t reserved = 0;            // reservations of the running requests
  std::vector<Worker> workers;
  std::deque<uint64_t> queue;
  std::unordered_map<uint64_t, std::shared_ptr<Request>> reqs;  // shared with result copies under way
  std::mutex mu;
  std::condition_variable cv_work, cv_done;
  bool stop = false;
  uint64_t next_id = 1;
  uint64_t admitted = 0, completed = 0, waits_for_memory = 0;
};

namespace {

uint64_t estimate(double per_point, uint64_t n) { return (uint64_t)(per_point * (double)n) + (64ull << 20); }

// True when the memory that the other idle workers keep fits beside the reservations and `need` more;
// else asks as many of them as it takes to give theirs back (the largest first).
bool idle_memory_fits(ehgp_server& s, uint32_t w, uint64_t need) {
  uint64_t all = 0, kept = 0;  // kept: by those that are not asked yet
  for (uint32_t i = 0; i < s.workers.size(); ++i) {
    const Worker& x = s.workers[i];
    if (i == w) continue;
    all += x.kept;
    kept += x.trim ? 0 : x.kept;
  }
  if (all == 0 || s.reserved + need + all <= s.budget) return true;
  while (s.reserved + need + kept > s.budget) {
    Worker* most = nullptr;
    for (uint32_t i = 0; i < s.workers.size(); ++i) {
      Worker& x = s.workers[i];
      if (i != w && x.kept && !x.trim && (!most || x.kept > most->kept)) most = &x;
    }
    if (!most) break;
    most->trim = true;
    kept -= most->kept;
  }
  s.cv_work.notify_all();
  return false;
}


// The whole chain for one request on the worker's context; fills the request's result.
int run_request(ehgp_ctx* ctx, Request& r) try {
  if (ehgp_step_begin(ctx) != EHGP_OK) return EHGP_ERR_CUDA;
  ehgp_lbvh_out none{};
  int st = r.f32 ? ehgp_lbvh_build_f32(ctx, r.xyz32.data(), r.n, &none) : ehgp_lbvh_build(ctx, r.xyz64.data(), r.n, &none);
  if (st != EHGP_OK) return st;
  if (r.n >= 2) {
    if (!r.emst_u.resize(r.n - 1) || !r.emst_v.resize(r.n - 1)) return EHGP_ERR_OUT_OF_MEMORY;
    ehgp_emst_out eo{};
    eo.u = r.emst_u.data();
    eo.v = r.emst_v.data();
    if ((st = ehgp_emst(ctx, &eo)) != EHGP_OK) return st;
  }
  st = ehgp_hierarchy(ctx, r.K, &r.counts);
  double ms = 0;
  ehgp_step_end(ctx, &ms);
  r.device_ms = ms;
  if (st != EHGP_OK) return st;
  const ehgp_hier_counts& c = r.counts;
  if (!r.nodes.resize(c.nodes) || !r.children.resize(c.children) || !r.batches.resize(c.journal_batches) ||
      !r.roots.resize(c.final_roots) || !r.vertical.resize(c.vertical_assignments) || !r.node_support.resize(5 * c.nodes))
    return EHGP_ERR_OUT_OF_MEMORY;
  ehgp_hier_out out{};
  out.nodes = r.nodes.data();
  out.children = r.children.data();
  out.batches = r.batches.data();
  out.roots = r.roots.data();
  out.vertical = r.vertical.data();
  if ((st = ehgp_hier_copy(ctx, &out)) != EHGP_OK) return st;
  std::vector<uint32_t> lev(c.nodes);
  for (uint64_t i = 0; i < c.nodes; ++i) lev[i] = r.nodes[i].level_event;
  return ehgp_event_supports(ctx, lev.data(), c.nodes, r.node_support.data());
} catch (const std::bad_alloc&) {
  return ehgp::abi_no_memory(ctx);
}

void worker_loop(ehgp_server* s, uint32_t w) {
  Worker& me = s->workers[w];
  for (;;) {
    Request* r = nullptr;
    {
      std::unique_lock<std::mutex> lock(s->mu);
      for (;;) {
        if (s->stop) return;
        if (!s->queue.empty()) {
          Request* head = s->reqs.at(s->queue.front()).get();
          const uint64_t est = estimate(s->bytes_per_point[head->K], head->n), need = std::max(est, me.kept);
          if (s->reserved + est > s->budget && s->reserved != 0) {  // FIFO; a lone request always runs
            ++s->waits_for_memory;
          } else if (me.kept > est && s->reserved + need > s->budget) {
            me.trim = true;
          } else if (idle_memory_fits(*s, w, need)) {
            me.kept = 0;  // within the reservation from here on
            me.trim = false;
            s->queue.pop_front();
            head->reserved = need;
            s->reserved += need;
            head->state = EHGP_REQ_RUNNING;
            head->worker = w;
            head->t_start = Clock::now();
            ++s->admitted;
            r = head;
            break;
          }
        }
        if (me.trim) {
          lock.unlock();
          ehgp::hier_trim(*me.ctx);
          lock.lock();
          me.trim = false;
          me.kept = 0;
          s->cv_work.notify_all();
          continue;
        }
        s->cv_work.wait(lock);
      }
    }
    const uint64_t held_before = ehgp_ctx_device_bytes(me.ctx);
    const int st = run_request(me.ctx, *r);
    const uint64_t held = ehgp_ctx_device_bytes(me.ctx), kept = me.ctx->hier_bytes;
    {
      std::lock_guard<std::mutex> lock(s->mu);
      me.max_n_seen = std::max(me.max_n_seen, r->n);
      me.kept = kept;
      if (st == EHGP_OK && r->n >= 1024) {  // the context's footprint per point of the largest cloud it holds
        double& all = s->bytes_per_point[r->K];
        if (held > held_before) all = std::max(all, (double)held / (double)me.max_n_seen);
        s->records_per_point = std::max(s->records_per_point, (double)(held - kept) / (double)me.max_n_seen);
      }
      r->status = st;
      if (st != EHGP_OK) r->error = ehgp_last_error(me.ctx);
      r->state = st == EHGP_OK ? EHGP_REQ_DONE : EHGP_REQ_FAILED;
      r->t_end = Clock::now();
      s->reserved -= r->reserved;
      r->reserved = 0;
      r->xyz64.clear();
      r->xyz64.shrink_to_fit();
      r->xyz32.clear();
      r->xyz32.shrink_to_fit();
      ++s->completed;
    }
    s->cv_done.notify_all();
    s->cv_work.notify_all();
  }
}

Request* find(ehgp_server* s, ehgp_request_id id) {
  auto it = s->reqs.find(id);
  return it == s->reqs.end() ? nullptr : it->second.get();
}

double ms_between(Clock::time_point a, Clock::time_point b) {
  return std::chrono::duration<double, std::milli>(b - a).count();
}

}  // namespace

extern "C" {

int ehgp_server_create(int device, const ehgp_server_limits* limits, ehgp_server** out) {
  if (!limits || !out || limits->workers == 0 || limits->workers > 64 || limits->max_points == 0 ||
      !(limits->hbm_fraction > 0.0 && limits->hbm_fraction <= 1.0))
    return EHGP_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  if (cudaSetDevice(device) != cudaSuccess) return EHGP_ERR_CUDA;
  size_t free_b = 0, total_b = 0;
  if (cudaMemGetInfo(&free_b, &total_b) != cudaSuccess) return EHGP_ERR_CUDA;
  std::unique_ptr<ehgp_server> s(new ehgp_server());
  s->device = device;
  s->limits = *limits;
  s->budget = (uint64_t)(limits->hbm_fraction * (double)total_b);
  s->records_per_point = 120.0 * 1024.0;  // before any measurement
  // 37 KB per point for index, lists and first record buffers, 0.95 KB per support event with the
  // hierarchy's: 502 KB per point at 50,653 lattice points and K = 10 (488 events), 82 KB at K = 4
  for (uint32_t k = 1; k <= 10; ++k)
    s->bytes_per_point[k] = 1024.0 * (40.0 + 1.05 * (7.0 + 483.0 * std::pow(k / 10.0, 2.3)));
  for (uint32_t w = 0; w < limits->workers; ++w) {
    ehgp_limits cl{limits->max_points, limits->hbm_fraction};
    Worker wk;
    const int st = ehgp_ctx_create(device, &cl, &wk.ctx);
    if (st != EHGP_OK) {
      for (auto& x : s->workers) ehgp_ctx_destroy(x.ctx);
      return st;
    }
    s->workers.push_back(std::move(wk));
  }
  for (uint32_t w = 0; w < limits->workers; ++w) s->workers[w].thread = std::thread(worker_loop, s.get(), w);
  *out = s.release();
  return EHGP_OK;
}

int ehgp_server_destroy(ehgp_server* s) {
  if (!s) return EHGP_OK;
  {
    std::lock_guard<std::mutex> lock(s->mu);
    s->stop = true;
  }
  s->cv_work.notify_all();
  for (auto& w : s->workers)
    if (w.thread.joinable()) w.thread.join();
  for (auto& w : s->workers) ehgp_ctx_destroy(w.ctx);
  delete s;
  return EHGP_OK;
}

int ehgp_cloud_submit(ehgp_server* s, const ehgp_cloud_desc* d, ehgp_request_id* id) {
  if (!s || !d || !id || !d->xyz || d->n == 0 || d->K == 0 || d->K > 10 || d->dtype > 1)
    return EHGP_ERR_INVALID_ARGUMENT;
  if (d->n > s->limits.max_points) return EHGP_ERR_CAPACITY;
  std::shared_ptr<Request> r(new Request());
  r->n = d->n;
  r->K = d->K;
  r->f32 = d->dtype == EHGP_DTYPE_F32;
  if (r->f32) r->xyz32.assign((const float*)d->xyz, (const float*)d->xyz + 3 * d->n);
  else r->xyz64.assign((const double*)d->xyz, (const double*)d->xyz + 3 * d->n);
  r->t_submit = Clock::now();
  {
    std::lock_guard<std::mutex> lock(s->mu);
    if (estimate(s->records_per_point, d->n) > s->budget) return EHGP_ERR_OUT_OF_MEMORY;
    r->id = s->next_id++;
    *id = r->id;
    s->queue.push_back(r->id);
    s->reqs.emplace(r->id, std::move(r));
  }
  s->cv_work.notify_one();
  return EHGP_OK;
}

int ehgp_poll(ehgp_server* s, ehgp_request_id id, int32_t* state) {
  if (!s || !state) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  Request* r = find(s, id);
  if (!r) return EHGP_ERR_INVALID_ARGUMENT;
  *state = r->state;
  return EHGP_OK;
}

int ehgp_wait(ehgp_server* s, ehgp_request_id id, uint64_t timeout_ns, int32_t* status) {
  if (!s) return EHGP_ERR_INVALID_ARGUMENT;
  std::unique_lock<std::mutex> lock(s->mu);
  Request* r = find(s, id);
  if (!r) return EHGP_ERR_INVALID_ARGUMENT;
  const auto done = [&] { return r->state == EHGP_REQ_DONE || r->state == EHGP_REQ_FAILED; };
  if (!s->cv_done.wait_for(lock, std::chrono::nanoseconds(timeout_ns), done)) return EHGP_ERR_TIMEOUT;
  if (status) *status = r->status;
  return EHGP_OK;
}

int ehgp_request_info(ehgp_server* s, ehgp_request_id id, ehgp_request_stats* info) {
  if (!s || !info) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  Request* r = find(s, id);
  if (!r) return EHGP_ERR_INVALID_ARGUMENT;
  *info = ehgp_request_stats{};
  info->state = r->state;
  info->status = r->status;
  info->points = r->n;
  info->K = r->K;
  info->worker = r->worker;
  const bool started = r->state != EHGP_REQ_QUEUED, ended = r->state == EHGP_REQ_DONE || r->state == EHGP_REQ_FAILED;
  info->queued_ms = started ? ms_between(r->t_submit, r->t_start) : ms_between(r->t_submit, Clock::now());
  info->service_ms = ended ? ms_between(r->t_start, r->t_end) : 0.0;
  info->latency_ms = ended ? ms_between(r->t_submit, r->t_end) : 0.0;
  info->device_ms = r->device_ms;
  info->counts = r->counts;
  return EHGP_OK;
}

const char* ehgp_request_error(ehgp_server* s, ehgp_request_id id) {
  if (!s) return "";
  std::lock_guard<std::mutex> lock(s->mu);
  Request* r = find(s, id);
  return r ? r->error.c_str() : "";
}

int ehgp_result_copy(ehgp_server* s, ehgp_request_id id, const ehgp_served_out* out) try {
  if (!s || !out) return EHGP_ERR_INVALID_ARGUMENT;
  std::shared_ptr<Request> r;  // a finished request's result does not change: copied outside the lock
  {
    std::lock_guard<std::mutex> lock(s->mu);
    auto it = s->reqs.find(id);
    if (it == s->reqs.end()) return EHGP_ERR_INVALID_ARGUMENT;
    if (it->second->state != EHGP_REQ_DONE) return EHGP_ERR_NOT_BUILT;
    r = it->second;
  }
  struct Piece {
    char* dst;
    const char* src;
    uint64_t bytes;
  };
  constexpr uint64_t kPiece = uint64_t{4} << 20;
  std::vector<Piece> pieces;
  uint64_t total = 0;
  auto put = [&](auto* dst, const auto& v) {
    if (!dst) return;
    total += v.bytes();
    for (uint64_t o = 0; o < v.bytes(); o += kPiece)
      pieces.push_back({reinterpret_cast<char*>(dst) + o, reinterpret_cast<const char*>(v.data()) + o,
                        std::min(kPiece, v.bytes() - o)});
  };
  put(out->nodes, r->nodes);
  put(out->children, r->children);
  put(out->batches, r->batches);
  put(out->roots, r->roots);
  put(out->vertical, r->vertical);
  put(out->node_supports, r->node_support);
  put(out->emst_u, r->emst_u);
  put(out->emst_v, r->emst_v);
  std::atomic<size_t> next{0};
  auto work = [&] {
    for (size_t i; (i = next.fetch_add(1)) < pieces.size();) std::memcpy(pieces[i].dst, pieces[i].src, pieces[i].bytes);
  };
  std::vector<std::thread> pool;
  if (total >= 4 * kPiece) {
    const unsigned hw = std::max(1u, std::thread::hardware_concurrency());
    try {
      for (unsigned i = 1; i < std::min(8u, hw); ++i) pool.emplace_back(work);
    } catch (...) {  // no more threads: this one copies too
    }
  }
  work();
  for (auto& t : pool) t.join();
  return EHGP_OK;
} catch (const std::bad_alloc&) {
  return EHGP_ERR_OUT_OF_MEMORY;
}

int ehgp_result_release(ehgp_server* s, ehgp_request_id id) {
  if (!s) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  auto it = s->reqs.find(id);
  if (it == s->reqs.end()) return EHGP_ERR_INVALID_ARGUMENT;
  if (it->second->state != EHGP_REQ_DONE && it->second->state != EHGP_REQ_FAILED) return EHGP_ERR_NOT_BUILT;
  s->reqs.erase(it);
  return EHGP_OK;
}

int ehgp_server_info(ehgp_server* s, uint64_t* info, uint32_t count) {
  if (!s || !info) return EHGP_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(s->mu);
  uint64_t held = 0, running = 0;
  for (const auto& w : s->workers) held += ehgp_ctx_device_bytes(w.ctx);
  for (const auto& kv : s->reqs) running += kv.second->state == EHGP_REQ_RUNNING;
  const uint64_t v[8] = {s->budget, s->reserved, held, (uint64_t)s->bytes_per_point[10], s->queue.size(), running,
                         s->completed, s->waits_for_memory};
  for (uint32_t i = 0; i < count && i < 8; ++i) info[i] = v[i];
  return EHGP_OK;
}

}  // extern "C"
