// The stream of a communicator's work and the fences around it (no counterpart in
// the reference).
#include <algorithm>
#include <chrono>

#include "internal.h"

namespace spmvb {

namespace {

// One event per thread and device, made on first use: it is recorded and the
// other stream made to wait for it at once, so a thread can use its own again
// for the next pair.
struct FenceEvents {
  std::vector<cudaEvent_t> ev;  // per device
  cudaEvent_t get(int device) {
    if (int(ev.size()) <= device) ev.resize(size_t(device) + 1, nullptr);
    if (!ev[size_t(device)])
      SPMVB_CUDA(cudaEventCreateWithFlags(&ev[size_t(device)], cudaEventDisableTiming));
    return ev[size_t(device)];
  }
  ~FenceEvents() {
    for (cudaEvent_t e : ev)
      if (e) soft_check(cudaEventDestroy(e), "cudaEventDestroy");
  }
};
thread_local FenceEvents g_fence;
// The communicator's stream whose direct fence this thread is in.
thread_local const WorkStream* g_direct = nullptr;
// The depth of this thread's library calls and the streams whose own_ they use.
thread_local int g_depth = 0;
thread_local std::vector<const WorkStream*> g_used;
// A direct fence only puts work on a stream; one that is never closed is the
// caller's error, which the call that waits for it reports.
constexpr std::chrono::seconds DIRECT_LIMIT(60);

}  // namespace

void order_streams(int device, cudaStream_t before, cudaStream_t after) {
  cudaEvent_t e = g_fence.get(device);
  SPMVB_CUDA(cudaEventRecord(e, before));
  SPMVB_CUDA(cudaStreamWaitEvent(after, e, 0));
}

CallScope::CallScope() { ++g_depth; }

CallScope::~CallScope() {
  if (--g_depth > 0 || g_used.empty()) return;
  for (const WorkStream* w : g_used) {
    const std::lock_guard<std::mutex> lock(w->mu_);
    --w->calls_;
  }
  g_used.clear();
}

WorkStream::~WorkStream() {
  g_used.erase(std::remove(g_used.begin(), g_used.end(), this), g_used.end());
  if (g_direct == this) g_direct = nullptr;
}

cudaStream_t WorkStream::get() const {
  std::unique_lock<std::mutex> lock(mu_);
  if (g_direct == this) {
    if (own_ahead_) {
      order_streams(device_, own_, nullptr);
      own_ahead_ = false;
    }
    default_ahead_ = true;
    return nullptr;
  }
  if (std::find(g_used.begin(), g_used.end(), this) == g_used.end()) {
    if (!closed_.wait_for(lock, DIRECT_LIMIT, [&] { return direct_ == 0; }))
      fail(SPMV_ERROR_INVALID_ARGUMENT,
           "spmv: another thread's fence (leave = 2) on the communicator was not ended");
    if (g_depth > 0) {
      g_used.push_back(this);
      ++calls_;
    }
  }
  if (default_ahead_) {
    order_streams(device_, nullptr, own_);
    default_ahead_ = false;
  }
  own_ahead_ = true;
  return own_;
}

void WorkStream::hand_out() const {
  (void)end_direct();  // (if this thread is in a fence: what follows is on the handle)
  (void)get();         // and behind the direct work
  const std::lock_guard<std::mutex> lock(mu_);
  given_ = true;
}

bool WorkStream::begin_direct(int device) const {
  const std::lock_guard<std::mutex> lock(mu_);
  if (given_ || g_direct != nullptr || calls_ > 0) return false;
  device_ = device;
  g_direct = this;
  ++direct_;
  return true;
}

bool WorkStream::end_direct() const {
  if (g_direct != this) return false;
  g_direct = nullptr;
  const std::lock_guard<std::mutex> lock(mu_);
  if (--direct_ == 0) closed_.notify_all();
  return true;
}

}  // namespace spmvb
