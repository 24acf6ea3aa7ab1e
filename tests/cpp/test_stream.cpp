// WorkStream (spmv_b200/csrc/stream.cpp) on a model of two CUDA streams: the
// runtime calls that it makes are the ones below, which keep each stream's work in
// order and a happens-before clock per item.  Every two items of work that threads
// put on a communicator must be ordered, whichever stream each went to.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>

#include "internal.h"

namespace {

// Stream 0 is the legacy default stream, 1 the library's own.
struct Clock {
  int n[2] = {0, 0};
};
struct Item {
  int stream;
  Clock clock;  // items of each stream that come before it (itself included)
};
std::mutex g_mu;
Clock g_now[2];
std::vector<Item> g_items;

cudaStream_t const OWN = reinterpret_cast<cudaStream_t>(uintptr_t(1));
int index_of(cudaStream_t s) { return s == OWN ? 1 : 0; }

void put_work(cudaStream_t stream) {
  const std::lock_guard<std::mutex> lock(g_mu);
  const int s = index_of(stream);
  ++g_now[s].n[s];
  g_items.push_back({s, g_now[s]});
}

bool before(const Item& a, const Item& b) { return b.clock.n[a.stream] >= a.clock.n[a.stream]; }

int unordered_pairs() {
  int bad = 0;
  for (size_t i = 0; i < g_items.size(); ++i)
    for (size_t j = 0; j < i; ++j)
      if (!before(g_items[i], g_items[j]) && !before(g_items[j], g_items[i])) ++bad;
  return bad;
}

void nap(int ms) { std::this_thread::sleep_for(std::chrono::milliseconds(ms)); }

// A call on device vectors of the default stream, as the Python layer makes it.
void fenced_call(spmvb::WorkStream& w, int ms, std::atomic<int>* got = nullptr) {
  const bool direct = w.begin_direct(0);
  {
    const spmvb::CallScope call;
    cudaStream_t s = w;
    if (got) ++*got;
    nap(ms);
    put_work(s);
  }
  if (direct) w.end_direct();
}
// A call without a fence: on the library's stream.
void plain_call(spmvb::WorkStream& w, int ms, std::atomic<int>* got = nullptr) {
  const spmvb::CallScope call;
  cudaStream_t s = w;
  if (got) ++*got;
  nap(ms);
  put_work(s);
}
void wait_for(const std::atomic<int>& n) {
  while (n.load() == 0) std::this_thread::yield();
}

int check(const char* name) {
  const int bad = unordered_pairs();
  std::printf("%s: %zu items, %d unordered pairs\n", name, g_items.size(), bad);
  g_items.clear();
  g_now[0] = g_now[1] = Clock{};
  return bad != 0;
}

}  // namespace

// The CUDA runtime, as far as stream.cpp uses it.
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) {
  *e = reinterpret_cast<cudaEvent_t>(new Clock);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  delete reinterpret_cast<Clock*>(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  const std::lock_guard<std::mutex> lock(g_mu);
  *reinterpret_cast<Clock*>(e) = g_now[index_of(s)];
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned int) {
  const std::lock_guard<std::mutex> lock(g_mu);
  const Clock& c = *reinterpret_cast<Clock*>(e);
  for (int i = 0; i < 2; ++i) g_now[index_of(s)].n[i] = std::max(g_now[index_of(s)].n[i], c.n[i]);
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return ""; }
}
namespace spmvb {
void soft_check(cudaError_t, const char*) {}
void set_last_error(const std::string&) {}
}  // namespace spmvb

int main() {
  int failed = 0;
  {
    // A plain call while another thread is between its stream and its launch.
    spmvb::WorkStream w;
    w.set(OWN);
    std::atomic<int> got{0};
    std::thread a([&] { fenced_call(w, 100, &got); });
    wait_for(got);
    plain_call(w, 0);
    a.join();
    failed |= check("plain call during a direct fence");
  }
  {
    // And the other way round.
    spmvb::WorkStream w;
    w.set(OWN);
    std::atomic<int> got{0};
    std::thread a([&] { plain_call(w, 100, &got); });
    wait_for(got);
    fenced_call(w, 0);
    fenced_call(w, 0);
    a.join();
    fenced_call(w, 0);
    failed |= check("fenced calls during a plain call");
    if (!w.begin_direct(0)) failed = 1;  // nobody works on own any more
    w.end_direct();
  }
  {
    // The handle given out, from inside a fence as well.
    spmvb::WorkStream w;
    w.set(OWN);
    fenced_call(w, 0);
    w.begin_direct(0);
    put_work(w);
    {
      const spmvb::CallScope call;
      w.hand_out();
      put_work(w.own());
    }
    if (w.end_direct()) failed = 1;
    fenced_call(w, 0);
    failed |= check("handle given out");
    if (w.begin_direct(0)) failed = 1;
  }
  {
    // A call that uses two communicators' streams, one of them dying in it.
    spmvb::WorkStream w;
    w.set(OWN);
    const spmvb::CallScope call;
    {
      spmvb::WorkStream v;
      v.set(OWN);
      (void)cudaStream_t(v);
      (void)cudaStream_t(w);
    }
  }
  {
    spmvb::WorkStream w;
    w.set(OWN);
    std::vector<std::thread> t;
    for (int i = 0; i < 4; ++i)
      t.emplace_back([&w, i] {
        std::minstd_rand rng(unsigned(i + 1));
        for (int k = 0; k < 250; ++k) {
          if (rng() % 2)
            fenced_call(w, 0);
          else
            plain_call(w, 0);
          if (rng() % 8 == 0) std::this_thread::yield();
        }
      });
    for (auto& q : t) q.join();
    failed |= check("four threads");
  }
  return failed;
}
