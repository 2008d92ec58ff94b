// The gate of call_gate.cuh: the count of threads inside and one bit for the
// thread that is alone, in one atomic.
#include "call_gate.cuh"

#include <atomic>
#include <mutex>
#include <vector>

namespace sl3dgpu {
namespace {

constexpr int kAlone = 1 << 30;
std::atomic<int> inside{0};
thread_local int depth = 0;       // this thread's calls, one within another
thread_local int aloneDepth = 0;  // its sections

std::mutex retiredLock;
std::vector<cudaGraphExec_t> retired;

// The gate keeps calls apart in time; what they share has locks of its own (the
// driver's, a grid's). So a call that ends does not order its stores: on Arm that
// would wait for its launches' writes to the device.
void Enter() {
  for (int now = inside.load(std::memory_order_relaxed);;) {
    if ((now & kAlone) != 0) {
      inside.wait(now);
      now = inside.load();
    } else if (inside.compare_exchange_weak(now, now + 1, std::memory_order_acquire, std::memory_order_relaxed)) {
      return;
    }
  }
}
void Leave() { inside.fetch_sub(1, std::memory_order_relaxed); }

}  // namespace

LibraryCall::LibraryCall() {
  if (depth++ == 0) Enter();
}
LibraryCall::~LibraryCall() {
  if (--depth == 0) Leave();
}

SeveralThreads::SeveralThreads(bool on) : on_(on) {
  if (on_) Enter();
}
SeveralThreads::~SeveralThreads() {
  if (on_) Leave();
}

Alone::Alone() : held_(false) {
  if (depth == 0) return;
  if (aloneDepth == 0) {
    int one = 1;
    if (!inside.compare_exchange_strong(one, 1 | kAlone)) return;
    std::lock_guard<std::mutex> guard(retiredLock);
    for (cudaGraphExec_t exec : retired) cudaGraphExecDestroy(exec);
    retired.clear();
  }
  ++aloneDepth;
  held_ = true;
}
Alone::~Alone() {
  if (!held_ || --aloneDepth > 0) return;
  inside.store(1);
  inside.notify_all();
}

void RetireGraph(cudaGraphExec_t exec) {
  if (exec == nullptr) return;
  if (const Alone alone; alone) {
    cudaGraphExecDestroy(exec);
    return;
  }
  std::lock_guard<std::mutex> guard(retiredLock);
  retired.push_back(exec);
}
int RetiredGraphs() {
  std::lock_guard<std::mutex> guard(retiredLock);
  return static_cast<int>(retired.size());
}

}  // namespace sl3dgpu
