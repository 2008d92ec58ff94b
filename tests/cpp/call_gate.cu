// The gate that keeps the correction's graphs to a thread that is alone in the
// library (csrc/call_gate.cuh): who may hold it, who waits for it, and what
// becomes of graphs that cannot be destroyed at once. No device is used.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "call_gate.cuh"

using namespace sl3dgpu;

namespace {
bool good = true;
void Check(bool ok, const char* what) {
  std::printf("%s: %s\n", ok ? "ok" : "FAIL", what);
  good = good && ok;
}
// never dereferenced: without a device the runtime refuses it before it looks
cudaGraphExec_t Fake() { return reinterpret_cast<cudaGraphExec_t>(256); }
}  // namespace

int main() {
  int devices = 0;
  if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0) return 2;  // run without a device
  {
    const Alone outside;
    Check(!outside, "no section outside a call");
    const LibraryCall call, nested;
    const Alone first, second;
    Check(first && second, "a thread alone holds the section, and again within it");
  }
  {
    const LibraryCall call;
    const SeveralThreads several(true);
    Check(!Alone(), "a call that drives others is not alone");
  }
  {
    const LibraryCall call;
    std::atomic<bool> otherIn{false}, done{false};
    std::thread other([&] {
      const LibraryCall theirs;
      otherIn = true;
      while (!done) std::this_thread::yield();
    });
    while (!otherIn) std::this_thread::yield();
    Check(!Alone(), "no section beside another thread's call");
    RetireGraph(Fake());
    Check(RetiredGraphs() == 1, "a graph retired beside it waits");
    done = true;
    other.join();
    Check(static_cast<bool>(Alone()) && RetiredGraphs() == 0, "and is destroyed by the next section");
  }
  {
    std::atomic<bool> otherIn{false};
    std::thread other;
    {
      const LibraryCall call;
      const Alone alone;
      other = std::thread([&] {
        const LibraryCall theirs;
        otherIn = true;
      });
      std::this_thread::sleep_for(std::chrono::milliseconds(200));
      Check(alone && !otherIn, "a call that starts during a section waits");
    }
    other.join();
    Check(otherIn, "and goes on after it");
  }
  // many threads: nobody is inside a call while another holds a section
  std::atomic<int> in{0}, sections{0};
  std::atomic<bool> clash{false};
  std::vector<std::thread> threads;
  for (int t = 0; t < 8; ++t)
    threads.emplace_back([&, t] {
      for (int i = 0; i < 20000; ++i) {
        const LibraryCall call;
        in.fetch_add(1);
        if (const Alone alone; alone) {
          sections.fetch_add(1);
          if (in.load() != 1) clash = true;
        }
        in.fetch_sub(1);
        std::atomic_thread_fence(std::memory_order_seq_cst);  // what calls share orders itself
        if (t % 2) std::this_thread::yield();
      }
    });
  for (auto& t : threads) t.join();
  Check(!clash && sections > 0, "sections and calls of eight threads exclude each other");
  return good ? 0 : 1;
}
