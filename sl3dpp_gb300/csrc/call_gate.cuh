// Which host threads are inside the library, and sections in which one thread
// is there alone.
//
// The FP32 correction's graphs hold a conditional node, and building, launching
// or destroying such a graph beside another thread's CUDA calls ended in a
// segmentation fault of the driver in some runs (a lock around the graph calls
// alone made no difference). So every call that may reach the GPU counts
// itself while it runs, and the graph calls are made in a section that a thread
// enters only when no other is inside and that keeps others from entering: a
// few milliseconds for a graph that is built, microseconds for a launch. A
// thread that is not alone keeps its loop on the host. (The graphs are kept for
// small operators: a mixed run at lmax 16, 32, 64 takes 19.0, 22.6, 42.5 ms
// with them and 21.6, 24.7, 45.3 without; from lmax 96 on there is no difference.)
#pragma once

#include <cuda_runtime.h>

namespace sl3dgpu {

// A call of the C interface, for as long as it runs; calls within it count once.
class LibraryCall {
 public:
  LibraryCall();
  ~LibraryCall();
  LibraryCall(const LibraryCall&) = delete;
  LibraryCall& operator=(const LibraryCall&) = delete;
};

// Counts as one more thread inside, for a call that drives others.
class SeveralThreads {
 public:
  explicit SeveralThreads(bool on);
  ~SeveralThreads();
  SeveralThreads(const SeveralThreads&) = delete;
  SeveralThreads& operator=(const SeveralThreads&) = delete;

 private:
  bool on_;
};

// A section in which this thread is alone in the library (within a
// LibraryCall; false when another is inside). Sections nest.
class Alone {
 public:
  Alone();
  ~Alone();
  Alone(const Alone&) = delete;
  Alone& operator=(const Alone&) = delete;
  explicit operator bool() const { return held_; }

 private:
  bool held_;
};

// Destroys a graph in such a section: now if there is one, else at the start of
// the next.
void RetireGraph(cudaGraphExec_t exec);
// Graphs waiting for that.
int RetiredGraphs();

}  // namespace sl3dgpu
