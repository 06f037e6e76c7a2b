// fake_cuda.h -- the CUDA runtime calls of ls_solver.cu on the host
// (fake_cuda.cpp), for tests of its orchestration on the CPU: device memory
// is host memory, a stream is a queue of work that runs when it is waited
// for, kernels are the closures of a KernelSet that the test supplies.  The
// runtime call number fail_at returns an error.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

namespace fake {
using Work = std::function<void()>;
struct Item {
  Work work;
  void* event;  // recorded here
};
struct Stream {
  std::vector<Item> queue;
};
struct Graph {
  std::vector<Work> work;  // what was captured into it, in order
};
struct State {
  Stream* stream = nullptr;           // the last one made
  std::vector<Work>* capture = nullptr;  // of the capture that is open
  long long calls = 0, fail_at = -1;
  std::string failed;  // name of the call that failed
  // work of a step graph's launch, given by the test
  Work step;
  int pageable = 1;  // cudaDevAttrPageableMemoryAccess
};
extern State st;

inline cudaError_t call(const char* name) {
  if (st.calls++ == st.fail_at) {
    st.failed = name;
    return cudaErrorUnknown;
  }
  return cudaSuccess;
}
inline void enqueue(Stream* s, Work w, void* event = nullptr) {
  if (st.capture) st.capture->push_back(std::move(w));
  else s->queue.push_back({std::move(w), event});
}
// runs a stream's work, up to the last place where `event` was recorded when given
inline void drain(Stream* s, void* event = nullptr) {
  size_t n = s->queue.size();
  while (event && n > 0 && s->queue[n - 1].event != event) --n;
  for (size_t i = 0; i < n; ++i) s->queue[i].work();
  s->queue.erase(s->queue.begin(), s->queue.begin() + n);
}
inline Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }
}  // namespace fake

#define FAKE_CALL(name)                                   \
  do {                                                    \
    const cudaError_t fake_e = fake::call(name);          \
    if (fake_e != cudaSuccess) return fake_e;             \
  } while (0)

