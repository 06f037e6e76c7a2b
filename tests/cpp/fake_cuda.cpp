// fake_cuda.cpp -- see fake_cuda.h.
#include "fake_cuda.h"

namespace fake {
State st;
}

extern "C" {
// launches through <<<>>> and their registration
struct FakeConfig { dim3 g, b; size_t m; cudaStream_t s; };
static FakeConfig fake_config;
unsigned CUDARTAPI __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
  fake_config = {g, b, m, s};
  return 0;
}
cudaError_t CUDARTAPI __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = fake_config.g; *b = fake_config.b; *m = fake_config.m;
  *reinterpret_cast<cudaStream_t*>(s) = fake_config.s;
  return cudaSuccess;
}
cudaError_t CUDARTAPI __cudaGetKernel(cudaKernel_t* k, const void* f) {
  *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
  return cudaSuccess;
}
cudaError_t CUDARTAPI __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t s) {
  FAKE_CALL("launch");
  fake::enqueue(fake::of(s), [] {});
  return cudaSuccess;
}
void** CUDARTAPI __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void CUDARTAPI __cudaRegisterFatBinaryEnd(void**) {}
void CUDARTAPI __cudaUnregisterFatBinary(void**) {}
void CUDARTAPI __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}

cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = 0; return fake::call("cudaGetDevice"); }
cudaError_t CUDARTAPI cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrPageableMemoryAccess ? fake::st.pageable : 152;
  return fake::call("cudaDeviceGetAttribute");
}
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaMalloc(void** p, size_t n) { FAKE_CALL("cudaMalloc"); *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t CUDARTAPI cudaMallocHost(void** p, size_t n) { FAKE_CALL("cudaMallocHost"); *p = std::calloc(n, 1); return cudaSuccess; }
cudaError_t CUDARTAPI cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t CUDARTAPI cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  FAKE_CALL("cudaStreamCreateWithFlags");
  fake::st.stream = new fake::Stream();
  *s = reinterpret_cast<cudaStream_t>(fake::st.stream);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamDestroy(cudaStream_t s) { delete fake::of(s); return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t s) {
  FAKE_CALL("cudaStreamSynchronize");
  fake::drain(fake::of(s));
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
  FAKE_CALL("cudaMemcpy");
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
  FAKE_CALL("cudaMemcpyAsync");
  fake::enqueue(fake::of(st), [=] { std::memcpy(d, s, n); });
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
  FAKE_CALL("cudaMemsetAsync");
  fake::enqueue(fake::of(st), [=] { std::memset(d, v, n); });
  return cudaSuccess;
}
// an event holds the stream that it was last recorded on
cudaError_t CUDARTAPI cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  FAKE_CALL("cudaEventCreate");
  *e = reinterpret_cast<cudaEvent_t>(new fake::Stream*(nullptr));
  return cudaSuccess;
}
#undef cudaEventCreate
cudaError_t CUDARTAPI cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t CUDARTAPI cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<fake::Stream**>(e); return cudaSuccess; }
cudaError_t CUDARTAPI cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
  FAKE_CALL("cudaEventRecord");
  *reinterpret_cast<fake::Stream**>(e) = fake::of(s);
  fake::enqueue(fake::of(s), [] {}, e);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventSynchronize(cudaEvent_t e) {
  FAKE_CALL("cudaEventSynchronize");
  fake::Stream* s = *reinterpret_cast<fake::Stream**>(e);
  if (s) fake::drain(s, e);
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return fake::call("cudaEventElapsedTime"); }

cudaError_t CUDARTAPI cudaGraphCreate(cudaGraph_t* g, unsigned) {
  FAKE_CALL("cudaGraphCreate");
  *g = reinterpret_cast<cudaGraph_t>(new fake::Graph());
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle* h, cudaGraph_t, unsigned, unsigned) {
  *h = 1;
  return fake::call("cudaGraphConditionalHandleCreate");
}
cudaError_t CUDARTAPI cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  FAKE_CALL("cudaStreamBeginCapture");
  fake::st.capture = new std::vector<fake::Work>();
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t g, const cudaGraphNode_t*, const cudaGraphEdgeData*,
                                                    size_t, cudaStreamCaptureMode) {
  FAKE_CALL("cudaStreamBeginCaptureToGraph");
  fake::st.capture = &reinterpret_cast<fake::Graph*>(g)->work;
  return cudaSuccess;
}
cudaError_t CUDARTAPI cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  fake::st.capture = nullptr;
  *g = reinterpret_cast<cudaGraph_t>(new fake::Graph());
  return fake::call("cudaStreamEndCapture");
}
cudaError_t CUDARTAPI cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus* s, unsigned long long*, cudaGraph_t*,
                                               const cudaGraphNode_t** deps, const cudaGraphEdgeData**, size_t* n) {
  static cudaGraphNode_t node;
  *s = cudaStreamCaptureStatusActive;
  *deps = &node;
  *n = 1;
  return fake::call("cudaStreamGetCaptureInfo");
}
cudaError_t CUDARTAPI cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                       cudaGraphNodeParams* p) {
  static cudaGraph_t body[1];
  body[0] = reinterpret_cast<cudaGraph_t>(new fake::Graph());
  p->conditional.phGraph_out = body;
  return fake::call("cudaGraphAddNode");
}
cudaError_t CUDARTAPI cudaGraphAddChildGraphNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, size_t, cudaGraph_t) {
  return fake::call("cudaGraphAddChildGraphNode");
}
cudaError_t CUDARTAPI cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(new int(0));
  return fake::call("cudaGraphInstantiate");
}
cudaError_t CUDARTAPI cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
  FAKE_CALL("cudaGraphLaunch");
  fake::enqueue(fake::of(s), fake::st.step);
  return cudaSuccess;
}
}
