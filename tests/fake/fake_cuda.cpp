// A stand-in for the CUDA runtime, for tests of the library's host code
// without a GPU: the library's own objects are linked against it instead of
// libcudart.  Device memory is host memory, kernels are recorded and do not
// run, every event is one millisecond after the one before it.  It records
// what the tests look at: live and peak device bytes, the launches, and
// launches that nothing orders after an upload they may read.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <string>
#include <vector>

namespace {

struct State {
  std::map<char*, size_t> live;
  size_t bytes = 0, peak = 0;
  // A copy from pageable memory on the legacy stream may return when the data
  // is staged; until that stream has been waited for, a launch on a
  // non-blocking stream may read what was there before.
  bool staged = false;
  int unordered = 0;
  std::map<const void*, std::string> kernels;
  std::string launches;
};

State& S() {
  static State s;
  return s;
}

// Host allocations of at least new_min bytes fail from the new_after-th on, once.
long long new_after = -1;
size_t new_min = 0;

bool non_blocking(cudaStream_t st) { return st != nullptr && st != cudaStreamLegacy; }

cudaError_t launched(const void* f, cudaStream_t st) {
  if (S().staged && non_blocking(st)) ++S().unordered;
  S().launches += S().kernels[f] + "\n";
  return cudaSuccess;
}

template <class T>
cudaError_t handle(T* out) {
  *out = reinterpret_cast<T>(std::malloc(8));
  return cudaSuccess;
}

}  // namespace

void* operator new(size_t n) {
  if (new_after >= 0 && n >= new_min && new_after-- == 0) throw std::bad_alloc();
  if (void* p = std::malloc(n ? n : 1)) return p;
  throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {

void fake_reset() {
  S().peak = S().bytes;
  S().unordered = 0;
  S().launches.clear();
}
void fake_fail_new(long long after, size_t min_bytes) {
  new_after = after;
  new_min = min_bytes;
}
int fake_new_pending() { return new_after >= 0; }
size_t fake_live_bytes() { return S().bytes; }
size_t fake_peak_bytes() { return S().peak; }
int fake_unordered() { return S().unordered; }
const char* fake_launches() { return S().launches.c_str(); }

cudaError_t cudaMalloc(void** p, size_t n) {
  *p = std::calloc(1, n);
  S().live[static_cast<char*>(*p)] = n;
  S().bytes += n;
  if (S().bytes > S().peak) S().peak = S().bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  const auto it = S().live.find(static_cast<char*>(p));
  if (it == S().live.end()) return cudaErrorInvalidValue;
  S().bytes -= it->second;
  S().live.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
  std::memcpy(d, s, n);
  S().staged = k == cudaMemcpyHostToDevice;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
  std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
  if (!non_blocking(st)) S().staged = false;
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  std::memset(a, 0, sizeof *a);
  auto it = S().live.upper_bound(static_cast<char*>(const_cast<void*>(p)));
  const bool in = it != S().live.begin() && p < std::prev(it)->first + std::prev(it)->second;
  a->type = in ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return (*p = std::malloc(n)), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }

cudaError_t cudaGetDevice(int* d) { return (*d = 0), cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return (*n = 1), cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof *p);
  p->major = 10;
  p->multiProcessorCount = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
  std::memset(a, 0, sizeof *a);
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
  return (*n = 1), cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
  // as a B200 answers for CTAs that have an SM to themselves
  static const int most[17] = {0, 148, 74, 45, 33, 26, 22, 15, 15, 15, 11, 7, 7, 7, 7, 7, 7};
  return (*n = most[c->attrs[0].val.clusterDim.x]), cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { return cudaMalloc(p, 16u << 20); }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle(g); }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  return (*s = cudaStreamCaptureStatusNone), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return handle(x); }
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return std::free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { return std::free(x), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return (*ms = 1.0f), cudaSuccess; }

// What nvcc's host stubs call: registration of the kernels and launches.
struct Launch {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
};
static std::vector<Launch>& pushed() {
  static std::vector<Launch> v;
  return v;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
  pushed().push_back({grid, block, smem, st});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
  const Launch l = pushed().back();
  pushed().pop_back();
  *grid = l.grid;
  *block = l.block;
  *smem = l.smem;
  *static_cast<cudaStream_t*>(st) = l.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t st) { return launched(f, st); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launched(f, c->stream); }
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  S().kernels[f] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

}  // extern "C"
