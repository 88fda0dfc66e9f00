// A stand-in for the CUDA runtime, preloaded over libcudart by test_host_paths.py,
// so that the library's host code runs without a GPU: "device" memory is host
// memory filled with 1.0, a launch checks its shape and runs nothing, a capture
// collects its launches.  The fake_* functions make a call fail and say what
// was called.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#define EXPORT extern "C" __attribute__((visibility("default")))

namespace {
struct Launch {
  const void* kernel;
  const void* second;  // its second argument, once set on the node
};
struct Graph {
  std::vector<Launch*> nodes;
};
cudaError_t last_error = cudaSuccess;
std::map<std::string, int> fail_at;  // calls until the one that fails
std::map<std::string, int> calls;
std::map<const void*, std::string> names;
std::map<const void*, int> limits;   // dynamic shared memory
int lowered = 0;
Graph* capture = nullptr;
Graph* launched = nullptr;           // of the last graph launch
const void* blank = nullptr;
void* blanks[8] = {&blank, &blank, &blank, &blank, &blank, &blank, &blank, &blank};

cudaError_t done(const char* name, cudaError_t e = cudaSuccess) {
  ++calls[name];
  auto f = fail_at.find(name);
  if (f != fail_at.end() && --f->second == 0) {
    fail_at.erase(f);
    e = cudaErrorUnknown;
  }
  if (e != cudaSuccess) last_error = e;
  return e;
}
}  // namespace

EXPORT void fake_fail(const char* name, int nth) { fail_at[name] = nth; }
EXPORT int fake_calls(const char* name) { return calls[name]; }
// Times a kernel's shared-memory limit was set below what it was.
EXPORT int fake_lowered() { return lowered; }
// Kernels of the last launched graph whose name holds `part`.
EXPORT int fake_launched(const char* part) {
  int count = 0;
  if (launched != nullptr)
    for (const Launch* n : launched->nodes)
      count += names[n->kernel].find(part) != std::string::npos;
  return count;
}
// Second argument of the last launched graph's first node, null if never set.
EXPORT const void* fake_entry_argument() {
  return launched == nullptr ? nullptr : launched->nodes.front()->second;
}

// ---- registration ---------------------------------------------------------
EXPORT void** __cudaRegisterFatBinary(void*) { return new void*(nullptr); }
EXPORT void __cudaRegisterFatBinaryEnd(void**) {}
EXPORT void __cudaUnregisterFatBinary(void**) {}
EXPORT void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
EXPORT void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*,
                                   uint3*, dim3*, dim3*, int*) {
  names[host] = name;
}
EXPORT unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t) { return 0; }
EXPORT cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }

// ---- device, memory, streams, events ----------------------------------------
EXPORT cudaError_t cudaGetLastError() {
  const cudaError_t e = last_error;
  last_error = cudaSuccess;
  return e;
}
EXPORT const char* cudaGetErrorString(cudaError_t) { return "refused by the stand-in"; }
EXPORT cudaError_t cudaGetDevice(int* device) { return *device = 0, cudaSuccess; }
EXPORT cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) {
  return *value = 148, cudaSuccess;
}
EXPORT cudaError_t cudaMalloc(void** p, size_t bytes) {
  double* d = static_cast<double*>(std::malloc(bytes + 8));
  for (size_t i = 0; i < bytes / 8 + 1; ++i) d[i] = 1.0;
  return *p = d, done("cudaMalloc");
}
EXPORT cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
EXPORT cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
  return *p = std::calloc(bytes, 1), done("cudaHostAlloc");
}
EXPORT cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
EXPORT cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind,
                                   cudaStream_t) {
  return std::memmove(to, from, bytes), done("cudaMemcpyAsync");
}
EXPORT cudaError_t cudaMemsetAsync(void* to, int value, size_t bytes, cudaStream_t) {
  // Clearing a whole arena would take the diagonals with it.
  if (bytes < (size_t(1) << 20)) std::memset(to, value, bytes);
  return done("cudaMemsetAsync");
}
EXPORT cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  *a = cudaPointerAttributes{};
  a->type = cudaMemoryTypeDevice;
  return done("cudaPointerGetAttributes");
}
static int address_range(unsigned long long* base, size_t* bytes, unsigned long long p) {
  *base = p;
  *bytes = size_t(1) << 40;
  return 0;
}
EXPORT cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned,
                                                    unsigned long long,
                                                    cudaDriverEntryPointQueryResult* found) {
  *f = reinterpret_cast<void*>(&address_range);
  return *found = cudaDriverEntryPointSuccess, cudaSuccess;
}
EXPORT cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  return *p = nullptr, cudaErrorInvalidSymbol;
}
EXPORT cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  return *s = reinterpret_cast<cudaStream_t>(std::malloc(1)), cudaSuccess;
}
EXPORT cudaError_t cudaStreamDestroy(cudaStream_t s) { return std::free(s), cudaSuccess; }
EXPORT cudaError_t cudaStreamSynchronize(cudaStream_t) { return done("cudaStreamSynchronize"); }
EXPORT cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  return *e = reinterpret_cast<cudaEvent_t>(std::malloc(1)), cudaSuccess;
}
EXPORT cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
EXPORT cudaError_t cudaEventDestroy(cudaEvent_t e) { return std::free(e), cudaSuccess; }
EXPORT cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
EXPORT cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
EXPORT cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  return *ms = 1.0f, cudaSuccess;
}

// ---- launches -----------------------------------------------------------------
EXPORT cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute what, int value) {
  if (what == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    if (limits.count(kernel) != 0 && value < limits[kernel]) ++lowered;
    limits[kernel] = value;
  }
  return done("cudaFuncSetAttribute");
}
EXPORT cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int,
                                                                          size_t, unsigned) {
  return *n = 1, cudaSuccess;
}
EXPORT cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* kernel, void**) {
  const dim3 g = c->gridDim, b = c->blockDim;
  const size_t shared = limits.count(kernel) != 0 ? limits[kernel] : 48 * 1024;
  cudaError_t e = cudaSuccess;
  if (g.x == 0 || g.y == 0 || g.z == 0 || g.x > 0x7fffffffu || g.y > 65535 || g.z > 65535 ||
      b.x * b.y * b.z == 0 || b.x * b.y * b.z > 1024)
    e = cudaErrorInvalidConfiguration;
  else if (c->dynamicSmemBytes > shared)
    e = cudaErrorInvalidValue;
  e = done("cudaLaunchKernelExC", e);
  if (e == cudaSuccess && capture != nullptr) capture->nodes.push_back(new Launch{kernel, nullptr});
  return e;
}
EXPORT cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
  return done("cudaLaunchKernel");
}

// ---- graphs -------------------------------------------------------------------
EXPORT cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  return capture = new Graph, done("cudaStreamBeginCapture");
}
EXPORT cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = reinterpret_cast<cudaGraph_t>(capture);
  capture = nullptr;
  return done("cudaStreamEndCapture");
}
EXPORT cudaError_t cudaStreamGetCaptureInfo_v3(cudaStream_t, cudaStreamCaptureStatus* status,
                                               unsigned long long*, cudaGraph_t*,
                                               const cudaGraphNode_t** last,
                                               const cudaGraphEdgeData** edges, size_t* count) {
  static cudaGraphNode_t node;
  *status = cudaStreamCaptureStatusActive;
  *edges = nullptr;
  *last = &node;
  *count = capture == nullptr || capture->nodes.empty() ? 0 : 1;
  if (*count != 0) node = reinterpret_cast<cudaGraphNode_t>(capture->nodes.back());
  return done("cudaStreamGetCaptureInfo_v3");
}
EXPORT cudaError_t cudaGraphGetNodes(cudaGraph_t g, cudaGraphNode_t*, size_t* count) {
  return *count = reinterpret_cast<Graph*>(g)->nodes.size(), cudaSuccess;
}
EXPORT cudaError_t cudaGraphInstantiate(cudaGraphExec_t* exec, cudaGraph_t g, unsigned long long) {
  return *exec = reinterpret_cast<cudaGraphExec_t>(g), done("cudaGraphInstantiate");
}
EXPORT cudaError_t cudaGraphKernelNodeGetParams(cudaGraphNode_t node, cudaKernelNodeParams* p) {
  *p = cudaKernelNodeParams{};
  p->kernelParams = blanks;
  return done("cudaGraphKernelNodeGetParams",
              node == nullptr ? cudaErrorInvalidValue : cudaSuccess);
}
EXPORT cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t, cudaGraphNode_t node,
                                                    const cudaKernelNodeParams* p) {
  const cudaError_t e = done("cudaGraphExecKernelNodeSetParams");
  if (e == cudaSuccess)
    std::memcpy(&reinterpret_cast<Launch*>(node)->second, p->kernelParams[1], sizeof(void*));
  return e;
}
EXPORT cudaError_t cudaGraphLaunch(cudaGraphExec_t exec, cudaStream_t) {
  launched = reinterpret_cast<Graph*>(exec);
  return done("cudaGraphLaunch");
}
EXPORT cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
EXPORT cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
