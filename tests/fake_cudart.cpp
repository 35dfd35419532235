// fake_cudart.cpp -- the CUDA runtime calls of libkg_b200.so without a GPU, for the
// tests of its host paths (tests/test_host_paths.py links it with the library's
// objects).  Nothing runs: device addresses are made up and never dereferenced,
// copies and fills do nothing, launches are checked and recorded.  What it knows:
//   * launch limits: grid and block extents, dynamic shared memory above 48 KB only
//     after cudaFuncSetAttribute on the launching device, the stream's device;
//   * the last-error slot of the calling thread;
//   * stream capture: allocations made during one, calls that end it;
//   * refusals that a test asks for (an allocation size, a kernel name).
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <cstdint>
#include <cstdlib>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace {

struct Stream {
  int device;
  bool capturing = false, broken = false;
  int allocs = 0;  // during the capture
};
struct Graph {
  int allocs, launches = 0;
};

std::recursive_mutex mu;
thread_local cudaError_t last = cudaSuccess;
thread_local int device = 0;
struct Config {
  dim3 grid, block;
  size_t smem;
  cudaStream_t st;
};
thread_local std::vector<Config> pushed;

std::map<const void*, std::string> names;                // host stub -> kernel
std::map<std::pair<int, const void*>, size_t> smem_set;  // (device, kernel) -> bytes
std::map<std::string, int> launched;
std::string refused_kernel;
size_t refused_size = 0;
int refused_count = 0, capture_allocs = 0;
uintptr_t next_addr = (uintptr_t)1 << 44;

cudaError_t fail(cudaError_t e) {
  if (e != cudaSuccess) last = e;
  return e;
}
Stream* S(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }

cudaError_t launch(const void* f, dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  const auto it = names.find(f);
  if (it == names.end()) return fail(cudaErrorInvalidDeviceFunction);
  if (!refused_kernel.empty() && it->second.find(refused_kernel) != std::string::npos)
    return fail(cudaErrorInvalidValue);
  if (!g.x || !g.y || !g.z || !b.x || !b.y || !b.z || g.x > 0x7fffffffu || g.y > 65535u || g.z > 65535u ||
      b.x * b.y * b.z > 1024u || b.z > 64u)
    return fail(cudaErrorInvalidConfiguration);
  if (st && S(st)->device != device) return fail(cudaErrorInvalidResourceHandle);
  if (smem > 48 * 1024) {
    const auto a = smem_set.find({device, f});
    if (a == smem_set.end() || a->second < smem) return fail(cudaErrorInvalidValue);
  }
  ++launched[it->second];
  return cudaSuccess;
}

CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t rank, void* base, const cuuint64_t* dims,
                const cuuint64_t* strides, const cuuint32_t* box, const cuuint32_t*, CUtensorMapInterleave,
                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
  if (reinterpret_cast<uintptr_t>(base) & 15u) return CUDA_ERROR_INVALID_VALUE;
  for (cuuint32_t i = 0; i < rank; ++i)
    if (!dims[i] || dims[i] > (1ull << 32) || !box[i] || box[i] > 256) return CUDA_ERROR_INVALID_VALUE;
  for (cuuint32_t i = 0; i + 1 < rank; ++i)
    if (strides[i] % 16 || strides[i] >= (1ull << 40)) return CUDA_ERROR_INVALID_VALUE;
  return CUDA_SUCCESS;
}

void* address(size_t n) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  const uintptr_t p = next_addr;
  next_addr += (n + 511) / 256 * 256;
  return reinterpret_cast<void*>(p);
}

}  // namespace

extern "C" {

// ---- the test's side -----------------------------------------------------------
void fake_reset() {
  std::lock_guard<std::recursive_mutex> lock(mu);
  refused_kernel.clear();
  refused_size = 0;
  refused_count = capture_allocs = 0;
  launched.clear();
  last = cudaSuccess;
}
void fake_refuse_alloc(size_t n) { refused_size = n; }
void fake_refuse_kernel(const char* part) { refused_kernel = part ? part : ""; }
int fake_refused() { return refused_count; }
int fake_capture_allocs() { return capture_allocs; }
int fake_launches(const char* part) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  int n = 0;
  for (const auto& l : launched)
    if (l.first.find(part) != std::string::npos) n += l.second;
  return n;
}
int fake_last_error() { return (int)last; }

// ---- registration and launches --------------------------------------------------
void** __cudaRegisterFatBinary(void* f) { return reinterpret_cast<void**>(f); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* stub, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*,
                            int*) {
  names[stub] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
  pushed.push_back({g, b, smem, reinterpret_cast<cudaStream_t>(st)});
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
  const Config c = pushed.back();
  pushed.pop_back();
  *g = c.grid;
  *b = c.block;
  *smem = c.smem;
  *reinterpret_cast<cudaStream_t*>(st) = c.st;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t smem, cudaStream_t st) {
  return launch(f, g, b, smem, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v > 227 * 1024) return fail(cudaErrorInvalidValue);
  smem_set[{device, f}] = (size_t)v;
  return cudaSuccess;
}

// ---- devices and errors -----------------------------------------------------------
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 2;
  return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
  if (d < 0 || d > 1) return fail(cudaErrorInvalidDevice);
  device = d;
  return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
  *d = device;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
  *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : 0;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() {
  const cudaError_t e = last;
  last = cudaSuccess;
  return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t e) {
  static thread_local std::string s;
  s = "error " + std::to_string((int)e);
  return s.c_str();
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  *p = reinterpret_cast<void*>(&encode);
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = address(1 << 22);
  return cudaSuccess;
}

// ---- memory ---------------------------------------------------------------------
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
  *p = reinterpret_cast<cudaMemPool_t>(address(1));
  return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t st) {
  std::lock_guard<std::recursive_mutex> lock(mu);
  if (S(st)->capturing) {  // an allocation node of the graph: always there, never of the pool
    ++capture_allocs;
    ++S(st)->allocs;
  } else if (refused_size && n == refused_size) {
    ++refused_count;
    return fail(cudaErrorMemoryAllocation);
  }
  *p = address(n);
  return cudaSuccess;
}
cudaError_t cudaFreeAsync(void*, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = address(n);
  return cudaSuccess;
}
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  *p = calloc(1, n);
  return *p ? cudaSuccess : fail(cudaErrorMemoryAllocation);
}
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFreeHost(void* p) {
  free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpy2DAsync(void*, size_t, const void*, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  const bool dev = reinterpret_cast<uintptr_t>(p) >= ((uintptr_t)1 << 44) &&
                   reinterpret_cast<uintptr_t>(p) < next_addr;
  a->type = dev ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
  a->device = device;
  return cudaSuccess;
}

// ---- streams, events, graphs -------------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
  *s = reinterpret_cast<cudaStream_t>(new Stream{device});
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  delete S(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (s && S(s)->capturing) {
    S(s)->broken = true;
    return fail(cudaErrorStreamCaptureUnsupported);
  }
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
  *S(s) = Stream{S(s)->device, true};
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
  S(s)->capturing = false;
  if (S(s)->broken) return fail(cudaErrorStreamCaptureInvalidated);
  *g = reinterpret_cast<cudaGraph_t>(new Graph{S(s)->allocs});
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
  *e = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
  delete reinterpret_cast<Graph*>(g);
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
  delete reinterpret_cast<Graph*>(e);
  return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
  Graph* g = reinterpret_cast<Graph*>(e);
  if (g->allocs && g->launches++) return fail(cudaErrorInvalidValue);  // its allocations were never freed
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = reinterpret_cast<cudaEvent_t>(address(1));
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* t, cudaEvent_t, cudaEvent_t) {
  *t = 0.f;
  return cudaSuccess;
}

}  // extern "C"
