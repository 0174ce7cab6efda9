// A CUDA runtime without a device, for tests of the library's host code: the
// library's objects are linked with it instead of cudart.  Device memory is
// addresses only, of which there is a settable amount; kernels do not run but
// are recorded by name with their stream; streams have priorities and may be
// said to belong to an SM partition.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
std::map<const void*, std::string> names;
std::string launched;
std::map<char*, size_t> held;
size_t limit = ~size_t(0), used = 0, peak = 0;
char* next_address = reinterpret_cast<char*>(uintptr_t(1) << 40);
struct Stream {
  int priority;
  bool partition;
};
std::map<cudaStream_t, Stream> streams;
uintptr_t next_handle = 1 << 20;
bool capturing = false;
int grown_in_capture = 0;
dim3 grid_, block_;
size_t smem_;
cudaStream_t stream_;

template <class T>
T handle() {
  return reinterpret_cast<T>(next_handle += 16);
}
cudaError_t record(const void* f, cudaStream_t s) {
  launched += names[f] + " " + std::to_string(reinterpret_cast<uintptr_t>(s)) + "\n";
  return cudaSuccess;
}
CUresult stream_green(CUstream s, CUgreenCtx* g) {
  auto it = streams.find(s);
  *g = it != streams.end() && it->second.partition ? reinterpret_cast<CUgreenCtx>(uintptr_t(64)) : nullptr;
  return CUDA_SUCCESS;
}
}  // namespace

#define OK(call) \
  extern "C" cudaError_t call { return cudaSuccess; }

extern "C" {
// what a test asks and says
void fake_reset(size_t bytes) {
  launched.clear();
  limit = bytes;
  peak = used;
  grown_in_capture = 0;
}
const char* fake_launches() { return launched.c_str(); }
size_t fake_used() { return used; }
size_t fake_peak() { return peak; }
int fake_grown_in_capture() { return grown_in_capture; }
void* fake_stream(int priority, int partition) {
  cudaStream_t s = handle<cudaStream_t>();
  streams[s] = Stream{priority, partition != 0};
  return s;
}
int fake_priority(uintptr_t s) { return streams.count((cudaStream_t)s) ? streams[(cudaStream_t)s].priority : 99; }
int fake_streams() { return (int)streams.size(); }

// what nvcc's host code calls
void** __cudaRegisterFatBinary(void*) {
  static void* h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
  names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) {
  grid_ = g, block_ = b, smem_ = m, stream_ = s;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
  *g = grid_, *b = block_, *m = smem_, *static_cast<cudaStream_t*>(s) = stream_;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t, cudaStream_t s) { return record(f, s); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return record(f, c->stream); }

cudaError_t cudaMalloc(void** p, size_t n) {
  if (capturing) {
    ++grown_in_capture;
    return cudaErrorStreamCaptureUnsupported;
  }
  if (n > limit - used || used > limit) return cudaErrorMemoryAllocation;
  *p = next_address;
  held[next_address] = n;
  next_address += (n + 511) / 512 * 512;
  used += n;
  peak = used > peak ? used : peak;
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  auto it = held.find(static_cast<char*>(p));
  if (it == held.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
  used -= it->second;
  held.erase(it);
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
  *p = std::calloc(1, n);
  return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
  std::free(p);
  return cudaSuccess;
}

cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int priority) {
  *s = static_cast<cudaStream_t>(fake_stream(priority, 0));
  return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) { return cudaStreamCreateWithPriority(s, f, 0); }
cudaError_t cudaStreamGetPriority(cudaStream_t s, int* p) {
  *p = streams.count(s) ? streams[s].priority : 0;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  streams.erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
  capturing = true;
  return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  capturing = false;
  *g = handle<cudaGraph_t>();
  return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = handle<cudaGraphExec_t>();
  return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = handle<cudaEvent_t>();
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = 0.f;
  return cudaSuccess;
}

cudaError_t cudaGetDevice(int* d) {
  *d = 0;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
  std::memset(p, 0, sizeof(*p));
  p->multiProcessorCount = 148;
  p->l2CacheSize = 126 << 20;
  p->sharedMemPerBlockOptin = 227 << 10;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = 148;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
  *lo = 0, *hi = -5;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int block, size_t, unsigned) {
  *n = 2048 / block;
  return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
  *p = next_address;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char* name, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
  const bool known = std::strcmp(name, "cuStreamGetGreenCtx") == 0;
  *p = known ? reinterpret_cast<void*>(&stream_green) : nullptr;
  *q = known ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
  return cudaSuccess;
}
}

OK(cudaDeviceSynchronize())
OK(cudaEventDestroy(cudaEvent_t))
OK(cudaEventRecord(cudaEvent_t, cudaStream_t))
OK(cudaEventSynchronize(cudaEvent_t))
OK(cudaFreeAsync(void*, cudaStream_t))
OK(cudaFuncSetAttribute(const void*, cudaFuncAttribute, int))
OK(cudaGetLastError())
OK(cudaGraphDestroy(cudaGraph_t))
OK(cudaGraphExecDestroy(cudaGraphExec_t))
OK(cudaGraphLaunch(cudaGraphExec_t, cudaStream_t))
OK(cudaMallocFromPoolAsync(void**, size_t, cudaMemPool_t, cudaStream_t))
OK(cudaMemPoolCreate(cudaMemPool_t*, const cudaMemPoolProps*))
OK(cudaMemPoolDestroy(cudaMemPool_t))
OK(cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*))
OK(cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t))
OK(cudaMemset(void*, int, size_t))
OK(cudaMemsetAsync(void*, int, size_t, cudaStream_t))
OK(cudaPeekAtLastError())
OK(cudaSetDevice(int))
OK(cudaStreamSynchronize(cudaStream_t))
OK(cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned))
