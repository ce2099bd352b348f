// fake_cudart.cpp -- a CUDA runtime without a device, for CPU tests of the
// library's host side: device memory is host memory, kernels and graphs do
// nothing, and the order of the calls is checked.
//
//  * A copy to the device, a device-to-device copy or a memset on the legacy
//    stream may still be on its way when it returns (pageable host memory), and
//    the library's streams do not wait for that stream: work given to one of
//    them before the legacy stream was waited for counts as unordered.
//  * Copies back to the host that no synchronisation of their stream has
//    covered yet are counted too: the caller's buffer may still be written.
//  * fake_fail_after(name, n) makes the call of that name fail after n more.
#include <cuda_runtime_api.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <vector>

namespace {

bool legacyPending = false;
int unordered = 0;
int launches = 0;  // kernels and graphs
std::map<cudaStream_t, int> backToHost;  // copies to the host not waited for
std::map<std::string, int> failAfter;
dim3 cfgGrid, cfgBlock;
size_t cfgSmem;
cudaStream_t cfgStream;

bool fails(const char *name) {
  auto it = failAfter.find(name);
  return it != failAfter.end() && it->second-- <= 0;
}

cudaError_t work(cudaStream_t st) {
  if (st && legacyPending) unordered++;
  return cudaSuccess;
}

cudaError_t legacy(void *dst, const void *src, size_t n, cudaMemcpyKind kind) {
  if (kind != cudaMemcpyDeviceToHost && fails("cudaMemcpy")) return cudaErrorUnknown;
  memcpy(dst, src, n);
  legacyPending = kind != cudaMemcpyDeviceToHost;  // a copy to the host waits for the stream
  return cudaSuccess;
}

cudaError_t handle(void **out) {
  *out = malloc(16);
  return cudaSuccess;
}

}  // namespace

extern "C" {

int fake_unordered(void) { return unordered; }
int fake_launches(void) { return launches; }
int fake_back_to_host(void) {
  int n = 0;
  for (auto &k : backToHost) n += k.second;
  return n;
}
void fake_reset(void) {
  unordered = launches = 0;
  legacyPending = false;
  backToHost.clear();
  failAfter.clear();
}
void fake_fail_after(const char *name, int calls) { failAfter[name] = calls; }

void **__cudaRegisterFatBinary(void *) {
  static void *h;
  return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *,
                            dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
  cfgGrid = g, cfgBlock = b, cfgSmem = smem, cfgStream = st;
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
  *g = cfgGrid, *b = cfgBlock, *smem = cfgSmem, *(cudaStream_t *)st = cfgStream;
  return cudaSuccess;
}

cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int,
                                                                   size_t, unsigned) {
  return *n = 1, cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n) {
  if (fails("cudaMalloc")) return cudaErrorMemoryAllocation;
  return *p = calloc(n ? n : 1, 1), cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) {
  if (fails("cudaMallocHost")) return cudaErrorMemoryAllocation;
  return *p = calloc(n ? n : 1, 1), cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFree(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *s) { return *p = (void *)s, cudaSuccess; }

cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  return legacy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  legacyPending = true;
  return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) {
  legacyPending = true;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t st) {
  if (fails(k == cudaMemcpyDeviceToHost ? "cudaMemcpyAsync to host" : "cudaMemcpyAsync"))
    return cudaErrorUnknown;
  memcpy(d, s, n);
  if (k == cudaMemcpyDeviceToHost) backToHost[st]++;
  return work(st);
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
  memset(d, v, n);
  return work(st);
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle((void **)s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return free(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  if (!s || s == cudaStreamLegacy) legacyPending = false;
  backToHost.erase(s);
  return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle((void **)e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle((void **)e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return free(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
  return *ms = 1.f, cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t st) {
  launches++;
  return work(st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
  launches++;
  return work(c->stream);
}

// captured work is checked when it is captured, and again as one launch
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle((void **)g); }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *, size_t *n) {
  return *n = 0, cudaSuccess;
}
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  return handle((void **)e);
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return free(g), cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return free(e), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
  if (fails("cudaGraphLaunch")) return cudaErrorUnknown;
  launches++;
  return work(st);
}

}  // extern "C"
