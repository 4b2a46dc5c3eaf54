// A CUDA runtime without a GPU, for tests of host code: preloaded before libcudart it gives the
// library one device of compute capability 10.3 that reads pageable memory, whose memory is
// the host's and whose kernels do nothing.  It remembers which streams hold work that nobody
// has waited for, the names of the kernels launched and the pages populated between them, and
// a test can make a later launch fail.
#include <cuda_runtime_api.h>
#include <sys/syscall.h>
#include <unistd.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

#define FAKE extern "C" __attribute__((visibility("default")))

namespace {
std::set<void *> pending; // streams with work in flight
long fail_in = 0;         // the launch that fails, counted down (0: none)
cudaError_t last = cudaSuccess;
std::map<const void *, std::string> &names() { // of kernels, by their host functions
	static std::map<const void *, std::string> m;
	return m;
}
std::string launched; // names, one per line
std::string populated; // "launches before it, bytes" of each MADV_POPULATE_WRITE, one per line
long n_launches = 0;
char handles[4096];
int n_handles = 0;

void *new_handle() { return &handles[n_handles++ % 4096]; }
cudaError_t queued(void *st) {
	pending.insert(st);
	return cudaSuccess;
}
cudaError_t launch(void *st, const void *fun = nullptr) {
	launched += names()[fun] + "\n";
	++n_launches;
	if (fail_in > 0 && --fail_in == 0)
		return last = cudaErrorLaunchOutOfResources;
	return queued(st);
}
} // namespace

FAKE void fake_fail_launch(long k) { fail_in = k; }
FAKE long fake_pending() { return (long)pending.size(); }
FAKE const char *fake_launched() { return launched.c_str(); }
FAKE void fake_forget_launched() { launched.clear(), populated.clear(), n_launches = 0; }
FAKE const char *fake_populated() { return populated.c_str(); }

FAKE int madvise(void *p, size_t n, int advice) noexcept {
	if (advice == 23) // MADV_POPULATE_WRITE
		populated += std::to_string(n_launches) + " " + std::to_string(n) + "\n";
	return (int)syscall(SYS_madvise, p, n, advice);
}

FAKE cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
FAKE cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
FAKE cudaError_t cudaSetDevice(int) { return cudaSuccess; }
FAKE cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
	*v = a == cudaDevAttrComputeCapabilityMajor   ? 10
	     : a == cudaDevAttrComputeCapabilityMinor ? 3
	     : a == cudaDevAttrMultiProcessorCount    ? 152
	                                              : 1;
	return cudaSuccess;
}
FAKE cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) {
	return *a = *b = 0, cudaSuccess;
}
FAKE cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
	std::memset(p, 0, sizeof *p);
	return cudaSuccess;
}
FAKE cudaError_t cudaDeviceSynchronize() { return pending.clear(), cudaSuccess; }
FAKE cudaError_t cudaGetLastError() {
	const cudaError_t e = last;
	last = cudaSuccess;
	return e;
}
FAKE const char *cudaGetErrorString(cudaError_t) { return "made up"; }

FAKE cudaError_t cudaMalloc(void **p, size_t n) {
	return (*p = std::calloc(1, n ? n : 1)) ? cudaSuccess : cudaErrorMemoryAllocation;
}
FAKE cudaError_t cudaFree(void *p) { return std::free(p), cudaSuccess; }
FAKE cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
FAKE cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
FAKE cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
FAKE cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) {
	return *d = h, cudaSuccess;
}
FAKE cudaError_t cudaMallocAsync(void **p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
FAKE cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
FAKE cudaError_t cudaGetSymbolAddress(void **p, const void *s) {
	return *p = const_cast<void *>(s), cudaSuccess;
}
FAKE cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) {
	std::memset(a, 0, sizeof *a);
	a->type = cudaMemoryTypeUnregistered;
	return cudaSuccess;
}
FAKE cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
	return std::memmove(d, s, n), cudaSuccess;
}
FAKE cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
	std::memmove(d, s, n);
	return queued(st);
}
FAKE cudaError_t cudaMemset(void *p, int v, size_t n) { return std::memset(p, v, n), cudaSuccess; }
FAKE cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t st) {
	std::memset(p, v, n);
	return queued(st);
}

FAKE cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
	return *s = static_cast<cudaStream_t>(new_handle()), cudaSuccess;
}
FAKE cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) {
	return cudaStreamCreateWithFlags(s, 0);
}
FAKE cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaStreamSynchronize(cudaStream_t s) { return pending.erase(s), cudaSuccess; }
FAKE cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
FAKE cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
	return *s = cudaStreamCaptureStatusNone, cudaSuccess;
}
FAKE cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
FAKE cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
	return *g = static_cast<cudaGraph_t>(new_handle()), cudaSuccess;
}
FAKE cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
	return *x = static_cast<cudaGraphExec_t>(new_handle()), cudaSuccess;
}
FAKE cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) { return launch(st); }
FAKE cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
FAKE cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventCreate(cudaEvent_t *e) {
	return *e = static_cast<cudaEvent_t>(new_handle()), cudaSuccess;
}
FAKE cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
FAKE cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
FAKE cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
	return *ms = 0.0f, cudaSuccess;
}

FAKE cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
FAKE cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int,
                                                                         size_t, unsigned) {
	return *n = 8, cudaSuccess;
}
FAKE cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *fun, void **) {
	return launch(c->stream, fun);
}
FAKE cudaError_t cudaLaunchKernel(const void *fun, dim3, dim3, void **, size_t, cudaStream_t st) {
	return launch(st, fun);
}
FAKE cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void **, size_t, cudaStream_t st) {
	return launch(st, k);
}
FAKE cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *fun) {
	return *k = static_cast<cudaKernel_t>(const_cast<void *>(fun)), cudaSuccess;
}
namespace {
cudaStream_t configured;
}
FAKE unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, cudaStream_t st) {
	return configured = st, 0u;
}
FAKE cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *st) {
	return *static_cast<cudaStream_t *>(st) = configured, cudaSuccess;
}
FAKE void **__cudaRegisterFatBinary(void *) { return static_cast<void **>(new_handle()); }
FAKE void __cudaRegisterFatBinaryEnd(void **) {}
FAKE void __cudaUnregisterFatBinary(void **) {}
FAKE void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, uint3 *,
                                 uint3 *, dim3 *, dim3 *, int *) {
	names()[fun] = name;
}
FAKE void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
