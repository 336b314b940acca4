// fake_cudart.cpp -- a stand-in for the CUDA runtime on the host, for tests of
// the engine's host code.  Device memory is heap memory, kernels do nothing, and
// work queued on a stream happens when the stream is waited for and no earlier:
// the latest a real device may do it.  Built with -fsanitize=address, so a copy
// whose host memory is gone by then, or that runs past an allocation, is reported.
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <vector>
#include <cuda_runtime_api.h>

struct CUstream_st { std::vector<std::function<void()>> queue; };

static std::vector<CUstream_st *> streams;
static bool capturing = false;
static long mallocs = 0, fail_at = -1, launches = 0, live = 0;
static cudaError_t last_error = cudaSuccess;
static std::map<void *, size_t> sizes;
static int handle;   // what every event, graph and function handle points to

static void run(CUstream_st *s)
{
	std::vector<std::function<void()>> q;
	q.swap(s->queue);
	for (auto &f : q) f();
}
static void run_all() { for (CUstream_st *s : streams) run(s); }
static void put(cudaStream_t s, std::function<void()> f)
{
	if (!capturing) s->queue.push_back(std::move(f));
}

// for the tests: the cudaMalloc call from now that is to fail (-1: none); kernels
// and graphs launched so far; device bytes allocated
extern "C" void fake_fail_malloc(long at) { fail_at = at < 0 ? -1 : mallocs+at; }
extern "C" long fake_launches() { return launches; }
extern "C" long fake_live() { return live; }

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
	if (mallocs++ == fail_at) { *p = nullptr; return last_error = cudaErrorMemoryAllocation; }
	*p = calloc(n ? n : 1, 1);
	live += n;
	sizes[*p] = n;
	return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { *p = calloc(n ? n : 1, 1); return cudaSuccess; }
cudaError_t cudaFree(void *p)
{
	run_all();
	live -= sizes[p];
	sizes.erase(p);
	free(p);
	return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { run_all(); free(p); return cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { run_all(); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t s)
{
	put(s, [=] { memset(p, v, n); });
	return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *p, size_t n, cudaMemcpyKind, cudaStream_t s)
{
	put(s, [=] { memcpy(d, p, n); });
	return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *p, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t s)
{
	put(s, [=] { for (size_t i = 0; i < h; i++) memcpy((char *)d+i*dp, (const char *)p+i*sp, w); });
	return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
	*s = new CUstream_st();
	streams.push_back(*s);
	return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s)
{
	run(s);
	for (size_t i = 0; i < streams.size(); i++)
		if (streams[i] == s) streams.erase(streams.begin()+i--);
	delete s;
	return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(s); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { run_all(); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { capturing = false; *g = (cudaGraph_t)&handle; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *, size_t *n) { *n = 0; return cudaSuccess; }
cudaError_t cudaGraphNodeGetType(cudaGraphNode_t, cudaGraphNodeType *t) { *t = cudaGraphNodeTypeEmpty; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)&handle; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { launches++; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = (cudaEvent_t)&handle; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { run_all(); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int)
{
	memset(p, 0, sizeof *p);
	p->major = 10; p->minor = 3; p->multiProcessorCount = 152;
	return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "fake error"; }
cudaError_t cudaGetLastError()
{
	const cudaError_t e = last_error;
	last_error = cudaSuccess;
	return e;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *)
{
	static void *scratch = calloc(1, 1 << 23);
	*p = scratch;
	return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
	memset(a, 0, sizeof *a);
	return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) { launches++; return cudaSuccess; }

// what compiled kernel launches and registrations call
void **__cudaRegisterFatBinary(void *) { static void *p; return &p; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { return cudaSuccess; }
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *) { *k = (cudaKernel_t)&handle; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void **, size_t, cudaStream_t) { launches++; return cudaSuccess; }
}
