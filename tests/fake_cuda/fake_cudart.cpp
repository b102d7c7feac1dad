// A CUDA runtime without a device, for tests of the library's host side on the CPU: device memory is host
// memory, copies are copies, kernels do nothing, and the calls are counted.  fake_fail_alloc = n: the n-th
// allocation from now on fails (0: none).
#include <cstdlib>
#include <cstring>

#include <cuda_runtime_api.h>

extern "C" {
int fake_syncs, fake_allocs, fake_launches, fake_uploads, fake_fail_alloc;

static cudaError_t take(void** p, size_t n) {
    ++fake_allocs;
    if (fake_fail_alloc > 0 && --fake_fail_alloc == 0) return cudaErrorMemoryAllocation;
    *p = std::calloc(n ? n : 1, 1);
    return cudaSuccess;
}

// what compiled kernel launches call
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction() {}
void __cudaRegisterVar() {}
unsigned __cudaPushCallConfiguration() { return 0; }
int __cudaPopCallConfiguration() { return 0; }
int __cudaGetKernel() { return 0; }
int __cudaLaunchKernel() { return ++fake_launches, 0; }

cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorInvalidValue; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) {
    return *p = nullptr, cudaErrorInvalidValue;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { return std::memset(a, 0, sizeof *a), cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::calloc(n, 1), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { return *p = (cudaMemPool_t) p, cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return take(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    fake_uploads += k == cudaMemcpyHostToDevice;
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemcpyToSymbolAsync(const void*, const void*, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyFromSymbolAsync(void* d, const void*, size_t n, size_t, cudaMemcpyKind, cudaStream_t) { return std::memset(d, 0, n), cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t) s, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return ++fake_syncs, cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { return *c = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t) e, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }

// no graphs here
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, cudaStreamCaptureMode) {
    return cudaErrorNotSupported;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t, cudaStreamCaptureStatus*, unsigned long long*, cudaGraph_t*, const cudaGraphNode_t**, const cudaGraphEdgeData**,
                                     size_t*) {
    return cudaErrorNotSupported;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t, cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t, cudaGraphNodeParams*) {
    return cudaErrorNotSupported;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
