// The CUDA runtime calls of the step calls' host side, in host memory and without
// a device.  A graph is the list of kernels launched while it was captured.
#include "fake_cudart.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <vector>

namespace {
struct FakeGraph {
    std::vector<std::function<void()>> ops;
};
std::vector<std::function<void()>> g_captured;
bool g_capturing = false;
int g_graph_launches = 0;
}  // namespace

bool fake_capturing() { return g_capturing; }
void fake_launch(std::function<void()> kernel) {
    if (g_capturing) g_captured.push_back(kernel);
    else kernel();
}
int& fake_graph_launches() { return g_graph_launches; }

extern "C" {
#define OK_FN(name, ...) \
    cudaError_t name(__VA_ARGS__) { return cudaSuccess; }
OK_FN(cudaSetDevice, int)
OK_FN(cudaGetLastError, void)
OK_FN(cudaStreamSynchronize, cudaStream_t)
OK_FN(cudaStreamDestroy, cudaStream_t)
OK_FN(cudaStreamWaitEvent, cudaStream_t, cudaEvent_t, unsigned)
OK_FN(cudaEventRecord, cudaEvent_t, cudaStream_t)
OK_FN(cudaEventSynchronize, cudaEvent_t)
OK_FN(cudaEventDestroy, cudaEvent_t)
OK_FN(cudaGraphDestroy, cudaGraph_t)
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    *p = cudaDeviceProp{};
    p->multiProcessorCount = 148;
    p->cooperativeLaunch = 1;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    g_capturing = true;
    g_captured.clear();
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    g_capturing = false;
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(new FakeGraph{g_captured});
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    delete reinterpret_cast<FakeGraph*>(e);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) {
    g_graph_launches += 1;
    for (auto& f : reinterpret_cast<FakeGraph*>(e)->ops) f();
    return cudaSuccess;
}
// the (empty) device image of the test program
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
}
