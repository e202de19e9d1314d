// A CUDA runtime for seq_host.cu that needs no GPU: prints what is launched and
// fails on request.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <new>

int g_fail_launch = -1;     // the kernel launch (by number) that fails
static int g_launch = 0;
bool g_fail_graph = false;  // cudaGraphLaunch fails
long g_fail_new = -1;       // the host allocation (counted from arming) that fails
int g_mode = 0;             // capture interaction mode of the thread
int g_graphs = 0;           // live graphs
static int g_nodes = 0;            // nodes of the graph built last
static int g_arg[64];              // the argument of each of its nodes

static int first_arg(void** p) { return *static_cast<int*>(p[0]); }

void* operator new(size_t n) {
    if (g_fail_new >= 0 && g_fail_new-- == 0) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

extern "C" {
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "error"; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void** args) {
    if (g_launch++ == g_fail_launch) return cudaErrorLaunchOutOfResources;
    std::printf("launch %d\n", first_arg(args));
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode* m) {
    const int was = g_mode;
    g_mode = *m;
    *m = (cudaStreamCaptureMode)was;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
    ++g_graphs;
    g_nodes = 0;
    *g = (cudaGraph_t)0x10;
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) {
    --g_graphs;
    return cudaSuccess;
}
cudaError_t cudaGraphAddNode_v2(cudaGraphNode_t* n, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                cudaGraphNodeParams* p) {
    g_arg[g_nodes] = first_arg(p->kernel.kernelParams);
    *n = (cudaGraphNode_t)(uintptr_t)++g_nodes;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = (cudaGraphExec_t)0x20;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphExecKernelNodeSetParams(cudaGraphExec_t, cudaGraphNode_t n, const cudaKernelNodeParams* p) {
    const int i = (int)(uintptr_t)n;
    if (i < 1 || i > g_nodes) return cudaErrorInvalidValue;
    g_arg[i - 1] = first_arg(p->kernelParams);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    if (g_fail_graph) return cudaErrorUnknown;
    std::printf("graph");
    for (int i = 0; i < g_nodes; ++i) std::printf(" %d", g_arg[i]);
    std::printf("\n");
    return cudaSuccess;
}
// registration of the (empty) device code
void** __cudaRegisterFatBinary(void*) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t __cudaGetKernel(void**, const void*) { return cudaSuccess; }
}
