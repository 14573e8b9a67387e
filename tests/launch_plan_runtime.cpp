// The CUDA runtime that launch_plan.cu is linked with: one device shaped like a B200, on which nothing runs.
#include <cuda_runtime_api.h>

int g_failing_queries = 0;

extern "C" {
cudaError_t CUDARTAPI cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t CUDARTAPI cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* cfg) {
    if (g_failing_queries > 0) { --g_failing_queries; return cudaErrorUnknown; }
    const unsigned C = cfg->attrs[0].val.clusterDim.x;
    *n = C == 2 ? 74 : C == 4 ? 33 : C == 8 ? 15 : 7;          // a B200's
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return cudaErrorUnknown; }
cudaError_t CUDARTAPI cudaGetLastError(void) { return cudaSuccess; }
const char* CUDARTAPI cudaGetErrorString(cudaError_t) { return "made up"; }
cudaError_t CUDARTAPI cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t CUDARTAPI cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
void** CUDARTAPI __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void CUDARTAPI __cudaRegisterFatBinaryEnd(void**) {}
void CUDARTAPI __cudaUnregisterFatBinary(void**) {}
void CUDARTAPI __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
cudaError_t CUDARTAPI __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaErrorUnknown; }
cudaError_t CUDARTAPI cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorUnknown; }
}
