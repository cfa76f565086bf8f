// The CUDA runtime calls of launch_pcg_amg on two devices, without a GPU:
// clusters of more than 8 blocks need a kernel attribute, which is set on the
// current device alone.  Each launch prints its status and its cluster size, 0 for
// a cooperative grid.  And what the compiler's start-up code calls to register
// kernels.
#include <cuda_runtime_api.h>

#include <cstdio>

int fake_device = 0, fake_largest[2] = {16, 16};

static bool allowed[2] = {false, false};
static cudaError_t check(unsigned blocks) {
    return blocks <= 8 || (allowed[fake_device] && (int)blocks <= fake_largest[fake_device])
               ? cudaSuccess
               : cudaErrorInvalidClusterSize;
}

extern "C" {
cudaError_t CUDARTAPI cudaGetDevice(int *d) { *d = fake_device; return cudaSuccess; }
cudaError_t CUDARTAPI cudaGetLastError() { return cudaSuccess; }
cudaError_t CUDARTAPI cudaFuncSetAttribute(const void *, cudaFuncAttribute attr, int v) {
    if (attr != cudaFuncAttributeNonPortableClusterSizeAllowed) return cudaErrorInvalidValue;
    if (fake_largest[fake_device] <= 8) return cudaErrorNotSupported;
    allowed[fake_device] = v != 0;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *c) {
    const cudaError_t e = check(c->attrs[0].val.clusterDim.x);
    *n = e == cudaSuccess ? 1 : 0;
    return e;
}
cudaError_t CUDARTAPI cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t,
                                                                            unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t CUDARTAPI cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **) {
    const unsigned k = c->attrs[0].val.clusterDim.x;
    std::printf("%d %u\n", (int)check(k), k);
    return check(k);
}
cudaError_t CUDARTAPI cudaLaunchCooperativeKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
    std::printf("0 0\n");
    return cudaSuccess;
}

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
unsigned __cudaPopCallConfiguration(void *, void *, size_t *, void *) { return 1; }
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, void *) { return 1; }
cudaError_t __cudaGetKernel(void **, const void *) { return cudaErrorUnknown; }
cudaError_t __cudaLaunchKernel(void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaErrorUnknown; }
}
