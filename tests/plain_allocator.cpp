// An allocator for torch.cuda.memory.CUDAPluggableAllocator: device memory as it comes, nothing cached, no questions answered.
#include <cuda_runtime_api.h>
#include <sys/types.h>

extern "C" void* plain_alloc(ssize_t bytes, int, cudaStream_t) {
    void* p = nullptr;
    return cudaMalloc(&p, (size_t)bytes) == cudaSuccess ? p : nullptr;
}

extern "C" void plain_free(void* p, ssize_t, int, cudaStream_t) { cudaFree(p); }
