// The launch helpers of csrc/common.cuh over a fake of the CUDA runtime whose next launch fails as told (see test_launch_status_cpu.py).
#include "../pam_b200/csrc/common.cu"

namespace {
cudaError_t next_launch = cudaSuccess, last = cudaSuccess;
void kernel(int) {}
}  // namespace

extern "C" {

cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) {
    const cudaError_t e = next_launch;
    if (e != cudaSuccess) last = e;                  // the runtime keeps a failed call's status until it is asked for
    next_launch = cudaSuccess;
    return e;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }

// Statuses of a launch that fails with `error` and of the check after the launch that follows it, which does not.
void shim_failed_launch(int error, int* status, int* recorded, int* status_after) {
    next_launch = (cudaError_t)error;
    *status = pamk::launch_behind(kernel, dim3(1), 32, nullptr, 1);
    *recorded = pamk_last_cuda_error();
    *status_after = pamk::check_launch();
}

// The same for a call that is not a launch (cudaMemsetAsync, cudaFuncSetAttribute), whose status goes to record_cuda_error.
void shim_failed_call(int error, int* status, int* recorded, int* status_after) {
    last = (cudaError_t)error;
    *status = pamk::record_cuda_error(last);
    *recorded = pamk_last_cuda_error();
    *status_after = pamk::check_launch();
}

}
