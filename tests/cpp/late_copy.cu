// A kernel that lets the kernel behind it start at once and writes its result late: copies `bytes` bytes from
// `src` to `dst` about `clocks` clocks after it has started (and always ends).
#include <cuda_runtime.h>

__global__ void late_copy_kernel(unsigned char* dst, const unsigned char* src, long long bytes, long long clocks) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const long long t0 = clock64();
    for (int i = 0; i < 1000000 && clock64() - t0 < clocks; ++i) __nanosleep(100);
    for (long long i = threadIdx.x; i < bytes; i += blockDim.x) dst[i] = src[i];
}

extern "C" int late_copy(void* dst, const void* src, long long bytes, long long clocks, void* stream) {
    late_copy_kernel<<<1, 1024, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<unsigned char*>(dst),
                                                                       static_cast<const unsigned char*>(src), bytes, clocks);
    return cudaPeekAtLastError();
}
