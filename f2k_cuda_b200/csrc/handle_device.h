// Which device a handle belongs to. Its status word, buffers, streams and events live on the device that was
// current when it was made; a kernel launched for it anywhere else would reach for them, and for the caller's
// tensors, from the wrong GPU. Host code only.
#pragma once

#include "f2k_attn.h"

#include <cuda_runtime.h>

#include <string>

namespace f2k {

// F2K_OK if `device` (that of a handle) is the calling thread's current one; otherwise an error code, with the
// reason in err. Every entry point that launches or queues something for a handle asks first.
inline int check_current_device(int device, std::string& err) {
    int current = -1;
    const cudaError_t e = cudaGetDevice(&current);
    if (e != cudaSuccess) {
        err = std::string("cudaGetDevice: ") + cudaGetErrorString(e);
        return F2K_ERR_CUDA;
    }
    if (current == device) return F2K_OK;
    err = "this handle was made on device " + std::to_string(device) + ", device " + std::to_string(current) + " is current";
    return F2K_ERR_INVALID;
}

// Makes `device` current while it lives: the readers of status words synchronise the handle's device,
// whichever one is current.
class OnDevice {
public:
    explicit OnDevice(int device) {
        error = cudaGetDevice(&before_);
        if (error == cudaSuccess && before_ != device) {
            error = cudaSetDevice(device);
            changed_ = error == cudaSuccess;
        }
    }
    ~OnDevice() {
        if (changed_) cudaSetDevice(before_);
    }
    OnDevice(const OnDevice&) = delete;
    OnDevice& operator=(const OnDevice&) = delete;
    cudaError_t error = cudaSuccess;

private:
    int  before_ = -1;
    bool changed_ = false;
};

}  // namespace f2k
