// Facts and set-up that belong to a kernel ON a device -- the opt-in to large shared memory, an occupancy -- held per device, so
// that a process that drives several GPUs sets each one up.  (Host only.)
#pragma once
#include <cuda_runtime_api.h>

namespace glmasr {

static constexpr int kMaxDevices = 64;

template <typename T>
class PerDevice {
    T v_[kMaxDevices] = {};

  public:
    // the current device's value; nullptr when there is none
    T *here() {
        int dev = -1;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
        return &v_[dev];
    }
};

// set_up() (returns cudaError_t) on the first call on each device and again after a failure.  A failure leaves no error behind.
template <typename F>
cudaError_t once_per_device(PerDevice<bool> &done, F set_up) {
    bool *d = done.here();
    if (d == nullptr) return cudaErrorInvalidDevice;
    if (*d) return cudaSuccess;
    const cudaError_t e = set_up();
    if (e == cudaSuccess) *d = true;
    else (void)cudaGetLastError();
    return e;
}

}  // namespace glmasr
