// lla_device.h -- what belongs to a device and is therefore asked of the device at
// hand: a process may run contexts on several (one per host thread).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace lla {

constexpr int kMaxDevices = 64;

// Multiprocessors of the current device (at least 1).
int device_sms();

// Lets `kernel` be launched on the current device with that much dynamic shared
// memory.  Called before every launch sequence: the attribute is the device's, and
// setting it again costs well under a microsecond.
template <typename K>
inline cudaError_t allow_dynamic_smem(K *kernel, size_t bytes) {
    return cudaFuncSetAttribute((const void *)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

}  // namespace lla
