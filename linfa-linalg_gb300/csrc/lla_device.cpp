// lla_device.cpp -- see lla_device.h.
#include "lla_device.h"

#include <atomic>

namespace lla {

static std::atomic<int> g_sms[kMaxDevices];  // 0: not asked yet

int device_sms() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 1;
    const bool keep = dev >= 0 && dev < kMaxDevices;
    if (keep && (sms = g_sms[dev].load(std::memory_order_relaxed)) > 0) return sms;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) return 1;
    if (keep) g_sms[dev].store(sms, std::memory_order_relaxed);
    return sms;
}

}  // namespace lla
