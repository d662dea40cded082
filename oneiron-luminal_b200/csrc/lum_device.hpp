// Set-up that belongs to a device.  A kernel's attributes are raised on the device that is current when they are set, so a launcher that keeps
// in mind that it has done so has to keep it per device, not per process: a second runtime may live on another GPU.
#pragma once
#include <atomic>
#include <cstdint>

namespace lum {

// work() on the current device unless `done` says that it succeeded there before.  get_device(int*) and work() return 0 or an error code, which
// is handed on; a failure is not remembered.  Threads may call it at the same time: at worst the work is done twice.  Devices from 64 on
// are asked every time.
template <typename GetDevice, typename Work>
int once_per_device(std::atomic<uint64_t>& done, GetDevice get_device, Work work) {
    int dev = 0;
    if (const int e = get_device(&dev)) return e;
    const uint64_t bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
    if (done.load(std::memory_order_acquire) & bit) return 0;
    if (const int e = work()) return e;
    done.fetch_or(bit, std::memory_order_release);
    return 0;
}

}  // namespace lum
