// Something that has to be done once on each device before a kernel's first launch there (raising its limit of dynamic
// shared memory), whichever host thread comes first.
#ifndef VDNN_B200_ONCE_H_
#define VDNN_B200_ONCE_H_

#include <atomic>
#include <mutex>

namespace vdnn {

// run() returns when `prepare` has succeeded on the device, by this thread or another; a failure is returned and tried again
// by the next call.  Statically initialised; one for each kernel.
class OncePerDevice {
public:
    constexpr OncePerDevice() : done_(0) {}
    template <class Prepare> auto run(int device, Prepare prepare) -> decltype(prepare()) {
        typedef decltype(prepare()) Status;
        if (device < 0 || device >= 64) return prepare();       // repeating it does no harm
        const unsigned long long bit = 1ull << device;
        if (done_.load(std::memory_order_acquire) & bit) return Status(0);
        std::lock_guard<std::mutex> lock(mu_);
        if (done_.load(std::memory_order_relaxed) & bit) return Status(0);
        const Status status = prepare();
        if (status == Status(0)) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }

private:
    std::atomic<unsigned long long> done_;
    std::mutex mu_;
};

}  // namespace vdnn

#endif
