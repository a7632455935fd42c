// once_per_device.h -- a set-up step that holds for one device at a time
// (cudaFuncSetAttribute speaks for the current device only): done at the first
// call on each, and tried again by the next call when it failed.
#ifndef RMS_ONCE_PER_DEVICE_H
#define RMS_ONCE_PER_DEVICE_H

#include <mutex>
#include <set>

namespace rms {

class OncePerDevice {
  public:
    // f() returns 0 or an error code, as this does
    template <class F>
    int operator()(int device, F&& f) {
        std::lock_guard<std::mutex> lk(mu_);
        if (done_.count(device)) return 0;
        const int e = (int)f();
        if (!e) done_.insert(device);
        return e;
    }

  private:
    std::mutex mu_;
    std::set<int> done_;
};

}  // namespace rms
#endif
