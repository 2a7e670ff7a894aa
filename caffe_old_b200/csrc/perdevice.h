// Answers that hold for one device: function attributes, which are set on the device that is current, and what a
// device is asked once (its SMs, whether a cluster fits).  A handle names its device, so one process may use
// several.
#pragma once
#include <mutex>

namespace cb {

template <class T>
class PerDevice {
  public:
    static constexpr int DEVICES = 64;
    // make() on the first call for a device, its answer afterwards; from any thread
    template <class F>
    T get(int device, F make) {
        if (device < 0 || device >= DEVICES) return make();
        std::lock_guard<std::mutex> guard(lock_);
        if (!known_[device]) {
            value_[device] = make();
            known_[device] = true;
        }
        return value_[device];
    }

  private:
    std::mutex lock_;
    bool known_[DEVICES] = {};
    T value_[DEVICES] = {};
};

}  // namespace cb
