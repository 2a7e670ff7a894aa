// PerDevice: one answer per device, asked once each, from any thread.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
#include "perdevice.h"

int main() {
    cb::PerDevice<int> p;
    std::atomic<int> asked[3] = {};
    std::atomic<int> wrong{0};
    auto use = [&](int dev) {
        if (p.get(dev, [&] { ++asked[dev]; return 10 + dev; }) != 10 + dev) ++wrong;
    };
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; ++t)
        ts.emplace_back([&, t] { for (int k = 0; k < 300; ++k) use((t + k) % 3); });
    for (auto& t : ts) t.join();
    int beyond = 0;
    for (int k = 0; k < 2; ++k) p.get(cb::PerDevice<int>::DEVICES, [&] { return ++beyond; });
    std::printf("%d %d %d wrong %d beyond %d\n", asked[0].load(), asked[1].load(), asked[2].load(), wrong.load(), beyond);
    return 0;
}
