// PerDevice (csrc/per_device.cuh): each device's value is found once, by one
// of the threads that ask first, and every caller gets its own device's.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include "../../masterthesis_gb300/csrc/per_device.cuh"

int main() {
    for (int round = 0; round < 200; ++round) {
        scafes::PerDevice p;
        std::atomic<int> finds{0}, wrong{0}, ready{0};
        std::vector<std::thread> threads;
        for (int t = 0; t < 8; ++t)
            threads.emplace_back([&, t] {
                ++ready;
                while (ready < 8) {}
                const int dev = t % 4;
                const int v = p.get(dev, [&] {
                    ++finds;
                    return dev == 0 ? 0 : 16 >> dev;  // a device may hold none
                });
                if (v != (dev == 0 ? 0 : 16 >> dev)) ++wrong;
            });
        for (auto& t : threads) t.join();
        if (finds != 4 || wrong != 0) {
            std::printf("%d finds, %d wrong\n", finds.load(), wrong.load());
            return 1;
        }
    }
    std::puts("ok");
    return 0;
}
