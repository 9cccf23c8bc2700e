// PerDevice: every device has its own value, found once however many threads ask.
#include "per_device.cuh"

#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

int main() {
    static eg::PerDevice<int> values;
    std::atomic<int> found[80] = {};
    auto ask = [&](int dev) {
        return values.get(dev, [&] {
            found[dev]++;
            return 100 + dev;
        });
    };
    std::vector<std::thread> ts;
    std::atomic<bool> ok{true};
    for (int t = 0; t < 16; t++)
        ts.emplace_back([&] {
            for (int i = 0; i < 4000; i++)
                if (ask(i % 8) != 100 + i % 8) ok = false;
        });
    for (auto &t : ts) t.join();
    for (int d = 0; d < 8; d++) ok = ok && found[d] == 1;
    for (int i = 0; i < 3; i++) ok = ok && ask(70) == 170; // beyond the table: asked for every time
    ok = ok && found[70] == 3 && found[9] == 0;
    std::puts(ok ? "per device ok" : "per device FAILED");
    return ok ? 0 : 1;
}
