// Set-up once per device (csrc/lum_device.hpp), with made-up devices.
#include <cstdio>
#include <thread>
#include <vector>

#include "lum_device.hpp"

#define CHECK(c) do { if (!(c)) { std::printf("line %d: %s\n", __LINE__, #c); return 1; } } while (0)

int main() {
    std::atomic<uint64_t> done{0};
    int current = 0, calls[70] = {0}, fail = 0;
    auto get = [&](int* dev) { *dev = current; return 0; };
    auto work = [&] { calls[current]++; return fail; };
    for (int round = 0; round < 3; round++)
        for (int dev : {0, 1, 63, 5}) {
            current = dev;
            CHECK(lum::once_per_device(done, get, work) == 0);
        }
    for (int dev : {0, 1, 63, 5}) CHECK(calls[dev] == 1);
    // a failure is reported and tried again
    current = 7; fail = 3;
    CHECK(lum::once_per_device(done, get, work) == 3 && lum::once_per_device(done, get, work) == 3 && calls[7] == 2);
    fail = 0;
    CHECK(lum::once_per_device(done, get, work) == 0 && lum::once_per_device(done, get, work) == 0 && calls[7] == 3);
    // beyond what is kept: every time
    current = 64;
    CHECK(lum::once_per_device(done, get, work) == 0 && lum::once_per_device(done, get, work) == 0 && calls[64] == 2);
    CHECK(lum::once_per_device(done, [](int*) { return 9; }, work) == 9);
    // threads on devices of their own
    std::atomic<uint64_t> shared{0};
    std::atomic<int> n[8] = {};
    std::vector<std::thread> t;
    for (int dev = 0; dev < 8; dev++)
        t.emplace_back([&, dev] { for (int i = 0; i < 1000; i++) lum::once_per_device(shared, [&](int* d) { *d = dev; return 0; }, [&] { n[dev]++; return 0; }); });
    for (auto& x : t) x.join();
    for (auto& x : n) CHECK(x == 1);
    std::printf("ok\n");
    return 0;
}
