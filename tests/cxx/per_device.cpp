// Once per device, from several threads: counts of the makes for the test.
#include "per_device.cuh"
#include <atomic>
#include <thread>
#include <vector>
static std::atomic<int> makes[80];
static xbg::PerDevice value;
extern "C" {
int get(int dev, int result) {
    return value.get(dev, [&] { makes[dev]++; return result; });
}
int made(int dev) { return makes[dev].load(); }
int race(int dev, int threads) {   // how many of the threads got the value
    std::atomic<int> good{0};
    std::vector<std::thread> t;
    for (int k = 0; k < threads; k++)
        t.emplace_back([&] { for (int j = 0; j < 1000; j++) good += get(dev, 5) == 5; });
    for (auto& x : t) x.join();
    return good.load();
}
}
