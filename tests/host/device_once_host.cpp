// Set-up once per device, compiled for the host against a fake current device, for tests/test_device_once.py.
#include <thread>
#include <vector>

static thread_local int current = 0;
static int cudaGetDevice(int *dev) { return *dev = current, 0; }
#define FLG_CUDA(call)       \
    do {                     \
        if (call) return -1; \
    } while (0)
#include "../../fluidlets_gb300/csrc/device_once.cuh"

static std::atomic<int> calls[128];
static int attribute(int fails) { return calls[current]++, fails; }
static int launch(int fails) {
    FLG_ONCE_PER_DEVICE(FLG_CUDA(attribute(fails)));
    return 0;
}

extern "C" int launch_on(int dev, int fails) {
    current = dev;
    return launch(fails);
}
extern "C" int set_ups(int dev) { return calls[dev].load(); }
extern "C" void launch_threads(int dev, int n) {
    std::vector<std::thread> t;
    for (int k = 0; k < n; k++)
        t.emplace_back([=] {
            current = dev;
            for (int i = 0; i < 100; i++) launch(0);
        });
    for (auto &x : t) x.join();
}
