// gb_device_once.h as host code, for test_device_once.py
#include "gb_device_once.h"

static gb::device_once once;
static std::atomic<int> steps[gb::kMaxDevices];

// 0 = taken or already taken, 1 = the step threw, 2 = no such device
extern "C" int take(int device, int fail)
{
    try {
        once.run(device, [&] {
            if (fail) throw std::runtime_error("step");
            steps[device]++;
        });
    } catch (const std::out_of_range &) {
        return 2;
    } catch (const std::runtime_error &) {
        return 1;
    }
    return 0;
}

extern "C" int taken(int device) { return steps[device]; }
