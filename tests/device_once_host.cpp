// device_once_host.cpp -- DeviceOnce of utr_public_gb300/csrc/device_once.h: prints how
// often the action ran for each device when eight threads ask for devices 0, 1, 63 a
// hundred times each, and for device 64 in one thread.  TEST ONLY.
#include <cstdio>
#include <thread>
#include <vector>

#include "device_once.h"

int main()
{
    msk::DeviceOnce once;
    std::atomic<int> ran[65] = {};
    std::atomic<bool> early{false};
    std::vector<std::thread> ts;
    for (int t = 0; t < 8; t++)
        ts.emplace_back([&, t] {
            for (int k = 0; k < 100; k++)
                for (int d : {0, 1, 63}) {
                    once.run(d, [&] { ran[d]++; });
                    if (ran[d] == 0) early = true;  // returned before the action ran
                }
            if (t == 0)
                for (int k = 0; k < 3; k++) once.run(64, [&] { ran[64]++; });
        });
    for (auto &t : ts) t.join();
    printf("%d %d %d %d %d\n", (int)ran[0], (int)ran[1], (int)ran[63], (int)ran[64], (int)early);
    return 0;
}
