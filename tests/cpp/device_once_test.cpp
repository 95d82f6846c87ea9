// State kept per device (device_once.h), with the devices and the calls faked by
// the host.  Exits 0 if every check holds, else with the number of the first that
// does not.
#include "device_once.h"

#define CHECK(n, cond) \
    if (!(cond)) return n

int main()
{
    agb::DeviceOnce once;
    int calls[3] = {0, 0, 0};
    bool fails = false;
    auto use = [&](int dev) {
        return once.run(dev, [&] {
            calls[dev]++;
            return !fails;
        });
    };
    CHECK(1, use(0) && use(0) && calls[0] == 1);
    CHECK(2, use(1) && calls[1] == 1 && use(0) && calls[0] == 1);   // another device makes its own
    fails = true;
    CHECK(3, !use(2) && !use(2) && calls[2] == 2 && use(0));        // a failure is tried again
    fails = false;
    CHECK(4, use(2) && use(2) && calls[2] == 3);

    agb::DevicePointer<int> ptr;
    int a = 0, b = 0, made = 0;
    CHECK(5, ptr.get(0, [&] { made++; return &a; }) == &a);
    CHECK(6, ptr.get(1, [&] { made++; return &b; }) == &b);
    CHECK(7, ptr.get(0, [&] { made++; return &b; }) == &a && made == 2);
    CHECK(8, ptr.get(5, [&] { made++; return (int*)nullptr; }) == nullptr && ptr.get(5, [&] { made++; return &a; }) == &a);

    // past the table (and without a device): made every time
    int over = 0;
    for (int q = 0; q < 2; q++) CHECK(9, once.run(agb::MAX_DEVICES, [&] { over++; return true; }) && once.run(-1, [&] { over++; return true; }));
    CHECK(10, over == 4);
    return 0;
}
