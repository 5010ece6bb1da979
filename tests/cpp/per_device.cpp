// Numbers that are found once per device (per_device.hpp).
#include <initializer_list>

#include "per_device.hpp"

int main() {
    static umapb::PerDevice v;
    int found = 0;
    auto of = [&](int device) { return v.get(device, [&] { return ++found, int64_t(100 + device); }); };
    for (int round = 0; round < 3; ++round)
        for (int device : {1, 0, 63, 7})
            if (of(device) != 100 + device) return 1;
    if (found != 4) return 2;
    return of(64) == 164 && of(-1) == 99 ? 0 : 3;   // beyond the table: found every time
}
