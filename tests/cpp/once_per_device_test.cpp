// OncePerDevice (pulsatrix_b200/csrc/once_per_device.hpp): once on every device, again after a failure, always from device 64 on.
#include <cstdio>
#include <initializer_list>

#include "../../pulsatrix_b200/csrc/once_per_device.hpp"

int main() {
    enum Result { kOk = 0, kFailed = 7 };
    psx::OncePerDevice once;
    int calls[66] = {};
    bool failing = true;
    auto work_on = [&](int device) {
        return once.run(device, [&] {
            ++calls[device];
            return device == 5 && failing ? kFailed : kOk;
        });
    };
    int bad = 0;
    auto check = [&](bool ok, const char* what) {
        if (!ok) {
            std::printf("failed: %s\n", what);
            ++bad;
        }
    };
    for (int turn = 0; turn < 3; ++turn) {
        for (int device : {0, 1, 63, 64, 65}) check(work_on(device) == kOk, "the result is passed on");
    }
    check(calls[0] == 1 && calls[1] == 1 && calls[63] == 1, "once on every device, whatever was done on the others");
    check(calls[64] == 3 && calls[65] == 3, "every time where there is no flag");
    check(work_on(5) == kFailed && work_on(5) == kFailed, "a failure is passed on and not noted");
    failing = false;
    check(work_on(5) == kOk && work_on(5) == kOk && calls[5] == 3, "noted once it has succeeded");
    return bad;
}
