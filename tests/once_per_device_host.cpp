// OncePerDevice: what set() returned is not kept unless it succeeded, and holds for its
// device only.
#include "../falcon_gb300/csrc/once_per_device.h"
enum Error { kSuccess = 0, kFailure = 2 };
int main() {
    falcon::OncePerDevice once;
    int calls = 0;
    auto call = [&](int device, Error e) {
        return once(device, [&] {
            ++calls;
            return e;
        });
    };
    if (call(0, kFailure) != kFailure || calls != 1) return 1;   // a failure is returned ...
    if (call(0, kSuccess) != kSuccess || calls != 2) return 2;   // ... and tried again
    if (call(0, kFailure) != kSuccess || calls != 2) return 3;   // a success is not
    if (call(1, kFailure) != kFailure || calls != 3) return 4;   // another device
    if (call(1, kSuccess) != kSuccess || call(1, kSuccess) != kSuccess || calls != 4) return 5;
    if (call(64, kSuccess) != kSuccess || call(64, kSuccess) != kSuccess || calls != 6) return 6;
    return 0;
}
