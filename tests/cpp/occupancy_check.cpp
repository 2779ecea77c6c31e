// cached_occupancy with a fake driver: a failed answer is not kept, a good one is,
// each device for itself, and devices past the table are asked every time.
#include <cstdio>

#include "../../compute_rasterizer_gb300/csrc/cr_occupancy.h"

int main() {
    static cr::OccupancyCache cache;
    int calls = 0, answer = 0;
    const auto ask = [&](int device) {
        return cr::cached_occupancy(cache, device, [&] { calls++; return answer; });
    };
    bool ok = ask(0) == 1 && calls == 1;  // the driver fails
    answer = 9;
    ok = ok && ask(0) == 9 && calls == 2;
    answer = 0;
    ok = ok && ask(0) == 9 && calls == 2;  // kept
    ok = ok && ask(1) == 1 && calls == 3;  // another device: not device 0's 9
    answer = 5;
    ok = ok && ask(1) == 5 && ask(0) == 9 && calls == 4;
    ok = ok && ask(64) == 5 && ask(64) == 5 && ask(-1) == 5 && calls == 7;
    printf("%s\n", ok ? "ok" : "wrong");
    return ok ? 0 : 1;
}
