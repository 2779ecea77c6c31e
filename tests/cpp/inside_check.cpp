// The cull's inside proof (compute_rasterizer_gb300/csrc/cr_inside.h) on random
// transforms and boxes, some with infinite or NaN entries and flat boxes: wherever
// it holds, every sampled point of the box must have |x / w| <= 1 and |y / w| <= 1
// in float, a NaN failing.  Prints "proofs P special S bad B": proofs that held,
// transforms with an entry that is not finite, and points outside a proof.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../compute_rasterizer_gb300/csrc/cr_inside.h"

int main(int argc, char** argv) {
    const long n = argc > 1 ? strtol(argv[1], nullptr, 10) : 100000;
    std::mt19937 rng(7);
    std::uniform_real_distribution<float> u(-1.0f, 1.0f);
    unsigned long proofs = 0, special = 0, bad = 0;
    for (long i = 0; i < n; i++) {
        float T[16];
        for (float& t : T) t = u(rng);
        T[15] = 2.0f + 6.0f * std::fabs(T[15]);  // w well above x and y for most boxes
        if (i % 4 == 3) {  // one entry of rows x, y that no finite point survives
            const int e = 4 * (int)(rng() % 4u) + (int)(rng() % 2u);
            const float v[3] = {INFINITY, -INFINITY, NAN};
            T[e] = v[rng() % 3u];
            special++;
        }
        float mn[3], mx[3];
        for (int k = 0; k < 3; k++) {
            const float a = u(rng), b = u(rng);
            mn[k] = std::fmin(a, b);
            mx[k] = std::fmax(a, b);
            if (rng() % 4u == 0u) mn[k] = mx[k] = 0.0f;  // flat, on the axis: inf * 0
        }
        if (!cr::all_inside(T, mn[0], mn[1], mn[2], mx[0], mx[1], mx[2])) continue;
        proofs++;
        for (int s = 0; s < 64; s++) {
            float p[3];
            for (int k = 0; k < 3; k++) {
                const float f = s < 8 ? (float)((s >> k) & 1) : 0.5f + 0.5f * u(rng);
                p[k] = std::fmin(std::fmax(std::fmaf(f, mx[k] - mn[k], mn[k]), mn[k]), mx[k]);
            }
            float q[3];
            for (int r = 0; r < 3; r++) {
                const int c = r == 2 ? 3 : r;
                q[r] = std::fmaf(T[8 + c], p[2], std::fmaf(T[4 + c], p[1], std::fmaf(T[c], p[0], T[12 + c])));
            }
            const float rw = 1.0f / q[2];
            bad += !(std::fabs(q[0] * rw) <= 1.0f && std::fabs(q[1] * rw) <= 1.0f);
        }
    }
    printf("%lu %lu %lu\n", proofs, special, bad);
    return bad == 0 ? 0 : 1;
}
