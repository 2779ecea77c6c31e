// Checks quant_quick (compute_rasterizer_gb300/csrc/cr_quant.h) against
// quant_fast: wherever the quick form decides, quant_fast decides the same
// integer.  Setups as the GPU builders make them: encoder boxes (30 bits, the X
// range of a batch) and Morton cubes (21 bits, every int32), points uniform, at
// the range's ends and next to cell boundaries.  Prints the points checked and
// the uniform points drawn and decided; exits 1 on the first disagreement.
#include <cinttypes>
#include <cstdio>
#include <cstdlib>

#include "../../compute_rasterizer_gb300/csrc/cr_quant.h"

namespace {

uint64_t g_state = 0x1234567ull;
uint64_t next_u64() {
    uint64_t z = (g_state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
double uni() { return (double)(next_u64() >> 11) * 0x1p-53; }
int64_t irange(int64_t a, int64_t b) { return a + (int64_t)(next_u64() % (uint64_t)(b - a + 1)); }

long long checked = 0, uniform = 0, decided = 0;

bool point(const cr::QuantFx& q, const cr::QuantQuick& qq, int64_t X, uint32_t qmax, bool count) {
    uint32_t a = 0, b = 0;
    const bool quick = cr::quant_quick(qq, (int32_t)X, qmax, &a);
    checked++;
    if (count) {
        uniform++;
        decided += quick;
    }
    if (!quick) return true;
    if (cr::quant_fast(q, (int32_t)X, qmax, &b) && a == b) return true;
    std::printf("MISMATCH X=%" PRId64 " quick %u fast %u\n", X, a, b);
    return false;
}

bool setup(double s, double o, double m1, double m2, bool has_m2, double size, int K, int64_t lo, int64_t hi,
           int64_t xlo, int64_t xhi) {
    const cr::QuantFx q = cr::quant_setup(s, o, m1, m2, has_m2, size, K, (int32_t)xlo, (int32_t)xhi);
    const cr::QuantQuick qq = cr::quant_quick_setup(q);
    const uint32_t qmax = (1u << K) - 1u;
    for (int r = 0; r < 48; r++)
        if (!point(q, qq, irange(lo, hi), qmax, q.ok && size > 0.0)) return false;
    const int64_t ends[5] = {xlo, xhi, lo, hi, irange(xlo, xhi)};
    for (int64_t X : ends)
        if (!point(q, qq, X, qmax, false)) return false;
    const double A = std::fabs(s) * std::ldexp(1.0, K) / size, C = (double)q.c.i + std::ldexp((double)q.c.f, -64);
    for (int r = 0; r < 16 && A > 0.0; r++) {
        const double dx = std::floor(((double)irange(-2, 1ll << K) - C) / A);
        if (!(dx > -4.0 && dx < 4294967300.0)) continue;
        for (int64_t d = -1; d <= 2; d++) {
            const int64_t X = q.neg ? q.xc - ((int64_t)dx + d) : q.xc + (int64_t)dx + d;
            if (X >= xlo && X <= xhi && !point(q, qq, X, qmax, false)) return false;
        }
    }
    return true;
}

}  // namespace

int main(int argc, char** argv) {
    const int setups = argc > 1 ? std::atoi(argv[1]) : 20000;
    for (int n = 0; n < setups; n++) {
        double s = std::ldexp(uni() + 0.5, -(int)(next_u64() % 24));
        if (n % 3 == 0) s = 0.001;
        if (n % 5 == 0) s = 0.25;  // exact cells: every point on a boundary
        if (n % 7 == 0) s = -s;
        const double o = n % 2 ? std::floor(uni() * 1e7) : 0.0;
        const int64_t span = (int64_t)1 << (next_u64() % 32);
        const int64_t lo = irange(INT32_MIN, (int64_t)INT32_MAX - span), hi = lo + irange(0, span);
        const double a = (double)lo * s + o, b = (double)hi * s + o;
        const double bm = std::fmin(a, b) - (n % 3 ? uni() * 1e3 : 0.0);
        const double vlo = a - bm, vhi = b - bm;
        const double b0 = s < 0.0 ? vhi : vlo, b1 = s < 0.0 ? vlo : vhi;
        if (!setup(s, o, bm, b0, true, b1 - b0, 30, lo, hi, lo, hi)) return 1;
        const double cube = std::fabs(b - a) * (n % 4 ? 1.0 : 1.0 + 3.0 * uni());
        if (!setup(s, o, std::fmin(a, b), 0.0, false, cube, 21, lo, hi, INT32_MIN, INT32_MAX)) return 1;
    }
    std::printf("%lld %lld %lld\n", checked, uniform, decided);
    return 0;
}
