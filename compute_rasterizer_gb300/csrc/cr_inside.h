// The cull's proof that a batch projects inside the view, shared with its host
// test (tests/cpp/inside_check.cpp).  Compiled without contraction on both sides.
#pragma once

#include <math.h>

#ifdef __CUDACC__
#define CR_IN __host__ __device__ __forceinline__
#else
#define CR_IN inline
#endif

namespace cr {

// Whether every point decoded from a batch that w_safe() passed projects inside
// the view (|x / w| <= 1 and |y / w| <= 1): w - |x| and w - |y| are minima of
// linear functions, so over the AABB they are least at corners.  The margin,
// 2^-15 of the term sums of both rows, is far above the rounding of the two
// rows (see w_safe) and of the quotient (2^-22 of w).  The body that trusts the
// proof tests nothing, so the term sums must be finite at every corner: an
// infinite or NaN entry of T makes x / w a NaN, which no pixel follows from, and
// fmaxf and fminf would drop it.
CR_IN bool all_inside(const float* T, float mnx, float mny, float mnz, float mxx, float mxy,
                      float mxz) {
    float slack = 0.0f, mag = 0.0f;
    bool finite = true;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const float x = (k & 1) ? mxx : mnx, y = (k & 2) ? mxy : mny, z = (k & 4) ? mxz : mnz;
        float p[3], m[3];
#pragma unroll
        for (int r = 0; r < 3; r++) {
            const int c = r == 2 ? 3 : r;
            p[r] = fmaf(T[8 + c], z, fmaf(T[4 + c], y, fmaf(T[c], x, T[12 + c])));
            m[r] = ((fabsf(T[c] * x) + fabsf(T[4 + c] * y)) + fabsf(T[8 + c] * z)) + fabsf(T[12 + c]);
        }
        const float s = p[2] - fmaxf(fabsf(p[0]), fabsf(p[1]));
        const float sum = (m[0] + m[1]) + m[2];
        finite = finite && sum - sum == 0.0f;
        slack = k == 0 ? s : fminf(slack, s);
        mag = fmaxf(mag, sum);
    }
    return finite && slack >= mag * 0x1p-15f;
}

}  // namespace cr
