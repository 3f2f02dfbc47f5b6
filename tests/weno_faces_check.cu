// weno_faces_check.cu -- host program: the interleaved FP64 WENO faces (weno_faces_up) against
// the face evaluated by itself (weno_face_up), and the branch-free divisions against the
// compiler's, bit for bit, over seeded operands that reach every branch: smooth and rough
// stencils, the switch's threshold, zero and tiny fields (the limiter), values out of the
// range of the exact residuals, NaN and infinity.  Prints one line per check.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>

#include "schemes.cuh"

static uint64_t state = 88172645463325252ull;
static uint64_t rnd()
{
    state ^= state << 13;
    state ^= state >> 7;
    state ^= state << 17;
    return state;
}
static double uni() { return (double)(rnd() >> 11) * 0x1p-53; }
static double bits(uint64_t u)
{
    double x;
    memcpy(&x, &u, 8);
    return x;
}
static bool same(double a, double b) { return a == b || (a != a && b != b); }

int main()
{
    long bad_rcp = 0, bad_div = 0;
    for (long i = 0; i < 2000000; i++) {
        uint64_t a = (rnd() >> 12) | 0x3ff0000000000000ull, b = (rnd() >> 12) | 0x3ff0000000000000ull;
        if (i % 4 == 1) { b = 0x3ffffffffffffffeull - rnd() % 1000; a = b - rnd() % 2000; }   // quotients next to 1
        if (i % 4 == 2) b = 0x3ff0000000000000ull + rnd() % 1000;
        if (i % 4 == 3) a = 0x3fffffffffffffffull - rnd() % 1000;
        const double x = bits(a), y = bits(b);
        if (y != bits(0x3fffffffffffffffull) && rcp_cr(y) != 1. / y) bad_rcp++;
        if (div_known(x, y, 1. / y) != x / y) bad_div++;
    }
    printf("rcp %ld div %ld\n", bad_rcp, bad_div);
    long bad = 0, n_lim = 0, n_nl = 0;
    for (long i = 0; i < 1000000; i++) {
        const int kind = (int)(i % 8);
        const double base[8] = {0., 300., 1e8 * uni(), uni(), 1e-20 * uni(), 1e-200 * uni(), 1e10 * uni(), 330.};
        const double b0 = base[kind], sc = std::pow(10., -18. * uni()) * (b0 == 0. ? 1. : b0);
        double s[4], t[4];
        for (int q = 0; q < 4; q++) { s[q] = kind == 3 ? uni() : b0 + sc * (uni() - 0.3); t[q] = 300. + uni(); }
        if (i % 97 == 0) s[1] = 0.;
        if (i % 101 == 0) s[2] = s[1];
        if (i % 103 == 0) s[0] = s[1] = s[2] = s[3] = 1.;
        if (i % 1009 == 0) s[0] = 1e160;
        if (i % 1013 == 0) s[rnd() % 4] = i % 2 ? NAN : INFINITY;
        if (kind == 7 && i % 3 == 0) {   // squared differences in a ratio within a few ulps of 20
            const double d = uni();
            s[1] = 0.; s[0] = -d; s[2] = d * std::sqrt(20.) * (1. + ((double)(rnd() % 9) - 4.) * 1e-16); s[3] = s[2] + uni();
        }
        const double u = i % 53 == 0 ? 0. : uni() - 0.5, v = uni() - 0.5;
        const bool full = i % 5 != 0;
        const double xm[2] = {s[0], t[0]}, x0[2] = {s[1], t[1]}, xp[2] = {s[2], t[2]}, xq[2] = {s[3], t[3]}, uu[2] = {u, v};
        double F[2];
        weno_faces_up<2>(xm, x0, xp, xq, uu, full, F);
        if (!same(F[0], weno_face_up<double>(s[0], s[1], s[2], s[3], u, full))) bad++;
        if (!same(F[1], weno_face_up<double>(t[0], t[1], t[2], t[3], v, full))) bad++;
        const double lo = std::fmin(std::fmin(-(0.5 * s[0]) + 1.5 * s[1], 0.5 * s[1] + 0.5 * s[2]), 1.5 * s[2] - 0.5 * s[3]);
        if (std::fabs(s[1]) < std::fabs((lo - s[1]) + 1e-15)) n_lim++;
        const double eo = std::pow(s[1] - s[0], 2.), em = std::pow(s[2] - s[1], 2.);
        if (full && ratio_gt(std::fmax(eo, em), std::fmin(eo, em) + 1e-15, 20.)) n_nl++;
    }
    printf("faces %ld limited %ld nonlinear %ld\n", bad, n_lim, n_nl);
    return 0;
}
