// Leading coefficients of the local expansion summed over many sources on one
// side, against FP64 sums of the same terms.  A term carries a few FP32
// roundings of its own (at most 16 x 2^-24, independent from source to
// source); the (hi, lo) sums must add nothing of note to
// 16 x 2^-24 x sqrt(sum of the terms' squares).
#include <cmath>
#include <cstdio>
#include <random>

#include "pgf_localexp.cuh"

int main() {
    using namespace pgf;
    std::mt19937 rng(1);
    std::uniform_real_distribution<double> u(0.2, 1.0), s(-1.0, 1.0);
    const int n = 100000;
    float L[kFarCoefs] = {}, lo[4] = {};
    double ref[4] = {}, sq[4] = {};
    for (int k = 0; k < n; ++k) {
        const float X = (float)u(rng), Y = (float)u(rng), Z = (float)u(rng), m = (float)u(rng);
        const double r2 = (double)X * X + (double)Y * Y + (double)Z * Z, r = std::sqrt(r2);
        // traceless moments, up to a third of m r^2
        const double f = 0.3 * m * r2;
        const float qxx = (float)(f * s(rng)), qyy = (float)(f * s(rng)), qzz = -(qxx + qyy);
        const float qxy = (float)(f * s(rng)), qxz = (float)(f * s(rng)), qyz = (float)(f * s(rng));
        add_source(X, Y, Z, (float)(1.0 / r), m, quad_op(qxx, qyy, qzz, qxy, qxz, qyz), L, lo);
        const double tz = -((double)qxx + (double)qyy);
        const double qd[3] = {(double)qxx * X + (double)qxy * Y + (double)qxz * Z,
                              (double)qxy * X + (double)qyy * Y + (double)qyz * Z,
                              (double)qxz * X + (double)qyz * Y + tz * Z};
        const double dqd = qd[0] * X + qd[1] * Y + qd[2] * Z, r3 = r * r2, r5 = r3 * r2, r7 = r5 * r2;
        const double x[3] = {X, Y, Z};
        double t[4];  // potential, then its gradient along z, x, y (rows 0 and 1 as stored)
        t[0] = m / r + 0.5 * dqd / r5;
        const int axis[3] = {2, 0, 1};
        for (int c = 0; c < 3; ++c) {
            const int d = axis[c];
            t[1 + c] = m * x[d] / r3 - qd[d] / r5 + 2.5 * dqd * x[d] / r7;
        }
        // the terms' magnitudes: monopole and quadrupole parts apart
        const double mag[4] = {m / r + std::fabs(0.5 * dqd / r5), 0, 0, 0};
        for (int c = 0; c < 4; ++c) {
            ref[c] += t[c];
            const double a = c == 0 ? mag[0]
                                    : std::fabs(m * x[axis[c - 1]] / r3) + std::fabs(qd[axis[c - 1]] / r5) +
                                          std::fabs(2.5 * dqd * x[axis[c - 1]] / r7);
            sq[c] += a * a;
        }
    }
    int bad = 0;
    for (int c = 0; c < 4; ++c) {
        const double err = std::fabs((double)L[c] + (double)lo[c] - ref[c]);
        const double tol = 16.0 * std::ldexp(1.0, -24) * std::sqrt(sq[c]);
        std::printf("coefficient %d: sum %.9g error %.3g tolerance %.3g\n", c, ref[c], err, tol);
        if (!(err <= tol)) bad = 1;
    }
    return bad;
}
