// Local expansions of the gravity of distant superparticles about a walk's
// centre, in real solid harmonics.
//
// The potential -G phi of a mass m with traceless quadrupole Q at D (relative
// to the centre) is, for |x| < |D|,
//   phi(x) = m / |D - x| + (D - x).Q.(D - x) / (2 |D - x|^5)
//          = sum_n [ L_n0 R_n0(x) + 2 Re sum_{m>0} conj(R_nm(x)) L_nm ],
//   R_nm(x) = |x|^n P_n^m e^{im phi} / (n+m)!,
//   S_nm(D) = (n-m)! P_n^m e^{im phi} / |D|^{n+1},
//   L_nm = m S_nm + (1/6) (Q : grad grad) S_nm,
// with the derivatives of S_nm again members of row n + 1 of S:
//   (dx + i dy) S_nm = -S_{n+1,m+1}, (dx - i dy) S_nm = S_{n+1,m-1},
//   dz S_nm = -S_{n+1,m}.
// The expansion keeps monopole terms to order P and quadrupole terms to order
// P - 2 (both read rows up to P of S).
//
// Row n is stored as 2n + 1 reals: [0] m = 0, [2m - 1], [2m] the real and
// imaginary parts for m > 0; rows follow each other (row n starts at n^2).
#pragma once

#ifdef __CUDACC__
#define PGF_HD __host__ __device__ __forceinline__
#define PGF_UNROLL _Pragma("unroll")
#else
#include <cmath>
#define PGF_HD inline
#define PGF_UNROLL
#endif

namespace pgf {

constexpr int kFarOrder = 8;
constexpr int kFarCoefs = (kFarOrder + 1) * (kFarOrder + 1);

// Row n + 1 of S from rows n and n - 1 (z = Z / r^2, xy = (X, Y) / r^2).
template <int N>
PGF_HD void irregular_row(const float (&p1)[2 * kFarOrder + 1], const float (&p2)[2 * kFarOrder + 1], float zr, float xr,
                          float yr, float ir2, float (&o)[2 * kFarOrder + 1]) {
    constexpr int n = N - 1;  // source row
    const float a = float(2 * n + 1) * zr;
    PGF_UNROLL
    for (int m = 0; m <= n; ++m) {
        const float b = float(n * n - m * m) * ir2;
        if (m == 0) {
            o[0] = n > 0 ? fmaf(a, p1[0], -b * p2[0]) : a * p1[0];
        } else if (m < n) {
            o[2 * m - 1] = fmaf(a, p1[2 * m - 1], -b * p2[2 * m - 1]);
            o[2 * m] = fmaf(a, p1[2 * m], -b * p2[2 * m]);
        } else {  // m == n: the second term vanishes
            o[2 * m - 1] = a * p1[2 * m - 1];
            o[2 * m] = a * p1[2 * m];
        }
    }
    const float fx = float(2 * n + 1) * xr, fy = float(2 * n + 1) * yr;
    if (n == 0) {
        o[1] = fx * p1[0];
        o[2] = fy * p1[0];
    } else {
        const float re = p1[2 * n - 1], im = p1[2 * n];
        o[2 * N - 1] = fmaf(fx, re, -fy * im);
        o[2 * N] = fmaf(fx, im, fy * re);
    }
}

// Moments of Q/6 : grad grad in the ladder operators: d+^2 (complex), d+ dz
// (complex), dz^2 (real), with d+ d- = -dz^2 on harmonic functions.
struct QuadOp {
    float ppr, ppi, pzr, pzi, zz;
};

PGF_HD QuadOp quad_op(float qxx, float qyy, float qzz, float qxy, float qxz, float qyz) {
    const float c = 1.f / 6.f;
    QuadOp q;
    q.ppr = (0.25f * c) * (qxx - qyy);
    q.ppi = (-0.5f * c) * qxy;
    q.pzr = c * qxz;
    q.pzi = -c * qyz;
    q.zz = c * (qzz - 0.5f * (qxx + qyy));
    return q;
}

// Adds the quadrupole's terms of L row K - 2 from row K of S.
template <int K, int C>
PGF_HD void quad_row(const QuadOp& q, const float (&s)[2 * kFarOrder + 1], float (&L)[C]) {
    constexpr int n = K - 2;
    constexpr int b = n * n;
    // m = 0: 2 Re(pp S_2) + 2 Re(pz S_1) + zz S_0
    L[b] = fmaf(2.f * q.ppr, s[3], fmaf(-2.f * q.ppi, s[4], fmaf(2.f * q.pzr, s[1], fmaf(-2.f * q.pzi, s[2], fmaf(q.zz, s[0], L[b])))));
    PGF_UNROLL
    for (int m = 1; m <= n; ++m) {
        float re = L[b + 2 * m - 1], im = L[b + 2 * m];
        re = fmaf(q.zz, s[2 * m - 1], re);
        im = fmaf(q.zz, s[2 * m], im);
        // pp S_{m+2} + conj(pp) S_{m-2}
        const float ur = s[2 * m + 3], ui = s[2 * m + 4];
        float vr, vi;
        if (m == 1) {  // S_{-1} = -conj(S_1)
            vr = -s[1];
            vi = s[2];
        } else if (m == 2) {
            vr = s[0];
            vi = 0.f;
        } else {
            vr = s[2 * m - 5];
            vi = s[2 * m - 4];
        }
        re = fmaf(q.ppr, ur, fmaf(-q.ppi, ui, re));
        im = fmaf(q.ppr, ui, fmaf(q.ppi, ur, im));
        re = fmaf(q.ppr, vr, m == 2 ? re : fmaf(q.ppi, vi, re));
        im = fmaf(-q.ppi, vr, m == 2 ? im : fmaf(q.ppr, vi, im));
        // pz S_{m+1} - conj(pz) S_{m-1}
        const float wr = s[2 * m + 1], wi = s[2 * m + 2];
        re = fmaf(q.pzr, wr, fmaf(-q.pzi, wi, re));
        im = fmaf(q.pzr, wi, fmaf(q.pzi, wr, im));
        if (m == 1) {
            re = fmaf(-q.pzr, s[0], re);
            im = fmaf(q.pzi, s[0], im);
        } else {
            const float tr = s[2 * m - 3], ti = s[2 * m - 2];
            re = fmaf(-q.pzr, tr, fmaf(-q.pzi, ti, re));
            im = fmaf(-q.pzr, ti, fmaf(q.pzi, tr, im));
        }
        L[b + 2 * m - 1] = re;
        L[b + 2 * m] = im;
    }
}

PGF_HD void two_sum_le(float a, float b, float& s, float& e) {
    s = a + b;
    const float bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}

// Rows N .. kFarOrder of one source, after rows N - 1 (p1) and N - 2 (p2).
// lead collects the source's terms of rows 0 and 1 (its monopole's from rows 0
// and 1 of S, its quadrupole's from rows 2 and 3).
template <int N>
PGF_HD void source_rows(const float (&p1)[2 * kFarOrder + 1], const float (&p2)[2 * kFarOrder + 1], float zr, float xr,
                        float yr, float ir2, float m, const QuadOp& q, float (&L)[kFarCoefs], float (&lo)[4],
                        float (&lead)[4]) {
    if constexpr (N <= kFarOrder) {
        float o[2 * kFarOrder + 1];
        irregular_row<N>(p1, p2, zr, xr, yr, ir2, o);
        PGF_UNROLL
        for (int k = 0; k < 2 * N + 1; ++k) {
            if (N == 1)
                lead[1 + k] = m * o[k];
            else
                L[N * N + k] = fmaf(m, o[k], L[N * N + k]);
        }
        if constexpr (N == 2 || N == 3)
            quad_row<N>(q, o, lead);
        else if constexpr (N > 3)
            quad_row<N>(q, o, L);
        if constexpr (N == 3) {
            PGF_UNROLL
            for (int k = 0; k < 4; ++k) {
                float s, e;
                two_sum_le(L[k], lead[k], s, e);
                L[k] = s;
                lo[k] += e;
            }
        }
        source_rows<N + 1>(o, p1, zr, xr, yr, ir2, m, q, L, lo, lead);
    }
}

// Adds one source at (X, Y, Z), 1/r = ri, to L.  lo holds the rounding errors
// of the sums of rows 0 and 1, the leading terms of the potential and the
// force: a source's monopole and quadrupole terms of these rows are added up
// first and enter the (hi, lo) sums once (100,000 sources on one side with
// quadrupole terms of up to a third of the monopole's: the sums are off by
// 1e-5 of themselves when the quadrupole's terms are added to the running sum
// one by one, by 3e-10 so).
PGF_HD void add_source(float X, float Y, float Z, float ri, float m, const QuadOp& q, float (&L)[kFarCoefs],
                       float (&lo)[4]) {
    const float ir2 = ri * ri;
    const float zr = Z * ir2, xr = X * ir2, yr = Y * ir2;
    float s0[2 * kFarOrder + 1], z0[2 * kFarOrder + 1];
    s0[0] = ri;
    float lead[4] = {m * ri, 0.f, 0.f, 0.f};
    source_rows<1>(s0, z0, zr, xr, yr, ir2, m, q, L, lo, lead);
}

// Row N of R from rows N - 1 (p1) and N - 2 (p2):
// R_{n+1,m} = ((2n+1) z R_nm - r^2 R_{n-1,m}) / ((n+1)^2 - m^2).
template <int N>
PGF_HD void regular_row(const float (&p1)[2 * kFarOrder + 1], const float (&p2)[2 * kFarOrder + 1], float x, float y,
                        float z, float r2, float (&o)[2 * kFarOrder + 1]) {
    constexpr int n = N - 1;
    PGF_UNROLL
    for (int m = 0; m <= n; ++m) {
        const float d = 1.f / float(N * N - m * m);
        const float a = float(2 * n + 1) * d, c = -d;
        if (m == 0) {
            o[0] = n > 0 ? fmaf(a * z, p1[0], (c * r2) * p2[0]) : a * z * p1[0];
        } else if (m < n) {
            o[2 * m - 1] = fmaf(a * z, p1[2 * m - 1], (c * r2) * p2[2 * m - 1]);
            o[2 * m] = fmaf(a * z, p1[2 * m], (c * r2) * p2[2 * m]);
        } else {
            o[2 * m - 1] = a * z * p1[2 * m - 1];
            o[2 * m] = a * z * p1[2 * m];
        }
    }
    const float f = 1.f / float(2 * N);
    if (n == 0) {
        o[1] = f * x * p1[0];
        o[2] = f * y * p1[0];
    } else {
        const float re = p1[2 * n - 1], im = p1[2 * n];
        o[2 * N - 1] = f * fmaf(x, re, -y * im);
        o[2 * N] = f * fmaf(x, im, y * re);
    }
}

// Coefficients of the expansion and of its gradient over the same R: entry k
// of row n is (phi, d phi/dx, d phi/dy, d phi/dz), each with the factor 2 of
// m > 0.  Uses (dx + i dy) R_nm = -R_{n-1,m+1}, (dx - i dy) R_nm = R_{n-1,m-1}
// and dz R_nm = R_{n-1,m}; the gradient's rows end at kFarOrder - 1.  get(i)
// returns L's real number i.
template <class Get>
PGF_HD void eval_coef(int n, int k, Get get, float& phi, float& gx, float& gy, float& gz) {
    const int m = (k + 1) / 2;
    const bool im = m > 0 && (k & 1) == 0;
    const float f = m == 0 ? 1.f : 2.f;
    phi = f * get(n * n + k);
    gx = gy = gz = 0.f;
    if (n >= kFarOrder) return;
    const int b = (n + 1) * (n + 1);  // row n + 1 of L
    gz = f * get(b + k);
    // Re/Im of L_{n+1,m+1} and L_{n+1,m-1}
    const float pr = get(b + 2 * m + 1), pi = get(b + 2 * m + 2);
    if (m == 0) {

        gx = pr;
        gy = pi;
        return;
    }
    float nr, ni;
    if (m == 1) {
        nr = get(b);
        ni = 0.f;
    } else {
        nr = get(b + 2 * m - 3);
        ni = get(b + 2 * m - 2);
    }
    if (!im) {
        gx = pr - nr;
        gy = pi + ni;
    } else {
        gx = pi - ni;
        gy = -pr - nr;
    }
}

}  // namespace pgf
