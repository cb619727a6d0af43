// The 3 x 3 (or smaller) normal equations of the offset fit: plain host and
// device code, so that a test can compile it for the CPU.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define XCG_FIT_FN __host__ __device__ inline
#else
#define XCG_FIT_FN inline
#endif

namespace xcg {

// S: w, wu, wv, wuu, wuv, wvv, wo, wuo, wvo summed over the points.

// Gaussian elimination with partial pivoting; singular systems leave the
// higher coefficients at 0.
XCG_FIT_FN void fit_solve(const double *S, int npar, double *c) {
    double A[3][4];
    const double M[3][3] = {{S[0], S[1], S[2]}, {S[1], S[3], S[4]}, {S[2], S[4], S[5]}};
    const double b[3] = {S[6], S[7], S[8]};
    for (int i = 0; i < npar; i++) {
        for (int j = 0; j < npar; j++) A[i][j] = M[i][j];
        A[i][3] = b[i];
    }
    for (int k = 0; k < 3; k++) c[k] = 0.0;
    int rank = npar;
    for (int k = 0; k < npar; k++) {
        int p = k;
        for (int i = k + 1; i < npar; i++)
            if (fabs(A[i][k]) > fabs(A[p][k])) p = i;
        if (!(fabs(A[p][k]) > 1e-300)) { rank = k; break; }
        if (p != k)
            for (int j = 0; j < 4; j++) { const double t = A[k][j]; A[k][j] = A[p][j]; A[p][j] = t; }
        for (int i = k + 1; i < npar; i++) {
            const double f = A[i][k] / A[k][k];
            for (int j = k; j < 4; j++) A[i][j] -= f * A[k][j];
        }
    }
    for (int k = rank - 1; k >= 0; k--) {
        double s = A[k][3];
        for (int j = k + 1; j < rank; j++) s -= A[k][j] * c[j];
        c[k] = s / A[k][k];
    }
}

// The same system by cofactors where that is as accurate: one division and a
// short chain of dependent operations (an FP64 operation's latency is what the
// serial part of a pass costs; elimination with its six divisions takes 4 us
// more per pass at npar 3).  Cofactors lose digits as the points near a line:
// with the determinant at 1e-3 of the diagonal's product their fitted offsets
// err 30 times as much as elimination's, at 1e-6 by 200 times, at 1e-8 by 190
// (medians over 1500 systems, against rational arithmetic); from 0.3 on both
// err by an ulp of the offset.  A grid of locations is at 0.9 or more.  (The
// diagonal is positive where any point has weight.)
XCG_FIT_FN void fit_solve_regular(const double *S, int npar, double *c) {
    const double a = S[0], b = S[1], d = S[2], e = S[3], f = S[4], g = S[5];
    c[0] = c[1] = c[2] = 0.0;
    if (npar == 1 && a > 1e-300) { c[0] = S[6] / a; return; }
    if (npar == 2) {
        const double det = fma(a, e, -b * b);
        if (det > 0.3 * a * e && det > 1e-300) {
            const double i = 1.0 / det;
            c[0] = fma(e, S[6], -b * S[7]) * i;
            c[1] = fma(a, S[7], -b * S[6]) * i;
            return;
        }
    }
    if (npar == 3) {
        const double m00 = fma(e, g, -f * f), m01 = fma(d, f, -b * g), m02 = fma(b, f, -d * e);
        const double m11 = fma(a, g, -d * d), m12 = fma(b, d, -a * f), m22 = fma(a, e, -b * b);
        const double det = fma(a, m00, fma(b, m01, d * m02));
        if (det > 0.3 * a * e * g && det > 1e-300) {
            const double i = 1.0 / det;
            c[0] = fma(m00, S[6], fma(m01, S[7], m02 * S[8])) * i;
            c[1] = fma(m01, S[6], fma(m11, S[7], m12 * S[8])) * i;
            c[2] = fma(m02, S[6], fma(m12, S[7], m22 * S[8])) * i;
            return;
        }
    }
    fit_solve(S, npar, c);
}

}  // namespace xcg
