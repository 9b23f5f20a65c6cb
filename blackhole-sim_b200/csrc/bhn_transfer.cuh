// bhn_transfer.cuh -- the exact constant-coefficient Stokes step (FP64).
//
// python/blackhole_sim/polarized_transfer.py:51-70 solves dS/ds = j - K S over
// one step as the 5x5 augmented exponential
//     [S'; 1] = exp(A ds) [S; 1],   A = [[-K, j], [0, 0]],
// through scipy.linalg.expm.  Here exp(A ds) = [[E, F], [0, 1]] is formed from
// its two blocks by scaling and squaring with a truncated Taylor series
// (Moler & Van Loan, "Nineteen dubious ways to compute the exponential of a
// matrix", 2003, method 3): with X = -K ds / 2^s and ||X||_1 <= 1/4,
//     E_s = sum_{m=0}^{16} X^m / m!,   F_s = sum_{m=0}^{16} X^m y / (m + 1)!,
// y = j ds / 2^s (truncation below 1e-20 relative), then s squarings of the
// block matrix, [[E, F], [0, 1]]^2 = [[E E, E F + F], [0, 1]].
//
// Up to ||K ds||_1 = 4 only the exponential's action on the one vector is
// taken, by its Taylor series over at most four equal steps (Al-Mohy & Higham,
// "Computing the action of the matrix exponential", 2011):
//     S' = S + h sum_{m=0}^{M} X^m (j - K S) / (m + 1)!,   X = -K h, ||X||_1 <= 1,
// M so that the dropped terms stay below 2^-56 of the first: 6 to 18 products
// with a vector in place of 16 (and a squaring per doubling) with a matrix.
// 2,000,003 cells at ||K ds|| ~ 0.05: 262 -> 69 us, where the cells' 304 MB
// take 47; beyond 4 the products outnumber the squarings.  A warp with norms on
// both sides of 4 takes both forms: 2M random cells of norms 0.3 to 5.4 take 549
// us, 335 by squaring alone; neighbouring cells of a brick are mostly alike (sorted
// by norm, 243 and 311).  Queueing each warp's cells by form brought the mixed case to
// 343, and the votes and reloads cost every other brick 4 to 6 %.

#pragma once

namespace bhn {

// K of native_kernels.py:213-222 / synchrotron.py:82-94 for the 11 COEFF_NAMES
// channels (j_I, j_Q, j_U, j_V, a_I, a_Q, a_U, a_V, r_V, r_Q, r_U).
__device__ inline void propagation_matrix(const double c[11], double K[4][4]) {
    const double ai = c[4], aq = c[5], au = c[6], av = c[7], rv = c[8], rq = c[9], ru = c[10];
    K[0][0] = ai; K[0][1] = aq;  K[0][2] = au;  K[0][3] = av;
    K[1][0] = aq; K[1][1] = ai;  K[1][2] = rv;  K[1][3] = -ru;
    K[2][0] = au; K[2][1] = -rv; K[2][2] = ai;  K[2][3] = rq;
    K[3][0] = av; K[3][1] = ru;  K[3][2] = -rq; K[3][3] = ai;
}

// 1 / (m + 1), the series' divisors.
static __constant__ double kSeriesInv[19] = {1.0,        1.0 / 2.0,  1.0 / 3.0,  1.0 / 4.0,  1.0 / 5.0,  1.0 / 6.0,  1.0 / 7.0,
                                             1.0 / 8.0,  1.0 / 9.0,  1.0 / 10.0, 1.0 / 11.0, 1.0 / 12.0, 1.0 / 13.0, 1.0 / 14.0,
                                             1.0 / 15.0, 1.0 / 16.0, 1.0 / 17.0, 1.0 / 18.0, 1.0 / 19.0};

// The series form of the step (norm = ||K ds||_1 <= 4), by Horner:
// S' = S + (d + X/2 (d + X/3 (... (d + X/(M+1) d)))), d = h (j - K S).
__device__ __forceinline__ void stokes_step_series(double S[4], const double c[11], double ds, double norm) {
    const int steps = norm <= 1.0 ? 1 : (norm <= 2.0 ? 2 : 4);
    const double h = ds / steps, nu = norm / steps;
    const int terms = nu <= 1.0 / 256 ? 6 : nu <= 1.0 / 64 ? 7 : nu <= 1.0 / 16 ? 9 : nu <= 0.25 ? 12 : nu <= 0.5 ? 15 : 18;
    const double a = -c[4] * h, q = -c[5] * h, u = -c[6] * h, v = -c[7] * h, rv = -c[8] * h, rq = -c[9] * h,
                 ru = -c[10] * h;
    for (int n = 0; n < steps; ++n) {
        const double d0 = fma(a, S[0], fma(q, S[1], fma(u, S[2], fma(v, S[3], h * c[0]))));
        const double d1 = fma(q, S[0], fma(a, S[1], fma(rv, S[2], fma(-ru, S[3], h * c[1]))));
        const double d2 = fma(u, S[0], fma(-rv, S[1], fma(a, S[2], fma(rq, S[3], h * c[2]))));
        const double d3 = fma(v, S[0], fma(ru, S[1], fma(-rq, S[2], fma(a, S[3], h * c[3]))));
        double t0 = d0, t1 = d1, t2 = d2, t3 = d3;
        for (int m = terms; m >= 1; --m) {
            const double inv = kSeriesInv[m];
            const double x0 = fma(fma(a, t0, fma(q, t1, fma(u, t2, v * t3))), inv, d0);
            const double x1 = fma(fma(q, t0, fma(a, t1, fma(rv, t2, -ru * t3))), inv, d1);
            const double x2 = fma(fma(u, t0, fma(-rv, t1, fma(a, t2, rq * t3))), inv, d2);
            t3 = fma(fma(v, t0, fma(ru, t1, fma(-rq, t2, a * t3))), inv, d3);
            t0 = x0;
            t1 = x1;
            t2 = x2;
        }
        S[0] += t0;
        S[1] += t1;
        S[2] += t2;
        S[3] += t3;
    }
}

// S <- E S + F for exp([[-K, j], [0, 0]] ds); ds <= 0 leaves S unchanged
// (polarized_transfer.py:56-57).
__device__ inline void stokes_step_exact(double S[4], const double c[11], double ds) {
    if (!(ds > 0.0)) return;
    double K[4][4];
    propagation_matrix(c, K);
    double norm = 0.0;  // ||K ds||_1 (largest column sum)
    for (int col = 0; col < 4; ++col) {
        double s = 0.0;
        for (int row = 0; row < 4; ++row) s += fabs(K[row][col]);
        norm = fmax(norm, s * ds);
    }
    if (norm <= 4.0) {
        stokes_step_series(S, c, ds, norm);
        return;
    }
    int sq = 0;
    double h = ds;
    while (norm > 0.25 && sq < 1100) {  // 2^-1100 scales any finite norm below 1/4
        norm *= 0.5;
        h *= 0.5;
        ++sq;
    }
    double X[4][4], y[4];
    for (int r = 0; r < 4; ++r) {
        for (int k = 0; k < 4; ++k) X[r][k] = -K[r][k] * h;
        y[r] = c[r] * h;
    }
    // Horner: E = I + X (I + X/2 (I + ... (I + X/16))), F = (I + X/2 (I + X/3 (... (I + X/17)))) y
    double E[4][4], F[4];
    for (int r = 0; r < 4; ++r) {
        for (int k = 0; k < 4; ++k) E[r][k] = r == k ? 1.0 : 0.0;
        F[r] = y[r];
    }
    for (int m = 16; m >= 1; --m) {
        double T[4][4], Fn[4];
        const double inv_e = 1.0 / m, inv_f = 1.0 / (m + 1);
        for (int r = 0; r < 4; ++r) {
            double fv = 0.0;
            for (int k = 0; k < 4; ++k) {
                double t = 0.0;
                for (int l = 0; l < 4; ++l) t += X[r][l] * E[l][k];
                T[r][k] = (r == k ? 1.0 : 0.0) + t * inv_e;
                fv += X[r][k] * F[k];
            }
            Fn[r] = y[r] + fv * inv_f;
        }
        for (int r = 0; r < 4; ++r) {
            for (int k = 0; k < 4; ++k) E[r][k] = T[r][k];
            F[r] = Fn[r];
        }
    }
    for (int it = 0; it < sq; ++it) {
        double E2[4][4], F2[4];
        for (int r = 0; r < 4; ++r) {
            double fv = 0.0;
            for (int k = 0; k < 4; ++k) {
                double t = 0.0;
                for (int l = 0; l < 4; ++l) t += E[r][l] * E[l][k];
                E2[r][k] = t;
                fv += E[r][k] * F[k];
            }
            F2[r] = fv + F[r];
        }
        for (int r = 0; r < 4; ++r) {
            for (int k = 0; k < 4; ++k) E[r][k] = E2[r][k];
            F[r] = F2[r];
        }
    }
    double out[4];
    for (int r = 0; r < 4; ++r) {
        double v = F[r];
        for (int k = 0; k < 4; ++k) v += E[r][k] * S[k];
        out[r] = v;
    }
    for (int r = 0; r < 4; ++r) S[r] = out[r];
}

}  // namespace bhn
