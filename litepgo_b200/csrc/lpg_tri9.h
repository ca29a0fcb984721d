// Eigenvalue clamp of a symmetric 9x9 matrix by the few eigenpairs of one sign, one thread per matrix:
// M+ = M + sum_{L < 0} |L| v v^T, or sum_{L > 0} L v v^T where those are fewer, so at most four of them (the
// projected Hessian's clamp of a tet's tangent in the q basis, mesh_energy.cpp:16-27). Compiled for the
// host as well, where a test checks it against an eigensolver.
//   1. Householder tridiagonalisation in registers (Golub & Van Loan, Matrix Computations, 8.3.1);
//   2. the number of eigenvalues of each sign by Sturm counts in FP64, and each wanted one to 3e-7 of the
//      norm by bisection in FP32, more closely near zero (Givens; Wilkinson, The Algebraic Eigenvalue Problem, 5.39);
//   3. Rayleigh quotient iteration from there (Parlett, The Symmetric Eigenvalue Problem, 4.6) with the
//      pivoted LU factors of T - s I, orthogonalised against the vectors already found, until the residual
//      is at round-off: two or three solves;
//   4. the reflectors applied to the vectors.
// What it returns is checked: k orthonormal vectors with residuals at round-off and Rayleigh quotients of
// the wanted sign, where the Sturm counts say that there are k such eigenvalues, span their eigenspace. A
// matrix that fails the check (the iteration can run to another eigenvalue) is left to the Jacobi method.
// Against that method's six sweeps of 36 rotations (a square root, a division and a reciprocal square root
// each, and 81 entries of eigenvectors) this is about a fifth of the operations.
#pragma once

#include "lpg_clamp9.h"

namespace lpg {

#ifdef __CUDA_ARCH__
#define C9_UNROLL _Pragma("unroll")
#define C9_LOOP _Pragma("unroll 1")
#else
#define C9_UNROLL
#define C9_LOOP
#endif

constexpr int kTri9Scratch = 75; // reflectors (35), four vectors, their eigenvalues (odd: conflict-free rows)

// Eigenvalues of the tridiagonal (d, squared off-diagonals e2) below x, by the signs of the leading
// principal minors. |d|, |e| <= a few (the matrix is scaled), nine rows: no rescaling in FP64. A minor that
// is exactly zero counts by the sign of its zero: x is then an eigenvalue of a leading block.
LPG_C9 int tri9_count(const double (&d)[9], const double (&e2)[8], double x) {
    double p2 = 1.0, p1 = d[0] - x;
    if (p1 == 0.0) p1 = -1e-30;
    int cnt = p1 < 0.0;
    C9_UNROLL
    for (int i = 1; i < 9; ++i) {
        double p = (d[i] - x) * p1 - e2[i - 1] * p2;
        if (p == 0.0) p = p1 < 0.0 ? 1e-30 : -1e-30;
        cnt += (p < 0.0) != (p1 < 0.0);
        p2 = p1;
        p1 = p;
    }
    return cnt;
}
// The same in FP32, to place a shift: a count that is one off there costs an iteration or the fallback. The
// signs go into a word, one instruction a row, and the pair is scaled up once where both have become small.
LPG_C9 int tri9_count_near(const float (&d)[9], const float (&e2)[8], float x) {
    float p2 = 1.f, p1 = d[0] - x;
    unsigned neg = p1 < 0.f;
    C9_UNROLL
    for (int i = 1; i < 9; ++i) {
        const float p = (d[i] - x) * p1 - e2[i - 1] * p2;
        neg = neg << 1 | (p < 0.f ? 1u : 0u);
        p2 = p1;
        p1 = p;
        if (i == 4 && C9F(fabs)(p1) < 1e-8f && C9F(fabs)(p2) < 1e-8f) {
            p1 *= 1e16f;
            p2 *= 1e16f;
        }
    }
    neg ^= neg >> 1; // bit: this minor's sign differs from the one before (the first from +1)
#ifdef __CUDA_ARCH__
    return __popc(neg);
#else
    return __builtin_popcount(neg);
#endif
}

// 1 / x to round-off for 1e-30 < |x| < 1e30: Newton's iteration r <- r + r (1 - x r) from the FP32
// reciprocal (7, 14, 28 digits), whose error only perturbs the elimination it is used in.
LPG_C9 double c9_recip(double x) {
#ifdef __CUDA_ARCH__
    double r = __fdividef(1.f, static_cast<float>(x));
#else
    double r = 1.f / static_cast<float>(x);
#endif
    r += r * (1.0 - x * r);
    return r + r * (1.0 - x * r);
}
LPG_C9 float c9_recip(float x) {
#ifdef __CUDA_ARCH__
    return __fdividef(1.f, x);
#else
    return 1.f / x;
#endif
}

// x <- (T - s I)^-1 x by Gaussian elimination with partial pivoting.
template <typename R> LPG_C9 void tri9_solve(const R (&d)[9], const R (&e)[8], R s, R (&x)[9]) {
    R ip[9], u1[8], u2[8]; // reciprocal pivots, the rows' other entries
    R a = d[0] - s, b = e[0];
    C9_UNROLL
    for (int i = 0; i < 8; ++i) {
        const R ei = e[i], dn = d[i + 1] - s, en = i < 7 ? e[i + 1] : R(0);
        const bool swap = C9F(fabs)(ei) > C9F(fabs)(a);
        R p = swap ? ei : a;
        const R q = swap ? dn : b, o = swap ? en : R(0), xp = swap ? x[i + 1] : x[i];
        const R a2 = swap ? a : ei, b2 = swap ? b : dn, c2 = swap ? R(0) : en, x2 = swap ? x[i] : x[i + 1];
        if (C9F(fabs)(p) < Eps<R>::v) p = Eps<R>::v;
        ip[i] = c9_recip(p);
        u1[i] = q;
        u2[i] = o;
        x[i] = xp;
        const R l = a2 * ip[i];
        a = b2 - l * q;
        b = c2 - l * o;
        x[i + 1] = x2 - l * xp;
    }
    if (C9F(fabs)(a) < Eps<R>::v) a = Eps<R>::v;
    ip[8] = c9_recip(a);
    x[8] *= ip[8];
    x[7] = (x[7] - u1[7] * x[8]) * ip[7];
    C9_UNROLL
    for (int i = 6; i >= 0; --i) x[i] = (x[i] - u1[i] * x[i + 1] - u2[i] * x[i + 2]) * ip[i];
}

// Step k of the tridiagonalisation and those after it: I - u u^T maps column k below the diagonal to
// (alpha, 0, ...); u goes to sc.
template <int k, typename R> LPG_C9 void tri9_reduce(R (&A)[45], R (&d)[9], R (&e)[8], R* sc) {
    constexpr int n = 8 - k; // length of u
    R u[8], w[8];
    R x2 = 0;
    const R x0 = A[sym9(k, k + 1)];
    C9_UNROLL
    for (int i = 1; i < n; ++i) x2 += A[sym9(k, k + 1 + i)] * A[sym9(k, k + 1 + i)];
    const bool any = x2 > Eps<R>::v * Eps<R>::v * R(1e-4); // else column k is as good as tridiagonal
    const R len = C9F(sqrt)(x0 * x0 + x2);
    const R alpha = any ? (x0 > R(0) ? -len : len) : x0;
    const R sc_k = any ? c9_rsqrt(len * (len + C9F(fabs)(x0))) : R(0);
    d[k] = A[sym9(k, k)];
    e[k] = alpha;
    u[0] = (x0 - alpha) * sc_k;
    C9_UNROLL
    for (int i = 1; i < n; ++i) u[i] = A[sym9(k, k + 1 + i)] * sc_k;
    R dot = 0;
    C9_UNROLL
    for (int i = 0; i < n; ++i) {
        R p = 0;
        C9_UNROLL
        for (int j = 0; j < n; ++j) p += A[sym9(k + 1 + i, k + 1 + j)] * u[j];
        w[i] = p;
        dot += p * u[i];
    }
    const R half = R(0.5) * dot;
    constexpr int at = 8 * k - (k * (k - 1)) / 2; // 0, 8, 15, 21, 26, 30, 33
    C9_UNROLL
    for (int i = 0; i < n; ++i) {
        w[i] -= half * u[i];
        sc[at + i] = u[i];
    }
    C9_UNROLL
    for (int i = 0; i < n; ++i)
        C9_UNROLL
        for (int j = i; j < n; ++j) A[sym9(k + 1 + i, k + 1 + j)] -= u[i] * w[j] + w[i] * u[j];
    if constexpr (k < 6) tri9_reduce<k + 1>(A, d, e, sc);
}

// v <- H_0 ... H_r v.
template <int r, typename R> LPG_C9 void tri9_back(const R* sc, R (&v)[9]) {
    constexpr int n = 8 - r, at = 8 * r - (r * (r - 1)) / 2;
    R g = 0;
    C9_UNROLL
    for (int i = 0; i < n; ++i) g += sc[at + i] * v[r + 1 + i];
    C9_UNROLL
    for (int i = 0; i < n; ++i) v[r + 1 + i] -= g * sc[at + i];
    if constexpr (r > 0) tri9_back<r - 1>(sc, v);
}

// The clamp of the packed upper triangle A (45 values). Returns 0: not accurate, A is spent; 1: A holds P with
// M+ = M + P; 2: A holds M+. sc is kTri9Scratch values of scratch.
template <typename R> LPG_C9 int tri9_clamp(R (&A)[45], R* sc) {
    R amax = 0;
    C9_UNROLL
    for (int t = 0; t < 45; ++t) amax = C9F(fmax)(amax, C9F(fabs)(A[t]));
    // Exact power-of-two scaling to max |entry| in [0.5, 1).
    int ex = 0;
    if (amax > R(0) && amax < R(INFINITY)) C9F(frexp)(amax, &ex);
    const R down = C9F(ldexp)(R(1), -ex), up = C9F(ldexp)(R(1), ex);
    C9_UNROLL
    for (int t = 0; t < 45; ++t) A[t] *= down;
    R d[9], e[8];
    tri9_reduce<0>(A, d, e, sc);
    d[7] = A[sym9(7, 7)];
    d[8] = A[sym9(8, 8)];
    e[7] = A[sym9(7, 8)];
    // Gershgorin's bound of |eigenvalue|, the inertia.
    R nrm = 0;
    double d64[9], e64[8];
    float d32[9], e32[8];
    C9_UNROLL
    for (int i = 0; i < 9; ++i) {
        nrm = C9F(fmax)(nrm, C9F(fabs)(d[i]) + (i > 0 ? C9F(fabs)(e[i - 1]) : R(0)) + (i < 8 ? C9F(fabs)(e[i]) : R(0)));
        d64[i] = d[i];
        d32[i] = static_cast<float>(d[i]);
        if (i < 8) {
            e64[i] = static_cast<double>(e[i]) * e[i];
            e32[i] = static_cast<float>(e64[i]);
        }
    }
    const double tol = (sizeof(R) == 8 ? 24.0 : 8.0) * Eps<R>::v * nrm; // eigenvalues this near zero count as zero
    const int nneg = tri9_count(d64, e64, -tol), npos = 9 - tri9_count(d64, e64, tol);
    const bool neg = nneg <= npos;
    const int k = neg ? nneg : npos;
    const R done = R(sizeof(R) == 8 ? 12 : 8) * Eps<R>::v * nrm; // a residual at round-off
    C9_LOOP
    for (int c = 0; c < k; ++c) {
        float lo = neg ? -1.0001f * static_cast<float>(nrm) : 0.f, hi = neg ? 0.f : 1.0001f * static_cast<float>(nrm);
        const int idx = neg ? c : 9 - k + c;
        C9_LOOP
        for (int it = 0; it < 23; ++it) {
            const float mid = 0.5f * (lo + hi);
            if (tri9_count_near(d32, e32, mid) > idx)
                hi = mid;
            else
                lo = mid;
        }
        R s = static_cast<R>(0.5f * (lo + hi)), x[9];
        bool good = false;
        // A second attempt, and one near zero, where FP32 does not tell eigenvalues apart, starts from FP64.
        C9_LOOP
        for (int attempt = sizeof(R) == 8 && C9F(fabs)(s) < R(1e-5) * nrm ? 1 : 0; attempt < 2 && !good; ++attempt) {
            R around = R(4e-6) * nrm;
            if (attempt > 0) {
                double l64 = lo - 2e-6 * nrm, h64 = hi + 2e-6 * nrm;
                C9_LOOP
                for (int it = 0; it < 20; ++it) {
                    const double mid = 0.5 * (l64 + h64);
                    if (tri9_count(d64, e64, mid) > idx)
                        h64 = mid;
                    else
                        l64 = mid;
                }
                s = static_cast<R>(0.5 * (l64 + h64));
                if (sizeof(R) == 8) around = R(1e-10) * nrm;
            }
            const R near = s;
            // A start of mixed signs and sizes, another for each vector and attempt.
            C9_UNROLL
            for (int i = 0; i < 9; ++i) {
                const unsigned h = (static_cast<unsigned>(36 * attempt + 9 * c + i) + 1u) * 2654435761u;
                const R v = R(0.5) + R(h >> 16) * R(0x1p-17);
                x[i] = (h & 0x8000u) ? -v : v;
            }
            C9_LOOP
            for (int it = 0; it < 8 && !good; ++it) {
                tri9_solve(d, e, s, x);
                for (int t = 0; t < c; ++t) { // orthogonal to the vectors before
                    const R* y = &sc[35 + 9 * t];
                    R g = 0;
                    C9_UNROLL
                    for (int i = 0; i < 9; ++i) g += x[i] * y[i];
                    C9_UNROLL
                    for (int i = 0; i < 9; ++i) x[i] -= g * y[i];
                }
                R nn = 0;
                C9_UNROLL
                for (int i = 0; i < 9; ++i) nn += x[i] * x[i];
                const R rn = c9_rsqrt(nn);
                R q = 0, res = 0, tx[9];
                C9_UNROLL
                for (int i = 0; i < 9; ++i) x[i] *= rn;
                C9_UNROLL
                for (int i = 0; i < 9; ++i) {
                    tx[i] = d[i] * x[i] + (i > 0 ? e[i - 1] * x[i - 1] : R(0)) + (i < 8 ? e[i] * x[i + 1] : R(0));
                    q += x[i] * tx[i];
                }
                C9_UNROLL
                for (int i = 0; i < 9; ++i) res += (tx[i] - q * x[i]) * (tx[i] - q * x[i]);
                // A quotient that has left the shift's surroundings is another eigenvalue's: the shift again.
                s = C9F(fabs)(q - near) <= around ? q : near;
                good = s == q && res <= (it < 4 ? R(1) : R(9)) * done * done; // rarely, it stays just above
            }
            // Orthogonal once more: beside a vector of the same cluster the first pass leaves round-off times
            // the amplification of the solve.
            for (int t = 0; t < c; ++t) {
                const R* y = &sc[35 + 9 * t];
                R g = 0;
                C9_UNROLL
                for (int i = 0; i < 9; ++i) g += x[i] * y[i];
                good = good && C9F(fabs)(g) <= R(16) * Eps<R>::v;
            }
        }
        if (!good || !((neg ? -s : s) > R(0.5 * tol))) return 0;
        C9_UNROLL
        for (int i = 0; i < 9; ++i) sc[35 + 9 * c + i] = x[i];
        sc[71 + c] = C9F(fabs)(s);
    }
    C9_UNROLL
    for (int t = 0; t < 45; ++t) A[t] = R(0);
    C9_LOOP
    for (int c = 0; c < k; ++c) {
        R v[9];
        C9_UNROLL
        for (int i = 0; i < 9; ++i) v[i] = sc[35 + 9 * c + i];
        tri9_back<6>(sc, v);
        const R lam = sc[71 + c] * up;
        C9_UNROLL
        for (int r = 0; r < 9; ++r) {
            const R lr = lam * v[r];
            C9_UNROLL
            for (int q = r; q < 9; ++q) A[sym9(r, q)] += lr * v[q];
        }
    }
    return neg ? 1 : 2;
}

} // namespace lpg
