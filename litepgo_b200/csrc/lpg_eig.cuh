// lpg_eig.cuh -- device code of the PSD projections of dense symmetric element Hessians (24 x 24 Q1
// hexes, one warp per element; 192 x 192 Hermite hexes, one block per element): what
// HessianKind::Projected asks for, V max(L, 0) V^T (mesh_energy.cpp:16-27, there by Eigen's
// SelfAdjointEigenSolver).
//
// Only the eigenpairs of one sign are needed: H+ = H + sum_{L_m < 0} |L_m| v_m v_m^T, or the sum over the
// positive ones where they are fewer, so at most N / 2 of them:
//   1. Householder tridiagonalisation (Golub & Van Loan, Matrix Computations, 8.3.1), reflectors kept;
//   2. the inertia and the wanted eigenvalues by Sturm counts (Givens' bisection; Wilkinson, The Algebraic
//      Eigenvalue Problem, 5.39), several points per eigenvalue and pass;
//   3. their eigenvectors by inverse iteration with the pivoted LU factors of T - lambda I (Wilkinson
//      5.54) from seeded starts, then modified Gram-Schmidt, twice. The solves leave the vectors of a multiple
//      eigenvalue almost parallel (they grow the most along one of its directions), and Gram-Schmidt then
//      magnifies the residual of what is left; such vectors are solved and orthogonalised again, up to
//      `rounds` times, until every residual of T x - lambda x is at round-off. Distinct eigenvalues take one
//      round, a 12-fold one at most three;
//   4. the reflectors applied to them, and the rank-k update.
// A matrix that is still off then goes to the Jacobi method. Orthonormal vectors with residuals at round-off
// for as many eigenvalues of one sign as the Sturm counts say there are span their eigenspace.
#pragma once

#include <cstdint>

#include "lpg_psd.h"

namespace lpg {

constexpr double kEigEps = 2.220446049250313e-16;
constexpr double kEigResidual = 1e-13; // accepted residual of an eigenvector, relative to the norm's bound

// Seeded start of an inverse iteration: entry i of vector c, +-[0.5, 1) (SplitMix64 finaliser).
__device__ __forceinline__ double eig_start(int i, int c) {
    unsigned long long z = (static_cast<unsigned long long>(c) << 32) + static_cast<unsigned>(i) + 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    z ^= z >> 31;
    const double u = 0.5 + static_cast<double>(z >> 12) * 0x1.0p-53;
    return (z & 1) ? -u : u;
}

// Eigenvalues of the n x n tridiagonal matrix (d, off-diagonals squared e2) below x, by the signs of the
// leading principal minors p_i = (d_i - x) p_{i-1} - e2_{i-1} p_{i-2}: no division in the chain, one
// dependent FMA per row. The matrix's entries are below 1, so |d| and |e| below N, and both terms of the
// pair are rescaled by a power of two every 8 rows.
template <int N> __device__ __forceinline__ int sturm_count(const double* d, const double* e2, double x) {
    double p2 = 1.0, p1 = d[0] - x;
    if (p1 == 0.0) p1 = -1e-30;
    int cnt = p1 < 0.0;
#pragma unroll 8
    for (int i = 1; i < N; ++i) {
        double p = fma(d[i] - x, p1, -(e2[i - 1] * p2));
        if (p == 0.0) p = -1e-30 * p1;
        cnt += (__double2hiint(p) ^ __double2hiint(p1)) < 0;
        p2 = p1;
        p1 = p;
        if ((i & 7) == 0) {
            // 2^-k with k the exponent of the larger of the two.
            const int h = max(__double2hiint(p1) & 0x7ff00000, __double2hiint(p2) & 0x7ff00000);
            const double s = __hiloint2double(0x7fe00000 - h, 0);
            p1 *= s;
            p2 *= s;
        }
    }
    return cnt;
}

// ---------------------------------------------------------------------------
// One warp, N <= 32: lane j holds column j of the matrix.
// ---------------------------------------------------------------------------
template <int N> struct WarpEig {
    static constexpr int K = N / 2; // most eigenpairs taken
    static constexpr int S = N + 1; // row stride of the staged matrix
    // Per-warp shared memory, in doubles. M is the staged matrix, then the LU factors, then the result;
    // the Jacobi iteration uses M and V | Z as its two matrices.
    double M[N * S];
    double V[N * N];     // reflector k at V + N k (entries i > k)
    double Z[K * N];     // eigenvectors, one per row
    double d[N], e[N], e2[N], beta[N], w[N];
    static_assert(2 * K * N <= N * S, "the LU factors fit the staged matrix");
    static_assert(N * S <= N * N + K * N, "Jacobi's eigenvectors fit V and Z");

    static __device__ __forceinline__ double sum(double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        return x;
    }

    // The projection of M (both triangles staged, scaled to max |entry| < 1): on return M holds P with
    // M+ = M_in + P (the return value 1) or M+ = P (2); 0: M is semi-definite (unchanged M+ = M_in);
    // -1: not accurate after the given rounds, the caller falls back. A team of 32 lanes, all converged.
    __device__ int project(int lane, int rounds) {
        const bool own = lane < N;
        {
            double a[N];
#pragma unroll
            for (int i = 0; i < N; ++i) a[i] = own ? M[i * S + lane] : 0.0;
            // Step k maps column k below the diagonal to (alpha, 0, ...) with I - beta v v^T.
#pragma unroll
            for (int k = 0; k < N - 2; ++k) {
                const double x = (own && lane > k) ? a[k] : 0.0; // A(k, lane) = A(lane, k)
                const double x2 = sum(lane == k + 1 ? 0.0 : x * x);
                const double x0 = __shfl_sync(0xffffffffu, x, k + 1);
                if (x2 <= 1e-40) { // nothing below the subdiagonal (of a matrix of entries near 1)
                    if (lane == 0) beta[k] = 0.0, e[k] = x0;
                    continue;
                }
                const double alpha = -copysign(sqrt(fma(x0, x0, x2)), x0);
                const double bk = 1.0 / (alpha * (alpha - x0)); // 2 / v^T v
                const double v = lane == k + 1 ? x0 - alpha : x;
                if (own) V[N * k + lane] = v;
                if (lane == 0) beta[k] = bk, e[k] = alpha;
                __syncwarp();
                double p0 = 0, p1 = 0;
#pragma unroll
                for (int i = k + 1; i < N; i += 2) {
                    p0 = fma(a[i], V[N * k + i], p0);
                    if (i + 1 < N) p1 = fma(a[i + 1], V[N * k + i + 1], p1);
                }
                const double p = lane > k ? bk * (p0 + p1) : 0.0;
                const double kk = 0.5 * bk * sum(p * v);
                const double wj = fma(-kk, v, p);
                if (own) w[lane] = wj;
                __syncwarp();
#pragma unroll
                for (int i = k + 1; i < N; ++i) a[i] -= fma(V[N * k + i], wj, w[i] * v);
                __syncwarp();
            }
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (lane == i) d[i] = a[i];
            if (lane == N - 2) e[N - 2] = a[N - 1];
        }
        __syncwarp();
        if (own) e2[lane] = lane < N - 1 ? e[lane] * e[lane] : 0.0;
        // Gershgorin's bound of |eigenvalue|.
        double nrm = own ? fabs(d[lane]) + (lane > 0 ? fabs(e[lane - 1]) : 0.0) + (lane < N - 1 ? fabs(e[lane]) : 0.0) : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
        __syncwarp();
        const double tol = 8 * kEigEps * nrm; // eigenvalues this near zero count as zero
        const int c2 = sturm_count<N>(d, e2, (lane & 1) ? tol : -tol);
        const int nneg = __shfl_sync(0xffffffffu, c2, 0), npos = N - __shfl_sync(0xffffffffu, c2, 1);
        const bool neg = nneg <= npos;
        const int k = neg ? nneg : npos;
        if (k == 0) {
            if (neg) return 0;
            for (int t = lane; t < N * S; t += 32) M[t] = 0.0; // no positive eigenvalue
            __syncwarp();
            return 2;
        }
        // Eigenvalue c = lane / ways by multisection: `ways` interior points per pass.
        const int ways = 32 / k, c = lane / ways, sub = lane - ways * c;
        double lo = neg ? -1.0000001 * nrm : 0.0, hi = neg ? 0.0 : 1.0000001 * nrm;
        const int idx = neg ? c : N - k + c;
        const double inv = 1.0 / (ways + 1);
        const unsigned mask = ways == 32 ? 0xffffffffu : (1u << ways) - 1u;
        double width = hi - lo;
        for (int it = 0; it < 60 && width > 2 * kEigEps * nrm; ++it, width *= inv) {
            const double step = (hi - lo) * inv;
            const double x = fma(step, sub + 1, lo);
            const bool above = c < k && sturm_count<N>(d, e2, x) > idx; // eigenvalue idx lies below x
            const unsigned b = __ballot_sync(0xffffffffu, above);
            const unsigned g = c < k ? (b >> (ways * c)) & mask : 0u;
            const int first = g ? __ffs(g) - 1 : ways;
            const double l0 = lo;
            if (first < ways) hi = fma(step, first + 1, l0);
            if (first > 0) lo = fma(step, first, l0);
        }
        // Lane c < k takes eigenvalue c and its vector.
        const double lam = __shfl_sync(0xffffffffu, 0.5 * (lo + hi), (lane * ways) & 31);
        const bool vec = lane < k;
        double x[N];
        unsigned sw = 0;
        double* f0 = M + lane;
        double* f1 = M + K * N + lane;
        if (vec) {
            // LU of T - lam I with row exchanges. Row i keeps 1 / pivot in f0 and in f1 the second
            // entry b of the row, or, where rows i and i + 1 were exchanged (bit i of sw), the entry a
            // that the exchange moved down (the pivot row is then T's row i + 1).
            double a = d[0] - lam, b = e[0];
            const double tiny = kEigEps * nrm;
#pragma unroll 4
            for (int i = 0; i < N - 1; ++i) {
                const double sb = e[i], dn = d[i + 1] - lam, sn = i + 2 < N ? e[i + 1] : 0.0;
                if (fabs(a) >= fabs(sb)) {
                    if (fabs(a) < tiny) a = copysign(tiny, a);
                    const double r = 1.0 / a;
                    f0[K * i] = r;
                    f1[K * i] = b;
                    a = fma(-(sb * r), b, dn);
                    b = sn;
                } else {
                    const double r = 1.0 / sb, l = a * r;
                    sw |= 1u << i;
                    f0[K * i] = r;
                    f1[K * i] = a;
                    a = fma(-l, dn, b);
                    b = -l * sn;
                }
            }
            if (fabs(a) < tiny) a = copysign(tiny, a);
            f0[K * (N - 1)] = 1.0 / a;
        }
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = vec ? eig_start(i, lane) : 0.0;
        bool bad = true;
#pragma unroll 1
        for (int round = 0; bad && round < rounds; ++round) {
            if (vec) {
#pragma unroll 1
                for (int it = round == 0 ? 0 : 1; it < 2; ++it) { // the first solve has no forward pass
                    if (it > 0) {
#pragma unroll
                        for (int i = 0; i < N - 1; ++i) {
                            if ((sw >> i) & 1u) {
                                const double t = x[i];
                                x[i] = x[i + 1];
                                x[i + 1] = fma(-(f1[K * i] * f0[K * i]), x[i], t);
                            } else {
                                x[i + 1] = fma(-(e[i] * f0[K * i]), x[i], x[i + 1]);
                            }
                        }
                    }
#pragma unroll
                    for (int i = N - 1; i >= 0; --i) {
                        double s = x[i];
                        if (i + 1 < N) {
                            const bool ex = (sw >> i) & 1u;
                            s = fma(-(ex ? d[i + 1] - lam : f1[K * i]), x[i + 1], s);
                            if (i + 2 < N && ex) s = fma(-e[i + 1], x[i + 2], s);
                        }
                        x[i] = s * f0[K * i];
                    }
                    double big = 0;
#pragma unroll
                    for (int i = 0; i < N; ++i) big = fmax(big, fabs(x[i]));
                    const double sc = 1.0 / big;
                    double q = 0;
#pragma unroll
                    for (int i = 0; i < N; ++i) {
                        x[i] *= sc;
                        q = fma(x[i], x[i], q);
                    }
                    const double r = rsqrt(q);
#pragma unroll
                    for (int i = 0; i < N; ++i) x[i] *= r;
                }
            }
            // Modified Gram-Schmidt over the lanes, twice.
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass)
#pragma unroll 1
                for (int m = 0; m < k; ++m) {
                    if (lane == m) {
                        double q = 0;
#pragma unroll
                        for (int i = 0; i < N; ++i) q = fma(x[i], x[i], q);
                        const double r = rsqrt(q);
#pragma unroll
                        for (int i = 0; i < N; ++i) {
                            x[i] *= r;
                            Z[N * m + i] = x[i];
                        }
                    }
                    __syncwarp();
                    if (vec && lane > m) {
                        double q0 = 0, q1 = 0;
#pragma unroll
                        for (int i = 0; i < N; i += 2) {
                            q0 = fma(Z[N * m + i], x[i], q0);
                            if (i + 1 < N) q1 = fma(Z[N * m + i + 1], x[i + 1], q1);
                        }
                        const double q = q0 + q1;
#pragma unroll
                        for (int i = 0; i < N; ++i) x[i] = fma(-q, Z[N * m + i], x[i]);
                    }
                    __syncwarp();
                }
            // The residuals of what Gram-Schmidt left.
            bool off = false;
            if (vec) {
#pragma unroll
                for (int i = 0; i < N; ++i) {
                    double t = (d[i] - lam) * x[i];
                    if (i > 0) t = fma(e[i - 1], x[i - 1], t);
                    if (i + 1 < N) t = fma(e[i], x[i + 1], t);
                    off = off || !(fabs(t) <= kEigResidual * nrm);
                }
            }
            bad = __any_sync(0xffffffffu, off);
        }
        if (bad) return -1;
        // Eigenvectors of the matrix: the reflectors from the last to the first, then scaled by
        // sqrt |lambda| (the update's terms are then products of two equal factors: bitwise symmetric).
        if (vec) {
#pragma unroll
            for (int q = N - 3; q >= 0; --q) {
                const double bq = beta[q];
                if (bq == 0.0) continue;
                double s0 = 0, s1 = 0;
#pragma unroll
                for (int i = q + 1; i < N; i += 2) {
                    s0 = fma(V[N * q + i], x[i], s0);
                    if (i + 1 < N) s1 = fma(V[N * q + i + 1], x[i + 1], s1);
                }
                const double f = bq * (s0 + s1);
#pragma unroll
                for (int i = q + 1; i < N; ++i) x[i] = fma(-f, V[N * q + i], x[i]);
            }
            const double r = sqrt(fabs(lam));
#pragma unroll
            for (int i = 0; i < N; ++i) Z[N * lane + i] = r * x[i];
        }
        __syncwarp();
        // The rank-k update, column per lane.
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] = 0.0;
        if (own) {
#pragma unroll 1
            for (int m = 0; m < k; ++m) {
                const double z = Z[N * m + lane];
#pragma unroll
                for (int i = 0; i < N; ++i) x[i] = fma(Z[N * m + i], z, x[i]);
            }
#pragma unroll
            for (int i = 0; i < N; ++i) M[i * S + lane] = x[i];
        }
        __syncwarp();
        return neg ? 1 : 2;
    }
};

// ---------------------------------------------------------------------------
// One block, N = 192 (tricubic Hermite elements): the lower triangle packed in shared memory, the LU
// factors and the inverse iteration's vectors in global scratch (kScratch doubles, resident in L2).
// ---------------------------------------------------------------------------
struct BlockEig {
    static constexpr int N = 192, K = N / 2;
    static constexpr int kThreads = 512, kWarps = kThreads / 32, kT = N / 32;
    static constexpr int kPacked = N * (N + 1) / 2;
    static constexpr int kStride = N + 1; // of an eigenvector in shared memory: K rows fill the triangle
    static constexpr size_t kScratch = 3 * static_cast<size_t>(N) * K;
    static_assert(N * N <= static_cast<int>(kScratch), "Jacobi's eigenvectors fit the scratch");
    static_assert(3 * K <= kWarps * N, "Jacobi's rotations fit the partial sums");
    static_assert(K * kStride <= kPacked, "the eigenvectors fit the matrix");
    double A[kPacked];       // lower triangle: row r at r (r + 1) / 2; then reflectors; then eigenvectors
    double part[kWarps * N]; // partial sums
    double v[2][N], w[N], y[N];
    double d[N], e[N], e2[N], beta[N], lam[K];
    double red[kWarps];
    unsigned sw[kT][K];
    int nneg, npos;

    static __device__ __forceinline__ int at(int r, int c) { return r * (r + 1) / 2 + c; } // r >= c

    // Block-wide sum, the same to every thread, in a fixed order; one barrier before the result and the
    // caller's next barrier before the next sum.
    __device__ __forceinline__ double sum(double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
        __syncthreads();
        double t = 0;
#pragma unroll
        for (int q = 0; q < kWarps; ++q) t += red[q];
        return t;
    }

    // Householder tridiagonalisation of A into (d, e); reflector k stays in column k below the diagonal.
    // Step k's rank-2 update of the trailing matrix and step k + 1's product with it are one pass.
    __device__ void tridiagonal() {
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        if (tid < N) v[1][tid] = w[tid] = 0.0;
        __syncthreads();
        for (int k = 0; k < N - 2; ++k) {
            const double* vo = v[(k & 1) ^ 1]; // the previous reflector (zero before the first)
            double* vn = v[k & 1];
            double x = 0;
            if (tid < N && tid >= k) {
                x = A[at(tid, k)] - fma(vo[tid], w[k], w[tid] * vo[k]);
                if (tid == k) {
                    d[k] = x;
                    x = 0;
                }
                if (tid == k + 1) y[0] = x;
            }
            const double x2 = sum(tid == k + 1 ? 0.0 : x * x);
            const double x0 = y[0];
            double alpha = x0, bk = 0;
            const bool flat = x2 <= 1e-40; // nothing below the subdiagonal (of a matrix of entries near 1)
            if (!flat) {
                alpha = -copysign(sqrt(fma(x0, x0, x2)), x0);
                bk = 1.0 / (alpha * (alpha - x0)); // 2 / v^T v
            }
            if (tid < N) {
                const double nv = flat || tid <= k ? 0.0 : tid == k + 1 ? x0 - alpha : x;
                vn[tid] = nv;
                if (tid > k) A[at(tid, k)] = nv;
            }
            if (tid == 0) {
                e[k] = alpha;
                beta[k] = bk;
            }
            __syncthreads();
            // Rows k + 1 .. N - 1 over the warps, columns over the lanes: update, store, and accumulate
            // A v (the row's part by shuffles, the transposed part per lane).
            double vj[kT], wj[kT], nj[kT], col[kT];
#pragma unroll
            for (int t = 0; t < kT; ++t) {
                const int j = 32 * t + lane;
                vj[t] = vo[j], wj[t] = w[j], nj[t] = vn[j], col[t] = 0;
            }
            for (int i = k + 1 + warp; i < N; i += kWarps) {
                const double vi = vo[i], wi = w[i], ni = vn[i];
                double row = 0;
                double* Ai = A + at(i, 0);
#pragma unroll
                for (int t = 0; t < kT; ++t) {
                    if (32 * t + 31 <= k || 32 * t > i) continue; // the same for the whole warp
                    const int j = 32 * t + lane;
                    if (j > k && j <= i) {
                        const double a = Ai[j] - fma(vi, wj[t], wi * vj[t]);
                        Ai[j] = a;
                        row = fma(a, nj[t], row);
                        if (j < i) col[t] = fma(a, ni, col[t]);
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) row += __shfl_xor_sync(0xffffffffu, row, o);
                if (lane == 0) y[i] = row;
            }
#pragma unroll
            for (int t = 0; t < kT; ++t) part[N * warp + 32 * t + lane] = col[t];
            __syncthreads();
            double p = 0;
            if (tid < N && tid > k) {
                double q[4] = {y[tid], 0, 0, 0};
#pragma unroll
                for (int g = 0; g < kWarps; ++g) q[g & 3] += part[N * g + tid];
                p = bk * ((q[0] + q[1]) + (q[2] + q[3]));
            }
            const double nv = tid < N ? vn[tid] : 0.0;
            const double kk = 0.5 * bk * sum(p * nv);
            if (tid < N) w[tid] = fma(-kk, nv, p);
            __syncthreads();
        }
        if (tid == 0) {
            const double* vo = v[(N - 3) & 1];
            d[N - 2] = A[at(N - 2, N - 2)] - 2 * vo[N - 2] * w[N - 2];
            d[N - 1] = A[at(N - 1, N - 1)] - 2 * vo[N - 1] * w[N - 1];
            e[N - 2] = A[at(N - 1, N - 2)] - fma(vo[N - 1], w[N - 2], w[N - 1] * vo[N - 2]);
            e[N - 1] = 0;
        }
        __syncthreads();
    }

    // LU of T - lambda_c I for eigenvector c < k by thread c.
    __device__ void factor(int c, double nrm, double* f0, double* f1) {
        const double lm = lam[c], tiny = kEigEps * nrm;
        double a = d[0] - lm, b = e[0];
        unsigned bits = 0;
#pragma unroll 4
        for (int i = 0; i < N - 1; ++i) { // rows as in WarpEig::project
            const double sb = e[i], dn = d[i + 1] - lm, sn = e[i + 1];
            double r, s;
            if (fabs(a) >= fabs(sb)) {
                if (fabs(a) < tiny) a = copysign(tiny, a);
                r = 1.0 / a;
                s = b;
                a = fma(-(sb * r), b, dn);
                b = sn;
            } else {
                r = 1.0 / sb;
                s = a;
                const double l = a * r;
                bits |= 1u << (i & 31);
                a = fma(-l, dn, b);
                b = -l * sn;
            }
            f0[K * i + c] = r;
            f1[K * i + c] = s;
            if ((i & 31) == 31) {
                sw[i >> 5][c] = bits;
                bits = 0;
            }
        }
        sw[kT - 1][c] = bits;
        if (fabs(a) < tiny) a = copysign(tiny, a);
        f0[K * (N - 1) + c] = 1.0 / a;
        f1[K * (N - 1) + c] = 0;
    }

    // Inverse iteration for eigenvector c < k by thread c: two solves from a seeded start (the first without
    // its forward pass), or one from the vector at X[K i + c], which the result replaces. Returns the
    // inverse of its 2-norm.
    __device__ double inverse_iteration(int c, bool first, const double* f0, const double* f1, double* X) {
        const double lm = lam[c];
        double scale = 1.0;
        constexpr int U = 8; // rows loaded ahead of the chain
        for (int it = first ? 0 : 1; it < 2; ++it) {
            if (it > 0) {
                double x = scale * X[c];
                for (int i0 = 0; i0 < N - 1; i0 += U) {
                    double g0[U], g1[U], xn[U];
#pragma unroll
                    for (int j = 0; j < U; ++j)
                        if (i0 + j < N - 1) g0[j] = f0[K * (i0 + j) + c], g1[j] = f1[K * (i0 + j) + c], xn[j] = X[K * (i0 + j + 1) + c];
                    const unsigned word = sw[i0 >> 5][c];
#pragma unroll
                    for (int j = 0; j < U; ++j) {
                        const int i = i0 + j;
                        if (i >= N - 1) break;
                        double nx = scale * xn[j];
                        if ((word >> (i & 31)) & 1u) {
                            const double t = x;
                            x = nx;
                            nx = fma(-(g1[j] * g0[j]), x, t);
                        } else {
                            nx = fma(-(e[i] * g0[j]), x, nx);
                        }
                        X[K * i + c] = x;
                        x = nx;
                    }
                }
                X[K * (N - 1) + c] = x;
            }
            double x1 = 0, x2 = 0, q = 0;
            for (int i0 = N - U; i0 >= 0; i0 -= U) {
                double g0[U], g1[U], xv[U];
#pragma unroll
                for (int j = U - 1; j >= 0; --j) {
                    g0[j] = f0[K * (i0 + j) + c], g1[j] = f1[K * (i0 + j) + c];
                    xv[j] = it == 0 ? eig_start(i0 + j, c) : X[K * (i0 + j) + c];
                }
                const unsigned word = sw[i0 >> 5][c];
#pragma unroll
                for (int j = U - 1; j >= 0; --j) {
                    const int i = i0 + j;
                    const bool ex = (word >> (i & 31)) & 1u;
                    const double dn = i + 1 < N ? d[i + 1] - lm : 0.0, sn = i + 1 < N ? e[i + 1] : 0.0;
                    double s = fma(-(ex ? dn : g1[j]), x1, xv[j]);
                    if (ex) s = fma(-sn, x2, s);
                    s *= g0[j];
                    q = fma(s, s, q);
                    X[K * i + c] = s;
                    x2 = x1;
                    x1 = s;
                }
            }
            scale = rsqrt(q);
        }
        return scale;
    }

    // Modified Gram-Schmidt, twice, over the k vectors of X times their factors in y, a column per half warp and
    // in registers (three columns a lane: half the shuffles and global sectors of a column per warp); the
    // reflectors stay in A. Returns whether a residual is above round-off.
    __device__ bool orthonormalise(int k, double nrm, double* X) {
        static_assert(K % (2 * kWarps) == 0, "columns per half warp");
        constexpr int J = K / (2 * kWarps), kH = N / 16;
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, l = lane & 15;
        double z[J][kH];
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int c = 2 * (warp + kWarps * j) + half;
            const double s = c < k ? y[c] : 0.0;
#pragma unroll
            for (int t = 0; t < kH; ++t) z[j][t] = c < k ? s * X[K * (16 * t + l) + c] : 0.0;
        }
        int off = 0;
#pragma unroll 1
        for (int pass = 0; pass < 2; ++pass)
#pragma unroll 1
            for (int m = 0; m < k; ++m) {
                double* u = v[m & 1]; // two buffers: one barrier per vector
                const bool mine = warp == ((m >> 1) & (kWarps - 1));
                if (mine)
#pragma unroll
                    for (int j = 0; j < J; ++j)
                        if (j == m / (2 * kWarps)) {
                            double q = 0;
#pragma unroll
                            for (int t = 0; t < kH; ++t) q = fma(z[j][t], z[j][t], q);
#pragma unroll
                            for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                            const double r = rsqrt(q);
                            if (half == (m & 1))
#pragma unroll
                                for (int t = 0; t < kH; ++t) {
                                    z[j][t] *= r;
                                    u[16 * t + l] = z[j][t];
                                }
                        }
                __syncthreads();
#pragma unroll
                for (int j = 0; j < J; ++j) {
                    const int c0 = 2 * (warp + kWarps * j), c = c0 + half;
                    if (c0 + 1 <= m || c0 >= k) continue; // the same for the whole warp
                    double q = 0;
#pragma unroll
                    for (int t = 0; t < kH; ++t) q = fma(u[16 * t + l], z[j][t], q);
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                    if (c > m)
#pragma unroll
                        for (int t = 0; t < kH; ++t) z[j][t] = fma(-q, u[16 * t + l], z[j][t]);
                }
                if (pass > 0 && mine) {
#pragma unroll
                    for (int t = 0; t < kT; ++t) {
                        const int i = 32 * t + lane;
                        double res = (d[i] - lam[m]) * u[i];
                        if (i > 0) res = fma(e[i - 1], u[i - 1], res);
                        if (i < N - 1) res = fma(e[i], u[i + 1], res);
                        if (!(fabs(res) <= kEigResidual * nrm)) off = 1;
                    }
                }
            }
#pragma unroll
        for (int j = 0; j < J; ++j) {
            const int c = 2 * (warp + kWarps * j) + half;
#pragma unroll
            for (int t = 0; t < kH; ++t)
                if (c < k) X[K * (16 * t + l) + c] = z[j][t];
        }
        return __syncthreads_or(off) != 0; // X is written
    }

    // All eigenpairs of the matrix in A by the cyclic Jacobi method in the round-robin ordering of lpg_psd.h: a
    // round's rotations act on disjoint 2 x 2 blocks of the packed triangle, one thread each. V is N N values
    // of scratch. Leaves what project() does and returns k. Tens of milliseconds; for what inverse iteration
    // does not resolve.
    __device__ __noinline__ int jacobi(double* V, int& kind) {
        using J = PsdJacobi<N>;
        const int tid = threadIdx.x;
        double* cs = part;                                // cosine and sine of each pair
        int* pq = reinterpret_cast<int*>(part + 2 * K); // its indices
        for (int t = tid; t < N * N; t += kThreads) V[t] = t / N == t % N ? 1.0 : 0.0;
        const auto entry = [&](int r, int c) -> double& { return A[r >= c ? at(r, c) : at(c, r)]; };
        for (int sweep = 0; sweep < J::kMaxSweeps; ++sweep) {
            double off = 0, diag = 0;
            for (int t = tid; t < N * N; t += kThreads) {
                const int r = t / N, c = t - N * r;
                if (r > c) off = fma(A[at(r, c)], A[at(r, c)], off);
                if (r == c) diag = fma(A[at(r, r)], A[at(r, r)], diag);
            }
            off = 2 * sum(off);
            __syncthreads();
            diag = sum(diag);
            if (!(off > J::kOffTol2 * (off + diag))) break;
            for (int round = 0; round < J::kRounds; ++round) {
                if (tid < K) {
                    int p, q;
                    J::pair(round, tid, p, q);
                    jacobi_rotation(entry(p, p), entry(q, q), entry(p, q), cs[2 * tid], cs[2 * tid + 1]);
                    pq[2 * tid] = p;
                    pq[2 * tid + 1] = q;
                }
                __syncthreads();
                for (int t = tid; t < K * K; t += kThreads) {
                    const int i = t / K, j = t - K * i;
                    if (j < i) continue;
                    const int p = pq[2 * i], q = pq[2 * i + 1], pp = pq[2 * j], qq = pq[2 * j + 1];
                    const double c = cs[2 * i], s = cs[2 * i + 1], c2 = cs[2 * j], s2 = cs[2 * j + 1];
                    const double b00 = entry(p, pp), b01 = entry(p, qq), b10 = entry(q, pp), b11 = entry(q, qq);
                    const double x0 = c2 * b00 - s2 * b01, x1 = s2 * b00 + c2 * b01; // the columns' rotation
                    const double y0 = c2 * b10 - s2 * b11, y1 = s2 * b10 + c2 * b11;
                    entry(p, pp) = c * x0 - s * y0;
                    entry(q, qq) = s * x1 + c * y1;
                    entry(q, pp) = i == j ? 0.0 : s * x0 + c * y0;
                    if (i != j) entry(p, qq) = c * x1 - s * y1;
                }
                for (int t = tid; t < N * K; t += kThreads) {
                    const int i = t / K, j = t - K * i;
                    double &a = V[N * i + pq[2 * j]], &b = V[N * i + pq[2 * j + 1]];
                    const double va = a, vb = b, c = cs[2 * j], s = cs[2 * j + 1];
                    a = c * va - s * vb;
                    b = s * va + c * vb;
                }
                __syncthreads();
            }
        }
        __syncthreads();
        if (tid < N) d[tid] = A[at(tid, tid)];
        __syncthreads();
        if (tid == 0) {
            int n = 0, p = 0;
            for (int m = 0; m < N; ++m) n += d[m] < 0.0, p += d[m] > 0.0;
            nneg = n, npos = p;
            for (int m = 0, c = 0; m < N; ++m)
                if (n <= p ? d[m] < 0.0 : d[m] > 0.0) pq[c++] = m;
        }
        __syncthreads();
        const bool neg = nneg <= npos;
        const int k = neg ? nneg : npos;
        kind = k == 0 ? (neg ? 0 : 2) : (neg ? 1 : 2);
        for (int t = tid; t < k * N; t += kThreads) {
            const int c = t / N, i = t - N * c, m = pq[c];
            A[kStride * c + i] = sqrt(fabs(d[m])) * V[N * i + m];
        }
        __syncthreads();
        return k;
    }

    // The reflectors applied to the k eigenvectors of T (X, times the column's entry of `scales`), which
    // then replace the reflectors in A (vector c at kStride c). Lanes are columns; a column's rows are dealt
    // to P warps (row p, p + P, ...), which add their parts of each product.
    template <int P> __device__ void back_transform(int k, const double* X, const double* scales) {
        constexpr int R = (N + P - 1) / P;
        const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
        const int g = warp / P, p = warp - P * g, c = 32 * g + lane;
        const bool on = g < (kWarps / P) && c < k;
        double x[R];
        const double sc = on ? scales[c] : 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r) x[r] = on && p + P * r < N ? sc * X[K * (p + P * r) + c] : 0.0;
        double* mine = part + 32 * warp + lane;
        int flip = 0; // two buffers: one barrier per reflector
        for (int q = N - 3; q >= 0; --q) {
            const double bq = beta[q];
            if (bq == 0.0) continue;
            flip ^= 32 * kWarps;
            double s0 = 0, s1 = 0;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + P * r;
                if (i > q && i < N) {
                    if (r & 1)
                        s1 = fma(A[at(i, q)], x[r], s1);
                    else
                        s0 = fma(A[at(i, q)], x[r], s0);
                }
            }
            mine[flip] = s0 + s1;
            __syncthreads();
            double s = 0;
            if (g < kWarps / P) {
                const double* all = part + flip + 32 * P * g + lane;
#pragma unroll
                for (int j = 0; j < P; ++j) s += all[32 * j];
            }
            const double f = bq * s;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int i = p + P * r;
                if (i > q && i < N) x[r] = fma(-f, A[at(i, q)], x[r]);
            }
        }
        __syncthreads(); // the reflectors are read
        if (on) {
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (p + P * r < N) A[kStride * c + p + P * r] = x[r];
        }
        __syncthreads();
    }

    // The matrix of an element's record times `down` into A. Block (a, b), a <= b, entry (i, c) of the record is
    // H(3 a + i, 3 b + c): the blocks of a are consecutive.
    __device__ void load(const double* rec, double down) {
        for (int a = threadIdx.x >> 5; a < N / 3; a += kWarps) {
            const double* ra = rec + 9 * (a * (N / 3) - a * (a - 1) / 2);
            for (int t = threadIdx.x & 31; t < 9 * (N / 3 - a); t += 32) {
                const int b = a + t / 9, ic = t - 9 * (t / 9), r = 3 * a + ic / 3, c = 3 * b + ic % 3;
                if (c >= r) A[at(c, r)] = down * ra[t];
            }
        }
        __syncthreads();
    }

    // Projection of the record's matrix times `down` (max |entry| < 1). Returns the number k of vectors
    // z_c = sqrt |lambda_c| v_c left in A (at kStride c) and the kind: 0 the matrix is its own projection,
    // 1 H+ = H + sum z z^T, 2 H+ = sum z z^T.
    __device__ int project(const double* rec, double down, double* scratch, int rounds, int& kind) {
        const int tid = threadIdx.x, lane = tid & 31;
        load(rec, down);
        tridiagonal();
        double nrm = 0;
        for (int i = lane; i < N; i += 32) {
            nrm = fmax(nrm, fabs(d[i]) + (i > 0 ? fabs(e[i - 1]) : 0.0) + fabs(e[i]));
            if (tid < 32) e2[i] = e[i] * e[i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm = fmax(nrm, __shfl_xor_sync(0xffffffffu, nrm, o));
        __syncthreads();
        const double tol = 8 * kEigEps * nrm; // eigenvalues this near zero count as zero
        if (tid < 2) {
            const int n = sturm_count<N>(d, e2, tid ? tol : -tol);
            if (tid)
                npos = N - n;
            else
                nneg = n;
        }
        __syncthreads();
        const bool neg = nneg <= npos;
        const int k = neg ? nneg : npos;
        kind = k == 0 ? (neg ? 0 : 2) : (neg ? 1 : 2);
        if (k == 0) return 0;
        // Eigenvalue c by multisection on 8 (or 4) neighbouring lanes.
        {
            const int lw = k <= kThreads / 8 ? 3 : 2, ways = 1 << lw, c = tid >> lw, sub = tid & (ways - 1);
            double lo = neg ? -1.0000001 * nrm : 0.0, hi = neg ? 0.0 : 1.0000001 * nrm;
            const int idx = neg ? c : N - k + c;
            const double inv = 1.0 / (ways + 1);
            const unsigned mask = (1u << ways) - 1u;
            double width = hi - lo;
            if (32 * (tid >> 5) < (k << lw)) // the same for the whole warp
                for (int it = 0; it < 60 && width > 2 * kEigEps * nrm; ++it, width *= inv) {
                    const double step = (hi - lo) * inv;
                    const bool above = c < k && sturm_count<N>(d, e2, fma(step, sub + 1, lo)) > idx;
                    const unsigned b = __ballot_sync(0xffffffffu, above);
                    const unsigned g = (b >> (lane & ~(ways - 1))) & mask;
                    const int first = g ? __ffs(g) - 1 : ways;
                    const double l0 = lo;
                    if (first < ways) hi = fma(step, first + 1, l0);
                    if (first > 0) lo = fma(step, first, l0);
                }
            if (c < k && sub == 0) lam[c] = 0.5 * (lo + hi);
        }
        __syncthreads();
        double *f0 = scratch, *f1 = scratch + N * K, *X = scratch + 2 * N * K;
        if (tid < k) factor(tid, nrm, f0, f1);
        bool bad = true;
        for (int round = 0; bad && round < rounds; ++round) {
            if (tid < k) y[tid] = inverse_iteration(tid, round == 0, f0, f1, X);
            __syncthreads();
            bad = orthonormalise(k, nrm, X);
        }
        if (bad) {
            load(rec, down);
            return jacobi(scratch, kind);
        }
        if (tid < k) y[tid] = sqrt(fabs(lam[tid]));
        __syncthreads();
        if (k <= 32)
            back_transform<16>(k, X, y);
        else if (k <= 64)
            back_transform<8>(k, X, y);
        else
            back_transform<5>(k, X, y);
        return k;
    }
};

} // namespace lpg
