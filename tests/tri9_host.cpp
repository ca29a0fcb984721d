// Test harness: the tet tangent's 9x9 clamp by few eigenpairs (litepgo_b200/csrc/lpg_tri9.h) on the host, for
// tests/test_tri9.py. The return value is tri9_clamp's; out is M+ unless that is 0.
#include "lpg_tri9.h"

namespace {
template <typename R> int run(const double* in, double* out) {
    R A[45], M[45], sc[lpg::kTri9Scratch];
    for (int i = 0; i < 9; ++i)
        for (int j = i; j < 9; ++j) M[lpg::sym9(i, j)] = A[lpg::sym9(i, j)] = static_cast<R>(in[9 * i + j]);
    const int how = lpg::tri9_clamp<R>(A, sc);
    for (int i = 0; i < 9; ++i)
        for (int j = i; j < 9; ++j)
            out[9 * i + j] = out[9 * j + i] = A[lpg::sym9(i, j)] + (how == 1 ? M[lpg::sym9(i, j)] : R(0));
    return how;
}
} // namespace

extern "C" int tri9_host(int fp32, const double* in, double* out) {
    return fp32 ? run<float>(in, out) : run<double>(in, out);
}
