// Host build of the neo-Hookean tangent's semi-definiteness test (litepgo_b200/csrc/lpg_psd.h).
#include "lpg_psd.h"

extern "C" void nh_semidefinite_host(int n, const double* G, const double* J, const double* theta, int* out) {
    for (int k = 0; k < n; ++k) {
        const double l = theta[2 * k] / theta[2 * k + 1];
        out[k] = lpg::nh_semidefinite(G + 9 * k, l * log(J[k]) - 1.0, l);
    }
}
