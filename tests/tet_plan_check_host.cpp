// Test harness: the tet plan's invariant checks (litepgo_b200/csrc/lpg_plan.cpp) on a plan whose table of the
// gradient pass's contributors is changed. Returns 0 where check_tet_clusters accepts it, else -1.
#include <string>

#include "lpg_internal.h"

namespace lpg {
[[noreturn]] void fail(int code, const std::string& what) { throw Error{code, what}; }
void check_cuda(cudaError_t, const char*) {}
} // namespace lpg

extern "C" int check_plan(int V, int T, const int32_t* tets, int cluster, int add, int drop) {
    lpg::HostPlan p;
    lpg::build_plan(V, T, tets, p, 4);
    const int ncl = static_cast<int>(p.tc_row_ptr.size()) - 1;
    p.tc_dent[(cluster + ncl) % ncl] += add;
    p.tc_dent.resize(p.tc_dent.size() - drop);
    try {
        lpg::check_tet_clusters(p, tets);
    } catch (const lpg::Error&) {
        return -1;
    }
    return 0;
}
