// Test-only: the FP32 forward kernel's choice of form and its shared-memory plan
// (forward32_plan.h) compiled for the host.
#include "forward32_plan.h"

using namespace awg::fwd32;

// The bytes that an instance (S, M, nodes) lays out in a launch for a batch of largest sizes
// (bS, bM, bnodes); *smem: what the launch allocates, form: states a thread, buffers, staged,
// owner threads.
extern "C" int plan_bytes(int S, int M, int nodes, int bS, int bM, int bnodes, int is_long, int least,
                          int *smem, int *form) {
    const Sizes z{S, M, nodes};
    *smem = launch_bytes(Sizes{bS, bM, bnodes});
    const Form f = form_of(z, *smem, is_long != 0, bS > 4 * OWNERS, least);
    form[0] = f.kpt;
    form[1] = f.bufs;
    form[2] = f.staged;
    form[3] = f.owners;
    return SmemPlan(z, f.bufs, f.staged).total;
}
