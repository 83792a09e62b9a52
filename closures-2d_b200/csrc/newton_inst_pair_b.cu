// newton_inst_pair_b.cu -- the fourfold-direction instances (Gaunt orders 3-6);
// see newton_inst_pair.cu.
#include "newton_kernel.cuh"

namespace clb {

bool newton_run_exact_pair_b(const NewtonArgs &a, int grid, cudaStream_t s, int mode, int *occ, cudaError_t *err)
{
#define CLB_QUAD(N_)                                                                            \
    if (a.prob.n == N_) {                                                                      \
        constexpr int NT_ = quad_groups(N_, false).tile[4];                                    \
        *err = newton_run<1, NT_, 0, NT_, 1, 0, kQuad, 16, N_>(a, grid, s, mode, occ);          \
        return true;                                                                           \
    }
    CLB_QUAD(10)
    CLB_QUAD(15)
    CLB_QUAD(21)
    CLB_QUAD(28)
#undef CLB_QUAD
    return false;
}

}  // namespace clb
