// newton_inst_pair_b.cu -- the larger instances of the direction-pair layout
// (Gaunt orders 5 and 6, direct order 4); see newton_inst_pair.cu.
#include "newton_kernel.cuh"

namespace clb {

bool newton_run_exact_pair_b(const NewtonArgs &a, int grid, cudaStream_t s, int mode, int *occ, cudaError_t *err)
{
#define CLB_PAIR(NT_, NBK_, N_, NTE_, NBE_)                                                     \
    if (a.ntExact == NT_ && a.nbk == NBK_ && a.prob.n == N_ && a.prob.K2e == 8 * NTE_ &&   \
        a.prob.nbe == 8 * NBE_) {                                                            \
        *err = newton_run<1, NT_, 0, NT_, NBK_, 0, 16 * NTE_ + NBE_, 16, N_>(a, grid, s, mode, occ); \
        return true;                                                                           \
    }
    CLB_PAIR(9, 4, 21, 5, 2)
    CLB_PAIR(13, 4, 28, 7, 2)
    CLB_PAIR(16, 3, 15, 9, 2)
#undef CLB_PAIR
    return false;
}

}  // namespace clb
