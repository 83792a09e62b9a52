// newton_inst_pair_c.cu -- direction pairs of the Gaunt orders 3-6, in both launch
// shapes, for tables symmetric under phi -> phi + pi but not under phi -> -phi
// (a quadrature with its azimuths turned); see newton_inst_pair.cu.  8000
// vectors on such tables, M3 / M4 / M5 (Q = 30) / M6 (Q = 40): 382, 526, 714 and
// 1229 us, one direction per row 552, 698, 1107 and 2188.
#include "newton_kernel.cuh"

namespace clb {

bool newton_run_exact_pair_c(const NewtonArgs &a, int grid, cudaStream_t s, int mode, int *occ, cudaError_t *err)
{
#define CLB_PAIR(NT_, NBK_, N_, NTE_, NBE_)                                                     \
    if (a.ntExact == NT_ && a.nbk == NBK_ && a.prob.n == N_ && a.prob.K2e == 8 * NTE_ &&        \
        a.prob.nbe == 8 * NBE_) {                                                               \
        *err = a.nw == 4                                                                        \
                   ? newton_run<1, NT_, 0, NT_, NBK_, 0, 16 * NTE_ + NBE_, 8, N_>(a, grid, s, mode, occ)   \
                   : newton_run<1, NT_, 0, NT_, NBK_, 0, 16 * NTE_ + NBE_, 16, N_>(a, grid, s, mode, occ); \
        return true;                                                                            \
    }
    CLB_PAIR(4, 2, 10, 2, 1)
    CLB_PAIR(7, 3, 15, 4, 2)
    CLB_PAIR(9, 4, 21, 5, 2)
    CLB_PAIR(13, 4, 28, 7, 2)
#undef CLB_PAIR
    return false;
}

}  // namespace clb
