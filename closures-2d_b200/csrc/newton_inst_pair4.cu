// newton_inst_pair4.cu -- the direction-pair Mn instances in the 16-slot
// launch shape (8 warps, two staged chunks, two CTAs per SM), for the
// Gaunt orders 3-6 and the direct order 4: the larger contractions, where
// overlapping one CTA's per-slot Newton logic with the other's contractions
// can pay.  The autotuner chooses between this shape and the 32-slot one.
#include "newton_kernel.cuh"

namespace clb {

namespace {
constexpr int kPair4Shapes[][3] = {{4, 2, 10}, {7, 3, 15}, {9, 4, 21}, {13, 4, 28}, {16, 3, 15}};
}  // namespace

bool newton_pair4_supported(int nt, int nbk, int n)
{
    for (const auto &s : kPair4Shapes)
        if (s[0] == nt && s[1] == nbk && s[2] == n)
            return true;
    return false;
}

bool newton_run_exact_pair4(const NewtonArgs &a, int grid, cudaStream_t s, int mode, int *occ, cudaError_t *err)
{
    if (a.momentType != 0 || a.mixed || a.nw != 4)
        return false;
#define CLB_PAIR4(NT_, NBK_, N_, NTE_, NBE_)                                                     \
    if (a.ntExact == NT_ && a.nbk == NBK_ && a.prob.n == N_ && a.prob.K2e == 8 * NTE_ &&   \
        a.prob.nbe == 8 * NBE_) {                                                            \
        *err = newton_run<1, NT_, 0, NT_, NBK_, 0, 16 * NTE_ + NBE_, 8, N_>(a, grid, s, mode, occ); \
        return true;                                                                           \
    }
    CLB_PAIR4(4, 2, 10, 2, 1)
    CLB_PAIR4(7, 3, 15, 4, 2)
    CLB_PAIR4(9, 4, 21, 5, 2)
    CLB_PAIR4(13, 4, 28, 7, 2)
    CLB_PAIR4(16, 3, 15, 9, 2)
#undef CLB_PAIR4
    return false;
}

}  // namespace clb
