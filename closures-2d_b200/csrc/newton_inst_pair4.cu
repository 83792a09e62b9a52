// newton_inst_pair4.cu -- the Mn instances of the folded layouts in the 16-slot
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
    if (a.prob.quad) {
#define CLB_QUAD4(N_)                                                                           \
    if (a.prob.n == N_) {                                                                      \
        constexpr int NT_ = quad_groups(N_, false).tile[4];                                    \
        *err = newton_run<1, NT_, 0, NT_, 1, 0, kQuad, 8, N_>(a, grid, s, mode, occ);           \
        return true;                                                                           \
    }
        CLB_QUAD4(10)
        CLB_QUAD4(15)
        CLB_QUAD4(21)
        CLB_QUAD4(28)
#undef CLB_QUAD4
        return false;
    }
    if (a.ntExact == 16 && a.nbk == 3 && a.prob.n == 15 && a.prob.K2e == 72 && a.prob.nbe == 16) {
        *err = newton_run<1, 16, 0, 16, 3, 0, 16 * 9 + 2, 8, 15>(a, grid, s, mode, occ);
        return true;
    }
    return newton_run_exact_pair_c(a, grid, s, mode, occ, err);
}

}  // namespace clb
