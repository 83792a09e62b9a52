// newton_inst_pair.cu -- Mn instances of the folded layouts.  Direction pairs:
// one per (column tiles, k-steps, moments) of orders 1 and 2, the direct
// orders 3 and 4, and the Gaunt orders 3-6 for tables that have no fourfold
// symmetry (newton_inst_pair_c.cu).  Fourfold directions: the Gaunt orders
// 3-6, where the four column groups pad to fewer MMAs per direction than two
// (orders 1 and 2: as many).  The moment count is part of the key: the per-slot logic is unrolled
// for exactly that many rows.
#include "newton_kernel.cuh"

namespace clb {

namespace {
// (tiles, k-steps, n) of the pair layouts: N = 1, 2 -> (2,2,3) (3,2,6), Gaunt or
// direct; Gaunt N = 3..6 -> (4,2,10) (7,3,15) (9,4,21) (13,4,28); direct N = 3, 4 -> (7,2,10) (16,3,15).  The pair instances also
// carry the even tiles and k-steps: E = sum over even degrees of l + 1 columns,
// or the products of two moments of one parity, padded to 8.
constexpr int kPairShapes[][3] = {{2, 2, 3}, {3, 2, 6}, {4, 2, 10}, {7, 2, 10}, {7, 3, 15}, {9, 4, 21}, {13, 4, 28},
                                  {16, 3, 15}};
}  // namespace

bool newton_pair_supported(int nt, int nbk, int n)
{
    for (const auto &s : kPairShapes)
        if (s[0] == nt && s[1] == nbk && s[2] == n)
            return true;
    return false;
}

bool newton_quad_supported(int n) { return n == 10 || n == 15 || n == 21 || n == 28; }

bool newton_run_exact_pair(const NewtonArgs &a, int grid, cudaStream_t s, int mode, int *occ, cudaError_t *err)
{
    if (a.momentType != 0 || a.mixed)
        return false;
    if (a.prob.quad)
        return newton_run_exact_pair_b(a, grid, s, mode, occ, err);
#define CLB_PAIR(NT_, NBK_, N_, NTE_, NBE_)                                                     \
    if (a.ntExact == NT_ && a.nbk == NBK_ && a.prob.n == N_ && a.prob.K2e == 8 * NTE_ &&   \
        a.prob.nbe == 8 * NBE_) {                                                            \
        *err = newton_run<1, NT_, 0, NT_, NBK_, 0, 16 * NTE_ + NBE_, 16, N_>(a, grid, s, mode, occ); \
        return true;                                                                           \
    }
    CLB_PAIR(2, 2, 3, 1, 1)
    CLB_PAIR(3, 2, 6, 2, 1)
    CLB_PAIR(7, 2, 10, 4, 1)
    CLB_PAIR(16, 3, 15, 9, 2)
#undef CLB_PAIR
    return newton_run_exact_pair_c(a, grid, s, mode, occ, err);
}

}  // namespace clb
