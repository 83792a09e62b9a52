// newton.cu -- launch planning and instance selection of the persistent
// dual-Newton kernel (device code in newton_kernel.cuh).
#include "newton.cuh"

#include "angular.h"

#include <cfloat>
#include <cmath>
#include <mutex>

namespace clb {

cudaError_t raise_smem_limit(const void *kernel, int bytes)
{
    static std::mutex m;   // two threads' reads and writes in turn
    std::lock_guard<std::mutex> lock(m);
    cudaFuncAttributes at;
    const cudaError_t e = cudaFuncGetAttributes(&at, kernel);
    if (e != cudaSuccess || at.maxDynamicSharedSizeBytes >= bytes)
        return e;
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

int plan_newton(NewtonArgs &a)
{
    const NewtonProblem &pb = a.prob;
    const int nbMax = pb.nb > 8 ? pb.nb : 8, ldPMax = pb.ldP, nMax = pb.n;
    const int K2tot = pb.K2p + (a.momentType == 1 ? pb.nb : 0);
    int ellGroups = pb.ellGroups, ellChunks = pb.ellChunks;
    if (a.nw == 0)
        a.nw = kWarps;
    if (a.nw != kWarps && a.nw != 4)
        return -1;
    const int nw = a.nw;
    a.T = 4 * nw;
    // fused contractions when the problem's G fits in 16 column tiles; in
    // FP64 one warp per 8 slots x 8 quadrature rows of a 32-row chunk, mixed
    // one per 16 slots x 8 rows
    const int nt2 = K2tot / 8;
    a.ntf = (nt2 <= 16) ? ((nt2 + 7) / 8) * 8 : 0;
    a.warps = (a.ntf > 0 && !a.mixed) ? 2 * nw : nw;
    a.kq = 32;
    a.ntq = a.kq / 8;
    a.ldv = nbMax + 4;
    a.ldE = a.kq + 4;
    a.ldG = K2tot + 4;
    // even: 16-byte row pairs for the broadcast loads; half of it odd: a column's
    // entries, or eight rows' pairs, spread over the banks (with 16 all 15 rows
    // of M4 fell in one: a step of 200 x 200 cells 3.13 ms, with 18 2.97)
    a.ldh = (nMax | 1) + 1;
    if (a.ldh % 4 == 0)
        a.ldh += 2;
    const int T = a.T;
    int off = 0;
    auto take = [&](int ndoubles) {
        int o = off;
        off += (ndoubles + 1) & ~1;   // keep 16-byte alignment
        return o;
    };
    a.offAlpha = take(T * a.ldv);
    a.offAold = take(T * a.ldv);
    a.offD = take(T * a.ldv);
    a.offU = take(T * a.ldv);
    a.offScal = take(T * SC_N);
    a.offInt = take((T * SI_N + 1) / 2);
    a.offFpart = take(T * a.ntq);
    a.offStat = take(kStatU64 + 1);
    // the 16-slot shape reads the Gaunt table through L1 so that two CTAs fit
    a.stageEll = (nw == kWarps) ? 1 : 0;   // matches the kernel's compile-time choice
    if (!a.stageEll)
        ellGroups = ellChunks = 0;
    a.offEllVal = take(ellGroups * kEllGroup);
    a.offEllIdx = take(ellGroups * kEllGroup / 4);
    a.offEllPair = take(ellChunks * 64 / 4);
    a.offEllOff = take((ellChunks + 2) / 2);
    a.offExp = take(64);
    a.offBar = take(6);

    exp_consts_init(a.ex);
    const int unionBase = off;
    const int ntiles2 = (T / 16) * (K2tot / 8);
    a.tpw = (ntiles2 + nw - 1) / nw;
    a.ntExact = a.ntf > 0 ? nt2 : 0;
    a.nbk = a.ntf > 0 ? pb.nb / 8 : 0;
    if (a.mixed && a.ntExact == 0)
        return -2;
    if (nw != kWarps && (a.ntExact == 0 || !pb.paired || a.mixed || a.optType != 0 ||
                         !(pb.quad ? newton_quad_supported(pb.n) : newton_pair4_supported(a.ntExact, a.nbk, pb.n))))
        return -1;   // the 16-slot shape: direction-pair Newton only
    // phase-B region
    int offG = unionBase;
    a.strideH = nMax * a.ldh;   // ldh is even
    int offH = offG + ((T * a.ldG + 1) & ~1);
    int offVec = offH + a.warps * a.strideH;
    int endB = offVec + a.warps * 64;

    // phase-A region
    const int maxDoubles = (232448 - 1024) / 8;   // opt-in limit minus static shared
    if (a.ntf > 0) {
        const int depth = (nw == kWarps) ? 3 : 2;
        const int endA = unionBase + depth * (a.kq * ldPMax + a.kq);   // staged chunks
        const int end = endA > endB ? endA : endB;
        if (end <= maxDoubles) {
            a.doubleBuffer = 1;
            a.offP = unionBase;
            a.offE = a.offEg = 0;
            a.offG = offG;
            a.offH = offH;
            a.offVec = offVec;
            a.smemBytes = end * 8;
            return 0;
        }
        // a Gaunt table too long to be staged beside 32 slots (order 6 with
        // Q = 12: 26 entry groups instead of 12): 16 slots, whose instances
        // read it through L1 (32,000 vectors 2.4 ms; unfolded, with the
        // general contractions, 4.0)
        if (pb.paired && nw == kWarps) {
            NewtonArgs b = a;
            b.nw = 4;
            if (plan_newton(b) == 0) {
                a = b;
                return 0;
            }
        }
        a.ntf = 0;
        a.ntExact = a.nbk = 0;
        if (a.mixed)
            return -2;
        if (nw != kWarps)
            return -1;
        a.warps = nw;
    }
    // General contractions: where their regions start within a 128-byte line
    // decides up to 8 % of the time (4736 vectors of direct order 6: 3.08 ms at
    // 112 bytes, 3.13 at 16, 48 or 80, 3.27 at 0 or 96, 3.36 at 32 or 64; order 5
    // 1.68 to 1.82, PPn order 4 0.80 to 0.85 in the same order; the fused
    // instances take the same time at all of them).
    const int base = (unionBase + 1) / 16 * 16 + 14;
    offG = base;
    offH = offG + ((T * a.ldG + 1) & ~1);
    offVec = offH + a.warps * a.strideH;
    endB = offVec + a.warps * 64;
    for (int db = 1; db >= 0; db--) {
        int offP = base;
        int offE = offP + (db ? 2 : 1) * (a.kq * ldPMax + a.kq);
        int offEg = offE + T * a.ldE;
        int endA = offEg + T * a.ldE;
        int end = endA > endB ? endA : endB;
        if (end <= maxDoubles) {
            a.doubleBuffer = db;
            a.offP = offP;
            a.offE = offE;
            a.offEg = offEg;
            a.offG = offG;
            a.offH = offH;
            a.offVec = offVec;
            a.smemBytes = end * 8;
            return 0;
        }
    }
    return -1;
}

// Instance selection: the kernel specialised to the problem's exact column-tile
// and k-step counts where there is one, else the fused instance with runtime
// counts or the general contractions.  mode: 0 launch, 1 shared-memory attribute, 2 occupancy.
static cudaError_t run(const NewtonArgs &a, int grid, cudaStream_t stream, int mode, int *occ)
{
    cudaError_t e = cudaErrorInvalidValue;
    if (a.mixed) {
        if (newton_run_mixed_mn(a, grid, stream, mode, occ, &e) || newton_run_mixed_ppn(a, grid, stream, mode, occ, &e))
            return e;
        return cudaErrorInvalidValue;
    }
    if (a.prob.paired) {
        // the direction-pair layout runs only its own fused instances
        if (a.nw == 4)
            return (a.ntf > 0 && a.ntExact > 0 && newton_run_exact_pair4(a, grid, stream, mode, occ, &e))
                       ? e
                       : cudaErrorInvalidValue;
        if (a.ntf > 0 && a.ntExact > 0 && newton_run_exact_pair(a, grid, stream, mode, occ, &e))
            return e;
        return cudaErrorInvalidValue;
    }
    if (a.nw != kWarps)
        return cudaErrorInvalidValue;
    if (a.ntf > 0 && a.ntExact > 0) {
        if (newton_run_exact_mn_a(a, grid, stream, mode, occ, &e) ||
            newton_run_exact_mn_b(a, grid, stream, mode, occ, &e) ||
            newton_run_exact_ppn_a(a, grid, stream, mode, occ, &e) ||
            newton_run_exact_ppn_b(a, grid, stream, mode, occ, &e))
            return e;
    }
    if (newton_run_generic(a, grid, stream, mode, occ, &e))
        return e;
    return cudaErrorInvalidValue;
}

cudaError_t prepare_newton(const NewtonArgs &a) { return run(a, 0, nullptr, 1, nullptr); }

cudaError_t launch_newton(const NewtonArgs &a, int grid, cudaStream_t stream)
{
    return run(a, grid, stream, 0, nullptr);
}

int newton_ctas_per_sm(const NewtonArgs &a)
{
    int occ = 1;
    if (run(a, 0, nullptr, 2, &occ) != cudaSuccess)
        return 1;
    return occ;
}

}  // namespace clb
