// newton_inst_screen.cu -- the screening pass of K1 (screen_kernel in
// newton_kernel.cuh): layout planning and its instances, one per (gradient
// column tiles, k-steps) of the direction-pair layouts: orders 1-3 -> (2, 2),
// 4 -> (3, 3), 5 and 6 -> (4, 4); and one per Gaunt order 3-6 (fourfold).
#include "newton_kernel.cuh"

#include <algorithm>

namespace clb {

bool screen_supported(int nt, int nbk) { return nt == nbk && nt >= 2 && nt <= 4; }

int plan_screen(NewtonArgs &a)
{
    const NewtonProblem &pb = a.prob;
    if (!pb.paired || a.momentType != 0 || a.mixed || a.optType != 0)
        return -1;
    a.nw = a.warps = kWarps;
    a.T = pb.quad ? 16 : 32;
    a.kq = 32;
    a.ntq = a.kq / 8;
    a.ldv = pb.nb + 4;
    a.ldE = a.kq + 4;
    a.ldG = pb.K2p + 4;
    a.ldh = (pb.n | 1) + 1;
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
    a.stageEll = 0;
    a.offEllVal = a.offEllIdx = a.offEllPair = a.offEllOff = off;
    a.offExp = take(64);
    a.offBar = take(6);
    a.offEg = take(4 * a.ldv);   // the representative start and results
    a.offE = 0;
    exp_consts_init(a.ex);
    const int unionBase = off;
    const int endG = unionBase + ((T * a.ldG + 1) & ~1);
    const int endA = unionBase + (pb.quad ? 2 : 3) * (a.kq * pb.ldP + a.kq);   // staged chunks
    a.offP = unionBase;
    a.offG = unionBase;
    a.offH = a.offVec = endG;
    a.doubleBuffer = 1;
    a.ntf = 8;
    a.ntExact = pb.K2p / 8;
    a.nbk = pb.nb / 8;
    a.tpw = 0;
    a.smemBytes = (endA > endG ? endA : endG) * 8;
    if ((pb.quad ? !newton_quad_supported(pb.n) : !screen_supported(a.ntExact, a.nbk)) || a.smemBytes > 232448 - 1024)
        return -1;
    return 0;
}

static cudaError_t screen_dispatch(const NewtonArgs &a, int grid, cudaStream_t s, int mode, int *occ)
{
    if (a.prob.quad) {
        switch (a.prob.n) {
        case 10:
            return screen_run<quad_groups(10, true).tile[4], 1, 10>(a, grid, s, mode, occ);
        case 15:
            return screen_run<quad_groups(15, true).tile[4], 1, 15>(a, grid, s, mode, occ);
        case 21:
            return screen_run<quad_groups(21, true).tile[4], 1, 21>(a, grid, s, mode, occ);
        case 28:
            return screen_run<quad_groups(28, true).tile[4], 1, 28>(a, grid, s, mode, occ);
        default:
            return cudaErrorInvalidValue;
        }
    }
    switch (a.ntExact) {
    case 2:
        return screen_run<2, 2, 0>(a, grid, s, mode, occ);
    case 3:
        return screen_run<3, 3, 0>(a, grid, s, mode, occ);
    case 4:
        return screen_run<4, 4, 0>(a, grid, s, mode, occ);
    default:
        return cudaErrorInvalidValue;
    }
}

cudaError_t prepare_screen(const NewtonArgs &a) { return screen_dispatch(a, 0, nullptr, 1, nullptr); }

cudaError_t launch_screen(const NewtonArgs &a, int grid, cudaStream_t stream)
{
    return screen_dispatch(a, grid, stream, 0, nullptr);
}

cudaError_t launch_screen_gate(const int *iters, int first, int count, int *out, cudaStream_t stream)
{
    int blocks = (count + 255) / 256;
    blocks = blocks < 1 ? 1 : (blocks > 1184 ? 1184 : blocks);
    screen_gate_kernel<<<blocks, 256, 0, stream>>>(iters, first, count, out);
    return cudaGetLastError();
}

namespace {
// What K1's order is taken over: the screened list when the gate is open, else
// the range when it is small enough; -1: K1 takes the range in cell order.
__device__ __forceinline__ int order_count(const int *list, const int *listCount, int count, const int *gateCount,
                                           int gateMin, int wholeMax, bool &useList)
{
    useList = list != nullptr && (gateCount == nullptr || *gateCount >= gateMin);
    if (!useList && count > wholeMax)
        return -1;
    return useList ? *listCount : count;
}

// Bucket of a cell: 31 - min(iterations, 31), the longest chains first.
__device__ __forceinline__ int order_bucket(const int *iters, int cell) { return 31 - min(iters[cell], 31); }

// Counting sort over several CTAs: counts of every bucket, then each CTA
// reserves its part of every bucket and fills it.  (One CTA took 450 us for
// 300,000 cells.)  work: [0, 32) bucket counts, [32, 64) cells handed out.
__global__ void __launch_bounds__(1024) order_count_kernel(const int *list, const int *listCount, int first, int count,
                                                           const int *gateCount, int gateMin, int wholeMax,
                                                           const int *iters, int *work, int *outCount)
{
    __shared__ int hist[32];
    bool useList;
    const int cnt = order_count(list, listCount, count, gateCount, gateMin, wholeMax, useList);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        *outCount = cnt;
    if (cnt < 0)
        return;
    if (threadIdx.x < 32)
        hist[threadIdx.x] = 0;
    __syncthreads();
    const unsigned lane = threadIdx.x & 31u;
    for (int base = blockIdx.x * blockDim.x; base < cnt; base += gridDim.x * blockDim.x) {
        const int i = base + (int)threadIdx.x;
        const int b = (i < cnt) ? order_bucket(iters, useList ? list[i] : first + i) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        if (b >= 0 && lane == (unsigned)(__ffs(peers) - 1))
            atomicAdd(&hist[b], __popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < 32 && hist[threadIdx.x] > 0)
        atomicAdd(&work[threadIdx.x], hist[threadIdx.x]);
}

__global__ void __launch_bounds__(1024) order_fill_kernel(const int *list, const int *listCount, int first, int count,
                                                          const int *gateCount, int gateMin, int wholeMax,
                                                          const int *iters, int *work, int *out)
{
    __shared__ int hist[32], start[32];
    bool useList;
    const int cnt = order_count(list, listCount, count, gateCount, gateMin, wholeMax, useList);
    if (cnt < 0)
        return;
    const unsigned lane = threadIdx.x & 31u;
    for (int base = blockIdx.x * blockDim.x; base < cnt; base += gridDim.x * blockDim.x) {
        if (threadIdx.x < 32)
            hist[threadIdx.x] = 0;
        __syncthreads();
        const int i = base + (int)threadIdx.x;
        const int c = (i < cnt) ? (useList ? list[i] : first + i) : 0;
        const int b = (i < cnt) ? order_bucket(iters, c) : -1;
        const unsigned peers = __match_any_sync(0xffffffffu, b);
        const int leader = __ffs(peers) - 1;
        int pos = 0;
        if (b >= 0 && lane == (unsigned)leader)
            pos = atomicAdd(&hist[b], __popc(peers));
        pos = __shfl_sync(0xffffffffu, pos, leader);
        __syncthreads();
        if (threadIdx.x < 32) {
            int before = 0;
            for (int k = 0; k < (int)threadIdx.x; k++)
                before += work[k];
            start[threadIdx.x] = hist[threadIdx.x] > 0 ? before + atomicAdd(&work[32 + threadIdx.x], hist[threadIdx.x]) : 0;
        }
        __syncthreads();
        if (b >= 0)
            out[start[b] + pos + __popc(peers & ((1u << lane) - 1u))] = c;
        __syncthreads();
    }
}
}  // namespace

cudaError_t launch_order_cells(const int *list, const int *listCount, int first, int count, const int *gateCount,
                               int gateMin, int wholeMax, const int *iters, int *work, int *out, int *outCount,
                               cudaStream_t stream, int *kernels)
{
    cudaError_t e = cudaMemsetAsync(work, 0, kOrderWork * sizeof(int), stream);
    if (e != cudaSuccess)
        return e;
    const int blocks = std::max(1, std::min(148, (count + 1023) / 1024));
    order_count_kernel<<<blocks, 1024, 0, stream>>>(list, listCount, first, count, gateCount, gateMin, wholeMax, iters,
                                                    work, outCount);
    order_fill_kernel<<<blocks, 1024, 0, stream>>>(list, listCount, first, count, gateCount, gateMin, wholeMax, iters,
                                                   work, out);
    *kernels += 2;
    return cudaGetLastError();
}

int screen_ctas_per_sm(const NewtonArgs &a)
{
    int occ = 1;
    if (screen_dispatch(a, 0, nullptr, 2, &occ) != cudaSuccess)
        return 1;
    return occ;
}

}  // namespace clb
