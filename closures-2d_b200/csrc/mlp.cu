// mlp.cu -- learned warm start for the dual Newton solve.
//
// A small multilayer perceptron maps the normalised moments u/u0 of a cell to
// the multipliers alpha of the scaled problem (u0 = 1).  Newton then starts
// from the prediction and runs to the same tolerance; where the prediction is
// not finite the caller's fallback multipliers (previous step, or isotropic)
// are used, so the network changes iteration counts, not the converged
// answer.  There is no counterpart in the reference, which starts each solve
// from the previous stage's alpha (momopt_update.cpp:236-238).
//
// Network: n -> W -> W -> W -> n with GELU (exact erf form) between layers,
// BF16 weights and activations feeding tensor-core MMAs (forward: tcgen05;
// backward: mma.sync m16n8k16, BF16 x BF16 -> FP32), FP32 master weights, FP32
// Adam.  Outputs are the
// multipliers standardised per component with the training set's mean and
// standard deviation.  Training and inference both run on these kernels.
#include "closures_gpu.h"

#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include "tc_gemm.cuh"
#include "uploads.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace {

constexpr int kLayers = 4;
constexpr double kSqrtPi = 1.7724538509055160273;
constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z)
{
    const float phi = 0.39894228040143268f * __expf(-0.5f * z * z);
    return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * phi;
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Asynchronous 16-byte copy to shared memory, zero-filled when !valid.
__device__ __forceinline__ void cp16_zfill(void *smem, const void *gmem, bool valid)
{
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    const int bytes = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes) : "memory");
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(unsigned (&r)[4], unsigned addr)
{
    if (TRANS)
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr));
    else
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(addr));
}

// One layer of the backward pass in one launch.  Its three products need
// only the layer's dZ, so their CTAs run side by side:
//   dW = in^T . dZ           64 x 64 tiles, K = rows
//   db = column sums of dZ   32 columns per CTA
//   dA . gelu'(Z) = next dZ  64 x 64 tiles of dZ . W^T, K = N (layers above 0)
// Every sum runs in the order of a plain loop over K in steps of 16 (mma.sync
// m16n8k16, the k-steps of one output a single chain; db one addition per
// row), so the gradients do not depend on the tiling, and training, whose
// first Adam steps divide gradients by their own size, is reproducible to the
// bit.  A chain of 256 dependent MMAs (4096 rows) or 4096 additions is some 5
// to 8 us of a layer's 35; the rest is the 64 stages, about 900 cycles each: a
// wait for the staged operands, a CTA barrier, sixteen-byte copies by every
// thread, the fragment loads.  The operands come four stages deep (through
// scalar loads the four dW took 1810 us a step at 4096 x 512, the column sums
// 910, dA 164).
// Row strides (ldin, ldz, ldw) are multiples of 8.
struct BackArgs {
    const __nv_bfloat16 *in;   // [rows][ldin], K columns
    const __nv_bfloat16 *dZ;   // [rows][ldz], N columns
    const float *dZf;          // [rows][ldz]
    const __nv_bfloat16 *W;    // [K][ldw]: row i the weights of input i (ldw >= N, zero padded)
    const float *Zprev;        // [rows][K] pre-activations of the layer below; null for layer 0
    float *gW, *gb;            // [K][N], [N]
    __nv_bfloat16 *dZnext;     // [rows][ldn], K columns
    float *dZfnext;
    int rows, K, N, ldin, ldz, ldw, ldn;
    int tilesW, tilesB;        // dW tiles, db CTAs; the rest are dA tiles
};
constexpr int kBackStages = 4, kBackK = 64;
constexpr int kBackTile = 64 * (kBackK + 8);   // bf16 of one staged operand (rows padded by 16 bytes)
constexpr int kBackSmem = kBackStages * 2 * kBackTile * 2;

// One 64 x 64 tile, eight warps of 32 x 16.  C [M x N] = A . B over kTot: dW
// (W): A = in^T, B = dZ, both staged as [k][64]; dA: A = dZ, B = W^T, staged as
// [64][k].  A stage is latency bound, so what a warp issues in it
// counts (addresses are fixed before the loop and advance by one stride), and
// eight warps hide more than four did (a layer's launch 54 us with addresses
// formed per piece, 35 us with fixed ones, four warps each).
template <bool W>
__device__ __forceinline__ void backward_tile(const BackArgs &a, int block, unsigned char *smraw)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int M = W ? a.K : a.rows, N = W ? a.N : a.K, kTot = W ? a.rows : a.ldw;
    const int tn = (N + 63) / 64;
    const int m0 = (block / tn) * 64, n0 = (block % tn) * 64;
    const __nv_bfloat16 *A = W ? a.in : a.dZ, *B = W ? a.dZ : a.W;
    const int lda = W ? a.ldin : a.ldz, ldb = W ? a.ldz : a.ldw;
    constexpr int LD = kBackK + 8;   // also 64 + 8 for the [k][64] form
    __nv_bfloat16 *sA = reinterpret_cast<__nv_bfloat16 *>(smraw), *sB = sA + kBackStages * kBackTile;
    const int nst = (kTot + kBackK - 1) / kBackK;
    // this thread's two 16-byte pieces of each operand: rows lr + 32 q
    const int lr = tid >> 3, lc = (tid & 7) * 8;
    const __nv_bfloat16 *pA = W ? A + (size_t)lr * lda + m0 + lc : A + (size_t)(m0 + lr) * lda + lc;
    const __nv_bfloat16 *pB = W ? B + (size_t)lr * ldb + n0 + lc : B + (size_t)(n0 + lr) * ldb + lc;
    const size_t stepA = W ? (size_t)kBackK * lda : kBackK, stepB = W ? (size_t)kBackK * ldb : kBackK;
    const size_t rowA = (size_t)32 * lda, rowB = (size_t)32 * ldb;
    bool inA[2], inB[2];   // the bounds that do not depend on the stage
#pragma unroll
    for (int q = 0; q < 2; q++) {
        inA[q] = W ? m0 + lc < lda : m0 + lr + 32 * q < M;
        inB[q] = W ? n0 + lc < ldb : n0 + lr + 32 * q < N;
    }
    int kLeft = kTot - (W ? lr : lc);   // k of this thread's first piece still inside
    const unsigned dstA = (unsigned)__cvta_generic_to_shared(sA + lr * LD + lc);
    const unsigned dstB = (unsigned)__cvta_generic_to_shared(sB + lr * LD + lc);
    auto cp = [](unsigned dst, const void *src, bool ok) {
        const int bytes = ok ? 16 : 0;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
    };
    auto load = [&](int buf) {   // the next stage into buffer buf
        const unsigned off = (unsigned)(buf * kBackTile * 2);
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const bool okK = W ? kLeft > 32 * q : kLeft > 0;
            const bool okA = okK && inA[q], okB = okK && inB[q];
            cp(dstA + off + q * 32 * LD * 2, okA ? pA + q * rowA : A, okA);
            cp(dstB + off + q * 32 * LD * 2, okB ? pB + q * rowB : B, okB);
        }
        pA += stepA;
        pB += stepB;
        kLeft -= kBackK;
    };
    const int wm = (warp >> 2) * 32, wn = (warp & 3) * 16;
    // fragment addresses: W: blocks (k, m) and (k, n) of [k][64] transposed;
    // else blocks of [m][k] and [n][k]
    const int l7 = lane & 7, l8 = (lane >> 3) & 1, l16 = lane >> 4;
    const unsigned fragA = (unsigned)__cvta_generic_to_shared(
        W ? sA + (l7 + l16 * 8) * LD + wm + l8 * 8 : sA + (wm + l7 + l8 * 8) * LD + l16 * 8);
    const unsigned fragB = (unsigned)__cvta_generic_to_shared(
        W ? sB + (l7 + l8 * 8) * LD + wn + l16 * 8 : sB + (wn + l7 + l16 * 8) * LD + l8 * 8);
    float acc[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
            acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.0f;
    for (int st = 0; st < kBackStages - 1; st++) {
        if (st < nst)
            load(st);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    int buf = 0;
    for (int st = 0; st < nst; st++) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kBackStages - 2) : "memory");
        __syncthreads();
        if (st + kBackStages - 1 < nst)
            load((buf + kBackStages - 1) % kBackStages);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const unsigned ta = fragA + buf * kBackTile * 2, tb = fragB + buf * kBackTile * 2;
#pragma unroll
        for (int kk = 0; kk < kBackK; kk += 16) {
            unsigned fa[2][4], fb[4];
            ldmatrix4<W>(fb, tb + (W ? kk * LD : kk) * 2);
#pragma unroll
            for (int i = 0; i < 2; i++)
                ldmatrix4<W>(fa[i], ta + (W ? kk * LD + i * 16 : i * 16 * LD + kk) * 2);
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++)
                    mma_bf16(acc[i][j], fa[i][0], fa[i][1], fa[i][2], fa[i][3], fb[2 * j], fb[2 * j + 1]);
        }
        buf = (buf + 1) % kBackStages;
    }
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
            for (int h = 0; h < 4; h++) {
                const int m = m0 + wm + i * 16 + g + ((h & 2) ? 8 : 0);
                const int nn = n0 + wn + j * 8 + 2 * t + (h & 1);
                // the padding columns of the next dZ are operands of its products
                if (!W && m < M && nn >= N && nn < a.ldn)
                    a.dZnext[(size_t)m * a.ldn + nn] = __float2bfloat16(0.0f);
                if (m >= M || nn >= N)
                    continue;
                if (W) {
                    a.gW[(size_t)m * N + nn] = acc[i][j][h];
                } else {
                    const float v = acc[i][j][h] * gelu_grad(a.Zprev[(size_t)m * N + nn]);
                    a.dZnext[(size_t)m * a.ldn + nn] = __float2bfloat16(v);
                    a.dZfnext[(size_t)m * a.ldn + nn] = v;
                }
            }
}

__global__ void __launch_bounds__(256) backward_kernel(const BackArgs a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int block = blockIdx.x;
    if (block >= a.tilesW && block < a.tilesW + a.tilesB) {
        // db: warp 0 adds the rows in order, all threads stage them
        constexpr int R = 64, S = 6;   // rows per stage, stages: 48 KB
        float *buf = reinterpret_cast<float *>(smraw);
        const int j0 = (block - a.tilesW) * 32;
        const int nst = (a.rows + R - 1) / R;
        auto load = [&](int st) {
            float *d = buf + (st % S) * (R * 32);
            for (int i = tid; i < R * 8; i += 256) {
                const int r = st * R + i / 8, c = j0 + (i % 8) * 4;
                const bool ok = r < a.rows && c < a.ldz;
                cp16_zfill(d + (i / 8) * 32 + (i % 8) * 4, a.dZf + (ok ? (size_t)r * a.ldz + c : 0), ok);
            }
        };
        for (int st = 0; st < S - 1; st++) {
            if (st < nst)
                load(st);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        }
        float s = 0.0f;
        for (int st = 0; st < nst; st++) {
            asm volatile("cp.async.wait_group %0;\n" ::"n"(S - 2) : "memory");
            __syncthreads();
            if (st + S - 1 < nst)
                load(st + S - 1);
            asm volatile("cp.async.commit_group;\n" ::: "memory");
            if (warp == 0) {
                const float *d = buf + (st % S) * (R * 32) + lane;
                const int cnt = min(R, a.rows - st * R);
                if (cnt == R) {
                    // loads well ahead of the chain of additions
                    float x[2][16];
#pragma unroll
                    for (int q = 0; q < 16; q++)
                        x[0][q] = d[q * 32];
#pragma unroll
                    for (int r = 0; r < R; r += 16) {
                        if (r + 16 < R) {
#pragma unroll
                            for (int q = 0; q < 16; q++)
                                x[(r / 16 + 1) & 1][q] = d[(r + 16 + q) * 32];
                        }
#pragma unroll
                        for (int q = 0; q < 16; q++)
                            s += x[(r / 16) & 1][q];
                    }
                } else {
                    for (int r = 0; r < cnt; r++)
                        s += d[r * 32];
                }
            }
        }
        if (warp == 0 && j0 + lane < a.N)
            a.gb[j0 + lane] = s;
        return;
    }
    if (block < a.tilesW)
        backward_tile<true>(a, block, smraw);
    else
        backward_tile<false>(a, block - a.tilesW - a.tilesB, smraw);
}

// W [K x N] FP32 -> W16 [K x ldw] BF16, zero columns N..ldw-1
__global__ void cast_bf16_kernel(const float *W, int K, int N, int ldw, __nv_bfloat16 *W16)
{
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= (size_t)K * ldw)
        return;
    const int r = (int)(i / ldw), c = (int)(i % ldw);
    W16[i] = __float2bfloat16(c < N ? W[(size_t)r * N + c] : 0.0f);
}

// dY = 2 (Y - T) / (B n) for the mean squared error over B x n entries, row
// stride ld; returns per-block partial losses.
__global__ void mse_grad_kernel(const float *Y, const float *T, __nv_bfloat16 *dY, float *dYf, int total, int n, int ld,
                                float scale, float *lossPart)
{
    __shared__ float red[256];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (i < total) {
        float d = Y[i] - T[i];
        l = d * d;
        float gval = 2.0f * d * scale;
        const size_t at = (size_t)(i / n) * ld + i % n;
        dY[at] = __float2bfloat16(gval);
        dYf[at] = gval;
        if (i % n == n - 1)   // the padding columns are operands too
            for (int k = 1; k <= ld - n; k++)
                dY[at + k] = __float2bfloat16(0.0f);
    }
    red[threadIdx.x] = l;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s)
            red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        lossPart[blockIdx.x] = red[0];
}

__device__ __forceinline__ float adam(float w, float *m, float *v, float gi, float lr, float b1, float b2, float eps,
                                      float c1, float c2)
{
    float mi = b1 * *m + (1.0f - b1) * gi;
    float vi = b2 * *v + (1.0f - b2) * gi * gi;
    *m = mi;
    *v = vi;
    w -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    return w;
}

// Adam on every parameter, and the BF16 copies of the weights the GEMMs read
// (row-major and transposed), in one launch: 32 x 32 tiles of each weight
// matrix, transposed through shared memory, then the biases 256 to a block.
// (Eight launches of Adam and eight of the copies took 50 us a step.)
struct UpdateArgs {
    float *W[kLayers], *mW[kLayers], *vW[kLayers], *b[kLayers], *mb[kLayers], *vb[kLayers];
    const float *gW[kLayers], *gb[kLayers];
    __nv_bfloat16 *W16[kLayers], *Wt16[kLayers];
    int dims[kLayers + 1], first[kLayers + 1];   // first tile of each layer; first[kLayers]: of the biases
    float lr, b1, b2, eps, c1, c2;
};

__global__ void __launch_bounds__(256) update_kernel(const UpdateArgs a)
{
    __shared__ __nv_bfloat16 tile[32][34];
    int block = blockIdx.x;
    const int tid = threadIdx.x;
    if (block >= a.first[kLayers]) {
        int j = (block - a.first[kLayers]) * 256 + tid;
        for (int l = 0; l < kLayers; l++) {
            const int N = a.dims[l + 1];
            if (j < N) {
                a.b[l][j] = adam(a.b[l][j], a.mb[l] + j, a.vb[l] + j, a.gb[l][j], a.lr, a.b1, a.b2, a.eps, a.c1, a.c2);
                return;
            }
            j -= N;
        }
        return;
    }
    int l = 0;
    while (block >= a.first[l + 1])
        l++;
    block -= a.first[l];
    const int K = a.dims[l], N = a.dims[l + 1], ldw = (N + 7) / 8 * 8, Kp = (K + 7) / 8 * 8;
    const int tn = (N + 31) / 32, i0 = (block / tn) * 32, j0 = (block % tn) * 32;
    const int x = tid & 31, y = tid >> 5;
    for (int r = y; r < 32; r += 8) {
        const int i = i0 + r, j = j0 + x;
        if (i < K && j < N) {
            const size_t at = (size_t)i * N + j;
            const float w = adam(a.W[l][at], a.mW[l] + at, a.vW[l] + at, a.gW[l][at], a.lr, a.b1, a.b2, a.eps, a.c1, a.c2);
            a.W[l][at] = w;
            const __nv_bfloat16 h = __float2bfloat16(w);
            a.W16[l][(size_t)i * ldw + j] = h;
            tile[r][x] = h;
        }
    }
    __syncthreads();
    for (int r = y; r < 32; r += 8) {
        const int j = j0 + r, i = i0 + x;
        if (i < K && j < N)
            a.Wt16[l][(size_t)j * Kp + i] = tile[x][r];
    }
}

// Linear part of the closure near isotropy (Mn): for u/u0 = (1, x_1, ...)
// close to isotropic, exp(alpha.m) ~ e^{alpha0 p0} (1 + sum alpha_k m_k) with
// orthonormal m_k gives alpha_k ~ 4 pi p0 x_k = 2 sqrt(pi) x_k, and alpha_0 the
// isotropic value 2 sqrt(pi) log(1/(2 sqrt(pi))).  The network learns the
// remainder, so near-isotropic cells need only a small correction.
__device__ __forceinline__ double alpha_linear(int k, double x, int momentType)
{
    if (momentType != CL_MN)
        return 0.0;
    return k == 0 ? 2.0 * kSqrtPi * log(0.5 / kSqrtPi) : 2.0 * kSqrtPi * x;
}

// Inputs: x = u/u0 (BF16, row stride np); targets (alpha_scaled - linear -
// mean)/std (FP32).  With perm (nullable) row c comes from vector perm[c].
__global__ void prep_kernel(const double *u, const double *alpha, const int *perm, int count, int n, int np,
                            int momentType, const float *mean, const float *stdv, __nv_bfloat16 *X, float *Tgt)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count * n)
        return;
    int c = i / n, k = i % n;
    const size_t row = (size_t)(perm ? perm[c] : c) * n;
    double u0 = u[row];
    double x = u[row + k] / u0;
    X[(size_t)c * np + k] = __float2bfloat16((float)x);
    if (Tgt) {
        double a = alpha[row + k];
        if (momentType == CL_MN) {
            if (k == 0)
                a -= log(u0) * 2.0 * kSqrtPi;
        } else {
            a /= u0;
        }
        a -= alpha_linear(k, x, momentType);
        Tgt[i] = (float)((a - mean[k]) / stdv[k]);
    }
}

// alpha = unscale(Y * std + mean); non-finite predictions (or u0 <= 0) take
// the fallback multipliers.  fallbackKind: 0 = keep alpha as given (previous
// stage), 1 = isotropic alpha for this u0, 2 = write NaN so that the Newton
// kernel's start falls back to its own multipliers.
// With idx (nullable), row r of Y is cell idx[off + r] (rows past *cnt - off
// are not there).
__global__ void predict_out_kernel(const float *Y, const double *u, double *alpha, int count, int n,
                                   int momentType, double delta, const float *mean, const float *stdv,
                                   int fallbackKind, int *fallbacks, const int *idx = nullptr,
                                   const int *cnt = nullptr, int off = 0)
{
    int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= count || (idx && off + r >= *cnt))
        return;
    // Y row r; u and alpha rows of cell c (with an index list) or r
    const int c = idx ? idx[off + r] : r;
    const float *Yr = Y + (size_t)r * n;
    double u0 = u[(size_t)c * n];
    bool ok = u0 > 0.0;
    double a[32];
    for (int k = 0; k < n && ok; k++) {
        double x = u[(size_t)c * n + k] / u0;
        double v = (double)Yr[k] * stdv[k] + mean[k] + alpha_linear(k, x, momentType);
        if (!isfinite(v))
            ok = false;
        a[k] = v;
    }
    if (ok) {
        if (momentType == CL_MN)
            a[0] += log(u0) * 2.0 * kSqrtPi;
        else
            for (int k = 0; k < n; k++)
                a[k] *= u0;
        for (int k = 0; k < n; k++)
            alpha[(size_t)c * n + k] = a[k];
        return;
    }
    atomicAdd(fallbacks, 1);
    if (fallbackKind == 2) {
        // mark the start as unusable: the Newton kernel then starts from its
        // fallback multipliers
        alpha[(size_t)c * n] = __longlong_as_double(0x7ff8000000000000ll);
    } else if (fallbackKind == 1 && u0 > 0.0) {
        double a0 = (momentType == CL_MN) ? 2.0 * kSqrtPi * log(u0 / (2.0 * kSqrtPi))
                                          : u0 - 4.0 * delta * kPi / u0;
        alpha[(size_t)c * n] = a0;
        for (int k = 1; k < n; k++)
            alpha[(size_t)c * n + k] = 0.0;
    }
}

// Cells whose last optimisation took at least minIters iterations are listed
// in idx (count in *cnt, order arbitrary); the others get a NaN start, so the
// Newton kernel starts them from their own (previous-stage) multipliers.
__global__ void select_kernel(const int *iters, int count, int minIters, int *idx, int *cnt, double *alpha, int n)
{
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= count)
        return;
    if (iters[c] >= minIters)
        idx[atomicAdd(cnt, 1)] = c;
    else
        alpha[(size_t)c * n] = __longlong_as_double(0x7ff8000000000000ll);
}

// Inputs x = u/u0 of the listed cells idx[off + r], r < min(rows, *cnt - off).
__global__ void prep_idx_kernel(const double *u, const int *idx, const int *cnt, int off, int rows, int n, int np,
                                __nv_bfloat16 *X)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int r = i / n, k = i % n;
    if (r >= rows || off + r >= *cnt)
        return;
    const size_t c = (size_t)idx[off + r];
    X[(size_t)r * np + k] = __float2bfloat16((float)(u[c * n + k] / u[c * n]));
}

int blocks(size_t n, int t = 256) { return (int)((n + t - 1) / t); }

int round8(int x) { return (x + 7) / 8 * 8; }

// W [K x N] FP32 row-major -> Wt [N x Kp] BF16 (the K-major B operand), zero
// columns K..Kp-1
__global__ void transpose_cast_kernel(const float *W, int K, int N, int Kp, __nv_bfloat16 *Wt)
{
    size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i >= (size_t)N * Kp)
        return;
    const int c = (int)(i / Kp), k = (int)(i % Kp);
    Wt[i] = k < K ? __float2bfloat16(W[(size_t)k * N + c]) : __float2bfloat16(0.0f);
}

// The driver's tensor-map encoder, through the runtime's entry-point query
// (no link against the driver library).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    if (!fn) {
        cudaDriverEntryPointQueryResult q;
        void *p = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    }
    return fn;
}

// 2-D map of a row-major BF16 [rows x cols] matrix (cols a multiple of 8,
// base 16-byte aligned) in boxes of boxRows x 64 with the 128 B swizzle;
// reads past the matrix are zero.
bool bf16_map(CUtensorMap *map, const __nv_bfloat16 *base, int rows, int cols, int boxRows)
{
    auto enc = tensor_map_encoder();
    if (!enc || cols % 8 != 0 || ((uintptr_t)base & 15) != 0)
        return false;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)clb::tc::BK, (cuuint32_t)boxRows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)base, dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int sm_count_dev()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms < 1)
            sms = 1;
    }
    return sms;
}

// The persistent tensor-memory GEMM: one CTA per SM (or per tile, if fewer).
template <int BN, int EPI>
cudaError_t tc_gemm_bn(const CUtensorMap &ma, const CUtensorMap &mb, int M, int N, int K, float *Z, const float *bias,
                       __nv_bfloat16 *Act, int ldAct, const int *Mdev, int moff, int *err, cudaStream_t s)
{
    static bool attr = false;
    auto *k = clb::tc::tc_gemm_persistent_kernel<BN, EPI>;
    const int smem = clb::tc::smem_bytes_persistent(BN);
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess)
            return e;
        attr = true;
    }
    const int tiles = ((N + BN - 1) / BN) * ((M + clb::tc::BM - 1) / clb::tc::BM);
    const int grid = tiles < sm_count_dev() ? tiles : sm_count_dev();
    k<<<grid, 192, smem, s>>>(ma, mb, M, N, K, Z, bias, Act, ldAct, Mdev, moff, err);
    return cudaGetLastError();
}

// Z (nullable) [M x N] / Act (nullable) [M x ldAct] = epilogue(A [M x K] .
// B [N x K]^T): the tensor-memory GEMM (tc_gemm.cuh); K a multiple of 8.
template <int EPI>
cudaError_t tc_gemm(const __nv_bfloat16 *A, const __nv_bfloat16 *B, int M, int N, int K, float *Z, const float *bias,
                    __nv_bfloat16 *Act, int ldAct, const int *Mdev, int moff, int *err, cudaStream_t s)
{
    const int bn = N <= 32 ? 32 : (N <= 64 ? 64 : 128);
    CUtensorMap ma, mb;
    if (!bf16_map(&ma, A, M, K, clb::tc::BM) || !bf16_map(&mb, B, N, K, bn))
        return cudaErrorInvalidValue;
    if (bn == 32)
        return tc_gemm_bn<32, EPI>(ma, mb, M, N, K, Z, bias, Act, ldAct, Mdev, moff, err, s);
    if (bn == 64)
        return tc_gemm_bn<64, EPI>(ma, mb, M, N, K, Z, bias, Act, ldAct, Mdev, moff, err, s);
    return tc_gemm_bn<128, EPI>(ma, mb, M, N, K, Z, bias, Act, ldAct, Mdev, moff, err, s);
}

}  // namespace

struct cl_mlp {
    int n = 0, width = 0, momentType = CL_MN;
    double delta = 0;
    int dims[kLayers + 1];
    float *W[kLayers] = {}, *b[kLayers] = {}, *mW[kLayers] = {}, *vW[kLayers] = {}, *mb[kLayers] = {},
          *vb[kLayers] = {}, *gW[kLayers] = {}, *gb[kLayers] = {};
    __nv_bfloat16 *W16[kLayers] = {};    // [in x round8(out)] BF16, zero padded (the backward GEMMs' operand)
    __nv_bfloat16 *Wt16[kLayers] = {};   // [out x round8(in)] BF16, the K-major operand of the forward GEMMs
    float *mean = nullptr, *stdv = nullptr;  // device [n]
    std::vector<float> hmean, hstd;
    int adamStep = 0;
    // work buffers (grow only): rows of the forward pass, and of the backward
    size_t cap = 0, capBack = 0;
    // inputs [rows x round8(n)] and activations [rows x round8(width)], zero
    // padded; dZ of the layer at hand and of the one below, row stride wp
    __nv_bfloat16 *X = nullptr, *Act[kLayers] = {}, *dZ16[2] = {};
    float *dZ[2] = {};
    int *tcErr = nullptr;       // error word of the tensor-memory GEMM's bounded waits
    bool keepZ = true;          // forward keeps the hidden pre-activations (training)
    float *Z[kLayers] = {}, *T = nullptr, *loss = nullptr;
    // training: the epoch's permutation, the loss partials of kLossSteps steps
    int *perm = nullptr;
    size_t permCap = 0;
    float *lossBuf = nullptr;
    size_t lossCap = 0;
    int *fallbacks = nullptr;
    int *sel = nullptr;         // selected cells (+ their count) of cl_mlp_predict_selected
    size_t selCap = 0;
    cudaStream_t stream = nullptr;
    std::string err;
};

constexpr int kLossSteps = 256;   // training steps between readbacks of the loss

static void mlp_free_back(cl_mlp *m)
{
    cudaFree(m->T);
    cudaFree(m->loss);
    m->T = m->loss = nullptr;
    for (int h = 0; h < 2; h++) {
        cudaFree(m->dZ16[h]);
        cudaFree(m->dZ[h]);
        m->dZ16[h] = nullptr;
        m->dZ[h] = nullptr;
    }
    m->capBack = 0;
}

static void mlp_free_work(cl_mlp *m)
{
    mlp_free_back(m);
    cudaFree(m->X);
    m->X = nullptr;
    for (int l = 0; l < kLayers; l++) {
        cudaFree(m->Act[l]);
        cudaFree(m->Z[l]);
        m->Act[l] = nullptr;
        m->Z[l] = nullptr;
    }
    m->cap = 0;
}

// padding columns are zero: they are operands of the GEMMs.  Those of X and Act
// keep their place and stay as filled; dZ16 holds matrices of several strides
// in turn, whose writers fill their padding.
template <class T>
static bool mlp_zeroed(T **p, size_t cnt)
{
    return cudaMalloc(p, cnt * sizeof(T)) == cudaSuccess && cudaMemset(*p, 0, cnt * sizeof(T)) == cudaSuccess;
}

// Work buffers for `rows` rows; those of the backward pass (a third of the
// whole, 0.8 GB at 131072 x 512) only where it runs.
static int mlp_reserve(cl_mlp *m, size_t rows, bool back)
{
    const size_t w = (size_t)(m->width > m->n ? m->width : m->n), wp = (size_t)round8((int)w);
    const bool grow = rows > m->cap, growBack = back && rows > m->capBack;
    bool ok = true;
    if (grow) {
        mlp_free_work(m);
        ok = mlp_zeroed(&m->X, rows * round8(m->n));
        for (int l = 0; l < kLayers && ok; l++)
            ok = mlp_zeroed(&m->Act[l], rows * wp) && cudaMalloc(&m->Z[l], rows * w * sizeof(float)) == cudaSuccess;
    }
    if (growBack && ok) {
        mlp_free_back(m);
        ok = cudaMalloc(&m->T, rows * m->n * sizeof(float)) == cudaSuccess &&
             cudaMalloc(&m->loss, (rows * m->n / 256 + 2) * sizeof(float)) == cudaSuccess;
        for (int h = 0; h < 2 && ok; h++)
            ok = mlp_zeroed(&m->dZ16[h], rows * wp) && mlp_zeroed(&m->dZ[h], rows * wp);
    }
    if (!grow && !growBack)
        return CL_OK;
    ok = ok && cudaDeviceSynchronize() == cudaSuccess;   // the fills, before work on other streams
    if (!ok) {
        mlp_free_work(m);
        m->err = "MLP work buffer allocation failed";
        return CL_ERR_CUDA;
    }
    if (grow)
        m->cap = rows;
    if (growBack)
        m->capBack = rows;
    return CL_OK;
}

// forward over `rows` inputs already in m->X (with Mdev: min(rows, *Mdev -
// moff) of them); output pre-activations in Z[3]
//
// The layer GEMMs run on the tensor-memory path (tcgen05, tc_gemm.cuh): the
// input padded to round8(n) columns, the weights as K-major BF16 copies.
static cudaError_t mlp_forward(cl_mlp *m, int rows, const int *Mdev = nullptr, int moff = 0)
{
    cudaError_t e = cudaSuccess;
    const __nv_bfloat16 *in = m->X;
    for (int l = 0; l < kLayers && e == cudaSuccess; l++) {
        const int K = round8(m->dims[l]), N = m->dims[l + 1];
        if (l < kLayers - 1)
            e = tc_gemm<clb::tc::EPI_BIAS_GELU>(in, m->Wt16[l], rows, N, K, m->keepZ ? m->Z[l] : nullptr, m->b[l],
                                                 m->Act[l], round8(N), Mdev, moff, m->tcErr, m->stream);
        else
            e = tc_gemm<clb::tc::EPI_BIAS>(in, m->Wt16[l], rows, N, K, m->Z[l], m->b[l], nullptr, 0, Mdev, moff,
                                            m->tcErr, m->stream);
        in = m->Act[l];
    }
    return e;
}

static cudaError_t mlp_sync_weights(cl_mlp *m)
{
    for (int l = 0; l < kLayers; l++) {
        const int K = m->dims[l], N = m->dims[l + 1], Kp = round8(K), ldw = round8(N);
        cast_bf16_kernel<<<blocks((size_t)K * ldw), 256, 0, m->stream>>>(m->W[l], K, N, ldw, m->W16[l]);
        transpose_cast_kernel<<<blocks((size_t)N * Kp), 256, 0, m->stream>>>(m->W[l], K, N, Kp, m->Wt16[l]);
    }
    return cudaGetLastError();
}

static int loss_parts(const cl_mlp *m, int rows) { return blocks((size_t)rows * m->n); }

static float loss_value(const float *part, int parts, int total)
{
    double s = 0;
    for (int i = 0; i < parts; i++)
        s += part[i];
    return (float)(s / total);
}

// backward of the MSE loss for the batch in X/T; gradients into gW/gb, the
// loss partials (loss_parts of them) into `loss`
static cudaError_t mlp_backward(cl_mlp *m, int rows, float *loss)
{
    const int n = m->n, total = rows * n;
    // on the current device, whichever it is
    cudaError_t e = cudaFuncSetAttribute(backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kBackSmem);
    if (e != cudaSuccess)
        return e;
    mse_grad_kernel<<<loss_parts(m, rows), 256, 0, m->stream>>>(m->Z[kLayers - 1], m->T, m->dZ16[0], m->dZ[0], total, n,
                                                                round8(n), 1.0f / (float)total, loss);
    e = cudaGetLastError();
    for (int l = kLayers - 1, h = 0; l >= 0 && e == cudaSuccess; l--, h ^= 1) {
        BackArgs a;
        a.rows = rows;
        a.K = m->dims[l];
        a.N = m->dims[l + 1];
        a.in = (l == 0) ? m->X : m->Act[l - 1];
        a.ldin = round8(a.K);
        a.dZ = m->dZ16[h];
        a.dZf = m->dZ[h];
        a.ldz = a.ldw = round8(a.N);
        a.W = m->W16[l];
        a.Zprev = (l > 0) ? m->Z[l - 1] : nullptr;
        a.gW = m->gW[l];
        a.gb = m->gb[l];
        a.dZnext = m->dZ16[h ^ 1];
        a.dZfnext = m->dZ[h ^ 1];
        a.ldn = round8(a.K);
        auto tiles = [](int M, int N) { return ((M + 63) / 64) * ((N + 63) / 64); };
        a.tilesW = tiles(a.K, a.N);
        a.tilesB = (a.N + 31) / 32;
        const int grid = a.tilesW + a.tilesB + (l > 0 ? tiles(rows, a.K) : 0);
        backward_kernel<<<grid, 256, kBackSmem, m->stream>>>(a);
        e = cudaGetLastError();
    }
    return e;
}

// The tensor-memory GEMM's error word (a bounded wait that gave up), read
// after the stream has been synchronised, and cleared.
static int tc_error(cl_mlp *m)
{
    int h = 0;
    if (cudaMemcpy(&h, m->tcErr, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess)
        return CL_ERR_CUDA;
    if (h != 0) {
        cudaMemset(m->tcErr, 0, sizeof(int));
        clb::uploads_arrived();
        m->err = "tensor-memory GEMM: a bounded wait timed out";
        return CL_ERR_TIMEOUT;
    }
    return CL_OK;
}

extern "C" {

int cl_mlp_create(int n, int width, int moment_type, double delta_ppn, unsigned long long seed, cl_mlp **out)
{
    if (!out || n < 1 || n > 32 || width < 8 || width > 4096)
        return CL_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev < 1)
        return CL_ERR_CUDA;
    cl_mlp *m = new cl_mlp();
    m->n = n;
    m->width = width;
    m->momentType = moment_type;
    m->delta = delta_ppn;
    m->dims[0] = n;
    m->dims[1] = m->dims[2] = m->dims[3] = width;
    m->dims[4] = n;
    cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking);
    std::mt19937_64 rng(seed);
    bool ok = true;
    for (int l = 0; l < kLayers && ok; l++) {
        size_t cnt = (size_t)m->dims[l] * m->dims[l + 1];
        int N = m->dims[l + 1];
        // He-style uniform init scaled by fan-in
        std::uniform_real_distribution<float> U(-1.0f, 1.0f);
        float sc = std::sqrt(3.0f / (float)m->dims[l]);
        std::vector<float> w(cnt), z(cnt, 0.0f), bz(N, 0.0f);
        for (auto &v : w)
            v = U(rng) * sc;
        ok = cudaMalloc(&m->W[l], cnt * 4) == cudaSuccess && cudaMalloc(&m->mW[l], cnt * 4) == cudaSuccess &&
             cudaMalloc(&m->vW[l], cnt * 4) == cudaSuccess && cudaMalloc(&m->gW[l], cnt * 4) == cudaSuccess &&
             cudaMalloc(&m->W16[l], (size_t)m->dims[l] * round8(N) * 2) == cudaSuccess &&
             cudaMalloc(&m->Wt16[l], (size_t)N * round8(m->dims[l]) * 2) == cudaSuccess &&
             cudaMalloc(&m->b[l], N * 4) == cudaSuccess &&
             cudaMalloc(&m->mb[l], N * 4) == cudaSuccess && cudaMalloc(&m->vb[l], N * 4) == cudaSuccess &&
             cudaMalloc(&m->gb[l], N * 4) == cudaSuccess;
        if (ok) {
            cudaMemcpy(m->W[l], w.data(), cnt * 4, cudaMemcpyHostToDevice);
            cudaMemcpy(m->mW[l], z.data(), cnt * 4, cudaMemcpyHostToDevice);
            cudaMemcpy(m->vW[l], z.data(), cnt * 4, cudaMemcpyHostToDevice);
            cudaMemcpy(m->b[l], bz.data(), N * 4, cudaMemcpyHostToDevice);
            cudaMemcpy(m->mb[l], bz.data(), N * 4, cudaMemcpyHostToDevice);
            cudaMemcpy(m->vb[l], bz.data(), N * 4, cudaMemcpyHostToDevice);
        }
    }
    ok = ok && cudaMalloc(&m->mean, n * 4) == cudaSuccess && cudaMalloc(&m->stdv, n * 4) == cudaSuccess &&
         cudaMalloc(&m->fallbacks, sizeof(int)) == cudaSuccess && cudaMalloc(&m->tcErr, sizeof(int)) == cudaSuccess &&
         cudaMemset(m->tcErr, 0, sizeof(int)) == cudaSuccess;
    if (!ok) {
        cl_mlp_destroy(m);
        return CL_ERR_CUDA;
    }
    m->hmean.assign(n, 0.0f);
    m->hstd.assign(n, 1.0f);
    cudaMemcpy(m->mean, m->hmean.data(), n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(m->stdv, m->hstd.data(), n * 4, cudaMemcpyHostToDevice);
    clb::uploads_arrived();
    mlp_sync_weights(m);
    cudaStreamSynchronize(m->stream);
    *out = m;
    return CL_OK;
}

void cl_mlp_destroy(cl_mlp *m)
{
    if (!m)
        return;
    if (m->stream)
        cudaStreamSynchronize(m->stream);
    for (int l = 0; l < kLayers; l++) {
        cudaFree(m->W[l]);
        cudaFree(m->b[l]);
        cudaFree(m->mW[l]);
        cudaFree(m->vW[l]);
        cudaFree(m->mb[l]);
        cudaFree(m->vb[l]);
        cudaFree(m->gW[l]);
        cudaFree(m->gb[l]);
        cudaFree(m->W16[l]);
        cudaFree(m->Wt16[l]);
    }
    mlp_free_work(m);
    cudaFree(m->perm);
    cudaFree(m->lossBuf);
    cudaFree(m->mean);
    cudaFree(m->stdv);
    cudaFree(m->fallbacks);
    cudaFree(m->tcErr);
    cudaFree(m->sel);
    if (m->stream)
        cudaStreamDestroy(m->stream);
    delete m;
}

const char *cl_mlp_last_error(const cl_mlp *m) { return m ? m->err.c_str() : ""; }

// Standardisation of the targets (per-component mean and std, host arrays).
int cl_mlp_set_output_scaling(cl_mlp *m, const float *mean, const float *stdv)
{
    if (!m || !mean || !stdv)
        return CL_ERR_ARG;
    m->hmean.assign(mean, mean + m->n);
    m->hstd.assign(stdv, stdv + m->n);
    cudaMemcpy(m->mean, mean, m->n * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(m->stdv, stdv, m->n * 4, cudaMemcpyHostToDevice);
    return clb::uploads_arrived() == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

// Adam training on pairs (u, alpha) held on the device ([count x n] FP64).
// Minibatches are consecutive slices of a shuffled index order drawn on the
// host; losses[steps] (nullable) receives the batch loss per step.
int cl_mlp_train(cl_mlp *m, const double *d_u, const double *d_alpha, int count, int steps, int batch, float lr,
                 unsigned long long seed, float *losses)
{
    if (!m || !d_u || !d_alpha || count < batch || batch < 1 || steps < 0)
        return CL_ERR_ARG;
    int rc = mlp_reserve(m, batch, true);
    if (rc)
        return rc;
    const int n = m->n, np = round8(n), parts = loss_parts(m, batch);
    auto grow = [](auto **p, size_t &cap, size_t cnt) {
        if (cnt <= cap)
            return true;
        cudaFree(*p);
        *p = nullptr;
        cap = 0;
        if (cudaMalloc(p, cnt * sizeof(**p)) != cudaSuccess)
            return false;
        cap = cnt;
        return true;
    };
    if (!grow(&m->perm, m->permCap, (size_t)count) || !grow(&m->lossBuf, m->lossCap, (size_t)kLossSteps * parts)) {
        m->err = "minibatch allocation failed";
        return CL_ERR_CUDA;
    }
    std::mt19937_64 rng(seed);
    std::vector<int> order(count);
    for (int i = 0; i < count; i++)
        order[i] = i;
    std::vector<float> hloss(losses ? (size_t)kLossSteps * parts : 0);
    int pos = count;
    UpdateArgs up;
    int first = 0, biases = 0;
    for (int l = 0; l < kLayers; l++) {
        up.W[l] = m->W[l];
        up.mW[l] = m->mW[l];
        up.vW[l] = m->vW[l];
        up.gW[l] = m->gW[l];
        up.b[l] = m->b[l];
        up.mb[l] = m->mb[l];
        up.vb[l] = m->vb[l];
        up.gb[l] = m->gb[l];
        up.W16[l] = m->W16[l];
        up.Wt16[l] = m->Wt16[l];
        up.dims[l] = m->dims[l];
        up.first[l] = first;
        first += ((m->dims[l] + 31) / 32) * ((m->dims[l + 1] + 31) / 32);
        biases += m->dims[l + 1];
    }
    up.dims[kLayers] = m->dims[kLayers];
    up.first[kLayers] = first;
    up.b1 = 0.9f;
    up.b2 = 0.999f;
    up.eps = 1e-8f;
    cudaError_t e = cudaSuccess;
    for (int s = 0; s < steps && e == cudaSuccess; s++) {
        if (pos + batch > count) {
            // new epoch: a fresh permutation of the training pairs, drawn while
            // the device works on the steps already queued (the copy from
            // pageable memory returns once the source has been read)
            std::shuffle(order.begin(), order.end(), rng);
            e = cudaMemcpyAsync(m->perm, order.data(), (size_t)count * sizeof(int), cudaMemcpyHostToDevice, m->stream);
            pos = 0;
        }
        prep_kernel<<<blocks((size_t)batch * n), 256, 0, m->stream>>>(d_u, d_alpha, m->perm + pos, batch, n, np,
                                                                     m->momentType, m->mean, m->stdv, m->X, m->T);
        pos += batch;
        if (e == cudaSuccess)
            e = mlp_forward(m, batch);
        const int slot = s % kLossSteps;
        if (e == cudaSuccess)
            e = mlp_backward(m, batch, m->lossBuf + (size_t)slot * parts);
        m->adamStep++;
        up.c1 = 1.0f - std::pow(up.b1, (float)m->adamStep);
        up.c2 = 1.0f - std::pow(up.b2, (float)m->adamStep);
        up.lr = (s >= steps - steps / 5) ? 0.1f * lr : lr;   // step decay for the last fifth
        if (e == cudaSuccess) {
            update_kernel<<<first + (biases + 255) / 256, 256, 0, m->stream>>>(up);
            e = cudaGetLastError();
        }
        // the loss comes back every kLossSteps steps, not every step
        if (losses && e == cudaSuccess && (slot == kLossSteps - 1 || s == steps - 1)) {
            e = cudaMemcpyAsync(hloss.data(), m->lossBuf, (size_t)(slot + 1) * parts * sizeof(float),
                                cudaMemcpyDeviceToHost, m->stream);
            if (e == cudaSuccess)
                e = cudaStreamSynchronize(m->stream);
            for (int k = 0; k <= slot && e == cudaSuccess; k++)
                losses[s - slot + k] = loss_value(&hloss[(size_t)k * parts], parts, batch * n);
        }
    }
    const cudaError_t es = cudaStreamSynchronize(m->stream);
    if (e == cudaSuccess)
        e = es;
    if (e != cudaSuccess) {
        m->err = std::string("training: ") + cudaGetErrorString(e);
        return CL_ERR_CUDA;
    }
    return tc_error(m);
}

// Predicted multipliers for count vectors d_u (device, [count x n]) written to
// d_alpha; non-finite predictions keep d_alpha (fallback_kind 0, e.g. the
// previous stage) or take the isotropic multiplier (fallback_kind 1).
// *fallbacks (nullable) receives how many vectors fell back.
int cl_mlp_predict(cl_mlp *m, const double *d_u, double *d_alpha, int count, int fallback_kind, int *fallbacks,
                   void *stream)
{
    if (!m || !d_u || !d_alpha || count < 0)
        return CL_ERR_ARG;
    if (count == 0)
        return CL_OK;
    cudaStream_t st = stream ? (cudaStream_t)stream : m->stream;
    const int chunk = 1 << 18;
    int rc = mlp_reserve(m, count < chunk ? count : chunk, false);
    if (rc)
        return rc;
    cudaStream_t keep = m->stream;
    m->stream = st;
    cudaError_t e = cudaMemsetAsync(m->fallbacks, 0, sizeof(int), st);
    for (int c0 = 0; c0 < count && e == cudaSuccess; c0 += chunk) {
        int rows = count - c0 < chunk ? count - c0 : chunk;
        prep_kernel<<<blocks((size_t)rows * m->n), 256, 0, st>>>(d_u + (size_t)c0 * m->n, nullptr, nullptr, rows, m->n,
                                                                round8(m->n), m->momentType, m->mean, m->stdv, m->X,
                                                                nullptr);
        m->keepZ = false;
        e = mlp_forward(m, rows);
        m->keepZ = true;
        predict_out_kernel<<<blocks(rows), 256, 0, st>>>(m->Z[kLayers - 1], d_u + (size_t)c0 * m->n,
                                                         d_alpha + (size_t)c0 * m->n, rows, m->n, m->momentType,
                                                         m->delta, m->mean, m->stdv, fallback_kind, m->fallbacks);
    }
    m->stream = keep;
    if (fallbacks && e == cudaSuccess) {
        e = cudaMemcpyAsync(fallbacks, m->fallbacks, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess)
            e = cudaStreamSynchronize(st);
    }
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e != cudaSuccess) {
        m->err = std::string("predict: ") + cudaGetErrorString(e);
        return CL_ERR_CUDA;
    }
    return CL_OK;
}

// Predicted starts only for the cells whose last optimisation took at least
// min_iters iterations (d_iters, device [count]); the other cells' starts are
// NaN, so the Newton kernel starts them from their previous-stage
// multipliers.  The selection is compacted on the device and the network runs
// over it in chunks whose row counts the GEMMs read from device memory, so
// the call needs no host synchronisation and can be captured in a graph.
int cl_mlp_predict_selected(cl_mlp *m, const double *d_u, const int *d_iters, int min_iters, double *d_alpha,
                            int count, void *stream)
{
    if (!m || !d_u || !d_iters || !d_alpha || count < 0 || min_iters < 1)
        return CL_ERR_ARG;
    if (count == 0)
        return CL_OK;
    cudaStream_t st = stream ? (cudaStream_t)stream : m->stream;
    const int chunk = 1 << 18;
    int rc = mlp_reserve(m, count < chunk ? count : chunk, false);
    if (rc)
        return rc;
    if (!m->sel || m->selCap < (size_t)count) {
        cudaFree(m->sel);
        m->sel = nullptr;
        if (cudaMalloc(&m->sel, ((size_t)count + 1) * sizeof(int)) != cudaSuccess) {
            m->err = "selection buffer";
            return CL_ERR_CUDA;
        }
        m->selCap = count;
    }
    int *cnt = m->sel + count;
    cudaStream_t keep = m->stream;
    m->stream = st;
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int), st);
    if (e == cudaSuccess)
        e = cudaMemsetAsync(m->fallbacks, 0, sizeof(int), st);
    select_kernel<<<blocks(count), 256, 0, st>>>(d_iters, count, min_iters, m->sel, cnt, d_alpha, m->n);
    for (int c0 = 0; c0 < count && e == cudaSuccess; c0 += chunk) {
        const int rows = count - c0 < chunk ? count - c0 : chunk;
        prep_idx_kernel<<<blocks((size_t)rows * m->n), 256, 0, st>>>(d_u, m->sel, cnt, c0, rows, m->n, round8(m->n),
                                                                    m->X);
        m->keepZ = false;
        e = mlp_forward(m, rows, cnt, c0);
        m->keepZ = true;
        predict_out_kernel<<<blocks(rows), 256, 0, st>>>(m->Z[kLayers - 1], d_u, d_alpha, rows, m->n, m->momentType,
                                                         m->delta, m->mean, m->stdv, 2, m->fallbacks, m->sel, cnt,
                                                         c0);
    }
    m->stream = keep;
    if (e == cudaSuccess)
        e = cudaGetLastError();
    if (e != cudaSuccess) {
        m->err = std::string("selected predict: ") + cudaGetErrorString(e);
        return CL_ERR_CUDA;
    }
    return CL_OK;
}

// The network's GEMM on its own (device pointers): C [M x N] FP32 = A [M x K]
// . B [N x K]^T with BF16 A, B (row-major, K a multiple of 8).  Waits for the
// result; for the numerics test of the tensor-memory path.
int cl_tc_gemm_bf16(const void *d_A, const void *d_B, int M, int N, int K, float *d_C)
{
    if (!d_A || !d_B || !d_C || M < 1 || N < 1 || K < 8 || K % 8 != 0)
        return CL_ERR_ARG;
    int *err = nullptr;
    if (cudaMalloc(&err, sizeof(int)) != cudaSuccess)
        return CL_ERR_CUDA;
    cudaMemset(err, 0, sizeof(int));
    cudaError_t e = tc_gemm<clb::tc::EPI_STORE>((const __nv_bfloat16 *)d_A, (const __nv_bfloat16 *)d_B, M, N, K, d_C,
                                                 nullptr, nullptr, 0, nullptr, 0, err, nullptr);
    if (e == cudaSuccess)
        e = cudaDeviceSynchronize();
    int h = 0;
    if (e == cudaSuccess)
        e = cudaMemcpy(&h, err, sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(err);
    if (e != cudaSuccess)
        return CL_ERR_CUDA;
    return h ? CL_ERR_TIMEOUT : CL_OK;
}

// Gradient check support: loss and parameter gradients of one batch (host
// FP64 inputs), copied to host buffers grads[l] = {dW_l [in x out], db_l}.
int cl_mlp_loss_and_grads(cl_mlp *m, const double *u, const double *alpha, int rows, float *loss, float *const *gW,
                          float *const *gb)
{
    if (!m || !u || !alpha || rows < 1)
        return CL_ERR_ARG;
    int rc = mlp_reserve(m, rows, true);
    if (rc)
        return rc;
    const int n = m->n;
    double *bu = nullptr, *ba = nullptr;
    cudaMalloc(&bu, (size_t)rows * n * 8);
    cudaMalloc(&ba, (size_t)rows * n * 8);
    cudaMemcpy(bu, u, (size_t)rows * n * 8, cudaMemcpyHostToDevice);
    cudaMemcpy(ba, alpha, (size_t)rows * n * 8, cudaMemcpyHostToDevice);
    clb::order_after_uploads(m->stream);
    prep_kernel<<<blocks((size_t)rows * n), 256, 0, m->stream>>>(bu, ba, nullptr, rows, n, round8(n), m->momentType,
                                                                m->mean, m->stdv, m->X, m->T);
    cudaError_t e = mlp_forward(m, rows);
    if (e == cudaSuccess)
        e = mlp_backward(m, rows, m->loss);
    std::vector<float> part(loss_parts(m, rows));
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(part.data(), m->loss, sizeof(float) * part.size(), cudaMemcpyDeviceToHost, m->stream);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(m->stream);
    if (loss && e == cudaSuccess)
        *loss = loss_value(part.data(), (int)part.size(), rows * n);
    for (int l = 0; l < kLayers && e == cudaSuccess; l++) {
        size_t cnt = (size_t)m->dims[l] * m->dims[l + 1];
        if (gW && gW[l])
            e = cudaMemcpy(gW[l], m->gW[l], cnt * 4, cudaMemcpyDeviceToHost);
        if (gb && gb[l] && e == cudaSuccess)
            e = cudaMemcpy(gb[l], m->gb[l], m->dims[l + 1] * 4, cudaMemcpyDeviceToHost);
    }
    cudaFree(bu);
    cudaFree(ba);
    if (e != cudaSuccess) {
        m->err = std::string("loss/grad: ") + cudaGetErrorString(e);
        return CL_ERR_CUDA;
    }
    return tc_error(m);
}

// Parameters: W_l is [in x out] row-major (y = x W + b).  get/set copy FP32
// masters; set also refreshes the BF16 copies.
int cl_mlp_get_params(cl_mlp *m, float *const *W, float *const *b)
{
    if (!m)
        return CL_ERR_ARG;
    cudaStreamSynchronize(m->stream);
    for (int l = 0; l < kLayers; l++) {
        if (W && W[l])
            cudaMemcpy(W[l], m->W[l], (size_t)m->dims[l] * m->dims[l + 1] * 4, cudaMemcpyDeviceToHost);
        if (b && b[l])
            cudaMemcpy(b[l], m->b[l], m->dims[l + 1] * 4, cudaMemcpyDeviceToHost);
    }
    return CL_OK;
}

int cl_mlp_set_params(cl_mlp *m, float *const *W, float *const *b)
{
    if (!m)
        return CL_ERR_ARG;
    for (int l = 0; l < kLayers; l++) {
        if (W && W[l])
            cudaMemcpy(m->W[l], W[l], (size_t)m->dims[l] * m->dims[l + 1] * 4, cudaMemcpyHostToDevice);
        if (b && b[l])
            cudaMemcpy(m->b[l], b[l], m->dims[l + 1] * 4, cudaMemcpyHostToDevice);
    }
    clb::uploads_arrived();
    mlp_sync_weights(m);
    return cudaStreamSynchronize(m->stream) == cudaSuccess ? CL_OK : CL_ERR_CUDA;
}

}  // extern "C"

// Reserves inference buffers ahead of stream capture (used by the grid solver).
int clb_mlp_reserve_for(cl_mlp *m, size_t rows)
{
    const size_t chunk = 1 << 18;
    return mlp_reserve(m, rows < chunk ? rows : chunk, false);
}
