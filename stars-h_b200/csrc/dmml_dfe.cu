// TLR-by-dense product and Frobenius error on the device.
//
// dmml: B = alpha M A + beta B (reference src/backends/sequential/blrm/
// dmml.c:16-145: per far block T = V^T A[cols], B[rows] += U T, near
// blocks dense).  Here every T of one input block column comes from one
// GEMM over the concatenated right factors, and every block row
// accumulates sum_b U_b T_b + sum_near D_b A[cols] in one GEMM whose K runs
// over the row's concatenated left factors and near blocks, so no two CTAs
// write the same rows and the sum order is fixed (deterministic).  For
// symm == 'S' the transposed contribution of every off-diagonal block is
// added to the mirrored block row, as the reference does (:78-87, :111-117).
//
// dfe: ||A - M||_F / ||A||_F with every block regenerated in FP64
// (reference src/backends/sequential/blrm/dfe.c:16-134); off-diagonal
// blocks of a symmetric format count twice.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include "device_ctx.cuh"
#include "engine.cuh"
#include "records.cuh"
#include "smem_limit.cuh"
#include "starsh-b200.h"

namespace b200 {

__device__ __forceinline__ void dmma_884(double &c0, double &c1, double a,
                                         double b)
{
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
        "{%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// ------------------------------------------------------ product kernels
//
// B = alpha M A as two long GEMMs instead of one small GEMM per block.
// Phase 1, per input block column j: the rows of T are the columns of all
// right factors V_p that multiply A_j (far block p, or its mirror in a
// symmetric format), T(rho, :) = V_p(:, c)^T A_j -- M runs over the
// concatenated factor columns, K over the block column's rows.  Phase 2,
// per output block row i: B_i += [U_p1 U_p2 ...] [T_p1; T_p2; ...] +
// sum_near op(D_b) A_j -- K runs over the concatenated left-factor columns
// of the row, then over the near blocks' columns.  T is written by phase 1
// straight into the row-ordered layout phase 2 reads: block row i's rows
// of T form one column-major (S_i x nrhs) matrix, S_i = sum of the row's
// ranks.  Each output element is written by one CTA, its sum in a fixed
// order (deterministic).
//
// CTA tile 64 x BN (BN = 16 FN), 8 warps of FP64 mma.sync m8n8k4 fragments;
// K steps of 16 through a three-stage cp.async pipeline.  Shared-memory layouts are chosen so that the
// fragment reads and the copies are free of bank conflicts: B as [n][k]
// (row stride 20 doubles); A as [m][k] (stride 20) in phase 1, whose
// operand is contiguous along k in global memory, and as [k][m] (stride
// 68) in phase 2, whose operand is contiguous along m.

struct RowT {          // where phase 1 writes row rho of T
    long long base;    // first T row of the output block row (P_i)
    int kappa;         // row within the block row's T_i
    int ld;            // rows of T_i (S_i)
};

struct Job1 {          // phase 1: up to 128 rows of T that share A_j
    int rho0, rows;
    int K;             // rows of A_j
    long long in0;     // first row of A_j in A
};

struct NearPiece {
    long long off;     // its D, doubles after the first near block's
    int trans;         // 1: the mirrored block of a symmetric format
    int K;             // columns of op(D)
    int ld;            // leading dimension of D
    long long in0;     // first row of the input block in A
};

struct Job2 {          // phase 2: up to 128 rows of one output block row
    long long out0;    // first output row
    int m0, rows;      // rows m0 .. m0 + rows - 1 of the block row
    long long kap0;    // P_i (first concatenated column of the row)
    int kfar;          // S_i
    int near0, near1;  // the row's near pieces
};

constexpr int kPBM = 128, kPBK = 16, kPStages = 3;
constexpr int kPRows = 64;             // rows of a CTA
constexpr int kPAStage = kPRows * 20;  // phase 1

template <int FN>
constexpr int prod_stage_doubles() { return kPAStage + 20 * 16 * FN; }

__device__ __forceinline__ void cp_async8(double *dst, const double *src,
                                          bool ok)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(d),
                 "l"(src), "r"(ok ? 8 : 0));
}

__device__ __forceinline__ void cp_async_commit()
{
    asm volatile("cp.async.commit_group;\n" ::);
}

__device__ __forceinline__ void cp_async_wait_stages()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kPStages - 2));
}

// acc += A_stage B_stage for one K step: MI x NJ fragments of the warp at
// (wm, wn); A stored as [k][m] with stride LDA, or (LDA = 0) as [m][k].
template <int MI, int NJ, int LDA>
__device__ __forceinline__ void prod_step(const double *As, const double *Bs,
                                          double (&acc)[MI][NJ][2], int wm,
                                          int wn, int g, int tig)
{
    #pragma unroll
    for (int kk = 0; kk < kPBK; kk += 4) {
        double af[MI], bf[NJ];
        #pragma unroll
        for (int i = 0; i < MI; ++i)
            af[i] = LDA ? As[(kk + tig) * LDA + wm + 8 * i + g]
                        : As[(wm + 8 * i + g) * 20 + kk + tig];
        #pragma unroll
        for (int j = 0; j < NJ; ++j) bf[j] = Bs[(wn + 8 * j + g) * 20 + kk + tig];
        #pragma unroll
        for (int i = 0; i < MI; ++i)
            #pragma unroll
            for (int j = 0; j < NJ; ++j)
                dmma_884(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
    }
}

// Phase 1: 64 of the T rows of one job, columns n0 .. n0 + BN - 1 of the
// right-hand sides.
template <int FN>
__global__ void __launch_bounds__(256, 3)
k_prod_t(const Job1 *__restrict__ jobs, const double *const *__restrict__ vcol,
         const RowT *__restrict__ rowt, const double *__restrict__ A, int lda,
         double *__restrict__ T, int nrhs)
{
    constexpr int BN = 16 * FN;
    constexpr int STAGE = prod_stage_doubles<FN>();
    extern __shared__ double sm[];
    // warps along the rows and the columns, fragments of a warp
    constexpr int WM = FN == 1 ? 4 : 2, MI = kPRows / (8 * WM), NJ = 2 * FN * WM / 8;
    __shared__ const double *rowp[kPRows];
    Job1 jb = jobs[blockIdx.x];
    jb.rho0 += blockIdx.z * kPRows;
    jb.rows = min(kPRows, jb.rows - (int)blockIdx.z * kPRows);
    if (jb.rows <= 0) return;
    const int n0 = blockIdx.y * BN;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int wm = warp % WM * 8 * MI, wn = warp / WM * 8 * NJ;
    for (int r = t; r < kPRows; r += 256)
        rowp[r] = r < jb.rows ? vcol[jb.rho0 + r] : nullptr;
    __syncthreads();
    const int lk = t & 15, lr = t >> 4;
    const double *Aj = A + jb.in0;
    const int steps = (jb.K + kPBK - 1) / kPBK;
    auto issue = [&](int step, int st) {
        double *As = sm + st * STAGE, *Bs = As + kPAStage;
        const int k = step * kPBK + lk;
        const bool kin = k < jb.K;
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            const double *p = rowp[lr + 16 * q];
            const bool ok = kin && p != nullptr;
            cp_async8(As + (lr + 16 * q) * 20 + lk, ok ? p + k : A, ok);
        }
        #pragma unroll
        for (int q = 0; q < FN; ++q) {
            const int col = n0 + lr + 16 * q;
            const bool ok = kin && col < nrhs;
            cp_async8(Bs + (lr + 16 * q) * 20 + lk,
                      ok ? Aj + k + (size_t)col * lda : A, ok);
        }
    };
    double acc[MI][NJ][2] = {};
    #pragma unroll
    for (int s = 0; s < kPStages - 1; ++s) {
        if (s < steps) issue(s, s);
        cp_async_commit();
    }
    for (int s = 0; s < steps; ++s) {
        cp_async_wait_stages();
        __syncthreads();
        if (s + kPStages - 1 < steps)
            issue(s + kPStages - 1, (s + kPStages - 1) % kPStages);
        cp_async_commit();
        const double *As = sm + (s % kPStages) * STAGE;
        prod_step<MI, NJ, 0>(As, As + kPAStage, acc, wm, wn, g, tig);
    }
    #pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int r = wm + 8 * i + g;
        if (r >= jb.rows) continue;
        const RowT rt = rowt[jb.rho0 + r];
        double *out = T + (size_t)nrhs * rt.base + rt.kappa;
        #pragma unroll
        for (int j = 0; j < NJ; ++j)
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = n0 + wn + 8 * j + 2 * tig + h;
                if (col < nrhs) out[(size_t)col * rt.ld] = acc[i][j][h];
            }
    }
}

// *out = alpha v + beta *out (not read when beta is 0).
__device__ __forceinline__ void update(double *out, double alpha, double v,
                                       double beta)
{
    const double old = beta == 0.0 ? 0.0 : beta * *out;
    *out = fma(alpha, v, old);
}

// Phase 2: 64 of a job's rows of one output block row (a block row's K is
// long and uneven: with 128 rows a CTA, N = 32768 left 40 of 148 SMs half
// idle for the whole launch, the DMMA pipe 58 % busy).
constexpr int kPRowsLd = kPRows + 4;
template <int FN>
constexpr int prod_b_stage() { return kPBK * kPRowsLd + 20 * 16 * FN; }

template <int FN>
__global__ void __launch_bounds__(256, 3)
k_prod_b(const Job2 *__restrict__ jobs, const double *const *__restrict__ ucol,
         const double *__restrict__ T, int nrhs,
         const NearPiece *__restrict__ near, const double *__restrict__ nearD,
         const double *__restrict__ A, int lda, double *__restrict__ B, int ldb,
         double alpha, double beta)
{
    constexpr int BN = 16 * FN;
    constexpr int STAGE = prod_b_stage<FN>(), AST = kPBK * kPRowsLd;
    // warps along the rows and the columns, fragments of a warp
    constexpr int WM = FN == 1 ? 4 : 2, MI = kPRows / (8 * WM), NJ = 2 * FN * WM / 8;
    extern __shared__ double sm[];
    Job2 jb = jobs[blockIdx.x];
    jb.m0 += blockIdx.z * kPRows;
    jb.rows = min(kPRows, jb.rows - (int)blockIdx.z * kPRows);
    if (jb.rows <= 0) return;
    jb.out0 += blockIdx.z * kPRows;
    const int n0 = blockIdx.y * BN;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int wm = warp % WM * 8 * MI, wn = warp / WM * 8 * NJ;
    // A copies: row am and columns ak + 4 q (q < 4) of the step;
    // B copies: column lk of the step, right-hand sides lr + 16 q
    const int am = t & 63, ak = t >> 6;
    const int lk = t & 15, lr = t >> 4;
    const double *Tf = T + (size_t)nrhs * jb.kap0;
    int total = (jb.kfar + kPBK - 1) / kPBK;
    for (int q = jb.near0; q < jb.near1; ++q) total += (near[q].K + kPBK - 1) / kPBK;
    // issue position: piece (-1: the factors, else a near piece) and k0
    int piece = jb.kfar > 0 ? -1 : jb.near0, k0 = 0;
    const double *up[4];            // factor columns of the next far step
    auto fetch_ptrs = [&]() {
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int kap = k0 + ak + 4 * q;
            up[q] = piece < 0 && kap < jb.kfar ? ucol[jb.kap0 + kap] : nullptr;
        }
    };
    auto advance = [&]() {
        k0 += kPBK;
        const int K = piece < 0 ? jb.kfar : near[piece].K;
        if (k0 >= K) {
            piece = piece < 0 ? jb.near0 : piece + 1;
            k0 = 0;
        }
        fetch_ptrs();
    };
    auto issue = [&](int st) {
        double *As = sm + st * STAGE, *Bs = As + AST;
        if (piece < 0) {
            #pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool ok = up[q] != nullptr && am < jb.rows;
                cp_async8(As + (ak + 4 * q) * kPRowsLd + am,
                          ok ? up[q] + jb.m0 + am : A, ok);
            }
            #pragma unroll
            for (int q = 0; q < FN; ++q) {
                const int col = n0 + lr + 16 * q, kap = k0 + lk;
                const bool ok = kap < jb.kfar && col < nrhs;
                cp_async8(Bs + (lr + 16 * q) * 20 + lk,
                          ok ? Tf + kap + (size_t)col * jb.kfar : A, ok);
            }
        } else {
            const NearPiece np = near[piece];
            const double *D = nearD + np.off;
            #pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int kap = k0 + ak + 4 * q;
                const bool ok = kap < np.K && am < jb.rows;
                const size_t off = np.trans
                    ? (size_t)kap + (size_t)(jb.m0 + am) * np.ld
                    : (size_t)(jb.m0 + am) + (size_t)kap * np.ld;
                cp_async8(As + (ak + 4 * q) * kPRowsLd + am, ok ? D + off : A, ok);
            }
            #pragma unroll
            for (int q = 0; q < FN; ++q) {
                const int col = n0 + lr + 16 * q, kap = k0 + lk;
                const bool ok = kap < np.K && col < nrhs;
                cp_async8(Bs + (lr + 16 * q) * 20 + lk,
                          ok ? A + np.in0 + kap + (size_t)col * lda : A, ok);
            }
        }
    };
    fetch_ptrs();
    double acc[MI][NJ][2] = {};
    #pragma unroll
    for (int s = 0; s < kPStages - 1; ++s) {
        if (s < total) {
            issue(s);
            advance();
        }
        cp_async_commit();
    }
    for (int s = 0; s < total; ++s) {
        cp_async_wait_stages();
        __syncthreads();
        if (s + kPStages - 1 < total) {
            issue((s + kPStages - 1) % kPStages);
            advance();
        }
        cp_async_commit();
        const double *As = sm + (s % kPStages) * STAGE;
        prod_step<MI, NJ, kPRowsLd>(As, As + AST, acc, wm, wn, g, tig);
    }
    #pragma unroll
    for (int i = 0; i < MI; ++i) {
        const int m = wm + 8 * i + g;
        if (m >= jb.rows) continue;
        double *out = B + jb.out0 + m;
        #pragma unroll
        for (int j = 0; j < NJ; ++j)
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int col = n0 + wn + 8 * j + 2 * tig + h;
                if (col < nrhs) update(out + (size_t)col * ldb, alpha, acc[i][j][h], beta);
            }
    }
}

template <int FN>
static void launch_products(const Job1 *j1, int n1, const double *const *vcol,
                            const RowT *rowt, const Job2 *j2, int n2,
                            const double *const *ucol, const NearPiece *near,
                            const double *nearD, const double *A, int lda,
                            double *T, double *B, int ldb, int nrhs, double alpha,
                            double beta, cudaStream_t s)
{
    constexpr size_t smem = (size_t)kPStages * prod_stage_doubles<FN>() * sizeof(double);
    constexpr size_t smem_b = (size_t)kPStages * prod_b_stage<FN>() * sizeof(double);
    allow_smem<k_prod_t<FN>, smem>();
    allow_smem<k_prod_b<FN>, smem_b>();
    const unsigned ny = (unsigned)((nrhs + 16 * FN - 1) / (16 * FN));
    if (n1 > 0) {
        k_prod_t<FN><<<dim3((unsigned)n1, ny, kPBM / kPRows), 256, smem, s>>>(j1, vcol, rowt, A,
                                                              lda, T, nrhs);
        count_launch();
    }
    if (n2 > 0) {
        k_prod_b<FN><<<dim3((unsigned)n2, ny, kPBM / kPRows), 256, smem_b, s>>>(
            j2, ucol, T, nrhs, near, nearD, A, lda, B, ldb, alpha, beta);
        count_launch();
    }
}

// ------------------------------------------------ a few right-hand sides
//
// With up to kGemvRhs columns the product is bound by the read of the
// factors, and the tiles above spend their 16 columns on padding and their
// steps on 256-thread barriers (N = 25600 symmetric, one column: 39 + 68
// us, here 35 + 51; N = 10000 with many dense blocks 35 + 50, here 14 + 39;
// five and more columns are faster there).  Here a thread owns one element of T, or one output row, per column
// and sums it alone; its operands come through a ring of cp.async stages in
// shared memory deep enough to cover the memory latency, private to a warp.
// An FP64 mma.sync adds its four products to the accumulator one after
// another (k = 0, 1, 2, 3, each rounded), so a chain of FMAs over the whole
// K gives the same bits as the tiles above: an iterative solver takes the
// same iterations whichever kernels its products run on.
constexpr int kGemvRhs = 4;
constexpr int kGvKT = 64;            // phase 1: K of a stage
constexpr int kGvLd = kGvKT + 1;     // ... doubles per row of it
constexpr int kGvRowsT = 64;         // ... rows of T of a CTA
constexpr int kGvStagesT = 3;
constexpr int kGvKB = 32;            // phase 2: K of a stage
constexpr int kGvRowsB = 64;         // ... rows of a CTA
constexpr int kGvThreadsB = 2 * kGvRowsB;   // ... half of them sum, half copy
constexpr int kGvStagesB = 4;
constexpr int kGvAhead = 3;          // ... stages a column pointer is read ahead

// doubles of a stage: operand tile, then the other operand's NR rows
template <int NR>
constexpr int gv_stage_t() { return kGvRowsT * kGvLd + NR * kGvKT; }
template <int NR>
constexpr int gv_stage_b() { return kGvRowsB * kGvKB + NR * kGvKB; }

// Phase 1: a CTA takes 64 rows of T (factor columns); its four warps copy 64
// consecutive k of every row per stage (512 contiguous bytes: 128 left the
// HBM at 1.8 TB/s), two of them own the 64 chains, a row per lane.  The odd
// row stride keeps the lanes' reads on different banks.
template <int NR>
__global__ void __launch_bounds__(128)
k_gemv_t(const Job1 *__restrict__ jobs, const double *const *__restrict__ vcol,
         const RowT *__restrict__ rowt, const double *__restrict__ A, int lda,
         double *__restrict__ T, int nrhs)
{
    extern __shared__ double sm[];
    __shared__ const double *rowp[kGvRowsT];
    const Job1 jb = jobs[blockIdx.x];
    const int r0 = blockIdx.y * kGvRowsT, rows = min(kGvRowsT, jb.rows - r0);
    if (rows <= 0) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t < kGvRowsT) rowp[t] = t < rows ? vcol[jb.rho0 + r0 + t] : nullptr;
    __syncthreads();
    constexpr int STAGE = gv_stage_t<NR>();
    const double *Aj = A + jb.in0;
    const int steps = (jb.K + kGvKT - 1) / kGvKT;
    auto issue = [&](int st) {
        double *S = sm + st % kGvStagesT * STAGE, *X = S + kGvRowsT * kGvLd;
        const int k = st * kGvKT + lane;
        #pragma unroll 4
        for (int q = warp; q < rows; q += 4) {
            const double *p = rowp[q];
            cp_async8(S + q * kGvLd + lane, k < jb.K ? p + k : A, k < jb.K);
            cp_async8(S + q * kGvLd + 32 + lane, k + 32 < jb.K ? p + k + 32 : A,
                      k + 32 < jb.K);
        }
        for (int c = warp; c < NR; c += 4) {
            const double *p = Aj + (size_t)c * lda;
            const bool ok = c < nrhs;
            cp_async8(X + c * kGvKT + lane, ok && k < jb.K ? p + k : A, ok && k < jb.K);
            cp_async8(X + c * kGvKT + 32 + lane, ok && k + 32 < jb.K ? p + k + 32 : A,
                      ok && k + 32 < jb.K);
        }
    };
    double acc[NR] = {};
    #pragma unroll
    for (int p = 0; p < kGvStagesT - 1; ++p) {
        if (p < steps) issue(p);
        cp_async_commit();
    }
    for (int st = 0; st < steps; ++st) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kGvStagesT - 2));
        __syncthreads();               // landed for all; the refilled one is consumed
        if (st + kGvStagesT - 1 < steps) issue(st + kGvStagesT - 1);
        cp_async_commit();
        if (t < kGvRowsT) {
            const double *S = sm + st % kGvStagesT * STAGE, *X = S + kGvRowsT * kGvLd;
            #pragma unroll
            for (int h = 0; h < kGvKT; h += 16) {
                double v[16];
                #pragma unroll
                for (int k = 0; k < 16; ++k) v[k] = S[t * kGvLd + h + k];
                #pragma unroll
                for (int c = 0; c < NR; ++c)
                    #pragma unroll
                    for (int k = 0; k < 16; ++k)
                        acc[c] = fma(v[k], X[c * kGvKT + h + k], acc[c]);
            }
        }
    }
    if (t >= rows) return;
    const RowT rt = rowt[jb.rho0 + r0 + t];
    double *out = T + (size_t)nrhs * rt.base + rt.kappa;
    #pragma unroll
    for (int c = 0; c < NR; ++c)
        if (c < nrhs) out[(size_t)c * rt.ld] = acc[c];
}

// One stage of phase 2, as its copying warps see it.
struct GvStage {
    const double *col;   // lane u: the column at K index u of the stage
    const double *x;     // the other operand there, `ldx` between columns
    int ldx, k, rs;      // K indices in use; doubles between rows of col
};

// The copying and the summing warps meet once a stage, each in a loop of its
// own: a named barrier, which counts threads wherever they arrive from
// (__syncthreads() is one place that all threads of the CTA pass).  Warps
// arrive whole: both loops' conditions are the warp's.
__device__ __forceinline__ void gvb_sync()
{
    asm volatile("barrier.sync.aligned 1, %0;" ::"n"(kGvThreadsB) : "memory");
}

// Phase 2: 64 output rows (K over the row's left-factor columns, then its
// near blocks).  Two warps own the chains, a row per lane, and do nothing
// else; the other two keep the ring filled, their column pointers read
// three stages ahead.
template <int NR>
__global__ void __launch_bounds__(kGvThreadsB)
k_gemv_b(const Job2 *__restrict__ jobs, const double *const *__restrict__ ucol,
         const double *__restrict__ T, int nrhs,
         const NearPiece *__restrict__ near, const double *__restrict__ nearD,
         const double *__restrict__ A, int lda, double *__restrict__ B, int ldb,
         double alpha, double beta)
{
    extern __shared__ __align__(16) double gvb_sm[];
    const Job2 jb = jobs[blockIdx.x];
    const int r0 = blockIdx.y * kGvRowsB, rows = min(kGvRowsB, jb.rows - r0);
    if (rows <= 0) return;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    constexpr int STAGE = gv_stage_b<NR>();
    int total = (jb.kfar + kGvKB - 1) / kGvKB;
    for (int q = jb.near0; q < jb.near1; ++q) total += (near[q].K + kGvKB - 1) / kGvKB;
    if (warp >= 2) {
        const int row = (warp - 2) * 32 + lane;
        const int m = jb.m0 + r0 + min(row, rows - 1);
        const double *Tf = T + (size_t)nrhs * jb.kap0;
        // next stage to describe: piece (-1: the factors, else a near piece)
        // and k0
        int piece = jb.kfar > 0 ? -1 : jb.near0, k0 = 0;
        auto describe = [&]() {
            GvStage g{nullptr, A, 0, 0, 0};
            if (piece >= jb.near1) return g;
            int K;
            if (piece < 0) {
                K = jb.kfar;
                g.k = min(kGvKB, K - k0);
                if (lane < g.k) g.col = ucol[jb.kap0 + k0 + lane];
                g.x = Tf + k0;
                g.ldx = jb.kfar;
                g.rs = 1;
            } else {
                const NearPiece np = near[piece];
                K = np.K;
                g.k = min(kGvKB, K - k0);
                g.col = nearD + np.off + (size_t)(k0 + min(lane, g.k - 1)) * (np.trans ? 1 : np.ld);
                g.x = A + np.in0 + k0;
                g.ldx = lda;
                g.rs = np.trans ? np.ld : 1;
            }
            k0 += kGvKB;
            if (k0 >= K) {
                piece = piece < 0 ? jb.near0 : piece + 1;
                k0 = 0;
            }
            return g;
        };
        auto issue = [&](const GvStage &g, int st) {
            double *S = gvb_sm + st % kGvStagesB * STAGE, *X = S + kGvRowsB * kGvKB;
            const size_t mo = (size_t)m * g.rs;
            #pragma unroll
            for (int u = 0; u < kGvKB; ++u) {
                const double *p = (const double *)__shfl_sync(
                    0xffffffffu, (unsigned long long)g.col, u);
                cp_async8(S + u * kGvRowsB + row, u < g.k ? p + mo : A, u < g.k);
            }
            for (int c = warp - 2; c < NR; c += 2) {
                const bool ok = lane < g.k && c < nrhs;
                cp_async8(X + c * kGvKB + lane, ok ? g.x + lane + (size_t)c * g.ldx : A, ok);
            }
        };
        GvStage g[kGvAhead];
        #pragma unroll
        for (int q = 0; q < kGvAhead; ++q) g[q] = describe();
        static_assert(kGvStagesB - 1 == kGvAhead, "the prologue issues what it described");
        #pragma unroll
        for (int q = 0; q < kGvStagesB - 1; ++q) {
            if (q < total) issue(g[q], q);
            cp_async_commit();
            g[q] = describe();
        }
        for (int st0 = 0; st0 < total; st0 += kGvAhead)
            #pragma unroll
            for (int q = 0; q < kGvAhead; ++q) {
                const int st = st0 + q;
                if (st >= total) break;
                asm volatile("cp.async.wait_group %0;\n" ::"n"(kGvStagesB - 2));
                gvb_sync();
                if (st + kGvStagesB - 1 < total) {
                    issue(g[q], st + kGvStagesB - 1);
                    g[q] = describe();
                }
                cp_async_commit();
            }
        asm volatile("cp.async.wait_group 0;\n" ::);
        return;
    }
    double acc[NR] = {};
    for (int st = 0; st < total; ++st) {
        gvb_sync();                    // landed, and the refilled one consumed
        const double *S = gvb_sm + st % kGvStagesB * STAGE + t;
        const double2 *X = reinterpret_cast<const double2 *>(
            gvb_sm + st % kGvStagesB * STAGE + kGvRowsB * kGvKB);
        double v[kGvKB];
        #pragma unroll
        for (int k = 0; k < kGvKB; ++k) v[k] = S[k * kGvRowsB];
        #pragma unroll
        for (int c = 0; c < NR; ++c)
            #pragma unroll
            for (int k = 0; k < kGvKB; k += 2) {
                const double2 x = X[(c * kGvKB + k) / 2];
                acc[c] = fma(v[k], x.x, acc[c]);
                acc[c] = fma(v[k + 1], x.y, acc[c]);
            }
    }
    if (t >= rows) return;
    #pragma unroll
    for (int c = 0; c < NR; ++c)
        if (c < nrhs) update(B + jb.out0 + r0 + t + (size_t)c * ldb, alpha, acc[c], beta);
}

template <int NR>
static void launch_gemv(const Job1 *j1, int n1, const double *const *vcol,
                        const RowT *rowt, const Job2 *j2, int n2,
                        const double *const *ucol, const NearPiece *near,
                        const double *nearD, const double *A, int lda, double *T,
                        double *B, int ldb, int nrhs, double alpha, double beta,
                        cudaStream_t s)
{
    constexpr size_t smem_t = (size_t)kGvStagesT * gv_stage_t<NR>() * sizeof(double);
    constexpr size_t smem_b = (size_t)kGvStagesB * gv_stage_b<NR>() * sizeof(double);
    allow_smem<k_gemv_t<NR>, smem_t>();
    allow_smem<k_gemv_b<NR>, smem_b>();
    if (n1 > 0) {
        k_gemv_t<NR><<<dim3((unsigned)n1, kPBM / kGvRowsT), 128, smem_t, s>>>(
            j1, vcol, rowt, A, lda, T, nrhs);
        count_launch();
    }
    if (n2 > 0) {
        k_gemv_b<NR><<<dim3((unsigned)n2, kPBM / kGvRowsB), kGvThreadsB, smem_b, s>>>(
            j2, ucol, T, nrhs, near, nearD, A, lda, B, ldb, alpha, beta);
        count_launch();
    }
}

__global__ void k_scale_cols(double *B, int ldb, int rows, int cols,
                             double beta)
{
    const long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (idx >= (long long)rows * cols) return;
    const int i = (int)(idx % rows), j = (int)(idx / rows);
    double *p = B + (size_t)j * ldb + i;
    *p = beta == 0.0 ? 0.0 : beta * *p;
}

// -------------------------------------------------- record for any blrm

// Matrices from another engine (or whose device copy was released) get
// their factors uploaded once and a record attached.
static int ensure_record(STARSH_blrm *M, Context &ctx, Record **out)
{
    Record *rec = find_record(M);
    if (rec) {
        *out = rec;
        return STARSH_SUCCESS;
    }
    STARSH_blrf *F = M->format;
    cudaStream_t s = ctx.stream;
    rec = new Record();
    rec->points = new DevicePoints();
    int info = upload_problem(*rec->points, F->problem, F->row_cluster,
                              F->col_cluster, s);
    if (info) {
        delete rec;
        return info;
    }
    size_t nu = 0, nv = 0, nd = 0;
    for (STARSH_int b = 0; b < F->nblocks_far; ++b) {
        nu += M->far_U[b]->size;
        nv += M->far_V[b]->size;
    }
    if (M->onfly == 0)
        for (STARSH_int b = 0; b < F->nblocks_near; ++b) nd += M->near_D[b]->size;
    double *chunk = nullptr;
    if (nu + nv + nd > 0) {
        chunk = (double *)pool_alloc((nu + nv + nd) * sizeof(double), s);
        if (chunk == nullptr) {
            delete rec;
            return cuda_fail(cudaErrorMemoryAllocation, "uploaded factors");
        }
        rec->chunks.push_back(chunk);
    }
    size_t ou = 0, ov = nu, od = nu + nv;
    rec->dU.resize(F->nblocks_far);
    rec->dV.resize(F->nblocks_far);
    for (STARSH_int b = 0; b < F->nblocks_far; ++b) {
        rec->dU[b] = chunk + ou;
        rec->dV[b] = chunk + ov;
        cudaMemcpyAsync(chunk + ou, M->far_U[b]->data,
                        M->far_U[b]->size * sizeof(double),
                        cudaMemcpyHostToDevice, s);
        cudaMemcpyAsync(chunk + ov, M->far_V[b]->data,
                        M->far_V[b]->size * sizeof(double),
                        cudaMemcpyHostToDevice, s);
        ou += M->far_U[b]->size;
        ov += M->far_V[b]->size;
    }
    rec->dD.assign(F->nblocks_near, nullptr);
    if (M->onfly == 0)
        for (STARSH_int b = 0; b < F->nblocks_near; ++b) {
            rec->dD[b] = chunk + od;
            cudaMemcpyAsync(chunk + od, M->near_D[b]->data,
                            M->near_D[b]->size * sizeof(double),
                            cudaMemcpyHostToDevice, s);
            od += M->near_D[b]->size;
        }
    rec->u_total = nu;
    rec->v_total = nv;
    rec->d_total = nd;
    rec->host_filled = true;
    add_record(M, rec);
    *out = rec;
    return STARSH_SUCCESS;
}

// ---------------------------------------------------------------- dmml

// The product plan of a matrix (device arrays, built on its first product
// and kept with its record): phase-1 jobs with their factor-column
// pointers and T destinations, phase-2 jobs with the concatenated
// left-factor columns of every block row and the near pieces.
struct ProductPlan {
    void *dev = nullptr;
    const double **vcol = nullptr;
    RowT *rowt = nullptr;
    const double **ucol = nullptr;
    Job1 *j1 = nullptr;
    Job2 *j2 = nullptr;
    NearPiece *near = nullptr;
    int n1 = 0, n2 = 0, nnear = 0;
    bool covers = false;       // phase 2 writes every output row
    size_t near_total = 0;     // doubles of the near blocks
    long long trows = 0;       // rows of T over all block rows
    cudaEvent_t ready = nullptr;   // the upload has completed
    ~ProductPlan()
    {
        if (ready) cudaEventDestroy(ready);
        if (dev) pool_free(dev);
    }
};

// A far block's place in the plan (or its mirror's).
struct PlanBlock {
    const double *U, *V;
    long long P, rho;      // first T row of its block row; its first phase-1 row
    int m, n, r, kap, S;   // sizes, rank, place in the block row's S columns
};

// The block's r columns in both phases' lists.  The lists have one entry per
// factor column (5e5 for 16384 blocks), which took the host 10 ms to fill;
// it now prepares one record per block.
__global__ void k_plan_columns(const PlanBlock *__restrict__ blocks,
                               const double **vcol, RowT *rowt, const double **ucol)
{
    const PlanBlock b = blocks[blockIdx.x];
    for (int c = threadIdx.x; c < b.r; c += blockDim.x) {
        vcol[b.rho + c] = b.V + (size_t)c * b.n;
        rowt[b.rho + c] = RowT{b.P, b.kap + c, b.S};
        ucol[b.P + b.kap + c] = b.U + (size_t)c * b.m;
    }
}

template <class T>
static size_t put(std::vector<char> &buf, const std::vector<T> &v)
{
    const size_t off = (buf.size() + 255) / 256 * 256;
    buf.resize(off + v.size() * sizeof(T));
    if (!v.empty()) memcpy(buf.data() + off, v.data(), v.size() * sizeof(T));
    return off;
}

static int build_plan(STARSH_blrm *M, const Record &rec, cudaStream_t s,
                      ProductPlan **out)
{
    STARSH_blrf *F = M->format;
    STARSH_cluster *R = F->row_cluster, *C = F->col_cluster;
    const bool symm = F->symm == 'S';
    // products: output block row, input block (of the column clustering,
    // or of the row clustering for a mirrored block), factors, sizes
    struct Prod { STARSH_int orow, icol; const double *U, *V; int m, n, r; long long in0; };
    std::vector<Prod> prods;
    for (STARSH_int b = 0; b < F->nblocks_far; ++b) {
        const int r = M->far_rank[b];
        if (r <= 0) continue;
        const STARSH_int i = F->block_far[2 * b], j = F->block_far[2 * b + 1];
        const int m = (int)R->size[i], n = (int)C->size[j];
        prods.push_back({i, j, rec.dU[b], rec.dV[b], m, n, r, (long long)C->start[j]});
        if (symm && i != j)
            prods.push_back({j, i, rec.dV[b], rec.dU[b], n, m, r, (long long)R->start[i]});
    }
    const STARSH_int nbr = F->nbrows, nbc = std::max(F->nbrows, F->nbcols);
    // phase 2 layout: per output row its products in list order
    std::vector<long long> P(nbr + 1, 0);
    std::vector<int> S(nbr, 0);
    std::vector<int> kap(prods.size());
    for (size_t p = 0; p < prods.size(); ++p) {
        kap[p] = S[prods[p].orow];
        S[prods[p].orow] += prods[p].r;
    }
    for (STARSH_int i = 0; i < nbr; ++i) P[i + 1] = P[i] + S[i];
    const long long trows = P[nbr];
    // phase 1: products grouped by input block, list order within a group
    std::vector<std::vector<int>> bycol(nbc);
    for (size_t p = 0; p < prods.size(); ++p) bycol[prods[p].icol].push_back((int)p);
    // (the columns themselves are spread out on the device, k_plan_columns)
    std::vector<PlanBlock> blocks(prods.size());
    std::vector<Job1> j1;
    long long rho = 0;
    for (STARSH_int j = 0; j < nbc; ++j) {
        if (bycol[j].empty()) continue;
        const long long rho0 = rho;
        for (int p : bycol[j]) {
            const Prod &q = prods[p];
            blocks[p] = PlanBlock{q.U, q.V, P[q.orow], rho, q.m, q.n, q.r, kap[p], S[q.orow]};
            rho += q.r;
        }
        const int cnt = (int)(rho - rho0);
        const Prod &q0 = prods[bycol[j][0]];
        for (int r0 = 0; r0 < cnt; r0 += kPBM)
            j1.push_back(Job1{(int)rho0 + r0, std::min(kPBM, cnt - r0), q0.n, q0.in0});
    }
    // near pieces per output row, in near-block order
    // (stored blocks by their place after the first one, regenerated ones
    // in list order)
    std::vector<std::vector<NearPiece>> rownear(nbr);
    size_t near_total = 0;
    for (STARSH_int b = 0; b < F->nblocks_near; ++b) {
        const STARSH_int i = F->block_near[2 * b], j = F->block_near[2 * b + 1];
        const int m = (int)R->size[i], n = (int)C->size[j];
        const long long off = M->onfly ? (long long)near_total
                                       : (long long)(rec.dD[b] - rec.dD[0]);
        near_total += (size_t)m * n;
        rownear[i].push_back(NearPiece{off, 0, n, m, (long long)C->start[j]});
        if (symm && i != j)
            rownear[j].push_back(NearPiece{off, 1, m, m, (long long)R->start[i]});
    }
    bool covers = true;
    std::vector<NearPiece> near;
    std::vector<Job2> j2;
    for (STARSH_int i = 0; i < nbr; ++i) {
        if (S[i] == 0 && rownear[i].empty()) {
            covers = false;
            continue;
        }
        const int near0 = (int)near.size();
        near.insert(near.end(), rownear[i].begin(), rownear[i].end());
        const int mi = (int)R->size[i];
        for (int m0 = 0; m0 < mi; m0 += kPBM)
            j2.push_back(Job2{(long long)R->start[i] + m0, m0, std::min(kPBM, mi - m0),
                              P[i], S[i], near0, (int)near.size()});
    }
    // longest K first: the CTAs of a launch start in this order
    {
        auto klen = [&](const Job2 &j) {
            long long k = j.kfar;
            for (int q = j.near0; q < j.near1; ++q) k += near[q].K;
            return k;
        };
        std::vector<std::pair<long long, int>> order(j2.size());
        for (size_t q = 0; q < j2.size(); ++q) order[q] = {-klen(j2[q]), (int)q};
        std::stable_sort(order.begin(), order.end(),
                         [](const auto &x, const auto &y) { return x.first < y.first; });
        std::vector<Job2> sorted(j2.size());
        for (size_t q = 0; q < j2.size(); ++q) sorted[q] = j2[order[q].second];
        j2.swap(sorted);
    }
    // one device allocation for every array
    std::vector<char> buf;
    const size_t o_j1 = put(buf, j1), o_j2 = put(buf, j2), o_near = put(buf, near),
                 o_blk = put(buf, blocks);
    // (behind the uploaded arrays: what the device fills)
    auto round256 = [](size_t n) { return (n + 255) / 256 * 256; };
    const size_t o_rowt = round256(buf.size());
    const size_t o_vcol = o_rowt + round256(trows * sizeof(RowT));
    const size_t o_ucol = o_vcol + round256(trows * sizeof(double *));
    const size_t all = o_ucol + trows * sizeof(double *);
    auto *plan = new ProductPlan();
    if (!buf.empty()) {
        char *d = (char *)pool_alloc(all, s);
        if (d == nullptr) {
            delete plan;
            return cuda_fail(cudaErrorMemoryAllocation, "product plan");
        }
        plan->dev = d;
        const cudaError_t e = cudaMemcpyAsync(d, buf.data(), buf.size(),
                                              cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) {
            delete plan;
            return cuda_fail(e, "product plan upload");
        }
        plan->vcol = (const double **)(d + o_vcol);
        plan->rowt = (RowT *)(d + o_rowt);
        plan->ucol = (const double **)(d + o_ucol);
        plan->j1 = (Job1 *)(d + o_j1);
        plan->j2 = (Job2 *)(d + o_j2);
        plan->near = (NearPiece *)(d + o_near);
        if (!blocks.empty()) {
            k_plan_columns<<<(unsigned)blocks.size(), 64, 0, s>>>(
                (const PlanBlock *)(d + o_blk), plan->vcol, plan->rowt, plan->ucol);
            count_launch();
        }
        // products on any stream wait for the upload
        if (cudaEventCreateWithFlags(&plan->ready, cudaEventDisableTiming) !=
                cudaSuccess ||
            cudaEventRecord(plan->ready, s) != cudaSuccess) {
            delete plan;
            return cuda_fail(cudaGetLastError(), "product plan event");
        }
    }
    plan->n1 = (int)j1.size();
    plan->n2 = (int)j2.size();
    plan->nnear = (int)near.size();
    plan->trows = trows;
    plan->covers = covers;
    plan->near_total = near_total;
    *out = plan;
    return STARSH_SUCCESS;
}

int dmml_device(STARSH_blrm *M, int nrhs, double alpha,
                const double *dA, int lda, double beta, double *dB,
                int ldb, cudaStream_t user_stream, Context &ctx)
{
    if (M == nullptr || nrhs < 0 || dA == nullptr || dB == nullptr)
        return STARSH_WRONG_PARAMETER;
    STARSH_blrf *F = M->format;
    STARSH_problem *P = F->problem;
    STARSH_cluster *R = F->row_cluster, *C = F->col_cluster;
    const STARSH_int nrows = P->shape[0];
    if (lda < P->shape[P->ndim - 1] || ldb < nrows)
        return STARSH_WRONG_PARAMETER;
    if (nrhs == 0) return STARSH_SUCCESS;
    Record *rec = nullptr;
    int info = ensure_record(M, ctx, &rec);
    if (info) return info;
    cudaStream_t s = ctx.stream;
    // Order the user's stream before ours and ours before the user's.
    struct Order {
        cudaEvent_t ev = nullptr;
        ~Order() { if (ev) cudaEventDestroy(ev); }
    } order;
    cudaEvent_t &ev = order.ev;
    if (user_stream != s) {
        B200_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "dmml event");
        cudaEventRecord(ev, user_stream);
        cudaStreamWaitEvent(s, ev, 0);
    }
    ProductPlan *plan = nullptr;
    {
        std::lock_guard<std::mutex> g(rec->plan_lock);
        if (!rec->plan) {
            ProductPlan *built = nullptr;
            if ((info = build_plan(M, *rec, s, &built))) return info;
            rec->plan = std::shared_ptr<void>(built, [](void *q) {
                delete (ProductPlan *)q;
            });
        }
        plan = (ProductPlan *)rec->plan.get();
    }
    if (plan->ready) cudaStreamWaitEvent(s, plan->ready, 0);
    // beta: with the product's last step, or first where it skips rows
    if (!plan->covers) {
        const long long tot = (long long)nrows * nrhs;
        k_scale_cols<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(
            dB, ldb, (int)nrows, nrhs, beta);
        count_launch();
        beta = 1.0;
    }
    // near blocks: dense D (stored, or regenerated when onfly)
    double *onfly_buf = nullptr;
    const double *nearD = nullptr;
    if (F->nblocks_near > 0) {
        if (M->onfly) {
            onfly_buf = (double *)pool_alloc(plan->near_total * sizeof(double), s);
            if (onfly_buf == nullptr) {
                return cuda_fail(cudaErrorMemoryAllocation, "onfly blocks");
            }
            std::vector<BlockJob> jobs;
            size_t off = 0;
            for (STARSH_int b = 0; b < F->nblocks_near; ++b) {
                const STARSH_int i = F->block_near[2 * b], j = F->block_near[2 * b + 1];
                BlockJob jb{R->start[i], C->start[j], (int)R->size[i],
                            (int)C->size[j], onfly_buf + off};
                off += (size_t)jb.m * jb.n;
                jobs.push_back(jb);
            }
            if ((info = gen_blocks(rec->points->K, jobs, s))) {
                pool_free(onfly_buf);
                return info;
            }
            nearD = onfly_buf;
        } else {
            nearD = rec->dD[0];
        }
    }
    // per call: T (rows of every block row x nrhs)
    const size_t tbytes = (size_t)plan->trows * nrhs * sizeof(double);
    char *scratch = nullptr;
    if (tbytes > 0) {
        scratch = (char *)pool_alloc(tbytes, s);
        if (scratch == nullptr) {
            if (onfly_buf) pool_free(onfly_buf);
            return cuda_fail(cudaErrorMemoryAllocation, "product scratch");
        }
    }
    double *T = (double *)scratch;
    auto tiles = [&](auto fn) {
        fn(plan->j1, plan->n1, plan->vcol, plan->rowt, plan->j2, plan->n2, plan->ucol,
           plan->near, nearD, dA, lda, T, dB, ldb, nrhs, alpha, beta, s);
    };
    if (nrhs <= kGemvRhs) {
        if (nrhs == 1) tiles(launch_gemv<1>);
        else if (nrhs == 2) tiles(launch_gemv<2>);
        else tiles(launch_gemv<kGemvRhs>);
    } else if (nrhs > 32) {
        tiles(launch_products<4>);
    } else if (nrhs > 16) {
        tiles(launch_products<2>);
    } else {
        tiles(launch_products<1>);
    }
    if (scratch) pool_free(scratch);
    if (onfly_buf) pool_free(onfly_buf);
    cudaError_t e = cudaGetLastError();
    if (user_stream != s) {
        cudaEventRecord(ev, s);
        cudaStreamWaitEvent(user_stream, ev, 0);
    }
    if (e != cudaSuccess) return cuda_fail(e, "dmml kernels");
    return STARSH_SUCCESS;
}

// ----------------------------------------------------------------- dfe

struct DfeJob {
    long long row0, col0;
    int m, n, r;
    const double *U, *V, *D;   // D: stored dense block or null
};

// Each CTA takes 64 rows and cb 64-column blocks (4, or 1 where that leaves
// too few CTAs) of a job: U V^T on the
// FP64 tensor path (8 warps of 32 x 16 outputs), and the block's entries
// evaluated by the thread that holds the same output in its accumulators, so
// nothing but the factors is read (or, for a stored dense block, its
// entries).  Coordinates are staged once per CTA, the kernel family is
// compiled in, and the factors' next K step of 16 is copied while the
// entries of the current block are evaluated.  The entries' FP64 work is
// what bounds it (the generator's bound without its store): N = 25600
// square exponential, tol 1e-7, 3.4 ms, against 11.2 with scalar products
// from shared memory and a family switch and two index loads per entry.
// The CTA's ||D||^2 and ||D - U V^T||^2 go to its own slot of `part` (slot =
// (job, tile row, column group)); k_dfe_sum adds a job's slots in a fixed
// order, so the error is the same on every run.
constexpr int kDfeCb = 4, kDfeLd = 68, kDfeDim = 4;
constexpr size_t kDfeStage = 2 * (size_t)kPBK * kDfeLd;   // doubles

// Entries (row i, columns c) of one block against the accumulators.
template <int FAM, int NDIM>
__device__ __forceinline__ void dfe_entries(
    const DevKernel &K, const DfeJob &jb, const double (*rc)[64],
    const double (*cc)[64 * kDfeCb], const long long *ri, const long long *ci,
    int i0, int j0, int jb0, int wm, int wn, int g, int tig,
    const double (&acc)[4][2][2], double &nrm, double &dif)
{
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int lr = wm + 8 * i + g;
        double xr[NDIM > 0 ? NDIM : 1];
        if constexpr (NDIM > 0) {
            #pragma unroll
            for (int d = 0; d < NDIM; ++d) xr[d] = rc[d][lr];
        }
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int lc = jb0 + wn + 8 * (q >> 1) + 2 * tig + (q & 1);
            double v;
            if (jb.D != nullptr) {
                v = i0 + lr < jb.m && j0 + lc < jb.n
                        ? jb.D[(size_t)(j0 + lc) * jb.m + i0 + lr] : 0.0;
            } else {
                double dist = 0.0;
                if constexpr (NDIM > 0) {
                    #pragma unroll
                    for (int d = 0; d < NDIM; ++d) {
                        const double t = __dsub_rn(xr[d], cc[d][lc]);
                        dist = __dadd_rn(dist, __dmul_rn(t, t));
                    }
                } else if constexpr (NDIM == 0) {
                    for (int d = 0; d < K.ndim; ++d) {
                        const double t = __dsub_rn(rc[d][lr], cc[d][lc]);
                        dist = __dadd_rn(dist, __dmul_rn(t, t));
                    }
                } else {
                    dist = sq_dist(K, ri[lr], ci[lc]);
                }
                v = entry_fam<FAM>(K, dist, ri[lr], ci[lc]);
            }
            if (i0 + lr < jb.m && j0 + lc < jb.n) {
                const double e = v - acc[i][q >> 1][q & 1];
                nrm += v * v;
                dif += e * e;
            }
        }
    }
}

template <int FAM>
__global__ void __launch_bounds__(256, 3)
k_dfe(DevKernel K, const DfeJob *__restrict__ jobs, double *__restrict__ part,
      int cb)
{
    extern __shared__ double dfe_sm[];         // [2][U 16 x 68, V 16 x 68]
    __shared__ double rc[kDfeDim][64], cc[kDfeDim][64 * kDfeCb];
    __shared__ long long ri[64], ci[64 * kDfeCb];
    __shared__ double red[2][8];
    const DfeJob jb = jobs[blockIdx.z];
    const int i0 = blockIdx.x * 64, j0 = blockIdx.y * 64 * cb;
    double *slot = part + 2 * (((size_t)blockIdx.z * gridDim.y + blockIdx.y) *
                               gridDim.x + blockIdx.x);
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (i0 >= jb.m || j0 >= jb.n) {
        if (t == 0) slot[0] = slot[1] = 0.0;
        return;
    }
    const int g = lane >> 2, tig = lane & 3;
    const int wm = (warp & 1) * 32, wn = (warp >> 1) * 16;
    const bool staged = !K.aos && K.ndim <= kDfeDim;
    if (t < 64) ri[t] = K.row_piv[jb.row0 + min(i0 + t, jb.m - 1)];
    ci[t] = K.col_piv[jb.col0 + min(j0 + t, jb.n - 1)];
    static_assert(64 * kDfeCb == 256, "a column index per thread");
    __syncthreads();
    if (staged)
        for (int d = 0; d < K.ndim; ++d) {
            if (t < 64) rc[d][t] = K.row_pt[d * K.row_count + ri[t]];
            cc[d][t] = K.col_pt[d * K.col_count + ci[t]];
        }
    const int nblk = min(cb, (jb.n - j0 + 63) / 64);
    const int ksteps = (jb.r + kPBK - 1) / kPBK;
    const int steps = nblk * ksteps;           // (block, K step), block-major
    auto issue = [&](int st) {
        double *Us = dfe_sm + (st & 1) * kDfeStage, *Vs = Us + kPBK * kDfeLd;
        const int b = st / ksteps, k0 = (st - b * ksteps) * kPBK;
        #pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int row = t & 63, k = (t >> 6) + 4 * q, p = k0 + k;
            const int i = i0 + row, j = j0 + b * 64 + row;
            const bool okU = p < jb.r && i < jb.m, okV = p < jb.r && j < jb.n;
            cp_async8(Us + k * kDfeLd + row, okU ? jb.U + (size_t)p * jb.m + i : jb.U, okU);
            cp_async8(Vs + k * kDfeLd + row, okV ? jb.V + (size_t)p * jb.n + j : jb.V, okV);
        }
    };
    if (steps > 0) issue(0);
    cp_async_commit();
    double nrm = 0.0, dif = 0.0;
    int st = 0;
    #pragma unroll 1
    for (int b = 0; b < nblk; ++b) {
        double acc[4][2][2] = {};
        #pragma unroll 1
        for (int k = 0; k < ksteps; ++k, ++st) {
            asm volatile("cp.async.wait_group 0;\n" ::);
            __syncthreads();                   // step st landed, st - 1 consumed
            if (st + 1 < steps) issue(st + 1);
            cp_async_commit();
            const double *Us = dfe_sm + (st & 1) * kDfeStage, *Vs = Us + kPBK * kDfeLd;
            #pragma unroll
            for (int kk = 0; kk < kPBK; kk += 4) {
                double af[4], bf[2];
                #pragma unroll
                for (int i = 0; i < 4; ++i) af[i] = Us[(kk + tig) * kDfeLd + wm + 8 * i + g];
                #pragma unroll
                for (int j = 0; j < 2; ++j) bf[j] = Vs[(kk + tig) * kDfeLd + wn + 8 * j + g];
                #pragma unroll
                for (int i = 0; i < 4; ++i)
                    #pragma unroll
                    for (int j = 0; j < 2; ++j)
                        dmma_884(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
            }
        }
        if (b == 0) __syncthreads();           // coordinates
        if (!staged)
            dfe_entries<FAM, -1>(K, jb, rc, cc, ri, ci, i0, j0, b * 64, wm, wn, g, tig, acc, nrm, dif);
        else if (K.ndim == 2)
            dfe_entries<FAM, 2>(K, jb, rc, cc, ri, ci, i0, j0, b * 64, wm, wn, g, tig, acc, nrm, dif);
        else if (K.ndim == 3)
            dfe_entries<FAM, 3>(K, jb, rc, cc, ri, ci, i0, j0, b * 64, wm, wn, g, tig, acc, nrm, dif);
        else
            dfe_entries<FAM, 0>(K, jb, rc, cc, ri, ci, i0, j0, b * 64, wm, wn, g, tig, acc, nrm, dif);
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        nrm += __shfl_down_sync(0xffffffffu, nrm, o);
        dif += __shfl_down_sync(0xffffffffu, dif, o);
    }
    if (lane == 0) {
        red[0][warp] = nrm;
        red[1][warp] = dif;
    }
    __syncthreads();
    if (t == 0) {
        double a = 0.0, b = 0.0;
        for (int w = 0; w < 8; ++w) {
            a += red[0][w];
            b += red[1][w];
        }
        slot[0] = a;
        slot[1] = b;
    }
}

// out[2 job + {0, 1}] = the sums of the job's nslot slots: one warp per job,
// lane l adds slots l, l + 32, ..., then a tree over the lanes.
__global__ void k_dfe_sum(const double *__restrict__ part, int nslot,
                          long long njobs, double *__restrict__ out)
{
    const long long j = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (j >= njobs) return;
    const double2 *p = reinterpret_cast<const double2 *>(part) + (size_t)j * nslot;
    double a = 0.0, b = 0.0;
    for (int q = lane; q < nslot; q += 32) {
        const double2 v = p[q];
        a += v.x;
        b += v.y;
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, o);
        b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
        out[2 * j] = a;
        out[2 * j + 1] = b;
    }
}

static void launch_dfe(const DevKernel &K, dim3 grid, const DfeJob *jobs,
                       double *part, int cb, cudaStream_t s)
{
    constexpr size_t smem = 2 * kDfeStage * sizeof(double);
    switch (K.family) {
    case FAM_EXP: k_dfe<FAM_EXP><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    case FAM_SQREXP: k_dfe<FAM_SQREXP><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    case FAM_MATERN: k_dfe<FAM_MATERN><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    case FAM_MATERN2: k_dfe<FAM_MATERN2><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    case FAM_COULOMB: k_dfe<FAM_COULOMB><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    case FAM_SIN: k_dfe<FAM_SIN><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    case FAM_COS: k_dfe<FAM_COS><<<grid, 256, smem, s>>>(K, jobs, part, cb); break;
    default: k_dfe<FAM_RBF><<<grid, 256, smem, s>>>(K, jobs, part, cb);
    }
}

// The weighted sums sum ||D_b - U_b V_b^T||_F^2 (far blocks) and
// sum ||D_b||_F^2 (all blocks) of M; returns STARSH_SUCCESS or an error.
static int dfe_sums_device(STARSH_blrm *M, Context &ctx, double *diff2,
                           double *norm2)
{
    *diff2 = *norm2 = 0.0;
    Record *rec = nullptr;
    if (ensure_record(M, ctx, &rec)) return STARSH_UNKNOWN_ERROR;
    STARSH_blrf *F = M->format;
    STARSH_cluster *R = F->row_cluster, *C = F->col_cluster;
    cudaStream_t s = ctx.stream;
    const STARSH_int nf = F->nblocks_far, nn = F->nblocks_near;
    const size_t njobs = nf + nn;
    if (njobs == 0) return STARSH_SUCCESS;
    std::vector<DfeJob> jobs(njobs);
    int mmax = 0, nmax = 0;
    for (STARSH_int b = 0; b < nf; ++b) {
        const STARSH_int i = F->block_far[2 * b], j = F->block_far[2 * b + 1];
        jobs[b] = DfeJob{R->start[i], C->start[j], (int)R->size[i],
                         (int)C->size[j], M->far_rank[b], rec->dU[b],
                         rec->dV[b], nullptr};
    }
    for (STARSH_int b = 0; b < nn; ++b) {
        const STARSH_int i = F->block_near[2 * b], j = F->block_near[2 * b + 1];
        jobs[nf + b] = DfeJob{R->start[i], C->start[j], (int)R->size[i],
                              (int)C->size[j], 0, nullptr, nullptr,
                              M->onfly ? nullptr : rec->dD[b]};
    }
    for (const auto &j : jobs) {
        mmax = std::max(mmax, j.m);
        nmax = std::max(nmax, j.n);
    }
    const int gx = (mmax + 63) / 64, gy1 = (nmax + 63) / 64;
    const int cb = (size_t)gx * ((gy1 + kDfeCb - 1) / kDfeCb) * njobs < 888 ? 1 : kDfeCb;
    const int gy = (gy1 + cb - 1) / cb;
    const size_t nslot = (size_t)gx * gy;
    double *sums = (double *)pool_alloc(2 * njobs * sizeof(double), s);
    double *part = (double *)pool_alloc(2 * njobs * nslot * sizeof(double), s);
    DfeJob *dj = (DfeJob *)pool_alloc(njobs * sizeof(DfeJob), s);
    if (!sums || !part || !dj) {
        pool_free(sums);
        pool_free(part);
        pool_free(dj);
        return cuda_fail(cudaErrorMemoryAllocation, "dfe buffers");
    }
    cudaMemcpyAsync(dj, jobs.data(), njobs * sizeof(DfeJob),
                    cudaMemcpyHostToDevice, s);
    for (size_t b0 = 0; b0 < njobs; b0 += 65535) {
        const unsigned nb = (unsigned)std::min<size_t>(65535, njobs - b0);
        dim3 grid(gx, gy, nb);
        launch_dfe(rec->points->K, grid, dj + b0, part + 2 * b0 * nslot, cb, s);
        count_launch();
    }
    k_dfe_sum<<<(unsigned)((njobs + 7) / 8), 256, 0, s>>>(
        part, (int)nslot, (long long)njobs, sums);
    count_launch();
    std::vector<double> h(2 * njobs);
    cudaMemcpyAsync(h.data(), sums, 2 * njobs * sizeof(double),
                    cudaMemcpyDeviceToHost, s);
    pool_free(sums);
    pool_free(part);
    pool_free(dj);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "dfe kernels");
    double diff = 0.0, norm = 0.0;
    const bool symm = F->symm == 'S';
    for (STARSH_int b = 0; b < nf; ++b) {
        const double w = (symm && F->block_far[2 * b] != F->block_far[2 * b + 1]) ? 2.0 : 1.0;
        norm += w * h[2 * b];
        diff += w * h[2 * b + 1];
    }
    for (STARSH_int b = 0; b < nn; ++b) {
        const double w = (symm && F->block_near[2 * b] != F->block_near[2 * b + 1]) ? 2.0 : 1.0;
        norm += w * h[2 * (nf + b)];
    }
    *diff2 = diff;
    *norm2 = norm;
    return STARSH_SUCCESS;
}

static double dfe_device(STARSH_blrm *M, Context &ctx)
{
    double diff = 0.0, norm = 0.0;
    if (dfe_sums_device(M, ctx, &diff, &norm) != STARSH_SUCCESS) return -1.0;
    return norm > 0.0 ? sqrt(diff) / sqrt(norm) : 0.0;
}

}  // namespace b200

using namespace b200;

extern "C" int starsh_b200_blrm_dmml_device(STARSH_blrm *matrix, int nrhs,
                                            double alpha, const double *dA,
                                            int lda, double beta, double *dB,
                                            int ldb, void *stream)
{
    Context *ctx = context();
    if (!ctx) return STARSH_UNKNOWN_ERROR;
    std::lock_guard<std::mutex> guard(ctx->lock);
    return dmml_device(matrix, nrhs, alpha, dA, lda, beta, dB, ldb,
                       stream ? (cudaStream_t)stream : ctx->stream, *ctx);
}

extern "C" int starsh_blrm__dmml_b200(STARSH_blrm *matrix, int nrhs,
                                      double alpha, double *A, int lda,
                                      double beta, double *B, int ldb)
{
    if (matrix == nullptr || A == nullptr || B == nullptr || nrhs < 0)
        return STARSH_WRONG_PARAMETER;
    Context *ctx = context();
    if (!ctx) return STARSH_UNKNOWN_ERROR;
    std::lock_guard<std::mutex> guard(ctx->lock);
    STARSH_problem *P = matrix->format->problem;
    const size_t nr = P->shape[0], nc = P->shape[P->ndim - 1];
    if (lda < (int)nc || ldb < (int)nr) return STARSH_WRONG_PARAMETER;
    cudaStream_t s = ctx->stream;
    double *dA = nullptr, *dB = nullptr;
    if (cudaMallocAsync((void **)&dA, nc * nrhs * sizeof(double) + 8, s) ||
        cudaMallocAsync((void **)&dB, nr * nrhs * sizeof(double) + 8, s))
        return cuda_fail(cudaGetLastError(), "cudaMallocAsync(dmml)");
    cudaMemcpy2DAsync(dA, nc * sizeof(double), A, (size_t)lda * sizeof(double),
                      nc * sizeof(double), nrhs, cudaMemcpyHostToDevice, s);
    if (beta != 0.0)
        cudaMemcpy2DAsync(dB, nr * sizeof(double), B,
                          (size_t)ldb * sizeof(double), nr * sizeof(double),
                          nrhs, cudaMemcpyHostToDevice, s);
    int info = dmml_device(matrix, nrhs, alpha, dA, (int)nc, beta, dB,
                           (int)nr, s, *ctx);
    if (!info)
        cudaMemcpy2DAsync(B, (size_t)ldb * sizeof(double), dB,
                          nr * sizeof(double), nr * sizeof(double), nrhs,
                          cudaMemcpyDeviceToHost, s);
    cudaFreeAsync(dA, s);
    cudaFreeAsync(dB, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (!info && e != cudaSuccess) info = cuda_fail(e, "dmml");
    return info;
}

extern "C" int starsh_blrm__dmml(STARSH_blrm *matrix, int nrhs, double alpha,
                                 double *A, int lda, double beta, double *B,
                                 int ldb)
{
    return starsh_blrm__dmml_b200(matrix, nrhs, alpha, A, lda, beta, B, ldb);
}

extern "C" double starsh_blrm__dfe_b200(STARSH_blrm *matrix)
{
    if (matrix == nullptr) return -1.0;
    Context *ctx = context();
    if (!ctx) return -1.0;
    std::lock_guard<std::mutex> guard(ctx->lock);
    return dfe_device(matrix, *ctx);
}

extern "C" double starsh_blrm__dfe(STARSH_blrm *matrix)
{
    return starsh_blrm__dfe_b200(matrix);
}

extern "C" int starsh_b200_blrm_dfe_sums(STARSH_blrm *matrix, double *diff2,
                                         double *norm2)
{
    if (matrix == nullptr || diff2 == nullptr || norm2 == nullptr)
        return STARSH_WRONG_PARAMETER;
    Context *ctx = context();
    if (!ctx) return STARSH_UNKNOWN_ERROR;
    std::lock_guard<std::mutex> guard(ctx->lock);
    return dfe_sums_device(matrix, *ctx, diff2, norm2);
}
