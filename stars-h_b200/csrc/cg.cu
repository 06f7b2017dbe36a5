// Conjugate gradients on a TLR matrix whose factors stay on the device:
// the iteration of starsh_itersolvers__dcg_omp (reference
// src/itersolvers/cg.c:24-95) with every product a device dmml and every
// vector operation a device kernel.  Per right-hand side j:
//     r = b - M x, p = r, rs = ||r||, check = tol rs;
//     repeat: q = M p; alpha = rs^2 / (p . q); x += alpha p; r -= alpha q;
//             rs' = ||r||; if rs' < check the column is finished;
//             else p = r + (rs'^2 / rs^2) p, rs = rs'.
// The result is the number of the iteration at which the last column
// finished (as the reference returns it) or -1 after n iterations.  Dot
// products and norms are reductions in a fixed order, so the iteration is
// deterministic.
//
// One launch does an iteration's vector work.  Thread t of a column's 256
// sums the rows t, t + 256, ... in order, then the warps' sums are added in
// order -- the iteration count of a symmetric matrix is sensitive to the
// last bit -- and the eight warps are the CTAs of a cluster, so that a
// column's loads spread over eight SMs, twenty rows of a thread at a time
// (n = 10000: 12 us; one CTA per column, two launches, a row at a time: 58).  The host reads an iteration's count of finished columns one
// iteration late: the iteration already queued then changes nothing, every
// column being finished.
#include <cmath>
#include <cooperative_groups.h>
#include <mutex>
#include <vector>

#include "device_ctx.cuh"
#include "records.cuh"
#include "starsh-b200.h"

namespace b200 {

constexpr int kCgThreads = 256;    // threads of a column
constexpr int kCgWarps = 8;        // ... one warp in each CTA of its cluster
constexpr int kCgUnroll = 20;

namespace cg = cooperative_groups;

// Per-column scalars of the iteration.
struct CgCol {
    double rsold;    // ||r||^2 of the previous iteration
    double check;    // tol ||r_0||
    int active;
};

// The column's sum of v over its 256 threads, tree in a warp, then the warps
// in order; every thread gets it.  `red`: kCgWarps doubles in each CTA, not
// read by an earlier call's readers any more.
__device__ __forceinline__ double column_sum(cg::cluster_group &cl, double v,
                                             double *red)
{
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x < kCgWarps)
        *cl.map_shared_rank(red + cl.block_rank(), (int)threadIdx.x) = v;
    cl.sync();
    double s = 0.0;
    for (int q = 0; q < kCgWarps; ++q) s += red[q];
    return s;
}

// This thread's rows i, i + 256, ... of the column in groups of kCgUnroll:
// load(i, u) for a whole group, then use(i, u) in order (u: place in the
// group).
template <class Load, class Use>
__device__ __forceinline__ void column_rows(int i, int n, const Load &load,
                                            const Use &use)
{
    for (; i < n; i += kCgThreads * kCgUnroll) {
        #pragma unroll
        for (int u = 0; u < kCgUnroll; ++u)
            if (i + u * kCgThreads < n) load(i + u * kCgThreads, u);
        #pragma unroll
        for (int u = 0; u < kCgUnroll; ++u)
            if (i + u * kCgThreads < n) use(i + u * kCgThreads, u);
    }
}

// r_j = b_j + r_j (r holds -M x), p_j = r_j, the column's initial scalars.
__global__ void __cluster_dims__(kCgWarps, 1, 1) __launch_bounds__(32)
k_cg_init(const double *__restrict__ B, int ldb, double *__restrict__ R,
          double *__restrict__ P, int n, double tol, CgCol *cols)
{
    __shared__ double red[kCgWarps];
    cg::cluster_group cl = cg::this_cluster();
    const int j = blockIdx.x / kCgWarps, i0 = blockIdx.x % kCgWarps * 32 + threadIdx.x;
    double *r = R + (size_t)j * n, *p = P + (size_t)j * n;
    const double *b = B + (size_t)j * ldb;
    double s = 0.0;
    double vr[kCgUnroll], vb[kCgUnroll];
    cl.sync();          // every CTA of the cluster runs: its shared memory is there
    column_rows(i0, n,
        [&](int i, int u) { vr[u] = r[i]; vb[u] = b[i]; },
        [&](int i, int u) {
            const double v = vr[u] + vb[u];
            r[i] = v;
            p[i] = v;
            s += v * v;
        });
    s = column_sum(cl, s, red);
    if (i0 == 0) {
        const double nrm = sqrt(s);
        cols[j].check = nrm * tol;
        cols[j].rsold = s;
        cols[j].active = 1;
    }
}

// alpha = rs^2 / (p . q); r -= alpha q, ||r||, the convergence test; x +=
// alpha p and, for columns still running, p = r + beta p.
__global__ void __cluster_dims__(kCgWarps, 1, 1) __launch_bounds__(32)
k_cg_iter(double *__restrict__ X, int ldx, double *__restrict__ R,
          double *__restrict__ P, const double *__restrict__ Q, int n,
          CgCol *cols, int *finished)
{
    __shared__ double red[2][kCgWarps];
    cg::cluster_group cl = cg::this_cluster();
    const int j = blockIdx.x / kCgWarps, i0 = blockIdx.x % kCgWarps * 32 + threadIdx.x;
    const CgCol c = cols[j];
    // (also: every CTA has read the scalars before the first one writes them)
    cl.sync();
    if (!c.active) return;
    double *x = X + (size_t)j * ldx, *r = R + (size_t)j * n;
    double *p = P + (size_t)j * n;
    const double *q = Q + (size_t)j * n;
    double va[kCgUnroll], vb[kCgUnroll], vc[kCgUnroll];
    double s = 0.0;
    column_rows(i0, n,
        [&](int i, int u) { va[u] = p[i]; vb[u] = q[i]; },
        [&](int, int u) { s += va[u] * vb[u]; });
    s = column_sum(cl, s, red[0]);
    const double alpha = c.rsold / s;
    s = 0.0;
    column_rows(i0, n,
        [&](int i, int u) { va[u] = r[i]; vb[u] = q[i]; },
        [&](int i, int u) {
            const double v = va[u] - alpha * vb[u];
            r[i] = v;
            s += v * v;
        });
    s = column_sum(cl, s, red[1]);
    const bool done = sqrt(s) < c.check;
    if (i0 == 0) {
        if (done) {
            cols[j].active = 0;
            atomicAdd(finished, 1);
        } else {
            cols[j].rsold = s;
        }
    }
    const double beta = s / c.rsold;
    column_rows(i0, n,
        [&](int i, int u) { va[u] = x[i]; vb[u] = p[i]; vc[u] = r[i]; },
        [&](int i, int u) {
            x[i] = va[u] + alpha * vb[u];
            if (!done) p[i] = vc[u] + beta * vb[u];
        });
}

// Device CG; returns the iteration count as the reference does, -1 when
// not converged within n iterations, or -2 - (STARSH error) on failure.
static int cg_device(STARSH_blrm *M, int nrhs, const double *dB, int ldb,
                     double *dX, int ldx, double tol, int maxiter,
                     cudaStream_t user, Context &ctx, int *info)
{
    *info = STARSH_SUCCESS;
    cudaStream_t s = ctx.stream;
    const int n = (int)M->format->problem->shape[0];
    double *work = (double *)pool_alloc((size_t)3 * n * nrhs * sizeof(double), s);
    CgCol *cols = (CgCol *)pool_alloc(nrhs * sizeof(CgCol), s);
    int *fin = (int *)pool_alloc(sizeof(int), s);
    int *seen = (int *)host_pinned_alloc(2 * sizeof(int));
    cudaEvent_t ev[3] = {nullptr, nullptr, nullptr};
    bool ok = work && cols && fin && seen;
    for (cudaEvent_t &e : ev)
        ok = ok && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) == cudaSuccess;
    int result = -1, e = ok ? STARSH_SUCCESS : STARSH_MALLOC_ERROR;
    if (!e) {
        // everything on the library stream, between the caller's work
        if (user != s) {
            cudaEventRecord(ev[2], user);
            cudaStreamWaitEvent(s, ev[2], 0);
        }
        double *R = work, *P = R + (size_t)n * nrhs, *Q = P + (size_t)n * nrhs;
        cudaMemsetAsync(fin, 0, sizeof(int), s);
        // r = -M x, then r += b
        e = dmml_device(M, nrhs, -1.0, dX, ldx, 0.0, R, n, s, ctx);
        if (!e) {
            k_cg_init<<<kCgWarps * nrhs, 32, 0, s>>>(dB, ldb, R, P, n, tol, cols);
            count_launch();
        }
        // finished columns after iteration `it`, in seen[it & 1]
        auto converged = [&](int it) {
            if (cudaEventSynchronize(ev[it & 1]) != cudaSuccess) {
                e = cuda_fail(cudaGetLastError(), "cg iteration");
                return true;
            }
            if (((volatile int *)seen)[it & 1] != nrhs) return false;
            result = it;
            return true;
        };
        bool stop = false;
        for (int it = 0; !e && !stop && it < maxiter; ++it) {
            const int cur = it & 1;
            if ((e = dmml_device(M, nrhs, 1.0, P, n, 0.0, Q, n, s, ctx))) break;
            k_cg_iter<<<kCgWarps * nrhs, 32, 0, s>>>(dX, ldx, R, P, Q, n, cols, fin);
            count_launch();
            if (cudaMemcpyAsync(seen + cur, fin, sizeof(int), cudaMemcpyDeviceToHost, s) !=
                    cudaSuccess ||
                cudaEventRecord(ev[cur], s) != cudaSuccess) {
                e = cuda_fail(cudaGetLastError(), "cg iteration");
                break;
            }
            if (it > 0) stop = converged(it - 1);
            if (!stop && it + 1 == maxiter) converged(it);
        }
        if (user != s) {
            cudaEventRecord(ev[2], s);
            cudaStreamWaitEvent(user, ev[2], 0);
        }
        const cudaError_t ce = cudaGetLastError();
        if (!e && ce != cudaSuccess) e = cuda_fail(ce, "cg kernels");
        // the copies into `seen` are done before it goes back
        cudaStreamSynchronize(s);
    }
    *info = e;
    for (cudaEvent_t x : ev)
        if (x) cudaEventDestroy(x);
    if (seen) host_pinned_free(seen);
    pool_free(work);
    pool_free(cols);
    pool_free(fin);
    return result;
}

}  // namespace b200

using namespace b200;

extern "C" int starsh_b200_dcg_device(STARSH_blrm *matrix, int nrhs,
                                      const double *dB, int ldb, double *dX,
                                      int ldx, double tol, int maxiter,
                                      void *stream, int *iterations)
{
    if (matrix == nullptr || nrhs <= 0 || dB == nullptr || dX == nullptr ||
        iterations == nullptr || !(tol >= 0.0))
        return STARSH_WRONG_PARAMETER;
    const int n = (int)matrix->format->problem->shape[0];
    if (ldb < n || ldx < n) return STARSH_WRONG_PARAMETER;
    Context *ctx = context();
    if (!ctx) return STARSH_UNKNOWN_ERROR;
    std::lock_guard<std::mutex> guard(ctx->lock);
    cudaStream_t s = stream ? (cudaStream_t)stream : ctx->stream;
    int info;
    *iterations = cg_device(matrix, nrhs, dB, ldb, dX, ldx, tol,
                            maxiter > 0 ? maxiter : n, s, *ctx, &info);
    return info;
}

// Signature of starsh_itersolvers__dcg_omp (reference include/starsh.h:671-672)
// with host B and X; `work` is not used (the iteration's vectors live on
// the device).  Returns the iteration count, or -1 if not converged (or on
// an error, which starsh_b200_last_error() describes).
extern "C" int starsh_itersolvers__dcg_b200(STARSH_blrm *matrix, int nrhs,
                                            double *B, int ldb, double *X,
                                            int ldx, double tol, double *work)
{
    (void)work;
    if (matrix == nullptr || nrhs <= 0 || B == nullptr || X == nullptr)
        return -1;
    const int n = (int)matrix->format->problem->shape[0];
    if (ldb < n || ldx < n) return -1;
    Context *ctx = context();
    if (!ctx) return -1;
    std::lock_guard<std::mutex> guard(ctx->lock);
    cudaStream_t s = ctx->stream;
    double *dB = (double *)pool_alloc((size_t)2 * n * nrhs * sizeof(double), s);
    if (dB == nullptr) {
        cuda_fail(cudaErrorMemoryAllocation, "cg vectors");
        return -1;
    }
    double *dX = dB + (size_t)n * nrhs;
    cudaMemcpy2DAsync(dB, n * sizeof(double), B, (size_t)ldb * sizeof(double),
                      n * sizeof(double), nrhs, cudaMemcpyHostToDevice, s);
    cudaMemcpy2DAsync(dX, n * sizeof(double), X, (size_t)ldx * sizeof(double),
                      n * sizeof(double), nrhs, cudaMemcpyHostToDevice, s);
    int info;
    const int it = cg_device(matrix, nrhs, dB, n, dX, n, tol, n, s, *ctx, &info);
    if (info == STARSH_SUCCESS)
        cudaMemcpy2DAsync(X, (size_t)ldx * sizeof(double), dX, n * sizeof(double),
                          n * sizeof(double), nrhs, cudaMemcpyDeviceToHost, s);
    cudaStreamSynchronize(s);
    pool_free(dB);
    return info == STARSH_SUCCESS ? it : -1;
}
