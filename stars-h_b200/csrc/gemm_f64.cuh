// Batched FP64 GEMM on the double-precision tensor-core path
// (mma.sync m8n8k4 .f64).  Every batch entry has its own operands and
// shape, so one launch covers all tiles of a batch even when their ranks
// differ:
//     C = alpha * op(A) * op(B) + beta * C,   op(A): M x K, op(B): K x N,
// all matrices column-major (gemm_f64.cu: one kernel for each shape of
// product).
#pragma once
#include <cuda_runtime.h>

namespace b200 {

struct GemmDesc {
    const double *A;
    const double *B;
    double *C;
    int M, N, K;
    int lda, ldb, ldc;
    double alpha, beta;
    // A B form: column k of A is column gather[k], column n of B column
    // gather_b[n] (or null)
    const int *gather, *gather_b;
};

constexpr int kGemmBK = 16;
constexpr int kGemmThreads = 256;
// Shared-memory row stride (doubles) of the [row][k] tiles: 20 puts the
// 4x4 (row, k) footprint of a half-warp fragment load on 16 distinct bank
// pairs.
constexpr int kGemmLds = kGemmBK + 4;

}  // namespace b200
