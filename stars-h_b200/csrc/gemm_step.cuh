// The product of one tile in a GEMM step of the engine: operands, shapes and
// leading dimensions from the tile's record and the workspace layout.  An
// empty product (M = 0) where the tile takes no part in the step.
#pragma once
#include "engine.cuh"

namespace b200 {

__device__ __forceinline__ GemmDesc gemm_desc(const GemmArgs &a, int index)
{
    const TileWork &tw = a.tiles[a.act ? a.act[index] : index];
    const Workspace &ws = a.ws;
    const int s = tw.slot;
    GemmDesc d;
    d.alpha = 1.0;
    d.beta = 0.0;
    d.M = d.N = d.K = 0;
    d.A = d.B = nullptr;
    d.C = nullptr;
    d.lda = d.ldb = d.ldc = 1;
    d.gather = d.gather_b = nullptr;
    const int ldm = ws.ldM(), ldk = ws.ldK();
    switch (a.step) {
    case STEP_SKETCH:
        d.A = ws.D(s); d.lda = ws.ldD();
        d.B = a.omega; d.ldb = a.ld_omega;
        d.C = ws.Y(s); d.ldc = ldm;
        d.M = tw.m; d.N = tw.k; d.K = tw.n;
        break;
    case STEP_GRAM_YR:  // TN, residual of pass B
        if (!tw.need_pass_b) break;
        d.A = ws.Y(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k; d.N = tw.k; d.K = tw.m;
        break;
    case STEP_GRAM_Y:   // TN
        d.A = ws.Y(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k; d.N = tw.k; d.K = tw.m;
        break;
    case STEP_Q1:       // NN: Q1buf = Qbuf(gathered) * T
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.T(s); d.ldb = ldk;
        d.C = ws.Q1(s); d.ldc = ldm;
        d.M = tw.m; d.N = tw.k1; d.K = tw.k1;
        break;
    case STEP_GRAM_Q1:  // TN
        d.A = ws.Q1(s); d.lda = ldm;
        d.B = ws.Q1(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.k1; d.K = tw.m;
        break;
    case STEP_Q:        // NN: Qbuf = Q1buf * T
        d.A = ws.Q1(s); d.lda = ldm;
        d.B = ws.T(s); d.ldb = ldk;
        d.C = ws.Q(s); d.ldc = ldm;
        d.M = tw.m; d.N = tw.k1; d.K = tw.k1;
        break;
    case STEP_RES_Z:    // TN: S = Q^T Y
        if (!tw.need_pass_b) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.k; d.K = tw.m;
        break;
    case STEP_RES_Y:    // NN: Y -= Q S
        if (!tw.need_pass_b) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.S(s); d.ldb = ldk;
        d.C = ws.Y(s); d.ldc = ldm;
        d.alpha = -1.0; d.beta = 1.0;
        d.M = tw.m; d.N = tw.k; d.K = tw.k1;
        break;
    case STEP_Q1B:      // NN: Ybuf = Q1buf(gathered residual) * T
        if (tw.kb <= 0) break;
        d.A = ws.Q1(s); d.lda = ldm;
        d.B = ws.T(s); d.ldb = ldk;
        d.C = ws.Y(s); d.ldc = ldm;
        d.M = tw.m; d.N = tw.kb; d.K = tw.kb;
        break;
    case STEP_RES_Z2:   // TN: S = Q^T Ybuf
        if (tw.kb <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.kb; d.K = tw.m;
        break;
    case STEP_RES_Q1B:  // NN: Ybuf -= Q S
        if (tw.kb <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.S(s); d.ldb = ldk;
        d.C = ws.Y(s); d.ldc = ldm;
        d.alpha = -1.0; d.beta = 1.0;
        d.M = tw.m; d.N = tw.kb; d.K = tw.k1;
        break;
    case STEP_GRAM_Q1B: // TN
        if (tw.kb <= 0) break;
        d.A = ws.Y(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.kb; d.N = tw.kb; d.K = tw.m;
        break;
    case STEP_QB:       // NN: Q[:, k1:k1+kb] = Ybuf T
        if (tw.kb <= 0) break;
        d.A = ws.Y(s); d.lda = ldm;
        d.B = ws.T(s); d.ldb = ldk;
        d.C = ws.Q(s) + (size_t)tw.k1 * ldm; d.ldc = ldm;
        d.M = tw.m; d.N = tw.kb; d.K = tw.kb;
        break;
    case STEP_PROJECT:  // TN: B = Q^T D
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.D(s); d.ldb = ws.ldD();
        d.C = ws.B(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.n; d.K = tw.m;
        if (tw.status & TILE_PROJ_I8) d.M = 0;   // on the tensor cores
        break;
    case STEP_GRAM_B:   // NT: S = B B^T
        d.A = ws.B(s); d.lda = ldk;
        d.B = ws.B(s); d.ldb = ldk;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.k1; d.K = tw.n;
        break;
    case STEP_ROTATE:   // TN: C = W^T B, W in T
        d.A = ws.T(s); d.lda = ldk;
        d.B = ws.B(s); d.ldb = ldk;
        d.C = ws.C(s); d.ldc = ldk;
        d.M = tw.k2; d.N = tw.n; d.K = tw.k1;
        break;
    case STEP_A_SKETCH: // NN: Y = D Omega[:, c:c+b]
        if (tw.bcur <= 0) break;
        d.A = ws.D(s); d.lda = ws.ldD();
        d.B = a.omega + (size_t)tw.cols_done * a.ld_omega; d.ldb = a.ld_omega;
        d.C = ws.Y(s); d.ldc = ldm;
        d.M = tw.m; d.N = tw.bcur; d.K = tw.n;
        break;
    case STEP_A_RES_Z:  // TN: S = Q^T Y
        if (tw.bcur <= 0 || tw.k1 <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.bcur; d.K = tw.m;
        break;
    case STEP_A_RES_Y:  // NN: Y -= Q S
        if (tw.bcur <= 0 || tw.k1 <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.S(s); d.ldb = ldk;
        d.C = ws.Y(s); d.ldc = ldm;
        d.alpha = -1.0; d.beta = 1.0;
        d.M = tw.m; d.N = tw.bcur; d.K = tw.k1;
        break;
    case STEP_A_GRAM:   // TN: S = Y^T Y
        if (tw.bcur <= 0) break;
        d.A = ws.Y(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.bcur; d.N = tw.bcur; d.K = tw.m;
        break;
    case STEP_A_RES_Z2: // TN: S = Q^T Y, repeat pass on the same sample
        if (!tw.need_pass_b || tw.bcur <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.bcur; d.K = tw.m;
        break;
    case STEP_A_RES_Y2: // NN: Y -= Q S
        if (!tw.need_pass_b || tw.bcur <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.S(s); d.ldb = ldk;
        d.C = ws.Y(s); d.ldc = ldm;
        d.alpha = -1.0; d.beta = 1.0;
        d.M = tw.m; d.N = tw.bcur; d.K = tw.k1;
        break;
    case STEP_A_GRAM2:  // TN: S = Y^T Y
        if (!tw.need_pass_b || tw.bcur <= 0) break;
        d.A = ws.Y(s); d.lda = ldm;
        d.B = ws.Y(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.bcur; d.N = tw.bcur; d.K = tw.m;
        break;
    case STEP_A_Q1B:    // NN: R = (pivot columns of the residual) T
        if (tw.kb <= 0) break;
        d.A = ws.Y(s); d.lda = ldm; d.gather = ws.Piv(s);
        d.B = ws.T(s); d.ldb = ldk;
        d.C = ws.R(s); d.ldc = ldm;
        d.M = tw.m; d.N = tw.kb; d.K = tw.kb;
        break;
    case STEP_A_ORTH_Z: // TN: S = Q^T R
        if (tw.kb <= 0 || tw.k1 <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.R(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.k1; d.N = tw.kb; d.K = tw.m;
        break;
    case STEP_A_ORTH_R: // NN: R -= Q S
        if (tw.kb <= 0 || tw.k1 <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.S(s); d.ldb = ldk;
        d.C = ws.R(s); d.ldc = ldm;
        d.alpha = -1.0; d.beta = 1.0;
        d.M = tw.m; d.N = tw.kb; d.K = tw.k1;
        break;
    case STEP_A_GRAM_R: // TN: S = R^T R
        if (tw.kb <= 0) break;
        d.A = ws.R(s); d.lda = ldm;
        d.B = ws.R(s); d.ldb = ldm;
        d.C = ws.S(s); d.ldc = ldk;
        d.M = tw.kb; d.N = tw.kb; d.K = tw.m;
        break;
    case STEP_A_QB:     // NN: Q[:, k1:k1+kb] = R T
        if (tw.kb <= 0) break;
        d.A = ws.R(s); d.lda = ldm;
        d.B = ws.T(s); d.ldb = ldk;
        d.C = ws.Q(s) + (size_t)tw.k1 * ldm; d.ldc = ldm;
        d.M = tw.m; d.N = tw.kb; d.K = tw.kb;
        break;
    case STEP_OUT_U:    // NN: U = Q W(:, ord), W in T
        if (tw.rank <= 0) break;
        d.A = ws.Q(s); d.lda = ldm;
        d.B = ws.T(s); d.ldb = ldk; d.gather_b = ws.Ord(s);
        d.C = a.out.U + tw.off_u; d.ldc = tw.m;
        d.M = tw.m; d.N = tw.rank; d.K = tw.k1;
        break;
    }
    return d;
}

}  // namespace b200
