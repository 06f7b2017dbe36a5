// Device kernels of the batched randomized-SVD engine (FP64 path).
//
// Per tile (D: m x n block, Omega: n x k Gaussian, k = min(maxrank +
// oversample, m, n)) the engine computes the same factorisation as the
// reference's starsh_dense_dlrrsdd (src/backends/sequential/dense/
// drsdd.c:16-93): Y = D Omega, an orthonormal basis Q of range(Y),
// B = Q^T D, the SVD of B, the rank cut of starsh_dense_dsvfr
// (src/backends/sequential/dense/dsvfr.c:16-47) and U = Q Us_r,
// V = (S_r Vs_r)^T.  The orthogonalisation and the small SVD are done with
// Gram matrices so that every O(m n k) and O(m k^2) step is a GEMM:
//   * basis: pivoted Cholesky of Y^T Y drops directions below the FP64
//     squared-noise floor or below (tol/10)^2 of the sketch energy, CholQR2
//     on the kept columns; when tol^2 is below the squared-noise floor a
//     second pass orthogonalises the explicit residual Y - Q Q^T Y, which
//     recovers the directions the squared Gram could not resolve;
//   * small SVD: B B^T = L L^T (pivoted Cholesky), one-sided Jacobi on L
//     gives the left singular vectors W of B; the energies of the rotated
//     rows C = W^T B are summed in FP64 directly from C, so the tail that
//     decides the rank is exact to FP64 rounding even where the Gram's
//     eigenvalues are not.
#include <cfloat>
#include <climits>
#include <cooperative_groups.h>
#include "engine.cuh"
#include "smem_limit.cuh"

namespace b200 {

// ------------------------------------------------------------ layout

size_t workspace_layout(Workspace &w, int m_max, int n_max, int k_max,
                        bool store_d, bool proj_digits)
{
    size_t o = 0;
    auto take = [&](size_t n) {
        const size_t r = o;
        o += (n + 31) & ~(size_t)31;   // 256-byte aligned fields
        return r;
    };
    w.m_max = m_max;
    w.n_max = n_max;
    w.k_max = k_max;
    w.oD = store_d ? take((size_t)m_max * n_max) : 0;
    w.oY = take((size_t)m_max * k_max);
    w.oQ1 = take((size_t)m_max * k_max);
    w.oQ = take((size_t)m_max * k_max);
    w.oS = take((size_t)k_max * k_max);
    w.oL = take((size_t)k_max * k_max);
    w.oT = take((size_t)k_max * k_max);
    w.oB = take((size_t)k_max * n_max);
    w.oC = take((size_t)k_max * n_max);
    w.oE = take(k_max);
    w.oSig = take(k_max);
    w.oPiv = take((k_max + 1) / 2);
    w.oOrd = take((k_max + 1) / 2);
    w.oNrm = take((size_t)((m_max + 63) / 64) * ((n_max + 63) / 64));
    w.oR = take((size_t)m_max * k_max);
    w.oRmx = take((size_t)m_max * ((n_max + 63) / 64));
    w.oQd = w.oQe = w.oQf = 0;
    if (proj_digits) {
        // 7 byte slices x 64 basis columns x ldQd bytes; m ints; 64 ints
        w.oQd = take((size_t)7 * 64 * ((m_max + 31) / 32 * 32) / 8);
        w.oQe = take(((size_t)m_max + 1) / 2);
        w.oQf = take(32);
    }
    w.stride = o;
    return o;
}

// -------------------------------------------------------- generation

// D(slot) = block of the tile, column-major with ld = m_max.  A CTA owns
// 64 rows and kGenCb column blocks of 64: the coordinates of its rows and
// columns are gathered through the cluster pivots into shared memory once
// (point-major layouts and dimensions above kStageDim read global memory
// directly), then each thread evaluates 16 entries of one row in each
// 64 x 64 block, so stores run down the columns and are coalesced.  Per
// 64 x 64 block the CTA writes the sum of squares of its entries to
// Nrm(slot) and each row's largest |D_ij| to Rmx(slot), reduced in a fixed
// order (deterministic per-tile norms for the adaptive sketch).  Several
// blocks per CTA spread the gathers and barriers of the staging over more
// entries.
constexpr int kStageDim = 4;
#ifndef GEN_CB
#define GEN_CB 4              // 64-column blocks of one generator CTA
#endif
constexpr int kGenCb = GEN_CB;
#ifndef GEN_MIN_BLOCKS
#define GEN_MIN_BLOCKS 3      // CTAs per SM the generator is compiled for
#endif
#ifndef GEN_MIN_BLOCKS_FIX
#define GEN_MIN_BLOCKS_FIX 4  // the same for a launch of one kernel family
#endif
#ifndef GEN_MIN_BLOCKS_MATERN
#define GEN_MIN_BLOCKS_MATERN 4   // ... of the Matérn family (its rare
#endif                            // series path spills; measured faster)
#ifndef GEN_UNROLL
#define GEN_UNROLL 8          // entries of a thread evaluated together
#endif
constexpr int kGenUnroll = GEN_UNROLL;
#ifndef GEN_UNROLL_MATERN
#define GEN_UNROLL_MATERN 2   // the same for the Matérn families
#endif

// The entries of one thread in a 64 x 64 block: rows ii, columns jj0,
// jj0 + 4, ... below jn, written to Dcol[jj * ld] (Dcol points at row ii of
// the block's first column); returns their sum of squares.  `amax` gets a
// value with the exponent of their largest |D_ij| (all that the row scales
// use): the maximum of the high words, one integer instruction per entry
// (the low words' bits where every high word is zero).  The generator is
// bound by issue slots (82 % busy), so what an entry does not need is left
// out at compile time: PLAIN is entry_plain, and the first squared
// difference starts the distance.  Two-dimensional square exponential, N =
// 102400: 30.2 -> 25.3 ms, the same bits.
template <int FAM, int NDIM, int LDC, bool PLAIN>
__device__ __forceinline__ double gen_entries(
    const DevKernel &K, bool staged, const double (*rc)[64],
    const double (*cc)[LDC], const long long *ri, const long long *ci, int ii,
    int jj0, int jn, double *Dcol, int ld, double &amax)
{
    // NDIM > 0: coordinates staged in shared memory, dimension known at
    // compile time (the row's coordinates held in registers); NDIM == 0:
    // staged, any dimension up to kStageDim; NDIM < 0: read through the
    // pivots from global memory
    double xr[NDIM > 0 ? NDIM : 1];
    if constexpr (NDIM > 0) {
        #pragma unroll
        for (int d = 0; d < NDIM; ++d) xr[d] = rc[d][ii];
    }
    double ss = 0.0;
    unsigned hmax = 0, lbits = 0;
    // the Matern entry (table piece per entry) keeps a shorter unroll:
    // more of its bodies cost more registers than they save
    constexpr int kUnroll =
        FAM == FAM_MATERN || FAM == FAM_MATERN2 ? GEN_UNROLL_MATERN : kGenUnroll;
    #pragma unroll kUnroll
    for (int jj = jj0; jj < jn; jj += 4) {
        double dist = 0.0;
        if constexpr (NDIM > 0) {
            #pragma unroll
            for (int d = 0; d < NDIM; ++d) {
                const double q = __dsub_rn(xr[d], cc[d][jj]);
                dist = d == 0 ? __dmul_rn(q, q) : __dadd_rn(dist, __dmul_rn(q, q));
            }
        } else if constexpr (NDIM == 0) {
            for (int d = 0; d < K.ndim; ++d) {
                const double q = __dsub_rn(rc[d][ii], cc[d][jj]);
                dist = __dadd_rn(dist, __dmul_rn(q, q));
            }
        } else {
            dist = sq_dist(K, ri[ii], ci[jj]);
        }
        double v;
        if constexpr (PLAIN) v = entry_plain<FAM>(K, dist);
        else v = entry_fam<FAM>(K, dist, ri[ii], ci[jj]);
        Dcol[(size_t)jj * ld] = v;
        ss += v * v;
        hmax = max(hmax, (unsigned)__double2hiint(v) & 0x7fffffffu);
        lbits |= (unsigned)__double2loint(v);
    }
    amax = __hiloint2double((int)hmax, hmax == 0 ? (int)lbits : 0);
    return ss;
}

// Dispatch on the staging dimension for one family.
template <int FAM, int LDC, bool PLAIN = false>
__device__ __forceinline__ double gen_entries_dim(
    const DevKernel &K, bool staged, const double (*rc)[64],
    const double (*cc)[LDC], const long long *ri, const long long *ci, int ii,
    int jj0, int jn, double *Dcol, int ld, double &amax)
{
    if (!staged)
        return gen_entries<FAM, -1, LDC, PLAIN>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    if (K.ndim == 2)
        return gen_entries<FAM, 2, LDC, PLAIN>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    if (K.ndim == 3)
        return gen_entries<FAM, 3, LDC, PLAIN>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    return gen_entries<FAM, 0, LDC, PLAIN>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
}

// The 16 entries of each thread in one 64 x 64 block of a generator CTA
// (columns jb0 .. jb0 + 63 of the tile), family dispatched once.
template <int LDC>
__device__ __forceinline__ double gen_block(
    const DevKernel &K, bool staged, const double (*rc)[64],
    const double (*cc)[LDC], const long long *ri, const long long *ci, int ii,
    int jj0, int jn, double *Dcol, int ld, double &amax)
{
    switch (K.family) {
    case FAM_EXP:
        return gen_entries_dim<FAM_EXP, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    case FAM_SQREXP:
        return gen_entries_dim<FAM_SQREXP, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    case FAM_MATERN:
        return gen_entries_dim<FAM_MATERN, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    case FAM_MATERN2:
        return gen_entries_dim<FAM_MATERN2, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    case FAM_COULOMB:
        return gen_entries_dim<FAM_COULOMB, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    case FAM_SIN:
        return gen_entries_dim<FAM_SIN, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    case FAM_COS:
        return gen_entries_dim<FAM_COS, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    default:
        return gen_entries_dim<FAM_RBF, LDC>(K, staged, rc, cc, ri, ci, ii, jj0, jn, Dcol, ld, amax);
    }
}

// FIX != 0: every tile of the launch has kernel family FIX (the family's
// entry code alone, compiled for MINB CTAs per SM); FIX == 0: the family
// is read per CTA.
template <int FIX, int MINB, bool PLAIN = false>
__global__ void __launch_bounds__(256, MINB)
k_gen_tiles(const DevKernel *__restrict__ kernels,
            const TileWork *__restrict__ tiles, Workspace ws, int need)
{
    constexpr int W = 64 * kGenCb;   // columns of the CTA
    const TileWork tw = tiles[blockIdx.z];
    if (blockIdx.x * 64 >= tw.m || blockIdx.y * W >= tw.n) return;
    if (need != 0 && (tw.status & need) == 0) return;
    __shared__ double rc[kStageDim][64], cc[kStageDim][W];
    __shared__ long long ri[64], ci[W];
    __shared__ double red[kGenCb][8];
    __shared__ double rmx[kGenCb][4][64];
    __shared__ DevKernel Ks;
    const int t = threadIdx.x;
    if (t == 0) Ks = kernels[tw.prob];
    __syncthreads();
    const DevKernel &K = Ks;
    const int i0 = blockIdx.x * 64, j0 = blockIdx.y * W;
    const int ncol = min(W, tw.n - j0);      // columns of this CTA
    const bool staged = !K.aos && K.ndim <= kStageDim;
    if (t < 64) {
        const int i = min(i0 + t, tw.m - 1);
        ri[t] = K.row_piv[tw.row0 + i];
    }
    for (int e = t; e < W; e += 256) {
        const int j = min(j0 + e, tw.n - 1);
        ci[e] = K.col_piv[tw.col0 + j];
    }
    __syncthreads();
    if (staged) {
        for (int q = t; q < 64 * K.ndim; q += 256) {
            const int d = q / 64, e = q % 64;
            rc[d][e] = K.row_pt[d * K.row_count + ri[e]];
        }
        for (int q = t; q < W * K.ndim; q += 256) {
            const int d = q / W, e = q % W;
            cc[d][e] = K.col_pt[d * K.col_count + ci[e]];
        }
    }
    __syncthreads();
    const int ii = t & 63, i = i0 + ii;
    double *D = ws.D(tw.slot);
    const int ld = ws.ldD();
    #pragma unroll 1
    for (int b = 0; b < kGenCb; ++b) {
        const int jb = b * 64;                // first column of the block
        if (jb >= ncol) break;
        double ss = 0.0, amax = 0.0;
        if (i < tw.m)
            ss = FIX == 0
                ? gen_block<W>(K, staged, rc, (const double (*)[W])&cc[0][jb],
                               ri, ci + jb, ii, t >> 6, min(64, ncol - jb),
                               D + (size_t)(j0 + jb) * ld + i, ld, amax)
                : gen_entries_dim<FIX == 0 ? FAM_EXP : FIX, W, PLAIN>(
                      K, staged, rc, (const double (*)[W])&cc[0][jb], ri,
                      ci + jb, ii, t >> 6, min(64, ncol - jb),
                      D + (size_t)(j0 + jb) * ld + i, ld, amax);
        // largest |D_ij| of each row of the block (the int8 sketch's row
        // scales): the four threads of a row combine through shared memory
        rmx[b][t >> 6][ii] = amax;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_down_sync(0xffffffffu, ss, o);
        if ((t & 31) == 0) red[b][t >> 5] = ss;
    }
    __syncthreads();
    const int nbc = (ws.n_max + 63) / 64;     // 64-column blocks of a tile row
    const int nblk = (ncol + 63) / 64;
    for (int q = t; q < 64 * nblk; q += 256) {
        const int b = q / 64, r = q % 64;
        if (i0 + r < tw.m)
            ws.Rmx(tw.slot)[(size_t)(i0 + r) * nbc + blockIdx.y * kGenCb + b] =
                fmax(fmax(rmx[b][0][r], rmx[b][1][r]), fmax(rmx[b][2][r], rmx[b][3][r]));
    }
    if (t < nblk) {
        double a = 0.0;
        for (int w = 0; w < 8; ++w) a += red[t][w];
        ws.Nrm(tw.slot)[blockIdx.x * nbc + blockIdx.y * kGenCb + t] = a;
    }
}

void launch_gen_tiles(const DevKernel *d_kernels, const TileWork *d_tiles,
                      int ntiles, Workspace ws, cudaStream_t stream, int need,
                      int family, bool plain)
{
    dim3 grid((ws.m_max + 63) / 64, (ws.n_max + 64 * kGenCb - 1) / (64 * kGenCb), ntiles);
    switch (family) {
    case FAM_EXP:
        if (plain) k_gen_tiles<FAM_EXP, GEN_MIN_BLOCKS_FIX, true><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        else k_gen_tiles<FAM_EXP, GEN_MIN_BLOCKS_FIX><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        break;
    case FAM_SQREXP:
        if (plain) k_gen_tiles<FAM_SQREXP, GEN_MIN_BLOCKS_FIX, true><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        else k_gen_tiles<FAM_SQREXP, GEN_MIN_BLOCKS_FIX><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        break;
    case FAM_MATERN:
        k_gen_tiles<FAM_MATERN, GEN_MIN_BLOCKS_MATERN><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        break;
    case FAM_COULOMB:
        k_gen_tiles<FAM_COULOMB, GEN_MIN_BLOCKS_FIX><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        break;
    case FAM_SIN:
        k_gen_tiles<FAM_SIN, GEN_MIN_BLOCKS_FIX><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
        break;
    default:
        k_gen_tiles<0, GEN_MIN_BLOCKS><<<grid, 256, 0, stream>>>(d_kernels, d_tiles, ws, need);
    }
}

// ---------------------------------------------------- Gaussian sketch

// Philox4x32-10 counter-based generator (J. K. Salmon, M. A. Moraes,
// R. O. Dror, D. E. Shaw, "Parallel random numbers: as easy as 1, 2, 3",
// SC'11); multipliers and Weyl increments are the published constants.
__device__ __forceinline__ uint4 philox4x32_10(uint4 c, uint2 k)
{
    #pragma unroll
    for (int r = 0; r < 10; ++r) {
        const unsigned lo0 = 0xD2511F53u * c.x;
        const unsigned hi0 = __umulhi(0xD2511F53u, c.x);
        const unsigned lo1 = 0xCD9E8D57u * c.z;
        const unsigned hi1 = __umulhi(0xCD9E8D57u, c.z);
        c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
        k.x += 0x9E3779B9u;
        k.y += 0xBB67AE85u;
    }
    return c;
}

// Omega entries N(0,1): one Philox block -> two 53-bit uniforms in (0,1]
// -> one Box-Muller pair (G. E. P. Box, M. E. Muller, Ann. Math. Stat. 29
// (1958) 610-611).
// Entries (2q, c) and (2q + 1, c) come from the Philox block with counter
// (q, c, 0, 0).
__global__ void k_gaussian(double *out, int rows, int cols, int ld,
                           unsigned long long seed)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = blockIdx.y;
    if (2 * q >= rows || col >= cols) return;
    const uint4 c = make_uint4((unsigned)q, (unsigned)col, 0u, 0u);
    const uint4 r = philox4x32_10(c, make_uint2((unsigned)seed,
                                                (unsigned)(seed >> 32)));
    const unsigned long long b1 = ((unsigned long long)r.x << 32) | r.y;
    const unsigned long long b2 = ((unsigned long long)r.z << 32) | r.w;
    const double u1 = ((b1 >> 11) + 1) * 0x1.0p-53;   // (0, 1]
    const double u2 = (b2 >> 11) * 0x1.0p-53;         // [0, 1)
    const double rad = sqrt(-2.0 * log(u1));
    double s, co;
    sincospi(2.0 * u2, &s, &co);
    double *o = out + (size_t)col * ld;
    o[2 * q] = rad * co;
    if (2 * q + 1 < rows) o[2 * q + 1] = rad * s;
}

void launch_gaussian(double *d_omega, int rows, int cols, int ld,
                     unsigned long long seed, cudaStream_t stream)
{
    if (rows <= 0 || cols <= 0) return;
    const int pairs = (rows + 1) / 2;
    dim3 grid((pairs + 255) / 256, cols);
    k_gaussian<<<grid, 256, 0, stream>>>(d_omega, rows, cols, ld, seed);
}

// Omega8(j, c) = clip(round(32 g(j, c)), -127, 127) with g the Gaussian of
// k_gaussian for the same (j, c); rows rows .. ld - 1 are zero.
__global__ void k_gaussian_i8(int8_t *out, int rows, int cols, int ld,
                              unsigned long long seed)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    const int col = blockIdx.y;
    if (2 * q >= ld || col >= cols) return;
    const uint4 c = make_uint4((unsigned)q, (unsigned)col, 0u, 0u);
    const uint4 r = philox4x32_10(c, make_uint2((unsigned)seed,
                                                (unsigned)(seed >> 32)));
    const unsigned long long b1 = ((unsigned long long)r.x << 32) | r.y;
    const unsigned long long b2 = ((unsigned long long)r.z << 32) | r.w;
    const double u1 = ((b1 >> 11) + 1) * 0x1.0p-53;
    const double u2 = (b2 >> 11) * 0x1.0p-53;
    const double rad = sqrt(-2.0 * log(u1));
    double s, co;
    sincospi(2.0 * u2, &s, &co);
    int8_t *o = out + (size_t)col * ld;
    auto q8 = [](double g) {
        return (int8_t)fmax(-127.0, fmin(127.0, rint(32.0 * g)));
    };
    o[2 * q] = 2 * q < rows ? q8(rad * co) : (int8_t)0;
    if (2 * q + 1 < ld) o[2 * q + 1] = 2 * q + 1 < rows ? q8(rad * s) : (int8_t)0;
}

void launch_gaussian_i8(int8_t *d_om8, int rows, int cols, int ld,
                        unsigned long long seed, cudaStream_t stream)
{
    if (cols <= 0 || ld <= 0) return;
    const int pairs = (ld + 1) / 2;
    dim3 grid((pairs + 255) / 256, cols);
    k_gaussian_i8<<<grid, 256, 0, stream>>>(d_om8, rows, cols, ld, seed);
}

// ------------------------------------------------- block reductions

struct MaxLoc {
    double v;
    int i;
};

// Block-wide argmax (largest value, then smallest index).  `red` holds one
// entry per warp.  All threads get the result.
__device__ MaxLoc block_argmax(MaxLoc x, MaxLoc *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        MaxLoc y;
        y.v = __shfl_down_sync(0xffffffffu, x.v, o);
        y.i = __shfl_down_sync(0xffffffffu, x.i, o);
        if (y.v > x.v || (y.v == x.v && y.i < x.i)) x = y;
    }
    __syncthreads();
    if (lane == 0) red[warp] = x;
    __syncthreads();
    if (warp == 0) {
        x = lane < (int)(blockDim.x >> 5) ? red[lane] : MaxLoc{-DBL_MAX, 1 << 30};
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            MaxLoc y;
            y.v = __shfl_down_sync(0xffffffffu, x.v, o);
            y.i = __shfl_down_sync(0xffffffffu, x.i, o);
            if (y.v > x.v || (y.v == x.v && y.i < x.i)) x = y;
        }
        if (lane == 0) red[0] = x;
    }
    __syncthreads();
    MaxLoc r = red[0];
    __syncthreads();
    return r;
}

// block_argmax of x and, in the same pass, the block sum of y (returned in
// *sum; `reds` holds one double per warp).
__device__ MaxLoc block_argmax_sum(MaxLoc x, double y, MaxLoc *red,
                                   double *reds, double *sum)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        MaxLoc z;
        z.v = __shfl_down_sync(0xffffffffu, x.v, o);
        z.i = __shfl_down_sync(0xffffffffu, x.i, o);
        if (z.v > x.v || (z.v == x.v && z.i < x.i)) x = z;
        y += __shfl_down_sync(0xffffffffu, y, o);
    }
    __syncthreads();
    if (lane == 0) {
        red[warp] = x;
        reds[warp] = y;
    }
    __syncthreads();
    if (warp == 0) {
        const bool in = lane < (int)(blockDim.x >> 5);
        x = in ? red[lane] : MaxLoc{-DBL_MAX, 1 << 30};
        y = in ? reds[lane] : 0.0;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            MaxLoc z;
            z.v = __shfl_down_sync(0xffffffffu, x.v, o);
            z.i = __shfl_down_sync(0xffffffffu, x.i, o);
            if (z.v > x.v || (z.v == x.v && z.i < x.i)) x = z;
            y += __shfl_down_sync(0xffffffffu, y, o);
        }
        if (lane == 0) {
            red[0] = x;
            reds[0] = y;
        }
    }
    __syncthreads();
    const MaxLoc r = red[0];
    *sum = reds[0];
    __syncthreads();
    return r;
}

__device__ double block_sum(double x, double *red)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    __syncthreads();
    if (lane == 0) red[warp] = x;
    __syncthreads();
    if (warp == 0) {
        x = lane < (int)(blockDim.x >> 5) ? red[lane] : 0.0;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
        if (lane == 0) red[0] = x;
    }
    __syncthreads();
    const double r = red[0];
    __syncthreads();
    return r;
}

// ------------------------------------------------ pivoted Cholesky

// Phases: A/B basis passes of the fixed-width sketch, H small SVD, R a
// round of the adaptive sketch, R2 its repeat pass on the same sample.
enum : int { PH_A = 0, PH_B = 1, PH_H = 2, PH_R = 3, PH_R2 = 4 };

constexpr int kSmallThreads = 256;
constexpr int kPivcholLanes = 4;                 // lanes per row, large phase-H factors
constexpr int kPivcholSplit = 128;               // "large": more rows than this
constexpr int kMaxK = 1024;   // largest sketch width handled by one CTA

// Left-looking pivoted Cholesky of the Gram in S(slot) (dimension nn):
// P^T G P ~ L L^T, L stored in L(slot) with rows in the original order
// (column j holds the multipliers of pivot j).  Stops when the largest
// remaining diagonal entry is <= thr.  For the basis phases (A, B) the
// pivot block R11 = L[piv, :]^T is inverted into T(slot).
//
// LPR lanes share a row's update (the left-looking product with the
// previous columns, read from L2): more loads in flight for the large
// factors of phase H, whose few tiles per batch bound the launch.  Tiles
// with nn outside [nn_lo, nn_hi] are left to another launch.
template <int LPR>
__global__ void __launch_bounds__(kSmallThreads * LPR)
k_pivchol(TileWork *__restrict__ tiles, Workspace ws, int phase, int nn_lo,
          int nn_hi, const int *__restrict__ act)
{
    TileWork &tw = tiles[act ? act[blockIdx.x] : blockIdx.x];
    const int s = tw.slot;
    const double tol = tw.tol;
    __shared__ double dg[kMaxK];
    __shared__ double lp[kMaxK];
    __shared__ unsigned char used[kMaxK];
    __shared__ MaxLoc red[32];
    __shared__ double redd[32];

    int nn;
    if (phase == PH_H) nn = tw.k1;
    else if (phase == PH_R) nn = tw.bcur;
    else if (phase == PH_R2) nn = tw.need_pass_b ? tw.bcur : 0;
    else nn = tw.k;
    if (nn < nn_lo || nn > nn_hi) return;   // another launch's tile
    if ((phase == PH_B && !tw.need_pass_b) ||
        ((phase == PH_R || phase == PH_R2) && nn <= 0)) {
        if (threadIdx.x == 0) {
            tw.kb = 0;
            if (phase == PH_R) tw.kround = 0;
            if (phase == PH_R2) tw.need_pass_b = 0;
        }
        return;
    }
    const double *G = ws.S(s);
    const int ld = ws.ldK();
    double *L = ws.L(s);
    int *piv = ws.Piv(s);

    double loc = 0.0;
    for (int i = threadIdx.x; i < nn; i += blockDim.x) {
        dg[i] = G[(size_t)i * ld + i];
        used[i] = 0;
        loc += dg[i];
    }
    const double trace = block_sum(loc, redd);
    MaxLoc mx{-DBL_MAX, 1 << 30};
    for (int i = threadIdx.x; i < nn; i += blockDim.x)
        if (dg[i] > mx.v) mx = MaxLoc{dg[i], i};
    const double dmax = block_argmax(mx, red).v;

    double thr;
    int cap = nn;
    double stop_trace = -1.0;   // PH_H: stop once the remaining trace is below
    if (phase == PH_A) {
        const double tol_floor = 0.01 * tol * tol * trace / nn;
        const double noise = 1e-15 * dmax;
        thr = fmax(noise, tol_floor);
        if (threadIdx.x == 0) {
            tw.tr_g = trace;
            tw.need_pass_b = noise > tol_floor && trace > 0.0;
        }
    } else if (phase == PH_B) {
        thr = fmax(1e-15 * dmax, 0.01 * tol * tol * tw.tr_g / tw.k);
        cap = tw.k - tw.k1;
    } else if (phase == PH_R || phase == PH_R2) {
        // residual columns r_i = (I - Q Q^T) D w_i have E||r_i||^2 =
        // ||(I - Q Q^T) D||_F^2: keep directions above (tol/10)^2 ||D||_F^2.
        // When the squared-noise floor of this Gram hides part of that
        // range, the same sample is projected and searched once more.
        // (E||r_i||^2 carries the variance of Omega's entries: 1 for the
        // Gaussian, about 32^2 for the int8 sketch matrix)
        const double noise = 1e-15 * dmax;
        const double var = tw.omega_var > 0.0 ? tw.omega_var : 1.0;
        const double floor_ = 0.01 * tol * tol * tw.dnorm2 * var;
        thr = fmax(noise, floor_);
        cap = min(nn, tw.k - tw.k1);
        // a repeat pass only where (tol/10)^2 lies below the squared-noise
        // floor at all (the same decision alone or in any batch)
        if (threadIdx.x == 0)
            tw.need_pass_b = phase == PH_R && noise > floor_ &&
                             0.01 * tol * tol < 1e-15;
    } else {
        thr = 1e-18 * dmax;
        if (threadIdx.x == 0) tw.tr_h = trace;
        // The energy the factor leaves out joins the rank rule's tail
        // (tail_h), so the factor may stop at 1% of the tile's error
        // budget: it, and the Jacobi SVD on it, are then no wider than the
        // tolerance needs (the rank grows by at most the directions that 1%
        // hides).
        const double energy = tw.dnorm2 > 0.0 ? fmax(tw.dnorm2, trace) : trace;
        stop_trace = 0.01 * tol * tol * energy;
        // A block whose energy outside the sketched basis, ||D||^2 -
        // ||B||^2 (less the rounding allowance of k_rank_cut), alone
        // exceeds the budget is stored dense whatever its small SVD says:
        // the rank cut reaches rank -1 from k2 = 0 by the same test, so the
        // factor and the Jacobi SVD are skipped.
        const double dn = tw.dnorm2;
        if (dn > 0.0 &&
            fmax(0.0, dn - trace - 2e-15 * dn) > tol * tol * fmax(dn, trace)) {
            if (threadIdx.x == 0) {
                tw.k2 = 0;
                tw.tail_h = trace;
                tw.status |= TILE_TAIL_LEFT;
            }
            return;
        }
    }
    if (!(dmax > 0.0)) thr = DBL_MAX;   // zero or invalid Gram: rank 0

    int j = 0;
    for (; j < cap; ++j) {
        MaxLoc cand{-DBL_MAX, 1 << 30};
        double rest = 0.0;          // remaining trace, for PH_H's stop
        for (int i = threadIdx.x; i < nn; i += blockDim.x)
            if (!used[i]) {
                if (dg[i] > cand.v) cand = MaxLoc{dg[i], i};
                rest += fmax(0.0, dg[i]);
            }
        MaxLoc best;
        if (stop_trace >= 0.0) {
            double total;
            best = block_argmax_sum(cand, rest, red, redd, &total);
            if (total <= stop_trace) break;
        } else {
            best = block_argmax(cand, red);
        }
        if (!(best.v > thr)) break;
        const int p = best.i;
        const double sp = sqrt(best.v);
        for (int l = threadIdx.x; l < j; l += blockDim.x)
            lp[l] = L[(size_t)l * ld + p];
        __syncthreads();
        if (threadIdx.x == 0) {
            piv[j] = p;
            used[p] = 1;
        }
        if constexpr (LPR == 1) {
        for (int i = threadIdx.x; i < nn; i += blockDim.x) {
            double v;
            if (i == p) {
                v = sp;
            } else if (used[i]) {
                v = 0.0;
            } else {
                // G(p, i) - sum_l L(i, l) L(p, l), in four independent
                // partial sums (the chain over l is the step's latency)
                double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
                int l = 0;
                for (; l + 3 < j; l += 4) {
                    a0 = fma(L[(size_t)l * ld + i], lp[l], a0);
                    a1 = fma(L[(size_t)(l + 1) * ld + i], lp[l + 1], a1);
                    a2 = fma(L[(size_t)(l + 2) * ld + i], lp[l + 2], a2);
                    a3 = fma(L[(size_t)(l + 3) * ld + i], lp[l + 3], a3);
                }
                for (; l < j; ++l) a0 = fma(L[(size_t)l * ld + i], lp[l], a0);
                const double acc = G[(size_t)p * ld + i] - ((a0 + a1) + (a2 + a3));
                v = acc / sp;
                dg[i] -= v * v;
            }
            L[(size_t)j * ld + i] = v;
        }
        } else {
        // lane q of a row's group sums l = q, q + LPR, ... (two chains);
        // the block-uniform row loop keeps every lane in the shuffles
        const int q = threadIdx.x % LPR;
        for (int i0 = 0; i0 < nn; i0 += blockDim.x / LPR) {
            const int i = i0 + threadIdx.x / LPR;
            const bool live = i < nn && i != p && !used[i];
            double a0 = 0.0, a1 = 0.0;
            if (live) {
                int l = q;
                for (; l + LPR < j; l += 2 * LPR) {
                    a0 = fma(L[(size_t)l * ld + i], lp[l], a0);
                    a1 = fma(L[(size_t)(l + LPR) * ld + i], lp[l + LPR], a1);
                }
                for (; l < j; l += LPR) a0 = fma(L[(size_t)l * ld + i], lp[l], a0);
            }
            double part = a0 + a1;
            #pragma unroll
            for (int o = LPR / 2; o > 0; o >>= 1)
                part += __shfl_xor_sync(0xffffffffu, part, o);
            if (i < nn && q == 0) {
                double v;
                if (i == p) {
                    v = sp;
                } else if (used[i]) {
                    v = 0.0;
                } else {
                    v = (G[(size_t)p * ld + i] - part) / sp;
                    dg[i] -= v * v;
                }
                L[(size_t)j * ld + i] = v;
            }
        }
        }
        __syncthreads();
    }
    const int cnt = j;
    if (threadIdx.x == 0) {
        if (phase == PH_A) tw.k1 = cnt;
        else if (phase == PH_B || phase == PH_R || phase == PH_R2) tw.kb = cnt;
        else tw.k2 = cnt;
        if (phase == PH_R) {
            tw.kround = cnt;
            if (cnt == 0) tw.need_pass_b = 0;
        }
    }
    if (phase == PH_H) {
        // energy of B outside the span of the factor's columns
        double rest = 0.0;
        for (int i = threadIdx.x; i < nn; i += blockDim.x)
            if (!used[i]) rest += fmax(0.0, dg[i]);
        rest = block_sum(rest, redd);
        if (threadIdx.x == 0) tw.tail_h = cnt > 0 ? rest : trace;
        return;
    }
    // T = R11^{-1}, R11(a, b) = L(piv[b], a) for a <= b (upper triangular).
    double *T = ws.T(s);
    for (int c = threadIdx.x; c < cnt; c += blockDim.x) {
        double *x = T + (size_t)c * ld;
        for (int a = c + 1; a < cnt; ++a) x[a] = 0.0;
        x[c] = 1.0 / L[(size_t)c * ld + piv[c]];
        for (int a = c - 1; a >= 0; --a) {
            double acc = 0.0;
            for (int b = a + 1; b <= c; ++b) acc += L[(size_t)a * ld + piv[b]] * x[b];
            x[a] = -acc / L[(size_t)a * ld + piv[a]];
        }
    }
}

// acc += sum of N products x[u sx] y[u sy], u ascending, all loads first.
template <int N>
__device__ __forceinline__ void chain_block(double &acc, const double *x, int sx,
                                            const double *y, int sy)
{
    double xv[N], yv[N];
    #pragma unroll
    for (int u = 0; u < N; ++u) {
        xv[u] = x[u * sx];
        yv[u] = y[u * sy];
    }
    #pragma unroll
    for (int u = 0; u < N; ++u) acc = fma(xv[u], yv[u], acc);
}

// a[u mod C] += x[u s] y[u s] for u = 0 .. N - 1, all loads first.
template <int C, int N>
__device__ __forceinline__ void chains_block(double (&a)[C], const double *x,
                                             const double *y, int s)
{
    double xv[N], yv[N];
    #pragma unroll
    for (int u = 0; u < N; ++u) {
        xv[u] = x[u * s];
        yv[u] = y[u * s];
    }
    #pragma unroll
    for (int u = 0; u < N; ++u) a[u % C] = fma(xv[u], yv[u], a[u % C]);
}

// X = R^{-1} for the upper triangular R(a, b) = R[a * ld_r + b] (a < b < cnt,
// diagonal in `diag`), in shared memory, one thread per column; X is stored
// as rows of ldx doubles, zero below the diagonal, and copied to
// T(:, 0:cnt).  A column's back substitution sums b = a + 1 .. c in that
// order, a chain of dependent products; a warp runs its 32 columns in step
// (the zeros change no sum), so the chain's loads go in whole blocks.
// Called by the whole block.
__device__ __forceinline__ void tri_inverse(const double *R, int ld_r,
                                            const double *diag, int cnt,
                                            double *X, int ldx, double *T, int ld)
{
    const int c = threadIdx.x, c_hi = min(cnt - 1, c | 31);
    const int lane = threadIdx.x & 31;
    if ((c & ~31) < cnt) {
        const bool in = c < cnt;
        double x = 0.0;                       // X(a + 1, c)
        for (int a = c_hi; a >= 0; --a) {
            double v = 0.0;
            if (a < c_hi) {
                const double *r = R + a * ld_r + a + 1;
                double acc = fma(*r, x, 0.0);
                const double *xp = X + (a + 2) * ldx + c;
                int n = c_hi - a - 1;
                ++r;
                for (; n >= 16; n -= 16, r += 16, xp += 16 * ldx)
                    chain_block<16>(acc, r, 1, xp, ldx);
                if (n & 8) {
                    chain_block<8>(acc, r, 1, xp, ldx);
                    r += 8;
                    xp += 8 * ldx;
                }
                if (n & 4) {
                    chain_block<4>(acc, r, 1, xp, ldx);
                    r += 4;
                    xp += 4 * ldx;
                }
                if (n & 2) {
                    chain_block<2>(acc, r, 1, xp, ldx);
                    r += 2;
                    xp += 2 * ldx;
                }
                if (n & 1) acc = fma(*r, *xp, acc);
                v = -acc;
            }
            if (a == c) v = 1.0;
            x = a <= c && in ? v / diag[a] : 0.0;
            if (in) X[a * ldx + c] = x;
        }
        if (in)
            for (int a = c_hi + 1; a < cnt; ++a) X[a * ldx + c] = 0.0;
    }
    __syncthreads();
    for (int q = threadIdx.x >> 5; q < cnt; q += blockDim.x >> 5)
        for (int a = lane; a < cnt; a += 32) T[(size_t)q * ld + a] = X[a * ldx + q];
}

// Order-preserving 64-bit key of a double.
__device__ __forceinline__ unsigned long long order_key(double v)
{
    const long long b = __double_as_longlong(v);
    return (unsigned long long)(b < 0 ? ~b : b | (long long)0x8000000000000000ull);
}

__device__ __forceinline__ double key_value(unsigned long long k)
{
    return __longlong_as_double((long long)(k >> 63 ? k & 0x7fffffffffffffffull : ~k));
}

// Block sum of one value per row in the order of block_sum (tree over the
// 32 rows of a warp, tree over the warps): every thread gets it.
template <int W>
__device__ __forceinline__ double row_sum(double x, double *red)
{
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if constexpr (W == 1) return x;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    if constexpr (W == 2) return red[0] + red[1];
    if constexpr (W == 3) return (red[0] + red[2]) + red[1];
    return (red[0] + red[2]) + (red[1] + red[3]);
}

// The same factorisation for at most 32 W rows: the Gram sits in shared
// memory, one thread per row, the diagonal in a register.  Step j's column
// of L takes slot j; the Gram column that was there moves to the slot of
// the pivot's column, which no later step reads (each thread moves its own
// row).  What bounds it is the chain of dependent steps -- pivot search,
// the left-looking product, quotient -- so the search is three integer
// warp reductions on an order-preserving key, the product walks
// consecutive slots (addresses known ahead, so its loads overlap), and a
// step has one block barrier (none for W = 1); the kernel above takes
// about 6 us a step (five barriers, the Gram and L read from L2).
// Every sum keeps the order of the kernel above (four partial sums of the
// left-looking product, trees over 32 rows and over warps), so both give
// the same bits.  Phases R, R2 (nn <= the round's columns) and H (tiles of
// 32 (W - 1) < nn <= 32 W rows: nn_lo, nn_hi).  81 tiles, 64 columns:
// 215 -> 75 us; 81 tiles of up to 128 rows in phase H 286 us in one launch ->
// 125 us for 97 .. 128 rows, with the narrower ranges beside it.
template <int W>
__global__ void __launch_bounds__(32 * W)
k_pivchol_rows(TileWork *__restrict__ tiles, Workspace ws, int phase, int nn_lo,
               int nn_hi, const int *__restrict__ act)
{
    extern __shared__ double pc_sm[];
    __shared__ double redd[4];
    __shared__ unsigned long long redk[2][4];
    __shared__ int redi[2][4];
    __shared__ int spiv[32 * W];
    __shared__ int pos[32 * W], at[32 * W];   // Gram column -> slot, and back
    TileWork &tw = tiles[act ? act[blockIdx.x] : blockIdx.x];
    const int s = tw.slot;
    const double tol = tw.tol;
    int nn;
    if (phase == PH_H) nn = tw.k1;
    else if (phase == PH_R) nn = tw.bcur;
    else nn = tw.need_pass_b ? tw.bcur : 0;
    const int i = threadIdx.x, lane = i & 31, warp = i >> 5;
    if (nn < nn_lo || nn > nn_hi) return;
    if (phase != PH_H && nn <= 0) {
        if (i == 0) {
            tw.kb = 0;
            if (phase == PH_R) tw.kround = 0;
            if (phase == PH_R2) tw.need_pass_b = 0;
        }
        return;
    }
    const double dn = tw.dnorm2, var0 = tw.omega_var;
    const int room = tw.k - tw.k1;
    constexpr int LD = 32 * W + 1;
    const double *G = ws.S(s);
    const int ld = ws.ldK();
    if (i < nn)
        for (int c = 0; c < nn; ++c) {
            const unsigned d = (unsigned)__cvta_generic_to_shared(pc_sm + c * LD + i);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                         :: "r"(d), "l"(G + (size_t)c * ld + i));
        }
    asm volatile("cp.async.commit_group;");
    pos[i] = at[i] = i;
    asm volatile("cp.async.wait_group 0;");
    __syncthreads();
    double dg = i < nn ? pc_sm[i * LD + i] : 0.0;
    bool open = i < nn;                    // not a pivot yet
    const double trace = row_sum<W>(dg, redd);

    // Largest value and its (smallest) row over the open rows, as keys;
    // values not above -DBL_MAX (NaN) never win.
    unsigned long long bk;
    int bi;
    auto search = [&](int par) {
        const bool in = open && dg > -DBL_MAX;
        const unsigned long long k = order_key(in ? dg : -DBL_MAX);
        const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        const unsigned row = in && hi == mh && lo == ml ? (unsigned)i : 1u << 30;
        bi = (int)__reduce_min_sync(0xffffffffu, row);
        bk = ((unsigned long long)mh << 32) | ml;
        if constexpr (W > 1) {
            if (lane == 0) {
                redk[par][warp] = bk;
                redi[par][warp] = bi;
            }
            __syncthreads();
            bk = redk[par][0];
            bi = redi[par][0];
            #pragma unroll
            for (int w = 1; w < W; ++w)
                if (redk[par][w] > bk) {
                    bk = redk[par][w];
                    bi = redi[par][w];
                }
        } else {
            __syncwarp();
        }
    };
    search(1);
    const double dmax = key_value(bk);

    double thr;
    int cap = nn;
    double stop_trace = -1.0;
    if (phase != PH_H) {
        const double noise = 1e-15 * dmax;
        const double var = var0 > 0.0 ? var0 : 1.0;
        const double floor_ = 0.01 * tol * tol * dn * var;
        thr = fmax(noise, floor_);
        cap = min(nn, room);
        if (i == 0)
            tw.need_pass_b = phase == PH_R && noise > floor_ &&
                             0.01 * tol * tol < 1e-15;
    } else {
        thr = 1e-18 * dmax;
        if (i == 0) tw.tr_h = trace;
        const double energy = dn > 0.0 ? fmax(dn, trace) : trace;
        stop_trace = 0.01 * tol * tol * energy;
        if (dn > 0.0 &&
            fmax(0.0, dn - trace - 2e-15 * dn) > tol * tol * fmax(dn, trace)) {
            if (i == 0) {
                tw.k2 = 0;
                tw.tail_h = trace;
                tw.status |= TILE_TAIL_LEFT;
            }
            return;
        }
    }
    if (!(dmax > 0.0)) thr = DBL_MAX;

    int j = 0;
    for (; j < cap; ++j) {
        search(j & 1);
        if (stop_trace >= 0.0) {
            const double total = row_sum<W>(open ? fmax(0.0, dg) : 0.0, redd);
            if (total <= stop_trace) break;
        }
        const double best = key_value(bk);
        if (!(best > thr)) break;
        const int p = bi;
        const double sp = sqrt(best);
        const int q = pos[p];
        double *colq = pc_sm + q * LD + i, *colj = pc_sm + j * LD + i;
        double v = 0.0, gq = 0.0;
        if (i < nn) {
            gq = *colq;                // the pivot's Gram column, this row
            *colq = *colj;             // slot j's column moves there
        }
        if (i == p) {
            v = sp;
            open = false;
            spiv[j] = p;
        } else if (open) {
            // blocks of sixteen, eight and four products, four chains; the
            // one to three left over join the first chain
            double a[4] = {};
            const double *li = pc_sm + i, *lp = pc_sm + p;
            int n = j;
            for (; n >= 16; n -= 16, li += 16 * LD, lp += 16 * LD)
                chains_block<4, 16>(a, li, lp, LD);
            if (n & 8) {
                chains_block<4, 8>(a, li, lp, LD);
                li += 8 * LD;
                lp += 8 * LD;
            }
            if (n & 4) {
                chains_block<4, 4>(a, li, lp, LD);
                li += 4 * LD;
                lp += 4 * LD;
            }
            if (n & 2) {
                chain_block<2>(a[0], li, LD, lp, LD);
                li += 2 * LD;
                lp += 2 * LD;
            }
            if (n & 1) a[0] = fma(*li, *lp, a[0]);
            v = (gq - ((a[0] + a[1]) + (a[2] + a[3]))) / sp;
            dg -= v * v;
        }
        if (i < nn) *colj = v;
        // pos and at of the moved column: every thread has read pos[p]
        // before the barrier of the next search; the entries written here
        // are read after it
        if constexpr (W == 1) __syncwarp();
        if (i == 0) {
            const int r = at[j];
            pos[r] = q;
            at[q] = r;
        }
        if constexpr (W == 1) __syncwarp();
    }
    const int cnt = j;
    __syncthreads();
    if (i == 0) {
        if (phase == PH_H) tw.k2 = cnt;
        else tw.kb = cnt;
        if (phase == PH_R) {
            tw.kround = cnt;
            if (cnt == 0) tw.need_pass_b = 0;
        }
    }
    if (phase == PH_H) {
        const double rest = row_sum<W>(open ? fmax(0.0, dg) : 0.0, redd);
        if (i == 0) tw.tail_h = cnt > 0 ? rest : trace;
        double *L = ws.L(s);
        if (i < nn)
            for (int c = 0; c < cnt; ++c) L[(size_t)c * ld + i] = pc_sm[c * LD + i];
        return;
    }
    int *piv = ws.Piv(s);
    __shared__ double diag[32 * W];
    const int mine = i < cnt ? spiv[i] : 0;
    if (i < cnt) {
        piv[i] = mine;
        diag[i] = pc_sm[i * LD + mine];
    }
    // rows in pivot order: slot a then holds R11(a, b) = L(piv[b], a)
    for (int a0 = 0; a0 < cnt; a0 += 8) {
        double v[8];
        #pragma unroll
        for (int u = 0; u < 8; ++u)
            v[u] = a0 + u < cnt ? pc_sm[(a0 + u) * LD + mine] : 0.0;
        __syncthreads();
        #pragma unroll
        for (int u = 0; u < 8; ++u)
            if (a0 + u < cnt && i < cnt) pc_sm[(a0 + u) * LD + i] = v[u];
    }
    __syncthreads();
    // T = R11^{-1} (upper triangular)
    tri_inverse(pc_sm, LD, diag, cnt, pc_sm + nn_hi * LD, LD, ws.T(s), ld);
}

template <int W>
static void pivchol_rows_launch(TileWork *d_tiles, int ntiles, Workspace ws,
                                int phase, int nn_lo, int nn_hi,
                                cudaStream_t stream, const int *act)
{
    // (the rounds, with two matrices, are launched for at most 64 rows)
    constexpr size_t most = (size_t)(W <= 2 ? 2 : 1) * (32 * W) * (32 * W + 1) * sizeof(double);
    const size_t smem = (size_t)(phase == PH_H ? 1 : 2) * nn_hi * (32 * W + 1) *
                        sizeof(double);
    allow_smem<k_pivchol_rows<W>, most>();
    k_pivchol_rows<W><<<ntiles, 32 * W, smem, stream>>>(d_tiles, ws, phase, nn_lo,
                                                        nn_hi, act);
}

// Phase H for factors above kPivcholSplit rows: a cluster of CTAs shares the
// rows in chunks of 32 (chunk w in CTA w mod CS), each CTA holding its rows
// of the Gram, and then of L, in its own shared memory.  A step exchanges
// the warps' pivot candidates and remaining-trace sums through distributed
// shared memory (one cluster barrier), reads the pivot's row of L from the
// CTA that owns it, and updates its rows.  Sums keep the order of
// k_pivchol<4> (eight partial sums of the product by l mod 8, lanes' trees
// over chunks), so both give the same bits; that kernel reads L from L2 in
// one CTA: about 9 us a step at 150 .. 270 rows, 1.5 ms and more for a
// launch with a few such tiles.
constexpr int kClusterRows = 128;     // most rows of one CTA of the cluster
constexpr int kClusterMaxChunks = 16;

template <int CS>
__host__ __device__ constexpr int pivchol_cluster_warps(int nn)
{
    return ((nn + 31) / 32 + CS - 1) / CS;
}

template <int CS>
__global__ void __launch_bounds__(kClusterRows)
k_pivchol_cluster(TileWork *__restrict__ tiles, Workspace ws, int nn_lo, int nn_hi,
                  const int *__restrict__ act)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ double pk_sm[];          // [slot][own rows]
    __shared__ unsigned long long ck[2][kClusterMaxChunks];
    __shared__ int ci[2][kClusterMaxChunks];
    __shared__ double cs[2][kClusterMaxChunks];
    __shared__ int pos[32 * kClusterMaxChunks], at[32 * kClusterMaxChunks];
    __shared__ __align__(16) double lp[32 * kClusterMaxChunks + 16];
    const int rank = (int)cl.block_rank();
    TileWork &tw = tiles[act ? act[blockIdx.x / CS] : blockIdx.x / CS];
    const int s = tw.slot, nn = tw.k1;
    if (nn < nn_lo || nn > nn_hi) return;       // cluster-uniform
    const double tol = tw.tol, dn = tw.dnorm2;
    const int nchunk = (nn + 31) / 32;
    const int nw = pivchol_cluster_warps<CS>(nn), rl = 32 * nw;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int chunk = warp * CS + rank;         // this warp's rows
    const int i = chunk * 32 + lane;
    const bool mine = warp < nw && i < nn;
    const double *G = ws.S(s);
    const int ld = ws.ldK();
    if (mine)
        for (int c = 0; c < nn; ++c) {
            const unsigned d = (unsigned)__cvta_generic_to_shared(pk_sm + c * rl + t);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;"
                         :: "r"(d), "l"(G + (size_t)c * ld + i));
        }
    asm volatile("cp.async.commit_group;");
    for (int q = t; q < 32 * kClusterMaxChunks; q += kClusterRows) pos[q] = at[q] = q;
    for (int q = t; q < 2 * kClusterMaxChunks; q += kClusterRows) {
        ck[q / kClusterMaxChunks][q % kClusterMaxChunks] = 0;
        ci[q / kClusterMaxChunks][q % kClusterMaxChunks] = 1 << 30;
        cs[q / kClusterMaxChunks][q % kClusterMaxChunks] = 0.0;
    }
    asm volatile("cp.async.wait_group 0;");
    cl.sync();
    double dg = mine ? pk_sm[i * rl + t] : 0.0;
    bool open = mine;
    // The chunks' best candidates and sums to every CTA, then the overall
    // best (largest value, then smallest row) and the sum in block_sum's
    // order (tree over the chunks).
    // (two sets of slots in turn: a set is written again only after the
    // barrier of the exchange between, which every reader has passed)
    unsigned long long bk;
    int bi, par = 1;
    double total;
    auto exchange = [&](double x) {
        par ^= 1;
        const bool in = open && dg > -DBL_MAX;
        const unsigned long long k = order_key(in ? dg : -DBL_MAX);
        const unsigned hi = (unsigned)(k >> 32), lo = (unsigned)k;
        const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
        const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
        const unsigned row = in && hi == mh && lo == ml ? (unsigned)i : 1u << 30;
        const int wi = (int)__reduce_min_sync(0xffffffffu, row);
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (warp < nw && chunk < nchunk && lane < CS) {
            *cl.map_shared_rank(&ck[par][chunk], lane) =
                ((unsigned long long)mh << 32) | ml;
            *cl.map_shared_rank(&ci[par][chunk], lane) = wi;
            *cl.map_shared_rank(&cs[par][chunk], lane) = x;
        }
        cl.sync();
        const int w = lane & (kClusterMaxChunks - 1);
        const unsigned long long kk = ck[par][w];
        const unsigned kh = (unsigned)(kk >> 32), kl = (unsigned)kk;
        const unsigned gh = __reduce_max_sync(0xffffffffu, kh);
        const unsigned gl = __reduce_max_sync(0xffffffffu, kh == gh ? kl : 0u);
        bi = (int)__reduce_min_sync(0xffffffffu,
                                    kh == gh && kl == gl ? (unsigned)ci[par][w] : 1u << 30);
        bk = ((unsigned long long)gh << 32) | gl;
        total = lane < kClusterMaxChunks ? cs[par][w] : 0.0;
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
    };
    exchange(dg);
    const double trace = total;
    const double dmax = key_value(bk);
    double thr = 1e-18 * dmax;
    const bool lead = rank == 0 && t == 0;
    if (lead) tw.tr_h = trace;
    const double energy = dn > 0.0 ? fmax(dn, trace) : trace;
    const double stop_trace = 0.01 * tol * tol * energy;
    if (dn > 0.0 &&
        fmax(0.0, dn - trace - 2e-15 * dn) > tol * tol * fmax(dn, trace)) {
        if (lead) {
            tw.k2 = 0;
            tw.tail_h = trace;
            tw.status |= TILE_TAIL_LEFT;
        }
        return;
    }
    if (!(dmax > 0.0)) thr = DBL_MAX;
    int j = 0;
    for (; j < nn; ++j) {
        exchange(open ? fmax(0.0, dg) : 0.0);
        if (total <= stop_trace) break;
        const double best = key_value(bk);
        if (!(best > thr)) break;
        const int p = bi;
        const double sp = sqrt(best);
        // row p of L from its CTA (chunk p / 32 is warp (p / 32) / CS of CTA
        // (p / 32) mod CS there)
        {
            const double *src = cl.map_shared_rank(pk_sm, (p >> 5) % CS) +
                                ((p >> 5) / CS * 32 + (p & 31));
            for (int l = t; l < j + 16; l += kClusterRows)
                lp[l] = l < j ? src[(size_t)l * rl] : 0.0;
        }
        const int q = pos[p], r = at[j];
        double gq = 0.0;
        if (mine) {
            gq = pk_sm[q * rl + t];
            pk_sm[q * rl + t] = pk_sm[j * rl + t];
        }
        __syncthreads();
        double v = 0.0;
        if (mine) {
            if (i == p) {
                v = sp;
                open = false;
            } else if (open) {
                // lane q of the replaced kernel summed l = q, q + 8, ... and
                // l = q + 4, q + 12, ...
                double a[8] = {};
                const double *li = pk_sm + t;
                const double2 *l2 = reinterpret_cast<const double2 *>(lp);
                int l = 0;
                for (; l + 15 < j; l += 16) {
                    double x[16];
                    double2 y[8];
                    #pragma unroll
                    for (int u = 0; u < 16; ++u) x[u] = li[(l + u) * rl];
                    #pragma unroll
                    for (int u = 0; u < 8; ++u) y[u] = l2[l / 2 + u];
                    #pragma unroll
                    for (int u = 0; u < 16; ++u)
                        a[u & 7] = fma(x[u], u & 1 ? y[u / 2].y : y[u / 2].x, a[u & 7]);
                }
                {
                    // up to fifteen more (lp is zero past j)
                    double x[16];
                    #pragma unroll
                    for (int u = 0; u < 16; ++u)
                        x[u] = l + u < j ? li[(l + u) * rl] : 0.0;
                    #pragma unroll
                    for (int u = 0; u < 15; ++u) a[u & 7] = fma(x[u], lp[l + u], a[u & 7]);
                }
                const double p0 = a[0] + a[4], p1 = a[1] + a[5];
                const double p2 = a[2] + a[6], p3 = a[3] + a[7];
                v = (gq - ((p0 + p2) + (p1 + p3))) / sp;
                dg -= v * v;
            }
            pk_sm[j * rl + t] = v;
        }
        // the moved column's place (every thread has read pos and at)
        if (t == 0) {
            pos[r] = q;
            at[q] = r;
        }
    }
    const int cnt = j;
    if (lead) {
        tw.k2 = cnt;
        if (cnt == 0) tw.tail_h = trace;
    }
    exchange(open ? fmax(0.0, dg) : 0.0);
    if (lead && cnt > 0) tw.tail_h = total;
    double *L = ws.L(s);
    if (mine)
        for (int c = 0; c < cnt; ++c) L[(size_t)c * ld + i] = pk_sm[c * rl + t];
    cl.sync();     // no CTA leaves while another may still read its rows
}

// Most rows k_pivchol_cluster<CS> takes: a CTA's share of the Gram within
// its shared memory.
constexpr size_t kClusterSmemMax = 208 * 1024;

template <int CS>
static int pivchol_cluster_fit(int kmax)
{
    int nn = std::min(kmax, 32 * kClusterMaxChunks);
    while (nn > 0 && (pivchol_cluster_warps<CS>(nn) * 32 > kClusterRows ||
                      (size_t)nn * 32 * pivchol_cluster_warps<CS>(nn) * sizeof(double) >
                          kClusterSmemMax))
        --nn;
    return nn;
}

template <int CS>
static void pivchol_cluster_launch(TileWork *d_tiles, int ntiles, Workspace ws,
                                   int nn_lo, int nn_hi, cudaStream_t stream,
                                   const int *act)
{
    size_t smem = 0;
    for (int nn = nn_lo; nn <= nn_hi; ++nn)
        smem = std::max(smem, (size_t)nn * 32 * pivchol_cluster_warps<CS>(nn) * sizeof(double));
    auto *fn = k_pivchol_cluster<CS>;
    allow_smem<k_pivchol_cluster<CS>, kClusterSmemMax>();
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ntiles * CS));
    cfg.blockDim = dim3(kClusterRows);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, fn, d_tiles, ws, nn_lo, nn_hi, act);
}

// Phase H above kPivcholSplit rows, `count` tiles (of `act`, or the first
// ones of the batch).  A few tiles: clusters of four as far as their shared
// memory reaches (277 rows), of eight from there (to 416); a cluster keeps
// its SMs to itself, so with more tiles than about two rounds of clusters the
// one-CTA kernel, two tiles to an SM, has more throughput.  The whole small
// SVD with one CTA a tile over that with clusters, random points, nearly all
// tiles in one range:
//   rows      16    36    64    81   100   144   225   324 tiles
//   138     1.06  1.06  1.05  1.05  1.05  1.31  1.01  0.99
//   181     1.06  1.06  1.06  1.01  0.99  0.95  0.92  0.88
//   232     1.12  1.09  1.05  0.97  0.94  0.95  0.93  0.92
//   291     1.10  1.18  0.89  0.92     -  0.85     -     -   (eight)
//   300     1.12  1.29  1.23  1.39     -  1.03     -     -   (eight)
//   362     0.98  0.96  0.94  0.93  0.96  0.91  0.91  0.93   (eight)
// (the last beside tiles of 509 rows, the longest chains, which no cluster
// holds; four tiles of 390 rows beside twelve of 291, the longest there: 15.7
// -> 12.9 ms).  Returns the number of launches.
constexpr int kPivcholClusterTiles = 74;

static int pivchol_large_launch(TileWork *d_tiles, int count, Workspace ws,
                                cudaStream_t stream, const int *act)
{
    const int kmax = ws.k_max;
    int lo = kPivcholSplit + 1, launches = 0;
    if (count <= kPivcholClusterTiles) {
        const int fit4 = pivchol_cluster_fit<4>(kmax), fit8 = pivchol_cluster_fit<8>(kmax);
        if (fit4 >= lo) {
            pivchol_cluster_launch<4>(d_tiles, count, ws, lo, fit4, stream, act);
            lo = fit4 + 1;
            ++launches;
        }
        if (kmax >= lo && fit8 >= lo) {
            pivchol_cluster_launch<8>(d_tiles, count, ws, lo, fit8, stream, act);
            lo = fit8 + 1;
            ++launches;
        }
    }
    if (kmax >= lo) {
        k_pivchol<kPivcholLanes><<<count, kSmallThreads * kPivcholLanes, 0, stream>>>(
            d_tiles, ws, PH_H, lo, INT_MAX, act);
        ++launches;
    }
    return launches;
}

// A round's pivoted Cholesky; `bmax` bounds the round's columns.
void launch_round_pivchol(TileWork *d_tiles, int ntiles, Workspace ws,
                          int repeat, int bmax, cudaStream_t stream,
                          const int *act)
{
    const int phase = repeat ? PH_R2 : PH_R;
    if (bmax <= 32)
        pivchol_rows_launch<1>(d_tiles, ntiles, ws, phase, INT_MIN, 32, stream, act);
    else if (bmax <= 64)
        pivchol_rows_launch<2>(d_tiles, ntiles, ws, phase, INT_MIN, 64, stream, act);
    else
        k_pivchol<1><<<ntiles, kSmallThreads, 0, stream>>>(d_tiles, ws, phase, 0,
                                                           INT_MAX, act);
}

// ||D||_F^2 of every block from the generator's per-CTA partial sums, in a
// fixed order.
__global__ void k_block_norms(TileWork *__restrict__ tiles, Workspace ws)
{
    TileWork &tw = tiles[blockIdx.x];
    const int gx = (tw.m + 63) / 64, gy = (tw.n + 63) / 64;
    const int ldn = (ws.n_max + 63) / 64;
    __shared__ double red[8];
    double a = 0.0;
    for (int q = threadIdx.x; q < gx * gy; q += blockDim.x)
        a += ws.Nrm(tw.slot)[(q / gy) * ldn + q % gy];
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_down_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = a;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
        tw.dnorm2 = s;
    }
}

void launch_block_norms(const TileWork *, TileWork *d_rw, int ntiles,
                        Workspace ws, cudaStream_t stream)
{
    k_block_norms<<<ntiles, 256, 0, stream>>>(d_rw, ws);
}

// Start of a sampling round: tiles not done sample min(block, k - cols)
// more columns; counts[0] counts them and act lists them, in any order.
// counts[1 + b] and the lists after act[0 .. ld - 1] collect the tiles by
// basis size (svd_bin), for the small SVD when no tile samples any more.
__global__ void k_round_setup(TileWork *__restrict__ tiles, int ntiles,
                              int block, int *counts, int *act, int ld)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    TileWork &tw = tiles[t];
    const int b = svd_bin(tw.k1);
    act[(size_t)(1 + b) * ld + atomicAdd(counts + 1 + b, 1)] = t;
    if (tw.done || tw.cols_done >= tw.k) {
        tw.bcur = 0;
        tw.done = 1;
        return;
    }
    tw.bcur = min(block, tw.k - tw.cols_done);
    tw.k1_round = tw.k1;
    tw.trunc_round = 0;
    act[atomicAdd(counts, 1)] = t;
}

void launch_round_setup(TileWork *d_tiles, int ntiles, int block,
                        int *d_counts, int *d_act, int ld, cudaStream_t stream)
{
    cudaMemsetAsync(d_counts, 0, (1 + kSvdBins) * sizeof(int), stream);
    k_round_setup<<<(ntiles + 127) / 128, 128, 0, stream>>>(d_tiles, ntiles, block,
                                                            d_counts, d_act, ld);
}

// End of a round: the new orthonormal columns join the basis.  The tile is
// finished when the round's sample left at least `verify` columns whose
// residuals against the grown basis all fell below the threshold (so the
// residual estimate rests on that many independent Gaussian samples), when
// it found no direction at all, or when the k columns are exhausted.
__global__ void k_round_end(TileWork *__restrict__ tiles, int ntiles,
                            int verify)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    TileWork &tw = tiles[t];
    if (tw.bcur <= 0) return;
    tw.cols_done += tw.bcur;
    const int added = tw.k1 + tw.kb - tw.k1_round;
    if (tw.kround == 0 || tw.cols_done >= tw.k ||
        (tw.bcur - added >= verify && !tw.trunc_round))
        tw.done = 1;
    tw.k1 += tw.kb;       // (kb is 0 here: each pass merged its columns)
    tw.kb = 0;
    tw.bcur = 0;
}

void launch_round_end(TileWork *d_tiles, int ntiles, int verify,
                      cudaStream_t stream)
{
    k_round_end<<<(ntiles + 127) / 128, 128, 0, stream>>>(d_tiles, ntiles,
                                                          verify);
}

void launch_pivchol(int phase, TileWork *d_tiles, int ntiles, Workspace ws,
                    cudaStream_t s)
{
    k_pivchol<1><<<ntiles, kSmallThreads, 0, s>>>(d_tiles, ws, phase, 0, INT_MAX,
                                                  nullptr);
}

// Gathers the pivot columns of Y into the Q buffer (phase A) or the Q1
// buffer (phase B).
__global__ void k_gather_cols(const TileWork *__restrict__ tiles,
                              Workspace ws, int phase)
{
    const TileWork tw = tiles[blockIdx.x];
    const int s = tw.slot;
    const int cnt = phase == PH_A ? tw.k1 : tw.kb;
    if (cnt <= 0) return;
    const int *piv = ws.Piv(s);
    const double *Y = ws.Y(s);
    double *dst = phase == PH_A ? ws.Q(s) : ws.Q1(s);
    const int ld = ws.ldM();
    for (int c = blockIdx.y; c < cnt; c += gridDim.y) {
        const double *src = Y + (size_t)piv[c] * ld;
        for (int i = threadIdx.x; i < tw.m; i += blockDim.x)
            dst[(size_t)c * ld + i] = src[i];
    }
}

void launch_gather_cols(int phase, const TileWork *d_tiles, int ntiles,
                        Workspace ws, cudaStream_t stream)
{
    dim3 grid(ntiles, 16);
    k_gather_cols<<<grid, 256, 0, stream>>>(d_tiles, ws, phase);
}

// Cholesky G = R^T R of the re-orthogonalisation Gram in S(slot)
// (dimension k1 for phase A, kb for phase B), R into L(slot), then
// T(slot) = R^{-1}.  For phase B the new columns are appended to the basis
// afterwards by the caller's merge step.
__global__ void __launch_bounds__(kSmallThreads)
k_chol_inv(TileWork *__restrict__ tiles, Workspace ws, int phase, int nn_lo,
           const int *__restrict__ act)
{
    TileWork &tw = tiles[act ? act[blockIdx.x] : blockIdx.x];
    const int s = tw.slot;
    const int nn = phase == PH_A ? tw.k1 : tw.kb;
    if (nn < nn_lo) return;
    const double *G = ws.S(s);
    double *R = ws.L(s);
    double *T = ws.T(s);
    const int ld = ws.ldK();
    __shared__ double diag;
    __shared__ int stop;
    if (threadIdx.x == 0) stop = 0;
    __syncthreads();
    int nn_ok = nn;
    for (int j = 0; j < nn; ++j) {
        if (threadIdx.x == 0) {
            const double gjj = G[(size_t)j * ld + j];
            double acc = gjj;
            for (int l = 0; l < j; ++l) {
                const double r = R[(size_t)j * ld + l];
                acc -= r * r;
            }
            // a column numerically inside the span of the previous ones:
            // the factor keeps the columns before it (they come in
            // decreasing pivot order) and the round may not finish the
            // tile on its verification columns
            if (!(acc > 1e-14 * gjj)) stop = 1;
            diag = sqrt(fmax(acc, 0.0));
            R[(size_t)j * ld + j] = diag;
        }
        __syncthreads();
        if (stop) { nn_ok = j; break; }
        const double rjj = diag;
        for (int c = j + 1 + threadIdx.x; c < nn; c += blockDim.x) {
            double acc = G[(size_t)c * ld + j];
            for (int l = 0; l < j; ++l)
                acc -= R[(size_t)j * ld + l] * R[(size_t)c * ld + l];
            R[(size_t)c * ld + j] = acc / rjj;
        }
        __syncthreads();
    }
    for (int c = threadIdx.x; c < nn_ok; c += blockDim.x) {
        double *x = T + (size_t)c * ld;
        for (int a = c + 1; a < nn_ok; ++a) x[a] = 0.0;
        x[c] = 1.0 / R[(size_t)c * ld + c];
        for (int a = c - 1; a >= 0; --a) {
            double acc = 0.0;
            for (int b = a + 1; b <= c; ++b) acc += R[(size_t)b * ld + a] * x[b];
            x[a] = -acc / R[(size_t)a * ld + a];
        }
    }
    if (threadIdx.x == 0 && nn_ok < nn) {
        if (phase == PH_A) tw.k1 = nn_ok;
        else tw.kb = nn_ok;
        tw.trunc_round = 1;
        tw.status |= TILE_CHOL_TRUNC;
    }
}

// The same for nn <= N, right-looking: thread (c, q) keeps the rows q, q +
// 4, ... of column c in registers, so a step is one square root, one
// quotient and one product per entry instead of a chain of l of them; every
// entry still subtracts its products in the order l = 0, 1, ..., so both
// kernels give the same bits.  Rows of the trailing matrix that are done,
// and entries below the diagonal, are updated along with the others and
// never read.
constexpr int kCholSmall = 64;

template <int N>
__global__ void __launch_bounds__(4 * N)
k_chol_inv_small(TileWork *__restrict__ tiles, Workspace ws, int phase,
                 const int *__restrict__ act)
{
    constexpr int LD = N + 1, E = N / 4;
    __shared__ double next[N], gd[N], diag[N];
    extern __shared__ double ci_sm[];
    TileWork &tw = tiles[act ? act[blockIdx.x] : blockIdx.x];
    const int s = tw.slot;
    const int nn = phase == PH_A ? tw.k1 : tw.kb;
    if (nn <= 0 || nn > N) return;
    double *R = ci_sm, *X = ci_sm + N * LD;     // R by rows
    const double *G = ws.S(s);
    const int ld = ws.ldK();
    const int c = threadIdx.x % N, q = threadIdx.x / N;
    double a[E];
    #pragma unroll
    for (int u = 0; u < E; ++u) {
        const int row = q + 4 * u;
        a[u] = row <= c && c < nn ? G[(size_t)c * ld + row] : 0.0;
        if (row == c) gd[c] = a[u];
    }
    for (int e = threadIdx.x; e < N * LD; e += 4 * N) R[e] = 0.0;
    if (q == 0) next[c] = a[0];
    __syncthreads();
    int nn_ok = nn;
    for (int l = 0; l < nn; ++l) {
        const double acc = next[l];
        // a column numerically inside the span of the previous ones ends
        // the factor (as above); the test is the same for every thread
        if (!(acc > 1e-14 * gd[l])) { nn_ok = l; break; }
        const double r = sqrt(fmax(acc, 0.0));
        // each of a column's four threads forms its R(l, c), one stores it
        const double rc = c > l && c < nn ? next[c] / r : 0.0;
        if (q == 0) R[l * LD + c] = rc;
        if (threadIdx.x == 0) diag[l] = r;
        __syncthreads();
        #pragma unroll
        for (int u = 0; u < E; ++u)
            if (4 * u + 3 > l) {                 // uniform
                const int j = q + 4 * u;
                a[u] -= R[l * LD + j] * rc;
                if (j == l + 1) next[c] = a[u];
            }
        __syncthreads();
    }
    tri_inverse(R, LD, diag, nn_ok, X, LD, ws.T(s), ld);
    if (threadIdx.x == 0 && nn_ok < nn) {
        if (phase == PH_A) tw.k1 = nn_ok;
        else tw.kb = nn_ok;
        tw.trunc_round = 1;
        tw.status |= TILE_CHOL_TRUNC;
    }
}

template <int N>
static void chol_small_launch(int phase, TileWork *d_tiles, int ntiles,
                              Workspace ws, cudaStream_t stream, const int *act)
{
    constexpr size_t smem = (size_t)2 * N * (N + 1) * sizeof(double);
    allow_smem<k_chol_inv_small<N>, smem>();
    k_chol_inv_small<N><<<ntiles, 4 * N, smem, stream>>>(d_tiles, ws, phase, act);
}

// `nmax` bounds the columns of every tile.
void launch_chol_inv(int phase, TileWork *d_tiles, int ntiles, Workspace ws,
                     int nmax, cudaStream_t stream, const int *act)
{
    if (nmax <= 32)
        chol_small_launch<32>(phase, d_tiles, ntiles, ws, stream, act);
    else
        chol_small_launch<kCholSmall>(phase, d_tiles, ntiles, ws, stream, act);
    if (nmax > kCholSmall)
        k_chol_inv<<<ntiles, kSmallThreads, 0, stream>>>(d_tiles, ws, phase,
                                                         kCholSmall + 1, act);
}

// -------------------------------------------------- one-sided Jacobi

// One-sided Jacobi (Hestenes) on the columns of A = L(slot) (k1 x k2):
// column pairs are rotated until mutually orthogonal; then the columns of
// A V are the eigenvectors of L L^T scaled by the singular values.  L comes
// from a pivoted Cholesky of B B^T (the transpose of a column-pivoted QR
// factor of B^T), the preconditioning under which one-sided Jacobi needs
// few sweeps (Z. Drmac, K. Veselic, SIAM J. Matrix Anal. Appl. 29 (2008)).
// Pairs follow the round-robin tournament ordering: k2/2 disjoint pairs per
// step, all rotated at once, a block barrier between steps.
//
// The cost is the chain of dependent steps (k2 - 1 per sweep), each issue
// bound on its SM for large tiles, so a pair is rotated by a group of G
// lanes holding E rows each in registers (G E >= k1): the group sizes its
// dot-product reduction to the column length, and a warp rotates 32 / G
// pairs at once, sharing the instructions of the rotation angle among
// them.  The kernel is instantiated per size
// class; tiles of one class share a launch, every other tile's CTA returns
// at once.  Columns live in shared memory when they fit, otherwise in
// global memory (L2-resident for the tiles of one launch).  W (normalised
// columns) goes to T(slot), squared norms to Sig(slot).
constexpr size_t kJacobiSmemMax = 220 * 1024;

// Size classes, by rows (k1), with G E just above the row count so that few
// lanes rotate padding; factors in shared memory when they fit, else the
// block kernel (k_jacobi_block).  The last class streams rows through
// registers for k1 > 512.
__host__ __device__ inline int jacobi_class(int rows, int cols)
{
    const size_t bytes = (size_t)(rows | 1) * cols * sizeof(double);
    const bool fits = bytes <= kJacobiSmemMax;
    if (rows <= 32) return 0;                     // G 4,  E 8,  64 threads
    if (rows <= 64) return 1;                     // G 4,  E 16, 128 threads
    if (rows <= 128) return 2;                    // G 8,  E 16, 512 threads
    if (rows <= 192) return fits ? 3 : 4;         // G 16, E 12, 512 threads
    if (rows <= 256) return fits ? 5 : 6;         // G 16, E 16, 512 threads
    if (rows <= 288) return 7;                    // G 16, E 18, blocks
    if (rows <= 320) return 8;                    // G 16, E 20, blocks
    if (rows <= 512) return 9;                    // G 32, E 16, blocks
    return 10;                                    // streamed, global
}

// Most columns a factor of the class can have (columns <= rows).
__host__ __device__ constexpr int jacobi_class_cols(int cls)
{
    return cls == 0 ? 32 : cls == 1 ? 64 : cls == 2 ? 128 : cls <= 4 ? 192
         : cls <= 6 ? 256 : cls == 7 ? 288 : cls == 8 ? 320 : cls == 9 ? 512
         : kMaxK;
}

// Convergence bookkeeping shared by the Jacobi kernels.  Every column
// pair is checked once per sweep at a fixed step of the schedule (T steps
// per sweep); lastrot[c] is the step at which column c was last rotated.
// A pair whose previous check (T steps ago) found it orthogonal and whose
// columns have not been rotated since is orthogonal still: it is skipped,
// so late sweeps, and the final sweep that confirms convergence, only
// look at the pairs that changed.  A sweep that rotates nothing ends the
// iteration exactly as when every pair is checked.
__device__ __forceinline__ bool jacobi_unchanged(const int *lastrot, int a,
                                                 int b, int since)
{
    return lastrot[a] < since && lastrot[b] < since;
}

// Where a lane keeps its E rows (gl + G q, q < E) of a column in shared
// memory.  PAIRED: rows q and q + 1 (q even) side by side, so that a lane
// moves two rows per 16-byte access and the column is padded with zero rows
// to G E (zeros change no sum); else row i at i, rows past `rows` skipped.
template <int G, bool PAIRED>
__device__ __forceinline__ int jacobi_at(int i)
{
    if constexpr (!PAIRED) return i;
    const int q = i / G;
    return (q >> 1) * 2 * G + (i - q * G) * 2 + (q & 1);
}

template <int G, int E, bool PAIRED>
__device__ __forceinline__ void jacobi_load(double (&x)[E], const double *col,
                                            int rows, int gl, bool valid)
{
    if constexpr (PAIRED) {
        static_assert(E % 2 == 0, "row pairs");
        const double2 *p = reinterpret_cast<const double2 *>(col) + gl;
        #pragma unroll
        for (int q = 0; q < E; q += 2) {
            const double2 v = valid ? p[q / 2 * G] : make_double2(0.0, 0.0);
            x[q] = v.x;
            x[q + 1] = v.y;
        }
    } else {
        #pragma unroll
        for (int q = 0; q < E; ++q) {
            const int i = gl + G * q;
            x[q] = valid && i < rows ? col[i] : 0.0;
        }
    }
}

template <int G, int E, bool PAIRED>
__device__ __forceinline__ void jacobi_store(const double (&x)[E], double *col,
                                             int rows, int gl)
{
    if constexpr (PAIRED) {
        double2 *p = reinterpret_cast<double2 *>(col) + gl;
        #pragma unroll
        for (int q = 0; q < E; q += 2) p[q / 2 * G] = make_double2(x[q], x[q + 1]);
    } else {
        #pragma unroll
        for (int q = 0; q < E; ++q) {
            const int i = gl + G * q;
            if (i < rows) col[i] = x[q];
        }
    }
}

// Rotation of a column pair whose rows are spread over the G lanes of one
// group, E per lane.  Every lane of the warp calls this (inactive groups
// with zero columns) because the reductions shuffle across the whole warp.
// Returns true if the pair was rotated.
template <int G, int E>
__device__ __forceinline__ bool jacobi_rotate(double (&xa)[E], double (&xb)[E],
                                              double eps2)
{
    double al = 0.0, be = 0.0, ga = 0.0;
    #pragma unroll
    for (int q = 0; q < E; ++q) {
        al = fma(xa[q], xa[q], al);
        be = fma(xb[q], xb[q], be);
        ga = fma(xa[q], xb[q], ga);
    }
    #pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        al += __shfl_xor_sync(0xffffffffu, al, o);
        be += __shfl_xor_sync(0xffffffffu, be, o);
        ga += __shfl_xor_sync(0xffffffffu, ga, o);
    }
    // |gamma| > eps sqrt(alpha beta), compared in squares
    if (!(ga * ga > eps2 * al * be) || !(al > 0.0) || !(be > 0.0))
        return false;
    // t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)), zeta = (beta - alpha) /
    // (2 gamma), rewritten with one division: t = sign(d) g / (|d| + h),
    // d = beta - alpha, g = 2 gamma, h = sqrt(d^2 + g^2).
    const double d = be - al, g = 2.0 * ga;
    const double h = sqrt(fma(d, d, g * g));
    const double t = (d >= 0.0 ? g : -g) / (fabs(d) + h);
    const double c = rsqrt(fma(t, t, 1.0));
    const double sn = c * t;
    #pragma unroll
    for (int q = 0; q < E; ++q) {
        const double a = xa[q], b = xb[q];
        xa[q] = c * a - sn * b;
        xb[q] = sn * a + c * b;
    }
    return true;
}

// The same for long columns: rows streamed in chunks of 32 per lane (one
// warp per pair), loaded twice (dot products, then rotation).
__device__ bool jacobi_rotate_stream(double *ca, double *cb, int rows,
                                     int lane, bool valid, double eps2)
{
    double al = 0.0, be = 0.0, ga = 0.0;
    if (valid) {
        for (int i = lane; i < rows; i += 32) {
            const double x = ca[i], y = cb[i];
            al = fma(x, x, al);
            be = fma(y, y, be);
            ga = fma(x, y, ga);
        }
    }
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        al += __shfl_xor_sync(0xffffffffu, al, o);
        be += __shfl_xor_sync(0xffffffffu, be, o);
        ga += __shfl_xor_sync(0xffffffffu, ga, o);
    }
    if (!(ga * ga > eps2 * al * be) || !(al > 0.0) || !(be > 0.0))
        return false;
    const double d = be - al, g = 2.0 * ga;
    const double h = sqrt(fma(d, d, g * g));
    const double t = (d >= 0.0 ? g : -g) / (fabs(d) + h);
    const double c = rsqrt(fma(t, t, 1.0));
    const double sn = c * t;
    for (int i = lane; i < rows; i += 32) {
        const double x = ca[i], y = cb[i];
        ca[i] = c * x - sn * y;
        cb[i] = sn * x + c * y;
    }
    return true;
}

// Doubles between the columns of the shared-memory kernel: padded to whole
// row pairs of the G lanes (PAIRED), and for G = 4, whose eight-lane access
// phases take two neighbouring columns, an odd multiple of 8 so that the
// two use different banks; else the row count, odd.
template <int G, int E, bool PAIRED>
__host__ __device__ constexpr int jacobi_stride(int rows)
{
    return !PAIRED ? (rows | 1) : G == 4 ? (E * G / 8 | 1) * 8 : E * G;
}

// The factor in shared memory (SMEM) or streamed from global memory (E = 0).
// The launch takes the tiles with rows_lo <= k1 <= rows_hi <= G E (of the
// classes 3 and 5 those that fit).  Shared-memory traffic and the FP64
// pipe bound a step, and with one CTA per SM its latency: the row pairs
// halve the accesses, the padding removes their bank conflicts (columns an
// odd number of doubles apart shared banks between the groups of a warp),
// E close to the row count leaves few lanes on padding, and the narrower
// ranges fit two CTAs on an SM.
template <int CLASS, int G, int E, int THREADS, int MINB, bool PAIRED>
__global__ void __launch_bounds__(THREADS, MINB)
k_jacobi(TileWork *__restrict__ tiles, Workspace ws, int rows_lo, int rows_hi,
         const int *__restrict__ act)
{
    constexpr bool SMEM = E > 0;
    constexpr int EE = SMEM ? E : 1;
    extern __shared__ double2 jac_sm[];
    double *sm = reinterpret_cast<double *>(jac_sm);
    __shared__ int rotated[2];
    __shared__ int lastrot[jacobi_class_cols(CLASS)];
    TileWork &tw = tiles[act ? act[blockIdx.x] : blockIdx.x];
    const int s = tw.slot;
    const int rows = tw.k1, cols = tw.k2;
    if (cols <= 0 || rows < rows_lo || rows > rows_hi ||
        jacobi_class(rows, cols) != CLASS) return;   // uniform
    for (int c = threadIdx.x; c < cols; c += THREADS) lastrot[c] = -1;
    // Relative orthogonality the rotations stop at: the rank cut needs the
    // left singular vectors orthonormal to well below tol (their overlap
    // enters the tail energies squared and the projector linearly): 1 % of
    // tol, at most 1e-7.
    const double eps = fmax(1e-15, fmin(1e-7, 0.01 * tw.tol));
    const double eps2 = eps * eps;
    const int ldg = ws.ldK();
    double *A = SMEM ? sm : ws.L(s);
    const int lda = SMEM ? jacobi_stride<G, EE, PAIRED>(rows) : ldg;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = THREADS / 32;
    if (SMEM) {
        const double *Lg = ws.L(s);
        const int fill = PAIRED ? G * EE : rows;
        for (int c = warp; c < cols; c += kWarps)
            for (int i = lane; i < fill; i += 32)
                A[(size_t)c * lda + jacobi_at<G, PAIRED>(i)] =
                    i < rows ? Lg[(size_t)c * ldg + i] : 0.0;
    }
    if (threadIdx.x == 0) rotated[0] = rotated[1] = 0;
    __syncthreads();
    constexpr int kGroupsPerWarp = 32 / G;
    const int gw = lane / G, gl = lane % G;
    const int nc = cols + (cols & 1);      // players, with a bye if odd
    const int npairs = nc / 2;
    const int T = nc - 1;                  // steps per sweep
    int sweep = 0;
    for (; sweep < 40; ++sweep) {
        bool any = false;
        for (int step = 0; step < nc - 1; ++step) {
            const int now = sweep * T + step;
            for (int base = warp * kGroupsPerWarp; base < npairs;
                 base += kWarps * kGroupsPerWarp) {
                const int p = base + gw;
                int a = 0, b = 0;
                if (p < npairs) {
                    // a = 1 + (p - 1 + step) mod (nc - 1) for p > 0,
                    // b = 1 + (nc - 2 - p + step) mod (nc - 1); both
                    // arguments lie in [0, 2 (nc - 1))
                    int x = p - 1 + step, y = nc - 2 - p + step;
                    if (x >= nc - 1) x -= nc - 1;
                    if (y >= nc - 1) y -= nc - 1;
                    a = p == 0 ? 0 : 1 + x;
                    b = 1 + y;
                }
                const bool valid = p < npairs && a < cols && b < cols &&
                                   !jacobi_unchanged(lastrot, a, b, now - T);
                if (!__any_sync(0xffffffffu, valid)) continue;   // warp-uniform
                double *ca = A + (size_t)a * lda, *cb = A + (size_t)b * lda;
                bool rot;
                if constexpr (SMEM) {
                    double xa[EE], xb[EE];
                    jacobi_load<G, EE, PAIRED>(xa, ca, rows, gl, valid);
                    jacobi_load<G, EE, PAIRED>(xb, cb, rows, gl, valid);
                    rot = jacobi_rotate<G, EE>(xa, xb, eps2);
                    if (rot) {
                        jacobi_store<G, EE, PAIRED>(xa, ca, rows, gl);
                        jacobi_store<G, EE, PAIRED>(xb, cb, rows, gl);
                    }
                } else {
                    rot = jacobi_rotate_stream(ca, cb, rows, lane, valid, eps2);
                }
                if (rot && gl == 0) lastrot[a] = lastrot[b] = now;
                any |= rot;
            }
            __syncthreads();
        }
        // double-buffered flag: cleared one sweep ahead, read after a barrier
        if (any) rotated[sweep & 1] = 1;
        if (threadIdx.x == 0) rotated[(sweep + 1) & 1] = 0;
        __syncthreads();
        if (!rotated[sweep & 1]) break;
    }
    // Normalise into W = T(slot); squared norms into Sig.
    double *W = ws.T(s);
    double *sig = ws.Sig(s);
    for (int c = warp; c < cols; c += kWarps) {
        const double *ca = A + (size_t)c * lda;
        double nrm = 0.0;
        for (int i = lane; i < rows; i += 32) {
            const double x = ca[jacobi_at<G, PAIRED>(i)];
            nrm = fma(x, x, nrm);
        }
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
        const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
        for (int i = lane; i < rows; i += 32)
            W[(size_t)c * ldg + i] = ca[jacobi_at<G, PAIRED>(i)] * inv;
        if (lane == 0) sig[c] = nrm;
    }
    if (threadIdx.x == 0) {
        tw.sweeps = sweep;
        if (sweep >= 40) tw.status |= TILE_JACOBI_SLOW;
    }
}

// Block one-sided Jacobi for the classes whose factor does not fit in
// shared memory (k1 <= 512).  The k2 columns form blocks of B = 512 / G;
// the blocks meet in a round-robin tournament, and each meeting brings the
// block pair (2B columns, 164 KB at most) into shared memory, rotates the
// B^2 column pairs across the two blocks there (B steps of B disjoint
// pairs, one group of G lanes per pair, E rows per lane) and writes it
// back; the pairs inside each block are rotated in the tournament's first
// round.  A sweep (one tournament) thus rotates every pair once, as the
// cyclic order does, but every rotation reads shared memory instead of L2
// and global traffic is a few copies of the factor per sweep.  Sweeps
// repeat until one rotates nothing.
//
// The meetings of one round touch disjoint blocks, so a tile is taken by a
// cluster of CTAs (jacobi_cluster) that share each round's meetings and meet
// at a cluster barrier between rounds (which also publishes the round's
// columns in global memory): a tile's latency, which is what bounds the
// batches that hold few such tiles, drops by up to that factor.  Times
// (for the convergence bookkeeping) count the steps of a round once,
// whichever CTA runs a meeting: round 0 takes steps [0, 2B - 1) (B - 1
// within blocks, B across), round r > 0 the B steps from B - 1 + r B; a
// column is only rotated by the one meeting of a round that holds it.
// lastrot lives in the slot's Sig buffer during the iteration (the
// normalisation overwrites it at the end), each meeting works on its own
// copy of its columns' entries.  Data another CTA of the cluster wrote is
// read past L1 (__ldcg).
constexpr int kJacobiClusterMax = 8;

// CTAs per tile.  With few tiles the chain of one tile is what the launch
// takes: one CTA for each meeting of a round (blocks of 512 / G columns, at
// most k1 of them).  With more tiles, meetings queue on the SMs anyway and a
// CTA per meeting only adds idle ones: 2, or 4 for the classes above 256 rows.
// The whole small SVD with 2 or 4 over that with a CTA per meeting (as above):
//   rows      16    36    64    81   121   144   169   225   324 tiles
//   181     1.28  1.27  1.28  1.26  1.16  1.05  1.36  1.12  0.94
//   232     1.54  1.40  1.13  1.34  1.05  1.21  1.06  1.03  0.94
//   276     1.35  1.32  1.11  1.09  0.99  1.00  0.98  0.91  0.81
//   362     1.25  1.27  1.11  0.99  0.95  0.91  0.89  0.82  0.82
// so the line lies at the SM count, and above 320 rows, where a CTA per meeting
// is a cluster of eight (blocks of 16 columns: up to 16 meetings) and not of
// three to five, at half of it (100 tiles of 362 rows: 0.94).  Without the tile
// count (no list) the batch's widest factor decides, as measured: 4 where kmax
// > 256, else 2.
// STARSH_B200_JACOBI_CLUSTER (1 .. 8) sets one size for all.
static int jacobi_cluster(int cls, int kmax, int count, bool known)
{
    static const int forced = [] {
        int v = 0;
        if (const char *e = getenv("STARSH_B200_JACOBI_CLUSTER"))
            v = std::max(1, std::min(kJacobiClusterMax, atoi(e)));
        return v;
    }();
    if (forced) return forced;
    if (known && count <= (cls == 9 ? 74 : 148)) {
        const int b = cls == 9 ? 16 : 32;
        const int nb = (std::min(kmax, jacobi_class_cols(cls)) + b - 1) / b;
        return std::max(2, std::min(kJacobiClusterMax, (nb + 1) / 2));
    }
    return cls >= 7 || (!known && kmax > 256) ? 4 : 2;
}

template <int CLASS, int G, int E>
__global__ void __launch_bounds__(512, 1)
k_jacobi_block(TileWork *__restrict__ tiles, Workspace ws,
               const int *__restrict__ act)
{
    constexpr int THREADS = 512;
    constexpr int B = THREADS / G;          // columns per block, pairs per step
    constexpr int P2 = 2 * B;               // columns in shared memory
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const int crank = (int)cl.block_rank(), csize = (int)cl.num_blocks();
    extern __shared__ double sm[];
    __shared__ int rotated[2];              // in the cluster's first CTA
    __shared__ int lr[P2];                  // lastrot of the meeting's slots
    TileWork &tw = tiles[act ? act[blockIdx.x / csize] : blockIdx.x / csize];
    const int s = tw.slot;
    const int rows = tw.k1, cols = tw.k2;
    if (cols <= 0 || jacobi_class(rows, cols) != CLASS) return;   // cluster-uniform
    const double eps = fmax(1e-15, fmin(1e-7, 0.01 * tw.tol));
    const double eps2 = eps * eps;
    const int ldg = ws.ldK();
    double *Lg = ws.L(s);
    int *lastrot = (int *)ws.Sig(s);
    int *rot0 = cl.map_shared_rank(rotated, 0);
    const int lds = rows | 1;
    const int nb = (cols + B - 1) / B;
    const int nbp = nb + (nb & 1);          // blocks, with a bye if odd
    const int gw = threadIdx.x / G, gl = threadIdx.x % G;
    for (int c = crank * THREADS + threadIdx.x; c < cols; c += csize * THREADS)
        lastrot[c] = -1;
    if (crank == 0 && threadIdx.x == 0) rotated[0] = rotated[1] = 0;
    cl.sync();
    auto column = [&](int q, int bi, int bj) {   // global column of slot q
        return q < B ? bi * B + q : bj * B + q - B;
    };
    const int T = (B - 1) + (nbp - 1) * B;      // steps per sweep
    int sweep = 0;
    for (; sweep < 40; ++sweep) {
        bool any = false;
        for (int rnd = 0; rnd < nbp - 1; ++rnd) {
            const int t0 = sweep * T + (rnd == 0 ? 0 : B - 1 + rnd * B);
            for (int pr = crank; pr < nbp / 2; pr += csize) {
                // block pair pr of round rnd (circle method, as for columns)
                int x = pr - 1 + rnd, y = nbp - 2 - pr + rnd;
                if (x >= nbp - 1) x -= nbp - 1;
                if (y >= nbp - 1) y -= nbp - 1;
                const int bi = pr == 0 ? 0 : 1 + x, bj = 1 + y;
                // Each block's own pairs are rotated once per sweep, in the
                // first round (where every block meets exactly one other,
                // or the bye); every meeting rotates the B^2 pairs across
                // its two blocks.
                const bool bye = bi >= nb || bj >= nb;
                if (bye && rnd > 0) continue;                   // uniform
                const int b0 = bye ? (bi < nb ? bi : bj) : bi;  // slots 0 .. B-1
                const int b1 = bye ? nb : bj;                   // slots B .. 2B-1
                const int nslots = bye ? B : P2;
                // A meeting none of whose columns has been rotated since
                // its previous occurrence (T steps ago, when all its pairs
                // were found orthogonal) is skipped with its copies.
                int hot = 0;
                for (int q = threadIdx.x; q < P2; q += THREADS) {
                    const int c = q < nslots ? column(q, b0, b1) : cols;
                    lr[q] = c < cols ? __ldcg(lastrot + c) : -1;
                    if (c < cols && lr[q] >= t0 - T) hot = 1;
                }
                if (!__syncthreads_or(hot)) continue;
                for (int e = threadIdx.x; e < nslots * rows; e += THREADS) {
                    const int q = e / rows, i = e - q * rows;
                    const int c = column(q, b0, b1);
                    sm[(size_t)q * lds + i] = c < cols ? __ldcg(Lg + (size_t)c * ldg + i) : 0.0;
                }
                __syncthreads();
                int now = t0;
                if (rnd == 0) {
                    // round-robin over the B columns of each block, B / 2
                    // pairs per block and step (groups B / 2 .. B - 1 take
                    // block b1, idle at the bye)
                    const int q = gw % (B / 2), off = gw < B / 2 ? 0 : B;
                    for (int step = 0; step < B - 1; ++step, ++now) {
                        int u = q - 1 + step, v = B - 2 - q + step;
                        if (u >= B - 1) u -= B - 1;
                        if (v >= B - 1) v -= B - 1;
                        const int a = off + (q == 0 ? 0 : 1 + u), b = off + 1 + v;
                        const bool valid = (off == 0 || !bye) &&
                                           column(a, b0, b1) < cols &&
                                           column(b, b0, b1) < cols &&
                                           !jacobi_unchanged(lr, a, b, now - T);
                        if (__any_sync(0xffffffffu, valid)) {
                            double *ca = sm + (size_t)a * lds, *cb = sm + (size_t)b * lds;
                            double xa[E], xb[E];
                            jacobi_load<G, E, false>(xa, ca, rows, gl, valid);
                            jacobi_load<G, E, false>(xb, cb, rows, gl, valid);
                            const bool rot = jacobi_rotate<G, E>(xa, xb, eps2);
                            if (rot) {
                                jacobi_store<G, E, false>(xa, ca, rows, gl);
                                jacobi_store<G, E, false>(xb, cb, rows, gl);
                                if (gl == 0) lr[a] = lr[b] = now;
                            }
                            any |= rot;
                        }
                        __syncthreads();
                    }
                }
                if (!bye) {
                    // the cross pairs: slot gw with slot B + (gw + step) mod
                    // B.  A group's own column a stays in its registers for
                    // the B steps (no other group touches it).
                    const int a = gw;
                    const bool in_a = column(a, b0, b1) < cols;
                    double *ca = sm + (size_t)a * lds;
                    double xa[E];
                    bool moved = false;
                    jacobi_load<G, E, false>(xa, ca, rows, gl, in_a);
                    for (int step = 0; step < B; ++step, ++now) {
                        const int b = B + (gw + step) % B;
                        const bool valid = in_a && column(b, b0, b1) < cols &&
                                           !jacobi_unchanged(lr, a, b, now - T);
                        if (__any_sync(0xffffffffu, valid)) {
                            double *cb = sm + (size_t)b * lds;
                            double xb[E];
                            // an inactive group's zero column b is never
                            // rotated
                            jacobi_load<G, E, false>(xb, cb, rows, gl, valid);
                            const bool rot = jacobi_rotate<G, E>(xa, xb, eps2);
                            if (rot) {
                                jacobi_store<G, E, false>(xb, cb, rows, gl);
                                if (gl == 0) lr[a] = lr[b] = now;
                                moved = true;
                            }
                            any |= rot;
                        }
                        __syncthreads();
                    }
                    if (moved) {
                        jacobi_store<G, E, false>(xa, ca, rows, gl);
                    }
                    __syncthreads();
                }
                for (int e = threadIdx.x; e < nslots * rows; e += THREADS) {
                    const int q = e / rows, i = e - q * rows;
                    const int c = column(q, b0, b1);
                    if (c < cols) Lg[(size_t)c * ldg + i] = sm[(size_t)q * lds + i];
                }
                for (int q = threadIdx.x; q < nslots; q += THREADS) {
                    const int c = column(q, b0, b1);
                    if (c < cols) lastrot[c] = lr[q];
                }
                __syncthreads();
            }
            // the round's columns and times, visible to the whole cluster
            cl.sync();
        }
        if (any) rot0[sweep & 1] = 1;
        if (crank == 0 && threadIdx.x == 0) rotated[(sweep + 1) & 1] = 0;
        cl.sync();
        if (!rot0[sweep & 1]) break;
    }
    // every CTA has read the first CTA's flag before any of them exits
    cl.sync();
    // Normalise into W = T(slot); squared norms into Sig (over lastrot).
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *W = ws.T(s);
    double *sig = ws.Sig(s);
    for (int c = crank * (THREADS / 32) + warp; c < cols;
         c += csize * (THREADS / 32)) {
        const double *ca = Lg + (size_t)c * ldg;
        double nrm = 0.0;
        for (int i = lane; i < rows; i += 32) {
            const double x = __ldcg(ca + i);
            nrm = fma(x, x, nrm);
        }
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
        const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
        for (int i = lane; i < rows; i += 32) W[(size_t)c * ldg + i] = __ldcg(ca + i) * inv;
        if (lane == 0) sig[c] = nrm;
    }
    if (crank == 0 && threadIdx.x == 0) {
        tw.sweeps = sweep;
        if (sweep >= 40) tw.status |= TILE_JACOBI_SLOW;
    }
}

template <int CLASS, int G, int E>
static void jacobi_block_launch(TileWork *d_tiles, int ntiles, Workspace ws,
                                int max_rows, cudaStream_t stream, const int *act)
{
    const int kmax = ws.k_max;
    auto *fn = k_jacobi_block<CLASS, G, E>;
    const size_t smem = (size_t)2 * (512 / G) * (max_rows | 1) * sizeof(double);
    // (max_rows: at most the class's, and so its columns)
    constexpr size_t most =
        (size_t)2 * (512 / G) * (jacobi_class_cols(CLASS) | 1) * sizeof(double);
    allow_smem<k_jacobi_block<CLASS, G, E>, most>();
    cudaLaunchConfig_t cfg = {};
    const int cs = jacobi_cluster(CLASS, kmax, ntiles, act != nullptr);
    cfg.gridDim = dim3((unsigned)(ntiles * cs));
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, fn, d_tiles, ws, act);
}

// Tiles with rows_lo <= k1 <= rows_hi of the class (k1 <= kmax, the batch's
// widest factor; k2 <= k1).
template <int CLASS, int G, int E, int THREADS, int MINB, bool PAIRED>
static void jacobi_rows_launch(TileWork *d_tiles, int ntiles, Workspace ws,
                               int rows_lo, int rows_hi, cudaStream_t stream,
                               const int *act)
{
    auto *fn = k_jacobi<CLASS, G, E, THREADS, MINB, PAIRED>;
    size_t smem = 0;
    if constexpr (E > 0) {
        const int r = std::min(rows_hi, ws.k_max);
        smem = (size_t)jacobi_stride<G, E, PAIRED>(r) * r * sizeof(double);
        if (!PAIRED) smem = std::min(smem, kJacobiSmemMax);
        // (rows_hi <= G E)
        constexpr size_t full =
            (size_t)jacobi_stride<G, E, PAIRED>(G * E) * (G * E) * sizeof(double);
        constexpr size_t most = !PAIRED && full > kJacobiSmemMax ? kJacobiSmemMax : full;
        allow_smem<k_jacobi<CLASS, G, E, THREADS, MINB, PAIRED>, most>();
    }
    fn<<<ntiles, THREADS, smem, stream>>>(d_tiles, ws, rows_lo, rows_hi, act);
}

__host__ __device__ int svd_bin(int rows)
{
    int b = 0;
    while (b + 1 < kSvdBins && rows > svd_bin_hi(b)) ++b;
    return b;
}

// Phase H of the pivoted Cholesky and the Jacobi SVD on its factor, by
// ranges of rows (svd_bin) on their own streams: the ranges are independent
// chains of a few long launches that seldom fill the GPU one by one (81
// tiles: 1.40 ms of Jacobi one after another, the longest of them 0.84).
// `count` (host) and `list` (device, kSvdBins lists of `list_ld` tiles) tell
// the tiles of each range, so that only they are launched; null: every
// range is launched over the whole batch, each CTA taking its tile or
// leaving it.  Without lanes everything runs on `stream`.
int launch_small_svd(TileWork *d_tiles, int ntiles, Workspace ws,
                     cudaStream_t stream, const SvdLanes &lanes,
                     const int *count, const int *list, int list_ld)
{
    const int kmax = ws.k_max;
    int launches = 0;
    const bool fork = lanes.fork != nullptr && kmax > 64;
    if (fork) cudaEventRecord(lanes.fork, stream);
    bool used[SvdLanes::kStreams] = {};
    // stream q of the lanes, waiting for the fork at its first use
    auto lane = [&](int q) {
        if (!fork) return stream;
        if (!used[q]) {
            cudaStreamWaitEvent(lanes.s[q], lanes.fork, 0);
            used[q] = true;
        }
        return lanes.s[q];
    };
    // the tiles of bin b: how many, and their list (null: the whole batch)
    auto num = [&](int b) {
        return svd_bin_lo(b) > kmax ? 0 : count ? count[b] : ntiles;
    };
    auto act = [&](int b) { return count ? list + (size_t)b * list_ld : nullptr; };
    // Above 128 rows first: the longest chains.  Their Gram factors run in
    // one launch per range, or one for the batch; the Jacobi SVDs of every
    // range follow on streams of their own: the block classes (factor in
    // global memory), and beside them the classes whose factor fits in
    // shared memory.
    for (int b = kSvdBinLarge; b < kSvdBins; ++b) {
        const int n = num(b);
        if (n == 0) continue;
        const int rows = std::min(kmax, svd_bin_hi(b));
        const cudaStream_t s = lane(count ? b - kSvdBinLarge : 0);
        if (count || b == kSvdBinLarge)
            launches += pivchol_large_launch(d_tiles, n, ws, s, act(b));
        switch (b) {
        case kSvdBinLarge:          // 129 .. 160
        case kSvdBinLarge + 1: {    // 161 .. 192
            const cudaStream_t m = count ? s : lane(SvdLanes::kStreams - 1);
            if (fork && !count && b == kSvdBinLarge) {
                cudaEventRecord(lanes.large, s);
                cudaStreamWaitEvent(m, lanes.large, 0);
            }
            if (b == kSvdBinLarge) {
                jacobi_rows_launch<3, 16, 10, 512, 1, false>(d_tiles, n, ws, 129, 160, m, act(b));
            } else {
                jacobi_rows_launch<3, 16, 12, 512, 1, false>(d_tiles, n, ws, 161, 192, m, act(b));
                jacobi_block_launch<4, 16, 12>(d_tiles, n, ws, rows, s, act(b));
                ++launches;
            }
            break;
        }
        case kSvdBinLarge + 2:      // 193 .. 256
            jacobi_block_launch<6, 16, 16>(d_tiles, n, ws, rows, s, act(b));
            jacobi_rows_launch<5, 16, 16, 512, 1, false>(
                d_tiles, n, ws, 193, 256, count ? s : lane(SvdLanes::kStreams - 1), act(b));
            ++launches;
            break;
        case kSvdBinLarge + 3:      // 257 .. 288
            jacobi_block_launch<7, 16, 18>(d_tiles, n, ws, rows, s, act(b));
            break;
        case kSvdBinLarge + 4:      // 289 .. 320
            jacobi_block_launch<8, 16, 20>(d_tiles, n, ws, rows, s, act(b));
            break;
        case kSvdBinLarge + 5:      // 321 .. 512
            jacobi_block_launch<9, 32, 16>(d_tiles, n, ws, rows, s, act(b));
            break;
        default:                    // above 512
            jacobi_rows_launch<10, 32, 0, 1024, 1, false>(d_tiles, n, ws, 513, kMaxK, s, act(b));
        }
        ++launches;
    }
    // 65 .. 128 rows: two ranges of the Gram factor, four of the Jacobi
    constexpr int kLane2 = SvdLanes::kMid, kLane1 = kLane2 + 1;
    if (num(kBin128)) {
        const cudaStream_t s = lane(kLane2);
        pivchol_rows_launch<4>(d_tiles, num(kBin128), ws, PH_H, 113, 128, s, act(kBin128));
        jacobi_rows_launch<2, 8, 16, 512, 1, true>(d_tiles, num(kBin128), ws, 113, 128, s, act(kBin128));
        launches += 2;
    }
    if (num(kBin112)) {
        const cudaStream_t s = lane(kLane2 + 2);
        pivchol_rows_launch<4>(d_tiles, num(kBin112), ws, PH_H, 97, 112, s, act(kBin112));
        jacobi_rows_launch<2, 8, 14, 448, 1, true>(d_tiles, num(kBin112), ws, 97, 112, s, act(kBin112));
        launches += 2;
    }
    if (num(kBin96)) {
        const cudaStream_t s = lane(kLane1);
        pivchol_rows_launch<3>(d_tiles, num(kBin96), ws, PH_H, 81, 96, s, act(kBin96));
        jacobi_rows_launch<2, 8, 12, 384, 2, true>(d_tiles, num(kBin96), ws, 81, 96, s, act(kBin96));
        launches += 2;
    }
    if (num(kBin80)) {
        const cudaStream_t s = lane(kLane1 + 2);
        pivchol_rows_launch<3>(d_tiles, num(kBin80), ws, PH_H, 65, 80, s, act(kBin80));
        jacobi_rows_launch<2, 8, 10, 320, 2, true>(d_tiles, num(kBin80), ws, 65, 80, s, act(kBin80));
        launches += 2;
    }
    if (num(kBin64)) {
        pivchol_rows_launch<2>(d_tiles, num(kBin64), ws, PH_H, 49, 64, stream, act(kBin64));
        jacobi_rows_launch<1, 4, 16, 128, 4, true>(d_tiles, num(kBin64), ws, 49, 64, stream, act(kBin64));
        launches += 2;
    }
    if (num(kBin48)) {
        pivchol_rows_launch<2>(d_tiles, num(kBin48), ws, PH_H, 33, 48, stream, act(kBin48));
        jacobi_rows_launch<1, 4, 12, 96, 5, true>(d_tiles, num(kBin48), ws, 33, 48, stream, act(kBin48));
        launches += 2;
    }
    if (num(kBin32)) {
        pivchol_rows_launch<1>(d_tiles, num(kBin32), ws, PH_H, INT_MIN, 32, stream, act(kBin32));
        jacobi_rows_launch<0, 4, 8, 64, 8, true>(d_tiles, num(kBin32), ws, 1, 32, stream, act(kBin32));
        launches += 2;
    }
    for (int q = 0; q < SvdLanes::kStreams; ++q)
        if (used[q]) {
            cudaEventRecord(lanes.done[q], lanes.s[q]);
            cudaStreamWaitEvent(stream, lanes.done[q], 0);
        }
    return launches;
}

// Appends the residual-pass columns to the basis: k1 += kb.
__global__ void k_merge_basis(TileWork *__restrict__ tiles, int ntiles)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < ntiles && tiles[t].kb > 0) {
        tiles[t].k1 += tiles[t].kb;
        tiles[t].kb = 0;
    }
}

void launch_merge_basis(TileWork *d_tiles, int ntiles, cudaStream_t stream)
{
    k_merge_basis<<<(ntiles + 127) / 128, 128, 0, stream>>>(d_tiles, ntiles);
}

// --------------------------------------------------------- rank cut

// Energies e_c = ||C(c, :)||^2 of the rotated rows, order by decreasing
// energy, then the smallest r >= 1 with
//   sum_{c >= r} e_c + tail_h + outside  <=  tol^2 ||D||_F^2,
// i.e. starsh_dense_dsvfr applied to the exact energies plus the energy the
// Gram factor (tail_h) and the sketch (outside) left out (0 if D = 0).
// rank = r if r <= maxrank, else -1.
// A row's energy is the sum of 32 strided partial sums (columns l, l + 32,
// ... each, then a tree over l); warp l takes the partial sums l of 32 rows
// at a time, so that its loads run along C's columns (a warp per row read a
// 32-byte sector for every 8 bytes: 81 tiles 60 us).
constexpr int kRankThreads = 1024;

__global__ void __launch_bounds__(kRankThreads)
k_rank_cut(TileWork *__restrict__ tiles, Workspace ws)
{
    TileWork &tw = tiles[blockIdx.x];
    const int s = tw.slot;
    const int k2 = tw.k2;
    const double tol = tw.tol;
    const int maxrank = tw.maxrank;
    __shared__ double e[kMaxK];
    __shared__ int ord[kMaxK];
    __shared__ double part[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double *C = ws.C(s);
    const int ld = ws.ldK();
    for (int c0 = 0; c0 < k2; c0 += 32) {
        const int c = c0 + lane;
        double acc = 0.0;
        if (c < k2) {
            const double *p = C + (size_t)warp * ld + c;
            int j = warp;
            for (; j + 96 < tw.n; j += 128, p += (size_t)128 * ld) {
                double v[4];
                #pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = p[(size_t)32 * u * ld];
                #pragma unroll
                for (int u = 0; u < 4; ++u) acc += v[u] * v[u];
            }
            for (; j < tw.n; j += 32, p += (size_t)32 * ld) acc += *p * *p;
        }
        part[warp][lane] = acc;
        __syncthreads();
        // warp w: row c0 + w, lane l its partial sum l
        double x = part[lane][warp];
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0 && c0 + warp < k2) e[c0 + warp] = x;
        __syncthreads();
    }
    // Position of c = number of entries ranked before it.
    for (int c = threadIdx.x; c < k2; c += blockDim.x) {
        int pos = 0;
        const double ec = e[c];
        for (int o = 0; o < k2; ++o)
            pos += (e[o] > ec) || (e[o] == ec && o < c);
        ord[pos] = c;
    }
    __syncthreads();
    int *gord = ws.Ord(s);
    double *ge = ws.E(s);
    for (int c = threadIdx.x; c < k2; c += blockDim.x) {
        gord[c] = ord[c];
        ge[c] = e[ord[c]];
    }
    if (threadIdx.x == 0) {
        // With the block's exact ||D||_F^2 (dnorm2, from the generator) the
        // energy outside the sketched basis, ||D||^2 - ||B||^2, is known
        // too: it joins the tail, less an allowance for the rounding of the
        // two sums, and the budget is tol^2 ||D||^2.  A block whose
        // outside energy alone exceeds the budget cannot meet tol with its
        // sketch: it is stored dense (rank -1), like a block above maxrank.
        // Without dnorm2 (dense tiles given by the caller) the rule is the
        // reference's: the tail of the projected block's spectrum against
        // tol^2 ||B||^2.
        const double dn = tw.dnorm2;
        const double outside = dn > 0.0
            ? fmax(0.0, dn - tw.tr_h - 2e-15 * dn) : 0.0;
        const double energy = dn > 0.0 ? fmax(dn, tw.tr_h) : tw.tr_h;
        int r;
        if (!(energy > 0.0) || k2 == 0) {
            r = outside <= tol * tol * energy ? 0 : -1;
        } else {
            const double budget = tol * tol * energy;
            // energy outside span(W): what the Gram factor left out
            const double missing = fmax(0.0, tw.tail_h) + outside;
            // tail(r) for r = k2 down to 1; keep the smallest r that fits
            double tail = missing;
            r = -1;
            if (tail <= budget) r = k2;
            for (int c = k2 - 1; c >= 1; --c) {
                tail += e[ord[c]];
                if (tail <= budget) r = c;
                else break;
            }
            if (r < 0) tw.status |= TILE_TAIL_LEFT;
        }
        tw.rank = r <= maxrank ? r : -1;
    }
}

void launch_rank_cut(TileWork *d_tiles, int ntiles, Workspace ws,
                     cudaStream_t stream)
{
    k_rank_cut<<<ntiles, kRankThreads, 0, stream>>>(d_tiles, ws);
}

// V(j, c) = C(ord[c], j): V is n x rank, leading dimension n.  A CTA
// transposes `cols` columns j of C at a time through shared memory: it reads
// their k2 rows (contiguous in C; every lane busy whatever k2) and writes
// the rank selected rows as consecutive entries of each column of V, so both
// sides are coalesced.  As many columns a pass as its shared memory holds
// (a multiple of 8), so that a pass has some 4000 loads in flight: with a
// warp per column and 32 columns a pass the N = 102400 square exponential
// spent 2.6 ms here for 1.2 GB.
constexpr int kWriteVDoubles = 5376;    // 42 KB

__global__ void __launch_bounds__(256)
k_write_v(const TileWork *__restrict__ tiles, Workspace ws, OutArena out,
          int doubles)
{
    extern __shared__ double wv_sm[];   // [cols][k2 | 1]
    const TileWork tw = tiles[blockIdx.x];
    if (tw.rank <= 0) return;
    const int s = tw.slot, ld = ws.ldK();
    const int *ord = ws.Ord(s);
    const double *C = ws.C(s);
    double *V = out.V + tw.off_v;
    const int kr = tw.k2, ls = kr | 1;   // rows of C; ord[c] < k2
    const int cols = max(8, min(256, doubles / ls / 8 * 8));
    const int t = threadIdx.x;
    for (int j0 = blockIdx.y * cols; j0 < tw.n; j0 += gridDim.y * cols) {
        const int nj = min(cols, tw.n - j0);
        const double *Cj = C + (size_t)j0 * ld;
        #pragma unroll 8
        for (int q = t; q < nj * kr; q += 256) {
            const int jj = q / kr, i = q - jj * kr;
            wv_sm[jj * ls + i] = Cj[(size_t)jj * ld + i];
        }
        __syncthreads();
        for (int q = t; q < nj * tw.rank; q += 256) {
            const int c = q / nj, jj = q - c * nj;
            V[(size_t)c * tw.n + j0 + jj] = wv_sm[jj * ls + ord[c]];
        }
        __syncthreads();
    }
}

void launch_write_v(const TileWork *d_tiles, int ntiles, Workspace ws,
                    OutArena out, cudaStream_t stream)
{
    // wide bases: at least 8 columns a pass
    const int doubles = std::max(kWriteVDoubles, 8 * (ws.k_max | 1));
    const size_t smem = (size_t)doubles * sizeof(double);
    allow_smem<k_write_v, (size_t)8 * (kMaxK | 1) * sizeof(double)>();
    dim3 grid(ntiles, ntiles >= 148 ? 4 : 8);
    k_write_v<<<grid, 256, smem, stream>>>(d_tiles, ws, out, doubles);
}

}  // namespace b200
