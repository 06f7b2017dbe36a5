// Batched FP64 GEMM (see gemm_f64.cuh): FP64 mma.sync m8n8k4, eight warps a
// CTA.  One kernel for each shape of product:
//   sketch (A B, long K)           k_gemm_f64
//   basis updates, U (A B, short K) k_gemm_f64_nn_short
//   rounds' A^T B, Gram B B^T      k_gemm_f64_tn_pipe, k_gemm_f64_nt_pipe
//   projection, rotation (A^T B, wide) k_gemm_f64_tn_wide
// Warps skip the DMMAs of output regions outside the tile's own M x N and of
// k4 steps past its K (those would add exact zeros); the order of each sum is
// the same in all of them (one chain over K, but for split_k).
#include <cstdint>
#include "gemm_step.cuh"
#include "smem_limit.cuh"

namespace b200 {

__device__ __forceinline__ void dmma_8x8x4(double &c0, double &c1, double a,
                                           double b)
{
    asm volatile(
        "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
        "{%0,%1}, {%2}, {%3}, {%0,%1};\n"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// A B with a long K, the sketch Y = D Omega: CTA tile 64 x 64 or (sketch
// blocks of 32 columns) 128 x 32, K step 16.  Operand tiles are staged in
// shared memory double-buffered, the next K step fetched into registers while
// the current one is multiplied; A lies there as [k][row] with stride rows +
// 4, B as [column][k] with stride 20, so that both the stores and the
// fragment reads are free of bank conflicts.  Three CTAs an SM.  Bound by the
// DMMA pipe (74 % busy in a launch of 90 tiles of 1024 x 1024 by 272, 26.7
// TFLOP/s); the three-stage cp.async kernel of the short
// products is no faster here.
template <int BM, int BN>
__global__ void __launch_bounds__(kGemmThreads, 3)
k_gemm_f64(const __grid_constant__ GemmArgs args, int tiles_n)
{
    // 8 warps of 32 x 16 output each, BM / 32 along M and BN / 16 along N
    constexpr int WARPS_M = BM / 32;
    static_assert(WARPS_M * (BN / 16) == kGemmThreads / 32, "warp grid");
    constexpr int RA = BM * kGemmBK / kGemmThreads;   // A loads per thread
    constexpr int RB = BN * kGemmBK / kGemmThreads;   // B loads per thread
    const GemmDesc d = gemm_desc(args, blockIdx.y);
    const int tm = blockIdx.x / tiles_n;
    const int tn = blockIdx.x % tiles_n;
    const int m0 = tm * BM, n0 = tn * BN;
    if (m0 >= d.M || n0 >= d.N) return;

    // [2][BM * kGemmLds] then [2][BN * kGemmLds], dynamic (above 48 KB
    // for the 128 x 32 shape)
    extern __shared__ double gemm_smem[];
    double (*As)[BM * kGemmLds] = reinterpret_cast<double (*)[BM * kGemmLds]>(gemm_smem);
    double (*Bs)[BN * kGemmLds] =
        reinterpret_cast<double (*)[BN * kGemmLds]>(gemm_smem + 2 * BM * kGemmLds);

    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const int wm = (warp % WARPS_M) * 32;   // warp row offset in the CTA tile
    const int wn = (warp / WARPS_M) * 16;   // warp column offset

    double acc[4][2][2];
    #pragma unroll
    for (int i = 0; i < 4; ++i)
        #pragma unroll
        for (int j = 0; j < 2; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    double ra[RA], rb[RB];
    // element e = t + 256 r of a tile, along the contiguous dimension: A
    // rows fastest, B k fastest
    constexpr int LDA = BM + 4;
    auto load_tiles = [&](int k0) {
        #pragma unroll
        for (int r = 0; r < RA; ++r) {
            const int e = t + kGemmThreads * r;
            const int gm = m0 + e % BM, gk = k0 + e / BM;
            ra[r] = gm < d.M && gk < d.K ? d.A[(size_t)gk * d.lda + gm] : 0.0;
        }
        #pragma unroll
        for (int r = 0; r < RB; ++r) {
            const int e = t + kGemmThreads * r;
            const int gn = n0 + e / kGemmBK, gk = k0 + e % kGemmBK;
            rb[r] = gn < d.N && gk < d.K ? d.B[(size_t)gn * d.ldb + gk] : 0.0;
        }
    };
    auto store_tiles = [&](int buf) {
        #pragma unroll
        for (int r = 0; r < RA; ++r) {
            const int e = t + kGemmThreads * r;
            As[buf][e / BM * LDA + e % BM] = ra[r];
        }
        #pragma unroll
        for (int r = 0; r < RB; ++r) {
            const int e = t + kGemmThreads * r;
            Bs[buf][e / kGemmBK * kGemmLds + e % kGemmBK] = rb[r];
        }
    };

    const int ktiles = (d.K + kGemmBK - 1) / kGemmBK;
    if (ktiles > 0) {
        load_tiles(0);
        store_tiles(0);
        __syncthreads();
    }
    // this warp's 32 x 16 output region holds part of the tile's M x N
    const bool live = m0 + wm < d.M && n0 + wn < d.N;
    for (int kt = 0; kt < ktiles; ++kt) {
        const int buf = kt & 1;
        if (kt + 1 < ktiles) load_tiles((kt + 1) * kGemmBK);
        // k4 steps of this warp in the K step (warp-uniform)
        const int kend = live ? min(kGemmBK, d.K - kt * kGemmBK) : 0;
        #pragma unroll
        for (int kk = 0; kk < kGemmBK; kk += 4) {
            if (kk >= kend) break;
            double af[4], bf[2];
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                af[i] = As[buf][(kk + tig) * LDA + wm + i * 8 + g];
            #pragma unroll
            for (int j = 0; j < 2; ++j)
                bf[j] = Bs[buf][(wn + j * 8 + g) * kGemmLds + kk + tig];
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                #pragma unroll
                for (int j = 0; j < 2; ++j)
                    dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
        if (kt + 1 < ktiles) {
            store_tiles(buf ^ 1);
        }
        __syncthreads();
    }

    // accumulator (i, j, h) holds C(wm + 8i + g, wn + 8j + 2 tig + h); a
    // sketch has no old C
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + wm + i * 8 + g;
        if (gm >= d.M) continue;
        #pragma unroll
        for (int j = 0; j < 2; ++j)
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gn = n0 + wn + j * 8 + 2 * tig + h;
                if (gn < d.N) d.C[(size_t)gn * d.ldc + gm] = d.alpha * acc[i][j][h];
            }
    }
}

// A^T B with 64 x 64 CTA tiles and a cp.async pipeline: the transposed
// products (Grams and projections onto the basis in the rounds) have outputs
// of a few tiles and K = the tile height, so one CTA walks a long K; a kernel
// that stages through registers has one K step in flight and waits on memory
// latency every step.  Operand tiles land in shared memory directly
// (16-byte cp.async, k contiguous in both operands).  Where a tile fills
// every warp's output region, the per-element accumulation order is that of
// k_gemm_f64 (the DMMA's k order, k4 steps in order), so results are
// identical to it; in a launch that asks for it (split_k), a tile with at
// most 32 rows or 48 columns of its own splits K over the spare warps (fixed
// slice order, deterministic).
//
// With few rows a step has little to multiply, and the instructions around
// it bound the kernel (16 tiles of 1024 rows, 32 columns: 212 a warp and
// step of 16, 0.7 us): a step is 32 deep, a warp walks its own k4 steps only,
// and copies advance their pointers.
constexpr int kShallow = 3;            // stages of the fitted 64 x 128 kernel
constexpr int kPipeK = 32;
constexpr int kPipeLds = kPipeK + 4;   // [row][k]: fragment reads free of conflicts
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem, bool pred)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    const int n = pred ? 16 : 0;   // zero-fill when outside the operand
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"(sa), "l"(gmem), "r"(n));
}

// A thread's share of an operand tile that is contiguous along k: rows t / 8 +
// 32 r (r < R) of the tile, k pair t % 8 of each K step, in stages of
// [row][kGemmLds], `pitch` rows apart.  What a row needs is worked out once (a K step of the
// pipelined kernels is short, and addresses and bounds worked out per piece
// took more issue slots than its products); rows outside the operand are
// zeroed in every stage at the start and not copied.
template <int R, int STAGES>
struct PipeRows {
    const double *src[R];
    double *dst;
    bool row_ok[R], even;

    __device__ __forceinline__ void init(const double *base, int ld, int g0, int lim,
                                         double *stages, int pitch, int tile_rows)
    {
        const int row = threadIdx.x >> 3, kk = (threadIdx.x & 7) * 2;
        even = (ld & 1) == 0 && ((uintptr_t)base & 15) == 0;
        dst = stages + row * kGemmLds + kk;
        #pragma unroll
        for (int r = 0; r < R; ++r) {
            const int g = g0 + row + 32 * r;
            row_ok[r] = row + 32 * r < tile_rows && g < lim;
            src[r] = base + (size_t)(row_ok[r] ? g : g0) * ld + kk;
            if (!row_ok[r] && row + 32 * r < tile_rows)
                for (int s = 0; s < STAGES; ++s) {
                    double *z = dst + (s * pitch + 32 * r) * kGemmLds;
                    z[0] = z[1] = 0.0;
                }
        }
    }
    // The K step at k0 into the stage whose first row is `at`.
    __device__ __forceinline__ void copy(int at, int k0, int K) const
    {
        const int gk = k0 + (threadIdx.x & 7) * 2;
        if (even && gk + 1 < K) {
            #pragma unroll
            for (int r = 0; r < R; ++r)
                if (row_ok[r])
                    cp_async16(dst + (at + 32 * r) * kGemmLds, src[r] + k0, true);
        } else {
            #pragma unroll
            for (int r = 0; r < R; ++r)
                if (row_ok[r]) {
                    double *q = dst + (at + 32 * r) * kGemmLds;
                    q[0] = gk < K ? src[r][k0] : 0.0;
                    q[1] = gk + 1 < K ? src[r][k0 + 1] : 0.0;
                }
        }
    }
};

// Output regions of 32 x 16, one per warp when the tile's own rows and
// columns fill the CTA tile.  A 64 x 64 tile with fewer (the products onto a
// narrow basis, Grams of a few columns) gives the spare warps a share of K
// instead: nreg regions (rounded up to rp, a power of two), warp w works on
// region w % rp over the k4 steps q = w / rp modulo nsl = 8 / rp, and the nsl
// partial sums are added in slice order through shared memory.  Every
// scheduler keeps the same share of the DMMA work.
struct PipeSplit {
    int rh = 2, rp = 8, nsl = 1;
    __device__ __forceinline__ PipeSplit(int rows, int cols, int split_k)
    {
        if (!split_k) return;
        rh = rows > 32 ? 2 : 1;
        const int nreg = rh * min(4, (cols + 15) / 16);
        rp = nreg <= 1 ? 1 : nreg <= 2 ? 2 : nreg <= 4 ? 4 : 8;
        nsl = 8 / rp;
    }
};

// acc += the k4 step at offset k4 of a stage: fragments A(wm + 8 i + g, k4 +
// tig), B(wn + 8 j + g, k4 + tig) at a + 8 i * ra, b + 8 j * rb.
__device__ __forceinline__ void pipe_k4(double (&acc)[4][2][2], const double *a, int ra,
                                        const double *b, int rb)
{
    double af[4], bf[2];
    #pragma unroll
    for (int i = 0; i < 4; ++i) af[i] = a[i * 8 * ra];
    #pragma unroll
    for (int j = 0; j < 2; ++j) bf[j] = b[j * 8 * rb];
    #pragma unroll
    for (int i = 0; i < 4; ++i)
        #pragma unroll
        for (int j = 0; j < 2; ++j)
            dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
}

// STAGES: three where the launch has at most one CTA per SM, else two (two
// CTAs per SM).
template <int STAGES>
__global__ void __launch_bounds__(kGemmThreads)
k_gemm_f64_tn_pipe(const __grid_constant__ GemmArgs args, int tiles_n, int split_k)
{
    constexpr int BM = 64, BN = 64;
    const GemmDesc d = gemm_desc(args, blockIdx.y);
    const int tm = blockIdx.x / tiles_n, tn = blockIdx.x % tiles_n;
    const int m0 = tm * BM, n0 = tn * BN;
    if (m0 >= d.M || n0 >= d.N) return;
    extern __shared__ double gemm_smem[];
    // [stage][64 rows of A^T, 64 rows of B^T][kPipeLds]
    constexpr int STAGE = (BM + BN) * kPipeLds;
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const PipeSplit sp(d.M - m0, d.N - n0, split_k);
    const int rh = sp.rh, rp = sp.rp, nsl = sp.nsl;
    const int reg = warp % rp, slice = warp / rp;
    const int wm = (reg % rh) * 32, wn = (reg / rh) * 16;
    const bool live = wm < BM && wn < BN && m0 + wm < d.M && n0 + wn < d.N;
    double acc[4][2][2] = {};
    // 16-byte pieces: rows t / 16 + 16 r of A and of B, k pair t % 16; rows
    // outside the operand are zeroed in every stage and not copied
    const int row = t >> 4, kk = (t & 15) * 2;
    const double *pa[4], *pb[4];
    bool oa[4], ob[4];
    double *dst = gemm_smem + row * kPipeLds + kk;
    #pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int ga = m0 + row + 16 * r, gb = n0 + row + 16 * r;
        oa[r] = ga < d.M;
        ob[r] = gb < d.N;
        pa[r] = d.A + (size_t)(oa[r] ? ga : m0) * d.lda + kk;
        pb[r] = d.B + (size_t)(ob[r] ? gb : n0) * d.ldb + kk;
        #pragma unroll
        for (int s = 0; s < STAGES; ++s) {
            double *z = dst + s * STAGE + 16 * r * kPipeLds;
            if (!oa[r]) z[0] = z[1] = 0.0;
            if (!ob[r]) z[BM * kPipeLds] = z[BM * kPipeLds + 1] = 0.0;
        }
    }
    const bool even = (d.lda & 1) == 0 && ((uintptr_t)d.A & 15) == 0 &&
                      (d.ldb & 1) == 0 && ((uintptr_t)d.B & 15) == 0;
    int left = d.K - kk;                       // k indices from this thread's next pair
    int ist = 0;                               // stage of the next copy
    auto issue = [&]() {
        double *q = dst + ist * STAGE;
        if (even && left >= 2) {
            #pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (oa[r]) cp_async16(q + 16 * r * kPipeLds, pa[r], true);
                if (ob[r]) cp_async16(q + (BM + 16 * r) * kPipeLds, pb[r], true);
            }
        } else {
            #pragma unroll
            for (int r = 0; r < 4; ++r) {
                double *za = q + 16 * r * kPipeLds, *zb = za + BM * kPipeLds;
                if (oa[r]) {
                    za[0] = left >= 1 ? pa[r][0] : 0.0;
                    za[1] = left >= 2 ? pa[r][1] : 0.0;
                }
                if (ob[r]) {
                    zb[0] = left >= 1 ? pb[r][0] : 0.0;
                    zb[1] = left >= 2 ? pb[r][1] : 0.0;
                }
            }
        }
        #pragma unroll
        for (int r = 0; r < 4; ++r) {
            pa[r] += kPipeK;
            pb[r] += kPipeK;
        }
        left -= kPipeK;
        ist = ist + 1 == STAGES ? 0 : ist + 1;
    };
    const int ktiles = (d.K + kPipeK - 1) / kPipeK;
    #pragma unroll
    for (int p = 0; p < STAGES - 1; ++p) {
        if (p < ktiles) issue();
        asm volatile("cp.async.commit_group;");
    }
    const double *fa = gemm_smem + (wm + g) * kPipeLds + tig;
    const double *fb = gemm_smem + (BM + wn + g) * kPipeLds + tig;
    int cst = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
        // the group of step kt has landed (at most STAGES - 2 newer ones
        // still in flight)
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2));
        __syncthreads();
        if (kt + STAGES - 1 < ktiles) issue();
        asm volatile("cp.async.commit_group;");
        const double *a = fa + cst * STAGE, *b = fb + cst * STAGE;
        if (live) {
            if (nsl == 1) {
                #pragma unroll
                for (int k4 = 0; k4 < kPipeK / 4; ++k4)
                    pipe_k4(acc, a + 4 * k4, kPipeLds, b + 4 * k4, kPipeLds);
            } else {
                // this warp's k4 steps (8 per step, a multiple of nsl)
                #pragma unroll 1
                for (int k4 = slice; k4 < kPipeK / 4; k4 += nsl)
                    pipe_k4(acc, a + 4 * k4, kPipeLds, b + 4 * k4, kPipeLds);
            }
        }
        cst = cst + 1 == STAGES ? 0 : cst + 1;
    }
    asm volatile("cp.async.wait_group 0;");
    if (nsl > 1) {
        // partial sums of the slices, [warp][16 accumulators][32 lanes]
        // over the stage buffers, added by slice 0 in slice order
        __syncthreads();
        double *part = gemm_smem + warp * 512;
        #pragma unroll
        for (int i = 0; i < 4; ++i)
            #pragma unroll
            for (int j = 0; j < 2; ++j)
                #pragma unroll
                for (int h = 0; h < 2; ++h) part[((i * 2 + j) * 2 + h) * 32 + lane] = acc[i][j][h];
        __syncthreads();
        if (slice != 0) return;
        for (int q = 1; q < nsl; ++q) {
            const double *pq = gemm_smem + (warp + q * rp) * 512;
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                #pragma unroll
                for (int j = 0; j < 2; ++j)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) acc[i][j][h] += pq[((i * 2 + j) * 2 + h) * 32 + lane];
        }
    }
    if (!live) return;
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + wm + i * 8 + g;
        if (gm >= d.M) continue;
        #pragma unroll
        for (int j = 0; j < 2; ++j) {
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gn = n0 + wn + j * 8 + 2 * tig + h;
                if (gn >= d.N) continue;
                double *c = d.C + (size_t)gn * d.ldc + gm;
                double v = d.alpha * acc[i][j][h];
                if (d.beta != 0.0) v += d.beta * *c;
                *c = v;
            }
        }
    }
}

// A^T B for wide outputs whose rows are a basis of a tile (the projection
// B = Q^T D, K = the tile height, and the rotation C = W^T B): a CTA takes
// 128 columns and up to 64 rows, each warp 16 columns and all of the rows,
// in 8 MF rows fitted to the tile's own basis (a loop compiled per MF).
// The DMMA pipe bounds a tile of many rows and the read of D one of few:
// with 32 x 128 CTA tiles the pipe multiplied the padding up to 32 rows and
// a basis of 33 .. 64 rows read D twice.  Per element the K order is that of
// k_gemm_f64 (bit-identical).  Three stages (90 KB), two CTAs per SM.
constexpr int kWideN = 128, kWideM = 64;

template <int MF>
__device__ __forceinline__ void tn_wide(const GemmDesc &d, int m0, int n0,
                                        double *smem)
{
    constexpr int STAGE = (kWideM + kWideN) * kGemmLds;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3, wn = warp * 16;
    PipeRows<(MF + 3) / 4, kShallow> ra;
    PipeRows<kWideN / 32, kShallow> rb;
    ra.init(d.A, d.lda, m0, d.M, smem, kWideM + kWideN, MF * 8);
    rb.init(d.B, d.ldb, n0, d.N, smem + kWideM * kGemmLds, kWideM + kWideN, kWideN);
    auto issue = [&](int kt) {
        const int at = kt % kShallow * (kWideM + kWideN), k0 = kt * kGemmBK;
        ra.copy(at, k0, d.K);
        rb.copy(at, k0, d.K);
        asm volatile("cp.async.commit_group;");
    };
    double acc[MF][2][2] = {};
    const int ktiles = (d.K + kGemmBK - 1) / kGemmBK;
    #pragma unroll
    for (int p = 0; p < kShallow - 1; ++p) {
        if (p < ktiles) issue(p);
        else asm volatile("cp.async.commit_group;");
    }
    for (int kt = 0; kt < ktiles; ++kt) {
        asm volatile("cp.async.wait_group %0;" :: "n"(kShallow - 2));
        __syncthreads();
        if (kt + kShallow - 1 < ktiles) issue(kt + kShallow - 1);
        else asm volatile("cp.async.commit_group;");
        const double *A = smem + kt % kShallow * STAGE, *B = A + kWideM * kGemmLds;
        #pragma unroll
        for (int k4 = 0; k4 < kGemmBK; k4 += 4) {
            double af[MF], bf[2];
            #pragma unroll
            for (int j = 0; j < 2; ++j) bf[j] = B[(wn + j * 8 + g) * kGemmLds + k4 + tig];
            #pragma unroll
            for (int i = 0; i < MF; ++i) af[i] = A[(i * 8 + g) * kGemmLds + k4 + tig];
            #pragma unroll
            for (int i = 0; i < MF; ++i)
                #pragma unroll
                for (int j = 0; j < 2; ++j)
                    dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;");
    #pragma unroll
    for (int i = 0; i < MF; ++i) {
        const int gm = m0 + i * 8 + g;
        if (gm >= d.M) continue;
        #pragma unroll
        for (int j = 0; j < 2; ++j)
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gn = n0 + wn + j * 8 + 2 * tig + h;
                if (gn >= d.N) continue;
                double *c = d.C + (size_t)gn * d.ldc + gm;
                double v = d.alpha * acc[i][j][h];
                if (d.beta != 0.0) v += d.beta * *c;
                *c = v;
            }
    }
}

__global__ void __launch_bounds__(kGemmThreads, 2)
k_gemm_f64_tn_wide(const __grid_constant__ GemmArgs args, int tiles_n)
{
    extern __shared__ double gemm_smem[];
    const GemmDesc d = gemm_desc(args, blockIdx.y);
    const int m0 = blockIdx.x / tiles_n * kWideM, n0 = blockIdx.x % tiles_n * kWideN;
    if (m0 >= d.M || n0 >= d.N) return;
    switch (min(kWideM, d.M - m0) + 7 >> 3) {
    case 1: tn_wide<1>(d, m0, n0, gemm_smem); break;
    case 2: tn_wide<2>(d, m0, n0, gemm_smem); break;
    case 3: tn_wide<3>(d, m0, n0, gemm_smem); break;
    case 4: tn_wide<4>(d, m0, n0, gemm_smem); break;
    case 5: tn_wide<5>(d, m0, n0, gemm_smem); break;
    case 6: tn_wide<6>(d, m0, n0, gemm_smem); break;
    case 7: tn_wide<7>(d, m0, n0, gemm_smem); break;
    default: tn_wide<8>(d, m0, n0, gemm_smem);
    }
}

// A B^T with 64 x 64 CTA tiles (the Gram B B^T of the small SVD, K = the
// tile width) through the same cp.async pipeline as the transposed
// products.  Here rows are contiguous in both operands and k is strided, so
// the tiles are staged as [k][row] (row stride 68 doubles: fragment reads free
// of bank conflicts); a 16-byte piece is two consecutive rows at one k.  Without split_k the per-element accumulation
// order is that of k_gemm_f64 (k4 steps in order), so results are
// identical to it; with it, K is split over the warps of empty output
// regions as in the transposed kernel.
// Three CTAs per SM where the launch has more than one CTA per SM (in 80
// registers; with the compiler's own 122, two: 256 tiles of 1024 columns 264
// -> 241 us, 2500 tiles of 400 columns and bases of about 130 1945 -> 1443).
// The A^T B kernel, whose copies hold more pointers, spills at three and is
// slower (554 -> 704 us over 16 launches).
constexpr int kNtLds = 64 + 4;

template <int STAGES>
__global__ void __launch_bounds__(kGemmThreads, STAGES == 2 ? 3 : 1)
k_gemm_f64_nt_pipe(const __grid_constant__ GemmArgs args, int tiles_n, int split_k)
{
    constexpr int BM = 64, BN = 64;
    const GemmDesc d = gemm_desc(args, blockIdx.y);
    const int tm = blockIdx.x / tiles_n, tn = blockIdx.x % tiles_n;
    const int m0 = tm * BM, n0 = tn * BN;
    if (m0 >= d.M || n0 >= d.N) return;
    extern __shared__ double gemm_smem[];
    // [stage][32 k of A, 32 k of B][kNtLds]
    constexpr int STAGE = 2 * kPipeK * kNtLds;
    const int t = threadIdx.x;
    const int lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3;
    const PipeSplit sp(d.M - m0, d.N - n0, split_k);
    const int rh = sp.rh, rp = sp.rp, nsl = sp.nsl;
    const int reg = warp % rp, slice = warp / rp;
    const int wm = (reg % rh) * 32, wn = (reg / rh) * 16;
    const bool live = wm < BM && wn < BN && m0 + wm < d.M && n0 + wn < d.N;
    double acc[4][2][2] = {};
    // 16-byte pieces: rows 2 (t % 32) and the next, k = t / 32 + 8 r of a K
    // step, of A and of B; rows outside the operand are zeroed in every
    // stage and not copied
    const int row = (t & 31) * 2, kk = t >> 5;
    const int na = max(0, min(2, d.M - m0 - row)), nb = max(0, min(2, d.N - n0 - row));
    const double *pa = d.A + m0 + (na ? row : 0) + (size_t)kk * d.lda;
    const double *pb = d.B + n0 + (nb ? row : 0) + (size_t)kk * d.ldb;
    const size_t sa = (size_t)8 * d.lda, sb = (size_t)8 * d.ldb;
    double *dst = gemm_smem + kk * kNtLds + row;
    #pragma unroll
    for (int s = 0; s < STAGES; ++s)
        #pragma unroll
        for (int r = 0; r < 4; ++r) {
            double *z = dst + s * STAGE + 8 * r * kNtLds;
            if (na < 2) z[1] = 0.0;
            if (na < 1) z[0] = 0.0;
            if (nb < 2) z[kPipeK * kNtLds + 1] = 0.0;
            if (nb < 1) z[kPipeK * kNtLds] = 0.0;
        }
    const bool even = (d.lda & 1) == 0 && ((uintptr_t)d.A & 15) == 0 &&
                      (d.ldb & 1) == 0 && ((uintptr_t)d.B & 15) == 0;
    const bool whole = even && na != 1 && nb != 1;
    int left = d.K - kk;
    int ist = 0;
    auto issue = [&]() {
        double *q = dst + ist * STAGE;
        #pragma unroll
        for (int r = 0; r < 4; ++r) {
            double *za = q + 8 * r * kNtLds, *zb = za + kPipeK * kNtLds;
            const bool in = left > 8 * r;
            if (whole && in) {
                if (na) cp_async16(za, pa, true);
                if (nb) cp_async16(zb, pb, true);
            } else {
                if (na > 0) za[0] = in ? pa[0] : 0.0;
                if (na > 1) za[1] = in ? pa[1] : 0.0;
                if (nb > 0) zb[0] = in ? pb[0] : 0.0;
                if (nb > 1) zb[1] = in ? pb[1] : 0.0;
            }
            pa += sa;
            pb += sb;
        }
        left -= kPipeK;
        ist = ist + 1 == STAGES ? 0 : ist + 1;
    };
    const int ktiles = (d.K + kPipeK - 1) / kPipeK;
    #pragma unroll
    for (int p = 0; p < STAGES - 1; ++p) {
        if (p < ktiles) issue();
        asm volatile("cp.async.commit_group;");
    }
    const double *fa = gemm_smem + tig * kNtLds + wm + g;
    const double *fb = gemm_smem + (kPipeK + tig) * kNtLds + wn + g;
    int cst = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2));
        __syncthreads();
        if (kt + STAGES - 1 < ktiles) issue();
        asm volatile("cp.async.commit_group;");
        const double *a = fa + cst * STAGE, *b = fb + cst * STAGE;
        if (live) {
            if (nsl == 1) {
                #pragma unroll
                for (int k4 = 0; k4 < kPipeK / 4; ++k4)
                    pipe_k4(acc, a + 4 * k4 * kNtLds, 1, b + 4 * k4 * kNtLds, 1);
            } else {
                #pragma unroll 1
                for (int k4 = slice; k4 < kPipeK / 4; k4 += nsl)
                    pipe_k4(acc, a + 4 * k4 * kNtLds, 1, b + 4 * k4 * kNtLds, 1);
            }
        }
        cst = cst + 1 == STAGES ? 0 : cst + 1;
    }
    asm volatile("cp.async.wait_group 0;");
    if (nsl > 1) {
        __syncthreads();
        double *part = gemm_smem + warp * 512;
        #pragma unroll
        for (int i = 0; i < 4; ++i)
            #pragma unroll
            for (int j = 0; j < 2; ++j)
                #pragma unroll
                for (int h = 0; h < 2; ++h) part[((i * 2 + j) * 2 + h) * 32 + lane] = acc[i][j][h];
        __syncthreads();
        if (slice != 0) return;
        for (int q = 1; q < nsl; ++q) {
            const double *pq = gemm_smem + (warp + q * rp) * 512;
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                #pragma unroll
                for (int j = 0; j < 2; ++j)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) acc[i][j][h] += pq[((i * 2 + j) * 2 + h) * 32 + lane];
        }
    }
    if (!live) return;
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + wm + i * 8 + g;
        if (gm >= d.M) continue;
        #pragma unroll
        for (int j = 0; j < 2; ++j) {
            #pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gn = n0 + wn + j * 8 + 2 * tig + h;
                if (gn >= d.N) continue;
                double *c = d.C + (size_t)gn * d.ldc + gm;
                double v = d.alpha * acc[i][j][h];
                if (d.beta != 0.0) v += d.beta * *c;
                *c = v;
            }
        }
    }
}

// A B with a short K (the basis updates: K and N a round's columns or the
// basis so far; U = Q W).  A CTA takes `iters` blocks of 64 rows and up to 64
// columns; K steps of 32 of the (row block, K step) sequence run through
// three cp.async stages, so a block's loads -- most often one step -- are in
// flight two blocks ahead, and the tile's record is read once for all of
// them.  The eight warps split the 64 rows finer where the tile has few
// columns (16 columns and 8, 16 or 32 rows a warp).  The register-staged
// kernel above waited a memory round trip in every K step of 16, and once
// more for C: 256 tiles of 1024 rows and about 25 columns 57 us.  Per
// element the K order is the same (bit-identical).
constexpr int kNnK = 32, kNnRows = 64, kNnStages = 3;
constexpr int kNnLdA = kNnRows + 4, kNnLdB = kNnK + 4;   // [k][row], [n][k]
constexpr int kNnStage = kNnK * kNnLdA + 64 * kNnLdB;

template <int MI>
__device__ __forceinline__ void nn_short(const GemmDesc &d, int m_first, int m_last,
                                         int n0, double *smem)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int g = lane >> 2, tig = lane & 3;
    constexpr int WM = kNnRows / (8 * MI);           // warps along the rows
    const int wm = warp % WM * 8 * MI, wn = warp / WM * 16;
    const bool live = n0 + wn < d.N;
    const int ksteps = max(1, (d.K + kNnK - 1) / kNnK);
    const int blocks = (m_last - m_first + kNnRows - 1) / kNnRows;
    const int total = blocks * ksteps;
    const bool evenA = (d.lda & 1) == 0 && ((uintptr_t)d.A & 15) == 0;
    const bool evenB = (d.ldb & 1) == 0 && ((uintptr_t)d.B & 15) == 0;
    // copies of A: rows 2 (t % 32) and the next, k = t / 32 + 8 r; of B: k
    // pair t % 16, columns t / 16 + 16 r
    const int ar = (t & 31) * 2, ak = t >> 5, bk = (t & 15) * 2, bn = t >> 4;
    int blk = 0, kst = 0;                            // next step to copy
    auto issue = [&](int st) {
        double *A = smem + st % kNnStages * kNnStage, *B = A + kNnK * kNnLdA;
        const int k0 = kst * kNnK, row = m_first + blk * kNnRows + ar;
        #pragma unroll
        for (int r = 0; r < kNnK / 8; ++r) {
            const int k = k0 + ak + 8 * r;
            double *dst = A + (ak + 8 * r) * kNnLdA + ar;
            if (k < d.K) {
                const double *src = d.A + row + (size_t)(d.gather ? d.gather[k] : k) * d.lda;
                if (evenA && row + 1 < m_last) {
                    cp_async16(dst, src, true);
                } else {
                    dst[0] = row < m_last ? src[0] : 0.0;
                    dst[1] = row + 1 < m_last ? src[1] : 0.0;
                }
            } else {
                dst[0] = dst[1] = 0.0;
            }
        }
        #pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int n = bn + 16 * r;
            if (n0 + n >= (d.N + 15) / 16 * 16) break;
            double *dst = B + n * kNnLdB + bk;
            const int k = k0 + bk;
            const bool in = n0 + n < d.N;
            const double *src = d.B + k +
                (size_t)(in && d.gather_b ? d.gather_b[n0 + n] : n0 + n) * d.ldb;
            if (in && evenB && k + 1 < d.K) {
                cp_async16(dst, src, true);
            } else {
                dst[0] = in && k < d.K ? src[0] : 0.0;
                dst[1] = in && k + 1 < d.K ? src[1] : 0.0;
            }
        }
        if (++kst == ksteps) {
            kst = 0;
            ++blk;
        }
    };
    #pragma unroll
    for (int p = 0; p < kNnStages - 1; ++p) {
        if (p < total) issue(p);
        asm volatile("cp.async.commit_group;");
    }
    const bool upd = d.beta != 0.0;
    int st = 0;
    #pragma unroll 1
    for (int b = 0; b < blocks; ++b) {
        const int m0 = m_first + b * kNnRows + wm;
        double acc[MI][2][2] = {}, cold[MI][2][2];
        // the old C of an update is read before the products need to be done
        if (upd) {
            #pragma unroll
            for (int i = 0; i < MI; ++i)
                #pragma unroll
                for (int j = 0; j < 2; ++j)
                    #pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int gm = m0 + i * 8 + g, gn = n0 + wn + j * 8 + 2 * tig + h;
                        cold[i][j][h] = gm < m_last && gn < d.N
                                            ? d.C[(size_t)gn * d.ldc + gm] : 0.0;
                    }
        }
        #pragma unroll 1
        for (int ks = 0; ks < ksteps; ++ks, ++st) {
            asm volatile("cp.async.wait_group %0;" :: "n"(kNnStages - 2));
            __syncthreads();
            if (st + kNnStages - 1 < total) issue(st + kNnStages - 1);
            asm volatile("cp.async.commit_group;");
            if (!live) continue;
            const double *A = smem + st % kNnStages * kNnStage, *B = A + kNnK * kNnLdA;
            const int kend = min(kNnK, d.K - ks * kNnK);
            #pragma unroll
            for (int kk = 0; kk < kNnK; kk += 4) {
                if (kk >= kend) break;
                double af[MI], bf[2];
                #pragma unroll
                for (int i = 0; i < MI; ++i) af[i] = A[(kk + tig) * kNnLdA + wm + i * 8 + g];
                #pragma unroll
                for (int j = 0; j < 2; ++j) bf[j] = B[(wn + j * 8 + g) * kNnLdB + kk + tig];
                #pragma unroll
                for (int i = 0; i < MI; ++i)
                    #pragma unroll
                    for (int j = 0; j < 2; ++j)
                        dmma_8x8x4(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
            }
        }
        if (!live) continue;
        #pragma unroll
        for (int i = 0; i < MI; ++i) {
            const int gm = m0 + i * 8 + g;
            if (gm >= m_last) continue;
            #pragma unroll
            for (int j = 0; j < 2; ++j)
                #pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int gn = n0 + wn + j * 8 + 2 * tig + h;
                    if (gn >= d.N) continue;
                    double v = d.alpha * acc[i][j][h];
                    if (upd) v += d.beta * cold[i][j][h];
                    d.C[(size_t)gn * d.ldc + gm] = v;
                }
        }
    }
    asm volatile("cp.async.wait_group 0;");
}

__global__ void __launch_bounds__(kGemmThreads, 2)
k_gemm_f64_nn_short(const __grid_constant__ GemmArgs args, int tiles_n, int iters)
{
    extern __shared__ __align__(16) double nn_smem[];
    const GemmDesc d = gemm_desc(args, blockIdx.y);
    const int m_first = blockIdx.x / tiles_n * iters * kNnRows;
    const int n0 = blockIdx.x % tiles_n * 64;
    if (m_first >= d.M || n0 >= d.N) return;
    const int m_last = min(d.M, m_first + iters * kNnRows);
    const int cols = min(64, d.N - n0);
    if (cols <= 16) nn_short<1>(d, m_first, m_last, n0, nn_smem);
    else if (cols <= 32) nn_short<2>(d, m_first, m_last, n0, nn_smem);
    else nn_short<4>(d, m_first, m_last, n0, nn_smem);
}

// One launch of Kernel with Smem bytes of dynamic shared memory.
template <auto Kernel, size_t Smem, class... Rest>
static cudaError_t launch_gemm(dim3 grid, cudaStream_t stream, const GemmArgs &args,
                               Rest... rest)
{
    allow_smem<Kernel, Smem>();
    Kernel<<<grid, kGemmThreads, Smem, stream>>>(args, rest...);
    return cudaGetLastError();
}

cudaError_t gemm_f64_batched(bool ta, bool tb, const GemmArgs &args, int batch,
                             int max_m, int max_n, cudaStream_t stream,
                             bool split_k)
{
    if (batch <= 0 || max_m <= 0 || max_n <= 0) return cudaSuccess;
    if (!ta && !tb) {
        const int tiles_n = (max_n + 63) / 64;
        if (args.step == STEP_SKETCH || args.step == STEP_A_SKETCH) {
            // 128 x 32 tiles for sketch blocks of at most 32 columns
            constexpr auto smem = [](int bm, int bn) {
                return 2 * (bm + bn) * kGemmLds * sizeof(double);
            };
            if (max_n <= 32 && max_m >= 128)
                return launch_gemm<k_gemm_f64<128, 32>, smem(128, 32)>(
                    dim3((max_m + 127) / 128 * tiles_n, batch), stream, args, tiles_n);
            return launch_gemm<k_gemm_f64<64, 64>, smem(64, 64)>(
                dim3((max_m + 63) / 64 * tiles_n, batch), stream, args, tiles_n);
        }
        // four row blocks to a CTA where that still leaves two rounds of
        // CTAs, else one
        const int blocks = (max_m + kNnRows - 1) / kNnRows;
        const int iters = (size_t)((blocks + 3) / 4) * tiles_n * batch >= 592 ? 4 : 1;
        constexpr size_t smem = (size_t)kNnStages * kNnStage * sizeof(double);
        return launch_gemm<k_gemm_f64_nn_short, smem>(
            dim3((blocks + iters - 1) / iters * tiles_n, batch), stream, args, tiles_n, iters);
    }
    if (ta == tb) return cudaErrorInvalidValue;   // (no step multiplies A^T B^T)
    // A^T B whose output is wide and (as for the projection B = Q^T D and the
    // rotation C = W^T B) has a basis much narrower than the batch maximum as
    // its rows: the fitted 64 x 128 kernel.  Else 64 x 64.
    const bool wide = ta && !split_k && max_n >= 256;
    const int tiles_m = (max_m + 63) / 64;
    const int tiles_n = (max_n + (wide ? kWideN : 64) - 1) / (wide ? kWideN : 64);
    const dim3 grid(tiles_m * tiles_n, batch);
    const bool alone = (size_t)grid.x * batch <= 148;
    if (wide) {
        constexpr size_t smem =
            (size_t)kShallow * (kWideM + kWideN) * kGemmLds * sizeof(double);
        return launch_gemm<k_gemm_f64_tn_wide, smem>(grid, stream, args, tiles_n);
    }
    const int split = split_k ? 1 : 0;
    constexpr size_t tn = 128 * kPipeLds * sizeof(double);          // a stage
    constexpr size_t nt = 2 * kPipeK * kNtLds * sizeof(double);
    if (ta && alone)
        return launch_gemm<k_gemm_f64_tn_pipe<3>, 3 * tn>(grid, stream, args, tiles_n, split);
    if (ta)
        return launch_gemm<k_gemm_f64_tn_pipe<2>, 2 * tn>(grid, stream, args, tiles_n, split);
    if (alone)
        return launch_gemm<k_gemm_f64_nt_pipe<3>, 3 * nt>(grid, stream, args, tiles_n, split);
    return launch_gemm<k_gemm_f64_nt_pipe<2>, 2 * nt>(grid, stream, args, tiles_n, split);
}

}  // namespace b200
