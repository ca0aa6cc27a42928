// Diagonal-block Cholesky and triangular inverse in shared memory (FP64).
//
// Replaces the per-tile potrf task (LAPACKE_dpotrf2 'L',
// core/src/cpu/adapter_cblas_fp64.cpp:14-22; cusolverDnXpotrf,
// core/src/gpu/adapter_cublas.cu:9-79).  One CTA of 16 warps factors a
// bs x bs (bs <= 128) diagonal block and inverts the factor, which turns every
// later triangular solve against this block (panel trsm, trsv, variance solve)
// into a GEMM; a block smaller than 128 is padded with the identity, so every
// loop below has a fixed trip count.
//
// The launch sits on the serial chain of every factorisation (n / 128 of them,
// one after another), and half of it is its own chain: 128 pivots, each
// the reciprocal of the pivot before it, a product and a shuffle.  So the
// chain runs alone on warp 0 and everything else beside it, in 32-wide
// sub-blocks s = 0..3:
//   warp 0      eliminates the 32 x 32 diagonal sub-block in registers (lane i
//               holds row i) without square roots, A = L~ D L~^T: the chain
//               needs one reciprocal per pivot instead of a reciprocal square
//               root and a scaling, and a pivot column is in shared memory
//               before its reciprocal is known;
//   warp 4      follows the pivots a group behind and forms X_s = L_ss^-1 =
//               D^-1/2 L~^-1 (lane c solves L~ x = e_c; the column of L~ D it
//               needs is the one warp 0 broadcast), done right after the last
//               pivot;
//   all warps   then only what the next chain waits for: the panel rows of
//               sub-block s+1, P = A X_s^T, and its diagonal A -= P P^T;
//   the others  beside the next chain, the rest of step s: the panel rows
//               below, the trailing update, the write-out of L's rows, and
//               row block s of the inverse,
//               Linv_s,<s = -X_s T_s, T_s = L_s,<s Linv_<s,  Linv_ss = X_s,
//               stored to memory from the accumulators, then T_s+1.
// After the last chain only Linv_3,<3 = -X_3 T_3 is left.  All products run on
// the FP64 tensor cores (mma.sync m16n8k8 f64).
// Measured per launch inside the pipelines: 21.3 us FP64, 25.1 us FP32 (43.1
// and 44.5 with square roots in the chain, the inverse of each sub-block after
// it and one barrier per phase).  By clock64() in a copy of the FP64 kernel, 39,900
// cycles: loads 2,200; four windows of 5,100, 7,200, 7,300 and 7,900; 2,000
// between two of them; 1,200 and the last stores, 3,200, after them.  In a window
// the 32 pivots take 4,200 cycles where nothing runs beside them (132 each, 95 of
// them latency) and 5,200 beside the products, the second half's tile 500; from the
// second window on the chain first waits 1,300 to 2,000 for the update of its
// sub-block's last tile.
// L is written back to the lower triangle only (the strict upper triangle in
// global memory is never touched, matching dpotrf2('L')).  A non-positive or
// NaN pivot is recorded in the status word (first failing global row,
// 1-based); the reference silently returns NaNs instead.
#include "common.cuh"

namespace gprat_cu
{
namespace
{

constexpr int PB = 128;                   // block size (padded)
constexpr int PS = PB + 4;                // smem row stride of the block (conflict-free fragment loads)
constexpr int SB = 32;                    // sub-block width
constexpr int XS = SB + 4;                // smem row stride of a sub-block inverse
constexpr int TS = 3 * SB + 4;            // smem row stride of the assembly temporary
constexpr int HB = SB / 2;                // pivots eliminated in registers at a time
constexpr int US = SB + 4;                // smem stride of a pivot column (conflict-free fragment loads)
constexpr int PTHREADS = 512;
constexpr int NWARPS = PTHREADS / 32;
// A warp's scheduler, with its FP64 pipe, is warp % 4: scheduler 0 runs the
// chain (warp 0), the inverse that follows it (warp 4) and the data movers
// (warps 8, 12), the other three the products: a product holds the pipe for 64
// cycles, a link of the chain for 2, so neither serial part shares a scheduler
// with them.
constexpr int CHASE_WARP = 4;
constexpr int MMA_WARPS = 12;
constexpr int MOVE_WARPS = 2;
constexpr int SIDE_WARPS = MMA_WARPS + MOVE_WARPS;
constexpr size_t SMEM_DOUBLES = PB * PS + 4 * SB * XS + SB * TS + 2 * SB * US + 3 * PB;
static_assert(SMEM_DOUBLES * sizeof(double) <= 227 * 1024, "shared memory of the diagonal-block kernel");

__device__ __forceinline__ void dmma(double (&c)[4], const double (&a)[4], const double (&b)[2])
{
    asm(
        "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// Fragment loads from row-major shared matrices (g = lane / 4, t = lane % 4).
// A: rows m0.., k-columns k0..
__device__ __forceinline__ void frag_a(double (&a)[4], const double *M, int ld, int m0, int k0, int g, int t)
{
    a[0] = M[(m0 + g) * ld + k0 + t];
    a[1] = M[(m0 + g + 8) * ld + k0 + t];
    a[2] = M[(m0 + g) * ld + k0 + t + 4];
    a[3] = M[(m0 + g + 8) * ld + k0 + t + 4];
}
// B = M^T with M row-major (N x K): B[k][n] = M[n][k]
__device__ __forceinline__ void frag_bt(double (&b)[2], const double *M, int ld, int n0, int k0, int g, int t)
{
    b[0] = M[(n0 + g) * ld + k0 + t];
    b[1] = M[(n0 + g) * ld + k0 + t + 4];
}
// B row-major (K x N)
__device__ __forceinline__ void frag_b(double (&b)[2], const double *M, int ld, int n0, int k0, int g, int t)
{
    b[0] = M[(k0 + t) * ld + n0 + g];
    b[1] = M[(k0 + t + 4) * ld + n0 + g];
}

// Stores a 16 x 8 accumulator tile at (m0, n0) of a row-major shared matrix.
__device__ __forceinline__ void store_tile(double *M, int ld, int m0, int n0, const double (&c)[4], int g, int t)
{
    *reinterpret_cast<double2 *>(M + (m0 + g) * ld + n0 + 2 * t) = make_double2(c[0], c[1]);
    *reinterpret_cast<double2 *>(M + (m0 + g + 8) * ld + n0 + 2 * t) = make_double2(c[2], c[3]);
}

// Barrier over the nthreads threads that name it (id 0 is __syncthreads), and
// its arrival without waiting (the producer's half).
__device__ __forceinline__ void bar_sync(int id, int nthreads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int nthreads)
{
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
constexpr int SIDE_BAR = 1;   // the warps beside the chain
constexpr int HALF_BAR = 2;   // a product warp -> warp 0: the sub-block's last 16 x 16 tile
constexpr int GROUP_BAR = 3;  // warp 0 -> warp 4, one barrier per pivot group

// The pivots warp 4 waits for at once: groups end after these many.  Short
// groups at the end, so that warp 4 finishes one pivot behind warp 0.
constexpr int GROUPS = 6;
__device__ __forceinline__ constexpr int group_end(int q)
{
    constexpr int ends[GROUPS] = { 8, 16, 24, 28, 30, 31 };
    return ends[q];
}

// The reciprocal of a pivot, in the two parts the chain uses at different times.
// With an approximation y of 1 / d and e = 1 - d y, 1 / d = y / (1 - e) = y (1 +
// e + e^2 + ..): the geometric series cut off after e^2, which is Householder's
// third-order iteration for 1 / x - d = 0 (A. S. Householder, The Numerical
// Treatment of a Single Nonlinear Equation, 1970).  What is cut off is e^3 of the
// result.  y is the hardware's approximation; measured over 97,600 values from
// 2^-1022 to 2^502, |e| is at most 2^-19.99, so that less than 2^-59 of the result
// is cut off, and 1 in 16 of the results differs from CUDA's 1 / d, by one unit in
// the last place.  With that division in the chain a block takes 0.3 to 0.6 us more
// (fit and predict at n = 1024 302 instead of 297 us).
__device__ __forceinline__ double rcp_seed(double d)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    return y;
}
// e + e^2, so that 1 / d = y + y (e + e^2)
__device__ __forceinline__ double rcp_series(double d, double y)
{
    const double e = fma(-d, y, 1.0);
    return fma(e, e, e);
}

// The chain wants pivots and their reciprocals to be normal numbers.  A block
// whose largest diagonal entry, which bounds its pivots, is not within 2^+-RANGE is
// therefore factored as 4^shift A, an exact multiple that brings that entry to [1,
// 4): L = 2^-shift L', L^-1 = 2^shift L'^-1.  A pivot below 2^-1022 (1e-157 of
// that entry or less) is reported like a non-positive one.  A block with an
// infinity or a NaN on its diagonal, or nothing positive, has no such entry and
// is eliminated with divisions.
constexpr int RANGE = 500;
constexpr double MIN_PIVOT = 2.2250738585072014e-308;  // 2^-1022

// By the high word of the largest diagonal entry (0: nothing positive).
__device__ __forceinline__ bool no_range(int top) { return top == 0 || top == 0x7ff00000; }
__device__ __forceinline__ int range_shift(int top)
{
    const int e = (top >> 20) - 1023;
    return no_range(top) || (e >= -RANGE && e < RANGE) ? 0 : -(e >> 1);
}

// v 2^e, |e| <= 512
__device__ __forceinline__ double times_pow2(double v, int e)
{
    return e == 0 ? v : v * __hiloint2double((1023 + e) << 20, 0);
}

// Warp 0: A = L~ D L~^T of the 32 x 32 sub-block at (c0, c0), lane i holding row
// i, 16 columns at a time; the last 16 x 16 tile is updated with the first 16
// pivots on the tensor cores (in registers it would double the chain's
// instructions, which is what the shared loads of a 32-column step cost:
// measured 143 against 95 cycles per pivot).  Leaves for warp 4 and the
// write-out: u[j][i] = (L~ D)_ij (column j as it stood when it became the
// pivot column), the pivots d and their reciprocals.  Fully unrolled, so every
// register index is a compile-time constant, and branch-free: a lane's entries
// above the diagonal receive values that are never read, which keeps the warp
// converged.
// The chain from pivot to pivot, d' = a - u^2 / d on lane j+1 and a shuffle:
// with 1 / d = y + y (e + e^2), d' = (a - u^2 y) - (u^2 y)(e + e^2), whose
// operands but the last are ready one step earlier (u^2 y as (u y) u: u^2 may
// underflow where u^2 / d does not).  FAST false: divisions.
template <bool FAST>
__device__ __forceinline__ void pivot_chain(double *a, int c0, double *u, double *piv, double *pinv)
{
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
        if (h == 1)
        {
            // the last 16 x 16 tile: A22 -= (U21 D^-1) U21^T
            double *c = a + (c0 + HB + g) * PS + c0 + HB + 2 * t;
            double af[2][4], bf[2][2][2], cf[2][4];
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
            {
                const double *k0 = u + (8 * kk + t) * US + HB, *k1 = k0 + 4 * US;
                const double p0 = pinv[8 * kk + t], p1 = pinv[8 * kk + t + 4];
                af[kk][0] = -k0[g] * p0;
                af[kk][1] = -k0[g + 8] * p0;
                af[kk][2] = -k1[g] * p1;
                af[kk][3] = -k1[g + 8] * p1;
#pragma unroll
                for (int n = 0; n < 2; ++n)
                {
                    bf[kk][n][0] = k0[8 * n + g];
                    bf[kk][n][1] = k1[8 * n + g];
                }
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
            {
                cf[n][0] = c[8 * n];
                cf[n][1] = c[8 * n + 1];
                cf[n][2] = c[8 * PS + 8 * n];
                cf[n][3] = c[8 * PS + 8 * n + 1];
            }
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
            {
#pragma unroll
                for (int n = 0; n < 2; ++n)
                {
                    dmma(cf[n], af[kk], bf[kk][n]);
                }
            }
            store_tile(a, PS, c0 + HB, c0 + HB, cf[0], g, t);
            store_tile(a, PS, c0 + HB, c0 + HB + 8, cf[1], g, t);
            __syncwarp();
        }
        double r[HB];  // r[c] = A[lane][c0 + 16 h + c]
        const double *arow = a + (c0 + lane) * PS + c0 + h * HB;
#pragma unroll
        for (int c = 0; c < HB; ++c)
        {
            r[c] = (h * HB + c <= lane) ? arow[c] : 0.0;
        }
        double d = __shfl_sync(0xffffffffu, r[0], h * HB);  // the current pivot
#pragma unroll
        for (int jj = 0; jj < HB; ++jj)
        {
            const int j = h * HB + jj;
            double *cb = u + j * US;
            cb[lane] = r[jj];
            const double y = FAST ? rcp_seed(d) : 1.0 / d;
            double dinv = y, dnext = 0.0;
            if (FAST)
            {
                const double ee = rcp_series(d, y);
                dinv = fma(y, ee, y);
                if (jj + 1 < HB)
                {
                    const double w = r[jj] * y;
                    dnext = fma(-(w * r[jj]), ee, fma(-w, r[jj], r[jj + 1]));
                }
            }
            else if (jj + 1 < HB)
            {
                dnext = fma(-r[jj] * y, r[jj], r[jj + 1]);
            }
            if (lane == 0)
            {
                piv[j] = d;
                pinv[j] = dinv;
            }
#pragma unroll
            for (int q = 0; q < GROUPS; ++q)
            {
                if (group_end(q) == j + 1)
                {
                    bar_arrive(GROUP_BAR + q, 64);
                }
            }
            if (jj + 1 < HB)
            {
                d = __shfl_sync(0xffffffffu, dnext, j + 1);
                const double w = r[jj] * dinv;  // L~[lane][j]
                __syncwarp();
                int c = jj + 1;
                if (c & 1)
                {
                    r[c] = fma(-w, cb[h * HB + c], r[c]);
                    ++c;
                }
#pragma unroll
                for (; c < HB; c += 2)
                {
                    const double2 v = *reinterpret_cast<const double2 *>(cb + h * HB + c);
                    r[c] = fma(-w, v.x, r[c]);
                    r[c + 1] = fma(-w, v.y, r[c + 1]);
                }
            }
        }
        __syncwarp();
    }
}

// Warp 4: X~ = L~^-1 (zero above the diagonal) of the sub-block warp 0 is
// eliminating, lane c column c, 16 rows at a time (the first half's part in the
// second half's rows on the tensor cores).  L^-1 = D^-1/2 X~: its readers scale
// the rows.  Waits for a group of pivots at a time.
__device__ __forceinline__ void chase_inverse(const double *u, const double *pinv, double *xinv)
{
    const int lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
        double x[HB];
        if (h == 0)
        {
#pragma unroll
            for (int i = 0; i < HB; ++i)
            {
                x[i] = (i == lane) ? 1.0 : 0.0;
            }
        }
        else
        {
            // rows 16 .. 31 of columns 0 .. 15: the first half's share,
            // -L~21 X~11 (L~_ij = u_ij / d_j), through their place in xinv
            __syncwarp();
            double cf[2][4] = {};
#pragma unroll
            for (int kk = 0; kk < 2; ++kk)
            {
                const double *k0 = u + (8 * kk + t) * US + HB, *k1 = k0 + 4 * US;
                const double p0 = -pinv[8 * kk + t], p1 = -pinv[8 * kk + t + 4];
                const double af[4] = { k0[g] * p0, k0[g + 8] * p0, k1[g] * p1, k1[g + 8] * p1 };
#pragma unroll
                for (int n = 0; n < 2; ++n)
                {
                    double bf[2];
                    frag_b(bf, xinv, XS, 8 * n, 8 * kk, g, t);
                    dmma(cf[n], af, bf);
                }
            }
            store_tile(xinv, XS, HB, 0, cf[0], g, t);
            store_tile(xinv, XS, HB, 8, cf[1], g, t);
            __syncwarp();
#pragma unroll
            for (int i = 0; i < HB; ++i)
            {
                x[i] = (lane < HB) ? xinv[(HB + i) * XS + lane] : (HB + i == lane ? 1.0 : 0.0);
            }
        }
#pragma unroll
        for (int jj = 0; jj < HB; ++jj)
        {
            const int j = h * HB + jj;
#pragma unroll
            for (int q = 0; q < GROUPS; ++q)
            {
                if ((q == 0 ? 0 : group_end(q - 1)) == j)  // (the last pivot's own column is not needed)
                {
                    bar_sync(GROUP_BAR + q, 64);
                }
            }
            const double *cb = u + j * US + h * HB;
            xinv[j * XS + lane] = x[jj];
            if (jj + 1 < HB)
            {
                const double w = x[jj] * pinv[j];
                int c = jj + 1;
                if (c & 1)
                {
                    x[c] = fma(-w, cb[c], x[c]);
                    ++c;
                }
#pragma unroll
                for (; c < HB; c += 2)
                {
                    const double2 v = *reinterpret_cast<const double2 *>(cb + c);
                    x[c] = fma(-w, v.x, x[c]);
                    x[c + 1] = fma(-w, v.y, x[c + 1]);
                }
            }
        }
    }
}

__device__ __forceinline__ void cp_async16_zfill(void *smem, const void *gmem, int bytes)
{
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(gmem), "r"(bytes) : "memory");
}

// True when the block and its rows start on 16-byte boundaries.
template <typename T>
__device__ __forceinline__ bool aligned16(const T *A, int64_t lda)
{
    return ((reinterpret_cast<uintptr_t>(A) | static_cast<uintptr_t>(lda * sizeof(T))) & 15) == 0;
}

// Rows [R_LO, R_HI) of the block's lower triangle into shared memory, all
// threads.  Nothing right of the block's diagonal is read; shared words right
// of it may receive zeros and are never read as part of L.  FP64 blocks on
// 16-byte boundaries: cp.async (the caller waits); everything else (FP32 is
// widened): plain loads, those of eight rows issued before the first is used.
template <int R_LO, int R_HI, typename T>
__device__ __forceinline__ void load_rows(const T *A, int64_t lda, bool al, int bs, double *sa)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int ROWS = (R_HI - R_LO) / NWARPS;  // per warp
    if (sizeof(T) == 8 && al)
    {
#pragma unroll
        for (int k = 0; k < ROWS; ++k)
        {
            const int i = R_LO + NWARPS * k + warp;
#pragma unroll
            for (int c0 = 0; c0 < R_LO + NWARPS * (k + 1); c0 += 64)
            {
                const int c = c0 + 2 * lane;
                if (c <= i && i < bs)
                {
                    cp_async16_zfill(sa + i * PS + c, A + static_cast<int64_t>(i) * lda + c, min(2, i + 1 - c) * 8);
                }
            }
        }
    }
    else
    {
#pragma unroll
        for (int k0 = 0; k0 < ROWS; k0 += 8)
        {
            T v[8][4];
#pragma unroll
            for (int q = 0; q < 8 && k0 + q < ROWS; ++q)
            {
                const int i = R_LO + NWARPS * (k0 + q) + warp;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    const int c = lane + 32 * k;
                    v[q][k] = (c <= i && i < bs) ? A[static_cast<int64_t>(i) * lda + c] : T(0);
                }
            }
#pragma unroll
            for (int q = 0; q < 8 && k0 + q < ROWS; ++q)
            {
                const int i = R_LO + NWARPS * (k0 + q) + warp;
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    sa[i * PS + lane + 32 * k] = static_cast<double>(v[q][k]);
                }
            }
        }
    }
    // identity rows below a block smaller than 128
    for (int i = max(R_LO, bs); i < R_HI; ++i)
    {
        if ((i & (NWARPS - 1)) == warp)
        {
            for (int c = lane; c <= i; c += 32)
            {
                sa[i * PS + c] = (i == c) ? 1.0 : 0.0;
            }
        }
    }
}

// One element pair (i, c), (i, c + 1) of an output matrix, c even: columns
// <= c_last are stored, as a pair where `pair` allows it.
template <typename T>
struct PairOf;
template <>
struct PairOf<double>
{
    using type = double2;
};
template <>
struct PairOf<float>
{
    using type = float2;
};
template <typename T>
__device__ __forceinline__ void store_pair(T *M, int64_t ld, int i, int c, int c_last, bool pair, double v0, double v1)
{
    using Pair = typename PairOf<T>::type;
    T *dst = M + static_cast<int64_t>(i) * ld + c;
    if (pair && c + 1 <= c_last)
    {
        Pair w;
        w.x = static_cast<T>(v0);
        w.y = static_cast<T>(v1);
        *reinterpret_cast<Pair *>(dst) = w;
        return;
    }
    if (c <= c_last)
    {
        dst[0] = static_cast<T>(v0);
    }
    if (c + 1 <= c_last)
    {
        dst[1] = static_cast<T>(v1);
    }
}

// Where the inverse goes: FP64 and / or FP32 (either may be null), rows and
// columns < bs.
struct InverseOut
{
    double *f64;
    int64_t ld64;
    float *f32;
    int64_t ld32;
    int bs;
    __device__ __forceinline__ void pair(int i, int c, double v0, double v1) const
    {
        if (i >= bs || c >= bs)
        {
            return;
        }
        if (f64 != nullptr)
        {
            store_pair(f64, ld64, i, c, bs - 1, true, v0, v1);
        }
        if (f32 != nullptr)
        {
            store_pair(f32, ld32, i, c, bs - 1, true, v0, v1);
        }
    }
};

// Row block s of the inverse left of its diagonal block: -X_s T_s (X_s = D^-1/2 X~_s), 16 x 16
// tiles over nwarps warps (this one is number w), to memory and, when
// keep, into sa in place of L_s,<s.
__device__ __forceinline__ void inverse_row_block(const InverseOut &out, double *sa, bool keep, const double *xs, const double *rsq,
                                                  const double *tbuf, int s, int w, int nwarps, int g, int t)
{
    const int c0 = s * SB;
    for (int tile = w; tile < 4 * s; tile += nwarps)
    {
        const int mi = tile / (2 * s), n0 = 16 * (tile % (2 * s));
        double cf[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
        {
            if (kk <= 2 * mi + 1)  // X is lower triangular
            {
                double af[4];
                frag_a(af, xs, XS, 16 * mi, 8 * kk, g, t);
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    double bf[2];
                    frag_b(bf, tbuf, TS, n0 + 8 * h, 8 * kk, g, t);
                    dmma(cf[h], af, bf);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
#pragma unroll
            for (int e = 0; e < 4; ++e)
            {
                cf[h][e] *= -rsq[c0 + 16 * mi + g + (e >> 1) * 8];
            }
            const int i = c0 + 16 * mi + g, c = n0 + 8 * h + 2 * t;
            out.pair(i, c, cf[h][0], cf[h][1]);
            out.pair(i + 8, c, cf[h][2], cf[h][3]);
            if (keep)
            {
                store_tile(sa, PS, c0 + 16 * mi, n0 + 8 * h, cf[h], g, t);
            }
        }
    }
}

// A -= P P^T on the 16 x 16 tile at (m0, n0), P the 32 columns from p0.
__device__ __forceinline__ void trailing_tile(double *sa, int m0, int n0, int p0, int g, int t)
{
    double cf[2][4] = {};
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
    {
        double af[4];
        frag_a(af, sa, PS, m0, p0 + 8 * kk, g, t);
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            double bf[2];
            frag_bt(bf, sa, PS, n0 + 8 * h, p0 + 8 * kk, g, t);
            dmma(cf[h], af, bf);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
    {
        const double *c = sa + (m0 + g) * PS + n0 + 8 * h + 2 * t;
        const double2 v0 = *reinterpret_cast<const double2 *>(c);
        const double2 v1 = *reinterpret_cast<const double2 *>(c + 8 * PS);
        const double tile[4] = { v0.x - cf[h][0], v0.y - cf[h][1], v1.x - cf[h][2], v1.y - cf[h][3] };
        store_tile(sa, PS, m0, n0 + 8 * h, tile, g, t);
    }
}

// T_s = L_s,<s Linv_<s  (32 x 32 s; Linv lower triangular: k >= n), 16 x 16
// tiles, those with the most products first.
__device__ __forceinline__ void inverse_temporary(double *tbuf, const double *sa, int s, int w, int nwarps, int g,
                                                  int t)
{
    for (int tile = w; tile < 4 * s; tile += nwarps)
    {
        const int mi = tile & 1, p = tile >> 1;
        double cf[2][4] = {};
#pragma unroll 2
        for (int kk = 2 * p; kk < 4 * s; ++kk)
        {
            double af[4];
            frag_a(af, sa, PS, s * SB + 16 * mi, 8 * kk, g, t);
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                double bf[2];
                frag_b(bf, sa, PS, 16 * p + 8 * h, 8 * kk, g, t);
                dmma(cf[h], af, bf);
            }
        }
        store_tile(tbuf, TS, 16 * mi, 16 * p, cf[0], g, t);
        store_tile(tbuf, TS, 16 * mi, 16 * p + 8, cf[1], g, t);
    }
}

// T: element type of the block in global memory (FP64, or FP32 for the
// mixed path, which then also receives Linv in FP32 and the FP64 diagonal of L).
template <typename T>
__global__ void __launch_bounds__(PTHREADS, 1) potrf_inv_kernel(T *A, int64_t lda, int bs, int row0, double *Linv,
                                                                int64_t ldi, float *Linv32, int64_t ldi32,
                                                                double *__restrict__ diag_out,
                                                                DeviceStatus *__restrict__ status, int write_l)
{
    extern __shared__ __align__(16) double sa[];  // [PB][PS]
    double *xall = sa + PB * PS;         // 4 x [SB][XS] sub-block inverses
    double *tbuf = xall + 4 * SB * XS;   // [SB][TS]
    double *ubuf = tbuf + SB * TS;       // 2 x [SB][US] pivot columns, alternating by sub-block
    double *piv = ubuf + 2 * SB * US;    // [PB] pivots
    double *pinv = piv + PB;             // [PB] their reciprocals
    double *rsq = pinv + PB;             // [PB] their reciprocal square roots (from the step after the pivots' on)
    __shared__ int bad;
    __shared__ int top_of[PB / 32];
    const int tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const bool mover = warp > CHASE_WARP && (warp & 3) == 0;
    const int mma_w = warp - 1 - (warp >> 2);                         // number among the product warps
    const int move_w = (warp >> 2) - 2, move_t = 32 * move_w + lane;  // among the data movers
    if (tid == 0)
    {
        bad = 0;
    }
    pdl_wait();  // the previous kernel's results are visible from here on
    const bool al = aligned16(A, lda);
    const double diag = tid < bs ? static_cast<double>(A[tid * (lda + 1)]) : 0.0;
    // the first sub-block's rows ahead of the rest: its chain starts on them
    load_rows<0, SB>(A, lda, al, bs, sa);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    load_rows<SB, PB>(A, lda, al, bs, sa);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 1;\n" ::: "memory");
    if (warp < PB / 32)
    {
        // the high words of positive numbers are in the numbers' order
        const int hi = __double2hiint(diag);
        const int key = (hi & 0x7ff00000) == 0x7ff00000 ? 0x7ff00000 : diag > 0.0 ? max(hi, 1) : 0;
        const int top = __reduce_max_sync(0xffffffffu, key);
        if (lane == 0)
        {
            top_of[warp] = top;
        }
    }
    __syncthreads();
    // (read again where it is needed: the chain leaves no registers to keep it in)
    auto top = [&]() { return max(max(top_of[0], top_of[1]), max(top_of[2], top_of[3])); };
    // (an FP32 block's numbers are in range)
    if (const int shift = sizeof(T) == 8 ? range_shift(top()) : 0; shift != 0)
    {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        for (int i = warp; i < bs; i += NWARPS)
        {
            for (int c = lane; c <= i; c += 32)
            {
                sa[i * PS + c] = times_pow2(times_pow2(sa[i * PS + c], shift), shift);
            }
        }
        __syncthreads();
    }
    const InverseOut out{ Linv, ldi, Linv32, ldi32, bs };

    // L's sub-block s (its columns u scaled by 1 / sqrt(d)) and diagonal, to
    // memory, by this thread as number me of count
    auto write_diag = [&](int s, int me, int count)
    {
        const double *u = ubuf + (s & 1) * SB * US;
        const int c0 = s * SB;
        for (int q = me; write_l && q < SB * SB / 2; q += count)
        {
            const int i = q >> 4, c = 2 * (q & 15);
            if (c <= i && c0 + i < bs)
            {
                store_pair(A, lda, c0 + i, c0 + c, c0 + i, al, u[c * US + i] * rsq[c0 + c],
                           u[(c + 1) * US + i] * rsq[c0 + c + 1]);
            }
        }
        for (int j = me; diag_out != nullptr && j < SB; j += count)
        {
            if (c0 + j < bs)
            {
                diag_out[c0 + j] = piv[c0 + j] * rsq[c0 + j];
            }
        }
    };
    // one warp: 1 / sqrt of sub-block s's pivots, and the first that is not positive
    auto finish_pivots = [&](int s)
    {
        const double d = piv[s * SB + lane];
        rsq[s * SB + lane] = rsqrt(d);
        const unsigned wrong = __ballot_sync(0xffffffffu, !(no_range(top()) ? d > 0.0 : d >= MIN_PIVOT) && s * SB + lane < bs);
        if (lane == 0 && wrong != 0 && bad == 0)
        {
            bad = row0 + s * SB + __ffs(wrong);
        }
    };
    // the inverse's diagonal block s, to memory and (keep) into sa
    auto write_xs = [&](int s, bool keep, int me, int count)
    {
        const double *xs = xall + s * SB * XS;
        const int c0 = s * SB;
        for (int q = me; q < SB * SB / 2; q += count)
        {
            const int i = q >> 4, c = 2 * (q & 15);
            double2 v = *reinterpret_cast<const double2 *>(xs + i * XS + c);
            v.x *= rsq[c0 + i];
            v.y *= rsq[c0 + i];
            out.pair(c0 + i, c0 + c, v.x, v.y);
            if (keep)
            {
                *reinterpret_cast<double2 *>(sa + (c0 + i) * PS + c0 + c) = v;
            }
        }
    };

#pragma unroll 1
    for (int s = 0; s < 4; ++s)
    {
        const int c0 = s * SB;
        const double *xs = xall + s * SB * XS;
        double *u = ubuf + (s & 1) * SB * US;
        if (warp == 0)
        {
            if (s > 0)
            {
                bar_sync(HALF_BAR, 64);  // the sub-block's last 16 x 16 tile is updated
            }
            if (!no_range(top()))
            {
                pivot_chain<true>(sa, c0, u, piv + c0, pinv + c0);
            }
            else
            {
                pivot_chain<false>(sa, c0, u, piv + c0, pinv + c0);
            }
        }
        else if (warp == CHASE_WARP)
        {
            chase_inverse(u, pinv + c0, xall + s * SB * XS);
        }
        else if (s == 0)
        {
            // zeros above the inverse's diagonal blocks
            for (int i = mover ? MMA_WARPS + move_w : mma_w; i < 3 * SB; i += SIDE_WARPS)
            {
                for (int c = (i / SB + 1) * SB + 2 * lane; c < PB; c += 64)
                {
                    out.pair(i, c, 0.0, 0.0);
                }
            }
        }
        else if (mover)
        {
            write_xs(s - 1, true, move_t, 32 * MOVE_WARPS);
            bar_sync(SIDE_BAR, 32 * SIDE_WARPS);
            // L's rows of sub-block s left of its diagonal
            if (write_l)
            {
#pragma unroll 4
                for (int i = c0 + move_w; i < c0 + SB; i += MOVE_WARPS)
                {
#pragma unroll
                    for (int c = 2 * lane; c < 3 * SB; c += 64)
                    {
                        if (i < bs && c < c0)
                        {
                            const double2 v = *reinterpret_cast<const double2 *>(sa + i * PS + c);
                            store_pair(A, lda, i, c, c0 - 1, al, v.x, v.y);
                        }
                    }
                }
            }
        }
        else
        {
            // the rest of step s - 1
            const int p = s - 1, p0 = p * SB;
            const double *xp = xall + p * SB * XS;
            const int b0 = c0 + SB;  // first row below the chain's sub-block
            if (mma_w == 0)
            {
                trailing_tile(sa, c0 + HB, c0 + HB, p0, g, t);
                bar_arrive(HALF_BAR, 64);
            }
            // panel rows b0 ..: P = A X_p^T, in place, a warp takes 16 rows
            for (int m0 = b0 + 16 * (mma_w - 1); m0 < PB && mma_w > 0; m0 += 16 * MMA_WARPS)
            {
                double af[4][4];
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                {
                    frag_a(af[kk], sa, PS, m0, p0 + 8 * kk, g, t);
                }
                __syncwarp();
#pragma unroll
                for (int nt = 0; nt < 4; ++nt)
                {
                    double cf[4] = { 0.0, 0.0, 0.0, 0.0 };
#pragma unroll
                    for (int kk = 0; kk <= nt; ++kk)  // X^T is zero where k > n
                    {
                        double bf[2];
                        frag_bt(bf, xp, XS, 8 * nt, 8 * kk, g, t);
                        dmma(cf, af[kk], bf);
                    }
                    const double r0 = rsq[p0 + 8 * nt + 2 * t], r1 = rsq[p0 + 8 * nt + 2 * t + 1];
                    cf[0] *= r0;
                    cf[1] *= r1;
                    cf[2] *= r0;
                    cf[3] *= r1;
                    store_tile(sa, PS, m0, p0 + 8 * nt, cf, g, t);
                }
            }
            // row block p of the inverse, from the warps without panel rows on (5, 6, ..)
            inverse_row_block(out, sa, true, xp, rsq, tbuf, p, (mma_w + MMA_WARPS - 5) % MMA_WARPS, MMA_WARPS, g, t);
            bar_sync(SIDE_BAR, 32 * SIDE_WARPS);
            // trailing update A -= P P^T of rows b0 .., columns c0 .. up to the diagonal, 16 x 16 tiles
            const int mt = (PB - b0) / 16;
            const int ntiles = mt * (mt + 5) / 2;  // sum over mi < mt of mi + 3
            for (int tile = mma_w; tile < ntiles; tile += MMA_WARPS)
            {
                int mi = 0, base = 0;
                while (base + mi + 3 <= tile)
                {
                    base += mi + 3;
                    ++mi;
                }
                const int m0 = b0 + 16 * mi, n0 = c0 + 16 * (tile - base);
                trailing_tile(sa, m0, n0, p0, g, t);
            }
            inverse_temporary(tbuf, sa, s, MMA_WARPS - 1 - mma_w, MMA_WARPS, g, t);
            write_diag(p, 32 * mma_w + lane, 32 * MMA_WARPS);
        }
        if (s == 0)
        {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        if (s == 3)
        {
            if (warp == 0)
            {
                finish_pivots(3);
            }
            __syncthreads();
            break;
        }
        // what the next chain waits for.  Panel rows of sub-block s+1: eight warps
        // take one 16 x 8 tile each (every scheduler the same number of products:
        // X^T is zero where k > n); all read before any writes.
        const int c1 = c0 + SB;
        const int mi = warp >> 2, nt = mi == 0 ? warp & 3 : 3 - (warp & 3);
        double af[4][4], bf[4][2], cf[4] = {};
        if (warp < 8)
        {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
            {
                if (kk <= nt)
                {
                    frag_a(af[kk], sa, PS, c1 + 16 * mi, c0 + 8 * kk, g, t);
                    frag_bt(bf[kk], xs, XS, 8 * nt, 8 * kk, g, t);
                    dmma(cf, af[kk], bf[kk]);
                }
            }
            // the scaling of X's rows, beside the products
            const double r0 = rsqrt(piv[c0 + 8 * nt + 2 * t]), r1 = rsqrt(piv[c0 + 8 * nt + 2 * t + 1]);
            cf[0] *= r0;
            cf[1] *= r1;
            cf[2] *= r0;
            cf[3] *= r1;
        }
        else if (warp == 8)
        {
            finish_pivots(s);
        }
        __syncthreads();
        if (warp < 8)
        {
            store_tile(sa, PS, c1 + 16 * mi, c0 + 8 * nt, cf, g, t);
        }
        __syncthreads();
        // the first 16 columns of its diagonal sub-block, one 16 x 8 tile per scheduler
        if (warp < 4)
        {
            const int m0 = c1 + 16 * (warp >> 1), n0 = c1 + 8 * (warp & 1);
            double ct[4] = {};
            const double *c = sa + (m0 + g) * PS + n0 + 2 * t;
            const double2 v0 = *reinterpret_cast<const double2 *>(c);
            const double2 v1 = *reinterpret_cast<const double2 *>(c + 8 * PS);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
            {
                frag_a(af[kk], sa, PS, m0, c0 + 8 * kk, g, t);
                frag_bt(bf[kk], sa, PS, n0, c0 + 8 * kk, g, t);
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
            {
                dmma(ct, af[kk], bf[kk]);
            }
            const double tile[4] = { v0.x - ct[0], v0.y - ct[1], v1.x - ct[2], v1.y - ct[3] };
            store_tile(sa, PS, m0, n0, tile, g, t);
        }
        __syncthreads();
    }
    pdl_launch_dependents();  // little more than the stores is left
    if (tid == 0 && bad != 0 && status != nullptr)
    {
        atomicCAS(&status->not_spd_row, 0, bad);
    }
    inverse_row_block(out, sa, false, xall + 3 * SB * XS, rsq, tbuf, 3, warp, NWARPS, g, t);
    write_xs(3, false, tid, PTHREADS);
    write_diag(3, tid, PTHREADS);
    if (const int shift = sizeof(T) == 8 ? range_shift(top()) : 0; shift != 0)
    {
        // (rare) what has been written, L' and its inverse, to the block's own scale
        __syncthreads();
        for (int i = warp; i < bs; i += NWARPS)
        {
            for (int c = lane; c <= i; c += 32)
            {
                if (write_l)
                {
                    T &l = A[static_cast<int64_t>(i) * lda + c];
                    l = static_cast<T>(times_pow2(static_cast<double>(l), -shift));
                }
                if (Linv != nullptr)
                {
                    double &x = Linv[static_cast<int64_t>(i) * ldi + c];
                    x = times_pow2(x, shift);
                }
            }
        }
    }
}

__global__ void reciprocal_kernel(const double *__restrict__ d, int n, double *__restrict__ seed,
                                  double *__restrict__ inv, double *__restrict__ quotient)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
    {
        const double y = rcp_seed(d[i]);
        seed[i] = y;
        inv[i] = fma(y, rcp_series(d[i], y), y);
        quotient[i] = 1.0 / d[i];
    }
}

}  // namespace

void pivot_reciprocals(const double *d, int n, double *seed, double *inv, double *quotient, cudaStream_t s)
{
    reciprocal_kernel<<<ceil_div(n, 256), 256, 0, s>>>(d, n, seed, inv, quotient);
    GPRAT_LAUNCH_CHECK();
}

void potrf_diag(double *A, int64_t lda, int bs, int row0, double *Linv, int64_t ldi, DeviceStatus *status,
                cudaStream_t s)
{
    if (bs <= 0 || bs > PB)
    {
        throw Error(1, "potrf_diag: block size must be in [1, 128]");
    }
    if ((ldi & 1) != 0 || (reinterpret_cast<uintptr_t>(Linv) & 15) != 0)
    {
        throw Error(1, "potrf_diag: Linv must be 16-byte aligned with an even leading dimension");
    }
    constexpr size_t smem = SMEM_DOUBLES * sizeof(double);
    ensure_smem_attr(reinterpret_cast<const void *>(potrf_inv_kernel<double>), static_cast<int>(smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(PTHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1] = { programmatic_launch_attr() };
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GPRAT_CUDA_CHECK(cudaLaunchKernelEx(&cfg, potrf_inv_kernel<double>, A, lda, bs, row0, Linv, ldi,
                                        static_cast<float *>(nullptr), int64_t{ 0 }, static_cast<double *>(nullptr),
                                        status, 1));
    GPRAT_LAUNCH_CHECK();
}

void potrf_diag_f32(float *A, int64_t lda, int bs, int row0, double *Linv, int64_t ldi, float *Linv32, int64_t ldi32,
                    double *diag, DeviceStatus *status, cudaStream_t s, bool write_l)
{
    if (bs <= 0 || bs > PB)
    {
        throw Error(1, "potrf_diag_f32: block size must be in [1, 128]");
    }
    if ((Linv != nullptr && ((ldi & 1) != 0 || (reinterpret_cast<uintptr_t>(Linv) & 15) != 0)) || (ldi32 & 1) != 0 ||
        (reinterpret_cast<uintptr_t>(Linv32) & 7) != 0)
    {
        throw Error(1, "potrf_diag_f32: Linv / Linv32 must be aligned with even leading dimensions");
    }
    constexpr size_t smem = SMEM_DOUBLES * sizeof(double);
    ensure_smem_attr(reinterpret_cast<const void *>(potrf_inv_kernel<float>), static_cast<int>(smem));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(PTHREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1] = { programmatic_launch_attr() };
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GPRAT_CUDA_CHECK(
        cudaLaunchKernelEx(&cfg, potrf_inv_kernel<float>, A, lda, bs, row0, Linv, ldi, Linv32, ldi32, diag, status,
                           write_l ? 1 : 0));
    GPRAT_LAUNCH_CHECK();
}

}  // namespace gprat_cu
