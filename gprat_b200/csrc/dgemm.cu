// FP64 products of the factorisation and of the solves on the DMMA tensor
// cores: the update C -= A B^T and the panel solve P := P Linv^T.
//
// Uses in the pipeline (reference tile tasks they replace):
//   Cholesky trailing and in-panel updates  C -= P P^T, lower only (syrk + gemm
//     tasks, core/src/cpu/tiled_algorithms.cpp:33-55), and with them, in the
//     same launch, the rows of a second matrix solved against the factor: the
//     variance solve's W (forward_solve_tiled_matrix, :117-149), the inverse's
//     identity, and y (forward_solve_tiled, :61-86)
//   Cholesky panel solve  P = P Linv_kk^T in place (trsm task, :21-32), with the
//     same further rows; row sums of squares of W
//     (symmetric_matrix_matrix_diagonal_tiled, :212-228) in its epilogue
#include "dgemm.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>

namespace gprat_cu
{
namespace gemm
{

void make_map(CUtensorMap &map, const double *base, int rows, int cols, int64_t ld, int box_rows)
{
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    static std::once_flag once;
    std::call_once(once,
                   []
                   {
                       void *p = nullptr;
                       cudaDriverEntryPointQueryResult q;
                       if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                                            &q) == cudaSuccess &&
                           q == cudaDriverEntryPointSuccess)
                       {
                           encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
                       }
                   });
    if (encode == nullptr)
    {
        throw Error(4, "cuTensorMapEncodeTiled is not available from the driver");
    }
    if ((ld & 1) || (reinterpret_cast<uintptr_t>(base) & 15))
    {
        throw Error(1, "dgemm: leading dimensions must be even and bases 16-byte aligned");
    }
    const bool grouped = grouped_map(cols);
    const cuuint64_t bytes = static_cast<cuuint64_t>(ld) * 8;
    const cuuint64_t dims[3] = { static_cast<cuuint64_t>(grouped ? KC : cols), static_cast<cuuint64_t>(rows),
                                 static_cast<cuuint64_t>(cols / KC) };
    const cuuint64_t strides[2] = { bytes, KC * 8 };
    const cuuint32_t box[3] = { KC, static_cast<cuuint32_t>(box_rows), 2 };
    const cuuint32_t elem[3] = { 1, 1, 1 };
    const CUresult r = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, grouped ? 3 : 2, const_cast<double *>(base), dims,
                              strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
    {
        throw Error(4, "cuTensorMapEncodeTiled failed with code " + std::to_string(static_cast<int>(r)));
    }
}

}  // namespace gemm

namespace
{

using namespace gemm;

// Device arguments of an update: C_a -= A_a B^T for the row groups a = 0 (the
// lower trapezoid or a full rectangle) and 1 (full), and the vector
// y -= B z.
struct UpdateParams
{
    int M[2];
    int N, K;
    double *C[2];
    int64_t ldc[2];
    bool lower;  // group 0
    int tiles0, tiles;
    const double *B;
    int64_t ldb;
    const double *z;
    double *y;
    DeviceStatus *status;
    int polls;
};

// y[c] -= B[c] . z for this warp's share of the rows of B, four at a time.
__device__ __forceinline__ void vector_update(const UpdateParams &p, int warp_id, int nwarps)
{
    const int lane = threadIdx.x & 31;
    for (int c0 = 4 * warp_id; c0 < p.N; c0 += 4 * nwarps)
    {
        double s[4] = { 0.0, 0.0, 0.0, 0.0 };
        for (int k = 2 * lane; k < p.K; k += 64)
        {
            const double z0 = p.z[k], z1 = k + 1 < p.K ? p.z[k + 1] : 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                const double2 v = *reinterpret_cast<const double2 *>(
                    p.B + static_cast<int64_t>(min(c0 + q, p.N - 1)) * p.ldb + k);
                s[q] += v.x * z0 + (k + 1 < p.K ? v.y * z1 : 0.0);
            }
        }
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                s[q] += __shfl_xor_sync(0xffffffffu, s[q], o);
            }
            if (lane == 0 && c0 + q < p.N)
            {
                p.y[c0 + q] -= s[q];
            }
        }
    }
}

// One group and one tile per CTA.  C_FIRST: the products are subtracted from C
// one after another, else summed and then subtracted (C is not needed until the
// end, and is on its way to L2 meanwhile).
template <int FM, int FN, int MIN_CTAS, bool C_FIRST>
__global__ void __launch_bounds__(GROUP_THREADS, MIN_CTAS)
    update_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                  const __grid_constant__ CUtensorMap map_b, const __grid_constant__ UpdateParams p)
{
    using T = Tile<FM, FN>;
    extern __shared__ __align__(128) double smem[];
    __shared__ RingBars bars;
    __shared__ int abort_flag;
    const int warp = threadIdx.x / 32, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int wm = warp >> 1, wn = warp & 1;
    if (threadIdx.x == 0)
    {
        abort_flag = 0;
        init_ring(bars);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tcx::fence_proxy_async_smem();
        prefetch_map(&map_a0);
        prefetch_map(&map_a1);
        prefetch_map(&map_b);
    }
    __syncthreads();
    pdl_wait();

    const int tile = blockIdx.x;
    if (tile < p.tiles)
    {
        TileJob j;
        j.k0 = 0;
        j.k1 = p.K;
        j.a = tile >= p.tiles0;
        if (j.a == 0 && p.lower)
        {
            trapezoid_tile<T::BM, T::BN>(tile, p.M[0], p.N, j.m0, j.n0);
        }
        else
        {
            const int q = tile - (j.a ? p.tiles0 : 0), nt = (p.N + T::BN - 1) / T::BN;
            j.m0 = (q / nt) * T::BM;
            j.n0 = (q % nt) * T::BN;
        }
        const Ring<FM, FN> ring{ smem, &bars, &abort_flag, j.a ? &map_a1 : &map_a0, &map_b, grouped_map(p.K),
                                 p.polls, j };
        ring.begin();
        __syncwarp();
        const int M = p.M[j.a];
        const int64_t ldc = p.ldc[j.a];
        const int row = j.m0 + wm * 16 * FM + g, col = j.n0 + wn * 8 * FN + 2 * t;
        double *C = p.C[j.a] + static_cast<int64_t>(row) * ldc + col;
        // tiles inside the matrix and clear of the diagonal need no tests
        const bool inside = j.m0 + T::BM <= M && j.n0 + T::BN <= p.N;
        const bool plain = inside && !(j.a == 0 && p.lower && j.n0 + T::BN > j.m0 + 1);
        double acc[FM][FN][4] = {};
        if (C_FIRST)
        {
#pragma unroll
            for (int mi = 0; mi < FM; ++mi)
            {
#pragma unroll
                for (int ni = 0; ni < FN; ++ni)
                {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                    {
                        const int r = row + 16 * mi + 8 * (e >> 1), c = col + 8 * ni + (e & 1);
                        acc[mi][ni][e] = r < M && c < p.N ? -p.C[j.a][static_cast<int64_t>(r) * ldc + c] : 0.0;
                    }
                }
            }
        }
        else
        {
            // C's tile towards L2 while the products run
            constexpr int LINES = T::BN / 16;  // 128-byte lines per row
            for (int q = threadIdx.x; q < T::BM * LINES; q += GROUP_THREADS)
            {
                const int r = j.m0 + q / LINES, c = j.n0 + 16 * (q % LINES);
                if (r < M && c < p.N)
                {
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(p.C[j.a] + static_cast<int64_t>(r) * ldc + c));
                }
            }
        }
        ring.run(acc, wm * 16 * FM + g, wn * 8 * FN + g, t);
        pdl_launch_dependents();  // C's read-modify-write is left
        if (plain && !C_FIRST)
        {
#pragma unroll
            for (int mi = 0; mi < FM; ++mi)
            {
                double2 v[2][FN];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
#pragma unroll
                    for (int ni = 0; ni < FN; ++ni)
                    {
                        v[h][ni] = *reinterpret_cast<const double2 *>(C + static_cast<int64_t>(16 * mi + 8 * h) * ldc +
                                                                      8 * ni);
                    }
                }
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
#pragma unroll
                    for (int ni = 0; ni < FN; ++ni)
                    {
                        *reinterpret_cast<double2 *>(C + static_cast<int64_t>(16 * mi + 8 * h) * ldc + 8 * ni) =
                            make_double2(v[h][ni].x - acc[mi][ni][2 * h], v[h][ni].y - acc[mi][ni][2 * h + 1]);
                    }
                }
            }
        }
        else
        {
#pragma unroll
            for (int mi = 0; mi < FM; ++mi)
            {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const int r = row + 16 * mi + 8 * h;
                    const int last = (j.a == 0 && p.lower) ? min(r, p.N - 1) : p.N - 1;
#pragma unroll
                    for (int ni = 0; ni < FN; ++ni)
                    {
                        double *c = C + static_cast<int64_t>(16 * mi + 8 * h) * ldc + 8 * ni;
                        const int cc = col + 8 * ni;
                        if (r < M && cc <= last)
                        {
                            c[0] = C_FIRST ? -acc[mi][ni][2 * h] : c[0] - acc[mi][ni][2 * h];
                        }
                        if (r < M && cc + 1 <= last)
                        {
                            c[1] = C_FIRST ? -acc[mi][ni][2 * h + 1] : c[1] - acc[mi][ni][2 * h + 1];
                        }
                    }
                }
            }
        }
    }
    if (p.y != nullptr)
    {
        vector_update(p, blockIdx.x * 4 + warp, gridDim.x * 4);
    }
    __syncthreads();
    if (abort_flag != 0)
    {
        if (threadIdx.x == 0 && p.status != nullptr)
        {
            atomicExch(&p.status->timeout, 1);
        }
        drain_after_abort();
    }
}

// Device arguments of a panel solve.
struct SolveParams
{
    int M[2];
    int bs;  // rows and columns of Linv, columns of P
    double *C[2];
    int64_t ldc[2];
    int ctas0, ctas;  // CTAs of row group 0, of both
    double *rowsq;    // group 1: rowsq[i] += sum_j C_new[i][j]^2
    const double *Linv;
    int64_t ldi;
    double *y;  // y := Linv y (bs values), by one further CTA
    DeviceStatus *status;
    int polls;
};

constexpr int SOLVE_THREADS = 256;
constexpr int SOLVE_CHUNKS = 8;  // chunks of 16 columns

template <int FM>
constexpr int solve_smem()
{
    return SOLVE_CHUNKS * (16 * FM + 128) * BK * 8;
}

// P := P Linv^T in place.  A CTA owns 16 FM rows with all bs <= 128 columns;
// warp w produces 16 of them.  Linv is lower triangular, so columns 16 c ..
// need only the first c + 1 chunks of 16 columns of P: a scheduler's two warps
// take column blocks c and 7 - c, which evens their products out, and of chunk
// c only the rows of Linv from 16 c on are copied.  The whole operands are
// requested at once (one memory latency); a warp stores its columns when
// chunks up to theirs have arrived, and the chunks after them hold other
// columns, so nothing is overwritten before it is read.
template <int FM>
__global__ void __launch_bounds__(SOLVE_THREADS, 1)
    solve_kernel(const __grid_constant__ CUtensorMap map_a0, const __grid_constant__ CUtensorMap map_a1,
                 const __grid_constant__ CUtensorMap map_b, const __grid_constant__ SolveParams p)
{
    constexpr int BM = 16 * FM;
    constexpr int CHUNK = (BM + 128) * BK;  // doubles
    extern __shared__ __align__(128) double smem[];
    __shared__ uint64_t full[SOLVE_CHUNKS];
    __shared__ double red[BM][8];
    __shared__ int abort_flag;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    if (static_cast<int>(blockIdx.x) == p.ctas)
    {
        // the vector: a warp takes rows warp, warp + 8, ..
        pdl_wait();
        double *ys = smem;
        if (threadIdx.x < 128)
        {
            ys[threadIdx.x] = static_cast<int>(threadIdx.x) < p.bs ? p.y[threadIdx.x] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int r = warp; r < p.bs; r += 8)
        {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                const int c = lane + 32 * q;
                s += c <= r ? p.Linv[r * p.ldi + c] * ys[c] : 0.0;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                s += __shfl_xor_sync(0xffffffffu, s, o);
            }
            if (lane == 0)
            {
                p.y[r] = s;
            }
        }
        return;
    }
    const int a = static_cast<int>(blockIdx.x) >= p.ctas0;
    const int m0 = (blockIdx.x - (a ? p.ctas0 : 0)) * BM;
    const int M = p.M[a];
    const int nchunks = (p.bs + BK - 1) / BK;
    if (threadIdx.x == 0)
    {
        abort_flag = 0;
        for (int c = 0; c < SOLVE_CHUNKS; ++c)
        {
            tcx::mbar_init(&full[c], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tcx::fence_proxy_async_smem();
    }
    __syncthreads();
    pdl_wait();
    if (threadIdx.x == 0)
    {
        const CUtensorMap *ma = a ? &map_a1 : &map_a0;
        for (int c = 0; c < nchunks; ++c)
        {
            double *dst = smem + c * CHUNK;
            tcx::mbar_expect_tx(&full[c], CHUNK * 8);
            load_boxes(dst, ma, grouped_map(p.bs), BK * c, m0, BM, &full[c]);
            load_boxes(dst + BM * BK, &map_b, grouped_map(p.bs), BK * c, BK * c, 128, &full[c]);
        }
    }
    __syncwarp();
    const int cb = warp < 4 ? warp : 11 - warp;
    double acc[FM][2][4] = {};
    if (BK * cb < p.bs)
    {
        for (int c = 0; c <= cb; ++c)
        {
            ring_wait(&full[c], 0, &abort_flag, p.polls);
            const double *box = smem + c * CHUNK;
#pragma unroll
            for (int ks = 0; ks < 2; ++ks)
            {
                double af[FM][4], bf[2][2];
                load_a(af, box + ks * BM * KC, g, t);
                load_b(bf, box + BM * BK + ks * 128 * KC, BK * (cb - c) + g, t);
                products(acc, af, bf);
            }
        }
    }
    pdl_launch_dependents();  // the stores are left
    const int col = BK * cb + 2 * t;
#pragma unroll
    for (int mi = 0; mi < FM; ++mi)
    {
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            const int r = m0 + 16 * mi + 8 * h + g;
            double *c = p.C[a] + static_cast<int64_t>(r) * p.ldc[a] + col;
            double s = 0.0;
#pragma unroll
            for (int ni = 0; ni < 2; ++ni)
            {
                const double2 v = make_double2(acc[mi][ni][2 * h], acc[mi][ni][2 * h + 1]);
                s += v.x * v.x + v.y * v.y;  // columns >= bs: products with zeros
                if (r < M && col + 8 * ni + 1 < p.bs)
                {
                    *reinterpret_cast<double2 *>(c + 8 * ni) = v;
                }
                else if (r < M && col + 8 * ni < p.bs)
                {
                    c[8 * ni] = v.x;
                }
            }
            if (a == 1 && p.rowsq != nullptr)
            {
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);
                if (t == 0)
                {
                    red[16 * mi + 8 * h + g][cb] = s;
                }
            }
        }
    }
    if (a == 1 && p.rowsq != nullptr)
    {
        __syncthreads();
        if (static_cast<int>(threadIdx.x) < BM && m0 + static_cast<int>(threadIdx.x) < M)
        {
            double s = 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q)
            {
                s += red[threadIdx.x][q];
            }
            p.rowsq[m0 + threadIdx.x] += s;
        }
    }
    __syncthreads();  // every chunk has been waited for by the warp of the last columns
    if (abort_flag != 0)
    {
        if (threadIdx.x == 0 && p.status != nullptr)
        {
            atomicExch(&p.status->timeout, 1);
        }
        drain_after_abort();
    }
}

template <typename Kernel, typename... Args>
void launch_pdl(Kernel kernel, int grid, int threads, int smem, cudaStream_t s, const Args &...args)
{
    ensure_smem_attr(reinterpret_cast<const void *>(kernel), smem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1] = { programmatic_launch_attr() };
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GPRAT_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, args...));
    GPRAT_LAUNCH_CHECK();
}

void check_rows(const RowGroup &g)
{
    if (g.M > 0 && ((g.ldc & 1) || (reinterpret_cast<uintptr_t>(g.C) & 15)))
    {
        throw Error(1, "dgemm: leading dimensions must be even and bases 16-byte aligned");
    }
}

template <int FM, int FN, int MIN_CTAS, bool C_FIRST>
void launch_update(const UpdateArgs &a, cudaStream_t s)
{
    using T = Tile<FM, FN>;
    CUtensorMap ma0, ma1, mb;
    make_map(mb, a.B, a.N, a.K, a.ldb, T::BN);
    const RowGroup &r0 = a.rows[0].M > 0 ? a.rows[0] : a.rows[1], &r1 = a.rows[1].M > 0 ? a.rows[1] : a.rows[0];
    make_map(ma0, r0.A, r0.M, a.K, r0.lda, T::BM);
    make_map(ma1, r1.A, r1.M, a.K, r1.lda, T::BM);
    UpdateParams p{};
    for (int q = 0; q < 2; ++q)
    {
        p.M[q] = std::max(a.rows[q].M, 0);
        p.C[q] = a.rows[q].C;
        p.ldc[q] = a.rows[q].ldc;
    }
    p.N = a.N;
    p.K = a.K;
    p.lower = a.lower;
    const int nt = ceil_div(a.N, T::BN);
    p.tiles0 = a.lower ? trapezoid_tiles<T::BM, T::BN>(p.M[0], a.N) : ceil_div(p.M[0], T::BM) * nt;
    p.tiles = p.tiles0 + ceil_div(p.M[1], T::BM) * nt;
    p.B = a.B;
    p.ldb = a.ldb;
    p.z = a.z;
    p.y = a.y;
    p.status = a.status;
    p.polls = wait_polls();
    launch_pdl(update_kernel<FM, FN, MIN_CTAS, C_FIRST>, p.tiles, GROUP_THREADS, T::RING_BYTES, s, ma0, ma1, mb, p);
}

template <int FM>
void launch_solve(const SolveArgs &a, cudaStream_t s)
{
    CUtensorMap ma0, ma1, mb;
    make_map(mb, a.Linv, a.bs, a.bs, a.ldi, 128);
    const RowGroup &r0 = a.rows[0].M > 0 ? a.rows[0] : a.rows[1], &r1 = a.rows[1].M > 0 ? a.rows[1] : a.rows[0];
    if (r0.M > 0)
    {
        make_map(ma0, r0.A, r0.M, a.bs, r0.lda, 16 * FM);
        make_map(ma1, r1.A, r1.M, a.bs, r1.lda, 16 * FM);
    }
    else
    {
        ma0 = mb;  // only the vector
        ma1 = mb;
    }
    SolveParams p{};
    for (int q = 0; q < 2; ++q)
    {
        p.M[q] = std::max(a.rows[q].M, 0);
        p.C[q] = a.rows[q].C;
        p.ldc[q] = a.rows[q].ldc;
    }
    p.bs = a.bs;
    p.ctas0 = ceil_div(p.M[0], 16 * FM);
    p.ctas = p.ctas0 + ceil_div(p.M[1], 16 * FM);
    p.rowsq = a.rowsq;
    p.Linv = a.Linv;
    p.ldi = a.ldi;
    p.y = a.y;
    p.status = a.status;
    p.polls = wait_polls();
    launch_pdl(solve_kernel<FM>, p.ctas + (a.y != nullptr ? 1 : 0), SOLVE_THREADS, solve_smem<FM>(), s, ma0, ma1, mb,
               p);
}

}  // namespace

void dgemm_update(const UpdateArgs &a, cudaStream_t s)
{
    const int m0 = std::max(a.rows[0].M, 0), m1 = std::max(a.rows[1].M, 0);
    if (m0 + m1 <= 0 || a.N <= 0 || a.K <= 0)
    {
        return;
    }
    check_rows(a.rows[0]);
    check_rows(a.rows[1]);
    if (a.lower && m0 < a.N)
    {
        throw Error(1, "dgemm_update: lower mode needs M >= N");
    }
    const bool timed = gemm_timing_enabled();
    if (timed)
    {
        gemm_timing_begin(s);
    }
    // Tile by the number of elements.  32 x 32 tiles, six CTAs per SM, spread a
    // small update over the chip and have the shorter latency (128 columns of
    // depth 384: 10.0 us at 256 rows against 21.2 with 64 x 64 tiles); 64 x 64
    // tiles read the operands half as often (8192 x 8192 lower, depth 512: 985
    // against 1031 us, 34.9 TFLOP/s).  They meet between 4096 x 512 (77 against
    // 71 us) and 8192 x 512 (130 against 136 us).
    const int64_t area = static_cast<int64_t>(m0 + m1) * a.N - (a.lower ? static_cast<int64_t>(a.N) * (a.N - 1) / 2 : 0);
    const bool large = a.tile != 0 ? a.tile == 1 : area >= 3 * 1024 * 1024;
    if (large)
    {
        a.c_first ? launch_update<2, 4, 3, true>(a, s) : launch_update<2, 4, 3, false>(a, s);
    }
    else
    {
        a.c_first ? launch_update<1, 2, 6, true>(a, s) : launch_update<1, 2, 6, false>(a, s);
    }
    if (timed)
    {
        gemm_timing_end(s, 2.0 * static_cast<double>(area) * a.K);
    }
}

void dgemm_solve(const SolveArgs &a, cudaStream_t s)
{
    const int rows = std::max(a.rows[0].M, 0) + std::max(a.rows[1].M, 0);
    if ((rows <= 0 && a.y == nullptr) || a.bs <= 0)
    {
        return;
    }
    if (a.bs > 128)
    {
        throw Error(1, "dgemm_solve: at most 128 columns");
    }
    check_rows(a.rows[0]);
    check_rows(a.rows[1]);
    const bool timed = gemm_timing_enabled();
    if (timed)
    {
        gemm_timing_begin(s);
    }
    // As few rows per CTA as one wave allows: 4.1, 5.5 and 8.3 us for one wave
    // of 16, 32 and 64 rows (1024, 4096 and 8192 rows), 13.2 us for four of 16.
    const int sms = device_sm_count();
    const int fm = a.tile != 0 ? a.tile : rows <= 16 * sms ? 1 : rows <= 32 * sms ? 2 : 4;
    switch (fm)
    {
    case 1:
        launch_solve<1>(a, s);
        break;
    case 2:
        launch_solve<2>(a, s);
        break;
    default:
        launch_solve<4>(a, s);
        break;
    }
    if (timed)
    {
        gemm_timing_end(s, static_cast<double>(rows) * a.bs * (a.bs + 1));
    }
}

}  // namespace gprat_cu
