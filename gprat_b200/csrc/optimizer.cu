// Adjoint gradient of the NLML and the Adam step, on the device.
//
// Reference (core/src/cpu/gp_functions.cpp:1032-1269, tiled_algorithms.cpp:296-448):
// materialise dK/dl and dK/dv tiles (gp_optimizer.cpp:115-150), form the
// explicit K^-1 by two tiled solves on the identity (2n^3 flops), then
//   g_theta = s_theta * 0.5/N * (tr(K^-1 dK) - alpha^T dK alpha),
//   g_noise = s_noise * 0.5/N * (tr(K^-1) - alpha^T alpha),
// with s = sigmoid(softplus^-1(theta)), and apply Adam on the unconstrained
// parameters (gp_optimizer.cpp:154-183).
//
// Here K^-1 = U U^T with U = L^-T (the rows of U L^T = I ride along with
// the factorisation, n^3/3 flops).  One fused kernel then forms each lower tile of U U^T on
// the DMMA tensor cores and, in its epilogue, regenerates the distance
// d_ij = -r_ij^2/(2 l^2) from the series, e_ij = exp(d_ij), and reduces
//   sum w_ij (K^-1_ij - a_i a_j) * (-2 v/l) d_ij e_ij,
//   sum w_ij (K^-1_ij - a_i a_j) * e_ij,       sum_i (K^-1_ii - a_i^2)
// (w = 2 off the diagonal, 1 on it).  Neither K^-1 nor the derivative
// matrices are ever stored.  A one-CTA kernel then reduces the per-tile
// partials in a fixed order and applies Adam to the device-resident
// parameters, so an optimisation loop never returns to the host.
#include "dgemm.cuh"

namespace gprat_cu
{
namespace
{

using namespace gemm;
constexpr int FM = 2, FN = 4;  // 64 x 64 tiles
using AT = Tile<FM, FN>;
constexpr int BM = AT::BM;
constexpr int BN = AT::BN;
constexpr int STAGED_REG = 128;  // up to this many regressors the tile's series windows are staged in shared memory

struct AdjointParams
{
    int n, d, tiles;
    const double *alpha, *x;
    const DeviceParams *p;
    double *partials;
    DeviceStatus *status;
    int polls;
};

// doubles of the epilogue area: series windows, alpha, the reduction
__host__ __device__ constexpr int epilogue_doubles(int d)
{
    return (d <= STAGED_REG ? BM + BN + 2 * d : 0) + BM + BN + 12;
}

// A 64 x 64 lower tile of K^-1 = U U^T per CTA.  U is upper triangular, so row
// m0's products start at column m0: the tiles come longest first, which is what
// keeps the last CTAs short.
__global__ void __launch_bounds__(GROUP_THREADS, 3)
    adjoint_kernel(const __grid_constant__ CUtensorMap map_u, const __grid_constant__ AdjointParams q)
{
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
    }
    __syncthreads();

    const int n = q.n, d = q.d;
    const int tile = blockIdx.x;
    {
        TileJob j;
        j.a = 0;
        trapezoid_tile<BM, BN>(tile, n, n, j.m0, j.n0);
        j.k0 = j.m0;
        j.k1 = n;
        const Ring<FM, FN> ring{ smem, &bars, &abort_flag, &map_u, &map_u, grouped_map(n), q.polls, j };
        ring.begin();
        __syncwarp();
        const int m0 = j.m0, n0 = j.n0;
        // the tile's series windows and alpha
        double *area = smem + AT::RING_BYTES / 8;
        double *ar = area, *ac = ar + BM, *red = ac + BN;  // red: [3][4]
        const double *xr = q.x + m0, *xc = q.x + n0;
        if (d <= STAGED_REG)
        {
            double *sr = red + 12, *sc = sr + BM + d;
            for (int r = threadIdx.x; r < BM + d - 1; r += GROUP_THREADS)
            {
                sr[r] = (m0 + r < n + d - 1) ? xr[r] : 0.0;
            }
            for (int r = threadIdx.x; r < BN + d - 1; r += GROUP_THREADS)
            {
                sc[r] = (n0 + r < n + d - 1) ? xc[r] : 0.0;
            }
            xr = sr;
            xc = sc;
        }
        for (int r = threadIdx.x; r < BM + BN; r += GROUP_THREADS)
        {
            const int i = r < BM ? m0 + r : n0 + r - BM;
            area[r] = i < n ? q.alpha[i] : 0.0;
        }
        __syncthreads();
        double acc[FM][FN][4] = {};
        ring.run(acc, wm * 16 * FM + g, wn * 8 * FN + g, t);

        const double l = q.p->hyper[0];
        const double v = q.p->hyper[1];
        const double nh = -0.5 / (l * l);
        const double fl = -2.0 * v / l;
        double gl = 0.0, gv = 0.0, gn = 0.0;
#pragma unroll
        for (int mi = 0; mi < FM; ++mi)
        {
#pragma unroll
            for (int ni = 0; ni < FN; ++ni)
            {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                {
                    const int li = wm * 16 * FM + 16 * mi + g + (e >> 1) * 8;
                    const int lj = wn * 8 * FN + 8 * ni + 2 * t + (e & 1);
                    const int i = m0 + li, jj = n0 + lj;
                    if (i >= n || jj > i)
                    {
                        continue;
                    }
                    double dist = 0.0;
                    for (int k = 0; k < d; ++k)
                    {
                        const double z = __dsub_rn(xr[li + k], xc[lj + k]);
                        dist = __dadd_rn(dist, __dmul_rn(z, z));
                    }
                    const double dd = __dmul_rn(nh, dist);
                    const double ex = exp(dd);
                    const double w = (i == jj) ? 1.0 : 2.0;
                    const double qv = acc[mi][ni][e] - ar[li] * ac[lj];
                    gl += w * qv * (fl * dd * ex);
                    gv += w * qv * ex;
                    if (i == jj)
                    {
                        gn += qv;
                    }
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            gl += __shfl_xor_sync(0xffffffffu, gl, o);
            gv += __shfl_xor_sync(0xffffffffu, gv, o);
            gn += __shfl_xor_sync(0xffffffffu, gn, o);
        }
        if (lane == 0)
        {
            red[warp] = gl;
            red[4 + warp] = gv;
            red[8 + warp] = gn;
        }
        __syncthreads();
        if (threadIdx.x < 3)
        {
            const double *w = red + 4 * threadIdx.x;
            q.partials[3 * tile + threadIdx.x] = (w[0] + w[1]) + (w[2] + w[3]);
        }
    }
    __syncthreads();
    if (abort_flag != 0)
    {
        if (threadIdx.x == 0 && q.status != nullptr)
        {
            atomicExch(&q.status->timeout, 1);
        }
        drain_after_abort();
    }
}

__device__ double to_constrained(double u, bool noise)
{
    // core/src/cpu/gp_optimizer.cpp:12-22
    return noise ? log(1.0 + exp(u)) + 1e-6 : log(1.0 + exp(u));
}

__device__ double to_unconstrained(double t, bool noise)
{
    // core/src/cpu/gp_optimizer.cpp:24-34
    return noise ? log(exp(t - 1e-6) - 1.0) : log(exp(t) - 1.0);
}

__device__ double sigmoid(double u) { return 1.0 / (1.0 + exp(-u)); }

constexpr int FINISH_THREADS = 256;

// One CTA: the per-tile partials in a fixed order (each thread its own, then a
// tree), then one thread's Adam step.
__global__ void __launch_bounds__(FINISH_THREADS) adjoint_finish_kernel(const double *__restrict__ partials, int np,
                                                                        int n, DeviceParams *__restrict__ p,
                                                                        int adam_step)
{
    __shared__ double part[3][FINISH_THREADS];
    double sum[3] = { 0.0, 0.0, 0.0 };
    for (int b = threadIdx.x; b < np; b += FINISH_THREADS)
    {
#pragma unroll
        for (int q = 0; q < 3; ++q)
        {
            sum[q] += partials[3 * b + q];
        }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q)
    {
        part[q][threadIdx.x] = sum[q];
    }
    __syncthreads();
    for (int w = FINISH_THREADS / 2; w > 0; w >>= 1)
    {
        if (static_cast<int>(threadIdx.x) < w)
        {
#pragma unroll
            for (int q = 0; q < 3; ++q)
            {
                part[q][threadIdx.x] += part[q][threadIdx.x + w];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x != 0)
    {
        return;
    }
    const double G[3] = { part[0][0], part[1][0], part[2][0] };
    const double scale = 0.5 / static_cast<double>(n);  // compute_gradient (gp_optimizer.cpp:222-225)
    double g[3];
    g[0] = sigmoid(to_unconstrained(p->hyper[0], false)) * (scale * G[0]);
    g[1] = sigmoid(to_unconstrained(p->hyper[1], false)) * (scale * G[1]);
    g[2] = sigmoid(to_unconstrained(p->hyper[2], true)) * (scale * G[2]);
    for (int q = 0; q < 3; ++q)
    {
        p->grad[q] = g[q];
    }
    if (!adam_step)
    {
        return;
    }
    const double lr = p->adam[0], b1 = p->adam[1], b2 = p->adam[2], eps = p->adam[3];
    for (int q = 0; q < 3; ++q)
    {
        if (!p->trainable[q])
        {
            continue;
        }
        // update_first/second_moment, adam_step (gp_optimizer.cpp:154-183)
        p->m_T[q] = b1 * p->m_T[q] + (1.0 - b1) * g[q];
        p->w_T[q] = b2 * p->w_T[q] + (1.0 - b2) * g[q] * g[q];
        const bool jitter = (q == 2);
        double u = to_unconstrained(p->hyper[q], jitter);
        double b1t = pow(b1, static_cast<double>(p->iter + 1));
        double b2t = pow(b2, static_cast<double>(p->iter + 1));
        double nu = lr * sqrt(1.0 - b2t) / (1.0 - b1t);
        u = u - nu * p->m_T[q] / (sqrt(p->w_T[q]) + eps);
        p->hyper[q] = to_constrained(u, jitter);
    }
    p->iter += 1;
}

}  // namespace

void adjoint_trace(const double *U, int64_t ldu, const double *alpha, const double *x, int n, int n_reg,
                   const DeviceParams *p, double *partials, int *n_partials, DeviceStatus *status, cudaStream_t s)
{
    static_assert(BM == BN, "one tensor map serves both operands");
    CUtensorMap map_u;
    make_map(map_u, U, n, n, ldu, BM);
    AdjointParams q{};
    q.n = n;
    q.d = n_reg;
    q.tiles = trapezoid_tiles<BM, BN>(n, n);
    q.alpha = alpha;
    q.x = x;
    q.p = p;
    q.partials = partials;
    q.status = status;
    q.polls = wait_polls();
    const int smem = AT::RING_BYTES + epilogue_doubles(n_reg) * 8;
    ensure_smem_attr(reinterpret_cast<const void *>(adjoint_kernel), smem);
    adjoint_kernel<<<q.tiles, GROUP_THREADS, smem, s>>>(map_u, q);
    GPRAT_LAUNCH_CHECK();
    *n_partials = q.tiles;
}

void adjoint_finish(const double *partials, int n_partials, int n, DeviceParams *p, bool adam_step, cudaStream_t s)
{
    adjoint_finish_kernel<<<1, FINISH_THREADS, 0, s>>>(partials, n_partials, n, p, adam_step ? 1 : 0);
    GPRAT_LAUNCH_CHECK();
}

}  // namespace gprat_cu
