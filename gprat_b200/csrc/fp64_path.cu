// The FP64 pipeline: blocked Cholesky on the DMMA tensor cores and the solves
// against its factor.
//
// The factorisation (reference right_looking_cholesky_tiled,
// core/src/cpu/tiled_algorithms.cpp:14-57) runs in outer panels of 128 to
// 512 columns, inside a panel by halving down to 128-column blocks:
//   potrf    L_kk and Linv_k (potrf_diag)
//   solve    rows below: P = P Linv_k^T
//   update   the panel's columns right of a finished half with that half
// and, per panel, one update of everything right of it.  Whatever else is to
// be solved against the factor, E L^T = E for further rows E (the variance
// solve's K*, the inverse's identity) and L z = y, takes part in the same
// launches: its rows ride along as a second row group, its z as a vector.
// That makes the solves free of launches and of a serial chain of their own,
// and the products larger.
//
// Look-ahead of one panel: the high-priority side stream applies panel k to
// the columns of panel k+1 and factors it while the main stream updates
// everything right of panel k+1 with panel k.  The update's CTAs end after one
// tile each, so the side stream's CTAs, which the scheduler prefers, get SMs at
// that rate and no SM is set aside.  Events order the
// streams: panel k+1's columns are complete up to panel k-1 when the side
// stream touches them, and panel k's update waits for its factorisation.
//
// Measured (one stream, separate solves and smaller tiles before): fit and
// predict with variances 1.38 -> 0.37 ms at n = 1024, 121 -> 76 ms at
// n = 16384, m = 4096 (33.6 of the chip's 37.2 TFLOP/s), 833 -> 591 ms at
// n = 32768, m = 8192; loss and gradient 33 -> 17.9 ms at n = 8192.
#include "gp_state.cuh"

#include <algorithm>

namespace gprat_cu
{
namespace
{

// Blocks of 128 columns per outer panel.  Narrow panels shorten the chain, wide
// ones make the large updates deeper.  1 / 2 / 4 blocks: fit and predict 364 /
// 371 / 385 us at n = 1024, 1.35 / 1.39 / 1.51 ms at n = 3250; loss and gradient
// 18.2 / 17.9 / 18.2 ms at n = 8192; fit and predict with 2 / 4 24.5 / 24.6 ms at n
// = 10240, 37.8 / 37.7 at 12288, 55.1 / 54.8 at 14336, 76.8 / 76.4 at 16384 (80.1
// with 1), 218.0 / 215.8 at 24576, - / 591 at 32768 (627 with 1, 589 with 8); runs
// differ by 0.1 %.
int panel_blocks(int n) { return knob("GPRAT_CU_FP64_PANEL_BLOCKS", n <= 4096 ? 1 : n <= 12288 ? 2 : 4, 1, 64); }

double *kat(const gprat_cu_gp *gp, int r, int c) { return gp->K.ptr + static_cast<int64_t>(r) * gp->ld + c; }

RowGroup row_group(double *base, int64_t ld, int from, int to, int rows)
{
    RowGroup g{};
    g.A = base + from;
    g.lda = ld;
    g.C = base + to;
    g.ldc = ld;
    g.M = rows;
    return g;
}

// Columns [c0, c1) -= columns [k0, k1): the factor's own rows (factor) and e's.
void update(gprat_cu_gp *gp, const SolveRows &e, bool factor, int k0, int k1, int c0, int c1, cudaStream_t s)
{
    UpdateArgs a{};
    if (factor)
    {
        a.rows[0] = row_group(gp->K.ptr + static_cast<int64_t>(c0) * gp->ld, gp->ld, k0, c0, gp->n - c0);
        a.lower = true;
    }
    a.rows[1] = row_group(e.ptr, e.ld, k0, c0, e.identity ? k1 : e.rows);
    a.B = kat(gp, c0, k0);
    a.ldb = gp->ld;
    a.N = c1 - c0;
    a.K = k1 - k0;
    if (e.vec != nullptr)
    {
        a.z = e.vec + k0;
        a.y = e.vec + c0;
    }
    a.c_first = e.c_first;
    a.status = gp->status.ptr;
    dgemm_update(a, s);
}

// Block column r0 (bs columns) := itself times Linv^T, likewise.
void solve(gprat_cu_gp *gp, const SolveRows &e, bool factor, int r0, int bs, cudaStream_t s)
{
    SolveArgs a{};
    if (factor)
    {
        a.rows[0] = row_group(gp->K.ptr + static_cast<int64_t>(r0 + bs) * gp->ld, gp->ld, r0, r0, gp->n - r0 - bs);
    }
    a.rows[1] = row_group(e.ptr, e.ld, r0, r0, e.identity ? r0 + bs : e.rows);
    a.rowsq = e.rowsq;
    a.Linv = gp->Linv.ptr + static_cast<int64_t>(r0 / NB) * NB * NB;
    a.ldi = NB;
    a.bs = bs;
    a.y = e.vec != nullptr ? e.vec + r0 : nullptr;
    a.status = gp->status.ptr;
    dgemm_solve(a, s);
}

// Columns [c0, c1) by halving: the left half, its update of the right half, the
// right half; block(r0, bs) does 128 columns or fewer.  As many updates as
// blocks, wide ones where they are deep.
template <typename Block, typename Update>
void in_halves(int c0, int c1, const Block &block, const Update &upd)
{
    if (c1 - c0 <= NB)
    {
        block(c0, c1 - c0);
        return;
    }
    const int mid = c0 + (ceil_div(c1 - c0, NB) + 1) / 2 * NB;
    in_halves(c0, mid, block, upd);
    upd(c0, mid, c1);
    in_halves(mid, c1, block, upd);
}

}  // namespace

void factor_solve_fp64(gprat_cu_gp *gp, const SolveRows &e, cudaStream_t s, cudaEvent_t rows_ready)
{
    const int n = gp->n;
    const int nbo = NB * panel_blocks(n);
    const int nout = ceil_div(n, nbo);
    StepScope step("cholesky", s);
    const bool ahead = nout > 1;
    if (ahead || rows_ready != nullptr)
    {
        ensure_lookahead(gp, lookahead_events(n));
    }
    cudaStream_t side = ahead ? gp->side : s;
    auto evF = [&](int k) { return gp->events[1 + k]; };
    auto evR = [&](int k) { return gp->events[1 + nout + k]; };
    auto factor_block = [&](int r0, int bs)
    {
        potrf_diag(kat(gp, r0, r0), gp->ld, bs, r0, gp->Linv.ptr + static_cast<int64_t>(r0 / NB) * NB * NB, NB,
                   gp->status.ptr, side);
        if (r0 == 0 && rows_ready != nullptr)
        {
            GPRAT_CUDA_CHECK(cudaStreamWaitEvent(side, rows_ready, 0));
        }
        solve(gp, e, true, r0, bs, side);
    };
    auto factor_panel = [&](int K0, int pend)
    {
        in_halves(K0, pend, factor_block, [&](int k0, int k1, int c1) { update(gp, e, true, k0, k1, k1, c1, side); });
    };
    if (ahead)
    {
        GPRAT_CUDA_CHECK(cudaEventRecord(gp->events[0], s));
        GPRAT_CUDA_CHECK(cudaStreamWaitEvent(side, gp->events[0], 0));
    }
    factor_panel(0, std::min(nbo, n));
    if (!ahead)
    {
        return;
    }
    GPRAT_CUDA_CHECK(cudaEventRecord(evF(0), side));
    for (int k = 0; k < nout; ++k)
    {
        const int K0 = k * nbo;
        const int pend = std::min(K0 + nbo, n);
        const int next_end = std::min(pend + nbo, n);
        // main: everything right of panel k+1, with panel k
        GPRAT_CUDA_CHECK(cudaStreamWaitEvent(s, evF(k), 0));
        if (next_end < n)
        {
            update(gp, e, true, K0, pend, next_end, n, s);
        }
        if (pend == n)
        {
            break;
        }
        GPRAT_CUDA_CHECK(cudaEventRecord(evR(k), s));
        // side: panel k applied to panel k+1's columns, then panel k+1 factored
        if (k >= 1)
        {
            GPRAT_CUDA_CHECK(cudaStreamWaitEvent(side, evR(k - 1), 0));
        }
        update(gp, e, true, K0, pend, pend, next_end, side);
        factor_panel(pend, next_end);
        GPRAT_CUDA_CHECK(cudaEventRecord(evF(k + 1), side));
    }
}

void solve_rows_fp64(gprat_cu_gp *gp, const SolveRows &e, cudaStream_t s)
{
    const int n = gp->n;
    for (int K0 = 0; K0 < n; K0 += NBO)
    {
        const int pend = std::min(K0 + NBO, n);
        in_halves(
            K0, pend, [&](int r0, int bs) { solve(gp, e, false, r0, bs, s); },
            [&](int k0, int k1, int c1) { update(gp, e, false, k0, k1, k1, c1, s); });
        if (pend < n)
        {
            update(gp, e, false, K0, pend, pend, n, s);
        }
    }
}

void fit_predict_fp64(gprat_cu_gp *gp, const double *d_xt, int m, double *d_mean, double *d_var, cudaStream_t s)
{
    const int n = gp->n;
    ensure_lookahead(gp, lookahead_events(n));
    // buffers first (an allocation must not fall between launches of different streams)
    gp->z.ensure(n);
    gp->W.ensure(static_cast<int64_t>(std::max(m, 1)) * gp->ld);
    gp->vacc.ensure(std::max(m, 1));
    const int ne = lookahead_events(n);
    cudaEvent_t begin = gp->events[ne - 1], rows_ready = gp->events[ne - 2];
    cudaStream_t vs = gp->vstream;
    GPRAT_CUDA_CHECK(cudaEventRecord(begin, s));
    GPRAT_CUDA_CHECK(cudaStreamWaitEvent(vs, begin, 0));
    // the test rows' covariances beside the training covariance and the first block
    GPRAT_CUDA_CHECK(cudaMemcpyAsync(gp->z.ptr, gp->y.ptr, n * sizeof(double), cudaMemcpyDeviceToDevice, vs));
    if (m > 0)
    {
        GPRAT_CUDA_CHECK(cudaMemsetAsync(gp->vacc.ptr, 0, m * sizeof(double), vs));
        assemble_cross(d_xt, m, gp->x.ptr, n, gp->d, gp->params.ptr, gp->W.ptr, gp->ld, nullptr, nullptr, 0, vs);
    }
    GPRAT_CUDA_CHECK(cudaEventRecord(rows_ready, vs));
    assemble_covariance(gp->x.ptr, n, gp->d, gp->T, gp->params.ptr, gp->K.ptr, gp->ld, s);
    SolveRows e{};
    e.ptr = gp->W.ptr;
    e.ld = gp->ld;
    e.rows = m;
    e.rowsq = gp->vacc.ptr;
    e.vec = gp->z.ptr;
    factor_solve_fp64(gp, e, s, rows_ready);
    if (m > 0)
    {
        // K* K^-1 y = (K* L^-T)(L^-1 y)
        cross_times_alpha(gp->W.ptr, gp->ld, m, n, gp->z.ptr, d_mean, s);
        finalize_variance(gp->vacc.ptr, m, gp->params.ptr, d_var, s);
    }
}

}  // namespace gprat_cu
