// FP64 tensor-core (DMMA, mma.sync m16n8k8 .f64) building blocks on sm_100a:
// the TMA-fed main loop shared by the updates (dgemm.cu) and the adjoint
// kernel (optimizer.cu).
//
// DMMA and the FP64 FMA units have the same peak here (128 flops per cycle and
// SM, 37.2 TFLOP/s), and one warp per scheduler with 16 independent products
// reaches 98 % of it (65.4 cycles per product instead of 64), so a main loop is
// as good as the time its warps are not stalled on anything else:
//   * a group of four warps (2 x 2) owns a C tile of 32 FM x 16 FN, a warp
//     FM x FN fragments of 16 x 8; no barrier inside the group: every warp
//     waits on the stage's full barrier and releases the stage by itself;
//   * the operand ring is filled by TMA copies, one per operand and stage;
//   * three CTAs of one 64 x 64 tile share an SM, so one's start and write-out
//     lie under the others' products (two groups of one persistent CTA with
//     128 x 64 tiles, which run in step, reach 29 TFLOP/s where this reaches
//     33.8, at 8192 x 8192 x 512);
//   * operand boxes are 8 columns (64 bytes) wide, and a thread takes columns
//     2t and 2t + 1 as the product's k = t and k = t + 4 (the order of k is free
//     as long as A and B agree): one 16-byte shared load per fragment row, and
//     eight lanes of a quarter warp read 128 contiguous bytes, so no bank
//     conflicts without padding or swizzle;
//   * the fragments of the next k step are loaded while the current one's
//     products are in the pipe.
// A copy fills what lies outside an operand with zeros, so ragged K needs no
// special case.  Waits are bounded: one that runs out raises the CTA's abort
// flag, later waits return at once, and the status word's timeout flag makes
// the host call fail.
#pragma once

#include "common.cuh"
#include "tcgen05_ptx.cuh"

namespace gprat_cu
{
namespace gemm
{

constexpr int KC = 8;      // columns of a TMA box (64 bytes)
constexpr int BK = 2 * KC;  // K per stage
constexpr int STAGES = 4;
constexpr int GROUP_THREADS = 128;

template <int FM, int FN>
struct Tile
{
    static constexpr int BM = 32 * FM;
    static constexpr int BN = 16 * FN;
    static constexpr int A_DOUBLES = BM * BK;
    static constexpr int STAGE_DOUBLES = (BM + BN) * BK;
    static constexpr int RING_BYTES = STAGES * STAGE_DOUBLES * 8;
};

// One tile of the stream a group works through: which A, where, and its K range.
struct TileJob
{
    int a;       // row group: which A operand (and C)
    int m0, n0;  // rows of A, rows of B
    int k0, k1;
};

// Barriers of one group's ring.
struct RingBars
{
    uint64_t full[STAGES];
    uint64_t empty[STAGES];
};

__device__ __forceinline__ void init_ring(RingBars &bars)
{
    for (int st = 0; st < STAGES; ++st)
    {
        tcx::mbar_init(&bars.full[st], 1);
        tcx::mbar_init(&bars.empty[st], 4);
    }
}

// Bounded wait for a barrier's phase: polls times where polls >= 0 (a test's
// budget), else about two seconds.  False: it gave up, now or before (the abort
// flag); a thread that sees false issues no further copy.
__device__ __forceinline__ bool ring_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int polls)
{
    if (tcx::mbar_test_wait(bar, parity))
    {
        return true;
    }
    if (polls < 0)
    {
        return tcx::mbar_wait(bar, parity, abort_flag);
    }
    for (int i = 0; i < polls; ++i)
    {
        if (*abort_flag != 0)
        {
            return false;
        }
        if (tcx::mbar_try_wait(bar, parity))
        {
            return true;
        }
    }
    *abort_flag = 1;
    return false;
}

__device__ __forceinline__ void dmma_16x8x8(double (&d)[4], const double (&a)[4], const double (&b)[2])
{
    asm("mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
        : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            tcx::smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(tcx::smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap *map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, int x, int y, int z, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(tcx::smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(tcx::smem_u32(bar))
        : "memory");
}

// An operand's tensor map: a matrix whose column count is a multiple of 8 as
// (8 columns, rows, column groups), so that one copy brings a stage's two boxes
// (`grouped`); any other as (columns, rows), one box per copy, whose fill of
// zeros ends at the last column.
// Columns k .. k + 15 of `rows` rows from `row`: two boxes.
__device__ __forceinline__ void load_boxes(double *dst, const CUtensorMap *map, bool grouped, int k, int row, int rows,
                                           uint64_t *bar)
{
    if (grouped)
    {
        tma_load_3d(dst, map, 0, row, k / KC, bar);
    }
    else
    {
        tma_load_2d(dst, map, k, row, bar);
        tma_load_2d(dst + rows * KC, map, k + KC, row, bar);
    }
}

// A fragment row pair / B fragment row: two columns per thread.
template <int FM>
__device__ __forceinline__ void load_a(double (&a)[FM][4], const double *box, int row, int t)
{
#pragma unroll
    for (int mi = 0; mi < FM; ++mi)
    {
        const double2 u = *reinterpret_cast<const double2 *>(box + (row + 16 * mi) * KC + 2 * t);
        const double2 v = *reinterpret_cast<const double2 *>(box + (row + 16 * mi + 8) * KC + 2 * t);
        a[mi][0] = u.x;
        a[mi][1] = v.x;
        a[mi][2] = u.y;
        a[mi][3] = v.y;
    }
}

template <int FN>
__device__ __forceinline__ void load_b(double (&b)[FN][2], const double *box, int row, int t)
{
#pragma unroll
    for (int ni = 0; ni < FN; ++ni)
    {
        const double2 u = *reinterpret_cast<const double2 *>(box + (row + 8 * ni) * KC + 2 * t);
        b[ni][0] = u.x;
        b[ni][1] = u.y;
    }
}

template <int FM, int FN>
__device__ __forceinline__ void products(double (&acc)[FM][FN][4], const double (&a)[FM][4], const double (&b)[FN][2])
{
#pragma unroll
    for (int mi = 0; mi < FM; ++mi)
    {
#pragma unroll
        for (int ni = 0; ni < FN; ++ni)
        {
            dmma_16x8x8(acc[mi][ni], a[mi], b[ni]);
        }
    }
}

// The group's operand ring for one tile, as its producer (one thread) and its
// four warps see it.
template <int FM, int FN>
struct Ring
{
    using T = Tile<FM, FN>;
    double *ring;
    RingBars *bars;
    volatile int *abort_flag;
    const CUtensorMap *map_a, *map_b;
    bool grouped;
    int polls;
    TileJob job;

    // producer: the copies of stage number `it` of the tile
    __device__ __forceinline__ void load(int it) const
    {
        const int st = it % STAGES, k = job.k0 + it * BK;
        double *dst = ring + st * T::STAGE_DOUBLES;
        tcx::mbar_expect_tx(&bars->full[st], T::STAGE_DOUBLES * 8);
        load_boxes(dst, map_a, grouped, k, job.m0, T::BM, &bars->full[st]);
        load_boxes(dst + T::A_DOUBLES, map_b, grouped, k, job.n0, T::BN, &bars->full[st]);
    }

    __device__ __forceinline__ int stages() const { return (job.k1 - job.k0 + BK - 1) / BK; }

    // one thread: the first stages
    __device__ __forceinline__ void begin() const
    {
        if (threadIdx.x == 0)
        {
#pragma unroll 1
            for (int q = 0; q < STAGES && q < stages(); ++q)
            {
                load(q);
            }
        }
    }

    // acc += A B^T over the tile's K range.  arow / brow: this thread's first
    // fragment rows in the tile.  The warps take turns at refilling stages
    // (issuing a copy costs a small tile's warp as much as its products).
    __device__ __forceinline__ void run(double (&acc)[FM][FN][4], int arow, int brow, int t) const
    {
        const int nk = stages(), warp = threadIdx.x >> 5;
        double a[2][FM][4], b[2][FN][2];
        const double *box = ring;
        ring_wait(&bars->full[0], 0, abort_flag, polls);
        load_a(a[0], box, arow, t);
        load_b(b[0], box + T::A_DOUBLES, brow, t);
#pragma unroll 1
        for (int kt = 0; kt < nk; ++kt)
        {
            load_a(a[1], box + T::BM * KC, arow, t);
            load_b(b[1], box + T::A_DOUBLES + T::BN * KC, brow, t);
            products(acc, a[0], b[0]);
            __syncwarp();
            if ((threadIdx.x & 31) == 0)
            {
                tcx::mbar_arrive(&bars->empty[kt % STAGES]);
                const int next = kt - 1 + STAGES;  // refills the stage the group left one step ago
                // (a warp that gave up arrives without having waited, so the flag is
                // looked at after the wait: a stage is never loaded twice at once)
                if (warp == (kt & 3) && kt > 0 && next < nk &&
                    ring_wait(&bars->empty[(kt - 1) % STAGES], ((kt - 1) / STAGES) & 1, abort_flag, polls) &&
                    *abort_flag == 0)
                {
                    load(next);
                }
            }
            if (kt + 1 < nk)
            {
                const int st = (kt + 1) % STAGES;
                box = ring + st * T::STAGE_DOUBLES;
                ring_wait(&bars->full[st], ((kt + 1) / STAGES) & 1, abort_flag, polls);
                load_a(a[0], box, arow, t);
                load_b(b[0], box + T::A_DOUBLES, brow, t);
            }
            products(acc, a[1], b[1]);
        }
    }
};

// After a timeout: copies may still be in flight towards this CTA's shared
// memory; they land long before this returns.
__device__ __forceinline__ void drain_after_abort()
{
    const unsigned long long t0 = tcx::global_ns();
    for (int i = 0; i < 100000 && tcx::global_ns() - t0 < 200000ull; ++i)
    {
        __nanosleep(1000);
    }
}

// Row tiles of the lower trapezoid C[i][j], j <= i, of an M x N product (M >= N)
// in BM x BN tiles, BM a multiple of BN: row tile i has min((i + 1) BM / BN, NT)
// column tiles.
template <int BM, int BN>
__host__ __device__ inline int trapezoid_tiles(int M, int N)
{
    constexpr int R = BM / BN;
    const int mt = (M + BM - 1) / BM, nt = (N + BN - 1) / BN;
    const int tri = mt < nt / R ? mt : nt / R;
    return R * tri * (tri + 1) / 2 + (mt - tri) * nt;
}

template <int BM, int BN>
__device__ __forceinline__ void trapezoid_tile(int q, int M, int N, int &m0, int &n0)
{
    constexpr int R = BM / BN;
    const int mt = (M + BM - 1) / BM, nt = (N + BN - 1) / BN;
    const int tri = mt < nt / R ? mt : nt / R;
    const int first = R * tri * (tri + 1) / 2;
    int i, j;
    if (q < first)
    {
        i = static_cast<int>((sqrtf(8.0f * static_cast<float>(q) / R + 1.0f) - 1.0f) * 0.5f);
        while (R * (i + 1) * (i + 2) / 2 <= q)
        {
            ++i;
        }
        while (i > 0 && R * i * (i + 1) / 2 > q)
        {
            --i;
        }
        j = q - R * i * (i + 1) / 2;
    }
    else
    {
        i = tri + (q - first) / nt;
        j = (q - first) % nt;
    }
    m0 = i * BM;
    n0 = j * BN;
}

// Tensor map of a row-major FP64 matrix (rows x cols, ld) for load_boxes
// (dgemm.cu).
void make_map(CUtensorMap &map, const double *base, int rows, int cols, int64_t ld, int box_rows);
// Whether a matrix with that many columns gets a grouped map.
constexpr bool grouped_map(int cols) { return cols % KC == 0; }

}  // namespace gemm
}  // namespace gprat_cu
