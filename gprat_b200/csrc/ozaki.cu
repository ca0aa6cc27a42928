// FP64 matrix products on the int8 tensor cores (Ozaki scheme); the method
// and the slice representation are described in ozaki.cuh.
//
// oz_split_kernel: one CTA per 128 x 128 block of the FP64 source, 8 warps of
// 16 rows; a lane holds 4 consecutive values of a row.  A warp loads its 16
// rows at once into registers (so the block's DRAM latency is paid once, not
// per row), finds the row maxima and, across the CTA, the block maximum,
// and writes s digit planes from the registers, 4 bytes per lane and plane
// (128-byte rows).  Up to five digits come straight from the value
// (direct_digit); more are peeled with the 1.5 * 2^52 rounding trick: y = t + 1.5 * 2^52 rounds t
// to the nearest integer d (ties to even), d is the low word of y, then
// t <- (t - d) * 254 (t - d is exact; the product rounds only once the
// remainder has used up the 53 bits), so D_0 .. D_{s-1} are the leading s
// balanced base-254 digits of x * 2^(6 - e): |D_0| <= 64, |D_p| <= 127.
//
// oz_gemm_kernel: persistent, warp-specialised CTA pair (cluster of 2, 384
// threads each), one 256 x 128 output tile per pair at a time:
//   warp 0, one lane (both CTAs): TMA producer.  For each 128-column block k
//     and group g it loads digit plane g of A (this CTA's 128 rows, 16 KB)
//     and of B (this CTA's 64 rows, 8 KB) into one slot of a ring of
//     OZ_RING, both counted by the slot's one barrier.  A block's planes stay
//     resident until its last group, so every digit tile crosses from L2
//     once per block; the spare slots let the next block's first planes load
//     while the current block's last groups run.
//   warp 2 (leader): scout.  Waits for what each unit needs and signals the
//     issuer through a hardware barrier, so that the thread that runs in step
//     with the tensor core tests no shared-memory barrier.
//   warp 1, one lane (leader): MMA issuer.  Group g of block k is one unit,
//     taken from the highest group down: for p = 0..g, four
//     tcgen05.mma.cta_group::2.kind::i8 (M 256, N 128, K 32) of A_p against
//     B_{g-p} into one int32 accumulator in tensor memory (four accumulators
//     of 128 columns rotate), all 2 G (G + 1) of a block unrolled;
//     tcgen05.commit frees plane g's slot and tells the epilogue.
//   warps 4..11 (both CTAs): epilogue.  Two warps per TMEM lane quarter, 64
//     columns each (224 registers after setmaxnreg).  3 and 5 groups: the two
//     highest are combined exactly in int32 as 254 P_{G-2} + P_{G-1}, kept in
//     registers while the others are multiplied, and the block's whole sum is
//     formed exactly in 64-bit integers, turned into FP64 by one subtraction
//     and added by one FMA with the scale 2^(eA + eB - 12) / 254^(G - 1) into
//     64 FP64 accumulators per thread.  Other G: pairs of groups, each
//     converted and added so (at most 2,112,012,032 in int32).  The next
//     block's exponents are loaded while a block is read.  After the tile's
//     last unit, alpha * acc (+ C, whose lines were sent for when the tile
//     began) is written 16 columns at a time through 4 KB of shared memory per
//     warp, whole 128-byte lines at once; on request the digits of the first
//     128 columns are written from the registers instead or as well.
// What bounds it: the epilogue.  FP64 instructions take 3.2 times as long
// while int8 MMAs stream (12 cycles a warp instruction and scheduler instead
// of 4), and so do integer ones between them, so what counts is the FP64
// instructions per element and block: 2 here (5 groups), 6 when each pair of
// groups is converted by itself.  One 256 x 128 x 128 block of 5 groups takes
// 8400 cycles, of which its MMAs are 3840 (64 each); with the epilogue's
// arithmetic left out 5400, with the integer sums alone 7100.  Against two issuing
// threads that waited for the barriers themselves and three pairs per block, both
// timed in turn on one box (launches one by one): 8192^3, 5 groups, 1808 -> 2111
// TOP/s; 3 groups 1301 -> 1500; 4 groups 1736 -> 1805; lower 28672^2 x 2048 1602 ->
// 1955; 8192 x 128 x 1920 97 -> 86 us; 8192 x 128 x 128 21 to 24 -> 19 to 24 us.
// (Rates below are of versions on the way here, each pair from one run.)
// Every mbarrier wait is bounded (tcgen05_ptx.cuh); a wait that gives up
// raises the CTA's abort flag, the roles leave their loops, TMA copies in
// flight get 200 us to land, the MMA issuer drains, TMEM is freed and the
// status word's timeout flag is set.  No TMA multicast is used.
#include "ozaki.cuh"
#include "tcgen05_ptx.cuh"

#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>
#include <string>

namespace gprat_cu
{
namespace
{

using namespace tcx;

constexpr int OZ_ZERO_EXP = -2000;  // an all-zero domain: digits 0
constexpr int OZ_BAD_EXP = 4000;    // a NaN or infinity in the domain: the product becomes NaN
constexpr double RND = 6755399441055744.0;      // 1.5 * 2^52
constexpr double I2D_BIAS = 4503601774854144.0;  // 2^52 + 2^31

__device__ __forceinline__ double pow2(int e)
{
    e = max(-1022, min(1023, e));
    return __longlong_as_double(static_cast<long long>(e + 1023) << 52);
}

// e with max|x| < 2^e over a domain whose maximum is vmax
__device__ __forceinline__ int exp_of(double vmax, bool bad)
{
    if (bad)
    {
        return OZ_BAD_EXP;
    }
    if (vmax == 0.0)
    {
        return OZ_ZERO_EXP;
    }
    const int e = ilogb(vmax) + 1;
    return e < -960 ? OZ_ZERO_EXP : e;
}

// The leading balanced base-254 digit of t (the low byte of the result), and
// t <- 254 (t - digit) if more are wanted: y holds the digit in its low word,
// 254 digit is exact from y by one FMA, and the next t is rounded once, as
// (t - digit) 254 would be (t - digit is exact).
template <bool MORE>
__device__ __forceinline__ uint32_t next_digit(double &t)
{
    const double y = __dadd_rn(t, RND);
    if (MORE)
    {
        t = __fma_rn(t, OZ_BASE, __fma_rn(y, -OZ_BASE, OZ_BASE * RND));
    }
    return static_cast<uint32_t>(__double2loint(y));
}

// The low bytes of four digits.
__device__ __forceinline__ uint32_t pack4(uint32_t d0, uint32_t d1, uint32_t d2, uint32_t d3)
{
    return __byte_perm(__byte_perm(d0, d1, 0x0040), __byte_perm(d2, d3, 0x0040), 0x5410);
}

// The digits of four consecutive values as bytes.
template <bool MORE>
__device__ __forceinline__ uint32_t next_digits(double *t)
{
    const uint32_t d0 = next_digit<MORE>(t[0]), d1 = next_digit<MORE>(t[1]);
    const uint32_t d2 = next_digit<MORE>(t[2]), d3 = next_digit<MORE>(t[3]);
    return pack4(d0, d1, d2, d3);
}

__device__ __forceinline__ double digit_scale(int e)
{
    return e == OZ_ZERO_EXP || e == OZ_BAD_EXP ? 0.0 : pow2(6 - e);
}

// Up to OZ_DIRECT digits come straight from v: with c_p = 254^p 2^(6 - e), the
// leading p + 1 digits as one integer are rint(c_p v) = 254 rint(c_(p-1) v) + d_p
// (254 is even, so ties round alike), and -254 = 2 modulo 256 leaves the byte of
// d_p as that of rint(c_p v) + 2 rint(c_(p-1) v): one FMA and one integer
// instruction a digit, without a chain from digit to digit, where peeling takes
// three FMAs' time.  Both are exact as long as the peeled remainder is, so that
// they may differ, in the last digit, where that has been rounded (once in
// 2^23 values with 5 digits); from 6 on, where it would be once in 2^15, the
// digits are peeled.  With 32-byte stores a tile's digits take 10,700 cycles of
// the epilogue instead of 13,300.
constexpr int OZ_DIRECT = 5;
__device__ __forceinline__ uint32_t direct_digit(double v, double c, uint32_t &prev)
{
    const uint32_t d = static_cast<uint32_t>(__double2loint(__fma_rn(v, c, RND)));
    const uint32_t byte = d + 2 * prev;
    prev = d;
    return byte;
}

__device__ __forceinline__ uint32_t direct_digits(const double *v, double c, uint32_t *prev)
{
    const uint32_t d0 = direct_digit(v[0], c, prev[0]), d1 = direct_digit(v[1], c, prev[1]);
    const uint32_t d2 = direct_digit(v[2], c, prev[2]), d3 = direct_digit(v[3], c, prev[3]);
    return pack4(d0, d1, d2, d3);
}

// S digit planes of 4 consecutive values (4 bytes per plane at out + p * plane)
template <int S>
__device__ __forceinline__ void write_digits(const double v[4], int e, int8_t *out, int64_t plane)
{
    const double sc = digit_scale(e);
    if (S <= OZ_DIRECT)
    {
        uint32_t prev[4] = { 0, 0, 0, 0 };
        double c = sc;
#pragma unroll
        for (int p = 0; p < S; ++p)
        {
            *reinterpret_cast<uint32_t *>(out + p * plane) = direct_digits(v, c, prev);
            c = __dmul_rn(c, OZ_BASE);
        }
        return;
    }
    double t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
        t[i] = __dmul_rn(v[i], sc);
    }
#pragma unroll
    for (int p = 0; p < S; ++p)
    {
        *reinterpret_cast<uint32_t *>(out + p * plane) = p + 1 < S ? next_digits<true>(t) : next_digits<false>(t);
    }
}

// Shared memory by its own address: a generic pointer would order these with
// the stores to global memory.
__device__ __forceinline__ void sts2(uint32_t a, double2 v)
{
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ double2 lds2(uint32_t a)
{
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void stg8(int8_t *a, const uint32_t (&w)[8])
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(a), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
}

// S digit planes of an epilogue thread's 64 values (64 bytes per plane), 32
// bytes, one memory sector, at a time.
__device__ __forceinline__ void write_row_digits(const double (&v)[64], int e, int8_t *out, int64_t plane, int S)
{
    const double sc = digit_scale(e);
    if (S <= OZ_DIRECT)
    {
#pragma unroll
        for (int c = 0; c < 2; ++c)
        {
            uint32_t prev[32];
#pragma unroll
            for (int i = 0; i < 32; ++i)
            {
                prev[i] = 0;
            }
            int8_t *dst = out + 32 * c;
            double cp = sc;
#pragma unroll 1
            for (int p = 0; p < S; ++p, dst += plane)
            {
                uint32_t w[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                {
                    w[i] = direct_digits(v + 32 * c + 4 * i, cp, prev + 4 * i);
                }
                stg8(dst, w);
                cp = __dmul_rn(cp, OZ_BASE);
            }
        }
        return;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
    {
        double t[16];
#pragma unroll
        for (int i = 0; i < 16; ++i)
        {
            t[i] = __dmul_rn(v[16 * c + i], sc);
        }
        int8_t *dst = out + 16 * c;
#pragma unroll 1
        for (int p = 1; p < S; ++p, dst += plane)
        {
            *reinterpret_cast<uint4 *>(dst) = make_uint4(next_digits<true>(t), next_digits<true>(t + 4),
                                                         next_digits<true>(t + 8), next_digits<true>(t + 12));
        }
        *reinterpret_cast<uint4 *>(dst) = make_uint4(next_digits<false>(t), next_digits<false>(t + 4),
                                                     next_digits<false>(t + 8), next_digits<false>(t + 12));
    }
}

constexpr int SPLIT_THREADS = 256;

// src is deliberately not __restrict__: loads through a const restrict
// pointer may be compiled as invariant loads, which the compiler is free to
// move above griddepcontrol.wait, before the producing kernel has finished.
template <int S>
__global__ void __launch_bounds__(SPLIT_THREADS) oz_split_kernel(const double *src, int64_t lds, int rows,
                                                                 int8_t *rdig, int64_t rld, int64_t rplane,
                                                                 int32_t *rexp, int rldE, int8_t *bdig, int64_t bld,
                                                                 int64_t bplane, int32_t *bexp, int bldE, int dst_row0,
                                                                 int dst_kb0)
{
    __shared__ double wmax[SPLIT_THREADS / 32];
    __shared__ int wbad[SPLIT_THREADS / 32];
    pdl_wait();
    const int rb = blockIdx.x, kb = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t col = static_cast<int64_t>(kb) * OZ_KB + lane * 4;
    const int r_first = rb * 128 + warp * 16;
    // the warp's 16 rows are loaded at once and kept in registers: the row
    // maxima, the block maximum and the digits all come from these values
    double v[16][4];
#pragma unroll
    for (int i = 0; i < 16; ++i)
    {
        const int r = r_first + i;
        if (r < rows)
        {
            const double2 *p2 = reinterpret_cast<const double2 *>(src + static_cast<int64_t>(r) * lds + col);
            const double2 a = p2[0], b = p2[1];
            v[i][0] = a.x;
            v[i][1] = a.y;
            v[i][2] = b.x;
            v[i][3] = b.y;
        }
        else
        {
            v[i][0] = v[i][1] = v[i][2] = v[i][3] = 0.0;
        }
    }
    int er[16];
    double bm = 0.0;
    bool bbad = false;
#pragma unroll
    for (int i = 0; i < 16; ++i)
    {
        double m = 0.0;
        bool bad = false;
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const double av = fabs(v[i][j]);
            bad = bad || !(av <= 1.0e308);
            m = fmax(m, av);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        }
        bad = __any_sync(0xffffffffu, bad);
        er[i] = exp_of(m, bad);
        const int r = r_first + i;
        if (rdig != nullptr && r < rows && lane == 0)
        {
            rexp[static_cast<int64_t>(dst_row0 + r) * rldE + dst_kb0 + kb] = er[i];
        }
        bm = fmax(bm, m);
        bbad = bbad || bad;
    }
    if (lane == 0)
    {
        wmax[warp] = bm;
        wbad[warp] = bbad ? 1 : 0;
    }
    __syncthreads();
    double blk = 0.0;
    bool blkbad = false;
#pragma unroll
    for (int w = 0; w < SPLIT_THREADS / 32; ++w)
    {
        blk = fmax(blk, wmax[w]);
        blkbad = blkbad || wbad[w] != 0;
    }
    const int eb = exp_of(blk, blkbad);
    if (bdig != nullptr && threadIdx.x == 0)
    {
        bexp[static_cast<int64_t>(dst_row0 / 128 + rb) * bldE + dst_kb0 + kb] = eb;
    }
    const int64_t dcol = static_cast<int64_t>(dst_kb0 + kb) * OZ_KB + lane * 4;
#pragma unroll
    for (int i = 0; i < 16; ++i)
    {
        const int r = r_first + i;
        if (r < rows)
        {
            if (rdig != nullptr)
            {
                write_digits<S>(v[i], er[i], rdig + static_cast<int64_t>(dst_row0 + r) * rld + dcol, rplane);
            }
            if (bdig != nullptr)
            {
                write_digits<S>(v[i], eb, bdig + static_cast<int64_t>(dst_row0 + r) * bld + dcol, bplane);
            }
        }
    }
    pdl_launch_dependents();
}

// ---------------------------------------------------------------------------
// GEMM

// warpgroup 0: warp 0 TMA, warp 1 MMA, warp 2 scout (warp 3 idle); warpgroups 1 and 2
// (warps 4..11): epilogue.  The kernel launches with 168 registers a thread;
// warpgroup 0 gives registers up (setmaxnreg) so that each epilogue thread
// holds 224: 128 * 56 + 256 * 224 = 384 * 168.
constexpr int OZ_THREADS = 384;
constexpr int OZ_REGS_PRODUCER = 56;
constexpr int OZ_REGS_EPILOGUE = 224;
static_assert(128 * OZ_REGS_PRODUCER + 256 * OZ_REGS_EPILOGUE <= OZ_THREADS * 168,
              "the register split exceeds the registers the block launches with");
constexpr int OZ_EPI_WARPS = 8;
constexpr int OZ_A_BYTES = 128 * 128;  // 128 rows x 128 digit bytes
constexpr int OZ_B_BYTES = 64 * 128;   // this CTA's half of the 128 B rows
// Slots of one A and one B digit plane: >= s + 1, so that the next block's first
// planes load early, and a power of two, so that a slot's index is a mask (9
// slots 4 % slower at 8192^3, 5 groups).
constexpr int OZ_RING = 8;
constexpr int OZ_NACC = 4;             // int32 accumulators of 128 TMEM columns
constexpr int OZ_NPHASE = 4;           // barriers of the epilogue's phases, in turn
constexpr int OZ_TMEM_COLS = OZ_NACC * 128;
constexpr int OZ_STAGE_BYTES = 32 * 128;  // an epilogue warp's 32 rows x 16 columns on their way to or from memory
constexpr int OZ_SMEM_BYTES =
    1024 + OZ_RING * (OZ_A_BYTES + OZ_B_BYTES) + OZ_EPI_WARPS * OZ_STAGE_BYTES + 512;
static_assert(OZ_SMEM_BYTES <= 232448, "shared memory of the int8 GEMM exceeds the per-CTA limit");
static_assert(OZ_RING >= OZ_MAX_SLICES + 1, "the ring must hold one block's planes plus one");
// D = S32, A and B signed 8-bit, K-major, N = 128, M = 256 (CTA pair)
constexpr uint32_t OZ_IDESC =
    (2u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((256u >> 4) << 24);
constexpr int OZ_GROUP_M = 8;  // row tiles per group of the non-lower tile order

// Whether the epilogue sums a block's groups in 64-bit integers: where that
// saves FP64 instructions enough to pay for its two widening multiplications.
// At 8192^3 against pairs: 3 groups 8 % faster, 5 groups 13 %; 4 groups 5 %
// slower, so pairs; above 5 the sum has more than 52 bits.
__host__ __device__ constexpr bool oz_sums(int G)
{
    return G == 3 || G == 5;
}

// Whether unit j of a block's G (groups G - 1 .. 0) ends a phase, after which
// the epilogue reads it and the units since the phase before.  With the sums
// the phases are the two highest groups and the rest; else pairs from the top,
// whose sum 254 P_{g-1} + P_g is exact in int32 up to the pair (5, 4), so
// group 6 is alone.
__host__ __device__ constexpr bool phase_ends(int j, int G)
{
    return j == G - 1 || (oz_sums(G) ? j == 1 : ((j & 1) != 0) == (G != 7));
}

// The scout's signal to the MMA issuer: a hardware barrier of their two warps
// per accumulator.
constexpr int OZ_SCOUT_BAR = 1;
__device__ __forceinline__ void scout_arrive(int u)
{
    asm volatile("bar.arrive %0, 64;" ::"r"(OZ_SCOUT_BAR + u) : "memory");
}
__device__ __forceinline__ void scout_sync(int u)
{
    asm volatile("bar.sync %0, 64;" ::"r"(OZ_SCOUT_BAR + u) : "memory");
}

struct OzKernelArgs
{
    int M, N, nkb;
    int a_row0, a_col0, b_row0, b_col0;
    const int32_t *ea;
    int ldea;
    const int32_t *eb;
    int ldeb;
    double *C;
    int64_t ldc;
    double alpha;
    int beta;
    int lower;
    double *rowsq;
    int64_t rowsq_half;
    DeviceStatus *status;
    int tiles_m, tiles_n, ntiles;
    double wpow[OZ_MAX_SLICES + 1];  // wpow[j] = 1 / OZ_BASE^j
    // digits of C's first 128 columns (emit_s planes; 0: none)
    int emit_s, emit_from, emit_row0, emit_kb, store_rows;
    int8_t *rdig, *bdig;
    int32_t *rexp, *bexp;
    int64_t rld, rplane, bld, bplane;
    int rldE, bldE;
};

__device__ __forceinline__ void tma_load_3d_pair(void *dst, const CUtensorMap *map, uint32_t leader_bar, int x, int y,
                                                 int z)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, "
        "%5}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(leader_bar), "r"(x), "r"(y), "r"(z)
        : "memory");
}

__device__ __forceinline__ void mma_i8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(OZ_IDESC), "r"(accumulate));
}

__device__ __forceinline__ void tmem_ld16_i(uint32_t taddr, int32_t *v)
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 16; ++j)
    {
        v[j] = static_cast<int32_t>(r[j]);
    }
}

__device__ __forceinline__ void tmem_ld8_i(uint32_t taddr, int32_t (&v)[8])
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int j = 0; j < 8; ++j)
    {
        v[j] = static_cast<int32_t>(r[j]);
    }
}

// Ties registers written by tcgen05.ld to the point after tcgen05.wait::ld:
// an empty volatile asm that reads and writes each one, so that no use is
// scheduled before the wait.
template <int N>
__device__ __forceinline__ void regs_loaded(int32_t (&v)[N])
{
#pragma unroll
    for (int j = 0; j < N; ++j)
    {
        asm volatile("" : "+r"(v[j]));
    }
}

// exact int32 -> FP64: the bit pattern 0x43300000:(v ^ 2^31) is 2^52 + 2^31 + v
__device__ __forceinline__ double i2d(int32_t v)
{
    return __dsub_rn(__hiloint2double(0x43300000, v ^ static_cast<int32_t>(0x80000000u)), I2D_BIAS);
}

// The sum of a block's G groups, V = sum_g 254^(G-1-g) P_g with |V| < 2^51
// (at most 2.217e15 of 2.252e15), as FP64: low = 254 P_{G-2} + P_{G-1} and the
// groups above it added in 64-bit integers to the bit pattern of
// 1.5 * 2^52 (+ 2^31, so that low enters as an unsigned word), which is then
// the pattern of 1.5 * 2^52 + 2^31 + V.
constexpr double V2D_BIAS = 6755399441055744.0 + 2147483648.0;
template <int G>
__device__ __forceinline__ double sum_of_groups(int32_t p0, int32_t p1, int32_t p2, int32_t low)
{
    int64_t v = (static_cast<int64_t>(0x43380000) << 32) | static_cast<uint32_t>(low ^ static_cast<int32_t>(0x80000000u));
    if (G == 3)
    {
        v += static_cast<int64_t>(p0) * (OZ_IBASE * OZ_IBASE);
    }
    else
    {
        v += static_cast<int64_t>(p2) * (OZ_IBASE * OZ_IBASE);
        v += static_cast<int64_t>(p0 * OZ_IBASE + p1) * (OZ_IBASE * OZ_IBASE * OZ_IBASE);
    }
    return __dsub_rn(__longlong_as_double(v), V2D_BIAS);
}

// pair tile t -> (m0, n0): 256-row x 128-column tiles.  Lower mode: row tile i
// holds the 2 i + 2 column tiles that reach its last row (the final one is
// dropped by the host when it lies right of N).
__device__ __forceinline__ void oz_tile(int t, bool lower, int tiles_m, int tiles_n, int &m0, int &n0)
{
    if (!lower)
    {
        const int span = OZ_GROUP_M * tiles_n;
        const int g = t / span;
        const int first = g * OZ_GROUP_M;
        const int gm = min(tiles_m - first, OZ_GROUP_M);
        const int r = t - g * span;
        m0 = (first + r % gm) * 256;
        n0 = (r / gm) * 128;
        return;
    }
    int i = static_cast<int>((sqrt(4.0 * t + 1.0) - 1.0) * 0.5);
    while ((i + 1) * (i + 2) <= t)
    {
        ++i;
    }
    while (i > 0 && i * (i + 1) > t)
    {
        --i;
    }
    m0 = i * 256;
    n0 = (t - i * (i + 1)) * 128;
}

// G: the number of groups.
template <int G>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    oz_gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, OzKernelArgs p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *aring = smem;
    uint8_t *bring = aring + OZ_RING * OZ_A_BYTES;
    uint8_t *stages = bring + OZ_RING * OZ_B_BYTES;
    uint64_t *full = reinterpret_cast<uint64_t *>(stages + OZ_EPI_WARPS * OZ_STAGE_BYTES);
    uint64_t *empty = full + OZ_RING;
    uint64_t *pfull = empty + OZ_RING;
    uint64_t *tempty = pfull + OZ_NPHASE;
    uint64_t *drain = tempty + OZ_NACC;
    uint64_t *xfull = drain + 1;  // the epilogue warps' exchange
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(xfull + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    const int pair = blockIdx.x >> 1;
    const int npairs = gridDim.x >> 1;
    constexpr bool SUM = oz_sums(G);

    if (threadIdx.x == 0)
    {
        for (int i = 0; i < OZ_RING; ++i)
        {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int u = 0; u < OZ_NPHASE; ++u)
        {
            mbar_init(&pfull[u], 1);
        }
        for (int u = 0; u < OZ_NACC; ++u)
        {
            mbar_init(&tempty[u], 2 * OZ_EPI_WARPS);
        }
        mbar_init(drain, 1);
        mbar_init(xfull, OZ_EPI_WARPS);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0)
    {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(OZ_TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    }
    tc_fence_before();
    cluster_sync_all();  // barriers of both CTAs initialised, TMEM allocated
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();  // the previous kernel's results are visible from here on
    if (warp < 4)
    {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(OZ_REGS_PRODUCER));
    }
    if (warp == 0)
    {
        if (lane == 0)
        {
            // ---------------- TMA producer (both CTAs) ----------------
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmA)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmB)) : "memory");
            uint32_t n = 0;  // digit-plane pairs loaded
            bool ok = true;
            for (int t = pair; ok && t < p.ntiles; t += npairs)
            {
                int m0, n0;
                oz_tile(t, p.lower != 0, p.tiles_m, p.tiles_n, m0, n0);
                const int arow = p.a_row0 + m0 + 128 * static_cast<int>(rank);
                const int brow = p.b_row0 + n0 + 64 * static_cast<int>(rank);
                for (int kb = 0; ok && kb < p.nkb; ++kb)
                {
                    const int xa = p.a_col0 + kb * OZ_KB, xb = p.b_col0 + kb * OZ_KB;
                    for (int g = G - 1; ok && g >= 0; --g)
                    {
                        // slot n % OZ_RING takes A_g and B_g; one barrier counts both
                        const int slot = n % OZ_RING;
                        if (!mbar_wait(&empty[slot], ((n / OZ_RING) & 1u) ^ 1u, abort_flag))
                        {
                            ok = false;
                            break;
                        }
                        if (leader)
                        {
                            mbar_expect_tx(&full[slot], 2 * (OZ_A_BYTES + OZ_B_BYTES));  // both CTAs' bytes
                        }
                        const uint32_t bar = map_to_rank(&full[slot], 0);
                        tma_load_3d_pair(aring + slot * OZ_A_BYTES, &tmA, bar, xa, arow, g);
                        tma_load_3d_pair(bring + slot * OZ_B_BYTES, &tmB, bar, xb, brow, g);
                        ++n;
                    }
                }
            }
            if (*abort_flag)
            {
                // give copies already in flight time to land before the CTA exits
                const unsigned long long t0 = global_ns();
                while (global_ns() - t0 < 200000ull)
                {
                }
            }
        }
    }
    else if (warp == 2 && leader)
    {
        // ---------------- scout (leader) ----------------
        // Waits for what each unit needs -- its accumulator read, and for a
        // block's first unit the block's digit planes -- and passes it on to
        // the issuer's warp through a hardware barrier.  The MMAs read their
        // operands at three quarters of the shared memory's bandwidth, so a
        // test of a shared-memory barrier takes 110 to 240 cycles beside them;
        // in the issuing thread, which runs in step with the tensor core, each
        // of these would be a gap.  The scout is at most four units ahead (it
        // waits for the accumulator of the unit four back), so no barrier is
        // arrived on twice; after a wait that gave up it only keeps pace.
        uint32_t n = 0, nu = 0;
        bool ok = true;
        for (int t = pair; t < p.ntiles; t += npairs)
        {
            for (int kb = 0; kb < p.nkb; ++kb, n += G)
            {
                for (int j = 0; j < G; ++j, ++nu)
                {
                    const int u = nu % OZ_NACC;
                    const bool was = ok;
                    // lane 31 the accumulator, lanes 0 .. G - 1 a plane each, at once
                    if (ok && lane == 31 && nu >= OZ_NACC)
                    {
                        ok = mbar_wait(&tempty[u], ((nu / OZ_NACC) & 1u) ^ 1u, abort_flag);
                    }
                    if (ok && j == 0 && lane < G)
                    {
                        ok = mbar_wait(&full[(n + lane) % OZ_RING], ((n + lane) / OZ_RING) & 1u, abort_flag);
                    }
                    ok = __all_sync(0xffffffffu, ok);
                    if (ok)
                    {
                        scout_arrive(u);
                        continue;
                    }
                    if (was)
                    {
                        // a millisecond for the issuer to take what has been
                        // signalled (it waits for nothing else)
                        const unsigned long long t0 = global_ns();
                        while (global_ns() - t0 < 1000000ull)
                        {
                            __nanosleep(1000);
                        }
                        __syncwarp();
                    }
                    scout_sync(u);
                }
            }
        }
    }
    else if (warp == 1 && leader)
    {
        // ---------------- MMA issuer (leader, one lane) ----------------
        // Descending groups, the largest first: the epilogue reads it and the
        // next while the others are multiplied.  Plane q is last read by group q, so its
        // slot is free long before the block's end, and the next block's
        // planes, loaded in the same order, find it.  Everything between two MMAs
        // is a gap (an issue returns about when the MMA before has completed),
        // so a block's MMAs are unrolled over descriptors made before it (2 %
        // faster at 8192^3, 5 groups).  Descriptors advance from
        // the ring bases (a slot is OZ_A_BYTES / 16 or OZ_B_BYTES / 16 units of
        // the descriptor's address field).
        const uint64_t adesc0 = sw128_desc(smem_u32(aring));
        const uint64_t bdesc0 = sw128_desc(smem_u32(bring));
        int s0 = 0;  // slot of the block's plane G - 1
        uint32_t nu = 0, np = 0;  // units, phases
        for (int t = pair; t < p.ntiles; t += npairs)
        {
            for (int kb = 0; kb < p.nkb; ++kb)
            {
                // the planes' slots and descriptors, before the block's first MMA
                int slot[G];
                uint64_t adesc[G], bdesc[G];
#pragma unroll
                for (int pl = 0; pl < G; ++pl)
                {
                    slot[pl] = s0 + G - 1 - pl;
                    slot[pl] -= slot[pl] >= OZ_RING ? OZ_RING : 0;
                    adesc[pl] = adesc0 + static_cast<uint64_t>(slot[pl] * (OZ_A_BYTES >> 4));
                    bdesc[pl] = bdesc0 + static_cast<uint64_t>(slot[pl] * (OZ_B_BYTES >> 4));
                }
#pragma unroll
                for (int j = 0; j < G; ++j, ++nu)
                {
                    const int g = G - 1 - j;
                    const int u = nu % OZ_NACC;
                    scout_sync(u);
                    if (lane == 0)
                    {
                        tc_fence_after();
                        const uint32_t d = tmem_base + static_cast<uint32_t>(u * 128);
#pragma unroll
                        for (int pa = 0; pa <= g; ++pa)  // A plane pa against B plane g - pa
                        {
#pragma unroll
                            for (int kk = 0; kk < OZ_KB / 32; ++kk)
                            {
                                // 32 bytes of K per instruction: advance the start address by 2 x 16 B
                                mma_i8_pair(d, adesc[pa] + 2 * kk, bdesc[g - pa] + 2 * kk, (pa | kk) != 0 ? 1u : 0u);
                            }
                        }
                        mma_commit_pair_both(&empty[slot[g]]);
                        if (phase_ends(j, G))
                        {
                            mma_commit_pair_both(&pfull[np % OZ_NPHASE]);
                        }
                    }
                    __syncwarp();
                    np += phase_ends(j, G) ? 1 : 0;
                }
                s0 += G;
                s0 -= s0 >= OZ_RING ? OZ_RING : 0;
            }
        }
        if (lane == 0)
        {
            // drain: completes once every MMA issued has completed (waited for
            // after an abort too)
            volatile int gave_up = 0;
            mma_commit_pair_local(drain);
            mbar_wait(drain, 0u, &gave_up);
        }
        __syncwarp();
    }
    else if (warp >= 4)
    {
        // ---------------- epilogue (warps 4..11 of both CTAs) ----------------
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(OZ_REGS_EPILOGUE));
        const int ew = warp - 4;
        const int q = warp & 3;  // TMEM lane quarter this warp may access
        const int h = ew >> 2;   // column half
        uint32_t nu = 0, np = 0, nx = 0;
        bool ok = true, there = false;
        for (int t = pair; ok && t < p.ntiles; t += npairs)
        {
            int mp, n0;
            oz_tile(t, p.lower != 0, p.tiles_m, p.tiles_n, mp, n0);
            const int row0w = mp + 128 * static_cast<int>(rank) + q * 32;  // this warp's first row of C
            const int row = row0w + lane;
            const bool rvalid = row < p.M;
            const int32_t *earow = p.ea + static_cast<int64_t>(p.a_row0 + (rvalid ? row : 0)) * p.ldea + p.a_col0 / OZ_KB;
            const int32_t *ebblk = p.eb + static_cast<int64_t>((p.b_row0 + n0) / 128) * p.ldeb + p.b_col0 / OZ_KB;
            double acc[64];
#pragma unroll
            for (int j = 0; j < 64; ++j)
            {
                acc[j] = 0.0;
            }
            if (p.beta && rvalid)
            {
                // the row's C values towards L2 while the products run
                const double *crow = p.C + static_cast<int64_t>(row) * p.ldc;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                {
                    const int col = n0 + h * 64 + 16 * c;
                    if (col < p.N && (!p.lower || col <= row))
                    {
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(crow + col));
                    }
                }
            }
            int ea_next = earow[0], eb_next = ebblk[0];
            for (int kb = 0; ok && kb < p.nkb; ++kb)
            {
                const int ea = ea_next;
                const int eb = eb_next;
                if (kb + 1 < p.nkb)
                {
                    // the next block's exponents load while this block's groups are read
                    ea_next = earow[kb + 1];
                    eb_next = ebblk[kb + 1];
                }
                const bool bad = ea == OZ_BAD_EXP || eb == OZ_BAD_EXP;
                if constexpr (SUM)
                {
                    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) +
                                               static_cast<uint32_t>(h * 64);
                    const double sc = bad ? __longlong_as_double(0x7ff8000000000000ll)
                                          : pow2(ea + eb - 12) * p.wpow[G - 1];
                    // Has phase np completed?  Its test is issued before the last
                    // products of the phase before it, so that a phase which is
                    // there by then costs no wait; else one lane polls (the others'
                    // polls would take shared-memory bandwidth from the MMAs).
                    auto phase_test = [&]()
                    { return mbar_test_wait(&pfull[np % OZ_NPHASE], (np / OZ_NPHASE) & 1u); };
                    auto phase_ready = [&]()
                    {
                        if (!__all_sync(0xffffffffu, there))
                        {
                            if (lane == 0)
                            {
                                ok = mbar_wait(&pfull[np % OZ_NPHASE], (np / OZ_NPHASE) & 1u, abort_flag);
                            }
                            ok = __all_sync(0xffffffffu, ok);
                        }
                        ++np;
                        return ok;
                    };
                    auto unit_base = [&](int j)
                    { return lane_base + static_cast<uint32_t>(((nu + j) % OZ_NACC) * 128); };
                    // every load of units j0 .. j1 - 1 has arrived: the MMAs may reuse them
                    auto release = [&](int j0, int j1)
                    {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0)
                        {
                            for (int j = j0; j < j1; ++j)
                            {
                                mbar_arrive_remote(map_to_rank(&tempty[(nu + j) % OZ_NACC], 0));
                            }
                        }
                    };
                    // the two highest groups, G - 1 (unit 0) and G - 2 (unit 1), the
                    // block's longest: 254 P_{G-2} + P_{G-1} kept in 64 registers
                    if (!phase_ready())
                    {
                        break;
                    }
                    tc_fence_after();
                    int32_t low[64];
                    {
                        const uint32_t t0 = unit_base(0), t1 = unit_base(1);
                        int32_t hi[2][16], lo[2][16];
                        tmem_ld16_i(t0, lo[0]);
                        tmem_ld16_i(t1, hi[0]);
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                        {
                            tmem_ld_wait();
                            regs_loaded(lo[c & 1]);
                            regs_loaded(hi[c & 1]);
                            if (c < 3)
                            {
                                tmem_ld16_i(t0 + (c + 1) * 16, lo[(c + 1) & 1]);
                                tmem_ld16_i(t1 + (c + 1) * 16, hi[(c + 1) & 1]);
                            }
                            else
                            {
                                release(0, 2);
                                there = phase_test();
                            }
#pragma unroll
                            for (int k = 0; k < 16; ++k)
                            {
                                low[16 * c + k] = hi[c & 1][k] * OZ_IBASE + lo[c & 1][k];
                            }
                        }
                    }
                    // the other groups, 8 columns at a time, and the block's sum
                    // into the accumulators; meanwhile the MMAs work on the next
                    // block's longest group.  The next columns are requested
                    // early once enough of `low` is used up to hold them.
                    if (!phase_ready())
                    {
                        break;
                    }
                    tc_fence_after();
                    {
                        constexpr int U = G - 2;      // units left: groups U - 1 .. 0
                        constexpr int AHEAD_FROM = U == 3 ? 2 : 0;
                        uint32_t tb[U];
#pragma unroll
                        for (int j = 0; j < U; ++j)
                        {
                            tb[j] = unit_base(G - 1 - j);  // group j
                        }
                        int32_t v[2][U][8];
#pragma unroll
                        for (int c = 0; c < 8; ++c)
                        {
                            if (c <= AHEAD_FROM)
                            {
#pragma unroll
                                for (int j = 0; j < U; ++j)
                                {
                                    tmem_ld8_i(tb[j] + 8 * c, v[c & 1][j]);
                                }
                            }
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < U; ++j)
                            {
                                regs_loaded(v[c & 1][j]);
                            }
                            if (c >= AHEAD_FROM && c < 7)
                            {
#pragma unroll
                                for (int j = 0; j < U; ++j)
                                {
                                    tmem_ld8_i(tb[j] + 8 * (c + 1), v[(c + 1) & 1][j]);
                                }
                            }
                            if (c == 7)
                            {
                                release(2, G);
                                there = phase_test();
                            }
#pragma unroll
                            for (int k = 0; k < 8; ++k)
                            {
                                const double x = sum_of_groups<G>(v[c & 1][0][k], U > 1 ? v[c & 1][U > 1 ? 1 : 0][k] : 0,
                                                                   U > 2 ? v[c & 1][U > 2 ? 2 : 0][k] : 0,
                                                                   low[8 * c + k]);
                                acc[8 * c + k] = fma(x, sc, acc[8 * c + k]);
                            }
                        }
                    }
                    nu += G;
                }
                // groups in pairs (g, g - 1) from the top: OZ_BASE P_{g-1} + P_g is
                // exact in int32, so one conversion and one FMA serve both
                for (int j = 0; !SUM && j < G; ++np)
                {
                    const int g = G - 1 - j;
                    const bool two = !phase_ends(j, G);
                    j += two ? 2 : 1;
                    const int u0 = nu % OZ_NACC;
                    const int u1 = (nu + 1) % OZ_NACC;
                    if (!__all_sync(0xffffffffu, there))
                    {
                        if (lane == 0)
                        {
                            ok = mbar_wait(&pfull[np % OZ_NPHASE], (np / OZ_NPHASE) & 1u, abort_flag);
                        }
                        ok = __all_sync(0xffffffffu, ok);
                    }
                    if (!ok)
                    {
                        break;
                    }
                    tc_fence_after();
                    const uint32_t lane_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) +
                                               static_cast<uint32_t>(h * 64);
                    const uint32_t t0 = lane_base + static_cast<uint32_t>(u0 * 128);
                    const uint32_t t1 = lane_base + static_cast<uint32_t>(u1 * 128);
                    const double sc = bad ? __longlong_as_double(0x7ff8000000000000ll)
                                          : pow2(ea + eb - 12) * p.wpow[g];
                    // 16 columns of each group at a time, double-buffered: the next
                    // chunk's tensor-memory loads are in flight while this chunk converts
                    auto chunk = [&](int32_t(&v)[16], int32_t(&w)[16], int32_t(&vn)[16], int32_t(&wn)[16], int c)
                    {
                        tmem_ld_wait();
                        regs_loaded(v);
                        regs_loaded(w);
                        if (c < 3)
                        {
                            tmem_ld16_i(t0 + (c + 1) * 16, vn);
                            if (two)
                            {
                                tmem_ld16_i(t1 + (c + 1) * 16, wn);
                            }
                            else
                            {
#pragma unroll
                                for (int k = 0; k < 16; ++k)
                                {
                                    wn[k] = 0;
                                }
                            }
                        }
                        else
                        {
                            // both accumulators are read: the MMA warp may reuse them
                            tc_fence_before();
                            __syncwarp();
                            if (lane == 0)
                            {
                                mbar_arrive_remote(map_to_rank(&tempty[u0], 0));
                                if (two)
                                {
                                    mbar_arrive_remote(map_to_rank(&tempty[u1], 0));
                                }
                            }
                            there = mbar_test_wait(&pfull[(np + 1) % OZ_NPHASE], ((np + 1) / OZ_NPHASE) & 1u);
                        }
#pragma unroll
                        for (int k = 0; k < 16; ++k)
                        {
                            acc[c * 16 + k] = fma(i2d(w[k] * OZ_IBASE + v[k]), sc, acc[c * 16 + k]);
                        }
                    };
                    int32_t va[16], wa[16], vb[16], wb[16];
                    tmem_ld16_i(t0, va);
                    if (two)
                    {
                        tmem_ld16_i(t1, wa);
                    }
                    else
                    {
#pragma unroll
                        for (int k = 0; k < 16; ++k)
                        {
                            wa[k] = 0;
                        }
                    }
                    chunk(va, wa, vb, wb, 0);
                    chunk(vb, wb, va, wa, 1);
                    chunk(va, wa, vb, wb, 2);
                    chunk(vb, wb, va, wa, 3);
                    nu += two ? 2 : 1;
                }
            }
            if (!ok)
            {
                break;
            }
            // ---- write alpha * acc, 16 columns at a time ----
            // Through the warp's 4 KB of shared memory (16-byte units, swizzled
            // by the row), so that 8 lanes move 128 consecutive bytes of a row:
            // with each lane at its own row a tile took 25,000 cycles, most of
            // them waiting for the C values (beta = 1).
            double sq = 0.0;
            // opaque, so that the addresses below are formed here and not kept in
            // registers through the products
            uint32_t stage = smem_u32(stages + ew * OZ_STAGE_BYTES);
            int ln = lane;
            int64_t ldc4 = 4 * p.ldc;
            asm volatile("" : "+r"(stage), "+r"(ln), "+l"(ldc4));
            // the 16-byte unit u of row r
            auto unit = [&](int r, int u) { return stage + static_cast<uint32_t>(r * 128 + ((u ^ (r & 7)) << 4)); };
            const int cl = ln & 7, rl = ln >> 3;  // this lane moves columns 2 cl, 2 cl + 1 of rows rl + 4 i
            double alpha = p.alpha;
            bool beta = p.beta != 0;
            int mst = p.M;  // rows written
            if (p.emit_s != 0 && n0 == 0)
            {
                // C's new values into the registers, each lane its own row, and
                // their digits from there: the next product's operand without
                // writing C, reading it again and another launch
#pragma unroll
                for (int c = 0; c < 4; ++c)
                {
                    if (beta)
                    {
                        const double *cptr = p.C + static_cast<int64_t>(row0w + rl) * p.ldc + h * 64 + c * 16 + 2 * cl;
                        if (row0w + 32 <= p.M)
                        {
                            double2 cold[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                            {
                                cold[i] = *reinterpret_cast<const double2 *>(cptr + i * ldc4);
                            }
#pragma unroll
                            for (int i = 0; i < 8; ++i)
                            {
                                const int rr = rl + 4 * i;
                                sts2(unit(rr, cl), cold[i]);
                            }
                        }
                        else
                        {
#pragma unroll 1
                            for (int rr = rl; rr < 32 && row0w + rr < p.M; rr += 4, cptr += ldc4)
                            {
                                sts2(unit(rr, cl), *reinterpret_cast<const double2 *>(cptr));
                            }
                        }
                        __syncwarp();
                    }
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                    {
                        const double2 o = beta ? lds2(unit(ln, u)) : make_double2(0.0, 0.0);
                        double &x = acc[c * 16 + 2 * u], &y = acc[c * 16 + 2 * u + 1];
                        // alpha is 1 or -1, so the product is exact
                        x = beta ? __fma_rn(alpha, x, o.x) : alpha < 0.0 ? -x : x;
                        y = beta ? __fma_rn(alpha, y, o.y) : alpha < 0.0 ? -y : y;
                    }
                    __syncwarp();
                }
                alpha = 1.0;
                beta = false;
                mst = min(mst, p.store_rows);
                // the row's maximum (infinity if a value is not finite), shared with
                // the warp that holds its other half, and the CTA's
                const bool emits = rvalid && row >= p.emit_from;
                unsigned long long mb = 0;
#pragma unroll
                for (int j = 0; j < 64; ++j)
                {
                    mb = max(mb, static_cast<unsigned long long>(__double_as_longlong(acc[j])) & 0x7fffffffffffffffull);
                }
                // larger than 1e308 or a NaN: infinity
                double m = emits ? __longlong_as_double(static_cast<long long>(mb)) : 0.0;
                m = m <= 1.0e308 ? m : __longlong_as_double(0x7ff0000000000000ll);
                double *mx = reinterpret_cast<double *>(stages);
                auto epi_sync = [&]()
                {
                    // the CTA's epilogue warps, with a bounded wait: one that
                    // gave up does not come
                    __syncwarp();
                    if (lane == 0)
                    {
                        mbar_arrive_remote(map_to_rank(xfull, rank));
                        ok = mbar_wait(xfull, nx & 1u, abort_flag);
                    }
                    ++nx;
                    ok = __all_sync(0xffffffffu, ok);
                    __syncwarp();
                    return ok;
                };
                auto row_max = [&](int w) -> double & { return mx[w * (OZ_STAGE_BYTES / 8) + lane]; };
                double wm = m;
                if (p.bdig != nullptr)
                {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1)
                    {
                        wm = fmax(wm, __shfl_xor_sync(0xffffffffu, wm, o));
                    }
                }
                row_max(ew) = m;
                if (lane == 0)
                {
                    mx[ew * (OZ_STAGE_BYTES / 8) + 32] = wm;
                }
                if (!epi_sync())
                {
                    break;
                }
                m = fmax(m, row_max(ew ^ 4));
                double bm = 0.0;
#pragma unroll
                for (int w = 0; w < OZ_EPI_WARPS; ++w)
                {
                    bm = fmax(bm, mx[w * (OZ_STAGE_BYTES / 8) + 32]);
                }
                if (!epi_sync())  // the stages are free again
                {
                    break;
                }
                const int64_t drow = p.emit_row0 + row;
                const int64_t dcol = static_cast<int64_t>(p.emit_kb) * OZ_KB + h * 64;
                if (p.rdig != nullptr && emits)
                {
                    const int e = exp_of(m, !(m <= 1.0e308));
                    if (h == 0)
                    {
                        p.rexp[drow * p.rldE + p.emit_kb] = e;
                    }
                    write_row_digits(acc, e, p.rdig + drow * p.rld + dcol, p.rplane, p.emit_s);
                }
                if (p.bdig != nullptr && emits)
                {
                    const int e = exp_of(bm, !(bm <= 1.0e308));
                    if (h == 0 && (row & 127) == 0)
                    {
                        p.bexp[drow / 128 * p.bldE + p.emit_kb] = e;
                    }
                    write_row_digits(acc, e, p.bdig + drow * p.bld + dcol, p.bplane, p.emit_s);
                }
            }
            if (p.rowsq != nullptr && rvalid)
            {
#pragma unroll
                for (int j = 0; j < 64; ++j)
                {
                    const double x = alpha * acc[j];
                    sq += n0 + h * 64 + j < p.N ? x * x : 0.0;
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
            {
                const int col0 = n0 + h * 64 + c * 16;
                // warp-uniform: chunk right of C, below C, or (lower) above the diagonal for all rows
                if (col0 >= p.N || row0w >= mst || (p.lower && col0 > row0w + 31))
                {
                    continue;
                }
                const int gc = col0 + 2 * cl;
                double *cptr = p.C + static_cast<int64_t>(row0w + rl) * p.ldc + gc;
                // every element of the chunk is written: no tests (they were most of the time)
                const bool whole = row0w + 32 <= mst && col0 + 16 <= p.N && (!p.lower || col0 + 15 <= row0w);
                double2 cold[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                {
                    cold[i] = whole && beta ? *reinterpret_cast<const double2 *>(cptr + i * ldc4) : make_double2(0.0, 0.0);
                }
#pragma unroll
                for (int u = 0; u < 8; ++u)
                {
                    sts2(unit(ln, u), make_double2(alpha * acc[c * 16 + 2 * u], alpha * acc[c * 16 + 2 * u + 1]));
                }
                __syncwarp();
                if (whole)
                {
#pragma unroll
                    for (int i0 = 0; i0 < 8; i0 += 4)
                    {
                        double2 o[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                        {
                            o[i] = lds2(unit(rl + 4 * (i0 + i), cl));
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                        {
                            if (beta)
                            {
                                o[i].x += cold[i0 + i].x;
                                o[i].y += cold[i0 + i].y;
                            }
                            *reinterpret_cast<double2 *>(cptr + (i0 + i) * ldc4) = o[i];
                        }
                    }
                }
                else
                {
#pragma unroll 1
                    for (int rr = rl; rr < 32; rr += 4, cptr += ldc4)
                    {
                        const int r = row0w + rr;
                        const double2 o = lds2(unit(rr, cl));
                        if (r < mst && gc < p.N && (!p.lower || gc <= r))
                        {
                            cptr[0] = beta ? cptr[0] + o.x : o.x;
                            if (gc + 1 < p.N && (!p.lower || gc + 1 <= r))
                            {
                                cptr[1] = beta ? cptr[1] + o.y : o.y;
                            }
                        }
                    }
                }
                __syncwarp();
            }
            __syncwarp();
            if (p.rowsq != nullptr && rvalid)
            {
                p.rowsq[h * p.rowsq_half + row] += sq;  // single writer per word and launch
            }
        }
        // the CTA's last tile is written: the next kernel in the stream may
        // start its set-up
        pdl_launch_dependents();
    }

    tc_fence_before();
    cluster_sync_all();  // no CTA leaves while its peer may still signal or read it
    if (warp == 0)
    {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(OZ_TMEM_COLS));
    }
    if (threadIdx.x == 0 && *abort_flag && p.status != nullptr)
    {
        atomicExch(&p.status->timeout, 1);
    }
}

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once,
                   []
                   {
                       void *q = nullptr;
                       cudaDriverEntryPointQueryResult r;
                       if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &q, 12000, cudaEnableDefault,
                                                            &r) == cudaSuccess &&
                           r == cudaDriverEntryPointSuccess)
                       {
                           fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(q);
                       }
                   });
    if (fn == nullptr)
    {
        throw Error(4, "cuTensorMapEncodeTiled is not available from the driver");
    }
    return fn;
}

void encode_digits(CUtensorMap *map, int8_t *base, int rows, int cols, int64_t ld, int64_t plane, int s, int box_rows)
{
    cuuint64_t dims[3] = { static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows), static_cast<cuuint64_t>(s) };
    cuuint64_t strides[2] = { static_cast<cuuint64_t>(ld), static_cast<cuuint64_t>(plane) };
    cuuint32_t box[3] = { 128u, static_cast<cuuint32_t>(box_rows), 1u };
    cuuint32_t estrides[3] = { 1u, 1u, 1u };
    CUresult r = encode_fn()(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, base, dims, strides, box, estrides,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
    {
        throw Error(4, "cuTensorMapEncodeTiled (digit planes) failed with code " + std::to_string(static_cast<int>(r)));
    }
}

}  // namespace

void oz_make_operand(OzOperand &op, int8_t *digits, int32_t *exps, int rows, int cols, int64_t ld, int64_t plane,
                     int ldE, int s, bool block)
{
    if (digits == nullptr || exps == nullptr || rows <= 0 || cols <= 0 || cols % OZ_KB != 0 || ld < cols ||
        ld % OZ_KB != 0 || plane < static_cast<int64_t>(rows) * ld || plane % 16 != 0 || ldE < cols / OZ_KB ||
        s < OZ_MIN_SLICES || s > OZ_MAX_SLICES || (reinterpret_cast<uintptr_t>(digits) & 127))
    {
        throw Error(1, "oz_make_operand: invalid digit-plane layout");
    }
    op.digits = digits;
    op.exps = exps;
    op.rows = rows;
    op.cols = cols;
    op.ld = ld;
    op.plane = plane;
    op.ldE = ldE;
    op.s = s;
    op.block = block;
    encode_digits(&op.map_a, digits, rows, cols, ld, plane, s, 128);
    encode_digits(&op.map_b, digits, rows, cols, ld, plane, s, 64);
}

void oz_split(const double *src, int64_t lds, int rows, int cols, const OzOperand *row_op, const OzOperand *blk_op,
              int dst_row0, int dst_col0, cudaStream_t s)
{
    if (rows <= 0 || cols <= 0)
    {
        return;
    }
    if (cols % OZ_KB != 0 || dst_col0 % OZ_KB != 0 || (lds & 1) || (reinterpret_cast<uintptr_t>(src) & 15) ||
        (row_op == nullptr && blk_op == nullptr))
    {
        throw Error(1, "oz_split: cols and dst_col0 must be multiples of 128, src 16-byte aligned with an even ld");
    }
    const int slices = row_op != nullptr ? row_op->s : blk_op->s;
    for (const OzOperand *op : { row_op, blk_op })
    {
        if (op == nullptr)
        {
            continue;
        }
        if (op->s != slices || dst_row0 < 0 || dst_row0 + rows > op->rows || dst_col0 + cols > op->cols)
        {
            throw Error(1, "oz_split: destination range exceeds the slice operand");
        }
    }
    if (blk_op != nullptr && dst_row0 % 128 != 0)
    {
        throw Error(1, "oz_split: block exponents need dst_row0 to be a multiple of 128");
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ceil_div(rows, 128), cols / OZ_KB);
    cfg.blockDim = dim3(SPLIT_THREADS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1] = { programmatic_launch_attr() };
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    void (*kern)(const double *, int64_t, int, int8_t *, int64_t, int64_t, int32_t *, int, int8_t *, int64_t,
                 int64_t, int32_t *, int, int, int) = nullptr;
    switch (slices)
    {
    case 3: kern = oz_split_kernel<3>; break;
    case 4: kern = oz_split_kernel<4>; break;
    case 5: kern = oz_split_kernel<5>; break;
    case 6: kern = oz_split_kernel<6>; break;
    case 7: kern = oz_split_kernel<7>; break;
    default: throw Error(1, "oz_split: unsupported digit-plane count");
    }
    static_assert(OZ_MAX_SLICES == 7 && OZ_MIN_SLICES == 3, "oz_split instantiates 3..7 digit planes");
    GPRAT_CUDA_CHECK(cudaLaunchKernelEx(
        &cfg, kern, src, lds, rows, row_op ? row_op->digits : static_cast<int8_t *>(nullptr),
        row_op ? row_op->ld : int64_t(0), row_op ? row_op->plane : int64_t(0),
        row_op ? row_op->exps : static_cast<int32_t *>(nullptr), row_op ? row_op->ldE : 0,
        blk_op ? blk_op->digits : static_cast<int8_t *>(nullptr), blk_op ? blk_op->ld : int64_t(0),
        blk_op ? blk_op->plane : int64_t(0), blk_op ? blk_op->exps : static_cast<int32_t *>(nullptr),
        blk_op ? blk_op->ldE : 0, dst_row0, dst_col0 / OZ_KB));
    GPRAT_LAUNCH_CHECK();
}

void oz_gemm(const OzOperand &A, const OzOperand &B, const OzGemmArgs &a, cudaStream_t s)
{
    if (a.M <= 0 || a.N <= 0)
    {
        return;
    }
    if (A.block || !B.block || A.s != B.s)
    {
        throw Error(1, "oz_gemm: A must be a row operand and B a block operand with the same slice count");
    }
    const int G = a.groups == 0 ? A.s : a.groups;
    if (G < 1 || G > A.s)
    {
        throw Error(1, "oz_gemm: groups must be in [1, s]");
    }
    if (a.K <= 0 || a.K % OZ_KB != 0 || a.a_col0 % OZ_KB != 0 || a.b_col0 % OZ_KB != 0 || a.b_row0 % 128 != 0 ||
        a.a_row0 < 0 || a.b_row0 < 0)
    {
        throw Error(1, "oz_gemm: K, a_col0, b_col0 and b_row0 must be multiples of 128");
    }
    if (a.a_row0 + a.M > A.rows || a.b_row0 + a.N > B.rows || a.a_col0 + a.K > A.cols || a.b_col0 + a.K > B.cols)
    {
        throw Error(1, "oz_gemm: range exceeds an operand");
    }
    if (a.C == nullptr || (reinterpret_cast<uintptr_t>(a.C) & 15) || (a.ldc & 1) || a.ldc < a.N)
    {
        throw Error(1, "oz_gemm: C must be 16-byte aligned with an even ldc >= N");
    }
    if (!(a.beta == 0.0 || a.beta == 1.0))
    {
        throw Error(1, "oz_gemm: beta must be 0 or 1");
    }
    if (a.lower && a.M != a.N)
    {
        throw Error(1, "oz_gemm: lower mode needs M == N");
    }
    if (a.rowsq != nullptr && (a.lower || a.beta != 0.0 || a.rowsq_half < a.M))
    {
        throw Error(1, "oz_gemm: rowsq needs beta = 0, no lower mode and rowsq_half >= M");
    }
    OzKernelArgs k{};
    k.M = a.M;
    k.N = a.N;
    k.nkb = a.K / OZ_KB;
    k.a_row0 = a.a_row0;
    k.a_col0 = a.a_col0;
    k.b_row0 = a.b_row0;
    k.b_col0 = a.b_col0;
    k.ea = A.exps;
    k.ldea = A.ldE;
    k.eb = B.exps;
    k.ldeb = B.ldE;
    k.C = a.C;
    k.ldc = a.ldc;
    k.alpha = a.alpha;
    k.beta = a.beta != 0.0 ? 1 : 0;
    k.lower = a.lower ? 1 : 0;
    k.rowsq = a.rowsq;
    k.rowsq_half = a.rowsq_half;
    k.status = a.status;
    if (a.emit_row != nullptr || a.emit_blk != nullptr)
    {
        for (const OzOperand *o : { a.emit_row, a.emit_blk })
        {
            if (o == nullptr)
            {
                continue;
            }
            if (a.lower || a.N < 128 || !(a.alpha == 1.0 || a.alpha == -1.0) || o->block != (o == a.emit_blk) || o->s != A.s || a.emit_col0 % OZ_KB != 0 ||
                a.emit_from < 0 || a.emit_row0 + a.emit_from < 0 || a.emit_row0 + a.M > o->rows ||
                a.emit_col0 + OZ_KB > o->cols || (o->block && (a.emit_row0 % 128 != 0 || a.emit_from % 128 != 0)) ||
                (reinterpret_cast<uintptr_t>(o->digits) & 31) != 0 || o->ld % 32 != 0 || o->plane % 32 != 0)
            {
                throw Error(1, "oz_gemm: the digits of C do not fit their operand");
            }
        }
        k.emit_s = A.s;
        k.emit_from = a.emit_from;
        k.emit_row0 = a.emit_row0;
        k.emit_kb = a.emit_col0 / OZ_KB;
        k.store_rows = a.store_rows;
        if (a.emit_row != nullptr)
        {
            k.rdig = a.emit_row->digits;
            k.rexp = a.emit_row->exps;
            k.rld = a.emit_row->ld;
            k.rplane = a.emit_row->plane;
            k.rldE = a.emit_row->ldE;
        }
        if (a.emit_blk != nullptr)
        {
            k.bdig = a.emit_blk->digits;
            k.bexp = a.emit_blk->exps;
            k.bld = a.emit_blk->ld;
            k.bplane = a.emit_blk->plane;
            k.bldE = a.emit_blk->ldE;
        }
    }
    double pw = 1.0;
    for (int j = 0; j <= OZ_MAX_SLICES; ++j)
    {
        k.wpow[j] = 1.0 / pw;  // OZ_BASE^j is exact up to j = 6
        pw *= OZ_BASE;
    }
    k.tiles_m = ceil_div(a.M, 256);
    k.tiles_n = ceil_div(a.N, 128);
    if (a.lower)
    {
        k.ntiles = k.tiles_m * (k.tiles_m + 1) - (2 * k.tiles_m > k.tiles_n ? 1 : 0);
    }
    else
    {
        k.ntiles = k.tiles_m * k.tiles_n;
    }
    const int sms = device_sm_count();
    int npairs = std::min(k.ntiles, sms / 2);
    if (a.max_ctas > 0)
    {
        npairs = std::min(npairs, std::max(1, a.max_ctas / 2));
    }
    const bool timed = gemm_timing_enabled();
    if (timed)
    {
        gemm_timing_begin(s);
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * npairs);
    cfg.blockDim = dim3(OZ_THREADS);
    cfg.dynamicSmemBytes = OZ_SMEM_BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1] = programmatic_launch_attr();
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    static_assert(OZ_MAX_SLICES == 7, "a kernel for each number of groups");
    constexpr decltype(&oz_gemm_kernel<1>) kernels[] = {oz_gemm_kernel<1>, oz_gemm_kernel<2>, oz_gemm_kernel<3>,
                                                        oz_gemm_kernel<4>, oz_gemm_kernel<5>, oz_gemm_kernel<6>,
                                                        oz_gemm_kernel<7>};
    const auto kern = kernels[G - 1];
    ensure_smem_attr(reinterpret_cast<const void *>(kern), OZ_SMEM_BYTES);
    GPRAT_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kern, A.map_a, B.map_b, k));
    GPRAT_LAUNCH_CHECK();
    if (timed)
    {
        // int8 tensor-core operations issued (the pipe this kernel is bound by)
        const double mn = a.lower ? 0.5 * static_cast<double>(a.M) * (a.M + 1) : static_cast<double>(a.M) * a.N;
        gemm_timing_end(s, 2.0 * mn * a.K * (G * (G + 1) / 2));
    }
}

}  // namespace gprat_cu
