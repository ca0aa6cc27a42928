// Kernel-level test entry points of the C ABI (gprat_cu_test_*): run one
// kernel on host-provided data so that tests can compare it in isolation
// (tcgen05 TF32/BF16 GEMM, the FP64 update and panel solve, fused triangular
// solves, the int8 digit split and the int8-emulated FP64 GEMM).
#include "common.cuh"
#include "gprat_cu.h"
#include "ozaki.cuh"
#include "tc_gemm.cuh"

#include <algorithm>
#include <memory>
#include <string>
#include <vector>

namespace gprat_cu
{
void set_last_error(const std::string &message);
}

namespace
{

using namespace gprat_cu;

struct Buf
{
    void *p = nullptr;
    explicit Buf(size_t bytes)
    {
        GPRAT_CUDA_CHECK(cudaMalloc(&p, bytes));
    }
    ~Buf()
    {
        if (p != nullptr)
        {
            cudaFree(p);
        }
    }
    Buf(const Buf &) = delete;
    Buf &operator=(const Buf &) = delete;
};

}  // namespace

extern "C" int gprat_cu_test_tc_gemm(int kind, int M, int N, int K, const float *A, int64_t lda, const float *B,
                                     int64_t ldb, float *C, int64_t ldc, float alpha, float beta, int lower,
                                     double *rowsq, int tile_mode)
{
    try
    {
        if (A == nullptr || B == nullptr || C == nullptr || M <= 0 || N <= 0 || K <= 0 || lda < K || ldb < K ||
            ldc < N || (kind != 0 && kind != 1) || tile_mode < 0 || tile_mode > 3)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_tc_gemm: invalid arguments");
        }
        cudaStream_t s = nullptr;
        // device copies with padded leading dimensions (multiples of 64 elements)
        const int64_t la = round_up(K, 64), lb = round_up(K, 64), lc = round_up(N, 4);
        Buf dA(static_cast<size_t>(M) * la * 4), dB(static_cast<size_t>(N) * lb * 4), dC(static_cast<size_t>(M) * lc * 4);
        GPRAT_CUDA_CHECK(cudaMemcpy2D(dA.p, la * 4, A, lda * 4, K * 4, M, cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy2D(dB.p, lb * 4, B, ldb * 4, K * 4, N, cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy2D(dC.p, lc * 4, C, ldc * 4, N * 4, M, cudaMemcpyHostToDevice));
        Buf dStatus(sizeof(DeviceStatus));
        GPRAT_CUDA_CHECK(cudaMemset(dStatus.p, 0, sizeof(DeviceStatus)));
        // two column-half accumulators: the caller's values in the first, zeros in the second
        Buf dRow(2 * static_cast<size_t>(M) * sizeof(double));
        if (rowsq != nullptr)
        {
            GPRAT_CUDA_CHECK(cudaMemset(dRow.p, 0, 2 * static_cast<size_t>(M) * sizeof(double)));
            GPRAT_CUDA_CHECK(cudaMemcpy(dRow.p, rowsq, M * sizeof(double), cudaMemcpyHostToDevice));
        }
        TcOperand oa, ob;
        Buf hA(kind == 1 ? static_cast<size_t>(M) * la * 2 : 16), hB(kind == 1 ? static_cast<size_t>(N) * lb * 2 : 16);
        if (kind == 1)
        {
            convert_f32_to_bf16(static_cast<const float *>(dA.p), la, hA.p, la, M, K, s);
            convert_f32_to_bf16(static_cast<const float *>(dB.p), lb, hB.p, lb, N, K, s);
            tc_make_operand(oa, hA.p, M, static_cast<int>(la), la, TcKind::BF16);
            tc_make_operand(ob, hB.p, N, static_cast<int>(lb), lb, TcKind::BF16);
        }
        else
        {
            tc_make_operand(oa, dA.p, M, static_cast<int>(la), la, TcKind::TF32);
            tc_make_operand(ob, dB.p, N, static_cast<int>(lb), lb, TcKind::TF32);
        }
        TcGemmArgs g{};
        g.M = M;
        g.N = N;
        g.K = K;
        g.C = static_cast<float *>(dC.p);
        g.ldc = lc;
        g.alpha = alpha;
        g.beta = beta;
        g.lower = lower != 0;
        g.rowsq = rowsq != nullptr ? static_cast<double *>(dRow.p) : nullptr;
        g.rowsq_half = M;
        g.tile_mode = tile_mode;
        g.status = static_cast<DeviceStatus *>(dStatus.p);
        tc_gemm(oa, ob, g, s);
        GPRAT_CUDA_CHECK(cudaStreamSynchronize(s));
        DeviceStatus st{};
        GPRAT_CUDA_CHECK(cudaMemcpy(&st, dStatus.p, sizeof(st), cudaMemcpyDeviceToHost));
        if (st.timeout != 0)
        {
            throw Error(GPRAT_CU_ERR_TIMEOUT, "tensor-core GEMM: a bounded wait timed out");
        }
        GPRAT_CUDA_CHECK(cudaMemcpy2D(C, ldc * 4, dC.p, lc * 4, N * 4, M, cudaMemcpyDeviceToHost));
        if (rowsq != nullptr)
        {
            std::vector<double> halves(2 * static_cast<size_t>(M));
            GPRAT_CUDA_CHECK(cudaMemcpy(halves.data(), dRow.p, halves.size() * sizeof(double), cudaMemcpyDeviceToHost));
            for (int i = 0; i < M; ++i)
            {
                rowsq[i] = halves[i] + halves[M + i];
            }
        }
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

extern "C" int gprat_cu_test_trsv(int kind, int n, const double *L, const double *b, double *x_fwd, double *x_bwd,
                                  int max_ctas)
{
    try
    {
        if (L == nullptr || b == nullptr || x_fwd == nullptr || x_bwd == nullptr || n <= 0 || (kind != 0 && kind != 1) ||
            max_ctas < 0)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_trsv: invalid arguments");
        }
        constexpr int B = 128;
        const int nblk = (n + B - 1) / B;
        const int64_t ld = round_up(n, 64);
        // inverses of the diagonal blocks (host, forward substitution per column)
        std::vector<double> inv(static_cast<size_t>(nblk) * B * B, 0.0);
        for (int k = 0; k < nblk; ++k)
        {
            const int r0 = k * B, bs = std::min(B, n - r0);
            double *X = inv.data() + static_cast<size_t>(k) * B * B;
            for (int c = 0; c < bs; ++c)
            {
                for (int r = c; r < bs; ++r)
                {
                    double s = (r == c) ? 1.0 : 0.0;
                    for (int t = c; t < r; ++t)
                    {
                        s -= L[static_cast<int64_t>(r0 + r) * n + r0 + t] * X[t * B + c];
                    }
                    X[r * B + c] = s / L[static_cast<int64_t>(r0 + r) * n + r0 + r];
                }
            }
        }
        const size_t es = kind == 0 ? sizeof(double) : sizeof(float);
        std::vector<char> hL(static_cast<size_t>(n) * ld * es, 0), hI(inv.size() * es, 0);
        for (int r = 0; r < n; ++r)
        {
            for (int c = 0; c <= r; ++c)
            {
                const double v = L[static_cast<int64_t>(r) * n + c];
                if (kind == 0)
                {
                    reinterpret_cast<double *>(hL.data())[static_cast<int64_t>(r) * ld + c] = v;
                }
                else
                {
                    reinterpret_cast<float *>(hL.data())[static_cast<int64_t>(r) * ld + c] = static_cast<float>(v);
                }
            }
        }
        for (size_t q = 0; q < inv.size(); ++q)
        {
            if (kind == 0)
            {
                reinterpret_cast<double *>(hI.data())[q] = inv[q];
            }
            else
            {
                reinterpret_cast<float *>(hI.data())[q] = static_cast<float>(inv[q]);
            }
        }
        Buf dL(hL.size()), dI(hI.size()), dx(n * sizeof(double)), dscr(n * sizeof(double)), dflags(16),
            dStatus(sizeof(DeviceStatus));
        GPRAT_CUDA_CHECK(cudaMemcpy(dL.p, hL.data(), hL.size(), cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy(dI.p, hI.data(), hI.size(), cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemset(dStatus.p, 0, sizeof(DeviceStatus)));
        cudaStream_t s = nullptr;
        auto *st = static_cast<DeviceStatus *>(dStatus.p);
        auto *x = static_cast<double *>(dx.p);
        for (int dir = 0; dir < 2; ++dir)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy(x, b, n * sizeof(double), cudaMemcpyHostToDevice));
            if (kind == 0)
            {
                const auto *l = static_cast<const double *>(dL.p);
                const auto *li = static_cast<const double *>(dI.p);
                if (dir == 0)
                {
                    trsv_fused_forward(l, ld, li, n, x, static_cast<int *>(dflags.p), static_cast<double *>(dscr.p),
                                       st, s, max_ctas);
                }
                else
                {
                    trsv_fused_backward(l, ld, li, n, x, static_cast<int *>(dflags.p), static_cast<double *>(dscr.p),
                                        st, s, max_ctas);
                }
            }
            else
            {
                const auto *l = static_cast<const float *>(dL.p);
                const auto *li = static_cast<const float *>(dI.p);
                if (dir == 0)
                {
                    trsv_fused_forward_f32(l, ld, li, n, x, static_cast<int *>(dflags.p),
                                           static_cast<double *>(dscr.p), st, s, max_ctas);
                }
                else
                {
                    trsv_fused_backward_f32(l, ld, li, n, x, static_cast<int *>(dflags.p),
                                            static_cast<double *>(dscr.p), st, s, max_ctas);
                }
            }
            GPRAT_CUDA_CHECK(cudaStreamSynchronize(s));
            GPRAT_CUDA_CHECK(cudaMemcpy(dir == 0 ? x_fwd : x_bwd, x, n * sizeof(double), cudaMemcpyDeviceToHost));
        }
        DeviceStatus hst{};
        GPRAT_CUDA_CHECK(cudaMemcpy(&hst, dStatus.p, sizeof(hst), cudaMemcpyDeviceToHost));
        if (hst.timeout != 0)
        {
            throw Error(GPRAT_CU_ERR_TIMEOUT, "triangular solve: a bounded wait timed out");
        }
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

namespace
{

// Digit planes + exponents of one slice operand on the device.
struct OzBuf
{
    Buf dig, exps;
    OzOperand op;
    OzBuf(int rows, int cols, int s, bool block)
        : dig(static_cast<size_t>(s) * round_up(rows, 128) * cols + 128),
          exps(static_cast<size_t>(block ? ceil_div(rows, 128) : rows) * (cols / OZ_KB) * sizeof(int32_t) + 16)
    {
        const int64_t plane = static_cast<int64_t>(round_up(rows, 128)) * cols;
        oz_make_operand(op, static_cast<int8_t *>(dig.p), static_cast<int32_t *>(exps.p), rows, cols, cols, plane,
                        cols / OZ_KB, s, block);
    }
};

}  // namespace

extern "C" int gprat_cu_test_oz_split(int rows, int cols, const double *src, int s, int block, int8_t *digits,
                                      int32_t *exps)
{
    try
    {
        if (src == nullptr || digits == nullptr || exps == nullptr || rows <= 0 || cols <= 0 || cols % OZ_KB != 0 ||
            s < OZ_MIN_SLICES || s > OZ_MAX_SLICES)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_oz_split: invalid arguments");
        }
        Buf dsrc(static_cast<size_t>(rows) * cols * sizeof(double));
        GPRAT_CUDA_CHECK(cudaMemcpy(dsrc.p, src, static_cast<size_t>(rows) * cols * sizeof(double),
                                    cudaMemcpyHostToDevice));
        OzBuf o(rows, cols, s, block != 0);
        cudaStream_t st = nullptr;
        oz_split(static_cast<const double *>(dsrc.p), cols, rows, cols, block ? nullptr : &o.op,
                 block ? &o.op : nullptr, 0, 0, st);
        GPRAT_CUDA_CHECK(cudaStreamSynchronize(st));
        for (int p = 0; p < s; ++p)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy(digits + static_cast<size_t>(p) * rows * cols,
                                        static_cast<int8_t *>(o.dig.p) + p * o.op.plane,
                                        static_cast<size_t>(rows) * cols, cudaMemcpyDeviceToHost));
        }
        const size_t ne = static_cast<size_t>(block ? ceil_div(rows, 128) : rows) * (cols / OZ_KB);
        GPRAT_CUDA_CHECK(cudaMemcpy(exps, o.exps.p, ne * sizeof(int32_t), cudaMemcpyDeviceToHost));
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

extern "C" int gprat_cu_test_oz_emit(int M, int N, int K, const double *A, const double *B, double *C, double beta, int s,
                                     int emit_from, int store_rows, int8_t *rdig, int32_t *rexp, int8_t *bdig,
                                     int32_t *bexp)
{
    try
    {
        if (A == nullptr || B == nullptr || C == nullptr || rdig == nullptr || rexp == nullptr || bdig == nullptr ||
            bexp == nullptr || M <= 0 || N < OZ_KB || N % 2 != 0 || K <= 0 || K % OZ_KB != 0 || s < OZ_MIN_SLICES ||
            s > OZ_MAX_SLICES || emit_from < 0 || emit_from % 128 != 0 || emit_from >= M || store_rows < 0)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_oz_emit: invalid arguments");
        }
        cudaStream_t st = nullptr;
        const size_t bytes = static_cast<size_t>(M) * N * 8;
        Buf dA(static_cast<size_t>(M) * K * 8), dB(static_cast<size_t>(N) * K * 8), dC(bytes);
        GPRAT_CUDA_CHECK(cudaMemcpy(dA.p, A, static_cast<size_t>(M) * K * 8, cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy(dB.p, B, static_cast<size_t>(N) * K * 8, cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy(dC.p, C, bytes, cudaMemcpyHostToDevice));
        const int rows = M - emit_from;
        OzBuf oa(M, K, s, false), ob(N, K, s, true), er(rows, OZ_KB, s, false), eb(rows, OZ_KB, s, true);
        oz_split(static_cast<const double *>(dA.p), K, M, K, &oa.op, nullptr, 0, 0, st);
        oz_split(static_cast<const double *>(dB.p), K, N, K, nullptr, &ob.op, 0, 0, st);
        Buf dStatus(sizeof(DeviceStatus));
        GPRAT_CUDA_CHECK(cudaMemset(dStatus.p, 0, sizeof(DeviceStatus)));
        OzGemmArgs g{};
        g.M = M;
        g.N = N;
        g.K = K;
        g.C = static_cast<double *>(dC.p);
        g.ldc = N;
        g.alpha = -1.0;
        g.beta = beta;
        g.status = static_cast<DeviceStatus *>(dStatus.p);
        g.emit_row = &er.op;
        g.emit_blk = &eb.op;
        g.emit_from = emit_from;
        g.emit_row0 = -emit_from;
        g.store_rows = store_rows;
        oz_gemm(oa.op, ob.op, g, st);
        GPRAT_CUDA_CHECK(cudaStreamSynchronize(st));
        DeviceStatus hs{};
        GPRAT_CUDA_CHECK(cudaMemcpy(&hs, dStatus.p, sizeof(hs), cudaMemcpyDeviceToHost));
        if (hs.timeout != 0)
        {
            throw Error(GPRAT_CU_ERR_TIMEOUT, "int8 GEMM: a bounded wait timed out");
        }
        GPRAT_CUDA_CHECK(cudaMemcpy(C, dC.p, bytes, cudaMemcpyDeviceToHost));
        const size_t pb = static_cast<size_t>(rows) * OZ_KB;
        for (int p = 0; p < s; ++p)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy(rdig + p * pb, er.op.digits + p * er.op.plane, pb, cudaMemcpyDeviceToHost));
            GPRAT_CUDA_CHECK(cudaMemcpy(bdig + p * pb, eb.op.digits + p * eb.op.plane, pb, cudaMemcpyDeviceToHost));
        }
        GPRAT_CUDA_CHECK(cudaMemcpy(rexp, er.exps.p, rows * sizeof(int32_t), cudaMemcpyDeviceToHost));
        GPRAT_CUDA_CHECK(
            cudaMemcpy(bexp, eb.exps.p, ceil_div(rows, 128) * sizeof(int32_t), cudaMemcpyDeviceToHost));
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

extern "C" int gprat_cu_test_oz_gemm(int M, int N, int K, const double *A, const double *B, double *C, double alpha,
                                     double beta, int lower, int s, int groups, double *rowsq, int max_ctas)
{
    try
    {
        if (A == nullptr || B == nullptr || C == nullptr || M <= 0 || N <= 0 || K <= 0 || K % OZ_KB != 0 ||
            s < OZ_MIN_SLICES || s > OZ_MAX_SLICES || groups < 0 || groups > s || max_ctas < 0)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_oz_gemm: invalid arguments");
        }
        cudaStream_t st = nullptr;
        const int64_t lc = round_up(N, 2);
        Buf dA(static_cast<size_t>(M) * K * 8), dB(static_cast<size_t>(N) * K * 8), dC(static_cast<size_t>(M) * lc * 8);
        GPRAT_CUDA_CHECK(cudaMemcpy(dA.p, A, static_cast<size_t>(M) * K * 8, cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy(dB.p, B, static_cast<size_t>(N) * K * 8, cudaMemcpyHostToDevice));
        GPRAT_CUDA_CHECK(cudaMemcpy2D(dC.p, lc * 8, C, N * 8, N * 8, M, cudaMemcpyHostToDevice));
        OzBuf oa(M, K, s, false), ob(N, K, s, true);
        oz_split(static_cast<const double *>(dA.p), K, M, K, &oa.op, nullptr, 0, 0, st);
        oz_split(static_cast<const double *>(dB.p), K, N, K, nullptr, &ob.op, 0, 0, st);
        Buf dStatus(sizeof(DeviceStatus));
        GPRAT_CUDA_CHECK(cudaMemset(dStatus.p, 0, sizeof(DeviceStatus)));
        Buf dRow(2 * static_cast<size_t>(M) * sizeof(double));
        if (rowsq != nullptr)
        {
            GPRAT_CUDA_CHECK(cudaMemset(dRow.p, 0, 2 * static_cast<size_t>(M) * sizeof(double)));
            GPRAT_CUDA_CHECK(cudaMemcpy(dRow.p, rowsq, M * sizeof(double), cudaMemcpyHostToDevice));
        }
        OzGemmArgs g{};
        g.M = M;
        g.N = N;
        g.K = K;
        g.C = static_cast<double *>(dC.p);
        g.ldc = lc;
        g.alpha = alpha;
        g.beta = beta;
        g.lower = lower != 0;
        g.rowsq = rowsq != nullptr ? static_cast<double *>(dRow.p) : nullptr;
        g.rowsq_half = M;
        g.status = static_cast<DeviceStatus *>(dStatus.p);
        g.max_ctas = max_ctas;
        g.groups = groups;
        oz_gemm(oa.op, ob.op, g, st);
        GPRAT_CUDA_CHECK(cudaStreamSynchronize(st));
        DeviceStatus hs{};
        GPRAT_CUDA_CHECK(cudaMemcpy(&hs, dStatus.p, sizeof(hs), cudaMemcpyDeviceToHost));
        if (hs.timeout != 0)
        {
            throw Error(GPRAT_CU_ERR_TIMEOUT, "int8 GEMM: a bounded wait timed out");
        }
        GPRAT_CUDA_CHECK(cudaMemcpy2D(C, N * 8, dC.p, lc * 8, N * 8, M, cudaMemcpyDeviceToHost));
        if (rowsq != nullptr)
        {
            std::vector<double> halves(2 * static_cast<size_t>(M));
            GPRAT_CUDA_CHECK(cudaMemcpy(halves.data(), dRow.p, halves.size() * sizeof(double), cudaMemcpyDeviceToHost));
            for (int i = 0; i < M; ++i)
            {
                rowsq[i] = halves[i] + halves[M + i];
            }
        }
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

extern "C" int gprat_cu_test_set_wait_budget(int64_t polls)
{
    try
    {
        set_wait_budget(polls);
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
}

extern "C" int gprat_cu_test_dgemm_update(int m0, int m1, int N, int K, const double *A0, const double *A1,
                                          const double *B, double *C0, double *C1, int lower, const double *z,
                                          double *y, int tile)
{
    try
    {
        if (m0 < 0 || m1 < 0 || m0 + m1 <= 0 || N <= 0 || K <= 0 || (m0 > 0 && (A0 == nullptr || C0 == nullptr)) ||
            (m1 > 0 && (A1 == nullptr || C1 == nullptr)) || B == nullptr || (lower != 0 && m0 < N) ||
            (z == nullptr) != (y == nullptr) || tile < 0 || tile > 2)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_dgemm_update: invalid arguments");
        }
        cudaStream_t s = nullptr;
        const int64_t lk = round_up(K, 8), ln = round_up(N, 8);
        // the padding columns hold NaN: nothing may read them as data
        auto upload = [&](int rows, int cols, int64_t ld, const double *src)
        {
            auto b = std::make_unique<Buf>(std::max<size_t>(static_cast<size_t>(rows) * ld * 8, 16));
            GPRAT_CUDA_CHECK(cudaMemset(b->p, 0xff, static_cast<size_t>(rows) * ld * 8));
            if (rows > 0)
            {
                GPRAT_CUDA_CHECK(cudaMemcpy2D(b->p, ld * 8, src, cols * 8, cols * 8, rows, cudaMemcpyHostToDevice));
            }
            return b;
        };
        auto dA0 = upload(m0, K, lk, A0), dA1 = upload(m1, K, lk, A1), dB = upload(N, K, lk, B);
        auto dC0 = upload(m0, N, ln, C0), dC1 = upload(m1, N, ln, C1);
        auto dz = upload(z != nullptr ? 1 : 0, K, K, z), dy = upload(y != nullptr ? 1 : 0, N, N, y);
        Buf dStatus(sizeof(DeviceStatus));
        GPRAT_CUDA_CHECK(cudaMemset(dStatus.p, 0, sizeof(DeviceStatus)));
        UpdateArgs a{};
        a.rows[0] = RowGroup{ static_cast<double *>(dA0->p), lk, static_cast<double *>(dC0->p), ln, m0 };
        a.rows[1] = RowGroup{ static_cast<double *>(dA1->p), lk, static_cast<double *>(dC1->p), ln, m1 };
        a.B = static_cast<double *>(dB->p);
        a.ldb = lk;
        a.N = N;
        a.K = K;
        a.lower = lower != 0;
        a.z = z != nullptr ? static_cast<double *>(dz->p) : nullptr;
        a.y = y != nullptr ? static_cast<double *>(dy->p) : nullptr;
        a.status = static_cast<DeviceStatus *>(dStatus.p);
        a.tile = tile;
        dgemm_update(a, s);
        GPRAT_CUDA_CHECK(cudaStreamSynchronize(s));
        DeviceStatus st{};
        GPRAT_CUDA_CHECK(cudaMemcpy(&st, dStatus.p, sizeof(st), cudaMemcpyDeviceToHost));
        if (st.timeout != 0)
        {
            throw Error(GPRAT_CU_ERR_TIMEOUT, "FP64 update: a bounded wait timed out");
        }
        if (m0 > 0)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy2D(C0, N * 8, dC0->p, ln * 8, N * 8, m0, cudaMemcpyDeviceToHost));
        }
        if (m1 > 0)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy2D(C1, N * 8, dC1->p, ln * 8, N * 8, m1, cudaMemcpyDeviceToHost));
        }
        if (y != nullptr)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy(y, dy->p, N * 8, cudaMemcpyDeviceToHost));
        }
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

extern "C" int gprat_cu_test_dgemm_solve(int m0, int m1, int bs, double *P0, double *P1, const double *Linv,
                                         double *rowsq, double *y, int tile)
{
    try
    {
        if (m0 < 0 || m1 < 0 || (m0 + m1 <= 0 && y == nullptr) || bs <= 0 || bs > 128 || (m0 > 0 && P0 == nullptr) ||
            (m1 > 0 && P1 == nullptr) || Linv == nullptr || (tile != 0 && tile != 1 && tile != 2 && tile != 4))
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_dgemm_solve: invalid arguments");
        }
        cudaStream_t s = nullptr;
        const int64_t ld = 128;
        auto upload = [&](int rows, int cols, int64_t l, const double *src)
        {
            auto b = std::make_unique<Buf>(std::max<size_t>(static_cast<size_t>(rows) * l * 8, 16));
            GPRAT_CUDA_CHECK(cudaMemset(b->p, 0xff, static_cast<size_t>(rows) * l * 8));
            if (rows > 0)
            {
                GPRAT_CUDA_CHECK(cudaMemcpy2D(b->p, l * 8, src, cols * 8, cols * 8, rows, cudaMemcpyHostToDevice));
            }
            return b;
        };
        auto d0 = upload(m0, bs, ld, P0), d1 = upload(m1, bs, ld, P1), dL = upload(bs, bs, ld, Linv);
        auto dr = upload(rowsq != nullptr && m1 > 0 ? 1 : 0, m1, m1, rowsq), dy = upload(y != nullptr ? 1 : 0, bs, bs, y);
        Buf dStatus(sizeof(DeviceStatus));
        GPRAT_CUDA_CHECK(cudaMemset(dStatus.p, 0, sizeof(DeviceStatus)));
        SolveArgs a{};
        a.rows[0] = RowGroup{ static_cast<double *>(d0->p), ld, static_cast<double *>(d0->p), ld, m0 };
        a.rows[1] = RowGroup{ static_cast<double *>(d1->p), ld, static_cast<double *>(d1->p), ld, m1 };
        a.Linv = static_cast<double *>(dL->p);
        a.ldi = ld;
        a.bs = bs;
        a.rowsq = rowsq != nullptr ? static_cast<double *>(dr->p) : nullptr;
        a.y = y != nullptr ? static_cast<double *>(dy->p) : nullptr;
        a.status = static_cast<DeviceStatus *>(dStatus.p);
        a.tile = tile;
        dgemm_solve(a, s);
        GPRAT_CUDA_CHECK(cudaStreamSynchronize(s));
        DeviceStatus st{};
        GPRAT_CUDA_CHECK(cudaMemcpy(&st, dStatus.p, sizeof(st), cudaMemcpyDeviceToHost));
        if (st.timeout != 0)
        {
            throw Error(GPRAT_CU_ERR_TIMEOUT, "FP64 panel solve: a bounded wait timed out");
        }
        if (m0 > 0)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy2D(P0, bs * 8, d0->p, ld * 8, bs * 8, m0, cudaMemcpyDeviceToHost));
        }
        if (m1 > 0)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy2D(P1, bs * 8, d1->p, ld * 8, bs * 8, m1, cudaMemcpyDeviceToHost));
        }
        if (rowsq != nullptr && m1 > 0)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy(rowsq, dr->p, m1 * 8, cudaMemcpyDeviceToHost));
        }
        if (y != nullptr)
        {
            GPRAT_CUDA_CHECK(cudaMemcpy(y, dy->p, bs * 8, cudaMemcpyDeviceToHost));
        }
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}

extern "C" int gprat_cu_test_pivot_reciprocals(int n, const double *d, double *seed, double *inv, double *quotient)
{
    try
    {
        if (n <= 0 || d == nullptr || seed == nullptr || inv == nullptr || quotient == nullptr)
        {
            throw Error(GPRAT_CU_ERR_INVALID_ARG, "gprat_cu_test_pivot_reciprocals: invalid arguments");
        }
        const size_t bytes = static_cast<size_t>(n) * 8;
        Buf dd(bytes), ds(bytes), di(bytes), dq(bytes);
        GPRAT_CUDA_CHECK(cudaMemcpy(dd.p, d, bytes, cudaMemcpyHostToDevice));
        pivot_reciprocals(static_cast<double *>(dd.p), n, static_cast<double *>(ds.p), static_cast<double *>(di.p),
                          static_cast<double *>(dq.p), nullptr);
        GPRAT_CUDA_CHECK(cudaMemcpy(seed, ds.p, bytes, cudaMemcpyDeviceToHost));
        GPRAT_CUDA_CHECK(cudaMemcpy(inv, di.p, bytes, cudaMemcpyDeviceToHost));
        GPRAT_CUDA_CHECK(cudaMemcpy(quotient, dq.p, bytes, cudaMemcpyDeviceToHost));
        set_last_error("");
        return GPRAT_CU_OK;
    }
    catch (const Error &e)
    {
        set_last_error(e.what());
        return e.code;
    }
    catch (const std::exception &e)
    {
        set_last_error(e.what());
        return GPRAT_CU_ERR_INVALID_ARG;
    }
}
