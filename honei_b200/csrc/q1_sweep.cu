// Which matrices the Q1 sweep kernel (q1_sweep.cuh) serves, and its launch.
#include "q1_sweep_impl.cuh"

namespace hb2
{
    int q1_sweep_f64(const Q1SweepArgs<double> & g, bool wide, bool uni, int S, int head, int tail, bool pvec,
                     const SweepLaunch & l);
    int q1_sweep_f32(const Q1SweepArgs<float> & g, bool wide, bool uni, int S, int head, int tail, bool pvec,
                     const SweepLaunch & l);

    // every row against the two kinds of rows of a Q1 grid operator: interior rows nine columns
    // in ascending order, boundary rows one diagonal entry in slot 0 (bad bit 0: another
    // structure); all interior rows with the values of the first one, all boundary rows with those
    // of row 0 (bit 1: other values).  ref: those ten values, for the host.
    template <typename T>
    struct GridCheck
    {
        T ref[10];
        int bad;
    };

    template <typename T>
    __global__ void q1_grid_check_kernel(EllView<T> A, uint32_t m, GridCheck<T> * out)
    {
        const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (r >= A.rows) return;
        T ref[10];
#pragma unroll
        for (int k = 0; k < 9; ++k) ref[k] = __ldg(A.val + k * A.ld + m + 1);
        ref[9] = __ldg(A.val);
        if (r == 0)
        {
#pragma unroll
            for (int k = 0; k < 10; ++k) out->ref[k] = ref[k];
        }
        const uint32_t i = (uint32_t)r / m, j = (uint32_t)r - i * m;
        const bool bnd = i == 0 || j == 0 || i == m - 1 || j == m - 1;
        bool shape = true, same = true;
#pragma unroll
        for (int k = 0; k < 9; ++k)
        {
            const int32_t c = A.col[k * A.ld + r];
            const T v = A.val[k * A.ld + r];
            if (bnd)
            {
                shape = shape && (k == 0 ? c == (int32_t)r : c < 0);
                if (k == 0) same = same && v == ref[9];
            }
            else
            {
                shape = shape && c == (int32_t)((int64_t)r + (k / 3 - 1) * (int64_t)m + (k % 3 - 1));
                same = same && v == ref[k];
            }
        }
        if (! shape) atomicOr(&out->bad, 1);
        if (! same) atomicOr(&out->bad, 2);
    }

    // points per line when the matrix can be a nine-point grid matrix, else 0
    static uint32_t grid_points(const hb2_ell_s * A)
    {
        if (A->rows != A->cols || A->K != 9 || A->rows < 9 || A->rows >= (1ull << 31)) return 0;
        uint64_t m = 3;
        while (m * m < A->rows) ++m;
        return m * m == A->rows ? (uint32_t)m : 0;
    }

    int launch_grid_check(hb2_ell_s * A, cudaStream_t stream)
    {
        const uint32_t m = grid_points(A);
        if (! m) return HB2_OK;
        const unsigned grid = ceil_div(A->rows, 256);
        if (A->dtype == HB2_F64)
            q1_grid_check_kernel<double><<<grid, 256, 0, stream>>>(A->view<double>(), m, (GridCheck<double> *)ell_scratch(A));
        else q1_grid_check_kernel<float><<<grid, 256, 0, stream>>>(A->view<float>(), m, (GridCheck<float> *)ell_scratch(A));
        count_launches(1);
        HB2_LAUNCH_CHECK("Q1 grid check");
        return HB2_OK;
    }

    template <typename T>
    static EllGrid grid_result_typed(uint32_t m, const void * scratch)
    {
        const GridCheck<T> & h = *(const GridCheck<T> *)scratch;
        static_assert(sizeof(h) <= kEllScratchBytes - sizeof(int), "scratch of the row check");
        EllGrid g;
        if (h.bad & 1) return g;
        g.m = m;
        g.q1 = h.bad == 0;
        for (int k = 0; k < 10; ++k) g.row[k] = (double)h.ref[k];
        return g;
    }

    EllGrid grid_check_result(const hb2_ell_s * A, const void * scratch)
    {
        const uint32_t m = grid_points(A);
        if (! m) return EllGrid();
        return A->dtype == HB2_F64 ? grid_result_typed<double>(m, scratch) : grid_result_typed<float>(m, scratch);
    }

    template <typename T>
    static int launch_typed(const hb2_ell_s * A, const Q1SweepPass & p, const SweepLaunch & l)
    {
        Q1SweepArgs<T> g = {};
        bool uni = true;
        for (int k = 0; k < 9; ++k)
        {
            g.v[k] = (T)A->q1g_v[k];
            if (k != 4) uni = uni && A->q1g_v[k] == A->q1g_v[0];
        }
        g.vb = (T)A->q1g_vb;
        g.m = (int)A->q1g_m;
        g.mc = (g.m + 1) / 2;
        g.x = (const T *)p.x;
        g.c = (const T *)p.c;
        g.b = (const T *)p.b;
        g.jac = (const T *)p.jac;
        g.y = (T *)p.y;
        g.cb = (T *)p.coarse_b;
        g.cz = (T *)p.coarse_zero;
        g.partials = p.ws ? p.ws->partials : nullptr;
        g.y32 = p.y32;
        g.z32 = p.z32;
        g.list = p.list;
        g.count = p.count;
        g.vs = p.vstride;
        g.cs = p.cstride;
        // columns a lane.  FP64: two from level 9 (9.4 us a pass against 9.9 with one), one
        // below (level 8: 6.7 us), where a strip of 20 owned columns leaves more warps.  FP32:
        // four from level 11 (35.1 / 38.9 us down / up against 37.1 / 45.4 with two), two below
        // (level 10: 11.9 / 15.3 us against 12.3 / 13.6; level 9: 6.9 / 9.4 against 8.5 / 9.9); the
        // line between 1,025 and 2,049 points is not measured
        const bool wide = g.m >= (sizeof(T) == 8 ? 400 : 1500);
        if constexpr (sizeof(T) == 8)
            return q1_sweep_f64(g, wide, uni, p.sweeps, p.zero_guess ? kSweepZero : kSweepLoad, p.tail, p.pvec, l);
        else
            return q1_sweep_f32(g, wide, uni, p.sweeps, p.zero_guess ? kSweepZero : kSweepLoad, p.tail, p.pvec, l);
    }

    int launch_q1_sweep(const hb2_ell_s * A, const Q1SweepPass & p, cudaStream_t stream)
    {
        if (! A->q1g_m || p.sweeps < (sweep_single(p.tail) ? 0 : 1) || p.sweeps > kQ1SweepMax) return fail(HB2_ERR_UNSUPPORTED, "Q1 sweep");
        SweepLaunch l;
        l.nvec = p.list ? p.nvec : 1;
        l.max_vec = p.list ? p.max_vec : 1;
        l.cap = p.cap;
        l.max_partials = p.ws ? p.ws->max_blocks : 0;
        l.blocks = p.blocks;
        l.stream = stream;
        return A->dtype == HB2_F64 ? launch_typed<double>(A, p, l) : launch_typed<float>(A, p, l);
    }

    // Product, defect (+ norm) and product with dot of a large Q1 grid operator as streaming
    // passes; below, the row kernels, whose layout was timed at creation, are as fast or faster.
    // Row kernel / streaming pass (B200, us, graphs of 20): product FP64 3.4 / 3.6 at 601 points a
    // line, 4.4 / 4.3 at 801, 5.8 / 4.9 at 1,001, 19.2 / 12.2 at 2,049, FP32 3.2 / 3.2 at 601,
    // 3.7 / 3.3 at 701; defect FP64 5.3 / 5.8 at 901,
    // 6.0 / 6.3 at 1,025, 6.9 / 6.5 at 1,101, FP32 5.0 / 5.1 at 901, 5.6 / 5.1 at 1,001; defect with
    // its norm FP64 5.6 / 5.9 at 513, 6.7 / 6.3 at 601, 34.2 / 19.1 at 2,049 (FP32 the same lines).
    bool q1_single_applies(const hb2_ell_s * A, int mode, bool reducing)
    {
        const bool f64 = A->dtype == HB2_F64;
        const uint32_t from = reducing ? 600 : mode == kPlain ? (f64 ? 768 : 640) : f64 ? 1100 : 950;
        return A->q1g_m >= from && (mode == kPlain || mode == kDefect || mode == kDot);
    }

    int launch_q1_single(const hb2_ell_s * A, int mode, const void * x, void * y, const void * b, double * red,
                         int want_sqrt, const Workspace * ws, cudaStream_t stream)
    {
        Q1SweepPass p;
        unsigned blocks = 0;
        p.tail = mode == kPlain ? kSweepProduct : (mode == kDefect ? kSweepDefect : kSweepDot);
        p.x = x;
        p.b = b;
        p.y = y;
        p.ws = red ? ws : nullptr;
        p.blocks = &blocks;
        const int st = launch_q1_sweep(A, p, stream);
        if (st || ! red) return st;
        launch_sum_partials(ws->partials, blocks, 1, red, want_sqrt, stream);
        HB2_LAUNCH_CHECK("Q1 pass: partials");
        return HB2_OK;
    }

    int launch_q1_ir_defect(const hb2_ell_s * A, const double * x, const double * b, float * b32, float * x32,
                            double * red, const Workspace * ws, cudaStream_t stream)
    {
        Q1SweepPass p;
        unsigned blocks = 0;
        p.tail = kSweepDefectIR;
        p.x = x;
        p.b = b;
        p.y32 = b32;
        p.z32 = x32;
        p.ws = ws;
        p.blocks = &blocks;
        const int st = launch_q1_sweep(A, p, stream);
        if (st) return st;
        launch_sum_partials(ws->partials, blocks, 1, red, 1, stream);
        HB2_LAUNCH_CHECK("IR defect: partials");
        return HB2_OK;
    }
}
