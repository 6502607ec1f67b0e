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
    // structure); all interior rows with the values ref[0 .. 8], all boundary rows with ref[9]
    // (bit 1: other values)
    template <typename T>
    __global__ void q1_grid_check_kernel(EllView<T> A, uint32_t m, const T * __restrict__ ref, int * bad)
    {
        const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (r >= A.rows) return;
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
        if (! shape) atomicOr(bad, 1);
        if (! same) atomicOr(bad, 2);
    }

    template <typename T>
    static int find_grid_typed(hb2_ell_s * A, uint32_t m, cudaStream_t stream)
    {
        const EllView<T> V = A->view<T>();
        // the row and the flag in the matrix's own scratch: a place shared by the stream's calls would
        // mix up two matrices that two threads make at the same time
        T ref[10];
        T * dref = (T *)(A->col + (uint64_t)A->K * A->ld);
        int * dbad = (int *)(dref + 10);
        static_assert(10 * sizeof(T) + sizeof(int) <= kEllScratchBytes, "reference row and flag");
        HB2_CUDA(cudaMemsetAsync(dbad, 0, sizeof(int), stream));
        HB2_CUDA(cudaMemcpy2DAsync(dref, sizeof(T), V.val + m + 1, V.ld * sizeof(T), sizeof(T), 9,
                                   cudaMemcpyDeviceToDevice, stream));
        HB2_CUDA(cudaMemcpyAsync(dref + 9, V.val, sizeof(T), cudaMemcpyDeviceToDevice, stream));
        q1_grid_check_kernel<T><<<ceil_div(A->rows, 256), 256, 0, stream>>>(V, m, dref, dbad);
        count_launches(1);
        HB2_LAUNCH_CHECK("Q1 grid check");
        int bad = 1;
        HB2_CUDA(cudaMemcpyAsync(ref, dref, sizeof(ref), cudaMemcpyDeviceToHost, stream));
        HB2_CUDA(cudaMemcpyAsync(&bad, dbad, sizeof(int), cudaMemcpyDeviceToHost, stream));
        HB2_CUDA(cudaStreamSynchronize(stream));
        if (bad == 2) A->g9_m = m;
        if (bad) return HB2_OK;
        for (int k = 0; k < 9; ++k) A->q1g_v[k] = (double)ref[k];
        A->q1g_vb = (double)ref[9];
        A->q1g_m = m;
        return HB2_OK;
    }

    int ell_find_q1_grid(hb2_ell_s * A, cudaStream_t stream)
    {
        A->q1g_m = A->g9_m = 0;
        if (A->rows != A->cols || A->K != 9 || A->rows < 9 || A->rows >= (1ull << 31)) return HB2_OK;
        uint64_t m = 3;
        while (m * m < A->rows) ++m;
        if (m * m != A->rows) return HB2_OK;
        return A->dtype == HB2_F64 ? find_grid_typed<double>(A, (uint32_t)m, stream)
                                   : find_grid_typed<float>(A, (uint32_t)m, stream);
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
        // (level 10: 11.9 / 15.3 us against 12.3 / 13.6; level 9: 6.9 / 9.4 against 8.5 / 9.9)
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
    // passes.  From 2^16 rows up: below, the one-row-per-thread kernels are as fast and their
    // layout was timed at creation.  Measured (B200), FP64 level 11: defect + norm 37.2 us
    // with the gather kernel, 26.6 as a streaming pass (a call, partial sums included).
    bool q1_single_applies(const hb2_ell_s * A, int mode)
    {
        return A->q1g_m >= 257 && (mode == kPlain || mode == kDefect || mode == kDot);
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
