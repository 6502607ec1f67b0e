// The bottom of a V-cycle over Q1 grid operators in one thread block: the levels of at most
// 33 x 33 points above the coarsest, and the coarsest CG (math/mg.hh:577-640).
//
// These levels have too few nodes to fill one SM, so a launch each way and per level is all
// latency: as sweep passes a level-5 grid cost about 4.7 us a pass, a level-4 one the same or
// 4 us as a cluster kernel, and the coarse solve a launch of its own between them.  Here the
// iterates live in shared memory and a phase (one sweep, the defect, a transfer) costs one
// block barrier.  A thread owns a few consecutive rows of one column, so a sweep reads three
// values a row and two more rows instead of nine a node; rhs and iterate stay in registers from
// phase to phase of a level.  256 threads, so that the coarse CG's warp may use 255 registers.
// Every node is computed with the products and slot-ordered sums of the single kernels: the
// bits are the same.
#include "cg_warp.cuh"

namespace hb2
{
    constexpr int kBottomThreads = 256;
    constexpr int kBottomRows = 5;      // rows a thread: 33 columns x 7 strips of 5 rows

    template <typename T>
    struct BottomLevel
    {
        T v[9], vb;
        const T * jac;
        int m;
    };

    template <typename T>
    struct BottomArgs
    {
        BottomLevel<T> lev[kQ1BottomLevels + 1];    // lev[0]: the coarsest (m only)
        int top, n_pre, n_post, zero_guess;
        const T * b;                                // of level top
        T * x;
        EllView<T> C;                               // coarsest operator
        EllView<double> C64;                        // its FP64 copy (mixed)
        int mixed, exact;
        int grid9;                                  // the coarsest is a 9 x 9 Q1 grid operator with equal
        double cv0, cv4, cvb;                       // couplings, solved in FP64 by cg_warp_grid9
        uint64_t max_iters;
        double eps;
        uint64_t * used;
        double * defect;
    };

    // a thread's nodes of a level: column j, rows i0 .. i0 + rows)
    struct BottomNodes
    {
        int m, j, i0, rows;
        __device__ __forceinline__ BottomNodes(int m_) : m(m_)
        {
            const int strips = kBottomThreads / m, per = (m + strips - 1) / strips, s = (int)threadIdx.x / m;
            j = (int)threadIdx.x - s * m;
            i0 = s * per;
            rows = s < strips ? max(0, min(per, m - i0)) : 0;
        }
    };

    // A x of R rows from the thread's first one, x in shared memory.  Without branches: rows
    // and columns outside the grid read a clamped neighbour and boundary rows are selected at
    // the end, so the chains of all rows run side by side.  UNI: all couplings equal, one
    // product per value.
    template <typename T, bool UNI, int R>
    __device__ __forceinline__ void bottom_product(const BottomLevel<T> & L, const BottomNodes & o, const T * x, T (&ax)[R],
                                                   T (&xc)[R])
    {
        typedef Arith<T> M;
        const int jw = max(o.j - 1, 0), je = min(o.j + 1, o.m - 1);
        const bool ecol = o.j == 0 || o.j == o.m - 1;
        T w[R + 2], c[R + 2], e[R + 2], pc[R + 2];
#pragma unroll
        for (int k = 0; k < R + 2; ++k)
        {
            const T * r = x + min(max(o.i0 + k - 1, 0), o.m - 1) * o.m;
            w[k] = r[jw];
            c[k] = r[o.j];
            e[k] = r[je];
        }
        if (UNI)
        {
#pragma unroll
            for (int k = 0; k < R + 2; ++k)
            {
                w[k] = M::fma(L.v[0], w[k], T(0));      // the sum 0 + p of the first slot folded in
                pc[k] = M::fma(L.v[0], c[k], T(0));
                e[k] = M::fma(L.v[0], e[k], T(0));
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
        {
            T s;
            if (UNI)
            {
                s = M::add(M::add(w[k], pc[k]), e[k]);
                s = M::add(M::add(M::add(s, w[k + 1]), M::mul(L.v[4], c[k + 1])), e[k + 1]);
                s = M::add(M::add(M::add(s, w[k + 2]), pc[k + 2]), e[k + 2]);
            }
            else
            {
                s = M::add(T(0), M::mul(L.v[0], w[k]));
                s = M::add(s, M::mul(L.v[1], c[k]));
                s = M::add(s, M::mul(L.v[2], e[k]));
                s = M::add(s, M::mul(L.v[3], w[k + 1]));
                s = M::add(s, M::mul(L.v[4], c[k + 1]));
                s = M::add(s, M::mul(L.v[5], e[k + 1]));
                s = M::add(s, M::mul(L.v[6], w[k + 2]));
                s = M::add(s, M::mul(L.v[7], c[k + 2]));
                s = M::add(s, M::mul(L.v[8], e[k + 2]));
            }
            const int i = o.i0 + k;
            xc[k] = c[k + 1];
            ax[k] = ecol || i == 0 || i >= o.m - 1 ? M::add(T(0), M::mul(L.vb, c[k + 1])) : s;
        }
    }

    // `sweeps` Jacobi sweeps from x0 (in shared memory) with ping-pong into x1, and with
    // DEFECT the defect of the result into the buffer that is then free; returns the buffer
    // that holds the result
    template <typename T, bool UNI, int R, bool DEFECT>
    __device__ __forceinline__ T * bottom_smooth_r(const BottomLevel<T> & L, const BottomNodes & o, T * x0, T * x1,
                                                   const T * b, int sweeps)
    {
        typedef Arith<T> M;
        const T Pi = L.jac[L.m + 1], Pb = L.jac[0];
        const bool ecol = o.j == 0 || o.j == o.m - 1;
        T rhs[R], P[R];
#pragma unroll
        for (int k = 0; k < R; ++k)
        {
            const int i = o.i0 + k;
            rhs[k] = k < o.rows ? b[i * o.m + o.j] : T(0);
            P[k] = ecol || i == 0 || i == o.m - 1 ? Pb : Pi;
        }
        T ax[R], xc[R];
        for (int s = 0; s < sweeps; ++s)
        {
            bottom_product<T, UNI, R>(L, o, x0, ax, xc);
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (k < o.rows) x1[(o.i0 + k) * o.m + o.j] = M::add(xc[k], M::mul(P[k], M::sub(rhs[k], ax[k])));
            __syncthreads();
            T * t = x0;
            x0 = x1;
            x1 = t;
        }
        if (DEFECT)
        {
            bottom_product<T, UNI, R>(L, o, x0, ax, xc);
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (k < o.rows) x1[(o.i0 + k) * o.m + o.j] = M::sub(rhs[k], ax[k]);
            __syncthreads();
        }
        return x0;
    }

    template <typename T, bool UNI, bool DEFECT>
    __device__ __forceinline__ T * bottom_smooth(const BottomLevel<T> & L, T * x0, T * x1, const T * b, int sweeps)
    {
        const BottomNodes o(L.m);
        return L.m > 2 * (kBottomThreads / L.m) ? bottom_smooth_r<T, UNI, kBottomRows, DEFECT>(L, o, x0, x1, b, sweeps)
                                                : bottom_smooth_r<T, UNI, 2, DEFECT>(L, o, x0, x1, b, sweeps);
    }

    template <typename TA, typename S>
    __device__ __forceinline__ void bottom_coarse(const EllView<TA> & A, const S * b, S * x, uint64_t max_iters, double eps,
                                                  int exact, uint64_t * used, double * defect, TA * smem)
    {
        switch ((A.rows + 31) / 32)
        {
            case 1: cg_warp_reg<TA, S, 1>(A, b, x, max_iters, eps, exact, used, defect, smem); break;
            case 2: cg_warp_reg<TA, S, 2>(A, b, x, max_iters, eps, exact, used, defect, smem); break;
            default: cg_warp_reg<TA, S, 3>(A, b, x, max_iters, eps, exact, used, defect, smem); break;
        }
    }

    template <typename T, bool MIXED, bool UNI>
    __global__ void __launch_bounds__(kBottomThreads, 1) q1_bottom_kernel(const __grid_constant__ BottomArgs<T> g)
    {
        typedef Arith<T> M;
        extern __shared__ __align__(16) unsigned char bottom_smem[];
        double * cgs = reinterpret_cast<double *>(bottom_smem);          // 3 * 96 + 1 for the CG
        T * mem = reinterpret_cast<T *>(cgs + 3 * 96 + 2);
        // per level: two iterates and the right-hand side, the coarsest first (x, b)
        T * xs[kQ1BottomLevels + 1], * ts[kQ1BottomLevels + 1], * bs[kQ1BottomLevels + 1];
#pragma unroll
        for (int l = 0; l <= kQ1BottomLevels; ++l)
        {
            const int n = l <= g.top ? g.lev[l].m * g.lev[l].m : 0;
            xs[l] = mem;
            ts[l] = mem + n;
            bs[l] = mem + 2 * n;
            mem += 3 * n;
        }
        pdl_entry();
#pragma unroll
        for (int l = kQ1BottomLevels; l >= 1; --l)
        {
            if (l > g.top) continue;
            const BottomLevel<T> & L = g.lev[l];
            const int n = L.m * L.m;
            if (l == g.top)
                for (int q = threadIdx.x; q < n; q += kBottomThreads)
                {
                    bs[l][q] = g.b[q];
                    xs[l][q] = g.zero_guess ? T(0) : g.x[q];
                }
            __syncthreads();
            T * cur = bottom_smooth<T, UNI, true>(L, xs[l], ts[l], bs[l], g.n_pre);
            T * r = cur == xs[l] ? ts[l] : xs[l];
            const int mc = g.lev[l - 1].m;
            for (int q = threadIdx.x; q < mc * mc; q += kBottomThreads)
            {
                bs[l - 1][q] = q1_restrict_row<T, false>(q, r, L.m, mc);
                xs[l - 1][q] = T(0);
            }
            __syncthreads();
            ts[l] = r;          // xs: the iterate, ts: free
            xs[l] = cur;
        }
        if (threadIdx.x < 32 && g.grid9)
            cg_warp_grid9<T>(g.cv0, g.cv4, g.cvb, bs[0], xs[0], g.max_iters, g.eps, g.used, g.defect, cgs);
        else if (threadIdx.x < 32)
        {
            if constexpr (MIXED)
                bottom_coarse<double, T>(g.C64, bs[0], xs[0], g.max_iters, g.eps, g.exact, g.used, g.defect, cgs);
            else
                bottom_coarse<T, T>(g.C, bs[0], xs[0], g.max_iters, g.eps, g.exact, g.used, g.defect, (T *)cgs);
        }
        __syncthreads();
#pragma unroll
        for (int l = 1; l <= kQ1BottomLevels; ++l)
        {
            if (l > g.top) continue;
            const BottomLevel<T> & L = g.lev[l];
            const int n = L.m * L.m;
            for (int q = threadIdx.x; q < n; q += kBottomThreads)
                xs[l][q] = M::add(xs[l][q], q1_prolong_row<T, false>(q, xs[l - 1], L.m, g.lev[l - 1].m));
            __syncthreads();
            xs[l] = bottom_smooth<T, UNI, false>(L, xs[l], ts[l], bs[l], g.n_post);
            if (l == g.top)
                for (int q = threadIdx.x; q < n; q += kBottomThreads) g.x[q] = xs[l][q];
        }
    }

    bool q1_bottom_fits(const hb2_ell_s * A) { return A->q1g_m >= 3 && A->q1g_m <= 33; }
    bool q1_bottom_coarse_fits(const hb2_ell_s * C) { return C->rows <= 96 && C->K >= 1 && C->K <= 9; }

    template <typename T>
    static int launch_typed(const Q1Bottom & p, cudaStream_t s)
    {
        BottomArgs<T> g = {};
        size_t elems = 0;
        g.lev[0].m = (int)((p.A[1]->q1g_m + 1) / 2);
        for (int l = 0; l <= p.top; ++l)
        {
            if (l > 0)
            {
                for (int k = 0; k < 9; ++k) g.lev[l].v[k] = (T)p.A[l]->q1g_v[k];
                g.lev[l].vb = (T)p.A[l]->q1g_vb;
                g.lev[l].m = (int)p.A[l]->q1g_m;
                g.lev[l].jac = (const T *)p.jac[l];
            }
            elems += 3 * (size_t)g.lev[l].m * g.lev[l].m;
        }
        g.top = p.top;
        g.n_pre = p.n_pre;
        g.n_post = p.n_post;
        g.zero_guess = p.zero_guess;
        g.b = (const T *)p.b;
        g.x = (T *)p.x;
        g.C = p.A[0]->view<T>();
        if (p.coarse64) g.C64 = p.coarse64->view<double>();
        g.exact = p.exact;
        // FP64 and the reordered recurrence only: the other modes sum in a given order.  Of the
        // sizes that fit one warp 9 x 9 is the one a hierarchy ends on by default (level 3).
        const hb2_ell_s * C = p.coarse64 ? p.coarse64 : p.A[0];
        g.grid9 = C->dtype == HB2_F64 && C->q1g_m == 9 && p.exact == kCgTreeOneReduction;
        for (int k = 0; k < 9; ++k) g.grid9 = g.grid9 && (k == 4 || C->q1g_v[k] == C->q1g_v[0]);
        g.cv0 = C->q1g_v[0];
        g.cv4 = C->q1g_v[4];
        g.cvb = C->q1g_vb;
        g.max_iters = p.max_iters;
        g.eps = p.eps;
        g.used = p.used;
        g.defect = p.defect;
        const size_t smem = (3 * 96 + 2) * sizeof(double) + elems * sizeof(T);
        bool uni = true;
        for (int l = 1; l <= p.top; ++l)
            for (int k = 0; k < 9; ++k) uni = uni && (k == 4 || p.A[l]->q1g_v[k] == p.A[l]->q1g_v[0]);
#define HB2_BOTTOM(M_, U_) launch_pdl(q1_bottom_kernel<T, M_, U_>, dim3(1), dim3(kBottomThreads), smem, s, g)
        if (p.coarse64) { if (uni) HB2_BOTTOM(true, true); else HB2_BOTTOM(true, false); }
        else { if (uni) HB2_BOTTOM(false, true); else HB2_BOTTOM(false, false); }
#undef HB2_BOTTOM
        count_launches(1);
        HB2_LAUNCH_CHECK("V-cycle bottom launch");
        return HB2_OK;
    }

    int launch_q1_bottom(int dtype, const Q1Bottom & p, cudaStream_t s)
    {
        return dtype == HB2_F64 ? launch_typed<double>(p, s) : launch_typed<float>(p, s);
    }
}
