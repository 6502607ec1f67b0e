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

    // A x of the thread's rows, x in shared memory
    template <typename T>
    __device__ __forceinline__ void bottom_product(const BottomLevel<T> & L, const BottomNodes & o, const T * x,
                                                   T (&ax)[kBottomRows], T (&xc)[kBottomRows])
    {
        typedef Arith<T> M;
        const bool ecol = o.j == 0 || o.j == o.m - 1;
        T w[3], c[3], e[3];                 // rows i - 1, i, i + 1
        auto load = [&](int k, int i) {
            const bool ok = i >= 0 && i < o.m;
            const T * r = x + i * o.m + o.j;
            w[k] = ok && ! ecol ? r[-1] : T(0);
            c[k] = ok ? r[0] : T(0);
            e[k] = ok && ! ecol ? r[1] : T(0);
        };
        if (o.rows == 0) return;
        load(0, o.i0 - 1);
        load(1, o.i0);
#pragma unroll
        for (int k = 0; k < kBottomRows; ++k)
        {
            if (k >= o.rows) break;
            const int i = o.i0 + k;
            load((k + 2) % 3, i + 1);
            const int a = k % 3, b = (k + 1) % 3, d = (k + 2) % 3;
            xc[k] = c[b];
            if (ecol || i == 0 || i == o.m - 1) ax[k] = M::add(T(0), M::mul(L.vb, c[b]));
            else
            {
                T s = M::add(T(0), M::mul(L.v[0], w[a]));
                s = M::add(s, M::mul(L.v[1], c[a]));
                s = M::add(s, M::mul(L.v[2], e[a]));
                s = M::add(s, M::mul(L.v[3], w[b]));
                s = M::add(s, M::mul(L.v[4], c[b]));
                s = M::add(s, M::mul(L.v[5], e[b]));
                s = M::add(s, M::mul(L.v[6], w[d]));
                s = M::add(s, M::mul(L.v[7], c[d]));
                ax[k] = M::add(s, M::mul(L.v[8], e[d]));
            }
        }
    }

    // `sweeps` Jacobi sweeps from x0 (in shared memory) with ping-pong into x1; returns the
    // buffer that holds the result
    template <typename T>
    __device__ __forceinline__ T * bottom_smooth(const BottomLevel<T> & L, const BottomNodes & o, T * x0, T * x1, const T * b,
                                                 int sweeps)
    {
        typedef Arith<T> M;
        const T Pi = L.jac[L.m + 1], Pb = L.jac[0];
        for (int s = 0; s < sweeps; ++s)
        {
            T ax[kBottomRows], xc[kBottomRows];
            bottom_product(L, o, x0, ax, xc);
#pragma unroll
            for (int k = 0; k < kBottomRows; ++k)
                if (k < o.rows)
                {
                    const int i = o.i0 + k, q = i * o.m + o.j;
                    const T P = i == 0 || i == o.m - 1 || o.j == 0 || o.j == o.m - 1 ? Pb : Pi;
                    x1[q] = M::add(xc[k], M::mul(P, M::sub(b[q], ax[k])));
                }
            __syncthreads();
            T * t = x0;
            x0 = x1;
            x1 = t;
        }
        return x0;
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

    template <typename T, bool MIXED>
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
            const BottomNodes o(L.m);
            T * cur = bottom_smooth(L, o, xs[l], ts[l], bs[l], g.n_pre);
            T * r = cur == xs[l] ? ts[l] : xs[l];
            T ax[kBottomRows], xc[kBottomRows];
            bottom_product(L, o, cur, ax, xc);
#pragma unroll
            for (int k = 0; k < kBottomRows; ++k)
                if (k < o.rows)
                {
                    const int q = (o.i0 + k) * o.m + o.j;
                    r[q] = M::sub(bs[l][q], ax[k]);
                }
            __syncthreads();
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
        if (threadIdx.x < 32)
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
            const BottomNodes o(L.m);
            xs[l] = bottom_smooth(L, o, xs[l], ts[l], bs[l], g.n_post);
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
        g.max_iters = p.max_iters;
        g.eps = p.eps;
        g.used = p.used;
        g.defect = p.defect;
        const size_t smem = (3 * 96 + 2) * sizeof(double) + elems * sizeof(T);
        if (p.coarse64) launch_pdl(q1_bottom_kernel<T, true>, dim3(1), dim3(kBottomThreads), smem, s, g);
        else launch_pdl(q1_bottom_kernel<T, false>, dim3(1), dim3(kBottomThreads), smem, s, g);
        count_launches(1);
        HB2_LAUNCH_CHECK("V-cycle bottom launch");
        return HB2_OK;
    }

    int launch_q1_bottom(int dtype, const Q1Bottom & p, cudaStream_t s)
    {
        return dtype == HB2_F64 ? launch_typed<double>(p, s) : launch_typed<float>(p, s);
    }
}
