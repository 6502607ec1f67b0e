// One-warp CG (CGSolver<Tag, methods::NONE>, math/cg.hh:64-135) for the
// smallest systems -- the MG coarsest level -- shared by the stand-alone
// coarse-solve kernels (cg.cu) and the fused small-level V-cycle (subcycle.cu).
#pragma once

#include <cfloat>
#include <type_traits>

#include "hb2_common.cuh"
#include "hb2_internal.hh"

namespace hb2
{
    template <typename T> struct Eps;
    template <> struct Eps<double> { static __device__ __forceinline__ double v() { return DBL_EPSILON; } };
    template <> struct Eps<float> { static __device__ __forceinline__ float v() { return FLT_EPSILON; } };

    // the `exact` argument of the coarse CG: the reference's sequential fma order
    // (bit-identical to it); the standard recurrence with tree-ordered dots; the
    // Chronopoulos-Gear recurrence with one fused reduction per iteration
    constexpr int kCgTreeOneReduction = 0;
    constexpr int kCgExact = 1;
    constexpr int kCgTreeStandard = 2;

    template <typename T> struct Recip;
    template <> struct Recip<double> { static __device__ __forceinline__ double rn(double v) { return __drcp_rn(v); } };
    template <> struct Recip<float> { static __device__ __forceinline__ float rn(float v) { return __frcp_rn(v); } };

    template <typename T>
    __device__ __forceinline__ T guard(T d)
    {
        return fabs(d) > Eps<T>::v() ? d : Eps<T>::v();
    }

    // The sum of v over the warp, in every lane, by two FP64 tensor-core products instead of
    // five shuffle rounds: ones(8x4) * B(4x8) with lane l's value in B[l % 4][l / 4] sums
    // groups of four lanes, each lane receives two neighbouring groups' sums and adds them,
    // and S(8x4) * ones(4x8) sums those four values.  Measured (B200): 66 cycles against 176
    // (a 64-bit shuffle and its add take 35, a product 29).  Every product is by one, so the
    // result is a sum of the 32 values in a fixed order.  Volatile: every lane has to take part
    // where the call stands, so the compiler must not sink it into a branch that alone uses the
    // result (the callers' "if (lane == 0) ... = sum").
    __device__ __forceinline__ double warp_sum_mma(double v)
    {
        double d0, d1, e0, e1;
        const double one = 1.0, zero = 0.0;
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %5};"
                     : "=d"(d0), "=d"(d1) : "d"(one), "d"(v), "d"(zero), "d"(zero));
        const double s = d0 + d1;
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%4, %5};"
                     : "=d"(e0), "=d"(e1) : "d"(s), "d"(one), "d"(zero), "d"(zero));
        return e0;
    }

    // the same for two values, whose instructions overlap (volatile ones keep their order)
    __device__ __forceinline__ void warp_sum_mma2(double & a, double & b)
    {
        double a0, a1, b0, b1;
        const double one = 1.0, zero = 0.0;
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%4}, {%5}, {%7, %7};\n\t"
                     "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%2, %3}, {%4}, {%6}, {%7, %7};"
                     : "=&d"(a0), "=&d"(a1), "=&d"(b0), "=&d"(b1) : "d"(one), "d"(a), "d"(b), "d"(zero));
        const double s = a0 + a1, t = b0 + b1;
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%4}, {%6}, {%7, %7};\n\t"
                     "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%2, %3}, {%5}, {%6}, {%7, %7};"
                     : "=&d"(a0), "=&d"(a1), "=&d"(b0), "=&d"(b1) : "d"(s), "d"(t), "d"(one), "d"(zero));
        a = a0;
        b = b0;
    }

    // ------------------------------------------------------------------ one warp
    // Latency-bound coarse solves (the MG coarsest level has 81 unknowns and runs
    // a hundred iterations per V-cycle): one warp, no block barriers, reductions
    // by shuffles.  The reference-order dot is one fma chain in lane 0 with the
    // operands fetched ahead of the chain.
    template <typename T>
    __device__ __forceinline__ T warp_dot_exact(const T * a, const T * b, int n)
    {
        T s = T(0);
        if ((threadIdx.x & 31) == 0)
        {
            int i = 0;
            for (; i + 8 <= n; i += 8)
            {
                T a0 = a[i], a1 = a[i + 1], a2 = a[i + 2], a3 = a[i + 3], a4 = a[i + 4], a5 = a[i + 5], a6 = a[i + 6],
                  a7 = a[i + 7];
                T b0 = b[i], b1 = b[i + 1], b2 = b[i + 2], b3 = b[i + 3], b4 = b[i + 4], b5 = b[i + 5], b6 = b[i + 6],
                  b7 = b[i + 7];
                s = Arith<T>::fma(a0, b0, s);
                s = Arith<T>::fma(a1, b1, s);
                s = Arith<T>::fma(a2, b2, s);
                s = Arith<T>::fma(a3, b3, s);
                s = Arith<T>::fma(a4, b4, s);
                s = Arith<T>::fma(a5, b5, s);
                s = Arith<T>::fma(a6, b6, s);
                s = Arith<T>::fma(a7, b7, s);
            }
            for (; i < n; ++i) s = Arith<T>::fma(a[i], b[i], s);
        }
        return __shfl_sync(0xffffffffu, s, 0);
    }

    // Register-resident variant for the smallest systems (n <= 32 * RPL, K = 9):
    // each lane keeps its RPL rows of A and of x, r, p, v in registers; only p
    // (gathered by the SpMV) and, for the reference-order dots, the dot operands
    // go through shared memory.
    // T: arithmetic and matrix type; S: element type of b and x in memory (an
    // FP32 hierarchy can run its coarsest solve in FP64 on an FP64 copy of the
    // coarse operator: b is widened on load, x rounded on store).
    //
    // cg_warp_reg runs in one full warp (lane = threadIdx.x & 31) and needs 3n + 1
    // elements of T in shared memory; it is called by cg_warp_reg_kernel and by
    // the fused small-level V-cycle kernel (subcycle.cu), which writes b earlier
    // in the same launch -- hence plain (coherent) loads of b, no __restrict__.
    template <typename T, typename S, int RPL>
    __device__ __forceinline__ void cg_warp_reg(const EllView<T> & Ag, const S * b, S * xg,
                                                uint64_t max_iters, double eps_d, int exact, uint64_t * used_out,
                                                double * defect_out, T * smem)
    {
        typedef Arith<T> M;
        constexpr int K = 9;
        const int n = (int)Ag.rows, lane = threadIdx.x & 31;
        // p (and x for the initial defect), then a zero that empty slots gather; the tree
        // modes alternate between two such vectors, so that one barrier an iteration orders
        // the gathers of the old one before the writes of the new one
        T * sp = smem;
        T * sp2 = sp + n + 1;
        T * sa = sp + n;          // first dot operand (exact mode, which has no such zero)
        T * sb = sa + n;          // second dot operand (exact mode)
        T av[RPL][K];
        int ac[RPL][K];
        T xr[RPL], rr[RPL], pr[RPL], vr[RPL];
#pragma unroll
        for (int j = 0; j < RPL; ++j)
        {
            const int row = lane + 32 * j;
            const bool ok = row < n;
#pragma unroll
            for (int k = 0; k < K; ++k)
            {
                const bool okk = ok && k < (int)Ag.K;     // up to 9 slots; the missing ones are skipped
                av[j][k] = okk ? Ag.val[(uint64_t)k * Ag.ld + row] : T(0);
                ac[j][k] = okk ? Ag.col[(uint64_t)k * Ag.ld + row] : -1;
            }
            xr[j] = ok ? T(xg[row]) : T(0);
            if (ok) sp[row] = xr[j];
        }
        __syncwarp();
        auto spmv = [&](T (&out)[RPL]) {
#pragma unroll
            for (int j = 0; j < RPL; ++j)
            {
                T s = T(0);
#pragma unroll
                for (int k = 0; k < K; ++k)
                    if (ac[j][k] >= 0) s = M::add(s, M::mul(av[j][k], sp[ac[j][k]]));
                out[j] = s;
            }
        };
        // dot of per-lane register vectors a, b over the valid rows; `order` is a constant, so that
        // neither mode's loop carries the other's instructions
        auto dot = [&](const T (&a)[RPL], const T (&bb)[RPL], auto order) -> T {
            if constexpr (decltype(order)::value)
            {
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                {
                    const int row = lane + 32 * j;
                    if (row < n) { sa[row] = a[j]; sb[row] = bb[j]; }
                }
                __syncwarp();
                T s = warp_dot_exact(sa, sb, n);
                __syncwarp();
                return s;
            }
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < RPL; ++j)
                if (lane + 32 * j < n) s = fma((double)a[j], (double)bb[j], s);
            return (T)warp_sum_mma(s);
        };
        // the tree modes' product: three chains of three fused terms a row, no branches
        auto spmv_tree = [&](T (&out)[RPL], const T * v) {
#pragma unroll
            for (int j = 0; j < RPL; ++j)
            {
                T s[3];
#pragma unroll
                for (int q = 0; q < 3; ++q)
                {
                    s[q] = M::mul(av[j][3 * q], v[ac[j][3 * q] >= 0 ? ac[j][3 * q] : n]);
                    s[q] = M::fma(av[j][3 * q + 1], v[ac[j][3 * q + 1] >= 0 ? ac[j][3 * q + 1] : n], s[q]);
                    s[q] = M::fma(av[j][3 * q + 2], v[ac[j][3 * q + 2] >= 0 ? ac[j][3 * q + 2] : n], s[q]);
                }
                out[j] = M::add(M::add(s[0], s[1]), s[2]);
            }
        };
        T tmp[RPL];
        spmv(tmp);
        __syncwarp();
#pragma unroll
        for (int j = 0; j < RPL; ++j)
        {
            const int row = lane + 32 * j;
            rr[j] = row < n ? M::sub(T(b[row]), tmp[j]) : T(0);
            pr[j] = rr[j];
            if (row < n) sp[row] = pr[j];
        }
        if (exact != kCgExact && lane == 0) sp[n] = sp2[n] = T(0);     // (the exact mode's dots use this memory)
        __syncwarp();
        const T eps = T(eps_d);
        T alpha = exact == kCgExact ? dot(rr, rr, std::true_type()) : dot(rr, rr, std::false_type());
        const T initial = sqrt(alpha);
        T current = initial;
        uint64_t it = 0, used = 0;
        if (exact == kCgTreeOneReduction && max_iters > 0)
        {
            // Chronopoulos-Gear recurrence (the same iterates as the loop below in
            // exact arithmetic): per iteration one product w = A r and both dots
            // (r, r), (w, r) in one shuffle tree, so the chain of an iteration holds
            // one reduction and one division instead of two of each; the
            // reciprocals the next iteration needs are formed off that chain.
            //   x += a p; r -= a s; w = A r; g = (r, r); d = (w, r);
            //   b = g / g_old; a = g / (d - b g / a_old); p = r + b p; s = w + b s
            T sr[RPL], wr[RPL];
            spmv_tree(wr, sp);   // w0 = A r0 (sp holds r0 = p0)
            T gam = alpha, del;
            {
                double s1 = 0.0;
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                    if (lane + 32 * j < n) s1 = fma((double)wr[j], (double)rr[j], s1);
                del = (T)warp_sum_mma(s1);
            }
            T a = M::div(gam, guard(del));
            T inv_a = Recip<T>::rn(guard(a)), inv_g = Recip<T>::rn(guard(gam));
            // the stop test on squared norms: no square root on the iteration's chain
            const T thr = M::mul(eps, initial), thr2 = M::mul(thr, thr), eps2 = M::mul(eps, eps);
#pragma unroll
            for (int j = 0; j < RPL; ++j) sr[j] = wr[j];
            const T inv_eps = Recip<T>::rn(Eps<T>::v());
            T * cur = sp, * nxt = sp2;
            while (it < max_iters)
            {
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                {
                    rr[j] = M::fma(-a, sr[j], rr[j]);
                    if (lane + 32 * j < n) nxt[lane + 32 * j] = rr[j];
                }
                __syncwarp();
                // ||r||^2 while the product's gathers are on their way
                double s1 = 0.0, s2 = 0.0;
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                    if (lane + 32 * j < n) s1 = fma((double)rr[j], (double)rr[j], s1);
                const T g = (T)warp_sum_mma(s1);
                spmv_tree(wr, nxt);
#pragma unroll
                for (int j = 0; j < RPL; ++j) xr[j] = M::fma(a, pr[j], xr[j]);
                T * t = cur;
                cur = nxt;
                nxt = t;
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                    if (lane + 32 * j < n) s2 = fma((double)wr[j], (double)rr[j], s2);
                del = (T)warp_sum_mma(s2);
                ++it;
                // single-rounded reciprocals instead of IEEE divisions (this mode is not the
                // reference's order anyway).  A warp issues in order, so what the next step
                // needs is formed before the sum (w, r) arrives -- b, 1/g and with them p and s --
                // and 1/a as t/g, not by a third reciprocal behind a
                const T b = M::mul(g, inv_g), bg = M::mul(M::mul(b, g), inv_a);
                const T ig = Recip<T>::rn(guard(g));
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                {
                    pr[j] = M::fma(b, pr[j], rr[j]);
                    sr[j] = M::fma(b, sr[j], wr[j]);
                }
                if (g < thr2 || g < eps2 || it == max_iters)
                {
                    current = sqrt(g);
                    used = it;
                    break;
                }
                const T d = guard(M::sub(del, bg));
                a = M::mul(g, Recip<T>::rn(d));
                inv_g = ig;
                inv_a = fabs(a) > Eps<T>::v() ? M::mul(d, ig) : inv_eps;
            }
            it = max_iters;   // done: skip the loop below
        }
        auto standard = [&](auto order) {
            constexpr bool EXACT = decltype(order)::value;
            while (it < max_iters)
            {
                // the tree-ordered mode takes the fused product and reciprocals, that of the old
                // alpha while the product's dot is on its way
                T inv_alpha = T(0);
                if constexpr (EXACT) spmv(vr);
                else
                {
                    spmv_tree(vr, sp);
                    inv_alpha = Recip<T>::rn(guard(alpha));
                }
                const T temp = dot(vr, pr, order);
                const T lambda = EXACT ? M::div(alpha, guard(temp)) : M::mul(alpha, Recip<T>::rn(guard(temp)));
                const T mlambda = -lambda;
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                {
                    xr[j] = M::add(xr[j], M::mul(lambda, pr[j]));
                    rr[j] = M::add(rr[j], M::mul(mlambda, vr[j]));
                }
                const T alpha_old = alpha;
                alpha = dot(rr, rr, order);
                const T talpha = EXACT ? M::div(alpha, guard(alpha_old)) : M::mul(alpha, inv_alpha);
                __syncwarp();   // every lane is done gathering the old p
#pragma unroll
                for (int j = 0; j < RPL; ++j)
                {
                    const int row = lane + 32 * j;
                    pr[j] = M::add(M::mul(pr[j], talpha), rr[j]);
                    if (row < n) sp[row] = pr[j];
                }
                __syncwarp();
                ++it;
                current = sqrt(alpha);
                if (current < M::mul(eps, initial) || current < eps) { used = it; break; }
                if (it == max_iters) used = it;
            }
        };
        if (exact == kCgExact) standard(std::true_type());
        else standard(std::false_type());
#pragma unroll
        for (int j = 0; j < RPL; ++j)
            if (lane + 32 * j < n) xg[lane + 32 * j] = S(xr[j]);
        if (lane == 0)
        {
            if (used_out) *used_out = used;
            if (defect_out) *defect_out = (double)current;
        }
    }

    // The one-reduction recurrence of cg_warp_reg (kCgTreeOneReduction) on a 9 x 9 Q1 grid
    // operator with equal couplings (interior diagonal v4, couplings v0, boundary diagonal vb),
    // FP64 arithmetic, one warp.  A lane owns three rows of one column (27 lanes), so a product
    // gathers 12 values instead of 27, keeps no matrix in registers and shares the line sums of
    // its rows.  Bound by the dependent chain of an iteration (two warp sums, a reciprocal, the
    // gather); measured (B200): 0.29 -> 0.26 us an iteration, a level-6 solve of 7 cycles 442 ->
    // 419 us, of level 10 with 8 cycles 1,354 -> 1,289.  smem: 2 x 81 doubles.
    template <typename S>
    __device__ __forceinline__ void cg_warp_grid9(double v0, double v4, double vb, const S * b, S * xg, uint64_t max_iters,
                                                  double eps, uint64_t * used_out, double * defect_out, double * smem)
    {
        typedef Arith<double> M;
        constexpr int m = 9, R = 3;
        const int lane = threadIdx.x & 31, j = lane % m, i0 = lane / m * R;
        const bool live = lane < m * (m / R);
        const int jw = max(j - 1, 0), je = min(j + 1, m - 1);
        int at[R + 2];          // the lines around the lane's rows
        bool edge[R];
#pragma unroll
        for (int k = 0; k < R + 2; ++k) at[k] = min(max(i0 + k - 1, 0), m - 1) * m;
#pragma unroll
        for (int k = 0; k < R; ++k) edge[k] = j == 0 || j == m - 1 || i0 + k == 0 || i0 + k >= m - 1;
        auto product = [&](double (&out)[R], const double * v, const double (&own)[R]) {
            double h[R + 2], H[R + 2];
#pragma unroll
            for (int k = 0; k < R + 2; ++k)
            {
                const double c = k >= 1 && k <= R ? own[k >= 1 && k <= R ? k - 1 : 0] : v[at[k] + j];
                h[k] = M::add(v[at[k] + jw], v[at[k] + je]);
                H[k] = M::add(h[k], c);
            }
#pragma unroll
            for (int k = 0; k < R; ++k)
            {
                const double s = M::fma(v0, M::add(M::add(H[k], H[k + 2]), h[k + 1]), M::mul(v4, own[k]));
                out[k] = edge[k] ? M::mul(vb, own[k]) : s;
            }
        };
        auto store = [&](double * v, const double (&a)[R]) {
#pragma unroll
            for (int k = 0; k < R; ++k)
                if (live) v[(i0 + k) * m + j] = a[k];
        };
        auto dot = [&](const double (&a)[R], const double (&c)[R]) -> double {
            double s = 0.0;
#pragma unroll
            for (int k = 0; k < R; ++k) s = fma(a[k], c[k], s);
            return warp_sum_mma(live ? s : 0.0);
        };
        double * cur = smem, * nxt = smem + m * m;
        double xr[R], rr[R], pr[R], sr[R], wr[R];
#pragma unroll
        for (int k = 0; k < R; ++k) xr[k] = live ? (double)xg[(i0 + k) * m + j] : 0.0;
        store(cur, xr);
        __syncwarp();
        product(wr, cur, xr);
#pragma unroll
        for (int k = 0; k < R; ++k) pr[k] = rr[k] = live ? M::sub((double)b[(i0 + k) * m + j], wr[k]) : 0.0;
        store(nxt, rr);
        __syncwarp();
        double g = dot(rr, rr);
        const double initial = sqrt(g);
        double current = initial;
        uint64_t it = 0, used = 0;
        if (max_iters > 0)
        {
            product(wr, nxt, rr);
            double a = M::div(g, guard(dot(wr, rr)));
            double inv_a = Recip<double>::rn(guard(a)), inv_g = Recip<double>::rn(guard(g));
            const double thr = M::mul(eps, initial), thr2 = M::mul(thr, thr), eps2 = M::mul(eps, eps);
            const double inv_eps = Recip<double>::rn(Eps<double>::v());
#pragma unroll
            for (int k = 0; k < R; ++k) sr[k] = wr[k];
            while (true)
            {
#pragma unroll
                for (int k = 0; k < R; ++k) rr[k] = M::fma(-a, sr[k], rr[k]);
                store(cur, rr);
                __syncwarp();
                g = dot(rr, rr);
                product(wr, cur, rr);
#pragma unroll
                for (int k = 0; k < R; ++k) xr[k] = M::fma(a, pr[k], xr[k]);
                double * t = cur;
                cur = nxt;
                nxt = t;
                const double del = dot(wr, rr);
                ++it;
                const double bt = M::mul(g, inv_g), bg = M::mul(M::mul(bt, g), inv_a);
                const double ig = Recip<double>::rn(guard(g));
#pragma unroll
                for (int k = 0; k < R; ++k)
                {
                    pr[k] = M::fma(bt, pr[k], rr[k]);
                    sr[k] = M::fma(bt, sr[k], wr[k]);
                }
                if (g < thr2 || g < eps2 || it == max_iters)
                {
                    current = sqrt(g);
                    used = it;
                    break;
                }
                const double d = guard(M::sub(del, bg));
                a = M::mul(g, Recip<double>::rn(d));
                inv_g = ig;
                inv_a = fabs(a) > Eps<double>::v() ? M::mul(d, ig) : inv_eps;
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (live) xg[(i0 + k) * m + j] = S(xr[k]);
        if (lane == 0)
        {
            if (used_out) *used_out = used;
            if (defect_out) *defect_out = current;
        }
    }

    template <typename T, typename S, int RPL>
    __global__ void __launch_bounds__(32)
    cg_warp_reg_kernel(EllView<T> Ag, const S * __restrict__ b, S * __restrict__ xg, uint64_t max_iters, double eps_d,
                       int exact, uint64_t * used_out, double * defect_out, uint64_t vstride, const uint8_t * active,
                       const uint32_t * list, const uint32_t * count)
    {
        extern __shared__ __align__(16) unsigned char smem_raw[];
        pdl_entry();
        if (list)
        {
            // work list: the systems of vectors list[0 .. *count - 1], one per warp in turn
            const uint32_t n = *count;
            for (uint32_t i = blockIdx.x; i < n; i += gridDim.x)
            {
                const uint64_t o = (uint64_t)list[i] * vstride;
                cg_warp_reg<T, S, RPL>(Ag, b + o, xg + o, max_iters, eps_d, exact, used_out, defect_out, (T *)smem_raw);
                __syncwarp();
            }
            return;
        }
        // batched launches: block j solves the system of vector j (b, x at j * vstride)
        if (active && ! active[blockIdx.x]) return;
        cg_warp_reg<T, S, RPL>(Ag, b + (uint64_t)blockIdx.x * vstride, xg + (uint64_t)blockIdx.x * vstride, max_iters,
                               eps_d, exact, used_out, defect_out, (T *)smem_raw);
    }
}
