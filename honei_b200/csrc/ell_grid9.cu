// ELL matrices with the rows of a nine-point operator on an m x m grid and any values: an
// interior row's columns are i - m - 1 .. i + m + 1 in ascending slot order, a boundary row
// holds its diagonal in slot 0 (the Q1 finite-element operator with varying coefficients;
// checked row by row at creation, launch_grid_check).  Their columns need not be read: a row
// moves 72 instead of 108 bytes of matrix in FP64, 36 instead of 72 in FP32.
//
// A thread takes 16 bytes of consecutive rows (two in FP64, four in FP32): nine 128-bit value
// loads, and three runs of R + 2 values of x instead of nine a row, all issued before the first
// product.  Products and slot-ordered sums of the plain kernel (la/product.hh:148-206), same
// bits.  Bound by HBM (inside L2, by its bandwidth): 88 bytes a row for y = A x in FP64.
#include "hb2_common.cuh"
#include "hb2_internal.hh"

namespace hb2
{
    template <typename T> struct Vec16;
    template <> struct Vec16<double> { typedef double2 type; };
    template <> struct Vec16<float> { typedef float4 type; };

    template <typename T, int MODE>
    __global__ void __launch_bounds__(kEllThreads)
    grid9_kernel(const T * __restrict__ val, uint64_t ld, uint32_t n, uint32_t m, const T * __restrict__ x,
                 T * __restrict__ y, const T * __restrict__ aux, const T * __restrict__ aux2, ReduceSlot rs, double * red,
                 int want_sqrt, int flags)
    {
        typedef Arith<T> M;
        typedef typename Vec16<T>::type V;
        constexpr int R = RowsPerThread<T>::value;
        pdl_entry();
        const uint32_t blk = (flags & kReverse) ? gridDim.x - 1 - blockIdx.x : blockIdx.x;
        const uint32_t r0 = (blk * kEllThreads + threadIdx.x) * R;
        double part = 0.0;
        if (r0 < n)
        {
            union { V v; T a[R]; } v[9];
#pragma unroll
            for (int k = 0; k < 9; ++k)
            {
                const V * p = (const V *)(val + (uint64_t)k * ld + r0);
                v[k].v = (flags & kKeepL2) ? __ldcg(p) : __ldcs(p);
            }
            // x of the three grid lines around the rows; outside the vector: any value, no
            // interior row reads it
            T xv[3][R + 2];
            const bool inside = r0 >= m + 1 && r0 + R + m < n;
#pragma unroll
            for (int l = 0; l < 3; ++l)
#pragma unroll
                for (int q = 0; q < R + 2; ++q)
                {
                    const int64_t i = (int64_t)r0 + (l - 1) * (int64_t)m + q - 1;
                    xv[l][q] = inside || (i >= 0 && i < (int64_t)n) ? __ldg(x + i) : T(0);
                }
            T ea[R], ep[R];
#pragma unroll
            for (int k = 0; k < R; ++k)
            {
                ea[k] = (MODE == kDefect || is_jacobi(MODE)) && r0 + k < n ? aux[r0 + k] : T(0);
                ep[k] = is_jacobi(MODE) && r0 + k < n ? aux2[r0 + k] : T(0);
            }
            uint32_t i = r0 / m, j = r0 - i * m;
#pragma unroll
            for (int k = 0; k < R; ++k)
            {
                const uint32_t r = r0 + k;
                if (r >= n) break;
                T acc = M::add(T(0), M::mul(v[0].a[k], xv[0][k]));
#pragma unroll
                for (int q = 1; q < 9; ++q) acc = M::add(acc, M::mul(v[q].a[k], xv[q / 3][k + q % 3]));
                const T xc = xv[1][k + 1];
                if (i == 0 || j == 0 || i == m - 1 || j == m - 1) acc = M::add(T(0), M::mul(v[0].a[k], xc));
                if (MODE == kPlain) y[r] = acc;
                else if (MODE == kDot)
                {
                    y[r] = acc;
                    part = fma((double)acc, (double)xc, part);
                }
                else
                {
                    const T d = M::sub(ea[k], acc);
                    y[r] = MODE == kDefect ? d : M::add(xc, M::mul(ep[k], d));
                    part = fma((double)d, (double)d, part);
                }
                if (++j == m) { j = 0; ++i; }
            }
        }
        if ((MODE == kDefect || MODE == kDot || MODE == kJacobiNorm) && red != 0)
        {
            __shared__ double scratch[32];
            ell_block_reduce(part, rs, red, want_sqrt, flags, scratch);
        }
    }

    bool grid9_applies(const hb2_ell_s * A, int mode, bool reducing)
    {
        return A->g9_m && A->layout[reducing ? 1 : 0] == kLayoutPlain &&
               (mode == kPlain || mode == kDefect || mode == kDot || mode == kJacobi);
    }

    template <typename T>
    static int launch_typed(const hb2_ell_s * A, int mode, const void * x, void * y, const void * aux, const void * aux2,
                            double * red, int want_sqrt, const Workspace * ws, cudaStream_t stream, int flags)
    {
        const uint32_t n = (uint32_t)A->rows, m = A->g9_m;
        const unsigned grid = ceil_div(n, (uint64_t)kEllThreads * RowsPerThread<T>::value);
        ReduceSlot rs = {};
        if (red)
        {
            if (! ws) return fail(HB2_ERR_ARG, "fused reduction without a workspace");
            if (grid > ws->max_blocks || (grid + kReduceGroup - 1) / kReduceGroup + 1 > ws->max_tickets)
                return fail(HB2_ERR_UNSUPPORTED, "matrix / batch too large for the reduction workspace");
            rs = ws->slot();
        }
        const bool split = red && grid >= kSplitSumMinBlocks;
        if (split) flags |= kSplitSum;
#define HB2_G9(M_) launch_pdl(grid9_kernel<T, M_>, dim3(grid), dim3(kEllThreads), 0, stream, (const T *)A->val, A->ld, n, m, \
                              (const T *)x, (T *)y, (const T *)aux, (const T *)aux2, rs, red, want_sqrt, flags)
        if (mode == kPlain) HB2_G9(kPlain);
        else if (mode == kDefect) HB2_G9(kDefect);
        else if (mode == kDot) HB2_G9(kDot);
        else if (red) HB2_G9(kJacobiNorm);
        else HB2_G9(kJacobi);
#undef HB2_G9
        count_launches(1);
        if (split) launch_sum_partials(rs.partials, grid, 1, red, want_sqrt, stream);
        HB2_LAUNCH_CHECK("nine-point ELL kernel launch");
        return HB2_OK;
    }

    int launch_grid9(const hb2_ell_s * A, int mode, const void * x, void * y, const void * aux, const void * aux2,
                     double * red, int want_sqrt, const Workspace * ws, cudaStream_t stream, int flags)
    {
        return A->dtype == HB2_F64 ? launch_typed<double>(A, mode, x, y, aux, aux2, red, want_sqrt, ws, stream, flags)
                                   : launch_typed<float>(A, mode, x, y, aux, aux2, red, want_sqrt, ws, stream, flags);
    }
}
