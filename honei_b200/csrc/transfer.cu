// Matrix-free grid transfer: Prolongation<Tag, NONE> (math/prolongation.hh:42-139)
// and Restriction<Tag, NONE> (math/restriction.hh:41-173), each followed by
// ApplyDirichletBoundaries (math/apply_dirichlet_boundaries.hh:29-84).
//
// The reference accumulates each node's value across several sequential
// sweeps over the grid.  Here one thread owns one output node and replays the
// contributions that reach that node in the reference's sweep order, with the
// same roundings, so the output is bit-identical and every node is written
// exactly once (no atomics, one pass over the input).
#include "hb2_common.cuh"
#include "hb2_internal.hh"
#include "transfer_free.cuh"

#include <cstdlib>

namespace hb2
{
    template <typename T>
    __global__ void prolongation_kernel(T * __restrict__ fine, const T * __restrict__ coarse, uint64_t mf, Mask mk)
    {
        const uint64_t f = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (f < mf * mf) fine[f] = free_prolong_node(coarse, f, mf, mk);
    }

    template <typename T>
    __global__ void restriction_kernel(T * __restrict__ coarse, const T * __restrict__ fine, uint64_t mf, Mask mk)
    {
        const uint64_t c = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, mc = (mf + 1) / 2;
        if (c < mc * mc) coarse[c] = free_restrict_node(fine, c, mf, mk);
    }

    static bool grid_side(uint64_t n, uint64_t * m)
    {
        uint64_t s = 1;
        while (s * s < n) ++s;
        *m = s;
        return s * s == n && s >= 3 && (s - 1) % 2 == 0;
    }

    // ------------------------------------------------------------------
    // The ProlongationMatrix of the identity index maps (math/prolongation_matrix.hh:44-100)
    // and its Transposition, applied without reading them.  Fine node (i, j) of a grid
    // with mf points per line, coarse node (I, J) = (i / 2, j / 2): the prolongation row
    // holds, in ascending column order, (I, J) with weight 1 (i, j even), (I, J) and
    // (I, J + 1) or (I, J) and (I + 1, J) with 1/2 (one odd), and (I, J), (I, J + 1),
    // (I + 1, J), (I + 1, J + 1) with 1/4 (both odd); the restriction row of (I, J)
    // holds the fine nodes (2I + di, 2J + dj), di, dj in -1..1 inside the grid, in
    // ascending column order, with weight (1 or 1/2) x (1 or 1/2).  Each row is summed
    // as the ELL kernels sum it (0 + v0 x0 + v1 x1 ..., products and sums rounded
    // separately; q1_prolong_row / q1_restrict_row), so the results are bit-identical
    // to the matrix products.
    // R fine rows per thread, interleaved over the block (every access coalesced); the
    // rows' y loads (kAdd) issued before their coarse gathers
    template <typename T, int MODE, int R>
    __global__ void __launch_bounds__(256)
    q1_prolong_kernel(const T * __restrict__ c, T * __restrict__ y, uint32_t mf, uint32_t mc, uint64_t nf,
                      int64_t pf)
    {
        typedef Arith<T> M;
        pdl_entry();
        const uint64_t r0 = (uint64_t)blockIdx.x * blockDim.x * R + threadIdx.x;
        T yv[R];
#pragma unroll
        for (int k = 0; k < R; ++k)
        {
            const uint64_t r = r0 + (uint64_t)k * blockDim.x;
            yv[k] = (MODE == kAdd && r < nf) ? y[r] : T(0);
            // the fine vector of a later wave of blocks into L2 (y += P c reads it)
            if (MODE == kAdd && pf && r + pf < nf) prefetch_l2(y + r + pf);
        }
#pragma unroll
        for (int k = 0; k < R; ++k)
        {
            const uint64_t r = r0 + (uint64_t)k * blockDim.x;
            if (r >= nf) break;
            const T acc = q1_prolong_row<T, false>(r, c, mf, mc);
            y[r] = MODE == kAdd ? M::add(yv[k], acc) : acc;
        }
    }

    // rows per thread of the prolongation kernel: 2 for fine grids of 2^21 rows or more,
    // else 1 (graph-timed at level 11 with an L2 prefetch: FP64 19.8 / 18.1 / 21.3 us for
    // 1 / 2 / 4 rows, FP32 18.9 / 16.1 / 16.1 us; the first form, one row and y loaded
    // after the gathers, 26.2 / 23.9 us; inside the MG solves two rows helped at level 11
    // and cost 0.5 % at levels 9 and 10, where the grid of blocks is small);
    // HB2_Q1_PROLONG_R (1, 2 or 4) overrides
    static int prolong_rows(uint64_t nf)
    {
        const char * v = getenv("HB2_Q1_PROLONG_R");
        const int r = v && *v ? atoi(v) : (nf >= (1u << 21) ? 2 : 1);
        return (r == 2 || r == 4) ? r : 1;
    }

    template <typename T, int MODE>
    __global__ void __launch_bounds__(256)
    q1_restrict_kernel(const T * __restrict__ x, T * __restrict__ y, T * __restrict__ zero, uint32_t mf,
                       uint32_t mc, uint64_t nc, int64_t pf)
    {
        pdl_entry();
        const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (r >= nc) return;
        if (pf && r + pf < nc)
        {
            // the three fine grid rows a later wave's coarse row reads, into L2
            const uint64_t rr = r + pf, I = rr / mc, J = rr - I * mc, f = 2 * I * mf + 2 * J, nf = (uint64_t)mf * mf;
            if (f >= mf) prefetch_l2(x + f - mf);
            prefetch_l2(x + f);
            if (f + mf < nf) prefetch_l2(x + f + mf);
        }
        y[r] = q1_restrict_row<T, false>(r, x, mf, mc);
        if (MODE == kRestrict) zero[r] = T(0);
    }

    template <typename T>
    static int q1_transfer_typed(const hb2_ell_s * A, int mode, const void * x, void * y, void * zero,
                                 cudaStream_t s)
    {
        const int L = A->q1_transfer > 0 ? A->q1_transfer : -A->q1_transfer;
        const uint32_t mf = (1u << L) + 1, mc = (1u << (L - 1)) + 1;
        const T * xp = (const T *)x;
        T * yp = (T *)y;
        const dim3 grid(ceil_div(A->rows, 256));
        const int64_t pf = l2_prefetch_rows(sizeof(T));
        if (A->q1_transfer > 0)
        {
            const int R = prolong_rows(A->rows);
            const dim3 pgrid(ceil_div(A->rows, 256 * R));
#define HB2_PROL(R_)                                                                                                   \
            if (mode == kAdd) launch_pdl(q1_prolong_kernel<T, kAdd, R_>, pgrid, dim3(256), 0, s, xp, yp, mf, mc, A->rows, pf); \
            else launch_pdl(q1_prolong_kernel<T, kPlain, R_>, pgrid, dim3(256), 0, s, xp, yp, mf, mc, A->rows, pf)
            if (R == 4) { HB2_PROL(4); }
            else if (R == 2) { HB2_PROL(2); }
            else { HB2_PROL(1); }
#undef HB2_PROL
        }
        else
        {
            if (mode == kRestrict)
                launch_pdl(q1_restrict_kernel<T, kRestrict>, grid, dim3(256), 0, s, xp, yp, (T *)zero, mf, mc, A->rows,
                           pf);
            else launch_pdl(q1_restrict_kernel<T, kPlain>, grid, dim3(256), 0, s, xp, yp, (T *)zero, mf, mc, A->rows,
                            pf);
        }
        return HB2_OK;
    }

    int launch_q1_transfer(const hb2_ell_s * A, int mode, const void * x, void * y, void * zero, cudaStream_t stream)
    {
        // a prolongation computes kPlain / kAdd rows, a restriction kPlain / kRestrict rows
        if ((A->q1_transfer > 0 && mode == kRestrict) || (A->q1_transfer < 0 && mode == kAdd))
            return fail(HB2_ERR_UNSUPPORTED, "Q1 transfer kernel: mode");
        const int st = A->dtype == HB2_F64 ? q1_transfer_typed<double>(A, mode, x, y, zero, stream)
                                           : q1_transfer_typed<float>(A, mode, x, y, zero, stream);
        count_launches(1);
        HB2_LAUNCH_CHECK("Q1 transfer kernel launch");
        return st;
    }
}

using namespace hb2;

extern "C" int hb2_prolongation(hb2_dtype dt, void * fine, uint64_t n_fine, const void * coarse, uint64_t n_coarse,
                                const uint64_t * mask, cudaStream_t stream)
{
    uint64_t mf = 0;
    if (! fine || ! coarse) return fail(HB2_ERR_ARG, "hb2_prolongation: null vector");
    if (! grid_side(n_fine, &mf) || ((mf + 1) / 2) * ((mf + 1) / 2) != n_coarse)
        return fail(HB2_ERR_SIZE, "hb2_prolongation: sizes are not (2m-1)^2 / m^2 grids");
    unsigned grid = ceil_div(n_fine, 256);
    Mask mk = make_mask(mask);
    if (dt == HB2_F64) prolongation_kernel<double><<<grid, 256, 0, stream>>>((double *)fine, (const double *)coarse, mf, mk);
    else prolongation_kernel<float><<<grid, 256, 0, stream>>>((float *)fine, (const float *)coarse, mf, mk);
    count_launches(1);
    HB2_LAUNCH_CHECK("hb2_prolongation");
    return HB2_OK;
}

extern "C" int hb2_restriction(hb2_dtype dt, void * coarse, uint64_t n_coarse, const void * fine, uint64_t n_fine,
                               const uint64_t * mask, cudaStream_t stream)
{
    uint64_t mf = 0;
    if (! fine || ! coarse) return fail(HB2_ERR_ARG, "hb2_restriction: null vector");
    if (! grid_side(n_fine, &mf) || ((mf + 1) / 2) * ((mf + 1) / 2) != n_coarse)
        return fail(HB2_ERR_SIZE, "hb2_restriction: sizes are not (2m-1)^2 / m^2 grids");
    unsigned grid = ceil_div(n_coarse, 256);
    Mask mk = make_mask(mask);
    if (dt == HB2_F64) restriction_kernel<double><<<grid, 256, 0, stream>>>((double *)coarse, (const double *)fine, mf, mk);
    else restriction_kernel<float><<<grid, 256, 0, stream>>>((float *)coarse, (const float *)fine, mf, mk);
    count_launches(1);
    HB2_LAUNCH_CHECK("hb2_restriction");
    return HB2_OK;
}
