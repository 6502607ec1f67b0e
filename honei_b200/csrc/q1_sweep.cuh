// Several damped Jacobi sweeps of a Q1 grid operator in one pass over memory, with
// the grid transfers and the defect around them (MGData's cycle, math/mg.hh:577-640;
// RISmoother, math/ri.hh:97-133).
//
// One sweep at a time reads x, b and P and writes x again (33 B a row in FP64): a
// V(4,4) cycle makes twelve such passes over its finest level.  Here a warp owns a strip
// of columns and marches along the grid rows with every sweep's stage in flight at once:
// stage t turns row a of iterate t into row a - 1 of iterate t + 1 as soon as row a
// exists, so x and b are read once and the last iterate is written once whatever the
// number of sweeps.  The optional last stage forms the defect of the new iterate and
// either restricts it (the coarser right-hand side is written instead of the defect) or
// sums its squares; an optional head adds the prolonged coarser correction to x on the
// way in, or starts from x = 0 without reading anything but b.
//
// Layout.  A lane holds C adjacent columns; the left and right neighbours' products come
// by shuffle, the rows above and below by keeping each stage's two partial sums in
// registers (row i's sum is three products of row i - 1, three of row i, three of
// row i + 1, in the ELL slot order -- la/product.hh:148-206 -- so marching upwards
// completes it in that order and the bits are those of the single sweeps).  All couplings
// of the constant-coefficient operator are equal (UNI): one product per node and stage
// serves its eight neighbours; the general form multiplies nine times.  Rows of x, b and
// of the coarser correction arrive through per-warp shared-memory rings filled by
// cp.async several rows ahead; there is no block barrier.  Each stage uses the row its
// predecessor finished one step earlier (skew of two rows per stage), so the stages of one
// step are independent instruction streams.
//
// What bounds it: instruction issue and the FP64 (FP32) pipe -- 13 operations per node and
// stage, plus the halo of NS columns each side of a strip and NS rows each end of a chunk;
// on the small grids the latency of a step times the rows of a chunk.  Measured (B200, graph
// of 20 passes over vector sets larger than L2), FP64: the level-11 pass of four sweeps,
// defect and restriction 49.8 us, of prolongation, four sweeps and norm 55.5 us, where the
// single passes took about 165 and 155 us; level 10 15.5 / 18.6 us; FP32 level 11 35.1 us.
#pragma once

#include "hb2_common.cuh"
#include "hb2_internal.hh"
#include "smem_opt_in.hh"

#include <algorithm>
#include <type_traits>

namespace hb2
{
    enum { kSweepLoad = 0, kSweepZero = 1 };                            // HEAD
    // TAIL; the last four without sweeps (S = 0): y = b - A x (+ ||y||^2), y = A x (+ <y, x>),
    // and the refinement's defect, rounded to FP32 into y32 with z32 cleared (+ ||b - A x||^2)
    enum { kSweepStore = 0, kSweepRestrict = 1, kSweepNorm = 2, kSweepDefect = 3, kSweepProduct = 4, kSweepDot = 5,
           kSweepDefectIR = 6 };
    __host__ __device__ constexpr bool sweep_single(int tail) { return tail >= kSweepDefect; }
    __host__ __device__ constexpr bool sweep_reads_b(int tail) { return tail != kSweepProduct && tail != kSweepDot; }
    __host__ __device__ constexpr bool sweep_reduces(int tail)
    {
        return tail == kSweepNorm || tail == kSweepDefect || tail == kSweepDot || tail == kSweepDefectIR;
    }

    template <typename T>
    struct Q1SweepArgs
    {
        T v[9];                 // the interior row, slot order
        T vb;                   // the boundary rows' diagonal
        int m, mc;              // points per line, fine and coarse
        const T * x;            // iterate in (kSweepLoad)
        const T * c;            // coarser correction to prolong and add to x (nullable)
        const T * b;            // right-hand side
        const T * jac;          // Jacobi vector; without PVEC entry 0 (boundary) and m + 1 (interior)
        T * y;                  // iterate out, != x
        T * cb;                 // kSweepRestrict: coarser right-hand side
        T * cz;                 // kSweepRestrict: coarser vector cleared on the way (nullable)
        double * partials;      // reducing tails: one partial per block (nullable but for kSweepNorm)
        float * y32, * z32;     // kSweepDefectIR (z32 nullable)
        int strips, chunks, rows;   // strips of columns x chunks of `rows` rows
        int bpv;                // blocks per vector
        // batched: vectors list[0 .. *count), the fine arrays vs elements apart, the coarse ones cs
        const uint32_t * list;
        const uint32_t * count;
        uint64_t vs, cs;
    };

    template <typename T, int C, int S, int HEAD, int TAIL>
    struct Q1SweepShape
    {
        static constexpr int NSM = HEAD == kSweepZero ? S - 1 : S;        // sweeps that need neighbours
        static constexpr int NS = NSM + (TAIL != kSweepStore ? 1 : 0);    // stencil stages
        static constexpr int HALO = NS + (TAIL == kSweepRestrict ? 1 : 0);
        static constexpr int W = 32 * C;                                  // columns of a warp
        static constexpr int HC = (HALO + 1) / 2 * 2;                     // column halo, even
        static constexpr int WV = W - 2 * HC;                             // columns it owns
        static constexpr int D = 6;                                       // rows in flight
        static constexpr int RB = 16, RX = 8, RC = 8;                     // ring sizes (rows)
        static constexpr int CW = W / 2 + 2;                              // coarse columns of a ring row
        static_assert(2 * NS + D <= RB, "b ring");
        static_assert(WV > 0, "strip");
        static constexpr size_t ring(bool pvec)                           // elements of one warp
        {
            return (size_t)RB * W * (pvec ? 2 : 1) + (HEAD == kSweepLoad ? (size_t)RX * W + (size_t)RC * CW : 0);
        }
    };

    constexpr int kSweepWarps = 4;
    // blocks per SM the registers are sized for: 3 (168 registers) with two FP64 columns a
    // lane, else 4.  Held to 128 registers the wide FP64 form spilled and its level-11 pass
    // took 142 us instead of 68 (before the steps were written in pairs).
    template <typename T, int C> constexpr int sweep_blocks_per_sm() { return C * sizeof(T) == 16 ? 3 : 4; }


    template <int BYTES>
    __device__ __forceinline__ void cp_async_elem(void * smem, const void * g)
    {
        const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
        if (BYTES == 8) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s), "l"(g) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(g) : "memory");
    }
    __device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
    template <int N>
    __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

    // C consecutive elements of shared memory, aligned to C * sizeof(T) (C = 1, 2, 4)
    template <typename T, int C>
    __device__ __forceinline__ void lds_vec(T (&o)[C], const T * p)
    {
        if constexpr (C == 1) o[0] = p[0];
        else if constexpr (C * sizeof(T) == 16)
        {
            const int4 q = *reinterpret_cast<const int4 *>(p);
            *reinterpret_cast<int4 *>(o) = q;
        }
        else
        {
#pragma unroll
            for (int c = 0; c < C; ++c) o[c] = p[c];
        }
    }

    template <typename T, int C, bool UNI, int S, int HEAD, int TAIL, bool PVEC>
    __global__ void __launch_bounds__(32 * kSweepWarps, sweep_blocks_per_sm<T, C>())
    q1_sweep_kernel(const __grid_constant__ Q1SweepArgs<T> g)
    {
        typedef Arith<T> M;
        typedef Q1SweepShape<T, C, S, HEAD, TAIL> K;
        constexpr int NS = K::NS, NSM = K::NSM, W = K::W, D = K::D, HALO = K::HALO;
        constexpr int RBM = K::RB - 1, RXM = K::RX - 1, RCM = K::RC - 1;
        extern __shared__ __align__(16) unsigned char sweep_smem[];
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        T * bring = reinterpret_cast<T *>(sweep_smem) + K::ring(PVEC) * warp;
        T * pring = bring + K::RB * W;                       // PVEC only
        T * xring = bring + K::RB * W * (PVEC ? 2 : 1);      // kSweepLoad only
        T * cring = xring + K::RX * W;
        const int m = g.m;
        pdl_entry();
        T Pi = T(0), Pb = T(0);
        if (! PVEC && ! sweep_single(TAIL)) { Pb = __ldg(g.jac); Pi = __ldg(g.jac + m + 1); }
        const uint32_t nblk = g.list ? *g.count * (uint32_t)g.bpv : gridDim.x;
        double part = 0.0;
        for (uint32_t blk = blockIdx.x; blk < nblk; blk += gridDim.x)
        {
            uint64_t vo = 0, co = 0;
            uint32_t item = blk;
            if (g.list)
            {
                const uint32_t j = blk / (uint32_t)g.bpv;
                item = blk - j * (uint32_t)g.bpv;
                const uint64_t vec = g.list[j];
                vo = vec * g.vs;
                co = vec * g.cs;
            }
            item = item * kSweepWarps + warp;
            if (item >= (uint32_t)(g.strips * g.chunks)) continue;     // whole warps
            const int chunk = (int)(item / (uint32_t)g.strips), strip = (int)item - chunk * g.strips;
            const int cb = strip * K::WV, base = cb - K::HC;           // first owned, first loaded column (even)
            const int r0 = chunk * g.rows, r1 = min(m, r0 + g.rows);   // owned rows
            const int kb = max(0, r0 - HALO) & ~1, ke = min(m - 1, r1 - 1 + HALO);   // rows read, from an even one
            const int last = (NS == 0 ? r1 - 1 : (TAIL == kSweepRestrict ? min(r1, m - 1) : r1 - 1) + 2 * NS - 1);
            const int col0 = base + lane * C;
            bool own[C], edge[C];
            T Pc[C];                                   // the Jacobi vector of an interior row's columns
#pragma unroll
            for (int c = 0; c < C; ++c)
            {
                const int col = col0 + c;
                own[c] = col >= cb && col < min(cb + K::WV, m);
                edge[c] = col == 0 || col == m - 1;
                Pc[c] = edge[c] ? Pb : Pi;
            }
            // rows kb .. ke of x, b (P, c) into the rings, D rows ahead
            const T * xg = HEAD == kSweepLoad ? g.x + vo : nullptr;
            const T * bg = sweep_reads_b(TAIL) ? g.b + vo : nullptr;
            const T * pg = PVEC ? g.jac : nullptr;
            const T * cg = (HEAD == kSweepLoad && ! sweep_single(TAIL) && g.c) ? g.c + co : nullptr;
            const int cbase = base >> 1;
            auto fetch_coarse = [&](int I) {
                for (int j = lane; j < K::CW; j += 32)
                {
                    const int J = cbase + j;
                    if (J >= 0 && J < g.mc && I < g.mc)
                        cp_async_elem<sizeof(T)>(cring + (I & RCM) * K::CW + j, cg + (int64_t)I * g.mc + J);
                }
            };
            // running pointers of the next row to fetch (this lane's first column)
            const int64_t fo = (int64_t)kb * m + base + lane;
            const T * xf = HEAD == kSweepLoad ? xg + fo : nullptr;
            const T * bf = sweep_reads_b(TAIL) ? bg + fo : nullptr;
            const T * pf = PVEC ? pg + fo : nullptr;
            bool in[C];
#pragma unroll
            for (int q = 0; q < C; ++q) in[q] = base + lane + 32 * q >= 0 && base + lane + 32 * q < m;
            auto fetch = [&](int f) {
                if (f <= ke)
                {
                    T * br = bring + (f & RBM) * W + lane, * xr = xring + (f & RXM) * W + lane;
#pragma unroll
                    for (int q = 0; q < C; ++q)
                        if (in[q])
                        {
                            if (sweep_reads_b(TAIL)) cp_async_elem<sizeof(T)>(br + 32 * q, bf + 32 * q);
                            if (HEAD == kSweepLoad) cp_async_elem<sizeof(T)>(xr + 32 * q, xf + 32 * q);
                            if (PVEC) cp_async_elem<sizeof(T)>(pring + (f & RBM) * W + lane + 32 * q, pf + 32 * q);
                        }
                    if (HEAD == kSweepLoad && cg && (f & 1)) fetch_coarse((f + 1) >> 1);
                }
                if (sweep_reads_b(TAIL)) bf += m;
                if (HEAD == kSweepLoad) xf += m;
                if (PVEC) pf += m;
                cp_async_commit();
            };
            __syncwarp();           // the rings' last reads of the previous item are done
            if (cg) fetch_coarse(kb >> 1);
#pragma unroll
            for (int f = 0; f < D; ++f) fetch(kb + f);

            constexpr int NA = NS > 0 ? NS : 1;
            T acc1[NA][C], acc2[NA][C], xprev[NA][C], cur[NA + 1][C], racc[C];
#pragma unroll
            for (int t = 0; t < NA; ++t)
#pragma unroll
                for (int c = 0; c < C; ++c) acc1[t][c] = acc2[t][c] = xprev[t][c] = cur[t][c] = T(0);
#pragma unroll
            for (int c = 0; c < C; ++c) cur[NA][c] = racc[c] = T(0);

            // running pointer of the row the last sweep completes in the next step
            constexpr int YLAG = NSM > 0 ? 2 * NSM - 1 : (sweep_single(TAIL) ? 1 : 0);
            T * yr = g.y + vo + col0 + ((int64_t)kb - YLAG) * m;
            const T * brl = bring + lane * C, * prl = pring + lane * C;
            auto step = [&](auto interior, auto parity, int s) {
                constexpr bool IN = decltype(interior)::value;      // no boundary row in a stage
                constexpr bool ODD = decltype(parity)::value;       // of s; the stages' rows have the other one
                cp_async_wait<D - 1>();
                __syncwarp();
                fetch(s + D);
                // ---- head: row s of the first iterate
                if (HEAD == kSweepLoad)
                {
                    lds_vec<T, C>(cur[0], xring + (s & RXM) * W + lane * C);
                    if (cg)
                    {
                        const int I = s >> 1;
                        const T h = T(0.5), q4 = T(0.25);
                        const T * c0 = cring + (I & RCM) * K::CW + ((lane * C) >> 1);
                        const T * c1 = cring + ((I + 1) & RCM) * K::CW + ((lane * C) >> 1);
#pragma unroll
                        for (int c = 0; c < C; ++c)
                        {
                            // powers of two: the products are exact, so each fma rounds as the sum does
                            const int j = C == 1 ? 0 : c >> 1;
                            const bool odd = C == 1 ? (lane & 1) != 0 : (c & 1) != 0;
                            T p;
                            if (! ODD) p = ! odd ? M::add(T(0), c0[j]) : M::fma(h, c0[j + 1], M::mul(h, c0[j]));
                            else if (! odd) p = M::fma(h, c1[j], M::mul(h, c0[j]));
                            else p = M::fma(q4, c1[j + 1], M::fma(q4, c1[j], M::fma(q4, c0[j + 1], M::mul(q4, c0[j]))));
                            cur[0][c] = M::add(cur[0][c], p);
                        }
                    }
                }
                else
                {
                    // the first sweep from x = 0: 0 + P (b - 0)
                    T bq[C], pq[C];
                    lds_vec<T, C>(bq, brl + (s & RBM) * W);
                    if (PVEC) lds_vec<T, C>(pq, prl + (s & RBM) * W);
                    const bool rb = ! IN && (s == 0 || s == m - 1);
#pragma unroll
                    for (int c = 0; c < C; ++c)
                    {
                        if (! PVEC) pq[c] = rb ? Pb : Pc[c];
                        cur[0][c] = M::add(T(0), M::mul(pq[c], bq[c]));
                    }
                    if (NSM == 0 && s >= r0 && s < r1)
                    {
#pragma unroll
                        for (int c = 0; c < C; ++c)
                            if (own[c]) yr[c] = cur[0][c];
                    }
                }
                // ---- the stages.  Each reads what its predecessor left a step ago, so they are
                // independent; written operation by operation over all of them, which the
                // compiler keeps as that many instruction streams side by side.
                // products of row q + 1 (UNI: one per node; the sum 0 + p of the first slot is
                // folded into p, which is never -0)
                T p[NA][C], pw[NA], pe[NA];
#pragma unroll
                for (int t = 0; t < NS; ++t)
#pragma unroll
                    for (int c = 0; c < C; ++c) p[t][c] = UNI ? M::fma(g.v[0], cur[t][c], T(0)) : cur[t][c];
#pragma unroll
                for (int t = 0; t < NS; ++t)
                {
                    pw[t] = __shfl_up_sync(0xffffffffu, p[t][C - 1], 1);
                    pe[t] = __shfl_down_sync(0xffffffffu, p[t][0], 1);
                }
                T ax[NA][C];
#pragma unroll
                for (int k = 0; k < 3; ++k)          // west, centre, east: one sum of each chain a round
#pragma unroll
                    for (int t = 0; t < NS; ++t)
#pragma unroll
                        for (int c = 0; c < C; ++c)
                        {
                            const T u = k == 0 ? (c ? p[t][c > 0 ? c - 1 : 0] : pw[t])
                                               : (k == 1 ? p[t][c] : (c < C - 1 ? p[t][c < C - 1 ? c + 1 : c] : pe[t]));
                            ax[t][c] = M::add(k == 0 ? acc2[t][c] : ax[t][c], UNI ? u : M::mul(g.v[6 + k], u));
                        }
#pragma unroll
                for (int k = 0; k < 3; ++k)
#pragma unroll
                    for (int t = 0; t < NS; ++t)
#pragma unroll
                        for (int c = 0; c < C; ++c)
                        {
                            const T u = k == 0 ? (c ? p[t][c > 0 ? c - 1 : 0] : pw[t])
                                               : (k == 1 ? p[t][c] : (c < C - 1 ? p[t][c < C - 1 ? c + 1 : c] : pe[t]));
                            const T d = k == 1 && UNI ? M::mul(g.v[4], cur[t][c]) : u;
                            acc2[t][c] = M::add(k == 0 ? acc1[t][c] : acc2[t][c], UNI ? d : M::mul(g.v[3 + k], u));
                            if (k == 0) acc1[t][c] = UNI ? u : M::fma(g.v[0], u, T(0));
                            else acc1[t][c] = M::add(acc1[t][c], UNI ? u : M::mul(g.v[k], u));
                        }
                T res[NA][C];
#pragma unroll
                for (int t = 0; t < NS; ++t)
                {
                    const int q = s - 2 * t - 1;                 // the row this stage completes
                    T bq[C];
                    if (sweep_reads_b(TAIL)) lds_vec<T, C>(bq, brl + (q & RBM) * W);
#pragma unroll
                    for (int c = 0; c < C; ++c)
                    {
                        if ((! IN && (q == 0 || q == m - 1)) || edge[c]) ax[t][c] = M::fma(g.vb, xprev[t][c], T(0));
                        res[t][c] = sweep_reads_b(TAIL) ? M::sub(bq[c], ax[t][c]) : ax[t][c];
                    }
                }
#pragma unroll
                for (int t = NS - 1; t >= 0; --t)
                {
                    const int q = s - 2 * t - 1;
                    T out[C], xq[C];
                    if (t < NSM)
                    {
                        T pq[C];
                        if (PVEC) lds_vec<T, C>(pq, prl + (q & RBM) * W);
#pragma unroll
                        for (int c = 0; c < C; ++c)
                        {
                            if (! PVEC) pq[c] = ! IN && (q == 0 || q == m - 1) ? Pb : Pc[c];
                            out[c] = M::add(xprev[t][c], M::mul(pq[c], res[t][c]));
                        }
                    }
                    else
                    {
#pragma unroll
                        for (int c = 0; c < C; ++c) out[c] = res[t][c];
                    }
#pragma unroll
                    for (int c = 0; c < C; ++c)
                    {
                        xq[c] = xprev[t][c];
                        xprev[t][c] = cur[t][c];
                    }
                    if (t < NSM)
                    {
#pragma unroll
                        for (int c = 0; c < C; ++c) cur[t + 1][c] = out[c];
                        if (t == NSM - 1 && q >= r0 && q < r1)
                        {
#pragma unroll
                            for (int c = 0; c < C; ++c)
                                if (own[c]) yr[c] = out[c];
                        }
                    }
                    else if (TAIL == kSweepNorm)
                    {
                        if (q >= r0 && q < r1)
                        {
#pragma unroll
                            for (int c = 0; c < C; ++c)
                                if (own[c]) part = fma((double)out[c], (double)out[c], part);
                        }
                    }
                    else if (sweep_single(TAIL))
                    {
                        if (q >= r0 && q < r1)
                        {
#pragma unroll
                            for (int c = 0; c < C; ++c)
                                if (own[c])
                                {
                                    if (TAIL == kSweepDefectIR)
                                    {
                                        const int64_t o = (int64_t)q * m + col0 + c;
                                        g.y32[o] = (float)out[c];
                                        if (g.z32) g.z32[o] = 0.f;
                                    }
                                    else yr[c] = out[c];
                                    if (sweep_reduces(TAIL))
                                        part = fma((double)out[c], (double)(TAIL == kSweepDot ? xq[c] : out[c]), part);
                                }
                        }
                    }
                    else if (TAIL == kSweepRestrict)
                    {
                        // row q of the defect into the coarse rows it touches (weights 1, 1/2,
                        // 1/4: exact products), the even columns' sums in column order
                        const T rw0 = __shfl_up_sync(0xffffffffu, out[C - 1], 1);
                        const T re0 = C == 1 ? __shfl_down_sync(0xffffffffu, out[0], 1) : T(0);
                        const T h = T(0.5), q4 = T(0.25);
#pragma unroll
                        for (int c = 0; c < C; c += 2)
                        {
                            const int col = col0 + c;
                            T w = c ? out[c > 0 ? c - 1 : 0] : rw0, e = C == 1 ? re0 : out[c + 1 < C ? c + 1 : c];
                            if (col <= 0) w = T(0);                 // outside the grid: no term
                            if (col >= m - 1) e = T(0);
                            if (! IN && q == 0) racc[c] = T(0);
                            bool done = false;
                            T v = T(0);
                            int I = 0;
                            if (! ODD)      // q odd
                            {
                                v = M::fma(q4, e, M::fma(h, out[c], M::fma(q4, w, racc[c])));
                                racc[c] = M::fma(q4, e, M::fma(h, out[c], M::fma(q4, w, T(0))));
                                done = q - 1 >= r0 && q - 1 < r1;
                                I = (q - 1) >> 1;
                            }
                            else
                            {
                                racc[c] = M::fma(h, e, M::add(M::fma(h, w, racc[c]), out[c]));
                                if (! IN && q == m - 1)
                                {
                                    v = racc[c];
                                    done = q >= r0 && q < r1;
                                    I = q >> 1;
                                }
                            }
                            if (done && own[c] && (C > 1 || ! (lane & 1)))
                            {
                                const int64_t o = (int64_t)co + (int64_t)I * g.mc + (col >> 1);
                                g.cb[o] = v;
                                if (g.cz) g.cz[o] = T(0);
                            }
                        }
                    }
                }
                yr += m;
            };
            // two steps at a time (the stages' rows change places without moves); a step
            // past `last` writes nothing
#pragma unroll 1
            for (int s = kb; s <= last; s += 2)
            {
                if (s >= 2 * NS + 1 && s + 1 < m - 1)
                {
                    step(std::true_type(), std::false_type(), s);
                    step(std::true_type(), std::true_type(), s + 1);
                }
                else
                {
                    step(std::false_type(), std::false_type(), s);
                    step(std::false_type(), std::true_type(), s + 1);
                }
            }
            cp_async_wait<0>();
        }
        if (sweep_reduces(TAIL) && g.partials)
        {
            __shared__ double scratch[32];
            const double sum = block_sum(part, scratch);
            if (threadIdx.x == 0) g.partials[blockIdx.x] = sum;
        }
    }

    // Rows per chunk: the smallest estimate of the pass's time over a few heights.  A warp
    // takes rows + 2 HALO + 2 NS - 1 steps; with 1, 2, 3 and 4 blocks on an SM a step of all
    // of them takes about 1, 1.25, 1.75 and 2.3 times that of one (measured on the FP64
    // passes of levels 7 to 11: 0.29 us alone, 0.36 and 0.5 us; the model picks the fastest
    // or within 5 % of the fastest measured height at each level -- level 11: 48 rows 49.8 us
    // against 60.5 at 24 and 55.7 at 56; level 10: 20 rows 15.5 us, 12 rows 16.6, 40 rows 18.4).
    // The FP32 passes, those with a given Jacobi vector and those without sweeps use the same step
    // costs; theirs were not measured.
    inline int sweep_chunk_rows(int m, int strips, int halo, int ns, int per_sm, uint64_t nvec)
    {
        static const int cand[] = {2, 4, 6, 8, 10, 12, 16, 20, 24, 28, 32, 36, 40, 44, 48, 52, 56, 60, 64, 72, 80, 96,
                                   112, 128, 160, 192, 256};
        static const double step[] = {0.0, 1.0, 1.25, 1.75, 2.3};
        const uint64_t sms = (uint64_t)num_sms(), wave = sms * per_sm;
        double best = 0;
        int rows = 8;
        for (int r : cand)
        {
            const uint64_t blocks = ceil_div((uint64_t)strips * ceil_div(m, r), kSweepWarps) * nvec;
            const uint64_t full = blocks / wave, rest = blocks % wave;
            const double t = (std::min(r, m) + 2 * halo + 2 * ns - 1) * (full * step[per_sm] + step[ceil_div(rest, sms)]);
            if (best == 0 || t < best) { best = t; rows = r; }
        }
        return rows;
    }

    template <typename T, int C, bool UNI, int S, int HEAD, int TAIL, bool PVEC>
    int q1_sweep_launch_one(Q1SweepArgs<T> g, uint64_t nvec, uint64_t max_vec, uint64_t cap, uint32_t max_partials, unsigned * blocks,
                            cudaStream_t stream)
    {
        typedef Q1SweepShape<T, C, S, HEAD, TAIL> K;
        g.strips = (g.m + K::WV - 1) / K::WV;
        g.rows = sweep_chunk_rows(g.m, g.strips, K::HALO, K::NS, sweep_blocks_per_sm<T, C>(), nvec);
        if (sweep_reduces(TAIL) && g.partials)
            while ((uint64_t)g.strips * ((g.m + g.rows - 1) / g.rows) / kSweepWarps + 1 > max_partials) g.rows *= 2;   // even stays even
        g.chunks = (g.m + g.rows - 1) / g.rows;
        g.bpv = (g.strips * g.chunks + kSweepWarps - 1) / kSweepWarps;
        const size_t smem = K::ring(PVEC) * sizeof(T) * kSweepWarps;
        auto kern = q1_sweep_kernel<T, C, UNI, S, HEAD, TAIL, PVEC>;
        const cudaError_t attr = smem_opt_in((const void *)kern, smem);
        if (attr != cudaSuccess) return cuda_status(attr, "Q1 sweep kernel: shared memory");
        uint64_t grid = (uint64_t)g.bpv * (g.list ? max_vec : 1);
        if (g.list && cap) grid = std::min(grid, cap);
        launch_pdl(kern, dim3((unsigned)grid), dim3(32 * kSweepWarps), smem, stream, g);
        count_launches(1);
        if (blocks) *blocks = (unsigned)grid;
        HB2_LAUNCH_CHECK("Q1 sweep launch");
        return HB2_OK;
    }
}
