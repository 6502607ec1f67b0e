// CGSolver<Tag, methods::NONE> (math/cg.hh:64-135) on a Q1 grid operator of a few hundred to
// some ten thousand rows, on one thread-block cluster.
//
// Such a solve is a chain of a few hundred steps with two dot products each; what it costs is
// the distance the data and the dots travel.  The cooperative form (cg.cu) keeps the vectors
// in global memory, reads the matrix again each step and meets three times at a grid barrier
// in global memory: 12 to 16 us a step at level 7.  Here a CTA owns a slab of grid lines with
// x, r, p and v in registers and p in shared memory with one halo line each side; the matrix
// is the nine kernel-parameter values.  A step meets twice, at the cluster's hardware barrier:
// once for <A p, p>, once for <r, r>, whose barrier also publishes the slab's first and last
// lines of r -- the neighbours form the halo lines of the next p from them by the same update
// (the same bits), instead of waiting for p at a third barrier.  Dots are FP64 tensor-core warp
// sums, one value per CTA written to every CTA's shared memory, and summed by each warp in rank
// order, so all CTAs hold the same bits and leave the loop together.
#include "cg_warp.cuh"
#include "smem_opt_in.hh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace hb2
{
    constexpr int kCgClusterMax = 16;

    template <typename T>
    struct CgClusterArgs
    {
        T v[9], vb;             // interior row, boundary diagonal
        int m, lines;           // points per line; lines per CTA
        const T * b;
        T * x;
        uint64_t max_iters;
        double eps;
        uint64_t * used;
        double * defect;
    };

    template <typename T, int E>
    __global__ void __launch_bounds__(1024 / (E > 4 ? 2 : 1), 1)
    cg_cluster_kernel(const __grid_constant__ CgClusterArgs<T> g)
    {
        typedef Arith<T> M;
        extern __shared__ __align__(16) unsigned char cgc_smem[];
        __shared__ double slots[2][kCgClusterMax], wred[32];
        cg::cluster_group cluster = cg::this_cluster();
        const int rank = (int)cluster.block_rank(), nc = (int)cluster.num_blocks();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
        const int m = g.m, l0 = rank * g.lines, nl = max(0, min(m, l0 + g.lines) - l0), cnt = nl * m;
        T * p = reinterpret_cast<T *>(cgc_smem);        // (lines + 2) * m: p with its halo lines
        T * rh = p + (size_t)(g.lines + 2) * m;         // r on the line before and the line after the slab
        const int64_t g0 = (int64_t)l0 * m;
        // the neighbours' copies of this slab's first and last line
        T * up = rank > 0 && nl > 0 ? cluster.map_shared_rank(rh, rank - 1) + m : nullptr;
        T * down = nl > 0 && l0 + nl < m ? cluster.map_shared_rank(rh, rank + 1) : nullptr;
        T xr[E], rr[E], vr[E];
        bool ok[E], bnd[E];
#pragma unroll
        for (int e = 0; e < E; ++e)
        {
            const int k = (int)threadIdx.x + e * (int)blockDim.x, i = l0 + k / m, j = k % m;
            ok[e] = k < cnt;
            bnd[e] = i == 0 || i == m - 1 || j == 0 || j == m - 1;
            xr[e] = ok[e] ? g.x[g0 + k] : T(0);
            rr[e] = vr[e] = T(0);
        }
        // x with its halo lines, for the first defect
        for (int k = threadIdx.x; k < (nl + 2) * m && nl > 0; k += blockDim.x)
        {
            const int64_t s = g0 - m + k;
            p[k] = s >= 0 && s < (int64_t)m * m ? g.x[s] : T(0);
        }
        cluster.sync();     // every CTA runs before its shared memory is written from another
        auto product = [&](int e) -> T {
            const T * c = p + m + (int)threadIdx.x + e * (int)blockDim.x;
            if (bnd[e]) return M::mul(g.vb, c[0]);
            T s = M::mul(g.v[0], c[-m - 1]);
            s = M::add(s, M::mul(g.v[1], c[-m]));
            s = M::add(s, M::mul(g.v[2], c[-m + 1]));
            s = M::add(s, M::mul(g.v[3], c[-1]));
            s = M::add(s, M::mul(g.v[4], c[0]));
            s = M::add(s, M::mul(g.v[5], c[1]));
            s = M::add(s, M::mul(g.v[6], c[m - 1]));
            s = M::add(s, M::mul(g.v[7], c[m]));
            s = M::add(s, M::mul(g.v[8], c[m + 1]));
            return s;
        };
        // the sum of `part` over the cluster, in every thread; the barrier also publishes what
        // the CTAs wrote into each other's shared memory before it
        auto total = [&](double part, double * slot) -> double {
            part = warp_sum_mma(part);
            if (lane == 0) wred[warp] = part;
            __syncthreads();
            if (warp == 0)
            {
                const double s = warp_sum_mma(lane < nwarps ? wred[lane] : 0.0);
                if (lane < nc) cluster.map_shared_rank(slot, lane)[rank] = s;
            }
            cluster.sync();
            return warp_sum_mma(lane < nc ? slot[lane] : 0.0);
        };
        auto publish = [&](int e) {
            const int k = (int)threadIdx.x + e * (int)blockDim.x;
            if (up && k < m) up[k] = rr[e];
            if (down && k >= cnt - m) down[k - (cnt - m)] = rr[e];
        };
        double part = 0.0;
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (ok[e])
            {
                rr[e] = M::sub(g.b[g0 + threadIdx.x + e * (int)blockDim.x], product(e));
                publish(e);
                part = fma((double)rr[e], (double)rr[e], part);
            }
        T alpha = (T)total(part, slots[1]);
        // p = r, the halo lines too
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (ok[e]) p[m + threadIdx.x + e * (int)blockDim.x] = rr[e];
        for (int k = threadIdx.x; k < m && nl > 0; k += blockDim.x)
        {
            p[k] = l0 > 0 ? rh[k] : T(0);
            p[m + cnt + k] = l0 + nl < m ? rh[m + k] : T(0);
        }
        __syncthreads();
        const T eps = T(g.eps), initial = sqrt(alpha);
        T current = initial;
        uint64_t it = 0, used = 0;
        while (it < g.max_iters)
        {
            part = 0.0;
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (ok[e])
                {
                    vr[e] = product(e);
                    part = fma((double)vr[e], (double)p[m + threadIdx.x + e * (int)blockDim.x], part);
                }
            const T temp = (T)total(part, slots[0]);
            const T lambda = M::div(alpha, guard(temp)), mlambda = -lambda;
            part = 0.0;
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (ok[e])
                {
                    xr[e] = M::add(xr[e], M::mul(lambda, p[m + threadIdx.x + e * (int)blockDim.x]));
                    rr[e] = M::add(rr[e], M::mul(mlambda, vr[e]));
                    publish(e);
                    part = fma((double)rr[e], (double)rr[e], part);
                }
            const T alpha_old = alpha;
            alpha = (T)total(part, slots[1]);
            ++it;
            current = sqrt(alpha);
            const bool stop = current < M::mul(eps, initial) || current < eps;
            if (stop || it == g.max_iters) used = it;
            if (stop) break;
            const T talpha = M::div(alpha, guard(alpha_old));
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (ok[e])
                {
                    T & q = p[m + threadIdx.x + e * (int)blockDim.x];
                    q = M::add(M::mul(q, talpha), rr[e]);
                }
            for (int k = threadIdx.x; k < m && nl > 0; k += blockDim.x)
            {
                if (l0 > 0) p[k] = M::add(M::mul(p[k], talpha), rh[k]);
                if (l0 + nl < m) p[m + cnt + k] = M::add(M::mul(p[m + cnt + k], talpha), rh[m + k]);
            }
            __syncthreads();
        }
#pragma unroll
        for (int e = 0; e < E; ++e)
            if (ok[e]) g.x[g0 + threadIdx.x + e * (int)blockDim.x] = xr[e];
        if (rank == 0 && threadIdx.x == 0)
        {
            *g.used = used;
            *g.defect = (double)current;
        }
        cluster.sync();     // no CTA leaves while others may still write into its shared memory
    }

    // the launch: `nc` CTAs of `threads` threads with E nodes a thread
    template <typename T, int E>
    static cudaError_t launch_e(const CgClusterArgs<T> & g, int nc, int threads, bool probe, cudaStream_t s)
    {
        const size_t smem = ((size_t)(g.lines + 4) * g.m) * sizeof(T) + 16;
        auto kern = cg_cluster_kernel<T, E>;
        cudaError_t e = smem_opt_in((const void *)kern, smem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess) return e;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(nc);
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = nc;
        at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (probe)
        {
            int n = 0;
            e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
            return e != cudaSuccess ? e : (n > 0 ? cudaSuccess : cudaErrorLaunchOutOfResources);
        }
        return cudaLaunchKernelEx(&cfg, kern, g);
    }

    template <typename T>
    static int solve_typed(const hb2_ell_s * A, const void * b, void * x, uint64_t max_iters, double eps,
                           uint64_t * used_dev, double * defect_dev, cudaStream_t s)
    {
        CgClusterArgs<T> g;
        for (int k = 0; k < 9; ++k) g.v[k] = (T)A->q1g_v[k];
        g.vb = (T)A->q1g_vb;
        g.m = (int)A->q1g_m;
        g.b = (const T *)b;
        g.x = (T *)x;
        g.max_iters = max_iters;
        g.eps = eps;
        g.used = used_dev;
        g.defect = defect_dev;
        // about 600 nodes a CTA (one CTA up to 1,200 nodes), at most 16 CTAs
        const int n = g.m * g.m;
        int nc = n <= 1200 ? 1 : std::min(kCgClusterMax, std::max(2, n / 600));
        while (nc & (nc - 1)) --nc;
        for (; nc >= 1; nc >>= 1)
        {
            g.lines = (g.m + nc - 1) / nc;
            const int cnt = g.lines * g.m;
            const int E = cnt <= 512 ? 1 : (cnt <= 2048 ? 2 : (cnt <= 4096 ? 4 : 9));
            const int threads = std::max(32, (int)(ceil_div(ceil_div(cnt, E), 32) * 32));
            if (threads > (E > 4 ? 512 : 1024)) break;
            cudaError_t e = cudaSuccess;
            for (int probe = 1; probe >= 0 && e == cudaSuccess; --probe)
                e = E == 1   ? launch_e<T, 1>(g, nc, threads, probe, s)
                    : E == 2 ? launch_e<T, 2>(g, nc, threads, probe, s)
                    : E == 4 ? launch_e<T, 4>(g, nc, threads, probe, s)
                             : launch_e<T, 9>(g, nc, threads, probe, s);
            if (e == cudaSuccess)
            {
                count_launches(1);
                return HB2_OK;
            }
            cudaGetLastError();     // this cluster width cannot be resident: the next narrower one
        }
        return HB2_ERR_UNSUPPORTED;
    }

    bool cg_cluster_applies(const hb2_ell_s * A)
    {
        return A->q1g_m >= 12 && A->q1g_m <= 270;      // below: one warp (cg.cu); above: no room for the slabs
    }

    int launch_cg_cluster(const hb2_ell_s * A, const void * b, void * x, uint64_t max_iters, double eps,
                          uint64_t * used_dev, double * defect_dev, cudaStream_t s)
    {
        return A->dtype == HB2_F64 ? solve_typed<double>(A, b, x, max_iters, eps, used_dev, defect_dev, s)
                                   : solve_typed<float>(A, b, x, max_iters, eps, used_dev, defect_dev, s);
    }
}
