// Instantiations of the Q1 sweep kernel for one element type (q1_sweep_f64.cu,
// q1_sweep_f32.cu): the runtime choices turned into template arguments.
#pragma once

#include "q1_sweep.cuh"

namespace hb2
{
    struct SweepLaunch
    {
        uint64_t nvec, max_vec, cap;
        uint32_t max_partials;
        unsigned * blocks;
        cudaStream_t stream;
    };

    template <typename T, int C, bool UNI, int HEAD, int TAIL, bool PVEC>
    static int q1_sweep_s(const Q1SweepArgs<T> & g, int S, const SweepLaunch & l)
    {
#define HB2_SW(S_) q1_sweep_launch_one<T, C, UNI, S_, HEAD, TAIL, PVEC>(g, l.nvec, l.max_vec, l.cap, l.max_partials, l.blocks, l.stream)
        switch (S)
        {
            case 1: return HB2_SW(1);
            case 2: return HB2_SW(2);
            case 3: return HB2_SW(3);
            default: return HB2_SW(4);
        }
#undef HB2_SW
    }

    template <typename T, int C, bool UNI>
    static int q1_sweep_kind(const Q1SweepArgs<T> & g, int S, int head, int tail, const SweepLaunch & l)
    {
        if (head == kSweepZero)
            return tail == kSweepRestrict ? q1_sweep_s<T, C, UNI, kSweepZero, kSweepRestrict, false>(g, S, l)
                                          : q1_sweep_s<T, C, UNI, kSweepZero, kSweepStore, false>(g, S, l);
        if (tail == kSweepRestrict) return q1_sweep_s<T, C, UNI, kSweepLoad, kSweepRestrict, false>(g, S, l);
        if (tail == kSweepNorm) return q1_sweep_s<T, C, UNI, kSweepLoad, kSweepNorm, false>(g, S, l);
        return q1_sweep_s<T, C, UNI, kSweepLoad, kSweepStore, false>(g, S, l);
    }

    // the passes without sweeps, on the wide form
    template <typename T, int C, bool UNI>
    static int q1_single(const Q1SweepArgs<T> & g, int tail, const SweepLaunch & l)
    {
#define HB2_SG(TAIL_) q1_sweep_launch_one<T, C, UNI, 0, kSweepLoad, TAIL_, false>(g, l.nvec, l.max_vec, l.cap, l.max_partials, l.blocks, l.stream)
        switch (tail)
        {
            case kSweepDefect: return HB2_SG(kSweepDefect);
            case kSweepProduct: return HB2_SG(kSweepProduct);
            case kSweepDot: return HB2_SG(kSweepDot);
            default:
                if constexpr (sizeof(T) == 8) return HB2_SG(kSweepDefectIR);
                else return fail(HB2_ERR_UNSUPPORTED, "Q1 pass");
        }
#undef HB2_SG
    }

    // CW columns a lane when wide, else CN; the general nine-value form in one width
    template <typename T, int CW, int CN>
    static int q1_sweep_typed(const Q1SweepArgs<T> & g, bool wide, bool uni, int S, int head, int tail, bool pvec,
                              const SweepLaunch & l)
    {
        // the passes without sweeps and the given Jacobi vector: the form that is fast on the
        // middle grids too (16 bytes a lane in FP64, 8 in FP32)
        constexpr int CM = sizeof(T) == 8 ? CW : CN;
        if (sweep_single(tail)) return uni ? q1_single<T, CM, true>(g, tail, l) : q1_single<T, CM, false>(g, tail, l);
        if (pvec)
            return uni ? q1_sweep_s<T, CM, true, kSweepLoad, kSweepStore, true>(g, S, l)
                       : q1_sweep_s<T, CM, false, kSweepLoad, kSweepStore, true>(g, S, l);
        if (! uni) return q1_sweep_kind<T, CM, false>(g, S, head, tail, l);
        return wide ? q1_sweep_kind<T, CW, true>(g, S, head, tail, l) : q1_sweep_kind<T, CN, true>(g, S, head, tail, l);
    }
}
