// The Q1 sweep kernel in FP32: four columns a lane on the largest grids, two below.
#include "q1_sweep_impl.cuh"

namespace hb2
{
    int q1_sweep_f32(const Q1SweepArgs<float> & g, bool wide, bool uni, int S, int head, int tail, bool pvec,
                     const SweepLaunch & l)
    {
        return q1_sweep_typed<float, 4, 2>(g, wide, uni, S, head, tail, pvec, l);
    }
}
