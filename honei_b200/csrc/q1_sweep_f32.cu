// The Q1 sweep kernel in FP32: two columns a lane (four: level 11 34.9 us against 35.4, but
// level 10 12.0 against 11.6 and more on the smaller grids).
#include "q1_sweep_impl.cuh"

namespace hb2
{
    int q1_sweep_f32(const Q1SweepArgs<float> & g, bool wide, bool uni, int S, int head, int tail, bool pvec,
                     const SweepLaunch & l)
    {
        return q1_sweep_typed<float, 2, 2>(g, wide, uni, S, head, tail, pvec, l);
    }
}
