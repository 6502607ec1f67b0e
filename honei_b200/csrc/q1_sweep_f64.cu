// The Q1 sweep kernel in FP64: 2 columns a lane on the large grids, 1 on the small ones.
#include "q1_sweep_impl.cuh"

namespace hb2
{
    int q1_sweep_f64(const Q1SweepArgs<double> & g, bool wide, bool uni, int S, int head, int tail, bool pvec,
                     const SweepLaunch & l)
    {
        return q1_sweep_typed<double, 2, 1>(g, wide, uni, S, head, tail, pvec, l);
    }
}
