// Moore-model marching FP64 step, LAT_F64_FAST variant (compiled with
// multiply-add contraction).
#include "moore_march.cuh"

namespace lat {

cudaError_t launch_moore_march_fast(const Geom& g, const Fields<double, 7>& f, const StepCoef& c, const DiagOut& d,
                                    bool diag, bool recip, cudaStream_t st)
{
    return launch_moore_march_t<false>(g, f, c, d, diag, recip, st);
}

}  // namespace lat
