// Moore-model step kernels, double instantiation: the marching step
// (moore_march.cuh) and the one-pass kernel kept for cross-checks.
#include "moore_march.cuh"
#include "moore_step.cuh"

namespace lat {

cudaError_t launch_moore_step_f64(const Geom& g, const Fields<double, 7>& f, const StepCoef& c, const DiagOut& d,
                                  bool diag, cudaStream_t st)
{
    return launch_moore_step_t<double>(g, f, c, d, diag, st);
}

int64_t moore_march_partials(const Geom& g) { return march64_ctas(g); }

cudaError_t launch_moore_march_strict(const Geom& g, const Fields<double, 7>& f, const StepCoef& c, const DiagOut& d,
                                      bool diag, bool recip, cudaStream_t st)
{
    return launch_moore_march_t<true>(g, f, c, d, diag, recip, st);
}

}  // namespace lat
