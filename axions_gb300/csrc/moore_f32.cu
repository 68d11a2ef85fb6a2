// Moore-model step kernels, float instantiation: the FP32 pair step
// (pair_step.cuh, the tiled step of tiled_step.cuh for checks, two scalars) and the one-pass kernel kept for cross-checks.
#include "moore_step.cuh"
#include "pair_step.cuh"
#include "tiled_step.cuh"

namespace lat {

cudaError_t launch_moore_step_f32(const Geom& g, const Fields<float, 7>& f, const StepCoef& c, const DiagOut& d,
                                  bool diag, cudaStream_t st)
{
    return launch_moore_step_t<float>(g, f, c, d, diag, st);
}

// variant 0: the pair step (pair_moore_ok), else the tiled step; 2: the tiled step staging one element per
// copy; 3: the tiled step with 16-byte staging where allowed.  *blocks: room for
// diagnostic partials in, the CTAs (and partials) of the kernel that ran out.
cudaError_t launch_moore_tiled_f32(const Geom& g, const Fields<float, 7>& f, const StepCoef& c, const DiagOut& d,
                                     bool diag, int chunk, cudaStream_t st, int variant, int* blocks)
{
    if (variant == 0 && pair_moore_ok(g, f)) return launch_pair_t<2>(g, f, c, d, diag, chunk, st, blocks);
    const dim3 t = tiled_grid(g, chunk);
    const int ctas = (int)(t.x * t.y * t.z);
    if (diag && ctas > *blocks) return cudaErrorInvalidConfiguration;
    *blocks = ctas;
    return launch_tiled_t<float, 2>(g, f, c, d, diag, chunk, st, variant != 2);
}

}  // namespace lat
