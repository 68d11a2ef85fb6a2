// Abelian-Higgs step kernels, float instantiation: the FP32 pair step
// (pair_step.cuh, the tiled step of tiled_step.cuh for checks) and the one-pass kernel kept for cross-checks.
#include <algorithm>

#include "ah_step.cuh"
#include "pair_step.cuh"
#include "tiled_step.cuh"

namespace lat {

cudaError_t launch_ah_step_f32(const Geom& g, const Fields<float, 5>& f, const StepCoef& c, const DiagOut& d, bool diag,
                               cudaStream_t st)
{
    return launch_ah_step_t<float>(g, f, c, d, diag, st);
}

// variant 0: the pair step; 2: the tiled step staging one element per
// copy; 3: the tiled step with 16-byte staging where allowed.  *blocks: room for
// diagnostic partials in, the CTAs (and partials) of the kernel that ran out.
cudaError_t launch_ah_tiled_f32(const Geom& g, const Fields<float, 5>& f, const StepCoef& c, const DiagOut& d,
                                  bool diag, int chunk, cudaStream_t st, int variant, int* blocks)
{
    if (variant == 0) return launch_pair_t<1>(g, f, c, d, diag, chunk, st, blocks);
    const dim3 t = tiled_grid(g, chunk);
    const int ctas = (int)(t.x * t.y * t.z);
    if (diag && ctas > *blocks) return cudaErrorInvalidConfiguration;
    *blocks = ctas;
    return launch_tiled_t<float, 1>(g, f, c, d, diag, chunk, st, variant != 2);
}

cudaError_t launch_divergence_f32(const Geom& g, const float* tx, const float* ty, const float* tz, const StepCoef& c,
                                  float* out, cudaStream_t st)
{
    return launch_divergence_t<float>(g, tx, ty, tz, c, out, st);
}

}  // namespace lat

namespace lat {

int64_t march_tiles(const Geom& g, bool moore)
{
    const dim3 t = pair_shape_grid(g, moore ? 32 : pair_tz2(g), 1), w = tiled_grid(g, 1);
    return !moore || pair_moore_fits(g) ? (int64_t)t.x * t.y : (int64_t)w.x * w.y;
}

int64_t march_tiles_most(const Geom& g)
{
    int64_t most = 0;
    for (const dim3 t : {pair_shape_grid(g, 32, 1), pair_shape_grid(g, 16, 1), tiled_grid(g, 1)})
        most = std::max(most, (int64_t)t.x * t.y);
    return most;
}

}  // namespace lat
