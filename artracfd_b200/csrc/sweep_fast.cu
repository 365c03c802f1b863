// Stage kernels, fast FP64 form (FMA-contracted).
#define ACFD_FORM 1
#define ACFD_NS form_fast
#include "sweep_impl.cuh"

namespace acfd {

int launch_stage_fast(const Grid &g, const ModelParams &m, const StageArgs &a, int s, bool viscous,
                       cudaStream_t st)
{
    return form_fast::launch_stage_impl(g, m, a, s, viscous, st);
}

int launch_weno_batch_fast(int scheme, const double *F, double *out, int count, cudaStream_t st)
{
    return form_fast::launch_weno_batch_impl(scheme, F, out, count, st);
}

int launch_fhat_batch_fast(const ModelParams &m, int s, const double *U, double *out, int count,
                            cudaStream_t st)
{
    return form_fast::launch_fhat_batch_impl(m, s, U, out, count, st);
}

}  // namespace acfd

#include "sweep_brick.cuh"

namespace acfd {

int launch_stage_brick_fast(const Grid &g, const ModelParams &m, const StageArgs &a, int s, bool viscous,
                            cudaStream_t st)
{
    return form_fast::launch_brick_impl(g, m, a, s, viscous, st);
}

}  // namespace acfd

#include "sweep_march.cuh"

namespace acfd {

int launch_stage_march_fast(const Grid &g, const ModelParams &m, const StageArgs &a, int s, bool viscous,
                            int target, cudaStream_t st)
{
    return form_fast::launch_march_impl(g, m, a, s, viscous, false, target, st);
}

}  // namespace acfd

#include "sweep_line.cuh"

namespace acfd {

int launch_stage_line(const Grid &g, const ModelParams &m, const StageArgs &a, int s, bool viscous, const LineTile &lt,
                      const CUtensorMap &map, const CUtensorMap &omap, cudaStream_t st)
{
    return form_fast::launch_line_impl(g, m, a, s, viscous, lt, map, omap, st);
}

int launch_line_roots(const double *x, double *rsqrt, double *rcp, int count, cudaStream_t st)
{
    if (count <= 0) return ACFD_OK;
    form_fast::line::roots<<<(unsigned)((count + 255LL) / 256), 256, 0, st>>>(x, rsqrt, rcp, count);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? ACFD_OK : cuda_status(e, "line roots launch");
}

}  // namespace acfd
