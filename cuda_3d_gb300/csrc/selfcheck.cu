// selfcheck.cu -- the short FP64 routines of the pose update (pose_math.cuh)
// against CUDA's IEEE division and sincos, on the device that runs them.
#include "pose_math.cuh"

#include <algorithm>

namespace gca3d
{

__device__ __forceinline__ void max_into(double *slot, double v)
{
    // non-negative doubles order as their bit patterns
    atomicMax(reinterpret_cast<unsigned long long *>(slot), (unsigned long long)__double_as_longlong(v));
}

__global__ void k_selfcheck_fp64(int n, double *out)
{
    constexpr double kEps = 2.220446049250313e-16;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        const double f = (double)i / (double)n;
        const double d = exp2(-60.0 + 120.0 * f) * (1.0 + 0.37 * sin((double)i));
        const double q = 1.0 / d;
        max_into(&out[0], fabs(rcp_nr(d) - q) / (fabs(q) * kEps));
        const double x = -kSmallAngle + 2.0 * kSmallAngle * f;
        double s0, c0;
        sincos(x, &s0, &c0);
        // as the finalize calls them: neighbouring lanes for neighbouring results
        const bool cosine = threadIdx.x & 1;
        const double ref = cosine ? c0 : s0, got = sin_or_cos_small(x, cosine);
        if (ref != 0.0)
            max_into(&out[cosine ? 2 : 1], fabs(got - ref) / (fabs(ref) * kEps));
        const double t = 0.05 + (kSmallAngle - 0.05) * f, t2 = t * t;
        const int m = threadIdx.x % 3;
        const double coeff = exp_coeff_small(t2, m);
        double st, ct;
        sincos(t, &st, &ct);
        const double coeff0 = m == 0 ? st / t : (m == 1 ? (1.0 - ct) / t2 : (t - st) / (t2 * t));
        // the closed forms cancel: 1 - cos t and t - sin t keep about t^2 / 2 and t^2 / 6
        // of their operands, so their rounding error is within eps (4 + 8 / t^2)
        const double bound = kEps * (4.0 + 8.0 / t2);
        max_into(&out[3], fabs(coeff - coeff0) / coeff0 / bound);
    }
}

} // namespace gca3d

using namespace gca3d;

extern "C" int gca3d_selfcheck_fp64(gca3d_context *ctx, int n, double out[4])
{
    if (!ctx || !out || n < 1)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "selfcheck: bad arguments");
    ctx->arena.reset();
    double *d_out = ctx->arena.get<double>(4);
    if (!d_out)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "selfcheck: scratch");
    GCA_CUDA(ctx, cudaMemsetAsync(d_out, 0, 4 * sizeof(double), ctx->stream));
    k_selfcheck_fp64<<<std::min((n + 255) / 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(n, d_out);
    GCA_CHECK_LAUNCH(ctx);
    GCA_CUDA(ctx, cudaMemcpyAsync(out, d_out, 4 * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    GCA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return consume_device_error(ctx, "selfcheck");
}
