// vjp.cu -- K unrolled Gauss-Newton steps of the colored-ICP objective and their
// adjoint with respect to the initial pose, the source points and the source
// colours.  No reference counterpart; the per-point rows are those of
// compute_JTJ_JTr_and_r_gauss_newton_functor
// (src/registration/cuda_color_icp_build_least_square.cu:184-253) and the step is
// solve_JTJ_JTr (src/registration/eigen_solver.hpp:44-85) with the chosen map.
//
// Forward: the ICP kernels run K + 1 evaluations of one pair from T_0 = Exp(xi0)
// with the convergence test switched off; every evaluation keeps its
// correspondences in its own buffer, and the finalize of each records the pose it
// started from, the summed system and the step (IcpTrace).  Evaluation K only
// supplies T_K and the objective E = sum of weighted r_g^2 + r_c^2 at T_K.
//
// Backward, from nothing but the recorded poses, systems and 6-vectors (the Jacobians are
// recomputed from the points, none is stored).  One launch prepares every step at once
// (k_vjp_prep, a block per step): U_k, dU_k / dx and the factored H_k, which do not depend on
// the cotangents.  Then evaluation k from K down to 0, one launch each (k_vjp_points):
//   point adjoint (FP32 per point): every row (j, r) of a correspondence gets
//     jbar = -y (j.x) - x (j.y) - r y  and  rbar = -(j.y) + 2 e r
//     (x = y = 0 and e = dE at evaluation K), pushed through j = w [p x dir; dir]
//     and r to pbar and to the source intensity; sbar = R_k^T pbar and
//     cbar = Ibar (0.2126, 0.7152, 0.0722); Tbar_k += sum over points of
//     pbar [s^T 1], compensated FP32 in the block and FP64 across blocks;
//   step adjoint (FP64, by the launch's last block, once Tbar_k is complete):
//     Ubar = Tbar_k T_{k-1}^T, xbar = dU/dx : Ubar, y = H_{k-1}^-1 xbar,
//     Tbar_{k-1} = U_{k-1}^T Tbar_k (x = -H^-1 b gives bbar = -y and Hbar = -y x^T);
//     after evaluation 0, xi0bar = dExp(xi0)/dxi : Tbar_0.
// Correspondences are held fixed: they are piecewise constant in the inputs.
//
// What bounds it is the chain of launches and of dependent FP64 operations, not the points.
// 100,000 points, K = 5 (GB300): a step adjoint in one thread was a launch of 51 us; what of
// it does not depend on the cotangents now runs once for all steps (13 us) and the rest, a
// few microseconds, in the point launch's last block.  The call: 904 to 680 us (612 with
// the shorter finalize and search of the forward pass).  The 391
// block partials are still added one after the other (12 us of a point launch: an FP64
// addition takes 64 cycles); running sums in a fixed order, as the finalize has them, would
// shorten that chain.
#include "icp.cuh"
#include "pose_math.cuh"
#include "stages.cuh"

#include <cmath>

using namespace gca3d;

namespace
{

constexpr int kVjpThreads = 256;
constexpr int kTb = 12; // entries of Tbar (rows 0-2 of the 4x4)
constexpr int kTbPad = 16;

struct Vec6
{
    double v[6];
};
struct Mat34
{
    double v[12];
};

// what a step's adjoint needs besides the cotangents: the step's pose increment U, its
// derivatives dU/dx, and the factored system; in the entry after the last step dU is
// dExp(xi0)/dxi
struct VjpStep
{
    double U[16];
    double dU[6][kTb];
    double A[6][6], D[6];
    int perm[6];
    int finite, singular;
};

// T_0 = Exp(xi0)
__global__ void k_vjp_init(PairState *st, Vec6 xi0)
{
    if (threadIdx.x != 0)
        return;
    double T[16];
    pose_from_x_device(xi0.v, GCA3D_UPDATE_SE3_EXP, T);
    for (int k = 0; k < 16; ++k)
        st[0].T[k] = T[k];
    for (int k = 0; k < 12; ++k)
        st[0].Tf[k] = (float)T[k];
    st[0].iters = 0;
    st[0].status = 0;
    st[0].rmse_ref = st[0].fitness = st[0].inlier_rmse = 0.0;
}

// block k < K: U_k, its derivatives (lane m of warp 0 by x_m) and, in warp 1, the factored
// system; block K: dExp(xi0)/dxi and the seed of Tbar_K
__global__ void __launch_bounds__(96) k_vjp_prep(const IcpTrace *trace, int K, int map, Vec6 xi0, Mat34 dT,
                                                 VjpStep *steps, double *Tbar)
{
    const int k = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool last = k == K;
    VjpStep &o = steps[k];
    if (warp == 0)
    {
        double x[6], d[kTb];
#pragma unroll
        for (int m = 0; m < 6; ++m)
            x[m] = last ? xi0.v[m] : trace[k].x[m];
        pose_derivative_device(x, last ? GCA3D_UPDATE_SE3_EXP : map, lane < 6 ? lane : 0, d);
        if (lane < 6)
#pragma unroll
            for (int c = 0; c < kTb; ++c)
                o.dU[lane][c] = d[c];
        if (last && lane < kTb)
            Tbar[lane] = dT.v[lane];
        return;
    }
    if (last)
    {
        if (warp == 1 && lane == 0)
            o.singular = 0;
        return;
    }
    if (warp == 2)
    {
        double U[16];
        pose_from_x_device(trace[k].x, map, U);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < 16; ++q)
                o.U[q] = U[q];
        return;
    }
    double S[21], A[6][6], D[6];
    int perm[6];
    bool finite;
#pragma unroll
    for (int q = 0; q < 21; ++q)
        S[q] = trace[k].S[q];
    const int singular = solve6_factor(S, A, D, perm, finite);
    if (lane == 0)
    {
#pragma unroll
        for (int i = 0; i < 6; ++i)
        {
#pragma unroll
            for (int j = 0; j < 6; ++j)
                o.A[i][j] = A[i][j];
            o.D[i] = D[i];
            o.perm[i] = perm[i];
        }
        o.finite = finite;
        o.singular = singular || trace[k].status;
    }
}

// the adjoint of T_{k+1} = U(x_k) T_k and of x_k = -H_k^-1 b_k by one warp, from Tbar_{k+1} in
// s_next: Tbar_k and y_k.  Every entry is summed in the order of its formula, one lane each.
__device__ __forceinline__ void step_adjoint(const VjpStep *s, const IcpTrace *tr, const double *s_next, double *s_Ub,
                                             double *s_rhs, double *Tbar, double *y, int *bad)
{
    const int lane = threadIdx.x & 31;
    if (lane < kTb)
    {
        const int a = lane >> 2, c = lane & 3;
        double u = 0.0, t = 0.0;
#pragma unroll
        for (int q = 0; q < 4; ++q)
            u += s_next[4 * a + q] * tr->T[4 * c + q];
#pragma unroll
        for (int q = 0; q < 3; ++q)
            t += s->U[4 * q + a] * s_next[4 * q + c];
        s_Ub[lane] = u;
        Tbar[lane] = t;
    }
    __syncwarp();
    if (lane < 6)
    {
        double v = 0.0;
#pragma unroll
        for (int c = 0; c < kTb; ++c)
            v += s_Ub[c] * s->dU[lane][c];
        s_rhs[lane] = -v; // the substitution returns -H^-1 (rhs): y = H^-1 xbar
    }
    __syncwarp();
    double yy[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    bool finite = s->finite != 0;
#pragma unroll
    for (int i = 0; i < 6; ++i)
        finite = finite && isfinite(s_rhs[i]);
    if (finite)
        solve6_substitute_warp(s->A, s->D, s->perm, s_rhs, yy);
    if (lane == 0)
    {
#pragma unroll
        for (int m = 0; m < 6; ++m)
            y[m] = yy[m];
        if (!finite)
            *bad = 1;
    }
}

__device__ __forceinline__ void two_sum_add(float &s, float &e, float x)
{
    const float t = s + x;
    const float bp = t - s;
    e += (s - (t - bp)) + (x - bp);
    s = t;
}

// adjoint of one row j = w [p x dir; dir], r: adds to pbar, returns rbar
__device__ __forceinline__ float row_adjoint(const float J[6], float r, float3 dir, float w, const float *x,
                                             const float *y, float e, float3 &pb)
{
    float jx = 0.0f, jy = 0.0f;
#pragma unroll
    for (int a = 0; a < 6; ++a)
    {
        jx += J[a] * x[a];
        jy += J[a] * y[a];
    }
    const float bx = -y[0] * jx - x[0] * jy - r * y[0];
    const float by = -y[1] * jx - x[1] * jy - r * y[1];
    const float bz = -y[2] * jx - x[2] * jy - r * y[2];
    const float rb = -jy + 2.0f * e * r;
    // d<jbar, p x dir> = <dp, dir x jbar>
    pb.x += w * (dir.y * bz - dir.z * by) + rb * w * dir.x;
    pb.y += w * (dir.z * bx - dir.x * bz) + rb * w * dir.y;
    pb.z += w * (dir.x * by - dir.y * bx) + rb * w * dir.z;
    return rb;
}

// evaluation k: First (evaluation K) stores the gradients, zero where a point has no
// correspondence, the later ones add theirs
template <bool First>
__global__ void __launch_bounds__(kVjpThreads)
    k_vjp_points(const float4 *__restrict__ src_pos, const int32_t *d_ns, const float4 *__restrict__ tpos,
                 const float4 *__restrict__ attr0, const float4 *__restrict__ attr1, const int2 *__restrict__ corr,
                 const IcpTrace *tr, double *y, float e, float slg, float slc, float *dxyz, float *drgb,
                 double *partials, unsigned *ticket, double *Tbar, VjpStep *prev, double *dxi)
{
    constexpr bool step = !First; // evaluation K takes no step
    __shared__ float s_T[12], s_x[6], s_y[6];
    __shared__ float s_s[kVjpThreads / 32][kTb], s_e[kVjpThreads / 32][kTb];
    __shared__ int s_last;
    if (threadIdx.x < 12)
        s_T[threadIdx.x] = (float)tr->T[threadIdx.x];
    if (threadIdx.x < 6)
    {
        s_x[threadIdx.x] = step ? (float)tr->x[threadIdx.x] : 0.0f;
        s_y[threadIdx.x] = step ? (float)y[threadIdx.x] : 0.0f;
    }
    __syncthreads();
    const int ns = *d_ns;
    float acc[kTb], err[kTb];
#pragma unroll
    for (int k = 0; k < kTb; ++k)
        acc[k] = err[k] = 0.0f;
    for (int i = blockIdx.x * kVjpThreads + threadIdx.x; i < ns; i += gridDim.x * kVjpThreads)
    {
        const int2 c = corr[i];
        if (c.x < 0)
        {
            if (First)
#pragma unroll
                for (int a = 0; a < 3; ++a)
                    dxyz[3 * i + a] = drgb[3 * i + a] = 0.0f;
            continue;
        }
        const float4 s4 = src_pos[i];
        const float3 p = apply_pose(s_T, s4);
        const float4 q = __ldg(&tpos[c.x]);
        const float4 a0 = __ldg(&attr0[c.x]);
        const float4 a1 = __ldg(&attr1[c.x]);
        const float3 n = make_float3(a0.x, a0.y, a0.z), d = make_float3(a1.x, a1.y, a1.z);
        GNTerms t;
        gn_terms(p, s4.w, make_float3(q.x, q.y, q.z), a0.w, n, d, slg, slc, t);
        const float nd = n.x * d.x + n.y * d.y + n.z * d.z;
        const float3 dt = make_float3(d.x - nd * n.x, d.y - nd * n.y, d.z - nd * n.z);
        float3 pb = make_float3(0.0f, 0.0f, 0.0f);
        row_adjoint(t.Jg, t.rg, n, slg, s_x, s_y, e, pb);
        const float rbc = row_adjoint(t.Jc, t.rc, dt, slc, s_x, s_y, e, pb);
        const float Ib = -rbc * slc;
        // p = R s + t
        const float gx[3] = {s_T[0] * pb.x + s_T[4] * pb.y + s_T[8] * pb.z,
                             s_T[1] * pb.x + s_T[5] * pb.y + s_T[9] * pb.z,
                             s_T[2] * pb.x + s_T[6] * pb.y + s_T[10] * pb.z};
        const float gc[3] = {Ib * 0.2126f, Ib * 0.7152f, Ib * 0.0722f};
#pragma unroll
        for (int a = 0; a < 3; ++a)
        {
            dxyz[3 * i + a] = First ? gx[a] : dxyz[3 * i + a] + gx[a];
            drgb[3 * i + a] = First ? gc[a] : drgb[3 * i + a] + gc[a];
        }
        const float pv[3] = {pb.x, pb.y, pb.z}, sv[3] = {s4.x, s4.y, s4.z};
#pragma unroll
        for (int r = 0; r < 3; ++r)
        {
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
                two_sum_add(acc[4 * r + cc], err[4 * r + cc], pv[r] * sv[cc]);
            two_sum_add(acc[4 * r + 3], err[4 * r + 3], pv[r]);
        }
    }
    // warp, then cross-warp two-sum reduction; one FP64 value per term and block
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < kTb; ++k)
        {
            const float s2 = __shfl_down_sync(0xffffffffu, acc[k], o);
            const float e2 = __shfl_down_sync(0xffffffffu, err[k], o);
            err[k] += e2;
            two_sum_add(acc[k], err[k], s2);
        }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < kTb; ++k)
        {
            s_s[warp][k] = acc[k];
            s_e[warp][k] = err[k];
        }
    __syncthreads();
    if (threadIdx.x < kTb)
    {
        float v = s_s[0][threadIdx.x], ev = s_e[0][threadIdx.x];
        for (int w = 1; w < kVjpThreads / 32; ++w)
        {
            ev += s_e[w][threadIdx.x];
            two_sum_add(v, ev, s_s[w][threadIdx.x]);
        }
        partials[(size_t)blockIdx.x * kTbPad + threadIdx.x] = (double)v + (double)ev;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last)
        return;
    // Tbar_k: the block partials in block order, kTile blocks at a time through shared memory
    // (loaded by the whole block, so the chain of additions waits on nothing else)
    constexpr int kTile = 64;
    __shared__ double s_part[2][kTile * kTb];
    __shared__ double s_Tb[kTb], s_Ub[kTb], s_rhs[6];
    // blocks first .. first + kTile - 1, by the threads from t0 on
    auto load = [&](int first, double *to, int t0) {
        const int n = min(kTile, (int)gridDim.x - first) * kTb;
        for (int j = (int)threadIdx.x - t0; j < n; j += kVjpThreads - t0)
            to[j] = __ldcg(partials + (size_t)(first + j / kTb) * kTbPad + j % kTb);
    };
    double v = 0.0;
    load(0, s_part[0], 0);
    __syncthreads();
    for (int first = 0, cur = 0; first < (int)gridDim.x; first += kTile, cur ^= 1)
    {
        if (first + kTile < (int)gridDim.x && warp > 0)
            load(first + kTile, s_part[cur ^ 1], 32);
        if (threadIdx.x < kTb)
        {
            const int n = min(kTile, (int)gridDim.x - first);
#pragma unroll 8
            for (int b = 0; b < n; ++b)
                v += s_part[cur][b * kTb + threadIdx.x];
        }
        __syncthreads();
    }
    if (warp > 0)
        return;
    if (lane < kTb)
        s_Tb[lane] = Tbar[lane] + v;
    if (lane == 0)
        *ticket = 0u;
    __syncwarp();
    if (dxi)
    {
        // evaluation 0: the initial pose's coordinates (prev: dExp(xi0)/dxi)
        if (lane < 6)
        {
            double d = 0.0;
            for (int c = 0; c < kTb; ++c)
                d += s_Tb[c] * prev->dU[lane][c];
            dxi[lane] = d;
        }
        return;
    }
    // the step before (tr - 1: its trace)
    step_adjoint(prev, tr - 1, s_Tb, s_Ub, s_rhs, Tbar - kTb, First ? y : y - 6, &prev->singular);
}

} // namespace

extern "C" int gca3d_color_icp_vjp(gca3d_context *ctx, gca3d_cloud *src, gca3d_cloud *tgt,
                                   const gca3d_vjp_params *p, const double xi0[6], const double dT[16], double dE,
                                   double T_out[16], double *E_out, double dxi0[6], float *d_dxyz, float *d_drgb,
                                   int32_t *d_corr)
{
    if (!ctx || !src || !tgt || !p || !xi0)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "icp vjp: null argument");
    if (p->K < 1 || p->K > GCA3D_VJP_MAX_STEPS || !(p->max_corr > 0.0f) || !(p->lambda >= 0.0f && p->lambda <= 1.0f) ||
        (p->update_map != GCA3D_UPDATE_EULER_ZYX && p->update_map != GCA3D_UPDATE_SE3_EXP))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "icp vjp: bad parameters (1 <= K <= 64, max_corr > 0)");
    if (!tgt->has_normals || !tgt->has_grad)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "icp vjp: the target needs normals and colour gradients");
    if (dT && (!dxi0 || !d_dxyz || !d_drgb))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "icp vjp: gradient outputs missing");
    const int K = p->K;
    ctx->arena.reset();
    // the point counts (the caller gets host results, so one read-back is due anyway)
    GCA_CUDA(ctx, cudaMemcpyAsync(ctx->h_pinned, src->d_count, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    GCA_CUDA(ctx,
             cudaMemcpyAsync(ctx->h_pinned + 1, tgt->d_count, sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    GCA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    const int64_t ns = ctx->h_pinned[0], nt = ctx->h_pinned[1];
    if (ns <= 0 || nt <= 0)
        return fail(ctx, GCA3D_ERR_NO_CORRESPONDENCES, "icp vjp: empty cloud");

    Batch bs, bt;
    int st;
    if ((st = cloud_batch(ctx, src, bs, false)) || (st = cloud_batch(ctx, tgt, bt, true)))
        return st;
    Grid g;
    if ((st = grid_build(ctx, bt, p->max_corr, kOriginPadF32, nullptr, g)))
        return st;
    const int max_blocks = std::max(div_up(src->capacity, kIcpChunk), 1);
    const int max_blocks_nn = std::max(div_up(src->capacity, kNNChunkSmall), 1);
    float4 *attr0 = ctx->arena.get<float4>(g.cap);
    float4 *attr1 = ctx->arena.get<float4>(g.cap);
    PairState *pst = ctx->arena.get<PairState>(1);
    int *bmap = ctx->arena.get<int>(3);
    int *bmap_nn = ctx->arena.get<int>(3);
    double *partials = ctx->arena.get<double>((size_t)max_blocks * kTermsPad);
    int2 *corr = ctx->arena.get<int2>((size_t)(K + 1) * src->capacity);
    const NNCerts cert{ctx->arena.get<float4>(src->capacity), ctx->arena.get<int>(src->capacity)};
    // what the host reads back in one copy: the traces, the step adjoints, the pose gradient
    const size_t rb_steps = sizeof(IcpTrace) * (K + 1), rb_dxi = rb_steps + sizeof(VjpStep) * (K + 1),
                 rb_bytes = rb_dxi + 6 * sizeof(double);
    static_assert((sizeof(IcpTrace) + sizeof(VjpStep)) * (GCA3D_VJP_MAX_STEPS + 1) + 48 <= kPinnedBytes - kPinnedBulk,
                  "the read-back fits the context's pinned buffer");
    char *readback = ctx->arena.get<char>(rb_bytes);
    IcpTrace *trace = reinterpret_cast<IcpTrace *>(readback);
    VjpStep *steps = reinterpret_cast<VjpStep *>(readback + rb_steps);
    double *d_dxi = reinterpret_cast<double *>(readback + rb_dxi);
    unsigned *fticket = ctx->arena.get<unsigned>(1);
    if (!attr0 || !attr1 || !pst || !bmap || !bmap_nn || !partials || !corr || !cert.pos || !cert.t || !readback ||
        !fticket)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "icp vjp: scratch");
    if ((st = gather_attrs(ctx, bt, g, tgt->nrm, tgt->grd, attr0, attr1)))
        return st;

    // forward: K steps plus the evaluation at T_K
    Vec6 x0;
    for (int m = 0; m < 6; ++m)
        x0.v[m] = xi0[m];
    k_vjp_init<<<1, 32, 0, ctx->stream>>>(pst, x0);
    GCA_CHECK_LAUNCH(ctx);
    const IcpShape shape;
    if ((st = icp_setup(ctx, pst, 1, bs.seg_off, bt.seg_off, bmap, bmap_nn, 0, shape.nn_chunk)))
        return st;
    IcpScale prm;
    prm.max_corr = p->max_corr;
    prm.sqrt_lg = sqrtf(p->lambda);
    prm.sqrt_lc = sqrtf(1.0f - p->lambda);
    prm.update_map = p->update_map;
    prm.cos_min = 2.0; // never converged: exactly K steps
    prm.trans_eps = -1.0;
    prm.trace = trace;
    prm.trace_cap = K + 1;
    GCA_CUDA(ctx, cudaMemsetAsync(fticket, 0, sizeof(unsigned), ctx->stream));
    IcpLoop loop;
    loop.ticket = fticket;
    for (int k = 0; k <= K; ++k)
        if ((st = icp_iteration(ctx, bs, g, attr0, attr1, pst, bmap, max_blocks, bmap_nn, max_blocks_nn, partials,
                                corr + (size_t)k * src->capacity, cert, prm, true,
                                d_corr ? d_corr + (size_t)k * ns : nullptr, loop, shape, k == 0)))
            return st;

    // backward
    if (dT)
    {
        const int nbv = std::max(std::min(div_up(ns, kVjpThreads), ctx->num_sms * 4), 1);
        double *Tbar = ctx->arena.get<double>((size_t)(K + 1) * kTb);
        double *ybuf = ctx->arena.get<double>((size_t)K * 6);
        double *vpart = ctx->arena.get<double>((size_t)nbv * kTbPad);
        unsigned *ticket = ctx->arena.get<unsigned>(1);
        if (!Tbar || !ybuf || !vpart || !ticket)
            return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "icp vjp: scratch");
        GCA_CUDA(ctx, cudaMemsetAsync(ticket, 0, sizeof(unsigned), ctx->stream));
        Mat34 seed;
        for (int k = 0; k < kTb; ++k)
            seed.v[k] = dT[k];
        k_vjp_prep<<<K + 1, 96, 0, ctx->stream>>>(trace, K, p->update_map, x0, seed, steps, Tbar + (size_t)K * kTb);
        GCA_CHECK_LAUNCH(ctx);
        const float slg = prm.sqrt_lg, slc = prm.sqrt_lc;
        k_vjp_points<true><<<nbv, kVjpThreads, 0, ctx->stream>>>(
            bs.pos, bs.seg_off + 1, g.dev.spos, attr0, attr1, corr + (size_t)K * src->capacity, trace + K,
            ybuf + 6 * (K - 1), (float)dE, slg, slc, d_dxyz, d_drgb, vpart, ticket, Tbar + (size_t)K * kTb,
            steps + K - 1, nullptr);
        GCA_CHECK_LAUNCH(ctx);
        for (int k = K - 1; k >= 0; --k)
        {
            k_vjp_points<false><<<nbv, kVjpThreads, 0, ctx->stream>>>(
                bs.pos, bs.seg_off + 1, g.dev.spos, attr0, attr1, corr + (size_t)k * src->capacity, trace + k,
                ybuf + 6 * k, 0.0f, slg, slc, d_dxyz, d_drgb, vpart, ticket, Tbar + (size_t)k * kTb,
                steps + (k ? k - 1 : K), k ? nullptr : d_dxi);
            GCA_CHECK_LAUNCH(ctx);
        }
    }
    GCA_CUDA(ctx, cudaMemcpyAsync(reinterpret_cast<char *>(ctx->h_pinned) + kPinnedBulk, readback, dT ? rb_bytes : rb_steps, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    if ((st = consume_device_error(ctx, "icp vjp"))) // synchronises
        return st;
    const char *host = reinterpret_cast<const char *>(ctx->h_pinned) + kPinnedBulk;
    const IcpTrace *h = reinterpret_cast<const IcpTrace *>(host);
    const VjpStep *h_steps = reinterpret_cast<const VjpStep *>(host + rb_steps);
    const double *h_dxi = reinterpret_cast<const double *>(host + rb_dxi);
    if (T_out)
        for (int k = 0; k < 16; ++k)
            T_out[k] = h[K].T[k];
    if (E_out)
        *E_out = h[K].S[27];
    if (dT)
        for (int m = 0; m < 6; ++m)
            dxi0[m] = h_dxi[m];
    for (int k = 0; k <= K; ++k)
        if (h[k].S[28] == 0.0)
            return fail(ctx, GCA3D_ERR_NO_CORRESPONDENCES, "icp vjp: an evaluation had no correspondences");
    bool singular = false;
    for (int k = 0; k < K; ++k)
        singular |= h[k].status != 0 || (dT && h_steps[k].singular);
    if (singular)
        return fail(ctx, GCA3D_ERR_SINGULAR, "icp vjp: a step's system was singular");
    return GCA3D_OK;
}
