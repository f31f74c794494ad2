// icp.cu -- colored ICP iteration (Park et al. 2017) for a batch of pairs.
//
// reference: color_icp::align (src/registration/color_icp.cu:151-234),
// compute_JTJ_JTr_and_r_gauss_newton_functor
// (src/registration/cuda_color_icp_build_least_square.cu:134-254) and
// solve_JTJ_JTr<true> (src/registration/eigen_solver.hpp:44-85).
//
// Three launches per Gauss-Newton iteration cover every pair (two with the fused
// finalize).  A block owns a chunk of one pair's source points.  k_icp_nn transforms
// them by the pair's current pose and finds the nearest target point inside max_corr
// (grid with a row table, ties to the smaller index); it keeps few registers so many warps
// hide the latency of the neighbour walk, and it skips the walk for points whose
// certificate from an earlier search of the scale still decides the answer
// (grid_query.cuh).  k_icp_accum builds the geometric and photometric residuals and
// their 6-vector Jacobians in FP32 and accumulates the 21 + 6 + 1 system terms plus
// the correspondence count and squared distances.  Accumulation is compensated FP32
// inside the block (two-sum per thread and per shuffle level) and FP64 across warps
// and blocks.  k_icp_finalize (a cluster of eight blocks per pair; k_icp_finalize_many,
// one block per pair, for several pairs of few points) -- or, fused, the last accumulate
// block of the pair to finish (atomic ticket, no waiting) -- sums the pair's block
// partials in FP64 in a fixed order, solves the 6x6 system by FP64 LDL^T, maps the step
// to SE(3) (Euler ZYX as the reference, or the exponential), composes the pose in
// FP64 and applies the reference's convergence test; a converged pair skips the
// remaining launches.  The source cloud is never rewritten: the pose is applied on
// the fly.
#include "grid_query.cuh"
#include "icp.cuh"
#include "pose_math.cuh"
#include "stages.cuh"

#include <algorithm>
#include <cooperative_groups.h>

namespace gca3d
{

// accumulator of kTerms values.  A thread sums its own few points (kIcpChunk /
// kIcpThreads = 4) in plain FP32; with Comp every combination above that -- the
// shuffle tree, the cross-warp sum -- is an error-free two-sum carrying an FP32
// error term, so the block sum is compensated where its error would grow.
template <bool Comp> struct Acc
{
    float s[kTerms];
    float e[kTerms];
    __device__ void zero()
    {
#pragma unroll
        for (int k = 0; k < kTerms; ++k)
            s[k] = 0.0f, e[k] = 0.0f;
    }
    __device__ __forceinline__ void add(int k, float x) { s[k] += x; }
    __device__ __forceinline__ void add_terms(const GNTerms &o, float d2)
    {
        int u = 0;
#pragma unroll
        for (int a = 0; a < 6; ++a)
#pragma unroll
            for (int b = a; b < 6; ++b)
                add(u++, o.Jg[a] * o.Jg[b] + o.Jc[a] * o.Jc[b]);
#pragma unroll
        for (int a = 0; a < 6; ++a)
            add(21 + a, o.Jg[a] * o.rg + o.Jc[a] * o.rc);
        add(27, o.rg * o.rg + o.rc * o.rc);
        add(28, 1.0f);
        add(29, d2);
    }
    // warp reduce-scatter by recursive halving: at the level of offset o a lane keeps
    // half of its current terms (the upper half when its lane bit o is set) and adds
    // the partner's copy of that half (xor o), sending the other half; 16 + 8 + 4 + 2 +
    // 1 exchanges per value instead of 5 per term.  Lane t < kTerms ends with term t
    // (value vs, error ve; terms 30 and 31 are zero padding).  The thread sums are
    // plain, so the first level has no error terms to exchange.
    __device__ __forceinline__ void warp_reduce_scatter(float &vs, float &ve) const
    {
        const unsigned full = 0xffffffffu;
        const int lane = threadIdx.x & 31;
        auto add2 = [](float a, float b, float ea, float eb, float &t, float &et) {
            if (Comp)
            {
                t = a + b;
                const float bp = t - a;
                et = ea + eb + ((a - (t - bp)) + (b - bp));
            }
            else
            {
                t = a + b;
                et = 0.0f;
            }
        };
        float s16[16], e16[16];
        {
            const bool up = lane & 16;
#pragma unroll
            for (int k = 0; k < 16; ++k)
            {
                const float lo = s[k], hi = k + 16 < kTerms ? s[k + 16] : 0.0f;
                const float keep = up ? hi : lo, send = up ? lo : hi;
                add2(keep, __shfl_xor_sync(full, send, 16), 0.0f, 0.0f, s16[k], e16[k]);
            }
        }
        float s8[8], e8[8];
        {
            const bool up = lane & 8;
#pragma unroll
            for (int k = 0; k < 8; ++k)
            {
                const float keep = up ? s16[k + 8] : s16[k], send = up ? s16[k] : s16[k + 8];
                const float ekeep = up ? e16[k + 8] : e16[k], esend = up ? e16[k] : e16[k + 8];
                add2(keep, __shfl_xor_sync(full, send, 8), ekeep, Comp ? __shfl_xor_sync(full, esend, 8) : 0.0f,
                     s8[k], e8[k]);
            }
        }
        float s4[4], e4[4];
        {
            const bool up = lane & 4;
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                const float keep = up ? s8[k + 4] : s8[k], send = up ? s8[k] : s8[k + 4];
                const float ekeep = up ? e8[k + 4] : e8[k], esend = up ? e8[k] : e8[k + 4];
                add2(keep, __shfl_xor_sync(full, send, 4), ekeep, Comp ? __shfl_xor_sync(full, esend, 4) : 0.0f,
                     s4[k], e4[k]);
            }
        }
        float s2[2], e2[2];
        {
            const bool up = lane & 2;
#pragma unroll
            for (int k = 0; k < 2; ++k)
            {
                const float keep = up ? s4[k + 2] : s4[k], send = up ? s4[k] : s4[k + 2];
                const float ekeep = up ? e4[k + 2] : e4[k], esend = up ? e4[k] : e4[k + 2];
                add2(keep, __shfl_xor_sync(full, send, 2), ekeep, Comp ? __shfl_xor_sync(full, esend, 2) : 0.0f,
                     s2[k], e2[k]);
            }
        }
        {
            const bool up = lane & 1;
            const float keep = up ? s2[1] : s2[0], send = up ? s2[0] : s2[1];
            const float ekeep = up ? e2[1] : e2[0], esend = up ? e2[0] : e2[1];
            add2(keep, __shfl_xor_sync(full, send, 1), ekeep, Comp ? __shfl_xor_sync(full, esend, 1) : 0.0f, vs,
                 ve);
        }
    }
    __device__ __forceinline__ double value(int k) const
    {
        return Comp ? (double)s[k] + (double)e[k] : (double)s[k];
    }
};

// sum of the block's kTerms values into part[kTerms].  Compensated: the per-warp
// (value, error) pairs are combined across warps by two-sum in FP32 and each of the
// 30 results is converted to FP64 once per block (FP64 issue is ~1/64 of FP32 on
// this part, so per-warp conversions would cost more than the sums).  Plain: FP32.
template <bool Comp>
__device__ __forceinline__ void block_reduce_store(Acc<Comp> &acc, double *part)
{
    __shared__ float s_s[kIcpThreads / 32][kTerms];
    __shared__ float s_e[kIcpThreads / 32][kTerms];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float vs, ve;
    acc.warp_reduce_scatter(vs, ve); // lane k holds term k
    if (lane < kTerms)
    {
        s_s[warp][lane] = vs;
        s_e[warp][lane] = ve;
    }
    __syncthreads();
    if (threadIdx.x < kTerms)
    {
        const int k = threadIdx.x;
        float v = s_s[0][k], e = Comp ? s_e[0][k] : 0.0f;
        for (int w = 1; w < kIcpThreads / 32; ++w)
        {
            const float x = s_s[w][k];
            if (Comp)
            {
                const float t = v + x;
                const float bp = t - v;
                e += s_e[w][k] + ((v - (t - bp)) + (x - bp));
                v = t;
            }
            else
                v += x;
        }
        part[k] = Comp ? (double)v + (double)e : (double)v;
    }
}

// exclusive prefix over the block's Threads threads of two per-thread counts: each
// thread gets its own prefixes back in a and b, and every thread the two totals
template <int Threads> __device__ __forceinline__ void block_prefix2(int &a, int &b, int &ta, int &tb)
{
    __shared__ int s_a[Threads], s_b[Threads];
    __shared__ int s_ta, s_tb;
    s_a[threadIdx.x] = a;
    s_b[threadIdx.x] = b;
    __syncthreads();
    if (threadIdx.x < 32)
    {
        // a few per lane, then across the warp
        constexpr int kPer = Threads / 32;
        const int l = threadIdx.x;
        int va[kPer], vb[kPer], sa = 0, sb = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            va[k] = s_a[l * kPer + k];
            vb[k] = s_b[l * kPer + k];
            sa += va[k];
            sb += vb[k];
        }
        int ia = sa, ib = sb;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const int ya = __shfl_up_sync(0xffffffffu, ia, o), yb = __shfl_up_sync(0xffffffffu, ib, o);
            if (l >= o)
                ia += ya, ib += yb;
        }
        int ra = ia - sa, rb = ib - sb;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            s_a[l * kPer + k] = ra;
            s_b[l * kPer + k] = rb;
            ra += va[k];
            rb += vb[k];
        }
        if (l == 31)
        {
            s_ta = ra;
            s_tb = rb;
        }
    }
    __syncthreads();
    a = s_a[threadIdx.x];
    b = s_b[threadIdx.x];
    ta = s_ta;
    tb = s_tb;
}

// per-scale setup: block map, per-pair counts, reset of the per-scale flags; the
// pairs split over the block's threads, the maps by a block prefix
__global__ void __launch_bounds__(kIcpThreads) k_icp_setup(PairState *st, int P, const int32_t *src_off,
                                                           const int32_t *tgt_off, int *bmap, int *bmap_nn, int scale,
                                                           int nn_chunk)
{
    __shared__ int s_nact;
    if (threadIdx.x == 0)
        s_nact = 0;
    __syncthreads();
    const int chunk = kIcpChunk;
    const int per = (P + kIcpThreads - 1) / kIcpThreads;
    const int p0 = min(P, (int)threadIdx.x * per), p1 = min(P, p0 + per);
    int b = 0, bn = 0, na = 0;
    for (int p = p0; p < p1; ++p)
    {
        PairState &S = st[p];
        const int ns = src_off[p + 1] - src_off[p];
        const int nt = tgt_off[p + 1] - tgt_off[p];
        const int nb = (ns > 0 && nt > 0) ? (ns + chunk - 1) / chunk : 0;
        const int nbn = (ns > 0 && nt > 0) ? (ns + nn_chunk - 1) / nn_chunk : 0;
        b += nb;
        bn += nbn;
        na += nb > 0;
        S.nblocks = nb;
        S.nblocks_nn = nbn;
        S.nsrc = ns;
        S.ntgt = nt;
        S.ticket = 0;
        S.active = nb > 0 ? 1 : 0;
        S.converged = 0;
        if (scale == 0)
        {
            S.iters = 0;
            S.status = 0;
            for (int k = 0; k < GCA3D_MAX_SCALES; ++k)
                S.scale_iters[k] = S.scale_nsrc[k] = S.scale_ntgt[k] = 0;
        }
        S.scale = scale;
        S.nn_warm = 0;
        S.scale_nsrc[scale] = ns;
        S.scale_ntgt[scale] = nt;
        if (nb == 0)
        {
            S.status = GCA3D_ERR_NO_CORRESPONDENCES;
            S.rmse_ref = S.fitness = S.inlier_rmse = 0.0;
        }
    }
    if (na)
        atomicAdd(&s_nact, na);
    int tb, tbn;
    block_prefix2<kIcpThreads>(b, bn, tb, tbn);
    for (int p = p0; p < p1; ++p)
    {
        bmap[p] = b;
        bmap_nn[p] = bn;
        b += st[p].nblocks;
        bn += st[p].nblocks_nn;
    }
    if (threadIdx.x == 0)
    {
        bmap[P] = tb;
        bmap[P + 1] = s_nact; // pairs the fused accumulate finalizes this iteration
        bmap_nn[P] = tbn;
        bmap_nn[P + 1] = 0; // the correspondence kernel's work queue
    }
}

__global__ void k_state_init(PairState *st, int P, const double *T_init)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= P)
        return;
    for (int k = 0; k < 16; ++k)
        st[p].T[k] = T_init ? T_init[16 * p + k] : (k % 5 == 0 ? 1.0 : 0.0);
    for (int k = 0; k < 12; ++k)
        st[p].Tf[k] = (float)st[p].T[k];
    st[p].iters = 0;
    st[p].status = 0;
    st[p].rmse_ref = st[p].fitness = st[p].inlier_rmse = 0.0;
}

// work item w -> (pair, chunk) of the pair's source points; the pair's pose as FP32 in shared
// memory.  Warp 0 does it, all lanes at once (its loads are the item's latency: one thread
// searching the map and converting the pose held a 256-point item for about 2 us); the block
// meets before it, so that the previous item's readers are done, and after it.
struct BlockPair
{
    int pair, start, end;
};

// the last pair whose first item is <= w (pairs without items share theirs with the next;
// bmap[0] is 0): 64 entries a round, so one round up to 64 pairs and two at 4096.  Its loads
// are most of an item's latency: with 32 entries a round in order, up to 128 rounds, 4096 pairs
// of 1000 points took 30,600 us (10 steps), now 28,500, and 64 pairs 884, 886.
__device__ __forceinline__ int item_pair(int w, const int *bmap, int P)
{
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int lo = 0, n = P;
    for (;;)
    {
        const int step = (n + 63) >> 6;
        const int a = lane * step, b = a + 32 * step;
        const bool la = a < n && bmap[lo + a] <= w, lb = b < n && bmap[lo + b] <= w;
        const int c = __popc(__ballot_sync(full, la)) + __popc(__ballot_sync(full, lb));
        lo += (c - 1) * step;
        if (step == 1)
            return lo;
        n = min(step, n - (c - 1) * step);
    }
}

__device__ __forceinline__ void item_setup(int w, int items, const int32_t *src_off, const PairState *st,
                                           const int *bmap, int P, int chunk, float *s_T, BlockPair *s_item)
{
    const int lane = threadIdx.x & 31;
    int p = -1;
    if (w < items)
    {
        p = item_pair(w, bmap, P);
        if (!st[p].active)
            p = -1;
    }
    if (p >= 0 && lane < 12)
        s_T[lane] = st[p].Tf[lane];
    if (lane == 0)
    {
        BlockPair b{p, 0, 0};
        if (p >= 0)
        {
            b.start = src_off[p] + (w - bmap[p]) * chunk;
            b.end = min(b.start + chunk, src_off[p + 1]);
        }
        *s_item = b;
    }
}

// step 1 of an iteration: the correspondence of every active source point
// (grid position and squared distance, -1 when none within max_corr).
// Phase 1, one thread per point: from the second iteration of a scale on, a point
// whose certificate from its last search still holds (it has not moved far enough
// for another target point to overtake its nearest one, grid_query.cuh) takes its
// correspondence without a search.  Phase 2, four lanes per point over the block's
// list of the others: the search, shrunk to the cells that overlap the ball
// through the last nearest point when that one is within max_corr (the ball holds
// the nearest point and all its ties); it renews the point's certificate.
// Cold: the first search of a scale, without certificates or last nearest points, in a
// kernel of its own, so that the second row loop of its search costs the warm ones no
// registers.
template <bool Cold>
__global__ void __launch_bounds__(kIcpThreads, 5) k_icp_nn(const float4 *__restrict__ src_pos, const int32_t *src_off,
                                                        GridDev g, const PairState *st, const int *bmap, int P,
                                                        float max_corr, int2 *corr, NNCerts cert, int32_t *nn_out,
                                                        int nn_chunk, int *queue, const int *stop_iter, int stop_at)
{
    // a search queued behind the iteration that spent the scale's budget has nothing to do
    if (stop_iter && *stop_iter >= stop_at)
        return;
    __shared__ BlockPair s_item;
    __shared__ int s_w;
    __shared__ float s_T[12];
    __shared__ int s_list[kNNChunkMax];
    __shared__ int4 s_box[kNNChunkMax]; // x0, y0, zlo, nx | ny << 8 | nz << 16 of the search box
    __shared__ float4 s_p[kNNChunkMax]; // the transformed point
    __shared__ int s_cnt;
    const KeyLayout L = *g.layout;
    const float rr = __fmul_rn(max_corr, max_corr);
    const int items = bmap[P];
    const int lane = threadIdx.x & 31;
    // a block's first work item is its own index, the later ones come from the
    // iteration's queue (drawn while the item before is searched): blocks that draw quick
    // items (mostly certified points) take more of them
    int next = (int)blockIdx.x;
    for (;;)
    {
    __syncthreads();
    if (threadIdx.x < 32)
    {
        const int w = __shfl_sync(0xffffffffu, next, 0);
        item_setup(w, items, src_off, st, bmap, P, nn_chunk, s_T, &s_item);
        if (lane == 0)
        {
            s_w = w;
            s_cnt = 0;
        }
    }
    __syncthreads();
    if (s_w >= items)
        break;
    if (threadIdx.x == 0)
        next = (int)gridDim.x + atomicAdd(queue, 1);
    const BlockPair b = s_item;
    if (b.pair < 0)
        continue;
    const float3 o = g.gmin[b.pair];
    const int tbase = g.seg_off[b.pair];
    const bool warm = !Cold && st[b.pair].nn_warm;
    for (int base = b.start; base < b.end; base += kIcpThreads)
    {
        const int i = base + (int)threadIdx.x;
        bool need = false;
        float3 p;
        CellBox B;
        if (i < b.end)
        {
            p = apply_pose(s_T, src_pos[i]);
            need = nn_full_box(g, L, o, p, B);
            if (!need)
            {
                // outside the grid's range: no candidates
                corr[i] = make_int2(-1, __float_as_int(rr));
                if (nn_out)
                    nn_out[i] = -1;
                cert.pos[i] = make_float4(p.x, p.y, p.z, 0.0f);
                cert.t[i] = -1;
            }
        }
        if (need && warm)
        {
            const int t1 = cert.t[i];
            int t;
            float d2;
            if (nn_certified(g, o, p, B, cert.pos[i], t1, rr, t, d2))
            {
                need = false;
                corr[i] = make_int2(t, __float_as_int(d2));
                if (nn_out)
                    nn_out[i] = t >= 0 ? __ldg(&g.sidx[t]) - tbase : -1;
            }
            else if (t1 >= 0)
            {
                // the ball through the last nearest point holds the nearest point and its ties
                const float4 q = __ldg(&g.spos[t1]);
                const float u2 = dist2_ref(q.x, q.y, q.z, p.x, p.y, p.z);
                if (u2 < rr)
                    nn_shrink_box(g, o, p, sqrtf(u2), B);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, need);
        int at = 0;
        if (lane == 0 && m)
            at = atomicAdd(&s_cnt, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (need)
        {
            const int k = at + __popc(m & ((1u << lane) - 1u));
            s_list[k] = i;
            s_box[k] = make_int4(B.x0, B.y0, B.zlo, B.nx | (B.ny << 8) | ((B.zhi - B.zlo + 1) << 16));
            s_p[k] = make_float4(p.x, p.y, p.z, 0.0f);
        }
    }
    __syncthreads();
    const int n = s_cnt;
    // four lanes per listed point (uniform trip count for the whole block)
    for (int base = 0; base < n; base += kIcpThreads / kSub)
    {
        const int k = base + (int)(threadIdx.x / kSub);
        const bool valid = k < n;
        const int kk = valid ? k : 0;
        NNBest2 best;
        CellBox searched;
        {
            const int4 bx = s_box[kk];
            const float4 p4 = s_p[kk];
            CellBox B{bx.x, bx.w & 0xff, bx.y, (bx.w >> 8) & 0xff, bx.z, bx.z + (bx.w >> 16) - 1};
            best = nn_search_box2<Cold>(g, L, b.pair, o, B, make_float3(p4.x, p4.y, p4.z), valid);
            if (Cold)
                searched = B;
        }
        if (valid && (threadIdx.x & (kSub - 1)) == 0)
        {
            // the point, its box and the grid origin read again (volatile: not kept
            // live in registers through the search)
            const volatile int *vl = s_list;
            const volatile int *vb = reinterpret_cast<const volatile int *>(&s_box[kk]);
            const volatile float *vp = reinterpret_cast<const volatile float *>(&s_p[kk]);
            const int i = vl[kk];
            const int bw = vb[3];
            const CellBox B = Cold ? searched
                                   : CellBox{vb[0], bw & 0xff, vb[1], (bw >> 8) & 0xff, vb[2], vb[2] + (bw >> 16) - 1};
            const float3 p = make_float3(vp[0], vp[1], vp[2]);
            const float3 og = g.gmin[b.pair];
            const bool hit = best.t >= 0 && best.d2 < rr;
            corr[i] = make_int2(hit ? best.t : -1, __float_as_int(hit ? best.d2 : rr));
            if (nn_out)
                nn_out[i] = hit ? __ldg(&g.sidx[best.t]) - tbase : -1;
            cert.pos[i] = make_float4(p.x, p.y, p.z, cert_bound(g, og, p, B, best.s2));
            cert.t[i] = best.t;
        }
    }
    }
}

// the pair's block partials in FP64, in a fixed order: group g of 8 takes blocks g, g + 8, ...
// as four running sums, (0 + 1) + (2 + 3), and the groups are added in order.  (Plain: FP32,
// one sum per group.)  The element of group g's running sum r at step q is block
// g + 8 (4 q + r); a remainder of fewer than four blocks goes to running sum 0.
constexpr int kSumGroups = 8;

// running sum `chain` of group grp (lane: term); chain 0 takes the remainder too.  Eight
// loads are in flight at once; an FP64 addition takes 64 cycles of the warp.
__device__ __forceinline__ double partial_chain(const double *src, int nb, int grp, int chain)
{
    constexpr int kW = kSumGroups, kAhead = 8;
    const int x = nb - grp - 3 * kW;
    const int full = x > 0 ? (x + 4 * kW - 1) / (4 * kW) : 0; // whole steps of four
    const int tail = grp + 4 * kW * full;                     // the remainder's first block
    const int rest = chain == 0 && nb > tail ? (nb - tail + kW - 1) / kW : 0;
    double v = 0.0;
    for (int q0 = 0; q0 < full + rest; q0 += kAhead)
    {
        double p[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
        {
            const int q = q0 + u;
            const int j = q < full ? grp + kW * (4 * q + chain) : tail + kW * (q - full);
            p[u] = q < full + rest ? __ldcg(src + (size_t)j * kTermsPad) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
            if (q0 + u < full + rest)
                v += p[u];
    }
    return v;
}

// one pair's sums by one whole block into s_S (the fused accumulate).  The partials are
// read from L2: other blocks of the same launch wrote them.
template <bool Comp>
__device__ __forceinline__ void finalize_sums(const PairState &Ps, const double *src, double *s_S)
{
    __shared__ double s_red[kSumGroups][kTermsPad];
    static_assert(kSumGroups == kIcpThreads / 32, "one warp per group");
    const int nb = Ps.nblocks;
    const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
    if (lane < kTerms)
    {
        if (Comp)
        {
            // the four chains side by side (each in its own order)
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            constexpr int kW = kSumGroups;
            int j = grp;
            for (; j + 3 * kW < nb; j += 4 * kW)
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    v[r] += __ldcg(src + (size_t)(j + r * kW) * kTermsPad + lane);
            for (; j < nb; j += kW)
                v[0] += __ldcg(src + (size_t)j * kTermsPad + lane);
            s_red[grp][lane] = (v[0] + v[1]) + (v[2] + v[3]);
        }
        else
        {
            float vf = 0.0f;
            for (int j = grp; j < nb; j += kSumGroups)
                vf += (float)__ldcg(src + (size_t)j * kTermsPad + lane);
            s_red[grp][lane] = (double)vf;
        }
    }
    __syncthreads();
    if (threadIdx.x < kTerms)
    {
        const int k = threadIdx.x;
        double v = 0.0;
        float vf = 0.0f;
        for (int w = 0; w < kSumGroups; ++w)
        {
            if (Comp)
                v += s_red[w][k];
            else
                vf += (float)s_red[w][k];
        }
        s_S[k] = Comp ? v : (double)vf;
    }
    __syncthreads();
}

// what a pair's finalize reads of its state, read before the sums are there
struct FinalizeIn
{
    double T; // entry `lane` of the pose (lanes 0..15)
    int iters, scale, scale_iter, status, nsrc;
};
__device__ __forceinline__ FinalizeIn finalize_in(const PairState &Ps)
{
    const int lane = threadIdx.x & 31;
    FinalizeIn in;
    in.T = lane < 16 ? Ps.T[lane] : 0.0;
    in.iters = Ps.iters;
    in.scale = Ps.scale;
    in.status = Ps.status;
    in.nsrc = Ps.nsrc;
    in.scale_iter = Ps.scale_iters[in.scale];
    return in;
}

// one pair's finalize from its sums: the 6x6 solve, the step map, the FP64 pose update and
// the reference's convergence test (color_icp.cu:216-228) by warp 0, the statistics by
// warp 1; other warps return at once
__device__ __forceinline__ void finalize_solve(PairState &Ps, int P, int pair, const double *s_S, const IcpScale &prm,
                                               const FinalizeIn &in)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0)
    {
        // solve, step map and composition over the lanes of warp 0
        double x[6];
        const int singular = solve6_warp(s_S, x);
        const double Ti = pose_from_x_warp(x, prm.update_map); // lanes 0..15: Ti[lane]
        const int r = (lane >> 2) & 3, c = lane & 3;
        const double Told = in.T;
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            v += __shfl_sync(0xffffffffu, Ti, 4 * r + k) * __shfl_sync(0xffffffffu, Told, 4 * k + c);
        // lane 0: the step's cosine, 0.5 (trace - 1); lane 1: its squared translation, negated
        // (compared as >= with cos_min and -trans_eps)
        const double d0 = __shfl_sync(0xffffffffu, Ti, lane == 1 ? 3 : 0),
                     d1 = __shfl_sync(0xffffffffu, Ti, lane == 1 ? 7 : 5),
                     d2 = __shfl_sync(0xffffffffu, Ti, lane == 1 ? 11 : 10);
        const double w0 = lane == 1 ? d0 : 1.0, w1 = lane == 1 ? d1 : 1.0, w2 = lane == 1 ? d2 : 1.0;
        const double dsum = fma(d2, w2, fma(d1, w1, d0 * w0));
        const double measure = fma(dsum, lane == 1 ? -1.0 : 0.5, lane == 1 ? 0.0 : -0.5);
        const unsigned small = __ballot_sync(0xffffffffu, measure >= (lane == 1 ? -prm.trans_eps : prm.cos_min));
        const int iters = in.iters;
        if (prm.trace && iters < prm.trace_cap)
        {
            IcpTrace &tr = prm.trace[(size_t)iters * P + pair];
            if (lane < 16)
                tr.T[lane] = Told;
            if (lane < kTerms)
                tr.S[lane] = s_S[lane];
            if (lane == 0)
            {
#pragma unroll
                for (int q = 0; q < 6; ++q)
                    tr.x[q] = x[q];
                tr.status = singular;
            }
        }
        __syncwarp();
        if (lane < 16)
            Ps.T[lane] = v;
        if (lane < 12)
            Ps.Tf[lane] = (float)v;
        if (lane == 0)
        {
            if (__double_as_longlong(s_S[28]) == 0ll) // a count: never -0
                Ps.status = GCA3D_ERR_NO_CORRESPONDENCES;
            else if (singular && in.status == 0)
                Ps.status = GCA3D_ERR_SINGULAR;
            Ps.iters = iters + 1;
            Ps.scale_iters[in.scale] = in.scale_iter + 1;
            Ps.nn_warm = 1;
            if ((small & 3u) == 3u)
            {
                Ps.converged = 1;
                Ps.active = 0;
            }
        }
    }
    else if (warp == 1)
    {
        // the statistics, on their own warp (one division per lane)
        const double ns = (double)in.nsrc;
        const int m = lane % 3;
        const double num = m == 0 ? s_S[27] : (m == 1 ? s_S[28] : s_S[29]);
        const double den = m == 2 ? s_S[28] : ns;
        double q = num / den;
        if (m == 2)
            q = s_S[28] > 0.0 ? sqrt(q) : 0.0;
        if (lane == 0)
            Ps.rmse_ref = q;
        else if (lane == 1)
            Ps.fitness = q;
        else if (lane == 2)
            Ps.inlier_rmse = q;
    }
}

// the work maps over the pairs still active (the next iteration's NN and accumulate
// launches get no items for converged pairs), their count and, in a captured
// schedule, the loop condition.  Run by one whole block once every pair of the
// iteration is finalized.
template <int Threads>
__device__ __forceinline__ void rebuild_maps_body(PairState *st, int P, int *bmap, int *bmap_nn, const IcpLoop &loop)
{
    __shared__ int s_nact;
    if (threadIdx.x == 0)
        s_nact = 0;
    __syncthreads();
    const int per = (P + Threads - 1) / Threads;
    const int p0 = min(P, (int)threadIdx.x * per), p1 = min(P, p0 + per);
    int a = 0, an = 0, na = 0;
    for (int q = p0; q < p1; ++q)
        if (__ldcg(&st[q].active))
        {
            a += st[q].nblocks;
            an += st[q].nblocks_nn;
            ++na;
        }
    if (na)
        atomicAdd(&s_nact, na);
    int ta, tn;
    block_prefix2<Threads>(a, an, ta, tn);
    if (threadIdx.x == 0)
    {
        bmap[P] = ta;
        bmap[P + 1] = s_nact;
        bmap_nn[P] = tn;
        bmap_nn[P + 1] = 0;
        *loop.ticket = 0u;
        if (loop.iter)
        {
            const int it = ++(*loop.iter);
            cudaGraphSetConditional(loop.handle, (tn > 0 && it < loop.max_iter) ? 1u : 0u);
        }
    }
    for (int q = p0; q < p1; ++q)
    {
        bmap[q] = a;
        bmap_nn[q] = an;
        if (__ldcg(&st[q].active))
        {
            a += st[q].nblocks;
            an += st[q].nblocks_nn;
        }
    }
}

// rebuild_maps_body for a single pair, by one thread; iter: the loop count so far
__device__ __forceinline__ void rebuild_single(int act, int nblocks, int nblocks_nn, int iter, int *bmap, int *bmap_nn,
                                               const IcpLoop &loop)
{
    const int tn = act ? nblocks_nn : 0;
    bmap[0] = bmap_nn[0] = 0;
    bmap[1] = act ? nblocks : 0;
    bmap[2] = act ? 1 : 0;
    bmap_nn[1] = tn;
    bmap_nn[2] = 0;
    *loop.ticket = 0u;
    if (loop.iter)
    {
        *loop.iter = iter + 1;
        cudaGraphSetConditional(loop.handle, (tn > 0 && iter + 1 < loop.max_iter) ? 1u : 0u);
    }
}

// the same two steps as calls, for the fused accumulate: compiled apart from the
// accumulation loop, whose registers they would otherwise crowd (the separate finalize
// kernel has its own sums)
template <bool Comp>
__device__ __noinline__ void finalize_pair(PairState *st, int P, int pair, const int *bmap, const double *partials,
                                           IcpScale prm)
{
    __shared__ double s_S[kTermsPad];
    finalize_sums<Comp>(st[pair], partials + (size_t)bmap[pair] * kTermsPad, s_S);
    finalize_solve(st[pair], P, pair, s_S, prm, finalize_in(st[pair]));
}

__device__ __noinline__ void rebuild_maps(PairState *st, int P, int *bmap, int *bmap_nn, IcpLoop loop)
{
    rebuild_maps_body<kIcpThreads>(st, P, bmap, bmap_nn, loop);
}

// step 2: residuals, Jacobians, block sums (one partial per block); three resident
// blocks per SM (80 registers: the 30 sums and two points' gathers in flight).
// Fused: after storing its partial a block takes the pair's ticket, and the pair's
// last block runs the pair's finalize; the last pair to be finalized rebuilds the
// work maps.  A block that starts after that rebuild finds no item: within a scale
// the active set only shrinks, so the next item count is at most this one, and every
// block below this count has work left until the rebuild.
template <bool Comp, bool Fused>
__global__ void __launch_bounds__(kIcpThreads, 3) k_icp_accum(const float4 *__restrict__ src_pos, const int32_t *src_off,
                                                           const float4 *__restrict__ tpos,
                                                           const float4 *__restrict__ attr0,
                                                           const float4 *__restrict__ attr1,
                                                           const int2 *__restrict__ corr, PairState *st,
                                                           int *bmap, int *bmap_nn, int P, double *partials,
                                                           float slg, float slc, const int32_t *d_nt, int *err,
                                                           IcpScale prm, IcpLoop loop)
{
    __shared__ BlockPair s_item;
    __shared__ float s_T[12];
    __shared__ int s_fin;
    const int items = bmap[P];
    const int nact = Fused ? bmap[P + 1] : 0;
    if (Fused && items == 0)
    {
        // no active pair: nothing to finalize, but the maps and the loop condition are set
        if (blockIdx.x == 0)
            rebuild_maps(st, P, bmap, bmap_nn, loop);
        return;
    }
    for (int w = blockIdx.x; w < items; w += gridDim.x)
    {
    __syncthreads();
    if (threadIdx.x < 32)
        item_setup(w, items, src_off, st, bmap, P, kIcpChunk, s_T, &s_item);
    __syncthreads();
    const BlockPair b = s_item;
    if (b.pair < 0)
        continue;
    Acc<Comp> acc;
    acc.zero();
    // a thread's points two at a time, all their loads issued before either is used
    // (the sums still run over the points in ascending order)
    constexpr int kPer = kIcpChunk / kIcpThreads;
#pragma unroll
    for (int j0 = 0; j0 < kPer; j0 += 2)
    {
        int2 c[2];
        float4 s4[2], q[2], a0[2], a1[2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
        {
            const int i = b.start + (int)threadIdx.x + kIcpThreads * (j0 + j);
            c[j] = i < b.end ? corr[i] : make_int2(-1, 0);
            if (c[j].x >= 0 && !GCA_INDEX_OK(c[j].x, *d_nt, err))
                c[j].x = -1;
            if (c[j].x >= 0)
            {
                s4[j] = src_pos[i];
                q[j] = __ldg(&tpos[c[j].x]);
                a0[j] = __ldg(&attr0[c[j].x]);
                a1[j] = __ldg(&attr1[c[j].x]);
            }
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
        {
            if (c[j].x < 0)
                continue;
            const float3 p = apply_pose(s_T, s4[j]);
            GNTerms terms;
            gn_terms(p, s4[j].w, make_float3(q[j].x, q[j].y, q[j].z), a0[j].w, make_float3(a0[j].x, a0[j].y, a0[j].z),
                     make_float3(a1[j].x, a1[j].y, a1[j].z), slg, slc, terms);
            acc.add_terms(terms, __int_as_float(c[j].y));
        }
    }
    block_reduce_store<Comp>(acc, partials + (size_t)w * kTermsPad);
    if (Fused)
    {
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0)
            s_fin = atomicAdd(&st[b.pair].ticket, 1u) == (unsigned)(st[b.pair].nblocks - 1);
        __syncthreads();
        if (s_fin)
        {
            __threadfence();
            finalize_pair<Comp>(st, P, b.pair, bmap, partials, prm);
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0)
            {
                st[b.pair].ticket = 0u;
                s_fin = P == 1 || atomicAdd(loop.ticket, 1u) == (unsigned)(nact - 1);
            }
            __syncthreads();
            if (s_fin)
            {
                __threadfence();
                rebuild_maps(st, P, bmap, bmap_nn, loop);
            }
        }
    }
    }
}

// the finalize as a launch of its own: a cluster of eight blocks per pair, block g summing
// group g with a warp per running sum (an SM adds one FP64 warp instruction in 19 cycles, so
// 200 partials took one block 3 us; eight SMs take 1), then block 0 solves.  The last pair's
// block rebuilds the work maps; a single pair's does so directly.  What bounds it is the chain
// of FP64 operations at 64 cycles each.  Cycles of a frame pair's finalize, one block before
// and a cluster now: sums 6900, 5430 (with the exchange); solve 7560, 7540; pose 2420 to
// 4090, 2210 to 3430; composition 1820, 1300; maps 3000, 200 to 840.  A launch went from 15.7
// to 10.5 us.
template <bool Comp>
__global__ void __launch_bounds__(128) k_icp_finalize(PairState *st, int P, int *bmap, int *bmap_nn,
                                                      const double *partials, IcpScale prm, IcpLoop loop)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double s_part[4][kTermsPad];
    __shared__ double s_group[kTermsPad]; // this block's group
    __shared__ double s_S[kTermsPad];
    const int grp = (int)cluster.block_rank(), pair = blockIdx.x / kSumGroups;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    PairState &Ps = st[pair];
    // everything read of the state and the maps, at once (the loads of one another's results
    // were half of the chain); the cluster's blocks see the same state: block 0 writes it
    // after the last barrier
    const bool active = Ps.active;
    const int nb = Ps.nblocks, nb_nn = Ps.nblocks_nn, first = bmap[pair];
    const int iter = loop.iter && P == 1 ? *loop.iter : 0;
    FinalizeIn in{};
    if (grp == 0)
        in = finalize_in(Ps);
    if (active)
    {
        const double *src = partials + (size_t)first * kTermsPad + lane;
        if (Comp)
        {
            if (lane < kTerms)
                s_part[warp][lane] = partial_chain(src, nb, grp, warp);
            __syncthreads();
            if (threadIdx.x < kTerms)
                s_group[threadIdx.x] = (s_part[0][threadIdx.x] + s_part[1][threadIdx.x]) +
                                       (s_part[2][threadIdx.x] + s_part[3][threadIdx.x]);
        }
        else
        {
            // FP32, one sum per group: the four warps read and round a tile of its partials,
            // eight loads in flight each, and one adds them up in order (one warp reading them
            // one after the other: 35 us a launch at 118 partials and at 293; so 11.3 and 12.2,
            // against 14.3 and 18.5 for one block)
            constexpr int kTile = 32;
            __shared__ float s_tile[kTile][kTermsPad];
            const int mine = nb > grp ? (nb - grp + kSumGroups - 1) / kSumGroups : 0;
            float vf = 0.0f;
            for (int q0 = 0; q0 < mine; q0 += kTile)
            {
                double p[kTile / 4];
#pragma unroll
                for (int u = 0; u < kTile / 4; ++u)
                {
                    const int q = q0 + 4 * u + warp;
                    p[u] = q < mine && lane < kTerms ? __ldcg(src + (size_t)(grp + kSumGroups * q) * kTermsPad) : 0.0;
                }
                __syncthreads(); // the tile before is added up
#pragma unroll
                for (int u = 0; u < kTile / 4; ++u)
                    s_tile[4 * u + warp][lane] = (float)p[u];
                __syncthreads();
                if (threadIdx.x < kTerms)
                    for (int u = 0; u < min(kTile, mine - q0); ++u)
                        vf += s_tile[u][threadIdx.x];
            }
            if (threadIdx.x < kTerms)
                s_group[threadIdx.x] = (double)vf;
        }
    }
    cluster.sync();
    if (grp == 0 && active && threadIdx.x < kTerms)
    {
        double part[kSumGroups];
#pragma unroll
        for (int w = 0; w < kSumGroups; ++w)
            part[w] = cluster.map_shared_rank(s_group, w)[threadIdx.x];
        double v = 0.0;
        float vf = 0.0f;
#pragma unroll
        for (int w = 0; w < kSumGroups; ++w)
        {
            if (Comp)
                v += part[w];
            else
                vf += (float)part[w];
        }
        s_S[threadIdx.x] = Comp ? v : (double)vf;
    }
    cluster.sync(); // the groups are read: the other blocks may leave
    if (grp != 0)
        return;
    if (active)
        finalize_solve(Ps, P, pair, s_S, prm, in);
    if (P == 1)
    {
        if (threadIdx.x == 0) // thread 0 wrote the state's flag itself
            rebuild_single(Ps.active, nb, nb_nn, iter, bmap, bmap_nn, loop);
        return;
    }
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(loop.ticket, 1u) == (unsigned)(P - 1);
    __syncthreads();
    if (!s_last)
        return;
    rebuild_maps_body<128>(st, P, bmap, bmap_nn, loop);
}

// The same by one block per pair.  A cluster per pair pays where the sums are long: for a
// single pair (whose maps it also rebuilds directly), and from about 48 partials a pair (48k
// points; max_blocks, by capacity).  Below, its eight blocks and two barriers cost more than
// the sums they share.  us for 30 steps, a cluster and one block: 1 pair of 1k points 874,
// 907, of 64k 993, 1064; 2 pairs of 4k 985, 963, of 16k 1050, 1037, of 48k 1144, 1158, of 128k
// 1700, 1750; 16 pairs of 4k 1134, 1086, of 32k 2548, 2530, of 64k 4397, 4412; 10 steps of
// 4096 pairs of 1k 28,710, 27,630.
constexpr int kClusterPartials = 48;
template <bool Comp>
__global__ void __launch_bounds__(kIcpThreads) k_icp_finalize_many(PairState *st, int P, int *bmap, int *bmap_nn,
                                                                   const double *partials, IcpScale prm, IcpLoop loop)
{
    __shared__ double s_S[kTermsPad];
    __shared__ int s_last;
    const int pair = blockIdx.x;
    PairState &Ps = st[pair];
    if (Ps.active)
    {
        const FinalizeIn in = finalize_in(Ps);
        finalize_sums<Comp>(Ps, partials + (size_t)bmap[pair] * kTermsPad, s_S);
        finalize_solve(Ps, P, pair, s_S, prm, in);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(loop.ticket, 1u) == (unsigned)(P - 1);
    __syncthreads();
    if (!s_last)
        return;
    rebuild_maps_body<kIcpThreads>(st, P, bmap, bmap_nn, loop);
}

IcpShape icp_shape(const gca3d_tuning &t, int P, int64_t src_cap)
{
    IcpShape s;
    s.nn_chunk = P == 1 || src_cap <= kNNSmallPoints ? kNNChunkSmall : kNNChunk;
    if (t.nn_item_points == 64 || t.nn_item_points == 128 || t.nn_item_points == 256 || t.nn_item_points == 512)
        s.nn_chunk = t.nn_item_points;
    if (t.nn_blocks_per_sm > 0)
        s.nn_bps = std::min(t.nn_blocks_per_sm, 64);
    if (t.accum_blocks_per_sm > 0)
        s.acc_bps = std::min(t.accum_blocks_per_sm, 64);
    s.fused = t.fused_finalize != 0;
    return s;
}

int icp_setup(gca3d_context *ctx, PairState *st, int P, const int32_t *src_off, const int32_t *tgt_off, int *bmap,
              int *bmap_nn, int scale, int nn_chunk)
{
    k_icp_setup<<<1, kIcpThreads, 0, ctx->stream>>>(st, P, src_off, tgt_off, bmap, bmap_nn, scale, nn_chunk);
    GCA_CHECK_LAUNCH(ctx);
    return GCA3D_OK;
}

int icp_state_init(gca3d_context *ctx, PairState *st, int P, const double *d_Tinit)
{
    k_state_init<<<grid_for(P, 128), 128, 0, ctx->stream>>>(st, P, d_Tinit);
    GCA_CHECK_LAUNCH(ctx);
    return GCA3D_OK;
}

int icp_search(gca3d_context *ctx, const Batch &src, const Grid &g, PairState *st, int *bmap_nn, int max_blocks_nn,
               int2 *corr, const NNCerts &cert, const IcpScale &prm, int32_t *nn_out, const IcpLoop *guard,
               const IcpShape &shape, bool cold)
{
    // work-item loop: enough blocks to fill the SMs a few times over, never more than
    // the items the capacity can produce
    const int grid_nn = std::max(std::min(max_blocks_nn, ctx->num_sms * shape.nn_bps), 1);
    GCA_PROF_BEGIN(ctx, kKidIcpIter);
    auto search = [&](auto kernel) {
        kernel<<<grid_nn, kIcpThreads, 0, ctx->stream>>>(src.pos, src.seg_off, g.dev, st, bmap_nn, src.P, prm.max_corr,
                                                         corr, cert, nn_out, shape.nn_chunk, bmap_nn + src.P + 1,
                                                         guard ? guard->iter : nullptr, guard ? guard->max_iter : 0);
    };
    if (cold)
        search(k_icp_nn<true>);
    else
        search(k_icp_nn<false>);
    GCA_CHECK_LAUNCH(ctx);
    GCA_PROF_END(ctx, kKidIcpIter);
    return GCA3D_OK;
}

int icp_update(gca3d_context *ctx, const Batch &src, const Grid &g, const float4 *attr0, const float4 *attr1,
               PairState *st, int *bmap, int max_blocks, int *bmap_nn, double *partials, const int2 *corr,
               const IcpScale &prm, bool compensated, const IcpLoop &loop, const IcpShape &shape)
{
    if (!loop.ticket)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "icp: iteration without a finalize ticket");
    const int grid_acc = std::max(std::min(max_blocks, ctx->num_sms * shape.acc_bps), 1);
    GCA_PROF_BEGIN(ctx, kKidIcpIter);
    const int32_t *d_nt = g.dev.d_n;
    if (shape.fused)
    {
        if (compensated)
            k_icp_accum<true, true><<<grid_acc, kIcpThreads, 0, ctx->stream>>>(
                src.pos, src.seg_off, g.dev.spos, attr0, attr1, corr, st, bmap, bmap_nn, src.P, partials,
                prm.sqrt_lg, prm.sqrt_lc, d_nt, ctx->d_err, prm, loop);
        else
            k_icp_accum<false, true><<<grid_acc, kIcpThreads, 0, ctx->stream>>>(
                src.pos, src.seg_off, g.dev.spos, attr0, attr1, corr, st, bmap, bmap_nn, src.P, partials,
                prm.sqrt_lg, prm.sqrt_lc, d_nt, ctx->d_err, prm, loop);
        GCA_CHECK_LAUNCH(ctx);
    }
    else
    {
        if (compensated)
            k_icp_accum<true, false><<<grid_acc, kIcpThreads, 0, ctx->stream>>>(
                src.pos, src.seg_off, g.dev.spos, attr0, attr1, corr, st, bmap, bmap_nn, src.P, partials,
                prm.sqrt_lg, prm.sqrt_lc, d_nt, ctx->d_err, prm, loop);
        else
            k_icp_accum<false, false><<<grid_acc, kIcpThreads, 0, ctx->stream>>>(
                src.pos, src.seg_off, g.dev.spos, attr0, attr1, corr, st, bmap, bmap_nn, src.P, partials,
                prm.sqrt_lg, prm.sqrt_lc, d_nt, ctx->d_err, prm, loop);
        GCA_CHECK_LAUNCH(ctx);
        if (src.P > 1 && max_blocks < kClusterPartials * src.P)
        {
            const auto kernel = compensated ? k_icp_finalize_many<true> : k_icp_finalize_many<false>;
            kernel<<<src.P, kIcpThreads, 0, ctx->stream>>>(st, src.P, bmap, bmap_nn, partials, prm, loop);
            GCA_CHECK_LAUNCH(ctx);
            GCA_PROF_END(ctx, kKidIcpIter);
            return GCA3D_OK;
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kSumGroups * src.P);
        cfg.blockDim = dim3(128);
        cfg.stream = ctx->stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kSumGroups;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        GCA_CUDA(ctx, cudaLaunchKernelEx(&cfg, compensated ? k_icp_finalize<true> : k_icp_finalize<false>, st, src.P,
                                         bmap, bmap_nn, partials, prm, loop));
        GCA_CHECK_LAUNCH(ctx);
    }
    GCA_PROF_END(ctx, kKidIcpIter);
    return GCA3D_OK;
}

int icp_iteration(gca3d_context *ctx, const Batch &src, const Grid &g, const float4 *attr0, const float4 *attr1,
                  PairState *st, int *bmap, int max_blocks, int *bmap_nn, int max_blocks_nn, double *partials,
                  int2 *corr, const NNCerts &cert, const IcpScale &prm, bool compensated, int32_t *nn_out,
                  const IcpLoop &loop, const IcpShape &shape, bool cold)
{
    if (!loop.ticket)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "icp: iteration without a finalize ticket");
    int st_ = icp_search(ctx, src, g, st, bmap_nn, max_blocks_nn, corr, cert, prm, nn_out, nullptr, shape, cold);
    if (!st_)
        st_ = icp_update(ctx, src, g, attr0, attr1, st, bmap, max_blocks, bmap_nn, partials, corr, prm, compensated,
                         loop, shape);
    return st_;
}

// ---------------------------------------------------------------------------
// system for given correspondences (cuda_build_gauss_newton_color_icp) and the
// per-point |r_g| + |r_c| (cuda_compute_abs_residual_color_icp)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kIcpThreads) k_build_gn(const float4 *__restrict__ sp, const int32_t *d_ns,
                                                          const float4 *__restrict__ tp, const float4 *__restrict__ tn,
                                                          const float4 *__restrict__ tg, const int32_t *nn,
                                                          float slg, float slc, double *partials,
                                                          unsigned *ticket, double *out, const int32_t *d_nt,
                                                          int *d_err)
{
    const int ns = *d_ns;
    const int nt = d_nt ? *d_nt : INT_MAX;
    Acc<true> acc;
    acc.zero();
    for (int i = blockIdx.x * kIcpThreads + threadIdx.x; i < ns; i += gridDim.x * kIcpThreads)
    {
        const int j = nn[i];
        if (j < 0)
            continue;
        if (j >= nt)
        {
            atomicOr(d_err, kErrInvalid);
            continue;
        }
        const float4 s4 = sp[i], q = tp[j], n = tn[j], d = tg[j];
        GNTerms t;
        gn_terms(make_float3(s4.x, s4.y, s4.z), s4.w, make_float3(q.x, q.y, q.z), q.w, make_float3(n.x, n.y, n.z),
                 make_float3(d.x, d.y, d.z), slg, slc, t);
        const float dx = q.x - s4.x, dy = q.y - s4.y, dz = q.z - s4.z;
        acc.add_terms(t, dx * dx + dy * dy + dz * dz);
    }
    block_reduce_store<true>(acc, partials + (size_t)blockIdx.x * kTermsPad);
    __threadfence();
    __syncthreads();
    __shared__ int s_last;
    if (threadIdx.x == 0)
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last)
        return;
    if (threadIdx.x < kTerms)
    {
        double v = 0.0;
        for (int b = 0; b < (int)gridDim.x; ++b)
            v += __ldcg(partials + (size_t)b * kTermsPad + threadIdx.x);
        out[threadIdx.x] = v;
    }
    if (threadIdx.x == 0)
        *ticket = 0;
}

__global__ void k_abs_residual(const float4 *__restrict__ sp, const int32_t *d_ns, const float4 *__restrict__ tp,
                               const float4 *__restrict__ tn, const float4 *__restrict__ tg, const int32_t *nn,
                               float slg, float slc, float *out, const int32_t *d_nt, int *d_err)
{
    const int ns = *d_ns;
    const int nt = *d_nt;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ns; i += gridDim.x * blockDim.x)
    {
        const int j = nn[i];
        if (j < 0 || j >= nt)
        {
            if (j >= nt)
                atomicOr(d_err, kErrInvalid); // an index beyond the target
            out[i] = 0.0f;
            continue;
        }
        const float4 s4 = sp[i], q = tp[j], n = tn[j], d = tg[j];
        GNTerms t;
        gn_terms(make_float3(s4.x, s4.y, s4.z), s4.w, make_float3(q.x, q.y, q.z), q.w, make_float3(n.x, n.y, n.z),
                 make_float3(d.x, d.y, d.z), slg, slc, t);
        out[i] = fabsf(t.rg) + fabsf(t.rc);
    }
}

int build_gn(gca3d_context *ctx, const gca3d_cloud *src, const gca3d_cloud *tgt, const int32_t *nn, float lambda,
             double *out30)
{
    const int blocks = std::min(grid_for(src->capacity, kIcpThreads * 4), ctx->num_sms * 2);
    double *partials = ctx->arena.get<double>((size_t)blocks * kTermsPad);
    unsigned *ticket = ctx->arena.get<unsigned>(1);
    double *d_out = ctx->arena.get<double>(kTermsPad);
    if (!partials || !ticket || !d_out)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "build_gn: scratch");
    GCA_CUDA(ctx, cudaMemsetAsync(ticket, 0, sizeof(unsigned), ctx->stream));
    k_build_gn<<<blocks, kIcpThreads, 0, ctx->stream>>>(src->pos, src->d_count, tgt->pos, tgt->nrm, tgt->grd, nn,
                                                        sqrtf(lambda), sqrtf(1.0f - lambda), partials, ticket, d_out,
                                                        tgt->d_count, ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    GCA_CUDA(ctx, cudaMemcpyAsync(out30, d_out, sizeof(double) * kTerms, cudaMemcpyDeviceToHost, ctx->stream));
    GCA_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return consume_device_error(ctx, "build_gauss_newton: a correspondence index lies beyond the target");
}

int abs_residual(gca3d_context *ctx, const gca3d_cloud *src, const gca3d_cloud *tgt, const int32_t *nn, float lambda,
                 float *out)
{
    k_abs_residual<<<grid_for(src->capacity), kBlock, 0, ctx->stream>>>(
        src->pos, src->d_count, tgt->pos, tgt->nrm, tgt->grd, nn, sqrtf(lambda), sqrtf(1.0f - lambda), out,
        tgt->d_count, ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    return consume_device_error(ctx, "abs_residual: a correspondence index lies beyond the target");
}

} // namespace gca3d
