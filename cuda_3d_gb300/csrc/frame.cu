// frame.cu -- depth filter + back-projection + colour fetch + compaction, two kernels.
//
// reference: __adaptive_bilateral_filter / __bilateral_filter / __gaussian*
// (src/geometry/cuda_point_cloud_factory.cu:19-129), __kernel_make_pointcloud_Z16_BGR8
// (:189-267), cuda_make_point_cloud (:269-313) and remove_invalid_points
// (src/geometry/geometry_util.cuh:124-130).
//
// The reference writes an organised W x H array of 28-byte points, synchronises the
// device and compacts with thrust::remove_if.  Here k_frame_filter filters pixel
// tiles staged in shared memory with their halo, decides which pixels become points and
// writes the filtered depth, one bit per pixel and one count per row of a tile;
// k_frame_points (one block per row) adds up the counts above its row, or takes their scan
// for a very tall frame, and writes the
// compacted SoA points in raster order.  Same arithmetic order as the reference (unfused
// multiply/add); the filter weights use det_expf below instead of expf, so the CPU oracle
// reproduces every output bit.
//
// Measured (GB300, ncu): the adaptive 1280 x 720 frame 62 + 15 us, issue-bound (82 % of
// the issue slots while its SMs are busy, 53 M warp instructions); evaluating both exps per
// tap took 596 us.
// The fixed 5 x 5 filter at 640 x 480: 11 + 10 us against 47 us for one kernel with a block
// per row, whose look-back chain over the rows, few warps and eight pixels of registers per
// thread left the SMs idle.  64 x 4 tiles give that small frame 1200 blocks; the adaptive
// filter's 64 x 8 share their larger tables over twice the pixels.
#include "stages.cuh"

#include <algorithm>
#include <type_traits>

namespace gca3d
{

constexpr int kFrameThreads = 256;
constexpr int kTileW = 64;         // pixels of a filter tile: 64 x 4 (fixed), 64 x 8 (adaptive)
constexpr int kRangeFixed = 1024;  // tabulated depth differences of the fixed filter
constexpr int kRangeAdaptive = 1536; // of the adaptive filter: past the last weight above zero
constexpr float kNoDepth = 1e9f;   // a tap without a depth: beyond every tabulated difference
// Up to so many additions of row counts (height x counts) k_frame_points adds up those above
// each row itself: that is quadratic in the height, but no launch.  Above, they are scanned
// first.  us summed / scanned: 640 x 480 (2.3 M) 37 / 45, 1920 x 1080 (35 M) 92 / 99,
// 64 x 8192 (67 M) 55 / 60, 2048 x 2048 (134 M) 165 / 165, 64 x 16,384 (268 M) 86 / 79,
// 64 x 65,536 414 / 221, 64 x 262,144 5370 / 803, 2048 x 8192 690 / 537.
constexpr int64_t kSummedCounts = int64_t(1) << 27;
constexpr int kAdaptiveSteps = 6;                                // adaptive filter: radius 0..5
constexpr int kAdaptiveRadius = kAdaptiveSteps - 1;
constexpr int kAdaptiveSq = 2 * kAdaptiveRadius * kAdaptiveRadius + 1; // squared offsets 0..50

// exp(x) in FP32: Cody-Waite reduction x = k ln2 + r (ln2 split into a 16-bit head
// and a tail so k * head is exact), degree-7 Taylor polynomial in Horner form, and
// 2^k applied in two exact power-of-two multiplies.  Only IEEE-rounded multiply
// and add, so the CPU oracle evaluates the identical sequence and the filtered
// depths (hence the colour lookups, which sit on pixel boundaries) agree bit for
// bit.  Within 2 ulp of exp(x) including the subnormal range.
__device__ __forceinline__ float det_expf(float x)
{
    if (x != x)
        return x;
    if (x > 88.72283935546875f)
        return __int_as_float(0x7f800000);
    if (x < -103.972084045410156f)
        return 0.0f;
    const float kf = rintf(__fmul_rn(x, 1.44269502162933349609f));
    const float r = __fsub_rn(__fsub_rn(x, __fmul_rn(kf, 0.693145751953125f)), __fmul_rn(kf, 1.428606765330187045e-06f));
    float p = 1.0f / 5040.0f;
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 720.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 120.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 24.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f / 6.0f);
    p = __fadd_rn(__fmul_rn(p, r), 0.5f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f);
    p = __fadd_rn(__fmul_rn(p, r), 1.0f);
    const int k = (int)kf;
    const int k1 = k / 2, k2 = k - k / 2;
    return __fmul_rn(__fmul_rn(p, __int_as_float((k1 + 127) << 23)), __int_as_float((k2 + 127) << 23));
}

__device__ __forceinline__ float gauss(float x, float s)
{
    return det_expf(__fdiv_rn(-__fmul_rn(x, x), __fmul_rn(s, s)));
}
__device__ __forceinline__ float gauss_sq(float x2, float s)
{
    return det_expf(__fdiv_rn(-x2, __fmul_rn(s, s)));
}

// the zero-skipping bilateral filter of the pixel at `c` (tile row pitch `pitch`, kNoDepth
// where there is none) with radius R, taps in raster order.  sp: the spatial weights of the
// (2 R + 1)^2 offsets (Square: indexed by the squared offset); range[d], d <= last: the
// weights of the depth differences.  With Cut range[last] is zero, and so is the weight of
// every larger difference (exp decreases): the difference is clamped to last, which also
// gives a tap without a depth a weight of zero, and a zero leaves both sums as they are, so
// no tap branches.  Without, differences above last are evaluated.
template <int R, bool Cut, bool Square>
__device__ __forceinline__ float bilateral(const float *c, int pitch, const float *sp, const float *range, int last,
                                           float sd)
{
    const float d0 = *c == kNoDepth ? 0.0f : *c;
    const float flast = (float)last;
    float sw = 0.0f, sum = 0.0f;
#pragma unroll 1
    for (int dy = -R; dy <= R; ++dy)
    {
        const float *row = c + dy * pitch;
        const float *sprow = Square ? sp + dy * dy : sp + (dy + R) * (2 * R + 1) + R;
#pragma unroll
        for (int dx = -R; dx <= R; ++dx)
        {
            const float nb = row[dx];
            const float diff = fabsf(__fsub_rn(d0, nb));
            // the integer of a float in [0, 2^22]: the low bits after adding 2^23
            const int k = __float_as_int(__fadd_rn(fminf(diff, flast), 8388608.0f)) - 0x4b000000;
            float wr = range[k];
            if (!Cut)
            {
                if (diff > flast && nb != kNoDepth)
                    wr = gauss(diff, sd);
            }
            float wgt = __fmul_rn(sprow[Square ? dx * dx : dx], wr);
            if (!Cut && nb == kNoDepth)
                wgt = 0.0f;
            sw = __fadd_rn(sw, wgt);
            sum = __fadd_rn(sum, __fmul_rn(wgt, nb));
        }
    }
    return __fdiv_rn(sum, sw);
}

// what the two kernels agree on: a pixel's back-projection and its colour pixel
struct FramePixel
{
    float X, Y;
    int tx, ty;
};
__device__ __forceinline__ FramePixel back_project(const FrameParams &P, int x, int y, float z)
{
    const float u = __fsub_rn((float)x, 0.5f), v = __fsub_rn((float)y, 0.5f);
    FramePixel f;
    f.X = __fdiv_rn(__fmul_rn(__fsub_rn(u, P.cx), z), P.fx);
    f.Y = __fdiv_rn(__fmul_rn(__fsub_rn(v, P.cy), z), P.fy);
    const float cxp = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(P.R[0], f.X), __fmul_rn(P.R[3], f.Y)), __fmul_rn(P.R[6], z)), P.t[0]);
    const float cyp = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(P.R[1], f.X), __fmul_rn(P.R[4], f.Y)), __fmul_rn(P.R[7], z)), P.t[1]);
    const float czp = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(P.R[2], f.X), __fmul_rn(P.R[5], f.Y)), __fmul_rn(P.R[8], z)), P.t[2]);
    const float cu = __fadd_rn(__fdiv_rn(__fmul_rn(cxp, P.cfx), czp), P.ccx);
    const float cv = __fadd_rn(__fdiv_rn(__fmul_rn(cyp, P.cfy), czp), P.ccy);
    f.tx = __float2int_rz(__fadd_rn(cu, 0.5f));
    f.ty = __float2int_rz(__fadd_rn(cv, 0.5f));
    return f;
}

// the filtered depth of every pixel, the pixels that become points (one bit each, 32
// pixels of a row per word) and their number in every row of the tile.  R is the radius
// of the fixed filter, kAdaptive or kNone; last the largest tabulated difference of the
// fixed filter.
constexpr int kNone = -1, kAdaptive = -2;
template <int R> constexpr int kTileHeight = R == kAdaptive ? 8 : 4;
template <int R>
__global__ void __launch_bounds__(kFrameThreads) k_frame_filter(const uint16_t *__restrict__ depth, FrameParams P,
                                                                float *zout, uint32_t *mask, int *count, int mask_pitch,
                                                                int tiles_x, int last)
{
    constexpr int kHalo = R == kAdaptive ? kAdaptiveRadius : (R == kNone ? 0 : R);
    constexpr int kTileH = kTileHeight<R>, kRowsPer = kTileW * kTileH / kFrameThreads;
    constexpr int kPitch = kTileW + 2 * kHalo;
    constexpr int kRange = R == kAdaptive ? kAdaptiveSteps * kRangeAdaptive : (R == kNone ? 1 : kRangeFixed);
    constexpr int kSp = R == kAdaptive ? kAdaptiveSteps * kAdaptiveSq : (2 * kHalo + 1) * (2 * kHalo + 1);
    __shared__ float s_depth[(kTileH + 2 * kHalo) * kPitch];
    __shared__ float s_range[kRange];
    __shared__ float s_sp[kSp];
    __shared__ int s_steps;
    __shared__ int s_cnt[kTileH][kTileW / 32];
    const int x0 = (int)(blockIdx.x % tiles_x) * kTileW, y0 = (int)(blockIdx.x / tiles_x) * kTileH;
    const int tid = threadIdx.x;
    if (R == kAdaptive && tid == 0)
        s_steps = 0;
    for (int i = tid; i < (kTileH + 2 * kHalo) * kPitch; i += kFrameThreads)
    {
        const int x = x0 + i % kPitch - kHalo, y = y0 + i / kPitch - kHalo;
        const uint16_t d = x >= 0 && x < P.w && y >= 0 && y < P.h ? depth[(int64_t)y * P.w + x] : (uint16_t)0;
        s_depth[i] = d || R == kNone ? (float)d : kNoDepth;
    }
    if (R >= 0)
    {
        for (int i = tid; i < kSp; i += kFrameThreads)
        {
            const int dy = i / (2 * kHalo + 1) - kHalo, dx = i % (2 * kHalo + 1) - kHalo;
            s_sp[i] = gauss_sq((float)(dx * dx + dy * dy), P.sigma_space);
        }
        for (int d = tid; d <= last; d += kFrameThreads)
            s_range[d] = gauss((float)d, P.sigma_depth);
    }
    __syncthreads();
    const int tx = tid % kTileW, ty0 = tid / kTileW * kRowsPer;
    const int x = x0 + tx;
    // whether a pixel's own depth lies in the range that is filtered, and its adaptive step
    auto in_range = [&](float d0, unsigned &step) {
        const float dv = __fmul_rn(d0, P.depth_scale);
        if (dv < P.tmin || dv > P.tmax)
            return false;
        if (R == kAdaptive)
            step = min((unsigned)__fdiv_rn(__fsub_rn(dv, P.tmin), 0.5f), (unsigned)kAdaptiveRadius);
        return true;
    };
    auto own_depth = [&](int r) {
        const float c = s_depth[(kHalo + ty0 + r) * kPitch + kHalo + tx];
        return R != kNone && c == kNoDepth ? 0.0f : c;
    };
    if (R == kAdaptive)
    {
        // the tables of the steps that this tile's pixels take (1.5 steps of the six on
        // average; a table's end is a weight of zero)
        unsigned seen = 0;
#pragma unroll
        for (int r = 0; r < kRowsPer; ++r)
        {
            unsigned step = 0;
            if (in_range(own_depth(r), step))
                seen |= 1u << step;
        }
        seen = __reduce_or_sync(0xffffffffu, seen);
        if ((tid & 31) == 0)
            atomicOr(&s_steps, (int)seen);
        __syncthreads();
        const int steps = s_steps;
        for (int k = 0; k < kAdaptiveSteps; ++k)
        {
            if (!((steps >> k) & 1))
                continue;
            const float ss = __fadd_rn(8.0f, __fmul_rn((float)k, 1.0f));
            const float sd = __fadd_rn(100.0f, __fmul_rn((float)k, 10.0f));
            for (int i = tid; i <= 2 * k * k; i += kFrameThreads)
                s_sp[k * kAdaptiveSq + i] = gauss_sq((float)i, ss);
            for (int d = tid; d < kRangeAdaptive; d += kFrameThreads)
                s_range[k * kRangeAdaptive + d] = gauss((float)d, sd);
        }
        __syncthreads();
    }
    // (a space sigma whose square is zero makes the centre's weight 0 / 0)
    const bool cut = R < 0 || (s_range[last] == 0.0f && __fmul_rn(P.sigma_space, P.sigma_space) > 0.0f);
#pragma unroll 1
    for (int r = 0; r < kRowsPer; ++r)
    {
        const int y = y0 + ty0 + r;
        const float *c = s_depth + (kHalo + ty0 + r) * kPitch + kHalo + tx;
        float fd = own_depth(r);
        unsigned step = 0;
        if (R >= 0)
        {
            if (in_range(fd, step))
                fd = cut ? bilateral<kHalo, true, false>(c, kPitch, s_sp, s_range, last, P.sigma_depth)
                         : bilateral<kHalo, false, false>(c, kPitch, s_sp, s_range, last, P.sigma_depth);
        }
        else if (R == kAdaptive)
        {
            // the lanes of one radius at a time: every radius has its own unrolled taps
            const int rad = in_range(fd, step) ? (int)step : -1;
            auto filter = [&](auto radius) {
                constexpr int K = decltype(radius)::value;
                if (rad == K)
                    fd = bilateral<K, true, true>(c, kPitch, s_sp + K * kAdaptiveSq, s_range + K * kRangeAdaptive,
                                                  kRangeAdaptive - 1, 0.0f);
            };
            filter(std::integral_constant<int, 0>{});
            filter(std::integral_constant<int, 1>{});
            filter(std::integral_constant<int, 2>{});
            filter(std::integral_constant<int, 3>{});
            filter(std::integral_constant<int, 4>{});
            filter(std::integral_constant<int, 5>{});
        }
        const float z = __fmul_rn(fd, P.depth_scale);
        bool valid = false;
        if (x < P.w && y < P.h && !(z < P.tmin || z > P.tmax))
        {
            const FramePixel f = back_project(P, x, y, z);
            valid = !(f.tx < 0 || f.tx >= P.w || f.ty < 0 || f.ty >= P.h);
            zout[(int64_t)y * P.w + x] = z;
        }
        const unsigned bits = __ballot_sync(0xffffffffu, valid);
        if ((tid & 31) == 0)
        {
            s_cnt[ty0 + r][tx >> 5] = __popc(bits);
            if (x < P.w && y < P.h)
                mask[y * mask_pitch + (x >> 5)] = bits;
        }
    }
    __syncthreads();
    if (tid < kTileH && y0 + tid < P.h)
    {
        int n = 0;
#pragma unroll
        for (int k = 0; k < kTileW / 32; ++k)
            n += s_cnt[tid][k];
        count[(y0 + tid) * tiles_x + (int)(blockIdx.x % tiles_x)] = n;
    }
}

// the length of the row counts, for their scan
__global__ void k_frame_counts(int32_t *d_counts, int32_t n) { *d_counts = n; }

// the points of one image row, after those of the rows above it.  Scanned: count holds the
// counts' exclusive prefixes; otherwise the counts, and every block sums those above its row
// (from L2), which needs no launch and no wait between blocks
template <bool Scanned>
__global__ void __launch_bounds__(kFrameThreads) k_frame_points(const uint8_t *__restrict__ bgr, FrameParams P,
                                                                const float *__restrict__ zin,
                                                                const uint32_t *__restrict__ mask,
                                                                const int *__restrict__ count, int mask_pitch,
                                                                int tiles_x, float4 *out_pos, float4 *out_col,
                                                                int32_t *d_count)
{
    __shared__ int s_sum[kFrameThreads / 32];
    const int y = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the words of this row (at most 2048 / 32 = 64) and their exclusive prefix, in every warp
    const int words = (P.w + 31) >> 5;
    const uint32_t w0 = lane < words ? mask[y * mask_pitch + lane] : 0u;
    const uint32_t w1 = lane + 32 < words ? mask[y * mask_pitch + lane + 32] : 0u;
    if (!Scanned)
    {
        int above = 0;
        for (int i = threadIdx.x; i < y * tiles_x; i += kFrameThreads)
            above += count[i];
        above = __reduce_add_sync(0xffffffffu, above);
        if (lane == 0)
            s_sum[warp] = above;
    }
    int p0 = __popc(w0), p1 = __popc(w1);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const int a = __shfl_up_sync(0xffffffffu, p0, o), b = __shfl_up_sync(0xffffffffu, p1, o);
        if (lane >= o)
            p0 += a, p1 += b;
    }
    p1 += __shfl_sync(0xffffffffu, p0, 31);
    int base = 0;
    if (Scanned)
        base = count[y * tiles_x];
    else
    {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kFrameThreads / 32; ++k)
            base += s_sum[k];
    }
    if (y == P.h - 1 && threadIdx.x == 31)
        *d_count = base + p1;
    for (int i = warp; i < words; i += kFrameThreads / 32)
    {
        const uint32_t bits = __shfl_sync(0xffffffffu, i < 32 ? w0 : w1, i & 31);
        const int incl = __shfl_sync(0xffffffffu, i < 32 ? p0 : p1, i & 31);
        if (!((bits >> lane) & 1u))
            continue;
        const int x = 32 * i + lane;
        const float z = zin[(int64_t)y * P.w + x];
        const FramePixel f = back_project(P, x, y, z);
        const int64_t ci = 3 * ((int64_t)f.ty * P.w + f.tx);
        const float sc = 1.0f / 255.0f;
        const float r = __fmul_rn((float)bgr[ci + 2], sc), g = __fmul_rn((float)bgr[ci + 1], sc),
                    b = __fmul_rn((float)bgr[ci + 0], sc);
        const int at = base + incl - __popc(bits) + __popc(bits & ((1u << lane) - 1u));
        out_pos[at] = make_float4(f.X, f.Y, z, intensity_of(r, g, b));
        out_col[at] = make_float4(r, g, b, 0.0f);
    }
}

int frame_to_cloud(gca3d_context *ctx, const uint16_t *depth, const uint8_t *bgr, const FrameParams &P,
                   gca3d_cloud *out)
{
    const int tiles_x = div_up(P.w, kTileW), words = div_up(P.w, 32);
    float *z = ctx->arena.get<float>((size_t)P.w * P.h);
    uint32_t *mask = ctx->arena.get<uint32_t>((size_t)words * P.h);
    const int64_t counts = (int64_t)tiles_x * P.h;
    int *count = ctx->arena.get<int>(counts);
    const bool scanned = counts * P.h > kSummedCounts;
    int *prefix = scanned ? ctx->arena.get<int>(counts) : nullptr;
    int *d_counts = scanned ? ctx->arena.get<int>(1) : nullptr;
    if (!z || !mask || !count || (scanned && (!prefix || !d_counts)))
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "frame_to_cloud: scratch");
    // the fixed filter's weights reach zero at a difference of 10.2 sigma (exp(-104)): the
    // table ends just past it, or at its capacity (then larger differences are evaluated)
    const int last = (int)std::min(10.3f * P.sigma_depth + 2.0f, (float)(kRangeFixed - 1));
    GCA_PROF_BEGIN(ctx, kKidFrame);
    auto filter = [&](auto radius) {
        constexpr int R = decltype(radius)::value;
        k_frame_filter<R><<<tiles_x * div_up(P.h, kTileHeight<R>), kFrameThreads, 0, ctx->stream>>>(
            depth, P, z, mask, count, words, tiles_x, last);
    };
    static_assert(kMaxFilterRadius == 7, "one instantiation per radius");
    const int R = P.mode == GCA3D_FILTER_ADAPTIVE ? kAdaptive : (P.mode == GCA3D_FILTER_NONE ? kNone : P.radius);
    switch (R)
    {
    case kAdaptive: filter(std::integral_constant<int, kAdaptive>{}); break;
    case kNone: filter(std::integral_constant<int, kNone>{}); break;
    case 0: filter(std::integral_constant<int, 0>{}); break;
    case 1: filter(std::integral_constant<int, 1>{}); break;
    case 2: filter(std::integral_constant<int, 2>{}); break;
    case 3: filter(std::integral_constant<int, 3>{}); break;
    case 4: filter(std::integral_constant<int, 4>{}); break;
    case 5: filter(std::integral_constant<int, 5>{}); break;
    case 6: filter(std::integral_constant<int, 6>{}); break;
    default: filter(std::integral_constant<int, 7>{}); break;
    }
    GCA_CHECK_LAUNCH(ctx);
    if (scanned)
    {
        k_frame_counts<<<1, 1, 0, ctx->stream>>>(d_counts, (int32_t)counts);
        GCA_CHECK_LAUNCH(ctx);
        const int st = exclusive_scan(ctx, count, prefix, d_counts, counts, nullptr);
        if (st)
            return st;
    }
    const auto points = scanned ? k_frame_points<true> : k_frame_points<false>;
    points<<<P.h, kFrameThreads, 0, ctx->stream>>>(bgr, P, z, mask, scanned ? prefix : count, words, tiles_x, out->pos,
                                                   out->col, out->d_count);
    GCA_CHECK_LAUNCH(ctx);
    GCA_PROF_END(ctx, kKidFrame);
    return GCA3D_OK;
}

} // namespace gca3d

using namespace gca3d;

namespace gca3d
{
// cuda_make_point_cloud (cuda_point_cloud_factory.cu:283-290): parameters present,
// depth_scale > 0; plus this kernel's limits (width, filter radius)
int frame_params(gca3d_context *ctx, int w, int h, const gca3d_intrinsics *di, const gca3d_intrinsics *ci,
                 const gca3d_extrinsics *d2c, float depth_scale, float tmin, float tmax, const gca3d_filter *filter,
                 FrameParams &P)
{
    if (!di || w <= 0 || h <= 0)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "frame_to_cloud: bad arguments");
    if (!(depth_scale > 0.0f))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "frame_to_cloud: depth_scale must be > 0");
    if (w > kMaxFrameWidth)
        return fail(ctx, GCA3D_ERR_NOT_SUPPORTED, "frame_to_cloud: width above 2048");
    P = FrameParams{};
    P.w = w, P.h = h;
    P.fx = di->fx, P.fy = di->fy, P.cx = di->cx, P.cy = di->cy;
    const gca3d_intrinsics *c = ci ? ci : di;
    P.cfx = c->fx, P.cfy = c->fy, P.ccx = c->cx, P.ccy = c->cy;
    for (int k = 0; k < 9; ++k)
        P.R[k] = d2c ? d2c->rotation[k] : (k % 4 == 0 ? 1.0f : 0.0f);
    for (int k = 0; k < 3; ++k)
        P.t[k] = d2c ? d2c->translation[k] : 0.0f;
    P.depth_scale = depth_scale, P.tmin = tmin, P.tmax = tmax;
    P.mode = filter ? filter->mode : GCA3D_FILTER_ADAPTIVE;
    P.radius = filter ? filter->radius : 0;
    P.sigma_space = filter ? filter->sigma_space : 0.0f;
    P.sigma_depth = filter ? filter->sigma_depth : 0.0f;
    if (P.mode < 0 || P.mode > 2 || (P.mode == GCA3D_FILTER_FIXED &&
                                     (P.radius < 0 || P.radius > kMaxFilterRadius || !(P.sigma_space > 0) ||
                                      !(P.sigma_depth > 0))))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "frame_to_cloud: bad filter parameters");
    return GCA3D_OK;
}
} // namespace gca3d

extern "C" int gca3d_frame_to_cloud(gca3d_context *ctx, const uint16_t *depth, const uint8_t *bgr, int w, int h,
                                    const gca3d_intrinsics *di, const gca3d_intrinsics *ci,
                                    const gca3d_extrinsics *d2c, float depth_scale, float tmin, float tmax,
                                    const gca3d_filter *filter, gca3d_cloud *out)
{
    if (!ctx || !depth || !bgr || !out)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "frame_to_cloud: bad arguments");
    FrameParams P;
    int st = frame_params(ctx, w, h, di, ci, d2c, depth_scale, tmin, tmax, filter, P);
    if (st)
        return st;
    if ((int64_t)w * h > out->capacity)
        return fail(ctx, GCA3D_ERR_CAPACITY, "frame_to_cloud: output capacity below w * h");
    ctx->arena.reset();
    if ((st = frame_to_cloud(ctx, depth, bgr, P, out)))
        return st;
    out->has_normals = out->has_grad = false;
    return GCA3D_OK;
}
