// sort_keys.cuh -- the keys of P point sets and what the radix sort needs to know of them:
// bounds and key layout in one launch, keys with their digit histograms and offsets in
// another (the passes are in sort_scan.cu).
//
// Both are bound by latency for one set (a launch with nothing to do takes 2 us: bounds,
// layout, keys, histogram and offsets were seven launches) and by reading the points for a
// batch; the histogram taken as the keys are made saves reading them back.
#pragma once

#include "stages.cuh"

#include <algorithm>

namespace gca3d
{

constexpr int kSortThreads = 256;
constexpr int kSortItems = 12;
constexpr int kSortTile = kSortThreads * kSortItems; // 3072 keys per tile
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kLookWindow = 8; // predecessor tiles read at once in the look-back
constexpr int kLookWide = 32;  // the same where all tiles start together

// Control words of one sort.  The keys come in P segments ([seg_off[s], seg_off[s+1]),
// the segment index being the key's most significant field, each segment's keys in
// ascending index order), so a segment's keys end up in its own range: the sort runs
// per segment -- digit offsets per segment, tiles that never straddle two segments,
// and a look-back that ends at the segment's first tile, so the look-back chains are
// as long as a segment, not as the batch.  A pass is skipped when every segment's
// keys share its digit (the segment field's digits always do).
struct SortCtl
{
    int nontrivial[8];
    int in_sel[8];
    uint32_t tile_ctr[8];
    uint32_t prep_ticket;
    int ntiles; // tiles over all segments
    uint32_t cells[3]; // largest cell per axis over the segments
    uint32_t bounds_ticket;
};

// per-segment scratch of a sort: hist[s][d][b] digit counts, doff[s][d][b] the first
// output position of bucket b of digit d in segment s, tile_first[s] the segment's
// first tile (P + 1 entries), ticket[2 P] the blocks done with a segment's bounds and keys
struct SortSeg
{
    uint32_t *hist;
    uint32_t *doff;
    int32_t *tile_first;
    uint32_t *ticket;
};

// the scratch of one sort; ctl, S.hist and S.ticket start at zero, and so do the caller's
// own bytes at zeroed (one memset)
struct SortPlan
{
    SortCtl *ctl;
    SortSeg S;
    uint32_t *status; // two buffers of status_words
    int64_t status_words, ntiles;
    void *zeroed;
};
int sort_plan(gca3d_context *ctx, int P, int64_t cap, size_t zero_bytes, SortPlan &sp);
// the passes over keys and histograms made by k_sort_keys; stable, segment by segment
int sort_passes(gca3d_context *ctx, SortBuffers &sb, const SortPlan &sp, const int32_t *seg_off, int P);

// the byte-digit d of a sort word: bits [ks + 8 d, ks + 8 d + 8), ks the key's lowest bit
// (SortBuffers::d_kshift), zero above bit 63
__device__ __forceinline__ uint32_t sort_digit(uint64_t k, int ks, int d)
{
    const int sh = ks + 8 * d;
    return sh < 64 ? (uint32_t)(k >> sh) & 255u : 0u;
}

// Maker: the points of P sets and their keys (also of cluster_sort.cuh).
//   int2 range(int seg) const                    elements [x, y) of set seg
//   float4 point(int seg, int i) const           element i
//   int sub_bits() const                         bits below the key proper (finer scales)
//   int segment(mn, mx, float3 &origin, uint32_t cells[3]) const
//                                                a set's origin and largest cells (cells
//                                                untouched when it is empty); error bits
//   int layout(cells, P, KeyLayout &) const      the layout they share; error bits
//   void begin(int n) const                      one set of n elements: tables of the maker's
//   uint64_t key(float4, seg, KeyLayout, float3 origin, int *d_err) const

// minima over the block of six values per thread, returned to threads 0..5
__device__ __forceinline__ float block_min6(const float v_in[6])
{
    __shared__ float s_red[kBlock / 32][6];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int a = 0; a < 6; ++a)
    {
        float v = v_in[a];
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            v = fminf(v, __shfl_xor_sync(0xffffffffu, v, d));
        if (lane == 0)
            s_red[warp][a] = v;
    }
    __syncthreads();
    float m = 0.0f;
    if (threadIdx.x < 6)
    {
        m = s_red[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < kBlock / 32; ++w)
            m = fminf(m, s_red[w][threadIdx.x]);
    }
    __syncthreads();
    return m;
}

// whether this block is the last of `of` to arrive at the ticket, with the others' writes
// visible if so; every thread of the block calls it
__device__ __forceinline__ bool last_arrival(uint32_t *ticket, uint32_t of)
{
    __shared__ int s_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(ticket, 1u) == of - 1u;
    __syncthreads();
    const bool last = s_last != 0;
    __syncthreads();
    if (last)
        __threadfence();
    return last;
}

// bounds of every set, its origin, and the key layout over all (block (x, s): part of set s).
// The last block of a set reduces its blocks' bounds, the last set's block lays out the keys.
template <class Maker>
__global__ void __launch_bounds__(kBlock) k_sort_bounds(Maker mk, int P, float *partial, SortCtl *ctl, SortSeg S,
                                                        float3 *origin, KeyLayout *lay, int index_bits, int *d_ib,
                                                        int *d_kshift, int *d_err)
{
    const int seg = blockIdx.y, gx = gridDim.x;
    const int2 r = mk.range(seg);
    constexpr float kMax = 3.402823466e38f;
    float v[6] = {kMax, kMax, kMax, kMax, kMax, kMax}; // minima of the coordinates and of their negatives
#pragma unroll 4
    for (int i = r.x + blockIdx.x * kBlock + threadIdx.x; i < r.y; i += gx * kBlock)
    {
        const float4 p = mk.point(seg, i);
        v[0] = fminf(v[0], p.x), v[1] = fminf(v[1], p.y), v[2] = fminf(v[2], p.z);
        v[3] = fminf(v[3], -p.x), v[4] = fminf(v[4], -p.y), v[5] = fminf(v[5], -p.z);
    }
    float *mine = partial + (size_t)seg * gx * 6;
    const float m = block_min6(v);
    if (threadIdx.x < 6)
        mine[blockIdx.x * 6 + threadIdx.x] = m;
    if (!last_arrival(S.ticket + seg, gx))
        return;
#pragma unroll
    for (int a = 0; a < 6; ++a)
        v[a] = kMax;
    for (int b = threadIdx.x; b < gx; b += kBlock)
#pragma unroll
        for (int a = 0; a < 6; ++a)
            v[a] = fminf(v[a], __ldcg(mine + b * 6 + a));
    const float t = block_min6(v);
    __shared__ float s_b[6];
    if (threadIdx.x < 6)
        s_b[threadIdx.x] = t;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        const float mn[3] = {s_b[0], s_b[1], s_b[2]}, mx[3] = {-s_b[3], -s_b[4], -s_b[5]};
        float3 o;
        uint32_t cells[3] = {0u, 0u, 0u};
        const int err = mk.segment(mn, mx, o, cells);
        if (err)
            atomicOr(d_err, err);
        origin[seg] = o;
#pragma unroll
        for (int a = 0; a < 3; ++a)
            atomicMax(&ctl->cells[a], cells[a]);
    }
    if (!last_arrival(&ctl->bounds_ticket, P) || threadIdx.x != 0)
        return;
    const uint32_t cells[3] = {__ldcg(&ctl->cells[0]), __ldcg(&ctl->cells[1]), __ldcg(&ctl->cells[2])};
    KeyLayout L;
    const int err = mk.layout(cells, P, L);
    if (err)
        atomicOr(d_err, err);
    *lay = L;
    const int ib = packed_index_bits(L.total_bits + mk.sub_bits(), index_bits);
    *d_ib = ib;
    *d_kshift = ib + mk.sub_bits();
    if (P == 1)
        mk.begin(r.y - r.x);
}

// per segment (the last block of its keys): bucket offsets of every digit, whether the
// segment's digit varies, and its tile count.  One warp per digit, each lane scanning 8
// consecutive buckets.
__device__ __forceinline__ void sort_segment_offsets(SortCtl *ctl, const SortSeg &S, int seg, int b, int n, int digits)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t *gh = S.hist + (size_t)seg * 8 * 256;
    uint32_t *go = S.doff + (size_t)seg * 8 * 256;
    for (int d = warp; d < digits; d += kBlock / 32)
    {
        uint32_t c[8], sum = 0;
        bool triv = n <= 1;
#pragma unroll
        for (int k = 0; k < 8; ++k)
        {
            c[k] = __ldcg(&gh[d * 256 + 8 * lane + k]);
            sum += c[k];
            triv |= (int)c[k] == n;
        }
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o)
                incl += y;
        }
        uint32_t run = (uint32_t)b + incl - sum;
#pragma unroll
        for (int k = 0; k < 8; ++k)
        {
            go[d * 256 + 8 * lane + k] = run;
            run += c[k];
        }
        triv = __any_sync(0xffffffffu, triv);
        if (lane == 0 && !triv)
            atomicOr(&ctl->nontrivial[d], 1);
    }
    if (threadIdx.x == 0)
        S.tile_first[seg + 1] = (n + kSortTile - 1) / kSortTile;
}

// the last segment's block: the segments' first tiles (exclusive prefix of the tile counts;
// P <= 4096: 16 per thread, then a block scan) and the ping-pong bookkeeping
__device__ __forceinline__ void sort_tiles(SortCtl *ctl, const SortSeg &S, int P, int *d_sel)
{
    if (P == 1)
    {
        if (threadIdx.x == 0)
        {
            S.tile_first[0] = 0;
            ctl->ntiles = S.tile_first[1];
        }
    }
    else
    {
        __shared__ int s_part[256];
        constexpr int kPer = (kMaxSegments + 255) / 256;
        const int p0 = threadIdx.x * kPer;
        int cnt[kPer], sum = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k)
        {
            cnt[k] = p0 + k < P ? __ldcg(&S.tile_first[p0 + k + 1]) : 0;
            sum += cnt[k];
        }
        s_part[threadIdx.x] = sum;
        __syncthreads();
        if (threadIdx.x < 32)
        {
            int v[8], t = 0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
            {
                v[k] = s_part[threadIdx.x * 8 + k];
                t += v[k];
            }
            int incl = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)threadIdx.x >= o)
                    incl += y;
            }
            int run = incl - t;
#pragma unroll
            for (int k = 0; k < 8; ++k)
            {
                s_part[threadIdx.x * 8 + k] = run;
                run += v[k];
            }
        }
        __syncthreads();
        int run = s_part[threadIdx.x];
#pragma unroll
        for (int k = 0; k < kPer; ++k)
            if (p0 + k < P)
            {
                S.tile_first[p0 + k] = run;
                run += cnt[k];
            }
        if (threadIdx.x == 255)
        {
            // the last thread's running sum is the total
            ctl->ntiles = run;
            S.tile_first[P] = run;
        }
    }
    if (threadIdx.x == 0)
    {
        int sel = 0;
        for (int d = 0; d < 8; ++d)
        {
            ctl->in_sel[d] = sel;
            if (__ldcg(&ctl->nontrivial[d]))
                sel ^= 1;
        }
        *d_sel = sel;
    }
}

// the sort words of every set with the histograms of their byte-digits (block (x, s): part of
// set s); also clears the first look-back status buffer
template <class Maker>
__global__ void __launch_bounds__(kBlock) k_sort_keys(Maker mk, int P, const float3 *origin, const KeyLayout *lay,
                                                      const int *d_ib, const int *d_kshift, uint64_t *keys,
                                                      int32_t *vals, SortCtl *ctl, SortSeg S, uint32_t *status0,
                                                      int64_t status_words, int *d_sel, int *d_err)
{
    __shared__ uint32_t h[8][256];
    const KeyLayout L = *lay;
    const int ib = *d_ib, ks = *d_kshift;
    const int digits = min((L.total_bits + 7) >> 3, 8); // the digits above are zero
    for (int i = threadIdx.x; i < digits * 256; i += kBlock)
        (&h[0][0])[i] = 0;
    __syncthreads();
    const int seg = blockIdx.y;
    const int2 r = mk.range(seg);
    const float3 o = origin[seg];
#pragma unroll 2
    for (int i = r.x + blockIdx.x * kBlock + threadIdx.x; i < r.y; i += gridDim.x * kBlock)
    {
        const uint64_t k = mk.key(mk.point(seg, i), seg, L, o, d_err);
        sort_store(keys, vals, i, k, ib);
        const uint64_t w = ib ? k << ib : k;
        for (int d = 0; d < digits; ++d)
            atomicAdd(&h[d][sort_digit(w, ks, d)], 1u);
    }
    const int64_t nb = (int64_t)gridDim.x * gridDim.y, bid = (int64_t)blockIdx.y * gridDim.x + blockIdx.x;
    for (int64_t i = bid * kBlock + threadIdx.x; i < status_words; i += nb * kBlock)
        status0[i] = 0;
    __syncthreads();
    uint32_t *gh = S.hist + (size_t)seg * 8 * 256;
    for (int i = threadIdx.x; i < digits * 256; i += kBlock)
    {
        const uint32_t c = (&h[0][0])[i];
        if (c)
            atomicAdd(&gh[i], c);
    }
    if (!last_arrival(S.ticket + P + seg, gridDim.x))
        return;
    sort_segment_offsets(ctl, S, seg, r.x, r.y - r.x, digits);
    if (!last_arrival(&ctl->prep_ticket, P))
        return;
    sort_tiles(ctl, S, P, d_sel);
}

// bounds, layout, keys and the stable sort of P sets (at most cap points in all and
// max_seg_cap in one), seg_off[P + 1] their element ranges; *zeroed: zero_bytes of cleared
// memory for the caller
template <class Maker>
int sort_by_keys(gca3d_context *ctx, const Maker &mk, SortBuffers &sb, const int32_t *seg_off, int P, int64_t cap,
                 int64_t max_seg_cap, KeyLayout *lay, float3 *origin, size_t zero_bytes, void **zeroed)
{
    SortPlan sp;
    int st = sort_plan(ctx, P, cap, zero_bytes, sp);
    if (st)
        return st;
    if (zeroed)
        *zeroed = sp.zeroed;
    // eight points per thread in the largest set, at most 16 blocks per SM over all sets
    const int gx = (int)std::max<int64_t>(1, std::min<int64_t>(grid_for(max_seg_cap, kBlock * 8),
                                                               ((int64_t)ctx->num_sms * 16 + P - 1) / P));
    float *partial = ctx->arena.get<float>((size_t)6 * gx * P);
    if (!partial)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "sort keys: scratch");
    k_sort_bounds<<<dim3(gx, P), kBlock, 0, ctx->stream>>>(mk, P, partial, sp.ctl, sp.S, origin, lay, index_bits(cap),
                                                           sb.d_ib, sb.d_kshift, ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    k_sort_keys<<<dim3(gx, P), kBlock, 0, ctx->stream>>>(mk, P, origin, lay, sb.d_ib, sb.d_kshift, sb.keys[0],
                                                         sb.vals[0], sp.ctl, sp.S, sp.status, sp.status_words, sb.d_sel,
                                                         ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    return sort_passes(ctx, sb, sp, seg_off, P);
}

} // namespace gca3d
