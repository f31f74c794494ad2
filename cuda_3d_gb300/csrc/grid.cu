// grid.cu -- uniform grid over a batch of point sets and its queries.
//
// reference: the grid build in src/geometry/cuda_nn_search.cu:573-608 (cell id, radix
// sort, reduce_by_key, dense cell table rebuilt per call), nn_search_functor
// (:113-214) and the radius-list passes (:216-414, 622-723).
//
// GB300 layout: points are physically reordered into cell order (float4 with the z
// cell in .w), so a query streams contiguous memory.  Instead of a dense
// nx*ny*nz table of cells the grid keeps [start, end) in the sorted arrays for the rows
// (segment, x, y): a direct table of runs of a row's z cells where the key is short enough
// for a few entries per point, a hash of the occupied rows elsewhere.  A 27-cell
// neighbourhood is 9 rows, each one or two entries (two where its window of z cells crosses
// a run) or a hash probe, and 9 contiguous scans over z.  Cells, rows and the scan order (x, then y, then z,
// then ascending original index) are the reference's, so radius lists come out in
// the reference's order for the same grid origin.  Memory is O(points), not
// O(bounding-box volume).
#include "cluster_sort.cuh"
#include "grid_query.cuh"
#include "stages.cuh"

#include <algorithm>

namespace gca3d
{

__device__ __forceinline__ float3 grid_origin(const float mn[3], float cell, int mode, float3 given)
{
    float o[3];
    const float g[3] = {given.x, given.y, given.z};
#pragma unroll
    for (int a = 0; a < 3; ++a)
        o[a] = mode == kOriginGiven
                   ? g[a]
                   : (mode == kOriginPadF64 ? (float)__dsub_rn((double)mn[a], __dmul_rn(1.5, (double)cell))
                                            : __fsub_rn(mn[a], __fmul_rn(1.5f, cell)));
    return make_float3(o[0], o[1], o[2]);
}

// the largest cell per axis of a set with bounds mn, mx (untouched when the set is empty);
// error bits
__device__ __forceinline__ int grid_extent(const float mn[3], const float mx[3], float3 origin, float cell,
                                           uint32_t cells[3])
{
    if (!(mx[0] >= mn[0]))
        return 0; // empty
    int err = 0;
    const float o[3] = {origin.x, origin.y, origin.z};
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        const int lo = cell_of(mn[a], o[a], cell);
        int hi = cell_of(mx[a], o[a], cell);
        if (lo < 0 || hi >= (1 << 21))
        {
            err = kErrKeyBits;
            hi = (1 << 21) - 1;
        }
        cells[a] = (uint32_t)max(hi, 0);
    }
    return err;
}

__device__ __forceinline__ uint64_t grid_key(float4 p, int seg, const KeyLayout &L, float3 o, float cell, float inv)
{
    // clamp defends the key fields against points outside the declared origin
    const uint64_t cx = (uint64_t)max(cell_of_inv(p.x, o.x, cell, inv), 0) & ((1ull << L.bx) - 1);
    const uint64_t cy = (uint64_t)max(cell_of_inv(p.y, o.y, cell, inv), 0) & ((1ull << L.by) - 1);
    const uint64_t cz = (uint64_t)max(cell_of_inv(p.z, o.z, cell, inv), 0) & ((1ull << L.bz) - 1);
    return ((uint64_t)seg << (L.bx + L.by + L.bz)) | (cx << (L.by + L.bz)) | (cy << L.bz) | cz;
}

// the grid keys of P sets; one set may come with its count alone (its offsets are then
// written by begin)
struct GridMaker
{
    const float4 *pos;
    int32_t *seg_off;
    const int32_t *d_count; // or null
    float cell, inv;
    int mode;
    float3 given;
    int table_bits; // a direct row table may have 2^table_bits entries
    __device__ int2 range(int seg) const
    {
        return d_count ? make_int2(0, *d_count) : make_int2(seg_off[seg], seg_off[seg + 1]);
    }
    __device__ float4 point(int, int i) const { return __ldg(&pos[i]); }
    __device__ int sub_bits() const { return 0; }
    __device__ void begin(int n) const
    {
        if (d_count)
        {
            seg_off[0] = 0;
            seg_off[1] = n;
        }
    }
    __device__ int segment(const float mn[3], const float mx[3], float3 &o, uint32_t cells[3]) const
    {
        o = grid_origin(mn, cell, mode, given);
        return grid_extent(mn, mx, o, cell, cells);
    }
    __device__ int layout(const uint32_t cells[3], int P, KeyLayout &L) const
    {
        L.bseg = bitlen_u32((uint32_t)(P - 1));
        L.bx = bitlen_u32(max(cells[0], 1u));
        L.by = bitlen_u32(max(cells[1], 1u));
        L.bz = bitlen_u32(max(cells[2], 1u));
        L.total_bits = L.bseg + L.bx + L.by + L.bz;
        L.morton = 0;
        // the shortest runs that fit the table, of four cells at least (a search's window of
        // three cells then lies in one run or two); without room for whole rows, the hash
        L.zs = max(min(2, L.bz), L.total_bits - table_bits);
        L.direct = L.zs <= L.bz && L.bz >= 1 && L.zs >= 1;
        return L.total_bits > 64 ? kErrKeyBits : 0;
    }
    __device__ uint64_t key(float4 p, int seg, const KeyLayout &L, float3 o, int *) const
    {
        return grid_key(p, seg, L, o, cell, inv);
    }
};

bool grid_cluster_enable() { return cluster_sort_enable<GridMaker>(); }

// the points in grid order, and the row table: the first point of a run (direct) or of a row
// (hash) finds its end by galloping and writes the entry
__global__ void __launch_bounds__(kBlock) k_grid_scatter(SortBuffers sb, const int32_t *d_n, const KeyLayout *lay,
                                                         const float4 *__restrict__ pos, float4 *spos, int32_t *sidx,
                                                         float *sint, int *scz, uint64_t *skey, RowSlot *slots,
                                                         uint32_t hmask, int *err)
{
    const int n = *d_n;
    const SortedView sv = sorted_view(sb);
    const KeyLayout L = *lay;
    const uint64_t mz = (1ull << L.bz) - 1;
    const int shift = L.direct ? L.zs : L.bz;
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
    {
        const uint64_t k = sv.key(s);
        const int g = sv.val(s);
        if (!GCA_INDEX_OK(g, n, err))
            continue;
        const float4 p = __ldg(&pos[g]);
        const unsigned long long rk = k >> shift;
        const bool first = s == 0 || (sv.key(s - 1) >> shift) != rk;
        spos[s] = make_float4(p.x, p.y, p.z, __int_as_float((int)(k & mz)));
        sidx[s] = g;
        sint[s] = p.w;
        scz[s] = (int)(k & mz);
        if (skey)
            skey[s] = k;
        if (!first)
            continue;
        // the end of the run (the keys are sorted): galloping from s, then bisection
        // of (lo, hi], where lo is in the run and hi is past it or n
        int lo = s, hi = s + 1, step = 1;
        while (hi < n && (sv.key(hi) >> shift) == rk)
        {
            lo = hi;
            step <<= 1;
            hi = s + step;
        }
        hi = min(hi, n);
        while (hi - lo > 1)
        {
            const int m = (lo + hi) >> 1;
            if ((sv.key(m) >> shift) == rk)
                lo = m;
            else
                hi = m;
        }
        if (L.direct)
        {
            if (GCA_INDEX_OK(rk, 1ll << (L.total_bits - L.zs), err))
                reinterpret_cast<int2 *>(slots)[rk] = make_int2(s, hi);
            continue;
        }
        uint32_t h = hash_u64(rk) & hmask;
        bool done = false;
        for (uint32_t probe = 0; probe <= hmask && !done; ++probe)
        {
            const unsigned long long prev = atomicCAS(&slots[h].key, kEmptyKey, rk);
            if (prev == kEmptyKey || prev == rk)
            {
                slots[h].start = s;
                slots[h].end = hi;
                done = true;
            }
            h = (h + 1) & hmask;
        }
        if (!done)
            atomicOr(err, kErrCapacity);
    }
}

// an empty row table of the size its layout takes
__global__ void __launch_bounds__(kBlock) k_grid_clear(const KeyLayout *lay, uint4 *slots, uint32_t hcap)
{
    const KeyLayout L = *lay;
    const uint32_t n = L.direct ? max(1u << (L.total_bits - L.zs) >> 1, 1u) : hcap; // 16-byte words
    const uint32_t ones = 0xffffffffu;
    for (uint32_t i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock)
        slots[i] = make_uint4(ones, ones, ones, ones);
}

int grid_build(gca3d_context *ctx, const Batch &b, float cell, int origin_mode, const float *host_origin,
               Grid &g)
{
    if (!(cell > 0.0f))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "grid cell must be > 0");
    if (origin_mode == kOriginGiven && (!host_origin || b.P != 1))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "grid: a given origin needs one segment");
    Arena &A = ctx->arena;
    const int P = b.P;
    const int64_t cap = std::max<int64_t>(b.cap, 1);
    uint32_t hcap = 1024;
    int table_bits = 10; // a direct table takes at most half the hash's memory: 8 bytes per entry
    while ((int64_t)hcap < 2 * cap)
    {
        hcap <<= 1;
        ++table_bits;
    }
    g.cap = cap;
    g.P = P;
    g.hcap = hcap;
    GridDev &d = g.dev;
    d.cell = cell;
    d.inv_cell = 1.0f / cell;
    d.gmin = A.get<float3>(P);
    d.layout = A.get<KeyLayout>(1);
    d.spos = A.get<float4>(cap);
    d.sidx = A.get<int32_t>(cap);
    d.sint = A.get<float>(cap);
    d.scz = A.get<int>(cap);
    d.skey = A.get<uint64_t>(cap);
    d.slots = A.get<RowSlot>(hcap);
    d.hmask = hcap - 1;
    d.seg_off = b.seg_off;
    d.d_n = b.seg_off + P;
    d.err = ctx->d_err;
    SortBuffers sb;
    sb.keys[0] = A.get<uint64_t>(cap);
    sb.keys[1] = A.get<uint64_t>(cap);
    sb.vals[0] = A.get<int32_t>(cap);
    sb.vals[1] = A.get<int32_t>(cap);
    sb.d_sel = A.get<int>(1);
    sb.d_ib = A.get<int>(1);
    sb.d_kshift = A.get<int>(1);
    if (!d.gmin || !d.layout || !d.spos || !d.sidx || !d.sint || !d.scz || !d.skey || !d.slots || !sb.keys[1] ||
        !sb.vals[1] || !sb.d_sel || !sb.d_ib || !sb.d_kshift)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "grid_build: scratch");
    cudaStream_t s = ctx->stream;
    const float3 given = host_origin ? make_float3(host_origin[0], host_origin[1], host_origin[2]) : make_float3(0, 0, 0);
    const GridMaker mk{b.pos, b.seg_off, b.d_count, cell, 1.0f / cell, origin_mode, given, table_bits};
    int st;
    if (cluster_sortable(ctx, P, cap))
        st = cluster_sort(ctx, mk, cap,
                          ClusterOut{sb.keys[0], sb.vals[0], sb.d_sel, sb.d_ib, sb.d_kshift, d.layout, d.gmin,
                                     ctx->d_err, nullptr, nullptr, nullptr, nullptr});
    else
        st = sort_by_keys(ctx, mk, sb, b.seg_off, P, cap, b.max_seg_cap, d.layout, d.gmin, 0, nullptr);
    if (st)
        return st;
    k_grid_clear<<<ctx->num_sms * 4, kBlock, 0, s>>>(d.layout, reinterpret_cast<uint4 *>(d.slots), hcap);
    GCA_CHECK_LAUNCH(ctx);
    GCA_PROF_BEGIN(ctx, kKidGridScatter);
    k_grid_scatter<<<std::min(grid_for(cap), ctx->num_sms * 8), kBlock, 0, s>>>(
        sb, b.seg_off + P, d.layout, b.pos, d.spos, d.sidx, d.sint, d.scz, P > 1 ? d.skey : nullptr, d.slots, d.hmask,
        ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    GCA_PROF_END(ctx, kKidGridScatter);
    return GCA3D_OK;
}

// ---------------------------------------------------------------------------
// queries against a single-segment grid
// ---------------------------------------------------------------------------
__global__ void k_nn_query(const float4 *__restrict__ q, const int32_t *d_nq, GridDev g, float radius, int32_t *out)
{
    const int nq = *d_nq;
    const KeyLayout L = *g.layout;
    const float3 o = g.gmin[0];
    const float rr = __fmul_rn(radius, radius);
    const int per_block = blockDim.x / kSub;
    for (int base = blockIdx.x * per_block; base < nq; base += gridDim.x * per_block)
    {
        const int i = base + (int)(threadIdx.x / kSub);
        const bool valid = i < nq;
        const float4 p = q[valid ? i : 0];
        const NNBest best = nn_search_sub(g, L, 0, o, make_float3(p.x, p.y, p.z), rr, valid);
        if (valid && (threadIdx.x & (kSub - 1)) == 0)
            out[i] = best.t >= 0 ? g.sidx[best.t] : -1;
    }
}

__global__ void k_radius_count(const float4 *__restrict__ q, const int32_t *d_nq, GridDev g, float radius,
                               int32_t *counts)
{
    const int nq = *d_nq;
    const KeyLayout L = *g.layout;
    const float3 o = g.gmin[0];
    const float rr = __fmul_rn(radius, radius);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x)
    {
        float4 p = q[i];
        int c = 0;
        grid_visit(g, L, 0, o, make_float3(p.x, p.y, p.z), [&](int t, float4 c4) {
            if (dist2_ref(c4.x, c4.y, c4.z, p.x, p.y, p.z) < rr)
                ++c;
        });
        counts[i] = c;
    }
}

__global__ void k_radius_fill(const float4 *__restrict__ q, const int32_t *d_nq, GridDev g, float radius,
                              const int32_t *starts, int32_t *list, int64_t cap, int *d_err)
{
    const int nq = *d_nq;
    const KeyLayout L = *g.layout;
    const float3 o = g.gmin[0];
    const float rr = __fmul_rn(radius, radius);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x)
    {
        float4 p = q[i];
        int64_t w = starts[i];
        grid_visit(g, L, 0, o, make_float3(p.x, p.y, p.z), [&](int t, float4 c4) {
            if (dist2_ref(c4.x, c4.y, c4.z, p.x, p.y, p.z) < rr)
            {
                if (w < cap)
                    list[w] = g.sidx[t];
                else
                    atomicOr(d_err, kErrCapacity);
                ++w;
            }
        });
    }
}

int nn_query(gca3d_context *ctx, const float4 *qpos, const int32_t *d_nq, int64_t qcap, const Grid &g, float radius,
             int32_t *out_idx)
{
    const int gs = std::min(grid_for(qcap, kBlock / kSub), ctx->num_sms * 16);
    k_nn_query<<<gs, kBlock, 0, ctx->stream>>>(qpos, d_nq, g.dev, radius, out_idx);
    GCA_CHECK_LAUNCH(ctx);
    return GCA3D_OK;
}

int radius_query(gca3d_context *ctx, const float4 *qpos, const int32_t *d_nq, int64_t qcap, const Grid &g,
                 float radius, int32_t *counts, int32_t *starts, int32_t *list, int64_t list_cap, int32_t *d_total)
{
    const int gs = std::min(grid_for(qcap), ctx->num_sms * 16);
    k_radius_count<<<gs, kBlock, 0, ctx->stream>>>(qpos, d_nq, g.dev, radius, counts);
    GCA_CHECK_LAUNCH(ctx);
    int st = exclusive_scan(ctx, counts, starts, d_nq, qcap, d_total);
    if (st)
        return st;
    k_radius_fill<<<gs, kBlock, 0, ctx->stream>>>(qpos, d_nq, g.dev, radius, starts, list, list_cap, ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    return GCA3D_OK;
}

} // namespace gca3d
