// voxel.cu -- batched voxel-grid downsampling.
//
// reference: cuda_voxel_grid_downsample (src/geometry/cuda_voxel_grid_down_sample.cu:123-161)
// and point_cloud::voxel_grid_down_sample (src/geometry/point_cloud.cu:198-229).
//
// Per segment (cloud) the key is floor((p - aabb_min) / v) per axis, as the
// reference computes it.  The three axis keys of every segment are packed, with the
// segment index above them, into one 64-bit key whose numeric order is the
// reference's lexicographic (kx, ky, kz) order; one stable radix sort then orders
// all segments at once.  A voxel's sum runs sequentially over its points in
// ascending original index (the sort is stable), so the downsampled set is
// bit-exact against the oracle; the mean is xyz / n and rgb * (1 / n) as in
// src/geometry/type.hpp:58-62.
#include "cluster_sort.cuh"
#include "stages.cuh"

#include <algorithm>

namespace gca3d
{

int batch_alloc(gca3d_context *ctx, Batch &b, int P, int64_t cap, int64_t max_seg_cap, bool nrm, bool grd)
{
    Arena &A = ctx->arena;
    b.P = P;
    b.cap = cap;
    b.max_seg_cap = max_seg_cap;
    int64_t c = std::max<int64_t>(cap, 1);
    b.pos = A.get<float4>(c);
    b.col = A.get<float4>(c);
    b.nrm = nrm ? A.get<float4>(c) : nullptr;
    b.grd = grd ? A.get<float4>(c) : nullptr;
    b.seg_off = A.get<int32_t>(P + 1);
    if (!b.pos || !b.col || (nrm && !b.nrm) || (grd && !b.grd) || !b.seg_off)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "batch_alloc: scratch");
    return GCA3D_OK;
}

// exclusive prefix of the segment sizes (one block)
__global__ void k_src_prefix(const SegSrc *src, int P, int32_t *off)
{
    __shared__ int32_t s_base;
    if (threadIdx.x == 0)
        s_base = 0;
    __syncthreads();
    for (int c0 = 0; c0 < P; c0 += blockDim.x)
    {
        int i = c0 + threadIdx.x;
        int v = i < P ? *src[i].d_n : 0;
        // block inclusive scan (Hillis-Steele over 256)
        __shared__ int32_t s[256];
        s[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < 256; o <<= 1)
        {
            int32_t y = threadIdx.x >= o ? s[threadIdx.x - o] : 0;
            __syncthreads();
            s[threadIdx.x] += y;
            __syncthreads();
        }
        if (i < P)
            off[i] = s_base + s[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 255)
            s_base += s[255];
        __syncthreads();
    }
    if (threadIdx.x == 0)
        off[P] = s_base;
}

// the bits of v (up to 21) at every third position (bit interleaving by masks)
__device__ __forceinline__ uint64_t spread3(uint64_t v)
{
    v &= 0x1fffffull;
    v = (v | (v << 32)) & 0x1f00000000ffffull;
    v = (v | (v << 16)) & 0x1f0000ff0000ffull;
    v = (v | (v << 8)) & 0x100f00f00f00f00full;
    v = (v | (v << 4)) & 0x10c30c30c30c30c3ull;
    v = (v | (v << 2)) & 0x1249249249249249ull;
    return v;
}

// the largest voxel key per axis of a set with bounds mn, mx (untouched when it is empty);
// error bits
__device__ __forceinline__ int voxel_extent(const float mn[3], const float mx[3], float voxel, uint32_t cells[3])
{
    if (!(mx[0] >= mn[0]))
        return 0;
    int err = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
    {
        int k = cell_of(mx[a], mn[a], voxel);
        if (k < 0 || k >= (1 << 21))
        {
            err = kErrKeyBits;
            k = (1 << 21) - 1;
        }
        cells[a] = (uint32_t)k;
    }
    return err;
}

// a point's voxel key with the sub-cell bits of the finer scales below it
__device__ __forceinline__ uint64_t voxel_key(float4 p, int seg, const KeyLayout &L, float3 o, float voxel,
                                              float inv, const SubLevels &sub, int *d_err)
{
    uint64_t kx = (uint32_t)cell_of_inv(p.x, o.x, voxel, inv), ky = (uint32_t)cell_of_inv(p.y, o.y, voxel, inv),
             kz = (uint32_t)cell_of_inv(p.z, o.z, voxel, inv);
    uint64_t key = ((uint64_t)seg << (L.bx + L.by + L.bz)) |
                   (L.morton ? (spread3(kx) << 2) | (spread3(ky) << 1) | spread3(kz)
                             : (kx << (L.by + L.bz)) | (ky << L.bz) | kz);
    // each finer scale's cells, as that scale computes them: with its voxel half the
    // previous one, its quotient is exactly twice the previous one, so each axis adds
    // one bit (x, y, z -- the next three bits of the finer Z-order key)
#pragma unroll
    for (int l = 0; l < kMaxSubLevels; ++l)
    {
        if (l >= sub.n)
            break;
        const float fv = sub.voxel[l], fi = sub.inv[l];
        const uint64_t fx = (uint32_t)cell_of_inv(p.x, o.x, fv, fi), fy = (uint32_t)cell_of_inv(p.y, o.y, fv, fi),
                       fz = (uint32_t)cell_of_inv(p.z, o.z, fv, fi);
        const uint64_t bx = fx - 2 * kx, by = fy - 2 * ky, bz = fz - 2 * kz;
        if ((bx | by | bz) > 1)
            atomicOr(d_err, kErrInvalid);
        key = (key << 3) | ((bx & 1) << 2) | ((by & 1) << 1) | (bz & 1);
        kx = fx, ky = fy, kz = fz;
    }
    return key;
}

// the voxel keys of P sets, read through the source table; a single source may come by value
// instead (begin then writes the table, which the reduction reads)
struct VoxelMaker
{
    SegSrc *table;
    SegSrc one;
    bool single, by_value;
    int32_t *in_off; // element ranges; written {0, n} by begin for a single source
    float voxel, inv;
    bool morton;
    SubLevels sub;
    __device__ int2 range(int seg) const
    {
        return single ? make_int2(0, by_value ? *one.d_n : *table->d_n) : make_int2(in_off[seg], in_off[seg + 1]);
    }
    __device__ float4 point(int seg, int i) const
    {
        return single ? __ldg((by_value ? one.pos : table->pos) + i) : __ldg(table[seg].pos + (i - in_off[seg]));
    }
    __device__ int sub_bits() const { return 3 * sub.n; }
    __device__ void begin(int n) const
    {
        in_off[0] = 0;
        in_off[1] = n;
        if (by_value)
            *table = one;
    }
    // the origin is the unpadded aabb min
    __device__ int segment(const float mn[3], const float mx[3], float3 &o, uint32_t cells[3]) const
    {
        o = make_float3(mn[0], mn[1], mn[2]);
        return voxel_extent(mn, mx, voxel, cells);
    }
    // With morton (and room in 64 bits) the three axis keys are bit-interleaved below the
    // segment index: the voxels then come out in Z-order, so runs of consecutive output
    // points are compact in space (the correspondence search of the ICP stages a block's
    // target cells once for such a run).
    __device__ int layout(const uint32_t cells[3], int P, KeyLayout &L) const
    {
        const int sub_bits = 3 * sub.n;
        L.bseg = bitlen_u32((uint32_t)(P - 1));
        L.bx = max(1, bitlen_u32(cells[0]));
        L.by = max(1, bitlen_u32(cells[1]));
        L.bz = max(1, bitlen_u32(cells[2]));
        L.total_bits = L.bseg + L.bx + L.by + L.bz;
        L.morton = L.direct = L.zs = 0;
        const int b = max(L.bx, max(L.by, L.bz));
        if (morton && L.bseg + 3 * b + sub_bits <= 64)
        {
            L.bx = L.by = L.bz = b;
            L.total_bits = L.bseg + 3 * b;
            L.morton = 1;
        }
        // sub-cell bits for finer scales ride below a Z-order key
        return L.total_bits + sub_bits > 64 || (sub_bits && !L.morton) ? kErrKeyBits : 0;
    }
    __device__ uint64_t key(float4 p, int seg, const KeyLayout &L, float3 o, int *d_err) const
    {
        return voxel_key(p, seg, L, o, voxel, inv, sub, d_err);
    }
};

bool voxel_cluster_enable() { return cluster_sort_enable<VoxelMaker>(); }

// segment offsets of the output; empty segments start where the next one does
__global__ void k_seg_first_to_offsets(const int32_t *seg_first, int P, const int32_t *d_m, int32_t *off)
{
    if (threadIdx.x != 0)
        return;
    int32_t next = *d_m;
    off[P] = next;
    for (int s = P - 1; s >= 0; --s)
    {
        if (seg_first[s] >= 0)
            next = seg_first[s];
        off[s] = next;
    }
}

__global__ void k_voxel_reduce(const SegSrc *src, const int32_t *in_off, SortBuffers sb, const int32_t *starts,
                               const int32_t *d_m, const KeyLayout *lay, float4 *opos, float4 *ocol, int *err)
{
    const int m = *d_m;
    const SortedView sv = sorted_view(sb);
    const KeyLayout L = *lay;
    const int segshift = L.bx + L.by + L.bz;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x)
    {
        const int s = starts[v], e = starts[v + 1];
        const int seg = L.bseg ? (int)(sv.key(s) >> segshift) : 0;
        const int base = in_off[seg];
        const float4 *ps = src[seg].pos;
        const float4 *cs = src[seg].col;
        int g = sv.val(s) - base;
        if (!GCA_INDEX_OK(g, in_off[seg + 1] - base, err))
            continue;
        float4 p = ps[g], c = cs[g];
        float sx = p.x, sy = p.y, sz = p.z, cr = c.x, cg = c.y, cb = c.z;
        // one thread adds up a voxel in order, so a large one is a chain of loads that do not
        // depend on the sums.  300k points in 1 / 29 / 3388 voxels: unrolled by the compiler's
        // choice 48,270 / 6930 / 217 us, by eight 37,060 / 5400 / 196, by sixteen 36,950 / 5440 /
        // 205, four points' loads in an array first 42,190 / 8300 / 229; with a few points to a
        // voxel all alike.
#pragma unroll 8
        for (int j = s + 1; j < e; ++j)
        {
            g = sv.val(j) - base;
            if (!GCA_INDEX_OK(g, in_off[seg + 1] - base, err))
                break;
            p = ps[g];
            c = cs[g];
            sx = __fadd_rn(sx, p.x);
            sy = __fadd_rn(sy, p.y);
            sz = __fadd_rn(sz, p.z);
            cr = __fadd_rn(cr, c.x);
            cg = __fadd_rn(cg, c.y);
            cb = __fadd_rn(cb, c.z);
        }
        const float fn = (float)(e - s);
        const float inv = __fdiv_rn(1.0f, fn);
        const float r = __fmul_rn(cr, inv), gg = __fmul_rn(cg, inv), b = __fmul_rn(cb, inv);
        opos[v] = make_float4(__fdiv_rn(sx, fn), __fdiv_rn(sy, fn), __fdiv_rn(sz, fn), intensity_of(r, gg, b));
        ocol[v] = make_float4(r, gg, b, 0.0f);
    }
}

// One finer scale from the previous one's sorted order: within each previous voxel's run
// the elements are split, stably, by the next three sub-cell bits below the key, which
// orders them by (finer key, index) -- what a full sort by the finer key gives.  One
// thread per previous voxel (a handful of points each); the output goes to the other
// buffer, and the finer scale's view and layout are written beside the previous ones.
__global__ void k_voxel_refine(SortBuffers sb, const int32_t *starts, const int32_t *d_m, const KeyLayout *lay_in,
                               int *d_sel_out, int *d_kshift_out, KeyLayout *lay_out)
{
    const int sel = *sb.d_sel;
    const int ks = *sb.d_kshift - 3; // the finer key's lowest bit
    const bool packed = *sb.d_ib != 0;
    const uint64_t *kin = sb.keys[sel];
    uint64_t *kout = sb.keys[sel ^ 1];
    const int32_t *vin = sb.vals[sel];
    int32_t *vout = sb.vals[sel ^ 1];
    if (blockIdx.x == 0 && threadIdx.x == 0)
    {
        *d_sel_out = sel ^ 1;
        *d_kshift_out = ks;
        KeyLayout L = *lay_in;
        L.bx += 1, L.by += 1, L.bz += 1;
        L.total_bits += 3;
        *lay_out = L;
    }
    const int m = *d_m;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x)
    {
        const int s = starts[v], e = starts[v + 1];
        if (e - s < 256)
        {
            // a run of fewer than 256 keys: the eight sub-cell counts are the bytes of one
            // register, and one multiplication by 0x0101..01 gives their running sums
            // (byte b of the product: the keys of sub-cells 0..b; shifted one byte up: the
            // keys of the sub-cells below b), all below 256, so no byte carries
            uint64_t c = 0;
            for (int j = s; j < e; ++j)
                c += 1ull << (8 * (int)((kin[j] >> ks) & 7));
            uint64_t at = (c * 0x0101010101010101ull) << 8;
            for (int j = s; j < e; ++j)
            {
                const uint64_t w = kin[j];
                const int sh = 8 * (int)((w >> ks) & 7);
                const int o = s + (int)((at >> sh) & 255u);
                at += 1ull << sh;
                kout[o] = w;
                if (!packed)
                    vout[o] = vin[j];
            }
            continue;
        }
        int off[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int j = s; j < e; ++j)
            ++off[(kin[j] >> ks) & 7];
        int run = s;
#pragma unroll
        for (int b = 0; b < 8; ++b)
        {
            const int c = off[b];
            off[b] = run;
            run += c;
        }
        for (int j = s; j < e; ++j)
        {
            const uint64_t w = kin[j];
            const int o = off[(w >> ks) & 7]++;
            kout[o] = w;
            if (!packed)
                vout[o] = vin[j];
        }
    }
}

// the sums of the voxels whose runs are known
static int voxel_sums(gca3d_context *ctx, const SegSrc *d_src, int64_t total_cap, const int32_t *in_off,
                      const SortBuffers &sb, const KeyLayout *lay, Batch &out, const int32_t *starts, const int32_t *d_m)
{
    const int gs = std::min(grid_for(total_cap), ctx->num_sms * 8);
    GCA_PROF_BEGIN(ctx, kKidVoxelReduce);
    k_voxel_reduce<<<gs, kBlock, 0, ctx->stream>>>(d_src, in_off, sb, starts, d_m, lay, out.pos, out.col, ctx->d_err);
    GCA_CHECK_LAUNCH(ctx);
    GCA_PROF_END(ctx, kKidVoxelReduce);
    return GCA3D_OK;
}

// the runs of equal keys (voxels) of the sorted view and their sums: the part of a voxel
// stage after its order is known
static int voxel_reduce_stage(gca3d_context *ctx, const SegSrc *d_src, int P, int64_t total_cap,
                              const int32_t *in_off, const SortBuffers &sb, const KeyLayout *lay, Batch &out,
                              int32_t *starts, int32_t *d_m, int32_t *d_count = nullptr, void *zeroed = nullptr)
{
    Arena &A = ctx->arena;
    const int64_t cap = std::max<int64_t>(total_cap, 1);
    const int32_t *d_n = in_off + P;
    int st;
    if (P == 1) // the scan writes the one segment's offsets itself
    {
        if ((st = run_scan(ctx, sb, d_n, cap, lay, starts, nullptr, d_m, out.seg_off, d_count, zeroed)))
            return st;
        return voxel_sums(ctx, d_src, total_cap, in_off, sb, lay, out, starts, d_m);
    }
    int32_t *seg_count = A.get<int32_t>(P);
    if (!seg_count)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "voxel_stage: scratch");
    cudaStream_t s = ctx->stream;
    GCA_CUDA(ctx, cudaMemsetAsync(seg_count, 0xFF, sizeof(int32_t) * P, s));
    if ((st = run_scan(ctx, sb, d_n, cap, lay, starts, seg_count, d_m, nullptr, nullptr, zeroed)))
        return st;
    if ((st = voxel_sums(ctx, d_src, total_cap, in_off, sb, lay, out, starts, d_m)))
        return st;
    k_seg_first_to_offsets<<<1, 32, 0, s>>>(seg_count, P, d_m, out.seg_off);
    GCA_CHECK_LAUNCH(ctx);
    return GCA3D_OK;
}

int voxel_refine(gca3d_context *ctx, const SegSrc *d_src, VoxelChain &c, Batch &out)
{
    if (c.used >= c.levels)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "voxel_refine: no finer scale carried");
    Arena &A = ctx->arena;
    const int64_t cap = std::max<int64_t>(c.total_cap, 1);
    SortBuffers sb = c.sb;
    sb.d_sel = A.get<int>(1);
    sb.d_kshift = A.get<int>(1);
    KeyLayout *lay = A.get<KeyLayout>(1);
    int32_t *starts = A.get<int32_t>(cap + 1);
    int32_t *d_m = A.get<int32_t>(1);
    if (!sb.d_sel || !sb.d_kshift || !lay || !starts || !d_m)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "voxel_refine: scratch");
    if (!out.pos)
    {
        int st = batch_alloc(ctx, out, c.P, c.total_cap, c.max_seg_cap, false, false);
        if (st)
            return st;
    }
    const int gs = std::min(grid_for(c.total_cap), ctx->num_sms * 8);
    k_voxel_refine<<<gs, kBlock, 0, ctx->stream>>>(c.sb, c.starts, c.d_m, c.lay, sb.d_sel, sb.d_kshift, lay);
    GCA_CHECK_LAUNCH(ctx);
    int st = voxel_reduce_stage(ctx, d_src, c.P, c.total_cap, c.in_off, sb, lay, out, starts, d_m);
    if (st)
        return st;
    c.sb = sb;
    c.lay = lay;
    c.starts = starts;
    c.d_m = d_m;
    c.used += 1;
    return GCA3D_OK;
}

int voxel_stage(gca3d_context *ctx, SegSrc *d_src, int P, int64_t total_cap, int64_t max_seg_cap,
                float voxel, Batch &out, bool morton, const SubLevels *finer, VoxelChain *chain, const SegSrc *one,
                int32_t *d_count)
{
    if (!(voxel > 0.0f))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "voxel size must be > 0");
    Arena &A = ctx->arena;
    const int64_t cap = std::max<int64_t>(total_cap, 1);
    int32_t *in_off = A.get<int32_t>(P + 1);
    float3 *origin = A.get<float3>(P);
    KeyLayout *lay = A.get<KeyLayout>(1);
    SortBuffers sb;
    sb.keys[0] = A.get<uint64_t>(cap);
    sb.keys[1] = A.get<uint64_t>(cap);
    sb.vals[0] = A.get<int32_t>(cap);
    sb.vals[1] = A.get<int32_t>(cap);
    sb.d_sel = A.get<int>(1);
    sb.d_ib = A.get<int>(1);
    sb.d_kshift = A.get<int>(1);
    int32_t *starts = A.get<int32_t>(cap + 1);
    int32_t *d_m = A.get<int32_t>(1);
    if (!in_off || !origin || !lay || !sb.keys[1] || !sb.vals[1] || !sb.d_sel || !sb.d_ib || !sb.d_kshift ||
        !starts || !d_m)
        return fail(ctx, GCA3D_ERR_OUT_OF_MEMORY, "voxel_stage: scratch");
    const SubLevels sub = finer ? *finer : SubLevels{};
    if (sub.n < 0 || sub.n > kMaxSubLevels || (sub.n && !morton))
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "voxel_stage: finer scales need Z-order keys");
    if (!out.pos)
    {
        int st = batch_alloc(ctx, out, P, total_cap, max_seg_cap, false, false);
        if (st)
            return st;
    }
    const VoxelMaker mk{d_src, one ? *one : SegSrc{}, P == 1, one != nullptr, in_off, voxel, 1.0f / voxel, morton, sub};
    int st;
    if (cluster_sortable(ctx, P, cap))
    {
        const ClusterOut co{sb.keys[0], sb.vals[0], sb.d_sel,     sb.d_ib,     sb.d_kshift, lay,
                            origin,     ctx->d_err, starts,       d_m,         out.seg_off, d_count};
        if ((st = cluster_sort(ctx, mk, cap, co)) ||
            (st = voxel_sums(ctx, d_src, total_cap, in_off, sb, lay, out, starts, d_m)))
            return st;
    }
    else
    {
        if (P > 1)
        {
            k_src_prefix<<<1, 256, 0, ctx->stream>>>(d_src, P, in_off);
            GCA_CHECK_LAUNCH(ctx);
        }
        void *zeroed = nullptr;
        if ((st = sort_by_keys(ctx, mk, sb, in_off, P, cap, max_seg_cap, lay, origin, run_scan_zero_bytes(cap), &zeroed)) ||
            (st = voxel_reduce_stage(ctx, d_src, P, total_cap, in_off, sb, lay, out, starts, d_m, d_count, zeroed)))
            return st;
    }
    if (chain)
    {
        chain->sb = sb;
        chain->in_off = in_off;
        chain->starts = starts;
        chain->d_m = d_m;
        chain->lay = lay;
        chain->levels = sub.n;
        chain->used = 0;
        chain->P = P;
        chain->total_cap = total_cap;
        chain->max_seg_cap = max_seg_cap;
    }
    return GCA3D_OK;
}

// copy segments into a contiguous batch (no downsampling)
__global__ void k_gather(const SegSrc *src, const int32_t *off, float4 *pos, float4 *col, float4 *nrm)
{
    const int seg = blockIdx.y;
    const int n = *src[seg].d_n;
    const int base = off[seg];
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    {
        pos[base + i] = src[seg].pos[i];
        col[base + i] = src[seg].col[i];
        if (nrm)
            nrm[base + i] = src[seg].nrm ? src[seg].nrm[i] : make_float4(0, 0, 0, 0);
    }
}

int gather_stage(gca3d_context *ctx, const SegSrc *d_src, int P, int64_t max_seg_cap, Batch &out,
                 bool with_normals)
{
    if (with_normals && !out.nrm)
        return fail(ctx, GCA3D_ERR_INVALID_VALUE, "gather_stage: batch has no normal storage");
    k_src_prefix<<<1, 256, 0, ctx->stream>>>(d_src, P, out.seg_off);
    GCA_CHECK_LAUNCH(ctx);
    const int gx = std::min(grid_for(max_seg_cap, kBlock * 4), ctx->num_sms * 4);
    k_gather<<<dim3(gx, P), kBlock, 0, ctx->stream>>>(d_src, out.seg_off, out.pos, out.col,
                                                     with_normals ? out.nrm : nullptr);
    GCA_CHECK_LAUNCH(ctx);
    return GCA3D_OK;
}

} // namespace gca3d
