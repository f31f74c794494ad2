// cluster_sort.cuh -- bounds, keys and stable radix sort of one point set in one launch.
//
// A set in a buffer of at most kClusterCap points (the host knows its capacity, not its count)
// fits in the shared memory of one cluster of 16 thread
// blocks (16 SMs), so its whole sort runs there: every block holds a sixteenth of the words,
// a pass ranks them warp by warp (one ballot per digit bit), the blocks exchange their digit
// counts, and every word goes straight to its place in its destination block through
// distributed shared memory.  Blocks meet at the cluster's hardware barrier; nothing polls.  No
// block touches another's shared memory before the barrier that all have started by, nor after
// the last one.
//
// What bounds the alternative (sort_keys.cuh, sort_scan.cu) at these sizes is latency: ten
// launches, half of them passes with nothing to do, and in a pass a chain of a dozen
// dependent memory accesses.  Here a pass of 8 bits takes 2 us plus 1 us per 1024 words of a
// block, about half of it ranking.  Measured (GB300, whole calls, this against the launches):
// voxel stage at 20k points 62 / 111 us, alignment of 64k 301 / 345, outlier removal at 180k
// 136 / 157, nearest neighbours in 200k 172 / 183, normals of 206k 203 / 217.  The line is
// drawn at 13 words per thread, 213k points: with 16 (256k, what the shared memory holds) a
// voxel stage at 256k took 143 / 134, a 250k pair 883 / 870, and the extra registers cost the
// 64k alignment 3 %, against 152 / 158 for neighbours in 256k.  Larger sets, and batches of
// several, have tiles enough to fill the
// GPU, of which a cluster is a tenth.
#pragma once

#include "sort_keys.cuh"

#include <cooperative_groups.h>
#include <utility>

namespace gca3d
{

constexpr int kClusterBlocks = 16;
constexpr int kClusterThreads = 1024;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterRounds = 13; // words per thread: 26 registers of the 64 there are, which spill a little
                                   // (ptxas: 124 bytes stored for grids, 144 for voxels)
constexpr int kClusterWordBits = 54; // of a word; a pass keeps its rank within the warp above them
constexpr int64_t kClusterCap = (int64_t)kClusterBlocks * kClusterThreads * kClusterRounds; // 212,992
constexpr int kClusterDigit = 10; // bits of the widest digit: 20 bits of key take two passes, 30 three
constexpr int kClusterBins = 1 << kClusterDigit;
static_assert(kClusterThreads * kClusterRounds < 65536 && kClusterBins <= kClusterThreads,
              "16-bit counts, a thread per bin");

// shared memory of a block: its words, its warps' digit counts and every block's digit
// counts (16 bits each)
inline size_t cluster_smem(int64_t cap)
{
    const size_t words = (size_t)((cap + kClusterBlocks - 1) / kClusterBlocks);
    return words * sizeof(uint64_t) + sizeof(uint16_t) * kClusterWarps * kClusterBins +
           sizeof(uint16_t) * kClusterBlocks * kClusterBins;
}

// where a cluster sort leaves its results; d_starts .. d_count may be null (no runs wanted)
struct ClusterOut
{
    uint64_t *keys; // SortBuffers' first arrays
    int32_t *vals;
    int *d_sel, *d_ib, *d_kshift;
    KeyLayout *layout;
    float3 *origin;
    int *d_err;
    // the runs of equal keys, as run_scan gives them, and the run count as a one-segment
    // offset table and as a cloud's count
    int32_t *d_starts, *d_runs, *seg_off, *d_count;
};

// the lanes among `in` whose low Width bits of d agree with this lane's
template <int Width> __device__ __forceinline__ unsigned cluster_peers(uint32_t d, unsigned in)
{
#pragma unroll
    for (int b = 0; b < Width; ++b)
    {
        const bool bit = (d >> b) & 1u;
        const unsigned v = __ballot_sync(0xffffffffu, bit);
        in &= bit ? v : ~v;
    }
    return in;
}

// a warp's words ranked by their digit (mask, at most Width bits, from lo): the rank among the warp's
// earlier words of that digit goes above each word, the digit's count into hist
template <int Width>
__device__ __forceinline__ void cluster_rank(uint64_t *words, uint16_t *hist, int e0, int cnt, int rounds, int lo,
                                             uint32_t mask)
{
    const int lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu, lt_mask = (1u << lane) - 1u;
#pragma unroll 1
    for (int it = 0; it < rounds; ++it)
    {
        const int e = e0 + 32 * it;
        const bool in = e < cnt;
        const uint64_t w = in ? words[e] : 0ull;
        const uint32_t d = (uint32_t)(w >> lo) & mask;
        const unsigned peers = cluster_peers<Width>(d, __ballot_sync(full, in));
        const uint32_t c = hist[d], r = c + __popc(peers & lt_mask);
        __syncwarp();
        if (in)
        {
            if ((peers & lt_mask) == 0u)
                hist[d] = (uint16_t)(c + __popc(peers));
            words[e] = w | (uint64_t)r << kClusterWordBits;
        }
        __syncwarp();
    }
}

// exclusive prefix over the block's threads (s_scan: a word per warp); every thread calls it
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *s_scan)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d)
            x += y;
    }
    if (lane == 31)
        s_scan[warp] = x;
    __syncthreads();
    uint32_t t = lane < warp ? s_scan[lane] : 0u;
    t = __reduce_add_sync(0xffffffffu, t);
    __syncthreads(); // s_scan may be written again
    return t + x - v;
}

// Maker: as in sort_keys.cuh, one set
template <class Maker>
__global__ void __launch_bounds__(kClusterThreads, 1) k_cluster_sort(Maker mk, ClusterOut o, int index_bits, int words)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // another block's shared memory may be accessed once that block has started: every block
    // arrives here and waits before its first remote write, behind its reading of the points
    auto started = cluster.barrier_arrive();
    extern __shared__ uint64_t s_words[];
    uint16_t *s_whist = reinterpret_cast<uint16_t *>(s_words + words); // [warp][bin]
    uint16_t *s_count = s_whist + kClusterWarps * kClusterBins; // [block][bin]
    __shared__ float s_bound[kClusterBlocks][6];
    __shared__ float s_red[kClusterWarps][6];
    __shared__ uint32_t s_scan[kClusterWarps];
    __shared__ uint32_t s_base[kClusterBins];
    __shared__ uint32_t s_runs[kClusterBlocks];
    __shared__ KeyLayout s_layout;
    __shared__ float3 s_origin;
    const int rank = (int)cluster.block_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned full = 0xffffffffu, lt_mask = (1u << lane) - 1u;
    const int n = mk.range(0).y;
    // block r holds the words [r chunk, r chunk + cnt); warp w of it the elements from
    // w * 32 * rounds on, 32 per round, so that element order is warp, round, lane
    const int chunk = (n + kClusterBlocks - 1) / kClusterBlocks;
    const int first = rank * chunk, cnt = max(0, min(chunk, n - first));
    const int rounds = (chunk + kClusterThreads - 1) / kClusterThreads;
    const int e0 = warp * 32 * rounds + lane;

    // bounds (exact, so the order of the minima does not matter)
    {
        float v[6] = {3.402823466e38f, 3.402823466e38f, 3.402823466e38f, 3.402823466e38f, 3.402823466e38f, 3.402823466e38f};
#pragma unroll 4
        for (int e = tid; e < cnt; e += kClusterThreads)
        {
            const float4 p = mk.point(0, first + e);
            v[0] = fminf(v[0], p.x), v[1] = fminf(v[1], p.y), v[2] = fminf(v[2], p.z);
            v[3] = fminf(v[3], -p.x), v[4] = fminf(v[4], -p.y), v[5] = fminf(v[5], -p.z);
        }
#pragma unroll
        for (int a = 0; a < 6; ++a)
        {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1)
                v[a] = fminf(v[a], __shfl_xor_sync(full, v[a], d));
            if (lane == 0)
                s_red[warp][a] = v[a];
        }
        __syncthreads();
        cluster.barrier_wait(std::move(started)); // every block has started
        if (tid < 6)
        {
            float m = s_red[0][tid];
            for (int w = 1; w < kClusterWarps; ++w)
                m = fminf(m, s_red[w][tid]);
            for (int b = 0; b < kClusterBlocks; ++b)
                *cluster.map_shared_rank(&s_bound[rank][tid], b) = m;
        }
        cluster.sync();
        if (tid < 6)
        {
            float m = s_bound[0][tid];
            for (int b = 1; b < kClusterBlocks; ++b)
                m = fminf(m, s_bound[b][tid]);
            s_red[0][tid] = m;
        }
        __syncthreads();
        if (tid == 0)
        {
            const float mn[3] = {s_red[0][0], s_red[0][1], s_red[0][2]};
            const float mx[3] = {-s_red[0][3], -s_red[0][4], -s_red[0][5]};
            uint32_t cells[3] = {0u, 0u, 0u};
            int err = mk.segment(mn, mx, s_origin, cells);
            err |= mk.layout(cells, 1, s_layout);
            if (rank == 0 && err)
                atomicOr(o.d_err, err);
        }
        __syncthreads();
    }
    const KeyLayout L = s_layout;
    const float3 origin = s_origin;
    const int sub = mk.sub_bits();
    // packed words (key << ib | index) when they fit; otherwise the key's low and high bits
    // are sorted one after the other, each part above the index, and the keys written out
    const int ib = index_bits;
    const bool packed = L.total_bits + sub + ib <= kClusterWordBits;
    constexpr uint64_t word_mask = (1ull << kClusterWordBits) - 1ull;
    const uint64_t index_mask = (1ull << ib) - 1ull;
    const int low_bits = packed ? L.total_bits : min(L.total_bits, kClusterWordBits - ib);

    // four points' loads in flight per thread
    for (int it = 0; it < rounds; it += 4)
    {
        float4 p[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            p[j] = mk.point(0, min(first + e0 + 32 * (it + j), n - 1)); // n > 0: there are rounds
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const int e = e0 + 32 * (it + j);
            if (it + j < rounds && e < cnt)
            {
                const uint64_t k = mk.key(p[j], 0, L, origin, o.d_err);
                s_words[e] = (((packed ? k : k >> sub) << ib) | (uint64_t)(uint32_t)(first + e)) & word_mask;
            }
        }
    }
    const uint64_t chunk_inv = chunk > 0 ? (1ull << 40) / (uint64_t)chunk + 1ull : 0ull; // p / chunk, p < 2^19

    for (int part = 0; part < (L.total_bits > low_bits ? 2 : 1); ++part)
    {
        if (part == 1)
        {
            for (int e = tid; e < cnt; e += kClusterThreads)
            {
                const uint64_t i = s_words[e] & index_mask;
                if (!GCA_INDEX_OK(i, n, o.d_err))
                    continue;
                const uint64_t k = mk.key(mk.point(0, (int)i), 0, L, origin, o.d_err);
                s_words[e] = ((((k >> sub) >> low_bits) << ib) | i) & word_mask;
            }
            __syncthreads();
        }
        // stable sort by the bits [lo, hi) of the words
        int lo = packed ? ib + sub : ib;
        const int hi = lo + (part == 0 ? low_bits : L.total_bits - low_bits);
        const int passes = (hi - lo + kClusterDigit - 1) / kClusterDigit;
        const int step = passes ? (hi - lo + passes - 1) / passes : 1;
#pragma unroll 1
        for (; lo < hi; lo += step)
        {
            const int width = min(step, hi - lo), bins = 1 << width;
            const uint32_t mask = (uint32_t)bins - 1u;
            uint16_t *hist = s_whist + warp * bins;
            for (int i = tid; i < kClusterWarps * bins / 2; i += kClusterThreads)
                reinterpret_cast<uint32_t *>(s_whist)[i] = 0u;
            __syncthreads();
            if (width == 10)
                cluster_rank<10>(s_words, hist, e0, cnt, rounds, lo, mask);
            else if (width == 9)
                cluster_rank<9>(s_words, hist, e0, cnt, rounds, lo, mask);
            else if (width == 8)
                cluster_rank<8>(s_words, hist, e0, cnt, rounds, lo, mask);
            else
                cluster_rank<7>(s_words, hist, e0, cnt, rounds, lo, mask);
            __syncthreads();
            // the block's counts, to every block, and where each digit starts in this one
            uint32_t mine = 0;
            if (tid < bins)
            {
#pragma unroll 8
                for (int w = 0; w < kClusterWarps; ++w)
                {
                    const uint32_t c = s_whist[w * bins + tid];
                    s_whist[w * bins + tid] = (uint16_t)mine;
                    mine += c;
                }
                uint16_t *slot = s_count + rank * kClusterBins + tid;
                for (int b = 0; b < kClusterBlocks; ++b)
                    *cluster.map_shared_rank(slot, b) = (uint16_t)mine;
            }
            const uint32_t local = block_exclusive(mine, s_scan);
            if (tid < bins)
                s_base[tid] = local;
            uint64_t k[kClusterRounds];
#pragma unroll
            for (int it = 0; it < kClusterRounds; ++it)
                k[it] = it < rounds && e0 + 32 * it < cnt ? s_words[e0 + 32 * it] : 0ull;
            __syncthreads();
            // into digit order within the block first: then a warp's words go to consecutive
            // places of the other blocks (one by one, 300k words took 14.5 us a pass, so 12)
#pragma unroll
            for (int it = 0; it < kClusterRounds; ++it)
                if (it < rounds && e0 + 32 * it < cnt)
                {
                    const uint32_t d = (uint32_t)(k[it] >> lo) & mask;
                    const uint32_t at = s_base[d] + hist[d] + (uint32_t)(k[it] >> kClusterWordBits);
                    if (GCA_INDEX_OK(at, cnt, o.d_err))
                        s_words[at] = k[it] & word_mask;
                }
            __syncthreads();
#pragma unroll
            for (int it = 0; it < kClusterRounds; ++it)
                k[it] = it < rounds && e0 + 32 * it < cnt ? s_words[e0 + 32 * it] : 0ull;
            cluster.sync(); // the counts are here, and every block's words are in registers
            uint32_t tot = 0, before = 0;
            if (tid < bins)
                for (int b = 0; b < kClusterBlocks; ++b)
                {
                    const uint32_t c = s_count[b * kClusterBins + tid];
                    before += b < rank ? c : 0u;
                    tot += c;
                }
            const uint32_t global = block_exclusive(tot, s_scan);
            if (tid < bins)
                s_base[tid] = global + before - local; // of the digit's first word here, less its place
            __syncthreads();
#pragma unroll
            for (int it = 0; it < kClusterRounds; ++it)
                if (it < rounds && e0 + 32 * it < cnt)
                {
                    const uint32_t at = s_base[(uint32_t)(k[it] >> lo) & mask] + (uint32_t)(e0 + 32 * it);
                    const uint32_t to = (uint32_t)(((uint64_t)at * chunk_inv) >> 40);
                    // (at < n: then to < 16 and the place in that block is below chunk)
                    if (GCA_INDEX_OK(at, n, o.d_err))
                        cluster.map_shared_rank(s_words, to)[at - to * (uint32_t)chunk] = k[it];
                }
            cluster.sync();
        }
    }
    if (!packed)
        for (int e = tid; e < cnt; e += kClusterThreads)
        {
            const int i = (int)(s_words[e] & index_mask);
            o.vals[first + e] = i;
            if (!GCA_INDEX_OK(i, n, o.d_err))
                continue;
            s_words[e] = mk.key(mk.point(0, i), 0, L, origin, o.d_err);
        }
    __syncthreads();
    for (int e = tid; e < cnt; e += kClusterThreads)
        o.keys[first + e] = s_words[e];
    const int kshift = packed ? ib + sub : sub;
    if (rank == 0 && tid == 0)
    {
        mk.begin(n);
        *o.d_sel = 0;
        *o.d_ib = packed ? ib : 0;
        *o.d_kshift = kshift;
        *o.layout = L;
        o.origin[0] = origin;
    }
    if (!o.d_starts)
        return;
    // run starts: counted per warp, then the blocks' totals exchanged
    cluster.sync(); // every block's words are final (the first word of a block looks at the block before)
    auto starts_run = [&](int e) {
        if (e >= cnt)
            return false;
        if (first + e == 0)
            return true;
        const uint64_t before = e > 0 ? s_words[e - 1] : cluster.map_shared_rank(s_words, rank - 1)[chunk - 1];
        return (before >> kshift) != (s_words[e] >> kshift);
    };
    uint32_t mine = 0, flags = 0; // flags: this thread's run starts, one bit per round
    for (int it = 0; it < rounds; ++it)
    {
        const bool st = starts_run(e0 + 32 * it);
        flags |= (uint32_t)st << it;
        mine += __popc(__ballot_sync(full, st));
    }
    if (lane == 0)
        s_scan[warp] = mine;
    __syncthreads();
    uint32_t run = 0, block_runs = 0;
    for (int w = 0; w < kClusterWarps; ++w)
    {
        const uint32_t c = s_scan[w];
        run += w < warp ? c : 0u;
        block_runs += c;
    }
    if (tid < kClusterBlocks)
        *cluster.map_shared_rank(&s_runs[rank], tid) = block_runs;
    cluster.sync();
    uint32_t total = 0;
    for (int b = 0; b < kClusterBlocks; ++b)
    {
        const uint32_t c = s_runs[b];
        run += b < rank ? c : 0u;
        total += c;
    }
    for (int it = 0; it < rounds; ++it)
    {
        const bool st = (flags >> it) & 1u;
        const unsigned m = __ballot_sync(full, st);
        const uint32_t at = run + __popc(m & lt_mask);
        if (st && GCA_INDEX_OK(at, n, o.d_err))
            o.d_starts[at] = first + e0 + 32 * it;
        run += __popc(m);
    }
    if (rank == 0 && tid == 0)
    {
        o.d_starts[total] = n;
        *o.d_runs = (int32_t)total;
        if (o.seg_off)
        {
            o.seg_off[0] = 0;
            o.seg_off[1] = (int32_t)total;
        }
        if (o.d_count)
            *o.d_count = (int32_t)total;
    }
    cluster.sync(); // no block leaves while another may read its words
}

// whether a stage of P sets of at most cap points in all takes the cluster sort
inline bool cluster_sortable(const gca3d_context *ctx, int P, int64_t cap)
{
    return ctx->cluster_sort && P == 1 && cap <= kClusterCap;
}

template <class Maker> int cluster_sort(gca3d_context *ctx, const Maker &mk, int64_t cap, const ClusterOut &o)
{
    const int words = (int)((cap + kClusterBlocks - 1) / kClusterBlocks);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClusterBlocks);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = cluster_smem(cap);
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterBlocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    GCA_PROF_BEGIN(ctx, kKidSortPass);
    GCA_CUDA(ctx, cudaLaunchKernelEx(&cfg, k_cluster_sort<Maker>, mk, o, index_bits(cap), words));
    GCA_CHECK_LAUNCH(ctx);
    GCA_PROF_END(ctx, kKidSortPass);
    return GCA3D_OK;
}

// lets a maker's kernel run with a cluster of 16 and the shared memory it needs on the
// current device; false where the device does not take it
template <class Maker> bool cluster_sort_enable()
{
    const auto kernel = k_cluster_sort<Maker>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cluster_smem(kClusterCap)) !=
            cudaSuccess)
    {
        cudaGetLastError();
        return false;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kClusterBlocks);
    cfg.blockDim = dim3(kClusterThreads);
    cfg.dynamicSmemBytes = cluster_smem(kClusterCap);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kClusterBlocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess)
    {
        cudaGetLastError();
        return false;
    }
    return clusters > 0;
}
bool grid_cluster_enable();
bool voxel_cluster_enable();

} // namespace gca3d
