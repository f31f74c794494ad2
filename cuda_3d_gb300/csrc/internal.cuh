// internal.cuh -- shared types and device helpers of the gca3d library.
#pragma once

#include "gca3d.h"

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <utility>
#include <vector>

namespace gca3d
{

// ---------------------------------------------------------------------------
// limits
// ---------------------------------------------------------------------------
constexpr int kMaxSegments = 4096;       // pairs / clouds in one batched stage
constexpr int kBlock = 256;              // threads per block for streaming kernels
constexpr int kPinnedBytes = 96 << 10;   // the context's pinned read-back buffer
constexpr int kPinnedBulk = 256;         // its part after the single words
constexpr int kWaitLimitDefault = 1 << 22; // polls before a cross-block wait gives up (about 0.3 s)

// device error word bits
enum : int
{
    kErrTimeout = 1,
    kErrCapacity = 2,
    kErrKeyBits = 4,
    kErrSingular = 8,
    kErrInvalid = 16,
    kErrBounds = 32, // an index check of the checked build failed
};

// Index checks of the checked build (compiled with -DGCA3D_CHECKED, the library
// libgca3d_checked.so): an index outside [0, n) sets kErrBounds in the context's error
// word and the access is skipped, so a bad index becomes a status, never a fault or a
// trap.  In the regular build the checks compile to nothing (n is not evaluated).
#ifdef GCA3D_CHECKED
#define GCA_INDEX_OK(i, n, err) ::gca3d::index_ok((long long)(i), (long long)(n), (err))
#else
#define GCA_INDEX_OK(i, n, err) true
#endif

// ---------------------------------------------------------------------------
// scratch memory: chunked bump allocator, reset per top-level call.  A replay
// of the same sequence of requests returns the same addresses, which is what
// graph capture relies on.
// ---------------------------------------------------------------------------
struct Arena
{
    struct Chunk
    {
        char *ptr = nullptr;
        size_t size = 0, used = 0;
    };
    std::vector<Chunk> chunks;
    size_t cur = 0;
    bool frozen = false; // no growth allowed (during capture)
    bool failed = false;
    gca3d_context *owner = nullptr; // the context whose allocations these are (not swapped)

    void *take(size_t bytes);
    void reset()
    {
        for (auto &c : chunks)
            c.used = 0;
        cur = 0;
        failed = false;
    }
    void release();
    size_t bytes() const
    {
        size_t n = 0;
        for (auto &c : chunks)
            n += c.size;
        return n;
    }
    void swap(Arena &o)
    {
        chunks.swap(o.chunks);
        std::swap(cur, o.cur);
        std::swap(frozen, o.frozen);
        std::swap(failed, o.failed);
    }
    Arena() = default;
    Arena(const Arena &) = delete;
    Arena &operator=(const Arena &) = delete;
    ~Arena() { release(); }
    template <typename T> T *get(size_t count) { return static_cast<T *>(take(count * sizeof(T))); }
};

} // namespace gca3d

// ---------------------------------------------------------------------------
// opaque handles
// ---------------------------------------------------------------------------
namespace gca3d
{
enum KernelId : int
{
    kKidNone = -1,
    kKidIcpIter = 0,
    kKidSortPass,
    kKidNormals,
    kKidVoxelReduce,
    kKidGridScatter,
    kKidFrame,
    kKidCount
};
struct Profiler
{
    int target = kKidNone;
    std::vector<cudaEvent_t> events; // start/stop pairs
    size_t used = 0;
};
} // namespace gca3d

struct gca3d_context
{
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int num_sms = 0;
    bool cluster_sort = false; // the device runs the one-launch sort (cluster_sort.cuh)
    gca3d::Arena arena;
    // device control words: [0] error bits (kErr*, set with atomicOr by kernels and
    // consumed by the host), [1] polls after which a cross-block wait gives up
    // (gca3d_set_wait_limit; kernels read it when they start)
    int *d_err = nullptr;
    int *h_pinned = nullptr; // pinned read-backs: 64 ints, and from kPinnedBulk bytes on larger ones
    int upload_mode = 0;     // GCA3D_UPLOAD_IN_PLACE or GCA3D_UPLOAD_COPY_ENGINE
    int64_t launches = 0;
    std::string last_error;
    gca3d::Profiler prof;
    // the workspace of the last one-shot registration, kept for the next (schedule.cu)
    gca3d_icp_plan *spare = nullptr;
};

struct gca3d_cloud
{
    int64_t capacity = 0;
    float4 *pos = nullptr; // x, y, z, intensity
    float4 *col = nullptr; // r, g, b, 0
    float4 *nrm = nullptr;
    float4 *grd = nullptr;
    int32_t *d_count = nullptr;
    bool has_normals = false;
    bool has_grad = false;
    float grad_radius = 0.0f;
    int device = 0;
};

namespace gca3d
{

// ---------------------------------------------------------------------------
// host helpers
// ---------------------------------------------------------------------------
int fail(gca3d_context *ctx, int status, const std::string &msg);
int cuda_fail(gca3d_context *ctx, cudaError_t e, const char *where);
#define GCA_CUDA(ctx, call)                                                                        \
    do                                                                                             \
    {                                                                                              \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return ::gca3d::cuda_fail((ctx), e_, #call);                                           \
    } while (0)
#define GCA_CHECK_LAUNCH(ctx)                                                                      \
    do                                                                                             \
    {                                                                                              \
        (ctx)->launches++;                                                                         \
        cudaError_t e_ = cudaGetLastError();                                                       \
        if (e_ != cudaSuccess)                                                                     \
            return ::gca3d::cuda_fail((ctx), e_, __func__);                                        \
    } while (0)

// event bracket around launches of the profiled kernel (no-op otherwise)
void prof_mark(gca3d_context *ctx, int kid);
#define GCA_PROF_BEGIN(ctx, kid) ::gca3d::prof_mark((ctx), (kid))
#define GCA_PROF_END(ctx, kid) ::gca3d::prof_mark((ctx), (kid))

inline int div_up(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }
inline int grid_for(int64_t n, int per_block = kBlock)
{
    int g = div_up(n > 0 ? n : 1, per_block);
    return g > 0 ? g : 1;
}
int ensure_attr(gca3d_context *ctx, gca3d_cloud *c, bool normals, bool grad);
// reads and clears the device error word; maps bits to a status
int consume_device_error(gca3d_context *ctx, const char *where);
// the status for an error word already read back (0: GCA3D_OK)
int device_error_status(gca3d_context *ctx, int word, const char *where);
// cudaMalloc; where it fails for want of memory, the context's kept workspace is given back
// and it is tried once more
cudaError_t device_malloc(gca3d_context *ctx, void **p, size_t bytes);
template <typename T> cudaError_t device_malloc(gca3d_context *ctx, T **p, size_t bytes)
{
    return device_malloc(ctx, reinterpret_cast<void **>(p), bytes);
}

// ---------------------------------------------------------------------------
// device helpers
// ---------------------------------------------------------------------------

// colour -> intensity in FP64 then rounded, without contraction, as
// color3::to_intensity (src/geometry/type.hpp:45-51)
static __device__ __noinline__ float intensity_f64(float r, float g, float b)
{
    double s = __dadd_rn(__dmul_rn(0.2126, (double)r), __dmul_rn(0.7152, (double)g));
    s = __dadd_rn(s, __dmul_rn(0.0722, (double)b));
    return (float)s;
}

// the same value from FP32 pairs: an SM issues two FP64 operations per clock, so the nine
// of intensity_f64 cost a warp 144 cycles of its SM's FP64 pipe and bound every kernel that
// writes points; this takes about 35 FP32 instructions.  Each product is an exact pair (FMA
// residual, the weight split in two floats), the sum a pair (hi, lo) within 2^-44 of the
// magnitudes' sum m of both the real value and the FP64 one.  When hi + lo rounds to hi
// from either end of an interval of m 2^-43 around it, FP64 rounds there too; otherwise
// (two in 10^6 random colours), and where a pair could lose bits to the exponent range, the FP64
// operations decide.
__device__ __forceinline__ float intensity_of(float r, float g, float b)
{
    constexpr float h0 = (float)0.2126, l0 = (float)(0.2126 - (double)h0);
    constexpr float h1 = (float)0.7152, l1 = (float)(0.7152 - (double)h1);
    constexpr float h2 = (float)0.0722, l2 = (float)(0.0722 - (double)h2);
    const float p0 = __fmul_rn(r, h0), p1 = __fmul_rn(g, h1), p2 = __fmul_rn(b, h2);
    const float e0 = __fmaf_rn(r, l0, __fmaf_rn(r, h0, -p0)), e1 = __fmaf_rn(g, l1, __fmaf_rn(g, h1, -p1)),
                e2 = __fmaf_rn(b, l2, __fmaf_rn(b, h2, -p2));
    const float s = __fadd_rn(p0, p1), sb = __fsub_rn(s, p0);
    const float t = __fadd_rn(__fsub_rn(p0, __fsub_rn(s, sb)), __fsub_rn(p1, sb));
    const float s2 = __fadd_rn(s, p2), sc = __fsub_rn(s2, s);
    const float t2 = __fadd_rn(__fsub_rn(s, __fsub_rn(s2, sc)), __fsub_rn(p2, sc));
    const float low = __fadd_rn(__fadd_rn(t, t2), __fadd_rn(__fadd_rn(e0, e1), e2));
    const float hi = __fadd_rn(s2, low), lo = __fsub_rn(low, __fsub_rn(hi, s2));
    const float m = __fadd_rn(__fadd_rn(fabsf(p0), fabsf(p1)), fabsf(p2));
    const float d = __fmul_rn(m, 1.1368683772161603e-13f); // 2^-43
    if (m > 1e-15f && m < 1e15f && __fadd_rn(hi, __fadd_rn(lo, d)) == hi && __fadd_rn(hi, __fsub_rn(lo, d)) == hi)
        return hi;
    if (r == 0.0f && g == 0.0f && b == 0.0f)
        return s2; // black, with the sign that FP64 gives
    return intensity_f64(r, g, b);
}

// float <-> order-preserving int (for atomicMin/atomicMax on floats)
__device__ __forceinline__ int float_to_ordered(float f)
{
    int i = __float_as_int(f);
    return i >= 0 ? i : i ^ 0x7FFFFFFF;
}
__device__ __forceinline__ float ordered_to_float(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }
inline float ordered_to_float_host(int i)
{
    int j = i >= 0 ? i : i ^ 0x7FFFFFFF;
    float f;
    memcpy(&f, &j, 4);
    return f;
}

// squared distance q - p, unfused, the reference's order (cuda_nn_search.cu:195-200)
__device__ __forceinline__ float dist2_ref(float qx, float qy, float qz, float px, float py, float pz)
{
    float dx = __fsub_rn(qx, px), dy = __fsub_rn(qy, py), dz = __fsub_rn(qz, pz);
    return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// floor((p - mn) / cell), IEEE sub and div (cuda_voxel_grid_down_sample.cu:40-45)
__device__ __forceinline__ int cell_of(float p, float mn, float cell)
{
    return __float2int_rd(__fdiv_rn(__fsub_rn(p, mn), cell));
}

// cell_of with inv = 1 / cell (rounded): the product is within three rounding units of
// (p - mn) / cell and the quotient within one, so where the product is further than that
// from an integer the two have the same floor; only the others are divided (a division is
// three times the instructions, and a key has three)
__device__ __forceinline__ int cell_of_inv(float p, float mn, float cell, float inv)
{
    const float d = __fsub_rn(p, mn);
    const float q = __fmul_rn(d, inv), f = floorf(q);
    const float r = __fsub_rn(q, f), slack = __fmul_rn(fabsf(q), 4.0e-7f);
    if (r > slack && __fsub_rn(1.0f, r) > slack && fabsf(q) < 4.0e6f && fabsf(q) > 1.0e-30f)
        return (int)f;
    return __float2int_rd(__fdiv_rn(d, cell));
}

__device__ __forceinline__ int bitlen_u32(uint32_t v) { return v ? 32 - __clz(v) : 0; }

// block-wide min/max of 3 components, then one atomic per component per block
// (per-warp atomics on the same few words serialise in one L2 slice)
__device__ __forceinline__ void block_bounds_commit(float mn[3], float mx[3], int *ord6)
{
    __shared__ float s_mn[3][32], s_mx[3][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            mn[a] = fminf(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
            mx[a] = fmaxf(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
        }
    if (lane == 0)
        for (int a = 0; a < 3; ++a)
            s_mn[a][warp] = mn[a], s_mx[a][warp] = mx[a];
    __syncthreads();
    if (threadIdx.x < 3)
    {
        const int a = threadIdx.x;
        float m = s_mn[a][0], M = s_mx[a][0];
        for (int w = 1; w < nw; ++w)
            m = fminf(m, s_mn[a][w]), M = fmaxf(M, s_mx[a][w]);
        atomicMin(ord6 + a, float_to_ordered(m));
        atomicMax(ord6 + 3 + a, float_to_ordered(M));
    }
}

// the wait limit of the context whose control words ctl points to (see gca3d_context)
__device__ __forceinline__ uint32_t wait_limit(const int *ctl)
{
    return (uint32_t)*(const volatile int *)(ctl + 1);
}

__device__ __forceinline__ bool index_ok(long long i, long long n, int *err)
{
    if (i >= 0 && i < n)
        return true;
    atomicOr(err, kErrBounds);
    return false;
}

// ---------------------------------------------------------------------------
// batched ("segmented") point sets: P clouds back to back
// ---------------------------------------------------------------------------

// parameters of one packed 64-bit cell key layout, shared by all segments
struct KeyLayout
{
    int bseg, bx, by, bz; // bits per field; key = seg|cx|cy|cz from MSB to LSB
    int total_bits;
    int morton; // voxel keys only: seg | bit-interleaved (cx, cy, cz), bx = by = bz
    // grid keys only: the row table is indexed by key >> zs, runs of 2^zs z cells of a row
    // (direct = 1), or is a hash of whole rows (direct = 0)
    int direct, zs;
};

// one open-addressing slot of the row hash: the key and the row's [start, end) in
// the sorted arrays, read with a single 16-byte load
struct __align__(16) RowSlot
{
    unsigned long long key;
    int start;
    int end;
};

// a grid over the target segments
struct GridDev
{
    // per segment
    float3 *gmin;  // grid origin
    float cell;     // cell edge
    float inv_cell; // 1 / cell (conservative bounds only; cells are assigned by division)
    KeyLayout *layout;
    // sorted points (global positions over all segments)
    float4 *spos;  // x, y, z, __int_as_float(cz)
    int32_t *sidx; // batch index of the point (original order)
    float *sint;   // intensity in sorted order
    int *scz;      // z cell in sorted order (compact copy for the in-row binary search)
    uint64_t *skey;
    // the row table (KeyLayout::direct): [start, end) per run of z cells, or a hash
    // (seg, cx, cy) -> [start, end) in 16-byte slots, at least twice as many as points, so
    // the first probe nearly always decides.  One memory serves both; empty is all ones.
    RowSlot *slots;
    uint32_t hmask;
    const int32_t *seg_off; // [P + 1] offsets of the segments in the sorted arrays
    const int32_t *d_n;     // points in the grid (seg_off[P])
    int *err;               // the context's error word (index checks of the checked build)
};

constexpr unsigned long long kEmptyKey = ~0ull;

__device__ __forceinline__ uint32_t hash_u64(unsigned long long k)
{
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdull;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ull;
    k ^= k >> 33;
    return (uint32_t)k;
}

__device__ __forceinline__ ulonglong2 slot_load(const RowSlot *slots, uint32_t h)
{
    return __ldg(reinterpret_cast<const ulonglong2 *>(slots + h));
}

// entry i of a direct row table; {-1, -1} when it is empty
__device__ __forceinline__ int2 run_load(const RowSlot *slots, uint32_t i)
{
    return __ldg(reinterpret_cast<const int2 *>(slots) + i);
}

// continue a linear probe after the first slot missed
static __device__ __noinline__ int2 row_probe_rest(const RowSlot *slots, uint32_t hmask, unsigned long long rk, uint32_t h)
{
    for (uint32_t probe = 1; probe <= hmask; ++probe)
    {
        h = (h + 1) & hmask;
        const ulonglong2 v = slot_load(slots, h);
        if (v.x == rk)
            return make_int2((int)(uint32_t)v.y, (int)(uint32_t)(v.y >> 32));
        if (v.x == kEmptyKey)
            break;
    }
    return make_int2(0, 0);
}

// ---------------------------------------------------------------------------
// stage entry points implemented in the .cu files (all stream-ordered)
// ---------------------------------------------------------------------------

// radix sort of (key, value) pairs by the low `max_bits` bits, n on the device.
// keys/vals are ping-pong buffers of capacity `cap`; on return *result_in_alt
// (device int) says whether the sorted data is in the alternate buffers.
// A sort of (key, index) pairs runs in one of two forms, chosen on the device by the
// kernel that writes the keys, once the key layout is known: packed, (key << ib) |
// index in one 64-bit word, when the key's bits and ib (the bits of the largest index)
// fit in 64 -- 8 bytes per element each way per pass instead of 12 -- or keys and
// indices in separate arrays.  The index is the element's position when the keys are
// written, so in both forms equal keys keep ascending index order.
struct SortBuffers
{
    uint64_t *keys[2];
    int32_t *vals[2];
    int *d_sel;    // device: index of the buffer holding the sorted data
    int *d_ib;     // device: index bits of the packed form, 0 for separate arrays
    int *d_kshift; // device: the key's lowest bit in a sort word (ib, plus sub-cell bits a
                   // voxel stage carries for finer scales); the digits start there
};

// index bits of a sort of at most cap elements
inline int index_bits(int64_t cap)
{
    int b = 1;
    while ((1ll << b) < cap)
        ++b;
    return b;
}

// the packed form's index bits for a key of key_bits bits, or 0 when it does not fit
__device__ __forceinline__ int packed_index_bits(int key_bits, int ib) { return key_bits + ib <= 64 ? ib : 0; }

// element i of the key kernels' output: the word w (the key, with any sub-cell bits
// below it) and index i
__device__ __forceinline__ void sort_store(uint64_t *keys, int32_t *vals, int i, uint64_t w, int ib)
{
    if (ib)
        keys[i] = (w << ib) | (uint64_t)(uint32_t)i;
    else
    {
        keys[i] = w;
        vals[i] = i;
    }
}

// the sorted keys and indices, whichever the form
struct SortedView
{
    const uint64_t *k;
    const int32_t *v;
    int ib, kshift;
    __device__ __forceinline__ uint64_t key(int i) const { return k[i] >> kshift; }
    __device__ __forceinline__ int32_t val(int i) const
    {
        return ib ? (int32_t)(k[i] & ((1ull << ib) - 1ull)) : v[i];
    }
};
__device__ __forceinline__ SortedView sorted_view(const SortBuffers &sb)
{
    const int sel = *sb.d_sel;
    return SortedView{sb.keys[sel], sb.vals[sel], *sb.d_ib, *sb.d_kshift};
}

// exclusive scan of int32 values (n on the device), writes total to *d_total
int exclusive_scan(gca3d_context *ctx, const int32_t *in, int32_t *out, const int32_t *d_n,
                   int64_t cap, int32_t *d_total);
// the runs of equal keys of a sorted view in one scan: starts[r] the first position of
// run r, starts[runs] = n, *d_runs the number of runs, seg_first[s] the first run of
// segment s (left untouched, e.g. -1, for an empty segment; may be null).  For one segment
// seg_off receives {0, runs} and *d_count the number of runs (either may be null).
// zeroed: run_scan_zero_bytes(cap) of memory that the caller has cleared, or null.
size_t run_scan_zero_bytes(int64_t cap);
int run_scan(gca3d_context *ctx, const SortBuffers &sb, const int32_t *d_n, int64_t cap, const KeyLayout *lay,
             int32_t *starts, int32_t *seg_first, int32_t *d_runs, int32_t *seg_off = nullptr,
             int32_t *d_count = nullptr, void *zeroed = nullptr);

} // namespace gca3d
