// Row-hash bucketize of a jagged batch for row-wise sharding: bucket = id % world,
// output grouped by (bucket, feature, sample) in input order, plus the permute
// that undoes it; optionally a first-occurrence dedup per (bucket, feature) with
// occurrence counts.  One thread walks one bag in order, which keeps the order
// inside a (bucket, feature, sample) cell identical to the sequential CPU loop.
#include "prims.cuh"

namespace recsdk {

constexpr int kMaxWorld = 64;

#define RECSDK_GRID_STRIDE(i, n)                                                        \
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < (n); \
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)

// offsets of the bags: exclusive scan of the int64 lengths, L + 1 values
struct LengthsIn {
    const int64_t* lengths;
    int64_t L;
    __device__ __forceinline__ int operator()(int64_t i) const { return i < L ? static_cast<int>(lengths[i]) : 0; }
};
struct OffsetsOut {
    int* offs;
    __device__ __forceinline__ void operator()(int64_t i, int, int prefix, int64_t) const { offs[i] = prefix; }
};

// bucketize.cpp:35-51
static __global__ void __launch_bounds__(128) bucket_count_kernel(const int* __restrict__ offs,
                                                                  const int64_t* __restrict__ indices, int64_t L, int W,
                                                                  int* __restrict__ nl)
{
    RECSDK_GRID_STRIDE(lin, L)
    {
        int cnt[kMaxWorld];
        for (int w = 0; w < W; ++w) cnt[w] = 0;
        for (int i = offs[lin]; i < offs[lin + 1]; ++i) cnt[static_cast<int>(indices[i] % W)]++;
        for (int w = 0; w < W; ++w) nl[static_cast<int64_t>(w) * L + lin] = cnt[w];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) nl[static_cast<int64_t>(W) * L] = 0;
}

// bucketize.cpp:54-76
static __global__ void __launch_bounds__(128) bucket_fill_kernel(const int* __restrict__ offs,
                                                                 const int64_t* __restrict__ indices, int64_t L, int W,
                                                                 const int* __restrict__ noffs,
                                                                 int64_t* __restrict__ new_indices,
                                                                 int64_t* __restrict__ perm)
{
    RECSDK_GRID_STRIDE(lin, L)
    {
        int cur[kMaxWorld];
        for (int w = 0; w < W; ++w) cur[w] = noffs[static_cast<int64_t>(w) * L + lin];
        for (int i = offs[lin]; i < offs[lin + 1]; ++i) {
            const int64_t id = indices[i];
            const int b = static_cast<int>(id % W);
            const int pos = cur[b]++;
            new_indices[pos] = id;
            perm[i] = pos;
        }
    }
}

static __global__ void set_i64_kernel(int64_t* p, int64_t v) { *p = v; }

// ---- dedup per (bucket, feature), bucketize.cpp:79-130 ----------------------
// An id has one bucket, so a (bucket, feature) segment holds it exactly when its feature does, and the segment's first
// occurrence is the feature's lowest position.  Positions are therefore grouped by (feature, id) through an
// open-addressing table of positions -- a slot names a position whose feature and id are the slot's key, and ends up
// with the lowest one -- instead of a sort of 64-bit ids: 852 K ids of 26
// features took 7 radix passes, 169 us, and nine more kernels over the pairs, 60 us; the probe of this table takes 37 us.
// The table holds at most half as many keys as slots.  Bound by the latency of its random L2 accesses.
constexpr uint32_t kNoPos = 0xffffffffu;
constexpr uint8_t kNotFirst = 0xff;  // a bucket number is below kMaxWorld

static inline int64_t dedup_capacity(int64_t n)
{
    int64_t cap = 64;
    while (cap < 2 * n) cap <<= 1;
    return cap;
}
__device__ __forceinline__ uint64_t mix_feature_id(uint64_t id, uint64_t f)
{
    uint64_t x = id + f * 0x9e3779b97f4a7c15ull;
    x ^= x >> 32;
    x *= 0xd6e8feb86659fd93ull;
    x ^= x >> 32;
    x *= 0xd6e8feb86659fd93ull;
    x ^= x >> 32;
    return x;
}

// ent[i] = slot of (feature of i, id of i); cnt[slot] counts occurrences, from -1
static __global__ void __launch_bounds__(256) dedup_insert_kernel(const int* __restrict__ offs, int64_t B, int64_t F,
                                                                  const int64_t* __restrict__ indices, int64_t n, int64_t cap,
                                                                  uint32_t* __restrict__ table, uint32_t* __restrict__ cnt,
                                                                  uint32_t* __restrict__ ent)
{
    RECSDK_GRID_STRIDE(i, n)
    {
        int64_t lo = 0, hi = F - 1;  // feature of i: the last f with offs[f * B] <= i
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (offs[mid * B] <= i) lo = mid; else hi = mid - 1;
        }
        const uint32_t f0 = static_cast<uint32_t>(offs[lo * B]), f1 = static_cast<uint32_t>(offs[(lo + 1) * B]);
        const int64_t id = indices[i];
        const uint32_t pos = static_cast<uint32_t>(i);
        uint64_t h = mix_feature_id(static_cast<uint64_t>(id), static_cast<uint64_t>(lo)) & (cap - 1);
        for (int64_t probes = 0; probes < cap; ++probes) {
            uint32_t s = *reinterpret_cast<volatile uint32_t*>(table + h);
            if (s == kNoPos) {
                s = atomicCAS(table + h, kNoPos, pos);
                if (s == kNoPos) break;
            }
            // whatever position the slot names now, its key stays the same
            if (s >= f0 && s < f1 && indices[s] == id) {
                if (pos < s) atomicMin(table + h, pos);
                break;
            }
            h = (h + 1) & (cap - 1);
        }
        ent[i] = static_cast<uint32_t>(h);
        if (cnt != nullptr) atomicAdd(cnt + h, 1u);
    }
}
// bucket of the first occurrences, kNotFirst for the others
static __global__ void __launch_bounds__(256) dedup_first_kernel(const int64_t* __restrict__ indices, int64_t n, int W,
                                                                 const uint32_t* __restrict__ table,
                                                                 const uint32_t* __restrict__ ent, uint8_t* __restrict__ first)
{
    RECSDK_GRID_STRIDE(i, n)
    first[i] = table[ent[i]] == static_cast<uint32_t>(i) ? static_cast<uint8_t>(indices[i] % W) : kNotFirst;
}
// first occurrences per (bucket, bag); the counters of a block's bags stand in shared memory, [bucket][bag]
constexpr int kDedupBags = 128;
static __global__ void __launch_bounds__(kDedupBags) dedup_count_kernel(const int* __restrict__ offs, int64_t L, int W,
                                                                        const uint8_t* __restrict__ first,
                                                                        int* __restrict__ nl)
{
    extern __shared__ int bucket_sm[];
    int* mine = bucket_sm + threadIdx.x;
    RECSDK_GRID_STRIDE(lin, L)
    {
        for (int w = 0; w < W; ++w) mine[w * kDedupBags] = 0;
        const int e = offs[lin + 1];
        for (int i = offs[lin]; i < e; ++i) {
            const int b = first[i];
            if (b < W) ++mine[b * kDedupBags];
        }
        for (int w = 0; w < W; ++w) nl[static_cast<int64_t>(w) * L + lin] = mine[w * kDedupBags];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) nl[static_cast<int64_t>(W) * L] = 0;
}
struct CellsIn {
    const int* nl;
    __device__ __forceinline__ int operator()(int64_t i) const { return nl[i]; }
};
struct CellsOut {
    int* noffs;
    int64_t* new_lengths;
    int64_t cells;
    __device__ __forceinline__ void operator()(int64_t i, int item, int prefix, int64_t) const
    {
        noffs[i] = prefix;
        if (i < cells) new_lengths[i] = item;
    }
};
// every first occurrence goes to its place, which takes the position's place in its slot
static __global__ void __launch_bounds__(kDedupBags) dedup_fill_kernel(const int* __restrict__ offs,
                                                                       const int64_t* __restrict__ indices, int64_t L, int W,
                                                                       const uint8_t* __restrict__ first,
                                                                       const int* __restrict__ noffs,
                                                                       const uint32_t* __restrict__ ent,
                                                                       const uint32_t* __restrict__ cnt,
                                                                       uint32_t* __restrict__ table,
                                                                       int64_t* __restrict__ out_indices,
                                                                       int64_t* __restrict__ counts)
{
    extern __shared__ int bucket_sm[];
    int* mine = bucket_sm + threadIdx.x;
    RECSDK_GRID_STRIDE(lin, L)
    {
        for (int w = 0; w < W; ++w) mine[w * kDedupBags] = noffs[static_cast<int64_t>(w) * L + lin];
        const int e = offs[lin + 1];
        for (int i = offs[lin]; i < e; ++i) {
            const int b = first[i];
            if (b >= W) continue;
            const int u = mine[b * kDedupBags]++;
            const uint32_t h = ent[i];
            out_indices[u] = indices[i];
            table[h] = static_cast<uint32_t>(u);
            if (counts != nullptr) counts[u] = static_cast<int64_t>(cnt[h] + 1u);
        }
    }
}
static __global__ void __launch_bounds__(256) dedup_perm_kernel(int64_t* __restrict__ perm, int64_t n,
                                                                const uint32_t* __restrict__ table,
                                                                const uint32_t* __restrict__ ent)
{
    RECSDK_GRID_STRIDE(i, n) perm[i] = table[ent[i]];
}

struct BucketWs {
    int *offs, *nl, *noffs, *scan_scratch;
    uint32_t *table, *cnt, *ent;
    uint8_t* first;
    int64_t cap;
    size_t bytes;
};
static BucketWs carve_bucket(void* base, int64_t N, int64_t L, int64_t W)
{
    WorkspaceCarver c(base);
    BucketWs w;
    const size_t n = static_cast<size_t>(N > 0 ? N : 1);
    const size_t cells = static_cast<size_t>(L * W);
    w.cap = dedup_capacity(N);
    w.offs = c.take<int>(static_cast<size_t>(L) + 1);
    w.nl = c.take<int>(cells + 1);
    w.noffs = c.take<int>(cells + 1);
    w.table = c.take<uint32_t>(static_cast<size_t>(w.cap) * 2);  // table and cnt: cleared together
    w.cnt = w.table + w.cap;
    w.ent = c.take<uint32_t>(n);
    w.first = c.take<uint8_t>(n);
    w.scan_scratch = c.take<int>(scan_scratch_ints(static_cast<int64_t>(cells) + 1));
    w.bytes = c.used();
    return w;
}

}  // namespace recsdk

using namespace recsdk;

extern "C" size_t recsdk_bucketize_workspace_bytes(int64_t n, int64_t lengths_size, int64_t world)
{
    return carve_bucket(nullptr, n, lengths_size, world).bytes;
}

extern "C" int recsdk_bucketize(const int64_t* lengths, int64_t lengths_size, const int64_t* indices, int64_t n,
                                int64_t num_features, int64_t world, int32_t do_unique, int32_t return_count,
                                int64_t* new_lengths, int64_t* new_indices, int64_t* unbucketize_permute,
                                int64_t* ids_counts, int64_t* num_out, void* workspace, size_t workspace_bytes,
                                void* stream)
{
    if (lengths_size <= 0 || n <= 0 || num_features <= 0 || world <= 0 || world > kMaxWorld) return RECSDK_ERR_INVALID_ARG;
    if (lengths_size % num_features != 0) return RECSDK_ERR_INVALID_ARG;
    if (!lengths || !indices || !new_lengths || !new_indices || !unbucketize_permute || !num_out) return RECSDK_ERR_INVALID_ARG;
    if (do_unique && return_count && !ids_counts) return RECSDK_ERR_INVALID_ARG;
    if (n >= (int64_t(1) << 31) || lengths_size * world >= (int64_t(1) << 31)) return RECSDK_ERR_TOO_LARGE;
    if (!workspace) return RECSDK_ERR_WORKSPACE;
    const int64_t L = lengths_size, W = world, F = num_features, B = L / F, cells = L * W;
    const BucketWs ws = carve_bucket(workspace, n, L, W);
    if (ws.bytes > workspace_bytes) return RECSDK_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int Wi = static_cast<int>(W);

    device_scan_fn<false>(LengthsIn{lengths, L}, OffsetsOut{ws.offs}, L + 1, ws.scan_scratch, nullptr, st);
    if (!do_unique) {
        bucket_count_kernel<<<grid_for(L, 128), 128, 0, st>>>(ws.offs, indices, L, Wi, ws.nl);
        device_scan_fn<false>(CellsIn{ws.nl}, CellsOut{ws.noffs, new_lengths, cells}, cells + 1, ws.scan_scratch, nullptr, st);
        bucket_fill_kernel<<<grid_for(L, 128), 128, 0, st>>>(ws.offs, indices, L, Wi, ws.noffs, new_indices,
                                                            unbucketize_permute);
        set_i64_kernel<<<1, 1, 0, st>>>(num_out, n);
        RECSDK_CUDA_CHECK_LAUNCH();
        return RECSDK_OK;
    }
    const int grid = grid_for(n, 256), bag_grid = grid_for(L, kDedupBags);
    const size_t smem = static_cast<size_t>(W) * kDedupBags * sizeof(int);  // 32 KB at kMaxWorld
    uint32_t* cnt = return_count ? ws.cnt : nullptr;
    cudaMemsetAsync(ws.table, 0xff, static_cast<size_t>(ws.cap) * sizeof(uint32_t) * (cnt ? 2 : 1), st);
    dedup_insert_kernel<<<grid, 256, 0, st>>>(ws.offs, B, F, indices, n, ws.cap, ws.table, cnt, ws.ent);
    dedup_first_kernel<<<grid, 256, 0, st>>>(indices, n, Wi, ws.table, ws.ent, ws.first);
    dedup_count_kernel<<<bag_grid, kDedupBags, smem, st>>>(ws.offs, L, Wi, ws.first, ws.nl);
    device_scan_fn<false>(CellsIn{ws.nl}, CellsOut{ws.noffs, new_lengths, cells}, cells + 1, ws.scan_scratch, num_out, st);
    dedup_fill_kernel<<<bag_grid, kDedupBags, smem, st>>>(ws.offs, indices, L, Wi, ws.first, ws.noffs, ws.ent, cnt, ws.table,
                                                          new_indices, return_count ? ids_counts : nullptr);
    dedup_perm_kernel<<<grid, 256, 0, st>>>(unbucketize_permute, n, ws.table, ws.ent);
    RECSDK_CUDA_CHECK_LAUNCH();
    return RECSDK_OK;
}
