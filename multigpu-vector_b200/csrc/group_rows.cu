// group_rows.cu -- a closed group-by's rows: taken out of its hash table,
// ordered by group on the device and written straight into pinned, mapped
// host memory, with the table left empty for the next open.
//
// Ordering is a sort of {group, source} pairs by one CTA per result: most
// results have at most a few tens of thousands of groups, so a device-wide sort
// would be launches and waits, and results of a batch run side by side on
// different SMs.  (Of a million groups one CTA still takes a third of the time
// that the host does: kDeviceOrderCap.)  On the host it cost about 35 us per
// 4096 groups and was half of a batch's time with its results read (366 K
// groups of 64 queries: 3.1 ms; here 64 us for the largest of them, 60 K
// groups).  The ordered rows are written to the host by many CTAs, at the host
// link's rate (8.8 MB in 118 us): one SM's stores to host memory reach about
// 8 GB/s.
#include <cuda_runtime.h>

#include <algorithm>

#include "device_common.cuh"
#include "mgv_internal.h"

namespace mgv {
namespace {

constexpr int kSortBlock = 1024;
constexpr uint32_t kSortWarps = kSortBlock / 32;
constexpr int kSortUnroll = 8;               // pairs per lane loaded before any is placed
constexpr uint32_t kDigits = 256;
constexpr uint32_t kCntStride = kSortWarps + 1;  // counters of one digit, a bank apart from the next digit's
constexpr size_t kCntBytes = sizeof(uint32_t) * kDigits * kCntStride;
constexpr uint32_t kRankSort = 512;          // pairs ordered by counting the smaller ones
constexpr uint32_t kBitmapWords = 4096;      // groups spanning 131072 values are placed by bitmap
static_assert(2 * sizeof(uint32_t) * kBitmapWords <= kCntBytes, "the bitmap and its counts take the counters' place");
constexpr uint32_t kSmemPairs = 8192;        // pairs sorted in shared memory (two buffers: 128 KiB)
constexpr size_t kSortSmem = kCntBytes + 2 * sizeof(unsigned long long) * kSmemPairs;

// {order-preserving group, source index}
__device__ __forceinline__ unsigned long long make_pair(int32_t group, uint32_t src) {
    return ((unsigned long long)((uint32_t)group ^ 0x80000000u) << 32) | src;
}
__device__ __forceinline__ int32_t pair_group(unsigned long long p) {
    return (int32_t)((uint32_t)(p >> 32) ^ 0x80000000u);
}

// Orders a[0..n) by group; the sorted pairs end in a or b, which is returned.
// Three ways: up to kRankSort pairs each count the smaller ones; groups that
// span at most kBitmapWords * 32 values (dictionary codes) take their place
// from a bitmap of the groups present, three short steps; others are radix
// sorted.  There each warp owns a contiguous segment and places its pairs in
// order, so every pass is stable: counters are kept per (digit, warp) and
// scanned digit-major.  5003 codes: radix 14 us, bitmap 2 us.
__device__ unsigned long long* sort_pairs(unsigned long long* a, unsigned long long* b, uint32_t n, uint32_t* cnt) {
    __shared__ uint32_t s_min, s_max;
    const uint32_t lane = lane_id(), warp = threadIdx.x / 32;
    if (n < 2) return a;
    if (n <= kRankSort) {
        for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) {
            const unsigned long long v = a[i];
            uint32_t rank = 0;
#pragma unroll 8
            for (uint32_t j = 0; j < n; ++j) rank += a[j] < v;
            b[rank] = v;
        }
        __syncthreads();
        return b;
    }
    if (threadIdx.x == 0) {
        s_min = 0xffffffffu;
        s_max = 0;
    }
    __syncthreads();
    uint32_t mn = 0xffffffffu, mx = 0;
#pragma unroll 8
    for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) {
        const uint32_t g = (uint32_t)(a[i] >> 32);
        mn = min(mn, g);
        mx = max(mx, g);
    }
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (lane == 0) {
        atomicMin(&s_min, mn);
        atomicMax(&s_max, mx);
    }
    __syncthreads();
    mn = s_min;
    mx = s_max;
    if (mx - mn < kBitmapWords * 32) {
        const uint32_t words = (mx - mn) / 32 + 1;
        uint32_t* bits = cnt;
        uint32_t* before = cnt + kBitmapWords;  // groups present in the words before
        for (uint32_t w = threadIdx.x; w < words; w += kSortBlock) bits[w] = 0;
        __syncthreads();
#pragma unroll 8
        for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) {
            const uint32_t d = (uint32_t)(a[i] >> 32) - mn;
            atomicOr(bits + d / 32, 1u << (d & 31));
        }
        __syncthreads();
        for (uint32_t w = threadIdx.x; w < words; w += kSortBlock) before[w] = __popc(bits[w]);
        __syncthreads();
        block_exclusive_scan<kSortBlock>(before, words);
        for (uint32_t i0 = threadIdx.x; i0 < n; i0 += kSortBlock * kSortUnroll) {
            unsigned long long v[kSortUnroll];
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) v[u] = i0 + u * kSortBlock < n ? a[i0 + u * kSortBlock] : 0ull;
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) {
                const uint32_t d = (uint32_t)(v[u] >> 32) - mn;
                if (i0 + u * kSortBlock < n) b[before[d / 32] + __popc(bits[d / 32] & ((1u << (d & 31)) - 1u))] = v[u];
            }
        }
        __syncthreads();
        return b;
    }
    const uint32_t bits = 32 - __clz(mn ^ mx);
    const uint32_t passes = (bits + 7) / 8, width = (bits + passes - 1) / passes, mask = (1u << width) - 1u;
    const uint32_t per = ((n + kSortWarps - 1) / kSortWarps + 31) & ~31u;
    const uint32_t lo = min(n, warp * per), hi = min(n, lo + per);
    const uint32_t counters = (mask + 1) * kCntStride;
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const uint32_t shift = 32 + pass * width;
        for (uint32_t i = threadIdx.x; i < counters; i += kSortBlock) cnt[i] = 0;
        __syncthreads();
        for (uint32_t i0 = lo + lane; i0 < hi; i0 += 32 * kSortUnroll) {
            unsigned long long v[kSortUnroll];
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) v[u] = i0 + 32 * u < hi ? a[i0 + 32 * u] : 0ull;
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u)
                if (i0 + 32 * u < hi) atomicAdd(cnt + ((uint32_t)(v[u] >> shift) & mask) * kCntStride + warp, 1u);
        }
        __syncthreads();
        block_exclusive_scan<kSortBlock>(cnt, counters);
        for (uint32_t i0 = lo; i0 < hi; i0 += 32 * kSortUnroll) {
            unsigned long long v[kSortUnroll];
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) {
                const uint32_t i = i0 + 32 * u + lane;
                v[u] = i < hi ? a[i] : 0ull;
            }
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) {
                const bool in = i0 + 32 * u + lane < hi;
                // a digit no pair has for the lanes past the end, so that they match none
                const uint32_t d = in ? (uint32_t)(v[u] >> shift) & mask : kDigits;
                const uint32_t peers = __match_any_sync(0xffffffffu, d);
                uint32_t* c = cnt + d * kCntStride + warp;
                const uint32_t base = in ? *c : 0u;
                __syncwarp();  // read by every peer before the last of them moves it on
                if (in) {
                    b[base + __popc(peers & ((1u << lane) - 1u))] = v[u];
                    if (lane == 31 - __clz(peers)) *c = base + __popc(peers);
                }
                __syncwarp();
            }
        }
        __syncthreads();
        unsigned long long* t = a;
        a = b;
        b = t;
    }
    return a;
}

// The landing zone's header: the error word, then the groups found.
__device__ __forceinline__ void land_header(GroupLanding* land, const uint32_t* err, uint32_t n) {
    const uint32_t e0 = err[0], e1 = err[1];  // both reads before a write they might alias
    land->err[0] = e0;
    land->err[1] = e1;
    land->count = n;
}

// A group table of up to kSmallGroupCap slots, closed by one CTA: its groups
// in order into the landing zone, its slots empty again.
__global__ void __launch_bounds__(kSortBlock) k_group_close(GroupTableView gt, GroupLanding* land, uint32_t sort,
                                                            const uint32_t* err) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem);
    unsigned long long* a = reinterpret_cast<unsigned long long*>(smem + kCntBytes);
    unsigned long long* b = a + gt.cap + 1;
    __shared__ uint32_t s_n;
    const uint32_t lane = lane_id();
    if (threadIdx.x == 0) s_n = 0;
    __syncthreads();
    for (uint32_t i0 = threadIdx.x & ~31u; i0 <= gt.cap; i0 += kSortBlock * kSortUnroll) {
        int32_t k[kSortUnroll];
#pragma unroll
        for (int u = 0; u < kSortUnroll; ++u) {
            const uint32_t i = i0 + u * kSortBlock + lane;
            k[u] = i < gt.cap ? gt.keys[i] : kEmptyKey;
        }
#pragma unroll
        for (int u = 0; u < kSortUnroll; ++u) {
            const uint32_t i = i0 + u * kSortBlock + lane;  // the slot past the last: the group INT32_MIN
            const bool keep = i == gt.cap ? gt.special[1] != 0 : k[u] != kEmptyKey;
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            uint32_t base = 0;
            if (lane == 0 && m) base = atomicAdd(&s_n, (uint32_t)__popc(m));
            base = __shfl_sync(0xffffffffu, base, 0);
            if (keep) a[base + __popc(m & ((1u << lane) - 1u))] = make_pair(k[u], i);
        }
    }
    __syncthreads();
    const uint32_t n = s_n;
    if (sort) a = sort_pairs(a, b, n, cnt);
    if (threadIdx.x == 0) land_header(land, err, n);
    // 64-bit words of the rows, so that a warp writes consecutive host addresses
    unsigned long long* out = reinterpret_cast<unsigned long long*>(land->rows);
    for (uint32_t w = threadIdx.x; w < 3 * n; w += kSortBlock) {
        const uint32_t i = w / 3, f = w - 3 * i, slot = (uint32_t)a[i];
        out[w] = f == 0 ? (unsigned long long)(uint32_t)pair_group(a[i])
                 : slot == gt.cap ? gt.special[f - 1]
                 : f == 1 ? gt.sums[slot] : gt.counts[slot];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) {
        const uint32_t slot = (uint32_t)a[i];
        if (slot == gt.cap) {
            gt.special[0] = gt.special[1] = 0;
        } else {
            gt.keys[slot] = kEmptyKey;
            gt.sums[slot] = 0;
            gt.counts[slot] = 0;
        }
    }
}

// The order of packed rows, one CTA per job: job.order[i] = the row that comes i-th.
__global__ void __launch_bounds__(kSortBlock) k_group_sort(const GroupSortJob* __restrict__ jobs, GroupSortJob job0,
                                                           uint32_t njobs) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem);
    for (uint32_t j = blockIdx.x; j < njobs; j += gridDim.x) {
        const GroupSortJob job = jobs ? jobs[j] : job0;
        const uint32_t found = *job.count, n = min(found, job.capacity);
        unsigned long long* a = n <= kSmemPairs ? reinterpret_cast<unsigned long long*>(smem + kCntBytes) : job.pairs;
        unsigned long long* b = n <= kSmemPairs ? a + kSmemPairs : job.pairs + job.capacity;
        __syncthreads();  // the previous job is done with the buffers
        for (uint32_t i0 = threadIdx.x; i0 < n; i0 += kSortBlock * kSortUnroll) {
            int32_t g[kSortUnroll];
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) {
                const uint32_t i = i0 + u * kSortBlock;
                g[u] = i < n ? job.rows[i].group : 0;
            }
#pragma unroll
            for (int u = 0; u < kSortUnroll; ++u) {
                const uint32_t i = i0 + u * kSortBlock;
                if (i < n) a[i] = make_pair(g[u], i);
            }
        }
        __syncthreads();
        a = sort_pairs(a, b, n, cnt);
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) job.order[i] = (uint32_t)a[i];
        if (threadIdx.x == 0) {
            *job.found = found;
            if (job.land) *job.count = 0;  // an operator's counter, ready for its next close
        }
    }
}

// The ordered rows to where the host reads them: CTA (j, y) takes every
// gridDim.y-th kEmitRows rows of job j, as 64-bit words, so that a warp
// writes consecutive addresses.
constexpr int kEmitBlock = 256;
constexpr uint32_t kEmitRows = 512;
constexpr int kEmitWords = 3 * kEmitRows / kEmitBlock;  // per thread, all in flight

__global__ void __launch_bounds__(kEmitBlock) k_group_emit(const GroupSortJob* __restrict__ jobs, GroupSortJob job0,
                                                           const uint32_t* err) {
    const GroupSortJob job = jobs ? jobs[blockIdx.x] : job0;
    const uint32_t found = *job.found, n = min(found, job.capacity);
    if (blockIdx.y == 0 && threadIdx.x == 0 && job.land) land_header(job.land, err, found);
    const unsigned long long* in = reinterpret_cast<const unsigned long long*>(job.rows);
    for (uint64_t r0 = (uint64_t)blockIdx.y * kEmitRows; r0 < n; r0 += (uint64_t)gridDim.y * kEmitRows) {
        const uint64_t end = 3 * min((uint64_t)n, r0 + kEmitRows);
        uint32_t src[kEmitWords], f[kEmitWords];
        unsigned long long v[kEmitWords];
#pragma unroll
        for (int u = 0; u < kEmitWords; ++u) {
            const uint64_t w = 3 * r0 + u * kEmitBlock + threadIdx.x;
            const uint32_t i = (uint32_t)(w / 3);
            f[u] = (uint32_t)(w - 3ull * i);
            src[u] = w < end ? job.order[i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < kEmitWords; ++u) v[u] = in[3ull * src[u] + f[u]];
#pragma unroll
        for (int u = 0; u < kEmitWords; ++u) {
            const uint64_t w = 3 * r0 + u * kEmitBlock + threadIdx.x;
            if (w >= end) continue;
            if (w < 3ull * job.out_rows) reinterpret_cast<unsigned long long*>(job.out)[w] = v[u];
            else reinterpret_cast<unsigned long long*>(job.more)[w - 3ull * job.out_rows] = v[u];
        }
    }
}

constexpr int kPackBlock = 256;
// The groups in slots [lo, hi) of a table (slot cap: the group INT32_MIN), by
// one CTA, into rows from *count on; rows past `capacity` are dropped and
// reported.  The loop is a chain of memory round trips (key, sums and counts,
// reservation, store), so a lane takes SLOTS slots through it at a time; one
// table is spread over more CTAs instead.  CLEAR empties the slots read.
template <bool CLEAR, int SLOTS>
__device__ __forceinline__ void pack_slots(const GroupTableView& gt, uint64_t lo, uint64_t hi, mgv_group_row* rows,
                                           uint32_t* count, uint32_t capacity, uint32_t* err) {
    const uint32_t lane = lane_id();
    for (uint64_t i0 = lo + (threadIdx.x / 32) * 32 * SLOTS; i0 < hi; i0 += kPackBlock * SLOTS) {
        int32_t k[SLOTS];
        unsigned long long sum[SLOTS], cnt[SLOTS];
#pragma unroll
        for (int u = 0; u < SLOTS; ++u) {
            const uint64_t i = i0 + 32 * u + lane;
            k[u] = i < hi && i < gt.cap ? gt.keys[i] : kEmptyKey;
        }
        uint32_t total = 0;
#pragma unroll
        for (int u = 0; u < SLOTS; ++u) {
            const uint64_t i = i0 + 32 * u + lane;
            const bool special = i == gt.cap && i < hi, slot = k[u] != kEmptyKey;
            sum[u] = special ? gt.special[0] : slot ? gt.sums[i] : 0ull;
            cnt[u] = special ? gt.special[1] : slot ? gt.counts[i] : 0ull;
        }
        unsigned m[SLOTS];
#pragma unroll
        for (int u = 0; u < SLOTS; ++u) {
            m[u] = __ballot_sync(0xffffffffu, cnt[u] != 0);
            total += __popc(m[u]);
        }
        if (total == 0) continue;
        uint32_t pos = 0;
        if (lane == 0) pos = atomicAdd(count, total);
        pos = __shfl_sync(0xffffffffu, pos, 0);
#pragma unroll
        for (int u = 0; u < SLOTS; ++u) {
            const uint64_t i = i0 + 32 * u + lane;
            const uint32_t at = pos + __popc(m[u] & ((1u << lane) - 1u));
            if (cnt[u] != 0) {
                if (at < capacity) rows[at] = mgv_group_row{k[u], 0, (int64_t)sum[u], (int64_t)cnt[u]};
                else set_error(err, kDevOverflow, 30);
                if (CLEAR) {
                    if (i == gt.cap) {
                        gt.special[0] = gt.special[1] = 0;
                    } else {
                        gt.keys[i] = kEmptyKey;
                        gt.sums[i] = 0;
                        gt.counts[i] = 0;
                    }
                }
            }
            pos += __popc(m[u]);
        }
    }
}

// Packs the groups of a table and empties its slots; the last CTA writes the
// header, when there is one, and readies the counters for the next close.
__global__ void __launch_bounds__(kPackBlock) k_group_pack(GroupTableView gt, mgv_group_row* __restrict__ rows,
                                                           uint32_t* count, GroupLanding* land, uint32_t* err) {
    for (uint64_t lo = (uint64_t)blockIdx.x * kPackBlock; lo <= gt.cap; lo += (uint64_t)gridDim.x * kPackBlock)
        pack_slots<true, 1>(gt, lo, min(lo + kPackBlock, (uint64_t)gt.cap + 1), rows, count, gt.cap + 1, err);
    if (!land) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(count + 1, 1u) == gridDim.x - 1) {  // every CTA has counted its groups
            land_header(land, err, atomicExch(count, 0u));
            count[1] = 0;
        }
    }
}

// Packs each query's groups into its output region (unsorted) and counts them.
__global__ void __launch_bounds__(kPackBlock) k_batch_compact(const BatchOut* __restrict__ outs,
                                                              const BatchItem* __restrict__ items, uint32_t nitems,
                                                              uint32_t* err) {
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        const BatchItem item = items[it];
        const BatchOut& o = outs[item.q];
        pack_slots<false, 8>(o.gt, item.lo, item.hi, o.rows, o.count, o.capacity, err);
    }
}

// A table emptied from any state.
__global__ void k_group_reset(GroupTableView gt, uint32_t* count) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < gt.cap; i += stride) {
        gt.keys[i] = kEmptyKey;
        gt.sums[i] = 0;
        gt.counts[i] = 0;
    }
    if (blockIdx.x == 0 && threadIdx.x < 2) {
        gt.special[threadIdx.x] = 0;
        count[threadIdx.x] = 0;
    }
}

size_t close_smem(uint32_t cap) { return kCntBytes + 2 * sizeof(unsigned long long) * ((size_t)cap + 1); }

}  // namespace

cudaError_t group_rows_init() {
    cudaError_t e = cudaFuncSetAttribute(k_group_close, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)close_smem(kSmallGroupCap));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_group_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortSmem);
    // the others are loaded now as well, not during an operator's first close
    cudaFuncAttributes fa;
    for (const void* k : {(const void*)k_group_pack, (const void*)k_group_emit, (const void*)k_group_reset})
        if (e == cudaSuccess) e = cudaFuncGetAttributes(&fa, k);
    return e;
}

cudaError_t launch_group_reset(const GroupTableView& gt, uint32_t* count, cudaStream_t s, Context* ctx) {
    const uint64_t want = ((uint64_t)gt.cap + 255) / 256;
    k_group_reset<<<(int)std::min<uint64_t>(want, (uint64_t)ctx->prop.multiProcessorCount * 8), 256, 0, s>>>(gt, count);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_group_close(const GroupTableView& gt, GroupLanding* land, bool sort, cudaStream_t s, Context* ctx) {
    k_group_close<<<1, kSortBlock, close_smem(gt.cap), s>>>(gt, land, sort ? 1u : 0u, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_group_pack(const GroupTableView& gt, mgv_group_row* rows, uint32_t* count, GroupLanding* land,
                              cudaStream_t s, Context* ctx) {
    const uint64_t want = ((uint64_t)gt.cap + kPackBlock) / kPackBlock;
    const int grid = (int)std::min<uint64_t>(want, (uint64_t)ctx->prop.multiProcessorCount * 8);
    k_group_pack<<<grid, kPackBlock, 0, s>>>(gt, rows, count, land, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_batch_compact(const BatchOut* d_outs, const BatchItem* items, uint32_t nitems, cudaStream_t s,
                                 Context* ctx) {
    if (nitems == 0) return cudaSuccess;
    const int grid = (int)std::min<uint64_t>((uint64_t)ctx->prop.multiProcessorCount * 4, nitems);
    k_batch_compact<<<grid, kPackBlock, 0, s>>>(d_outs, items, nitems, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_group_sort(const GroupSortJob* d_jobs, const GroupSortJob& job0, uint32_t njobs, uint32_t max_rows,
                              cudaStream_t s, Context* ctx) {
    if (njobs == 0) return cudaSuccess;
    const int grid = (int)std::min<uint32_t>(njobs, (uint32_t)ctx->prop.multiProcessorCount);
    k_group_sort<<<grid, kSortBlock, kSortSmem, s>>>(d_jobs, job0, njobs);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    // about two CTAs per SM over all jobs, and no more than the largest result has work for
    const uint32_t want = std::max<uint32_t>(1, 2 * (uint32_t)ctx->prop.multiProcessorCount / njobs);
    const uint32_t most = (max_rows + kEmitRows - 1) / kEmitRows;
    k_group_emit<<<dim3(njobs, std::min(want, most)), kEmitBlock, 0, s>>>(d_jobs, job0, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace mgv
