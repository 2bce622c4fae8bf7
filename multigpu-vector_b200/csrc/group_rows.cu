// group_rows.cu -- a closed group-by's rows: taken out of its hash table,
// ordered by group on the device and written straight into pinned, mapped
// host memory, with the table left empty for the next open.
//
// Ordering is an LSD radix sort of {group, source} pairs by one CTA per
// result: a result has at most a few tens of thousands of groups, so a
// device-wide sort would be launches and waits, and results of a batch run
// side by side on different SMs.  Only the bits in which the groups differ
// are sorted (dictionary codes below 65536 take two passes).  On the host the
// same sort cost about 35 us per 4096 groups and was half of a batch's time
// with its results read (366 K groups of 64 queries: 3.1 ms).
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
constexpr uint32_t kSmemPairs = kSmallGroupCap + 1;  // pairs sorted in shared memory (two buffers: 128 KiB)
constexpr size_t kSortSmem = kCntBytes + 2 * sizeof(unsigned long long) * kSmemPairs;

// {order-preserving group, source index}
__device__ __forceinline__ unsigned long long make_pair(int32_t group, uint32_t src) {
    return ((unsigned long long)((uint32_t)group ^ 0x80000000u) << 32) | src;
}
__device__ __forceinline__ int32_t pair_group(unsigned long long p) {
    return (int32_t)((uint32_t)(p >> 32) ^ 0x80000000u);
}

// Orders a[0..n) by group; the sorted pairs end in a or b, which is returned.
// Each warp owns a contiguous segment and places its pairs in order, so every
// pass is stable: counters are kept per (digit, warp) and scanned digit-major.
__device__ unsigned long long* sort_pairs(unsigned long long* a, unsigned long long* b, uint32_t n, uint32_t* cnt) {
    __shared__ uint32_t s_diff;
    const uint32_t lane = lane_id(), warp = threadIdx.x / 32;
    if (threadIdx.x == 0) s_diff = 0;
    __syncthreads();
    if (n < 2) return a;
    const uint32_t k0 = (uint32_t)(a[0] >> 32);
    uint32_t diff = 0;
    for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) diff |= (uint32_t)(a[i] >> 32) ^ k0;
    diff = __reduce_or_sync(0xffffffffu, diff);
    if (lane == 0 && diff) atomicOr(&s_diff, diff);
    __syncthreads();
    diff = s_diff;
    if (diff == 0) return a;
    if (n <= kRankSort) {  // few groups: each pair counts the smaller ones, one step instead of several per pass
        __syncthreads();
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
    const uint32_t low = __ffs(diff) - 1, bits = 32 - __clz(diff) - low;
    const uint32_t passes = (bits + 7) / 8, width = (bits + passes - 1) / passes, mask = (1u << width) - 1u;
    const uint32_t counters = (mask + 1) * kCntStride;
    const uint32_t per = ((n + kSortWarps - 1) / kSortWarps + 31) & ~31u;
    const uint32_t lo = min(n, warp * per), hi = min(n, lo + per);
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const uint32_t shift = 32 + low + pass * width;
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
    land->err[0] = err[0];
    land->err[1] = err[1];
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

// Orders packed rows, one CTA per job.
__global__ void __launch_bounds__(kSortBlock) k_group_sort(const GroupSortJob* __restrict__ jobs, GroupSortJob job0,
                                                           uint32_t njobs, const uint32_t* err) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t* cnt = reinterpret_cast<uint32_t*>(smem);
    for (uint32_t j = blockIdx.x; j < njobs; j += gridDim.x) {
        const GroupSortJob job = jobs ? jobs[j] : job0;
        const uint32_t found = *job.count, n = min(found, job.capacity);
        unsigned long long* a = n <= kSmemPairs ? reinterpret_cast<unsigned long long*>(smem + kCntBytes) : job.pairs;
        unsigned long long* b = n <= kSmemPairs ? a + kSmemPairs : job.pairs + job.capacity;
        __syncthreads();  // the previous job is done with the buffers
        for (uint32_t i = threadIdx.x; i < n; i += kSortBlock) a[i] = make_pair(job.rows[i].group, i);
        __syncthreads();
        a = sort_pairs(a, b, n, cnt);
        const unsigned long long* in = reinterpret_cast<const unsigned long long*>(job.rows);
        unsigned long long* out = reinterpret_cast<unsigned long long*>(job.out);
        unsigned long long* more = reinterpret_cast<unsigned long long*>(job.more);
        for (uint64_t w = threadIdx.x; w < 3ull * n; w += kSortBlock) {
            const uint32_t i = (uint32_t)(w / 3), f = (uint32_t)(w - 3ull * i);
            const unsigned long long v = in[3ull * (uint32_t)a[i] + f];
            if (i < job.out_rows) out[w] = v;
            else more[w - 3ull * job.out_rows] = v;
        }
        if (threadIdx.x == 0) {
            if (job.host_count) *job.host_count = found;
            if (job.land) {
                land_header(job.land, err, found);
                *job.count = 0;  // ready for the next close
            }
        }
    }
}

// Packs the groups of a table (the group INT32_MIN included) into rows, in
// slot order per warp, and empties their slots; the last CTA writes the
// header, when there is one, and readies the counters for the next close.
__global__ void k_group_pack(GroupTableView gt, mgv_group_row* __restrict__ rows, uint32_t* count, GroupLanding* land,
                             const uint32_t* err) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t end = ((uint64_t)gt.cap + 1 + 31) & ~31ull;  // whole warps take part in the ballots
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < end; i += stride) {
        const bool special = i == gt.cap;
        bool keep = false;
        mgv_group_row r{};
        if (i <= gt.cap) {
            r.group = special ? kEmptyKey : gt.keys[i];
            keep = special ? gt.special[1] != 0 : r.group != kEmptyKey;
            if (keep) {
                r.sum = (int64_t)(special ? gt.special[0] : gt.sums[i]);
                r.count = (int64_t)(special ? gt.special[1] : gt.counts[i]);
                if (special) {
                    gt.special[0] = gt.special[1] = 0;
                } else {
                    gt.keys[i] = kEmptyKey;
                    gt.sums[i] = 0;
                    gt.counts[i] = 0;
                }
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        uint32_t base = 0;
        if (lane_id() == 0 && m) base = atomicAdd(count, (uint32_t)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (keep) rows[base + __popc(m & ((1u << lane_id()) - 1u))] = r;
    }
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

int table_grid(const GroupTableView& gt, const Context* ctx) {
    const uint64_t want = ((uint64_t)gt.cap + 1 + 255) / 256;
    return (int)std::min<uint64_t>(want, (uint64_t)ctx->prop.multiProcessorCount * 8);
}

}  // namespace

cudaError_t group_rows_init() {
    cudaError_t e = cudaFuncSetAttribute(k_group_close, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortSmem);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_group_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSortSmem);
    return e;
}

cudaError_t launch_group_reset(const GroupTableView& gt, uint32_t* count, cudaStream_t s, Context* ctx) {
    k_group_reset<<<table_grid(gt, ctx), 256, 0, s>>>(gt, count);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_group_close(const GroupTableView& gt, GroupLanding* land, bool sort, cudaStream_t s, Context* ctx) {
    const size_t smem = kCntBytes + 2 * sizeof(unsigned long long) * ((size_t)gt.cap + 1);
    k_group_close<<<1, kSortBlock, smem, s>>>(gt, land, sort ? 1u : 0u, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_group_pack(const GroupTableView& gt, mgv_group_row* rows, uint32_t* count, GroupLanding* land,
                              cudaStream_t s, Context* ctx) {
    k_group_pack<<<table_grid(gt, ctx), 256, 0, s>>>(gt, rows, count, land, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_group_sort(const GroupSortJob* d_jobs, const GroupSortJob& job0, uint32_t njobs, cudaStream_t s,
                              Context* ctx) {
    if (njobs == 0) return cudaSuccess;
    const int grid = (int)std::min<uint32_t>(njobs, (uint32_t)ctx->prop.multiProcessorCount);
    k_group_sort<<<grid, kSortBlock, kSortSmem, s>>>(d_jobs, job0, njobs, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace mgv
