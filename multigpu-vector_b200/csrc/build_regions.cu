// build_regions.cu -- hash-table build through shared memory.
//
// Inserting build rows one 64-bit atomicCAS at a time into a table in global
// memory is bound by the L2's atomic throughput (about 20 G inserts/s on
// B200 even with the table in L2, and slower with more rows in flight).  Here
// the table is cut into regions of up to kRegionBuckets buckets (64 KiB) and
// built region by region in shared memory:
//   1. every row, packed {key, payload} (the key alone for a key-only table),
//      goes to its region's staging range.  k_region_tile_scatter sorts tiles
//      of thousands of rows by region in shared memory and stores runs: a lane per
//      row to a random address is bound by the memory pipeline's request rate
//      (4 M rows, 1024 regions: 57 us that way after a 17 us histogram and
//      scan).  Where the ranges lie:
//        - a table without a radix layout: the hash spreads its rows evenly,
//          so each region has a fixed share of the staging space, twice its
//          expected rows, and no row is counted beforehand; rows past the
//          share join the overflow list (step 3)
//        - a radix-laid-out table's regions follow the raw key bits, which may
//          be skewed: exact ranges, from a histogram and a scan
//          (k_region_hist, k_region_scan), or, for one run of a partition op
//          with whole-region slices, inside each partition's own range
//          (k_region_part_scatter, one CTA per partition, no global histogram)
//   2. k_region_build    one CTA per region: each row claims a slot with one
//                        shared atomicAdd on its bucket's fill counter (linear
//                        probing on a full bucket), one pass finds duplicate
//                        keys, and the region is written back with one bulk copy
//   3. k_region_overflow rows whose run leaves their region (rare) are
//                        inserted into the finished global table; its last CTA
//                        hands the table's counters to the host
// A table of one region and few rows is built by one CTA in one launch
// (k_build_small).
// The table is the same open-addressing table (hash_table.cuh): a row goes to
// the first empty slot of its run from its home bucket, slots fill in order,
// so probes are unchanged.  Rows with the reserved key INT32_MIN go to the
// side list during the scatter.
#include <cuda_runtime.h>

#include <algorithm>
#include <type_traits>

#include "device_common.cuh"
#include "hash_table.cuh"
#include "mgv_internal.h"

namespace mgv {
namespace {

constexpr int kRBlock = 512;       // histogram / scatter CTA
constexpr int kRBuildBlock = 512;  // region build CTA: a thread per 2 to 4 buckets
constexpr int kScanBlock = 1024;

// The job of item / region lookups, cached in shared memory by the caller.
__device__ __forceinline__ void load_job(RegionJob& dst, const RegionJob* jobs, const RegionJob& job0, uint32_t j) {
    static_assert(sizeof(RegionJob) % 4 == 0, "RegionJob is copied as 32-bit words");
    const uint32_t* src = jobs ? reinterpret_cast<const uint32_t*>(jobs + j) : reinterpret_cast<const uint32_t*>(&job0);
    for (uint32_t i = threadIdx.x; i < sizeof(RegionJob) / 4; i += blockDim.x) reinterpret_cast<uint32_t*>(&dst)[i] = src[i];
}

__device__ __forceinline__ BatchItem item_at(const BatchItem* items, uint32_t it, uint64_t n, uint64_t rpi) {
    if (items) return items[it];
    BatchItem b;
    b.q = 0;
    b.pad = 0;
    b.lo = (uint64_t)it * rpi;
    b.hi = min(n, b.lo + rpi);
    return b;
}

// Staging rows: {key, payload} as 8 bytes, or the key alone (4 bytes) for a
// key-only table -- half the scatter's stores and the build's loads.
template <bool KO>
__device__ __forceinline__ void stage_put(unsigned long long* staging, uint64_t pos, unsigned long long v) {
    if (KO) reinterpret_cast<uint32_t*>(staging)[pos] = (uint32_t)v;
    else staging[pos] = v;
}

template <bool KO>
__device__ __forceinline__ unsigned long long stage_get(const unsigned long long* staging, uint64_t i) {
    if (KO) return (unsigned long long)reinterpret_cast<const uint32_t*>(staging)[i];
    return staging[i];
}

// home_bucket (hash_table.cuh) and the region it lies in, with the table's
// constants in registers: a job in shared memory would be read again for every
// row, since the shared atomics between two rows could have changed it.
struct HomeFn {
    uint32_t radix_shift, radix_mask, bpp, shift;
    __device__ __forceinline__ explicit HomeFn(const RegionJob& j)
        : radix_shift(j.t.radix_shift), radix_mask(j.t.radix_mask), bpp(j.t.bpp), shift(j.shift) {}
    __device__ __forceinline__ uint32_t bucket(int32_t key) const {
        return (((uint32_t)key >> radix_shift) & radix_mask) * bpp + __umulhi(murmur32((uint32_t)key), bpp);
    }
    __device__ __forceinline__ uint32_t region(int32_t key) const { return bucket(key) >> shift; }
};

// Where a launch's rows go: staging and its region counters, and the rows
// for the global insert.
struct StageOut {
    const uint32_t* start;  // exact ranges: first staging row of each region; nullptr: job.stage0 + region * job.cap
    uint32_t* cursor;       // rows placed in each region so far
    unsigned long long* staging;
    unsigned long long* ovf;
    uint32_t* ovf_job;
    uint32_t* ctl;          // [0] rows in ovf, [1] CTAs done
};

__device__ __forceinline__ void overflow_put(const StageOut& o, unsigned long long v, uint32_t job) {
    const uint32_t i = atomicAdd(o.ctl, 1u);
    o.ovf[i] = v;
    if (o.ovf_job) o.ovf_job[i] = job;
}

// What a region build of several jobs leaves in the list when it has no job
// numbers of its own: the job above, below it the key of a key-only table's
// row, or the staging row (exact ranges: every row of the list is staged).
// The shared launch of a batch then takes 8 bytes a build row instead of 12.
template <bool KO>
__device__ __forceinline__ unsigned long long overflow_entry(uint32_t job, unsigned long long v, uint64_t staged) {
    return (unsigned long long)job << 32 | (KO ? (uint32_t)v : (uint32_t)staged);
}

// Row `i` of a region (counted from the region's first) into its range.
template <bool KO>
struct StageFn {
    const StageOut& o;
    const uint32_t* start;
    uint64_t stage0;
    uint32_t cap, q;
    __device__ __forceinline__ StageFn(const StageOut& out, const RegionJob& j, uint32_t job)
        : o(out), start(out.start ? out.start + j.region0 : nullptr), stage0(j.stage0), cap(j.cap), q(job) {}
    __device__ __forceinline__ void operator()(uint32_t region, uint32_t i, unsigned long long v) const {
        if (start) stage_put<KO>(o.staging, (uint64_t)start[region] + i, v);
        else if (i < cap) stage_put<KO>(o.staging, stage0 + (uint64_t)region * cap + i, v);
        else overflow_put(o, KO ? overflow_entry<KO>(q, v, 0) : v, q);
    }
};

// Loads of kPrefetch rows per thread are issued before any is used.
constexpr int kPrefetch = 8;

// Adds the item's rows to the shared per-region counters.
__device__ __forceinline__ void count_regions(const RegionJob& sj, const BatchItem& item, uint32_t* sh) {
    const HomeFn home(sj);
    for (uint64_t i0 = item.lo + threadIdx.x; i0 < item.hi; i0 += (uint64_t)kRBlock * kPrefetch) {
        int32_t key[kPrefetch];
        bool in[kPrefetch];
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u) {
            const uint64_t i = i0 + (uint64_t)u * kRBlock;
            in[u] = i < item.hi;
            key[u] = in[u] ? __ldg(sj.keys + i) : 0;
            if (in[u] && sj.filt) in[u] = __ldg(sj.filt + i) <= sj.bound;
        }
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u)
            if (in[u] && key[u] != kEmptyKey) atomicAdd(sh + home.region(key[u]), 1u);
    }
}

__global__ void __launch_bounds__(kRBlock) k_region_hist(const RegionJob* __restrict__ jobs, const __grid_constant__ RegionJob job0,
                                                         const BatchItem* __restrict__ items, uint32_t nitems,
                                                         uint64_t n, uint64_t rpi, uint32_t* __restrict__ hist) {
    extern __shared__ uint32_t sh[];
    __shared__ RegionJob sj;
    int64_t cur = -1;
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        const BatchItem item = item_at(items, it, n, rpi);
        __syncthreads();  // the previous item is done with sh and sj
        if ((int64_t)item.q != cur) {
            load_job(sj, jobs, job0, item.q);
            cur = item.q;
            __syncthreads();
        }
        for (uint32_t r = threadIdx.x; r < sj.nregions; r += kRBlock) sh[r] = 0;
        __syncthreads();
        count_regions(sj, item, sh);
        __syncthreads();
        for (uint32_t r = threadIdx.x; r < sj.nregions; r += kRBlock)
            if (sh[r]) atomicAdd(hist + sj.region0 + r, sh[r]);
    }
}

// One CTA: start[i] = sum of hist[0..i), start[regions] = total.
__global__ void __launch_bounds__(kScanBlock) k_region_scan(const uint32_t* __restrict__ hist, uint32_t regions,
                                                            uint32_t* __restrict__ start) {
    __shared__ uint32_t part[kScanBlock];
    const uint32_t per = (regions + kScanBlock - 1) / kScanBlock;
    const uint32_t lo = min(regions, threadIdx.x * per), hi = min(regions, lo + per);
    uint32_t sum = 0;
    for (uint32_t i = lo; i < hi; ++i) sum += hist[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t o = 1; o < kScanBlock; o <<= 1) {  // inclusive Hillis-Steele scan of the chunk sums
        const uint32_t add = threadIdx.x >= o ? part[threadIdx.x - o] : 0u;
        __syncthreads();
        part[threadIdx.x] += add;
        __syncthreads();
    }
    uint32_t run = part[threadIdx.x] - sum;
    for (uint32_t i = lo; i < hi; ++i) {
        start[i] = run;
        run += hist[i];
    }
    if (threadIdx.x == kScanBlock - 1) start[regions] = part[kScanBlock - 1];
}

// Rows to their regions' staging ranges one lane per row, for tables of more
// regions than a tile sorts (kTileRegions): per item, the rows per region are
// counted, one range per region is reserved, and shared cursors hand out its
// rows.
template <bool KO>
__global__ void __launch_bounds__(kRBlock) k_region_scatter(const RegionJob* __restrict__ jobs, const __grid_constant__ RegionJob job0,
                                                            const BatchItem* __restrict__ items, uint32_t nitems,
                                                            uint64_t n, uint64_t rpi, const __grid_constant__ StageOut out, uint32_t* err) {
    extern __shared__ uint32_t sh[];
    __shared__ RegionJob sj;
    int64_t cur = -1;
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        const BatchItem item = item_at(items, it, n, rpi);
        __syncthreads();
        if ((int64_t)item.q != cur) {
            load_job(sj, jobs, job0, item.q);
            cur = item.q;
            __syncthreads();
        }
        for (uint32_t r = threadIdx.x; r < sj.nregions; r += kRBlock) sh[r] = 0;
        __syncthreads();
        count_regions(sj, item, sh);
        __syncthreads();
        // one reservation per region and item; sh[r] becomes the region's next row
        for (uint32_t r = threadIdx.x; r < sj.nregions; r += kRBlock) {
            const uint32_t c = sh[r];
            if (c) sh[r] = atomicAdd(out.cursor + sj.region0 + r, c);
        }
        __syncthreads();
        const HomeFn home(sj);
        const StageFn<KO> stage(out, sj, item.q);
        for (uint64_t i0 = item.lo + threadIdx.x; i0 < item.hi; i0 += (uint64_t)kRBlock * kPrefetch) {
            int32_t key[kPrefetch], pay[kPrefetch];
            bool in[kPrefetch];
#pragma unroll
            for (int u = 0; u < kPrefetch; ++u) {
                const uint64_t i = i0 + (uint64_t)u * kRBlock;
                in[u] = i < item.hi;
                key[u] = in[u] ? __ldg(sj.keys + i) : 0;
                pay[u] = (in[u] && sj.pays) ? __ldg(sj.pays + i) : 0;
                if (in[u] && sj.filt) in[u] = __ldg(sj.filt + i) <= sj.bound;
            }
#pragma unroll
            for (int u = 0; u < kPrefetch; ++u) {
                if (!in[u]) continue;
                if (key[u] == kEmptyKey) {  // the side list (its duplicates are seen from its count)
                    bool dup, ok;
                    table_insert(sj.t, key[u], pay[u], err, dup, ok);
                    continue;
                }
                const uint32_t r = home.region(key[u]);
                const uint32_t i = atomicAdd(sh + r, 1u);
                stage(r, i, ((unsigned long long)(uint32_t)pay[u] << 32) | (uint32_t)key[u]);
            }
        }
    }
}

// ---- sorted tiles -------------------------------------------------------------

constexpr int kTileBlock = 512;
constexpr int kTileRows = 16;  // per thread, held in registers from load to placement
constexpr uint32_t kTileSize = kTileBlock * kTileRows;
constexpr uint32_t kTileRegions = 4096;   // most regions a tile sorts: runs of two rows on average
constexpr uint32_t kTileCounters = 1024;  // rank counters are replicated per lane while they are at most this many

// A tile's sorting space: two CTAs fit per SM up to 1024 regions.
template <bool KO>
struct TileSpace {
    typename std::conditional<KO, uint32_t, unsigned long long>::type* val;  // [kTileSize] rows in region order
    uint16_t* reg;     // [kTileSize] region of each sorted position
    uint32_t* off;     // [regions * copies] counts, then first sorted positions
    uint32_t* base;    // [regions] region row of sorted position 0 (mod 2^32)
    uint32_t copies;   // rank counters per region: lane & (copies - 1) picks one
};

__host__ __device__ constexpr uint32_t tile_copies(uint32_t regions) {
    uint32_t f = 1;
    while (f < 32 && 2 * f * regions <= kTileCounters) f *= 2;
    return f;
}
// Shared memory for jobs of up to `regions` regions: a smaller job may use more
// counters than the largest (200 regions x 4 copies, 128 x 8), but never more
// than kTileCounters while it has copies at all.
__host__ __device__ constexpr size_t tile_counter_bytes(uint32_t regions) {
    return 4ull * (regions > kTileCounters ? regions : kTileCounters);
}
constexpr bool tile_counters_fit() {
    for (uint32_t r = 1; r <= kTileRegions; ++r)
        if (4ull * r * tile_copies(r) > tile_counter_bytes(r)) return false;
    return true;
}
static_assert(tile_counters_fit(), "a job's counters fit the space of every launch it can be part of");
template <bool KO>
__host__ __device__ constexpr size_t tile_smem(uint32_t regions) {
    return (KO ? 6ull : 10ull) * kTileSize + tile_counter_bytes(regions) + 4ull * regions;
}
template <bool KO>
__device__ __forceinline__ TileSpace<KO> tile_space(unsigned char* base, uint32_t regions) {
    TileSpace<KO> s;
    s.val = reinterpret_cast<decltype(s.val)>(base);
    s.reg = reinterpret_cast<uint16_t*>(s.val + kTileSize);
    s.copies = tile_copies(regions);
    s.off = reinterpret_cast<uint32_t*>(s.reg + kTileSize);
    s.base = s.off + regions * s.copies;
    return s;
}

// One build row with the reserved key: the side list (its duplicates are seen
// from its count), as table_insert does it, without the rest of the insert.
__device__ __forceinline__ void side_list_row(const TableView& t, int32_t pay, uint32_t* err) {
    const unsigned long long i = atomicAdd(t.meta + 0, 1ull);
    atomicAdd(t.meta + 1, (unsigned long long)(long long)pay);
    if (i < t.side_cap) t.side_pay[i] = pay;
    else set_error(err, kDevTableFull, 1);
}

// Rows [lo, hi) (at most kTileSize) of a job to their regions: ranks by shared
// atomics, positions by a scan, one reserve(region, rows) -> first row per
// region, then put(region, row, value) in region order, so that a warp's
// stores are runs.  Every thread of the CTA calls it.
template <bool KO, class Region, class Reserve, class Put>
__device__ __forceinline__ void sort_tile(const RegionJob& job, const TileSpace<KO>& ts, uint32_t regions, uint64_t lo,
                                          uint64_t hi, uint32_t* err, uint32_t* side_rows, Region region,
                                          Reserve reserve, Put put) {
    __syncthreads();  // the previous tile is stored
    for (uint32_t r = threadIdx.x; r < regions * ts.copies; r += kTileBlock) ts.off[r] = 0;
    const uint32_t n = (uint32_t)(hi - lo);
    const int32_t* const keys = job.keys + lo;
    const int32_t* const pays = !KO && job.pays ? job.pays + lo : nullptr;
    const int32_t* const filt = job.filt ? job.filt + lo : nullptr;
    const int32_t bound = job.bound;
    int32_t key[kTileRows], pay[kTileRows];
    uint32_t at[kTileRows];  // region << 16 | rank, ~0 for no row
#pragma unroll
    for (int u = 0; u < kTileRows; ++u) {
        const uint32_t i = u * kTileBlock + threadIdx.x;
        key[u] = i < n ? __ldg(keys + i) : kEmptyKey;
        pay[u] = pays && i < n ? __ldg(pays + i) : 0;
        at[u] = filt && i < n && __ldg(filt + i) > bound ? ~0u : 0u;
    }
    __syncthreads();
    const uint32_t copy = lane_id() & (ts.copies - 1);
    bool reserved = false;
#pragma unroll
    for (int u = 0; u < kTileRows; ++u) {
        reserved |= key[u] == kEmptyKey && u * kTileBlock + threadIdx.x < n;
        at[u] = at[u] == 0 && key[u] != kEmptyKey ? region(key[u]) << 16 : ~0u;
    }
#pragma unroll
    for (int u = 0; u < kTileRows; ++u)
        if (at[u] != ~0u) at[u] |= atomicAdd(ts.off + (at[u] >> 16) * ts.copies + copy, 1u);
    if (reserved) {  // rare: the rows are read again, so that the common path holds nothing for them
#pragma unroll 1
        for (uint32_t i = threadIdx.x; i < n; i += kTileBlock) {
            if (__ldg(keys + i) != kEmptyKey || (filt && __ldg(filt + i) > bound)) continue;
            side_list_row(job.t, job.pays ? __ldg(job.pays + lo + i) : 0, err);
            if (side_rows) atomicAdd(side_rows, 1u);
        }
    }
    __syncthreads();
    const uint32_t total = block_exclusive_scan<kTileBlock>(ts.off, regions * ts.copies);
    for (uint32_t r = threadIdx.x; r < regions; r += kTileBlock) {
        const uint32_t first = ts.off[r * ts.copies];
        const uint32_t c = (r + 1 < regions ? ts.off[(r + 1) * ts.copies] : total) - first;
        ts.base[r] = (c ? reserve(r, c) : 0u) - first;
    }
#pragma unroll
    for (int u = 0; u < kTileRows; ++u) {
        if (at[u] == ~0u) continue;
        const uint32_t r = at[u] >> 16, p = ts.off[r * ts.copies + copy] + (at[u] & 0xffffu);
        if constexpr (KO) ts.val[p] = (uint32_t)key[u];
        else ts.val[p] = ((unsigned long long)(uint32_t)pay[u] << 32) | (uint32_t)key[u];
        ts.reg[p] = (uint16_t)r;
    }
    __syncthreads();
#pragma unroll 4
    for (uint32_t j = threadIdx.x; j < total; j += kTileBlock) {
        const uint32_t r = ts.reg[j];
        put(r, ts.base[r] + j, (unsigned long long)ts.val[j]);
    }
}

template <bool KO>
__global__ void __launch_bounds__(kTileBlock, 2)
    k_region_tile_scatter(const RegionJob* __restrict__ jobs, const __grid_constant__ RegionJob job0, const BatchItem* __restrict__ items,
                          uint32_t nitems, uint64_t n, uint64_t rpi, const __grid_constant__ StageOut out, uint32_t* err) {
    extern __shared__ __align__(16) unsigned char tile_raw[];
    __shared__ RegionJob sj;
    int64_t cur = -1;
    for (uint32_t it = blockIdx.x; it < nitems; it += gridDim.x) {
        const BatchItem item = item_at(items, it, n, rpi);
        if ((int64_t)item.q != cur) {
            __syncthreads();  // the previous job's tile is stored
            load_job(sj, jobs, job0, item.q);
            cur = item.q;
            __syncthreads();
        }
        const TileSpace<KO> ts = tile_space<KO>(tile_raw, sj.nregions);
        const HomeFn home(sj);
        const StageFn<KO> stage(out, sj, item.q);
        uint32_t* const cursor = out.cursor + sj.region0;
        for (uint64_t lo = item.lo; lo < item.hi; lo += kTileSize)
            sort_tile<KO>(sj, ts, sj.nregions, lo, min(item.hi, lo + kTileSize), err, nullptr,
                          [&](int32_t key) { return home.region(key); },
                          [&](uint32_t r, uint32_t c) { return atomicAdd(cursor + r, c); }, stage);
    }
}

__device__ __forceinline__ uint32_t job_of_region(const RegionJob* jobs, uint32_t njobs, uint32_t g) {
    uint32_t lo = 0, hi = njobs;  // last job whose region0 <= g
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (jobs[mid].region0 <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// 16-byte shared-memory read.
__device__ __forceinline__ uint4 lds_v4(const void* p) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "r"(smem_u32(p))
                 : "memory");
    return r;
}

// Slots per bucket: 4 {key, payload} slots, or 8 keys in a key-only table.
template <bool KO>
constexpr uint32_t slots_per_bucket() { return KO ? 8u : 4u; }

// The key words of shared bucket b (4, or 8 for a key-only table).
template <bool KO>
__device__ __forceinline__ void bucket_keys(const unsigned long long* tab, uint32_t b,
                                            uint32_t (&k)[slots_per_bucket<KO>()]) {
    const uint32_t* words = reinterpret_cast<const uint32_t*>(tab) + 8 * b;
    const uint4 s01 = lds_v4(words), s23 = lds_v4(words + 4);
    if constexpr (KO) {
        k[0] = s01.x; k[1] = s01.y; k[2] = s01.z; k[3] = s01.w;
        k[4] = s23.x; k[5] = s23.y; k[6] = s23.z; k[7] = s23.w;
    } else {
        k[0] = s01.x;
        k[1] = s01.z;
        k[2] = s23.x;
        k[3] = s23.z;
    }
}

// Inserts one staged row into the shared region.  fill[b] counts the rows
// that asked bucket b for a slot: the first four (eight in a key-only table)
// get slots 0, 1, ... in that order (so slots fill as a prefix, as the global
// insert leaves them), later ones move on to the next bucket.  A bucket that
// has turned a row away stays full, so every row ends in the first bucket of
// its run that had room.
template <bool KO>
__device__ __forceinline__ void region_put(unsigned long long* tab, uint32_t b, uint32_t q, unsigned long long v) {
    if (KO) reinterpret_cast<uint32_t*>(tab)[8 * b + q] = (uint32_t)v;  // the key alone
    else tab[4 * b + q] = v;
}
template <bool KO>
__device__ __forceinline__ bool region_insert(unsigned long long* tab, uint32_t* fill, uint32_t nb, uint32_t b,
                                              unsigned long long v) {
    for (; b < nb; ++b) {
        const uint32_t q = atomicAdd(fill + b, 1u);
        if (q < slots_per_bucket<KO>()) {
            region_put<KO>(tab, b, q, v);
            return true;
        }
    }
    return false;  // the run leaves the region
}

// Whether the table region holds two rows of one key: in one bucket, or in a
// full bucket and the buckets after it up to the first one that is not full.
// Two rows with one key share their home bucket, and every bucket between the
// two is full, so this finds every duplicate pair inside the region.  wrap:
// the region is the whole table, whose runs go round its end.  A lane looks
// into one bucket and, when it is full, walks on.  Of 8-slot buckets few are
// full at the usual load factors (1.6 of 32 at 0.5): those are compared with
// their successors by the whole warp, two pairs of keys a lane, instead of 64
// pairs by one or two of its lanes (2^24 keys: 133 -> 106 us); of 4-slot
// buckets more are (4.5 of 32), with 16 pairs each.
template <bool KO>
__device__ __forceinline__ bool region_has_dup(const unsigned long long* tab, const uint32_t* fill, uint32_t nb, bool wrap) {
    constexpr uint32_t S = slots_per_bucket<KO>();
    constexpr int kWarpWise = KO ? 4 : 0;  // full buckets of 32 that the warp takes one by one
    const uint32_t lane = lane_id();
    const uint32_t* words = reinterpret_cast<const uint32_t*>(tab);
    bool dup = false;
    // the bucket `step` after f; false past the region's end
    auto after = [&](uint32_t f, uint32_t step, uint32_t& c) {
        c = f + step;
        if (c < nb) return true;
        c -= nb;
        return wrap;
    };
    for (uint32_t b0 = threadIdx.x & ~31u; b0 < nb; b0 += blockDim.x) {
        const uint32_t b = b0 + lane;
        const uint32_t n = b < nb ? min(fill[b], S) : 0u;
        uint32_t k[S];
        if (n > 1) {
            bucket_keys<KO>(tab, b, k);
#pragma unroll
            for (int j = 1; j < (int)S; ++j) {
                bool eq = false;
#pragma unroll
                for (int i = 0; i < j; ++i) eq |= k[i] == k[j];
                dup |= eq && (uint32_t)j < n;
            }
        }
        unsigned full = __ballot_sync(0xffffffffu, n == S);
        if (__popc(full) > kWarpWise) {
            uint32_t c;
            for (uint32_t step = 1; n == S && !dup && step < nb && after(b, step, c); ++step) {
                const uint32_t m = min(fill[c], S);
                uint32_t o[S];
                bucket_keys<KO>(tab, c, o);
#pragma unroll
                for (int j = 0; j < (int)S; ++j) {
                    bool eq = false;
#pragma unroll
                    for (int i = 0; i < (int)S; ++i) eq |= k[i] == o[j];
                    dup |= eq && (uint32_t)j < m;
                }
                if (m < S) break;
            }
            continue;
        }
        for (; full; full &= full - 1) {
            const uint32_t f = b0 + __ffs(full) - 1;
            const uint32_t key = words[8 * f + lane / 4], j0 = lane % 4 * 2;  // against keys j0 and j0 + 1
            uint32_t c;
            for (uint32_t step = 1; step < nb && after(f, step, c); ++step) {
                const uint32_t m = min(fill[c], S);
                dup |= (j0 < m && words[8 * c + j0] == key) || (j0 + 1 < m && words[8 * c + j0 + 1] == key);
                if (m < S) break;
            }
        }
    }
    return dup;
}

// nb empty buckets in shared memory.
__device__ __forceinline__ void clear_table(unsigned long long* tab, uint32_t nb) {
    const uint4 empty = make_uint4(0x80000000u, 0x80000000u, 0x80000000u, 0x80000000u);  // 2 x kEmptySlot
    static_assert(kEmptySlot == 0x8000000080000000ull, "empty slot pattern");
    for (uint32_t w = threadIdx.x; w < 2 * nb; w += blockDim.x) reinterpret_cast<uint4*>(tab)[w] = empty;
}

// Staging rows per thread in one load batch.  Few: at 40 registers (three CTAs)
// the whole region's rows, 16 keys or 8 {key, payload}, spilled, and with the
// tables in shared memory there is hardly an L1 for spills (2^22 {key, payload}
// rows 51 -> 41 us, 2^24 keys 107 -> 92 us).
template <bool KO>
constexpr int region_batch() { return KO ? 4 : 2; }

// A region's staging rows.
struct RegionRows {
    uint64_t lo;
    uint32_t n;
};
__device__ __forceinline__ RegionRows region_rows(const StageOut& o, const RegionJob& job, uint32_t g) {
    if (o.start) return RegionRows{o.start[g], o.start[g + 1] - o.start[g]};
    return RegionRows{job.stage0 + (uint64_t)(g - job.region0) * job.cap, min(o.cursor[g], job.cap)};
}

// The next region of this CTA at or after g (stride gridDim.x); without
// `fresh`, regions that receive no rows are left as they are.
__device__ __forceinline__ uint32_t next_region(uint32_t g, uint32_t regions, const StageOut& o, uint32_t fresh) {
    for (; g < regions; g += gridDim.x)
        if (fresh || (o.start ? o.start[g] != o.start[g + 1] : o.cursor[g] != 0)) return g;
    return regions;
}

// A region's rows from `from` on, one load batch, into registers (past the
// last they read as empty).
template <bool KO, class T>
__device__ __forceinline__ void load_region_rows(const unsigned long long* staging, const RegionRows& rr, uint32_t from,
                                                 T (&v)[region_batch<KO>()]) {
#pragma unroll
    for (int u = 0; u < region_batch<KO>(); ++u) {
        const uint32_t i = from + threadIdx.x + u * blockDim.x;
        v[u] = i < rr.n ? (T)stage_get<KO>(staging, rr.lo + i) : (T)kEmptySlot;
    }
}

// Regions one at a time per CTA, several CTAs per SM; the next region's
// first rows are loaded into registers before this region's duplicate pass
// and bulk store, so their latency overlaps that work.  The phases of a
// region are separated by barriers, so the SM is kept busy by its other CTAs
// (three of 512 threads with 64 KiB regions; small tables use smaller regions
// and CTAs, so that every SM has some).
template <bool KO>
__global__ void __launch_bounds__(kRBuildBlock, 3) k_region_build(const RegionJob* __restrict__ jobs, const __grid_constant__ RegionJob job0,
                                                                  uint32_t njobs, uint32_t regions, const __grid_constant__ StageOut out,
                                                                  uint32_t fresh, uint32_t* err) {
    using Row = typename std::conditional<KO, uint32_t, unsigned long long>::type;
    extern __shared__ __align__(128) unsigned long long tab[];  // the region's slots, then the fill counters
    __shared__ RegionJob sj;
    __shared__ __align__(8) uint64_t bar;
    const uint32_t T = blockDim.x;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    uint32_t phase = 0;
    int64_t cur = -1;
    uint32_t g = next_region(blockIdx.x, regions, out, fresh);
    uint32_t j = (jobs && njobs > 1 && g < regions) ? job_of_region(jobs, njobs, g) : 0u;
    RegionRows rr{0, 0};
    Row v[region_batch<KO>()];
    if (g < regions) {
        rr = region_rows(out, *(jobs ? jobs + j : &job0), g);
        load_region_rows<KO>(out.staging, rr, 0, v);
    }
    while (g < regions) {
        __syncthreads();  // the previous region's store has read the buffer; sj is free
        if ((int64_t)j != cur) {
            load_job(sj, jobs, job0, j);
            cur = j;
            __syncthreads();
        }
        const HomeFn home(sj);
        const uint32_t rb = 1u << sj.shift;
        const uint32_t b0 = (g - sj.region0) << sj.shift;
        const uint32_t nb = min(rb, sj.t.nbuckets - b0);
        uint32_t* fill = reinterpret_cast<uint32_t*>(tab + 4 * rb);
        unsigned long long* gslots = sj.t.slots + 4ull * b0;
        if (fresh) {
            clear_table(tab, nb);
            for (uint32_t b = threadIdx.x; b < nb; b += T) fill[b] = 0;
        } else {
            if (threadIdx.x == 0) {  // the region's current contents, one bulk copy
                mbar_expect_tx(&bar, nb * 32);
                bulk_g2s(tab, gslots, nb * 32, &bar);
            }
            if (!mbar_wait_bounded(&bar, phase, 1u << 24)) {
                if (threadIdx.x == 0) {
                    set_error(err, kDevTimeout, 40);
                    bulk_wait_all();
                }
                return;
            }
            phase ^= 1u;
            // slots fill as a prefix: a bucket's count is the index of its first empty slot
            for (uint32_t b = threadIdx.x; b < nb; b += T) {
                uint32_t k[slots_per_bucket<KO>()];
                bucket_keys<KO>(tab, b, k);
                uint32_t n = 0;
#pragma unroll
                for (int q = 0; q < (int)slots_per_bucket<KO>(); ++q) n += k[q] != (uint32_t)kEmptyKey;
                fill[b] = n;
            }
        }
        __syncthreads();
        uint32_t ins = 0;
        for (uint32_t from = 0;;) {
#pragma unroll
            for (int u = 0; u < region_batch<KO>(); ++u) {
                // past the region, or a gap slot of a partition's range (the
                // reserved key goes to the side list, never into staging)
                if ((int32_t)(uint32_t)v[u] == kEmptyKey) continue;
                if (region_insert<KO>(tab, fill, nb, home.bucket((int32_t)(uint32_t)v[u]) - b0, v[u])) ++ins;
                else if (jobs && !out.ovf_job)  // the run leaves the region
                    overflow_put(out, overflow_entry<KO>(j, v[u], rr.lo + from + threadIdx.x + u * T), j);
                else overflow_put(out, v[u], j);
            }
            from += T * region_batch<KO>();
            if (from >= rr.n) break;
            load_region_rows<KO>(out.staging, rr, from, v);  // a large region
        }
        __syncthreads();
        const uint32_t gn = next_region(g + gridDim.x, regions, out, fresh);
        const uint32_t jn = (jobs && njobs > 1 && gn < regions) ? job_of_region(jobs, njobs, gn) : 0u;
        if (gn < regions) {
            rr = region_rows(out, *(jobs ? jobs + jn : &job0), gn);
            load_region_rows<KO>(out.staging, rr, 0, v);  // in flight from here on
        }
        const bool dup = region_has_dup<KO>(tab, fill, nb, false);
        fence_proxy_async_smem();  // the inserts, before the bulk store reads them
        __syncthreads();
        if (threadIdx.x == 0) {
            bulk_s2g(gslots, tab, nb * 32);
            bulk_commit();
            bulk_wait_reads();  // the buffer may be refilled; the write itself completes in the background
        }
        const unsigned long long tot = warp_sum_u64(ins);
        const bool any_dup = __any_sync(0xffffffffu, dup);
        if (lane_id() == 0) {
            if (tot) atomicAdd(sj.t.meta + 2, tot);
            if (any_dup) atomicOr(sj.t.meta + 3, 1ull);
        }
        g = gn;
        j = jn;
    }
    if (threadIdx.x == 0) bulk_wait_all();  // every region store is complete before the CTA ends
}

// The table's counters and the error word, to the host.  All six are read
// before the first is written: the host's words might alias them for all the
// compiler knows, and each read would wait for the one before it.
__device__ __forceinline__ void land_words(TableLanding* land, const unsigned long long (&meta)[4], const uint32_t* err) {
    const uint32_t e0 = *((volatile const uint32_t*)err), e1 = *((volatile const uint32_t*)(err + 1));
    land->err[0] = e0;
    land->err[1] = e1;
#pragma unroll
    for (int i = 0; i < 4; ++i) land->meta[i] = meta[i];
}
// own: the table's counters if t.meta was kept elsewhere during the build.
__device__ __forceinline__ void land_table(TableLanding* land, const TableView& t, unsigned long long* own, const uint32_t* err) {
    unsigned long long meta[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) meta[i] = *((volatile unsigned long long*)(t.meta + i));
    land_words(land, meta, err);
    if (own != t.meta) {
#pragma unroll
        for (int i = 0; i < 4; ++i) own[i] = meta[i];
    }
}

// Rows whose run left their region, into the global table; the last CTA then
// lands the table's counters (land != nullptr: one table) and leaves the
// scratch zeroed: the memsets it saves were 1.5 us each on the device and as
// much between them.  Few rows come here
// and none waits for another's; what takes the time is a chain of round trips
// (the list, the home bucket, the run, the claims lost to rows of the same
// run).  Reading four buckets of the run at once did not shorten it: 12.3 us for
// 12.2 at 2^22 distinct keys, 22.3 for 21.1 at 300 K rows of 100 K keys.
__global__ void k_region_overflow(const RegionJob* __restrict__ jobs, const __grid_constant__ RegionJob job0, const __grid_constant__ StageOut out, TableLanding* land,
                                  unsigned long long* meta, uint32_t zero_words, uint32_t* err) {
    __shared__ uint32_t s_last;
    const uint32_t cnt = *out.ctl;
    for (uint32_t x = blockIdx.x * blockDim.x + threadIdx.x; x < cnt; x += gridDim.x * blockDim.x) {
        unsigned long long v = out.ovf[x];
        uint32_t j = 0;
        if (jobs) {
            j = out.ovf_job ? out.ovf_job[x] : (uint32_t)(v >> 32);
            if (!out.ovf_job && !job0.t.key_only) v = out.staging[(uint32_t)v];
        }
        const TableView t = jobs ? jobs[j].t : job0.t;
        bool dup = false, ok = false;
        table_insert(t, (int32_t)(uint32_t)v, (int32_t)(uint32_t)(v >> 32), err, dup, ok);
        if (ok) atomicAdd(t.meta + 2, 1ull);
        if (dup) atomicOr(t.meta + 3, 1ull);
    }
    if (!land) return;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(out.ctl + 1, 1u) == gridDim.x - 1;
        if (s_last) {
            __threadfence();
            land_table(land, job0.t, meta, err);
        }
    }
    __syncthreads();
    if (!s_last) return;
    // every other CTA is done with the scratch: zero for the next build
    for (uint32_t i = threadIdx.x; i < zero_words; i += blockDim.x) out.cursor[i] = 0;
}

__global__ void k_table_land(TableView t, TableLanding* land, const uint32_t* err) {
    if (threadIdx.x == 0) land_table(land, t, t.meta, err);
}

// A table of one region built from all its rows by one CTA: clear, insert,
// duplicates, store, counters and the hand-over to the host in one launch.
// Runs wrap around the table here, as they do in the global insert.
constexpr int kSmallBlock = 1024;
template <bool KO>
__global__ void __launch_bounds__(kSmallBlock) k_build_small(const __grid_constant__ RegionJob job, uint32_t n, TableLanding* land, uint32_t* err) {
    extern __shared__ __align__(128) unsigned long long tab[];
    const uint32_t nb = job.t.nbuckets;
    uint32_t* fill = reinterpret_cast<uint32_t*>(tab + 4 * nb);
    __shared__ uint32_t s_side, s_ins, s_dup;
    __shared__ unsigned long long s_side_sum;
    if (threadIdx.x == 0) {
        s_side = s_ins = s_dup = 0;
        s_side_sum = 0;
    }
    clear_table(tab, nb);
    for (uint32_t b = threadIdx.x; b < nb; b += kSmallBlock) fill[b] = 0;
    __syncthreads();
    uint32_t ins = 0;
    for (uint32_t i0 = threadIdx.x; i0 < n; i0 += kSmallBlock * kPrefetch) {
        int32_t key[kPrefetch], pay[kPrefetch];
        bool in[kPrefetch];
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u) {
            const uint32_t i = i0 + u * kSmallBlock;
            in[u] = i < n;
            key[u] = in[u] ? __ldg(job.keys + i) : 0;
            pay[u] = (in[u] && job.pays) ? __ldg(job.pays + i) : 0;
            if (in[u] && job.filt) in[u] = __ldg(job.filt + i) <= job.bound;
        }
#pragma unroll
        for (int u = 0; u < kPrefetch; ++u) {
            if (!in[u]) continue;
            if (key[u] == kEmptyKey) {
                const uint32_t at = atomicAdd(&s_side, 1u);
                atomicAdd(&s_side_sum, (unsigned long long)(long long)pay[u]);
                if (at < job.t.side_cap) job.t.side_pay[at] = pay[u];
                else set_error(err, kDevTableFull, 1);
                continue;
            }
            const unsigned long long v = ((unsigned long long)(uint32_t)pay[u] << 32) | (uint32_t)key[u];
            const uint32_t hb = home_bucket(key[u], job.t);
            if (region_insert<KO>(tab, fill, nb, hb, v) || region_insert<KO>(tab, fill, hb, 0, v)) ++ins;
            else set_error(err, kDevTableFull, 2);
        }
    }
    __syncthreads();
    const bool dup = region_has_dup<KO>(tab, fill, nb, true);
    fence_proxy_async_smem();
    ins = __reduce_add_sync(0xffffffffu, ins);
    if (lane_id() == 0 && ins) atomicAdd(&s_ins, ins);
    if (dup) s_dup = 1;
    __syncthreads();
    if (threadIdx.x == 0) {
        bulk_s2g(job.t.slots, tab, nb * 32);
        bulk_commit();
        const unsigned long long meta[4] = {s_side, s_side_sum, s_ins, s_dup};
#pragma unroll
        for (int i = 0; i < 4; ++i) job.t.meta[i] = meta[i];
        land_words(land, meta, err);
        bulk_wait_all();
    }
}

// ---- staging of a partition op's single run ---------------------------------
//
// A partition op's single run gives each partition's rows as one range
// [ends[p-1], ends[p]), and when the table's partition slices are whole
// regions (bpp a multiple of kRegionBuckets) every region lies in one
// partition.  One CTA per partition then counts its rows per region in
// shared memory, and stages them region-major inside the partition's own
// range -- the regions' starts are the range's start plus a prefix sum, so
// no global histogram, scan or cursor is needed, and the partition's rows
// (just written by the partition op) are read from L2 twice.  Rows with the
// reserved key go to the side list; their slots at the range's end are
// filled with the reserved key, which the region build skips.  The rows are
// staged in sorted tiles (2^24 keys, 8 regions a partition: 89 us with a
// match and a shared atomic per row of a warp).
template <bool KO>
__global__ void __launch_bounds__(kTileBlock, 2) k_region_part_scatter(const __grid_constant__ RegionJob job,
                                                                       const unsigned long long* __restrict__ ends,
                                                                       uint32_t P, uint32_t rpp,
                                                                       uint32_t* __restrict__ start,
                                                                       unsigned long long* __restrict__ staging,
                                                                       uint32_t* err) {
    extern __shared__ __align__(16) unsigned char part_raw[];  // the tile space, then a row cursor per region
    const TileSpace<KO> ts = tile_space<KO>(part_raw, rpp);
    uint32_t* cur = ts.base + rpp;
    __shared__ uint32_t side_rows;
    const uint32_t bpp = job.t.bpp, copy = lane_id() & (ts.copies - 1);
    auto region = [&](int32_t key) { return __umulhi(murmur32((uint32_t)key), bpp) / kRegionBuckets; };
    for (uint32_t p = blockIdx.x; p < P; p += gridDim.x) {
        const uint64_t lo = p ? ends[p - 1] : 0ull, hi = ends[p];
        __syncthreads();  // the previous partition is done with the counters
        for (uint32_t r = threadIdx.x; r < rpp * ts.copies; r += kTileBlock) ts.off[r] = 0;
        if (threadIdx.x == 0) side_rows = 0;
        __syncthreads();
        // 1. rows per region
        for (uint64_t i0 = lo + threadIdx.x; i0 < hi; i0 += kTileSize) {
            int32_t key[kTileRows];
#pragma unroll
            for (int u = 0; u < kTileRows; ++u) {
                const uint64_t i = i0 + (uint64_t)u * kTileBlock;
                key[u] = i < hi ? __ldg(job.keys + i) : kEmptyKey;
            }
#pragma unroll
            for (int u = 0; u < kTileRows; ++u)
                if (key[u] != kEmptyKey) atomicAdd(ts.off + region(key[u]) * ts.copies + copy, 1u);
        }
        __syncthreads();
        // the regions' starts inside the partition's range
        block_exclusive_scan<kTileBlock>(ts.off, rpp * ts.copies);
        for (uint32_t r = threadIdx.x; r < rpp; r += kTileBlock) {
            cur[r] = (uint32_t)lo + ts.off[r * ts.copies];
            start[(uint64_t)p * rpp + r] = cur[r];
        }
        if (p == P - 1 && threadIdx.x == 0) start[(uint64_t)P * rpp] = (uint32_t)hi;
        // 2. the rows, region-major
        for (uint64_t t0 = lo; t0 < hi; t0 += kTileSize)
            sort_tile<KO>(job, ts, rpp, t0, min(hi, t0 + kTileSize), err, &side_rows, region,
                          [&](uint32_t r, uint32_t c) {  // one thread per region: no atomic
                              const uint32_t at = cur[r];
                              cur[r] = at + c;
                              return at;
                          },
                          [&](uint32_t, uint32_t i, unsigned long long v) { stage_put<KO>(staging, i, v); });
        __syncthreads();
        // the reserved-key rows' slots at the end of the range
        const uint32_t nside = side_rows;
        for (uint32_t k = threadIdx.x; k < nside; k += kTileBlock)
            stage_put<KO>(staging, hi - nside + k, kEmptySlot);
    }
}

}  // namespace

bool region_build_partitioned_fits(const TableView& t) {
    return t.bpp % kRegionBuckets == 0 && t.bpp / kRegionBuckets <= kTileRegions;
}

static StageOut stage_out(const RegionScratch& sc, bool exact) {
    return StageOut{exact ? sc.start : nullptr, sc.cursor, sc.staging, sc.ovf, sc.ovf_job, sc.ctl};
}

// Shared memory of k_region_build for regions of 2^shift buckets.
static size_t region_smem(uint32_t shift) { return (32ull + 4ull) << shift; }

// The region build and the global insert of what it leaves.
static cudaError_t build_staged(const RegionJob* d_jobs, const RegionJob& job0, uint32_t njobs, uint32_t regions,
                                uint32_t shift, const StageOut& out, bool fresh, TableLanding* land,
                                unsigned long long* meta, cudaStream_t s, Context* ctx) {
    const bool ko = job0.t.key_only != 0;
    const void* kb = ko ? (const void*)k_region_build<true> : (const void*)k_region_build<false>;
    const size_t smem = region_smem(shift);
    const int block = (int)std::min((uint32_t)kRBuildBlock, (1u << shift) / 2);
    const int grid = (int)std::min<uint64_t>(regions, (uint64_t)occupancy_grid(kb, block, smem, ctx));
    if (ko) k_region_build<true><<<grid, block, smem, s>>>(d_jobs, job0, njobs, regions, out, fresh ? 1u : 0u, ctx->d_err);
    else k_region_build<false><<<grid, block, smem, s>>>(d_jobs, job0, njobs, regions, out, fresh ? 1u : 0u, ctx->d_err);
    ctx->launches++;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_region_overflow<<<ctx->prop.multiProcessorCount, 256, 0, s>>>(d_jobs, job0, out, land, meta,
                                                                   (uint32_t)(region_zero_bytes(regions) / 4), ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t region_build_init() {
    const size_t tab = region_smem(kRegionShift), tile_ko = tile_smem<true>(kTileRegions) + 4 * kTileRegions,
                 tile = tile_smem<false>(kTileRegions) + 4 * kTileRegions, hist = 4ull * kMaxRegionsPerJob;
    const struct {
        const void* k;
        size_t smem;
    } all[] = {{(const void*)k_region_hist, hist},
               {(const void*)k_region_scatter<true>, hist},
               {(const void*)k_region_scatter<false>, hist},
               {(const void*)k_region_tile_scatter<true>, tile_ko},
               {(const void*)k_region_tile_scatter<false>, tile},
               {(const void*)k_region_part_scatter<true>, tile_ko},
               {(const void*)k_region_part_scatter<false>, tile},
               {(const void*)k_region_build<true>, tab},
               {(const void*)k_region_build<false>, tab},
               {(const void*)k_build_small<true>, tab},
               {(const void*)k_build_small<false>, tab}};
    for (const auto& x : all) {
        const cudaError_t e = cudaFuncSetAttribute(x.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)x.smem);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_build_regions_partitioned(const RegionJob& table_job, const unsigned long long* ends, uint64_t n,
                                             const RegionScratch& sc, TableLanding* land, bool zeroed, cudaStream_t s,
                                             Context* ctx) {
    RegionJob job = table_job;
    job.t.meta = sc.meta;
    const uint32_t P = job.t.radix_mask + 1;
    const uint32_t rpp = job.t.bpp / kRegionBuckets;
    const uint32_t regions = P * rpp;
    const bool ko = job.t.key_only != 0;
    cudaError_t e;
    if (!zeroed && (e = cudaMemsetAsync(sc.cursor, 0, region_zero_bytes(regions), s))) return e;
    if (n) {
        const size_t smem = (ko ? tile_smem<true>(rpp) : tile_smem<false>(rpp)) + 4ull * rpp;
        const void* kp = ko ? (const void*)k_region_part_scatter<true> : (const void*)k_region_part_scatter<false>;
        const int grid = (int)std::min<uint64_t>(P, (uint64_t)occupancy_grid(kp, kTileBlock, smem, ctx));
        if (ko)
            k_region_part_scatter<true><<<grid, kTileBlock, smem, s>>>(job, ends, P, rpp, sc.start, sc.staging, ctx->d_err);
        else
            k_region_part_scatter<false><<<grid, kTileBlock, smem, s>>>(job, ends, P, rpp, sc.start, sc.staging, ctx->d_err);
        ctx->launches++;
        if ((e = cudaGetLastError())) return e;
    } else {  // nothing staged: every region is empty
        if ((e = cudaMemsetAsync(sc.start, 0, 4ull * (regions + 1), s))) return e;
    }
    return build_staged(nullptr, job, 1, regions, kRegionShift, stage_out(sc, true), true, land, table_job.t.meta, s,
                        ctx);
}

static size_t align_scratch(size_t x) { return (x + 255) & ~(size_t)255; }

size_t region_zero_bytes(uint32_t regions) { return align_scratch(4ull * regions) + 8 + 32; }

// One job needs no numbers in its overflow list, and key-only rows and exact
// ranges have room for them in the entries (overflow_entry).
static bool job_list(bool one_job, bool key_only, bool exact) { return !one_job && !key_only && !exact; }

size_t region_scratch_bytes(uint32_t regions, uint64_t staged, uint64_t rows, bool one_job, bool key_only, bool exact) {
    auto a = align_scratch;
    return a(region_zero_bytes(regions)) + a(4ull * regions) + a(4ull * (regions + 1)) +
           a((key_only ? 4ull : 8ull) * staged) + a(8ull * rows) +
           (job_list(one_job, key_only, exact) ? a(4ull * rows) : 0);
}

RegionScratch carve_region_scratch(void* base, uint32_t regions, uint64_t staged, uint64_t rows, bool one_job,
                                   bool key_only, bool exact) {
    auto a = align_scratch;
    unsigned char* p = static_cast<unsigned char*>(base);
    RegionScratch s;
    s.cursor = reinterpret_cast<uint32_t*>(p);
    s.ctl = reinterpret_cast<uint32_t*>(p + a(4ull * regions));
    s.meta = reinterpret_cast<unsigned long long*>(s.ctl + 2);
    p += a(region_zero_bytes(regions));
    s.hist = reinterpret_cast<uint32_t*>(p);
    p += a(4ull * regions);
    s.start = reinterpret_cast<uint32_t*>(p);
    p += a(4ull * (regions + 1));
    s.staging = reinterpret_cast<unsigned long long*>(p);
    p += a((key_only ? 4ull : 8ull) * staged);
    s.ovf = reinterpret_cast<unsigned long long*>(p);
    p += a(8ull * rows);
    s.ovf_job = job_list(one_job, key_only, exact) ? reinterpret_cast<uint32_t*>(p) : nullptr;
    return s;
}

uint32_t region_share(uint64_t rows, uint32_t nregions, const TableView& t, uint32_t shift) {
    const uint64_t slots = (uint64_t)(t.key_only ? 8 : 4) << shift;
    const uint64_t expected = (rows + nregions - 1) / nregions;
    return (uint32_t)std::max<uint64_t>(1, std::min({slots, 2 * expected + 256, rows}));
}

cudaError_t launch_build_regions(const RegionJob* d_jobs, const RegionJob& table_job, uint32_t njobs,
                                 const BatchItem* items, uint32_t nitems, uint64_t n, uint32_t total_regions,
                                 uint32_t max_job_regions, const RegionScratch& sc, bool exact, bool fresh,
                                 TableLanding* land, bool zeroed, cudaStream_t s, Context* ctx) {
    if (total_regions == 0) return cudaSuccess;
    RegionJob job0 = table_job;
    if (fresh && land) job0.t.meta = sc.meta;
    // every job of one launch has the same slot layout (all key-only or none); a
    // key-only launch stages 4-byte keys
    const bool ko = job0.t.key_only != 0;
    const bool tiles = max_job_regions <= kTileRegions;
    const size_t hsmem = 4ull * std::max(max_job_regions, 1u);
    const size_t smem = !tiles ? hsmem : ko ? tile_smem<true>(max_job_regions) : tile_smem<false>(max_job_regions);
    const void* k = tiles ? (ko ? (const void*)k_region_tile_scatter<true> : (const void*)k_region_tile_scatter<false>)
                          : (ko ? (const void*)k_region_scatter<true> : (const void*)k_region_scatter<false>);
    const uint64_t ctas = (uint64_t)occupancy_grid(k, tiles ? kTileBlock : kRBlock, smem, ctx);
    uint64_t rpi = 0;
    if (!items && n) {
        // whole tiles dealt evenly over the CTAs, or items worth zeroing and flushing their region counters
        if (tiles) rpi = (n - 1) / (ctas * ((n - 1) / (ctas * kTileSize) + 1)) + 1;
        else rpi = std::max<uint64_t>({8ull * max_job_regions, 4096, n / (2ull * ctx->prop.multiProcessorCount) + 1});
        nitems = (uint32_t)((n + rpi - 1) / rpi);
    }
    cudaError_t e;
    if (!zeroed && (e = cudaMemsetAsync(sc.cursor, 0, region_zero_bytes(total_regions), s))) return e;
    if (exact) {
        if ((e = cudaMemsetAsync(sc.hist, 0, 4ull * total_regions, s))) return e;
        if (nitems) {
            const int grid = (int)std::min<uint64_t>(nitems, (uint64_t)occupancy_grid((const void*)k_region_hist, kRBlock,
                                                                                       hsmem, ctx));
            k_region_hist<<<grid, kRBlock, hsmem, s>>>(d_jobs, job0, items, nitems, n, rpi, sc.hist);
            ctx->launches++;
            if ((e = cudaGetLastError())) return e;
        }
        k_region_scan<<<1, kScanBlock, 0, s>>>(sc.hist, total_regions, sc.start);
        ctx->launches++;
        if ((e = cudaGetLastError())) return e;
    }
    const StageOut out = stage_out(sc, exact);
    if (nitems) {
        const int grid = (int)std::min<uint64_t>(nitems, ctas);
        if (tiles && ko)
            k_region_tile_scatter<true><<<grid, kTileBlock, smem, s>>>(d_jobs, job0, items, nitems, n, rpi, out, ctx->d_err);
        else if (tiles)
            k_region_tile_scatter<false><<<grid, kTileBlock, smem, s>>>(d_jobs, job0, items, nitems, n, rpi, out, ctx->d_err);
        else if (ko)
            k_region_scatter<true><<<grid, kRBlock, smem, s>>>(d_jobs, job0, items, nitems, n, rpi, out, ctx->d_err);
        else
            k_region_scatter<false><<<grid, kRBlock, smem, s>>>(d_jobs, job0, items, nitems, n, rpi, out, ctx->d_err);
        ctx->launches++;
        if ((e = cudaGetLastError())) return e;
    }
    return build_staged(d_jobs, job0, njobs, total_regions, job0.shift, out, fresh, land, table_job.t.meta, s, ctx);
}

cudaError_t launch_build_small(const RegionJob& job, uint32_t n, TableLanding* land, cudaStream_t s, Context* ctx) {
    const size_t smem = 36ull * job.t.nbuckets;
    if (job.t.key_only) k_build_small<true><<<1, kSmallBlock, smem, s>>>(job, n, land, ctx->d_err);
    else k_build_small<false><<<1, kSmallBlock, smem, s>>>(job, n, land, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

cudaError_t launch_table_land(const TableView& t, TableLanding* land, cudaStream_t s, Context* ctx) {
    k_table_land<<<1, 32, 0, s>>>(t, land, ctx->d_err);
    ctx->launches++;
    return cudaGetLastError();
}

}  // namespace mgv
