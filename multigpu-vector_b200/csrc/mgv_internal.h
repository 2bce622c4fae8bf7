// mgv_internal.h -- host-side objects behind the C ABI and the kernel
// launchers they call.  Not part of the public interface.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/mgv.h"
#include "launch_fits.h"

namespace mgv {

// ---- error reporting ---------------------------------------------------

void set_last_error(const std::string& msg);
mgv_status fail(mgv_status s, const std::string& msg);
mgv_status cuda_fail(cudaError_t e, const char* what);

#define MGV_CUDA_TRY(expr)                                    \
    do {                                                      \
        cudaError_t e_ = (expr);                              \
        if (e_ != cudaSuccess) return ::mgv::cuda_fail(e_, #expr); \
    } while (0)

// ---- device views passed to kernels by value ----------------------------

// Open-addressing join table: nbuckets buckets of 32 bytes (32-byte
// aligned), either 4 slots of 64-bit {key (low word), payload (high word)}
// or, for a build side without payloads (key_only), 8 slots of a 32-bit key
// (every match then has payload 0): half the bytes per key.
struct TableView {
    unsigned long long* slots;
    uint32_t nbuckets;
    // Radix layout: the home bucket of a key lies in the region of its
    // partition ((key >> radix_shift) & radix_mask), bpp buckets per region;
    // radix_mask 0 and bpp == nbuckets for an unpartitioned table.  Runs
    // continue linearly across regions.
    uint32_t radix_shift;
    uint32_t radix_mask;
    uint32_t bpp;
    uint32_t key_only;  // 1: 8 key slots per bucket, no payloads
    uint32_t pad;
    // Rows whose key is the reserved empty marker INT32_MIN:
    // meta[0] = their count, meta[1] = their payload sum, meta[2] = rows
    // inserted into the table, meta[3] = duplicate-key flag.
    unsigned long long* meta;
    int32_t* side_pay;      // payloads of those rows (for emitting matches)
    uint64_t side_cap;
};

// Group-by table in global memory: cap (power of two) slots of {key, sum,
// count}, empty key INT32_MIN; the group INT32_MIN has its own counters.
struct GroupTableView {
    int32_t* keys;
    unsigned long long* sums;
    unsigned long long* counts;
    unsigned long long* special;  // [0] sum, [1] count of group INT32_MIN
    uint32_t cap;
    uint32_t pad;
};

// Output rows appended to a chain of pool buffers.
struct SinkView {
    int32_t* slab;              // pool slab base
    unsigned long long* cursor; // rows reserved so far
    uint32_t* chain;            // buffer id per chunk, 0xffffffff = not yet taken
    uint32_t max_chunks;
    uint32_t capacity;          // rows per buffer
    uint32_t ncols;             // columns written
    uint32_t pool_ncols;
    struct PoolDev* pool;       // device free stack for swap-on-full
};

// Device free stack of a pool (tagged Treiber stack of buffer ids).
struct PoolDev {
    unsigned long long head;    // low 32 bits: top id (0xffffffff = empty), high: tag
    uint32_t available;
    uint32_t producers;
    uint32_t nbuffers;
    uint32_t pad;
    uint32_t next[1];           // nbuffers entries follow
};

constexpr uint32_t kNil = 0xffffffffu;
#ifndef MGV_BUILD_ROWS_PER_THREAD
#define MGV_BUILD_ROWS_PER_THREAD 1
#endif
constexpr int kBuildRows = MGV_BUILD_ROWS_PER_THREAD;  // build rows per thread in flight (1 measured fastest: more in flight contends in L2)
constexpr uint32_t kMaxSmemGroups = 8192;  // largest per-CTA shared group table (slots; 128 KiB)

// ---- host objects --------------------------------------------------------

struct Context;

struct Pool {
    Context* ctx = nullptr;
    uint32_t nbuffers = 0, capacity = 0, ncols = 0;
    int32_t* slab = nullptr;
    PoolDev* dev = nullptr;         // device free stack
    uint32_t* d_ids = nullptr;      // device scratch for host batch ops
    uint32_t* h_ids = nullptr;      // pinned mirror
    cudaStream_t stream = nullptr;  // the pool's own stream (release_streams)
    std::mutex mu;
    std::vector<uint32_t> host_cache;   // ids cached on the host side
    std::vector<mgv_buffer> bufs;       // descriptors, indexed by id
    std::vector<uint8_t> held;          // 1 = handed out to the caller
    uint32_t producers = 0;
};

struct Context {
    int device = 0;
    cudaDeviceProp prop{};
    cudaStream_t stream = nullptr;
    uint32_t* d_err = nullptr;      // device error word [code, detail]
    // pinned landing zone for close(): [0..1] error word, [2..] result words
    unsigned long long* h_stage = nullptr;
    std::atomic<uint64_t> launches{0};
    mgv_tuning tuning{0u, 4u, 4u, 3u, 0.5f, kMaxSmemGroups, 0u, 0u};
    mgv_batch_config batch_tuned{};  // the batch autotuner's last choice
    bool has_batch_tuned = false;
    std::mutex mu;
    mutable LaunchFits fits;  // CTAs per SM of the launch shapes used lately (blocks_per_sm)
};

enum class OpKind { Select, Aggregate, HashBuild, HashProbe, Sink, Groupby, Partition };
enum class OpState { Created, Open, Closed };

struct Op {
    OpKind kind;
    Context* ctx = nullptr;
    Op* parent = nullptr;
    OpState state = OpState::Created;
    bool graphed = false;  // an open or a consume of it was captured into a graph (for good)
    // select
    mgv_select_desc sel{};
    // aggregate
    mgv_aggregate_desc agg{};
    unsigned long long* d_acc = nullptr;    // [count, sum]
    unsigned long long* h_res = nullptr;    // pinned: the error word and the results read back at close
    unsigned long long* h_res_dev = nullptr;  // the same as the device addresses it (aggregate)
    bool agg_clean = false;                 // d_acc is zero on the device (a close leaves it so)
    mgv_agg_result agg_result{};
    // hash build
    mgv_hash_build_desc hb{};
    TableView table{};
    size_t table_bytes = 0;
    mgv_hash_build_info hb_info{};
    bool unique = false;
    // hash probe
    mgv_hash_probe_desc hp{};
    // sink
    mgv_sink_desc sk{};
    Pool* sink_pool = nullptr;
    SinkView sink{};
    uint64_t sink_rows = 0;
    std::vector<uint32_t> sink_chain;
    struct SinkLanding* sk_land = nullptr;  // pinned, mapped: max_chunks ids
    struct SinkLanding* sk_land_dev = nullptr;
    // delivery channel (mgv_sink_drain): copies run on their own stream; the
    // buffers of the copy in flight return to the pool when it completes
    cudaStream_t drain_stream = nullptr;
    cudaEvent_t drain_done = nullptr;
    std::vector<uint32_t> drain_ids;
    // group-by
    mgv_groupby_desc gb{};
    GroupTableView gtab{};
    const mgv_group_row* gb_view = nullptr;  // the closed result's rows: in the landing zone or gb_rows
    uint32_t gb_n = 0;
    std::vector<mgv_group_row> gb_rows;      // rows the landing zone does not hold, or ordered on the host
    bool gb_sorted = false;                  // gb_view is ordered by group (else done at the first result read)
    bool gb_unordered = false;               // nobody asks for an order: close leaves the rows as they come
    bool gb_clean = false;                   // the table is empty on the device (a close leaves it so)
    mgv_group_row* gb_dev_rows = nullptr;    // [cap + 1] packed by the close of a large table
    uint32_t* gb_dev_count = nullptr;        // {groups packed, CTAs done, groups found}
    unsigned long long* gb_pairs = nullptr;  // sorting space of a large table: pairs, then the order
    mgv_group_row* gb_dev_more = nullptr;    // ordered rows past the landing zone
    struct GroupLanding* gb_land = nullptr;  // pinned, mapped: gb_land_rows rows
    struct GroupLanding* gb_land_dev = nullptr;
    uint32_t gb_land_rows = 0;
    // partition
    mgv_partition_desc pt{};
    int32_t* pt_store = nullptr;          // ncols x capacity, partition-major runs
    uint32_t pt_ncols = 0;
    uint64_t pt_fill = 0;                 // rows stored (read back at close)
    uint64_t pt_offered = 0;              // rows consumed since open (host count)
    uint32_t pt_runs = 0;                 // consumes with rows since open (each stores one partition-major run)
    bool pt_filtered = false;             // a select fed a consume: only the device knows pt_fill
    bool pt_hist_valid = true;            // pt_hist read back (else read at mgv_op_result)
    cudaStream_t pt_close_stream = nullptr;
    unsigned long long* pt_dev = nullptr; // [P] histogram / cursors of a consume
    unsigned long long* pt_acc = nullptr; // [1 + P] rows stored, rows per partition
    std::vector<uint64_t> pt_hist;        // rows per partition (read back at close)
    bool hb_fresh = false;  // opened, nothing consumed yet: the table and its counters are not cleared yet
    bool hb_cleared = false;  // the open cleared them (a graph holds the operator)
    bool hb_landed = false;  // the last consume's kernels hand the table's counters to the host
    struct TableLanding* hb_land = nullptr;  // pinned, mapped
    struct TableLanding* hb_land_dev = nullptr;
    const unsigned long long* hb_part_ends = nullptr;  // that run's partition ends (device), when it is the only run
    // host ingest (mgv_op_consume_host): the copy stream and, per buffer in
    // flight, events for "slice copied" and "slice consumed"
    cudaStream_t in_stream = nullptr;
    std::vector<cudaEvent_t> in_copied, in_consumed;
    // shared-memory build scratch (hash_build), grown on demand
    void* rb_scratch = nullptr;
    size_t rb_bytes = 0;
    bool rb_exact = false;   // no room for staging shares: exact ranges
    uint32_t rb_zeroed = 0;  // regions for which the scratch was left zeroed (0: none)
    // device allocations owned by this op
    std::vector<void*> allocs;
};

// ---- kernel launchers (kernels.cu, pool.cu) -----------------------------

struct LaunchCfg {
    int grid;
    int block;
};

// CTAs of a launch shape that fit one SM (at least 1).  The first call for a
// shape also raises the kernel's dynamic shared memory limit to what the
// device allows; later ones are a look-up, where asking the runtime each time
// took 2 to 3 us of a launch.
int blocks_per_sm(const void* kernel, int block, size_t smem, const Context* ctx);
int occupancy_grid(const void* kernel, int block, size_t smem, const Context* ctx);

cudaError_t launch_fill_u64(unsigned long long* p, uint64_t n, unsigned long long v, cudaStream_t s,
                            Context* ctx);
cudaError_t launch_select_agg(const int32_t* filt, int32_t bound, bool has_sel, const int32_t* a,
                              const int32_t* b, uint64_t n, unsigned long long* acc, cudaStream_t s,
                              Context* ctx);
// {error word, count, sum} to the host (pinned, mapped), and the sums back to zero.
cudaError_t launch_agg_land(unsigned long long* acc, unsigned long long* land, cudaStream_t s, Context* ctx);
cudaError_t launch_build(const int32_t* keys, const int32_t* pays, const int32_t* filt,
                         int32_t bound, bool has_sel, uint64_t n, const TableView& t,
                         cudaStream_t s, Context* ctx);
// sum_mode bit 0: add build payload, bit 1: add probe payload column.
cudaError_t launch_probe_agg_staged(const int32_t* keys, const int32_t* pays, uint64_t n, const TableView& t,
                                    bool unique, uint32_t sum_mode, unsigned long long* acc, cudaStream_t s,
                                    Context* ctx);
cudaError_t launch_probe_agg(const int32_t* keys, const int32_t* pays, uint64_t n,
                             const TableView& t, bool unique, uint32_t sum_mode,
                             unsigned long long* acc, cudaStream_t s, Context* ctx);
// Generic fused chain (chain.cu): [select] -> [probe] -> terminal.
enum TermKind : int { kTermAgg = 0, kTermGroupby = 1, kTermSink = 2, kTermCells = 3 };

// A shared scan: several select -> join -> group-by requests over the same
// probe columns and join table that differ only in their filter bound read
// the columns and probe the table once.  The m distinct bounds, ascending,
// cut the filter values into m ranges (range j: b[j-1] < f <= b[j]); a
// matched row adds its (group, value) to one cell (range of its filter,
// group) only, whatever the number of requests.  A request with bound b[j]
// is then the sum of ranges 0..j, which one prefix pass over the ranges
// computes for every request at once.
//
// Cells live in m group tables that share one key array (the group
// directory, `cap` slots): range j's table is {keys, v + j*(2 cap + 2),
// +cap, +2 cap} over one block of u64 values, so a group has the same slot
// in every range and the prefix is a flat sum over the blocks.
struct CellsView {
    const int32_t* bounds;       // m ascending distinct filter bounds
    uint32_t m;
    uint32_t cap;                // directory slots, power of two
    int32_t* keys;               // the group directory (EMPTY = INT32_MIN)
    unsigned long long* vals;    // m blocks of [sums (cap) | counts (cap) | special sum, count]
    const uint16_t* lut;         // range of filter value lut_base + i, i < lut_len (0: none)
    uint32_t lut_len;
    int32_t lut_base;
};
constexpr uint32_t kCellRowBits = 20;        // ring entries: row offset (low bits) | range (high bits)
constexpr uint32_t kMaxCellRanges = 2048;    // distinct bounds per shared scan (range index < 2^11)
constexpr uint32_t kCellLut = 8192;          // longest range lookup table (filter values b[0]..b[m-1])
__host__ __device__ __forceinline__ size_t cell_block_words(uint32_t cap) { return 2ull * cap + 2; }
__host__ __device__ __forceinline__ GroupTableView cells_range(const CellsView& c, uint32_t j) {
    GroupTableView g;
    g.keys = c.keys;
    g.sums = c.vals + (size_t)j * cell_block_words(c.cap);
    g.counts = g.sums + c.cap;
    g.special = g.sums + 2ull * c.cap;
    g.cap = c.cap;
    g.pad = 0;
    return g;
}

struct ChainArgs {
    const int32_t* cols[MGV_MAX_COLS];
    uint32_t ncols;
    uint64_t n;
    bool has_sel;
    uint32_t sel_col;
    int32_t sel_bound;
    bool has_probe;
    uint32_t probe_col;
    TableView table;
    bool unique;
    int term;
    // terminal column references (input column, ncols = build payload, -1 none):
    //   aggregate: ref[0], ref[1] summed;  group-by: ref[0] group, ref[1] value;
    //   sink: ref[i] = source of output column i
    int32_t ref[MGV_MAX_COLS + 2];
    uint32_t nref;
    unsigned long long* acc;
    GroupTableView gt;
    uint32_t smem_groups;
    SinkView sink;
};
cudaError_t launch_chain(const ChainArgs& a, cudaStream_t s, Context* ctx);
// What a sink has gathered, handed to the host by one kernel.
struct SinkLanding {
    uint32_t err[2];
    unsigned long long rows;
    uint32_t chain[1];  // max_chunks buffer ids
};
cudaError_t launch_sink_land(const SinkView& sv, SinkLanding* land, cudaStream_t s, Context* ctx);

// Device-side parameters of one chain (one query of a batch).
struct ChainDev {
    const int32_t* cols[MGV_MAX_COLS];
    uint64_t n;
    uint32_t ncols;
    uint32_t nslots;                 // carried columns
    int32_t slot_src[MGV_MAX_COLS];  // input column of each carried slot
    uint32_t sel_col;
    int32_t sel_bound;
    int32_t probe_slot;
    uint32_t unique;  // the table has no duplicate keys: a probe stops at its match
    TableView table;
    // terminal column references: carried slot, kBP (build payload) or -1
    int32_t ref[MGV_MAX_COLS + 2];
    uint32_t nref;
    unsigned long long* acc;
    GroupTableView gt;
    uint32_t smem_groups;  // shared group-table slots: power of two <= kMaxSmemGroups, 0 = none
    SinkView sink;
    CellsView cells;       // shared scan (kTermCells): the ranges' cells
};

constexpr int32_t kBP = 100;  // terminal reference to the build payload

// Batched execution (chain.cu kernels, batch.cu host side).
struct BatchItem {  // rows [lo, hi) of query q
    uint32_t q;
    uint32_t pad;
    uint64_t lo, hi;
};
// Shared-memory hash-table build (build_regions.cu).  A table is cut into
// regions of kRegionBuckets buckets; build rows are bucketed by the region of
// their home bucket, then one CTA per region inserts the region's rows into
// a shared-memory copy of the region and writes it back with coalesced
// stores.  A row whose run leaves its region is inserted afterwards into the
// global table.  A "job" is one table's build; a launch can build many.
constexpr uint32_t kRegionShift = 11;
constexpr uint32_t kRegionBuckets = 1u << kRegionShift;  // 64 KiB of table per region
// Small tables: smaller regions, so that every SM gets some.  300 K {key,
// payload} rows, regions of 2^11 / 2^10 / 2^9 / 2^8 buckets: staging, build and
// global insert take 54 / 53 / 61 / 62 us (every region end adds rows to the insert).
constexpr uint32_t kMinRegionShift = 10;
constexpr uint32_t kMaxRegionsPerJob = 16384;  // per-CTA region histogram: 64 KiB
constexpr uint64_t kRegionBuildMinRows = 1u << 16;  // smaller builds: one global CAS per row
constexpr uint64_t kSmallBuildRows = 1u << 14;      // a one-region table of at most this many rows: one CTA, one launch
struct RegionJob {
    TableView t;
    const int32_t* keys;
    const int32_t* pays;      // nullable
    const int32_t* filt;      // nullable: rows with filt <= bound only
    int32_t bound;
    uint32_t region0;         // first region of this job in the launch
    uint32_t nregions;        // regions of 2^shift buckets
    uint32_t shift;
    uint64_t stage0;          // region r's staging rows: stage0 + r * cap on (when the ranges are not exact)
    uint32_t cap;
    uint32_t pad;
};
struct RegionScratch {
    // cursor, ctl and meta are zeroed together (region_zero_bytes), before a
    // launch and, where the launch lands one table's counters, again by its end
    uint32_t* cursor;         // [regions] rows placed
    uint32_t* ctl;            // [2] rows left for the global insert, CTAs done
    unsigned long long* meta; // [4] the counters of a fresh table while it is built (TableView::meta)
    uint32_t* hist;           // [regions] rows per region (exact ranges)
    uint32_t* start;          // [regions + 1] first staging row of each region (exact ranges)
    unsigned long long* staging;  // {key, payload}, region-major
    unsigned long long* ovf;  // [rows] {key, payload} left for the global insert
    uint32_t* ovf_job;        // [rows] their jobs; nullptr: one job, or the entries hold the jobs too
};
// A table's counters (TableView::meta) and the error word, handed to the host.
struct TableLanding {
    uint32_t err[2];
    unsigned long long meta[4];
};
// Host: group rows in ascending group order (radix sort).
void sort_group_rows(std::vector<mgv_group_row>& v);
inline uint32_t table_regions(const TableView& t) { return (t.nbuckets + kRegionBuckets - 1) / kRegionBuckets; }
size_t region_zero_bytes(uint32_t regions);
size_t region_scratch_bytes(uint32_t regions, uint64_t staged, uint64_t rows, bool one_job, bool key_only, bool exact);
RegionScratch carve_region_scratch(void* base, uint32_t regions, uint64_t staged, uint64_t rows, bool one_job,
                                   bool key_only, bool exact);
// Staging rows of each region when the ranges are fixed shares.
uint32_t region_share(uint64_t rows, uint32_t nregions, const TableView& t, uint32_t shift);
cudaError_t region_build_init();  // once per device: the kernels' shared memory limits
// Items: explicit (job, rows) items, or (items == nullptr) rows [0, n) of
// job0.  exact: staging ranges from a histogram (the jobs' stage0 and cap are
// not used).  fresh: the tables hold nothing yet and are not cleared
// beforehand; every region is written.  land: nullable, where one table's
// counters go afterwards; a fresh table's own need no clearing then.  zeroed:
// the scratch is as the last such launch over as many regions left it.
cudaError_t launch_build_regions(const RegionJob* d_jobs, const RegionJob& job0, uint32_t njobs,
                                 const struct BatchItem* items, uint32_t nitems, uint64_t n, uint32_t total_regions,
                                 uint32_t max_job_regions, const RegionScratch& sc, bool exact, bool fresh,
                                 TableLanding* land, bool zeroed, cudaStream_t s, Context* ctx);
// A fresh radix-laid-out table built from a partition op's single run on its
// radix bits (ends[p] = one past partition p's last row): per-partition
// staging in the partition's own range, then the region build.  Only when
// every partition slice is whole regions (region_build_partitioned_fits).
bool region_build_partitioned_fits(const TableView& t);
cudaError_t launch_build_regions_partitioned(const RegionJob& job, const unsigned long long* ends, uint64_t n,
                                             const RegionScratch& sc, TableLanding* land, bool zeroed, cudaStream_t s,
                                             Context* ctx);
// A fresh table of at most kRegionBuckets buckets from all its rows.
cudaError_t launch_build_small(const RegionJob& job, uint32_t n, TableLanding* land, cudaStream_t s, Context* ctx);
cudaError_t launch_table_land(const TableView& t, TableLanding* land, cudaStream_t s, Context* ctx);

struct BatchOut {  // packed result region of a query
    GroupTableView gt;
    mgv_group_row* rows;
    uint32_t* count;
    uint32_t capacity;
    uint32_t pad;
};
// A group-by operator's landing zone in pinned, mapped host memory.
struct GroupLanding {
    uint32_t err[2];
    uint32_t count;
    uint32_t pad;
    mgv_group_row rows[1];
};
// Packed rows to be ordered by group (group_rows.cu).
struct GroupSortJob {
    const mgv_group_row* rows;
    uint32_t* count;            // rows found (may exceed capacity: then an error is set)
    uint32_t* found;            // the same, kept for the writing of the rows
    unsigned long long* pairs;  // 2 * capacity, used when the rows do not fit shared memory
    uint32_t* order;            // capacity
    mgv_group_row* out;         // the first out_rows rows
    mgv_group_row* more;        // the rows past them
    GroupLanding* land;         // nullable: header to fill in
    uint32_t capacity;
    uint32_t out_rows;
};
constexpr uint32_t kSmallGroupCap = 2048;      // slots of a table that one CTA closes
// Slots of the largest table ordered on the device, by one CTA.  Close and read
// of a result on the host / on the device, us, dense and sparse group ids: 2^13
// groups 117 / 51 and 140 / 89, 2^16 1218 / 260 and 1530 / 538, 2^18 5742 / 2579
// and 7060 / 3000, 2^20 34085 / 10816 and 35070 / 11930.  (The close alone is the
// longer one of the two from 2^17 groups on: 505 / 670; 3699 / 8594 for 2^20.)
// Past this the sorting space is what counts against it.
constexpr uint32_t kDeviceOrderCap = 1u << 21;
cudaError_t group_rows_init();  // once per device: the kernels' shared memory limits
cudaError_t launch_group_reset(const GroupTableView& gt, uint32_t* count, cudaStream_t s, Context* ctx);
cudaError_t launch_group_close(const GroupTableView& gt, GroupLanding* land, bool sort, cudaStream_t s, Context* ctx);
cudaError_t launch_group_pack(const GroupTableView& gt, mgv_group_row* rows, uint32_t* count, GroupLanding* land,
                              cudaStream_t s, Context* ctx);
// Orders the jobs' rows (max_rows: the largest capacity) and writes them out.
cudaError_t launch_group_sort(const GroupSortJob* d_jobs, const GroupSortJob& job0, uint32_t njobs, uint32_t max_rows,
                              cudaStream_t s, Context* ctx);
cudaError_t launch_batch(const ChainDev* d_qs, const BatchItem* probe_items, uint32_t n_probe, int ctas_per_sm,
                         uint32_t item_order, cudaStream_t s, Context* ctx);
// Packs the groups of many tables (items: slots [lo, hi) of query q, at most
// kCompactSlots each) into their output regions.
constexpr uint64_t kCompactSlots = 4096;
cudaError_t launch_batch_compact(const BatchOut* d_outs, const BatchItem* items, uint32_t nitems, cudaStream_t s,
                                 Context* ctx);
// Shared scans: the persistent probe -> cells kernel over (scan, rows)
// items (rows per item < 2^kCellRowBits), then the prefix over each scan's
// ranges (`scans` are host-side copies of the device descriptors' cells).
cudaError_t launch_cells(const ChainDev* d_scans, const BatchItem* items, uint32_t nitems, cudaStream_t s,
                         Context* ctx);
cudaError_t launch_cells_prefix(const CellsView& c, cudaStream_t s, Context* ctx);

// partition.cu
cudaError_t launch_partition_hist(const int32_t* const* cols, uint64_t n, bool has_sel, uint32_t sel_col,
                                  int32_t sel_bound, uint32_t key_col, uint32_t shift, uint32_t bits,
                                  unsigned long long* hist, cudaStream_t s, Context* ctx);
cudaError_t launch_partition_cursors(unsigned long long* hc, uint32_t bits, unsigned long long* acc, uint64_t max_rows,
                                    cudaStream_t s, Context* ctx);
cudaError_t launch_partition_scatter(const int32_t* const* cols, uint32_t ncols, uint64_t n, bool has_sel,
                                     uint32_t sel_col, int32_t sel_bound, uint32_t key_col, uint32_t shift,
                                     uint32_t bits, unsigned long long* cursors, int32_t* out, uint64_t out_stride,
                                     cudaStream_t s, Context* ctx);
cudaError_t launch_fill_i32(int32_t* p, uint64_t n, int32_t v, cudaStream_t s, Context* ctx);

// pool.cu
cudaError_t pool_init_device(Pool* p);
// Pops up to `want` ids into p->h_ids (sync); returns the count taken or
// reports drained / timeout through *status.
cudaError_t pool_pop_batch(Pool* p, uint32_t want, uint32_t timeout_us, uint32_t* got,
                           mgv_status* status);
cudaError_t pool_push_batch(Pool* p, const uint32_t* ids, uint32_t n);
cudaError_t pool_read_counters(Pool* p, uint32_t* available, uint32_t* producers);
cudaError_t pool_add_producers(Pool* p, int delta);

}  // namespace mgv

struct mgv_ctx : mgv::Context {};
struct mgv_pool : mgv::Pool {};
struct mgv_op : mgv::Op {};
