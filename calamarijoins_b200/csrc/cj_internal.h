/*
 * cj_internal.h — types shared by the host engine and the sm_100a kernels.
 *
 * Device data layout (all in HBM, one allocation per array):
 *   pages        a column's 8 KiB pages, consecutive, exactly as on the host
 *   page index   u64 base per 256 pages and u32 loc per page, whose sum is
 *                the page's first row (a page holds n_rows rows, a
 *                long-string start page 0xffff one, a continuation page
 *                0xfffe none)
 *   values       dense fixed-width values, one per row (0 where NULL)
 *   valid        validity bitmap, u32 words, bit r = row r present
 *   str_desc     VARCHAR: one u64 per row, see CJ_DESC_* below
 *   rid vectors  u32 row ids (late materialisation of intermediates)
 *   hash table   u64 directory ((end << 16) | 16-bit Bloom tag) and a
 *                slot-ordered tuple array {key, row id}
 */
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/cj_b200.h"

namespace cj {

constexpr uint32_t kPageSize = CJ_PAGE_SIZE;
constexpr uint32_t kMaxShortString = kPageSize - 7; /* plan.h:331 */
constexpr uint32_t kLongChunk = kPageSize - 4;      /* plan.h:301 */
constexpr uint32_t kRowsPerPageInt32 = 1984;        /* ColumnInserter<int32_t> fill */
constexpr uint32_t kRowsPerPage8B = 1007;           /* ColumnInserter<int64_t/double> */

/* VARCHAR row descriptor.
 *   short string: bit 63 = 0, bits 62..24 = byte offset of the first
 *                 character inside the column's page blob, bits 23..0 =
 *                 length (<= 8185)
 *   long string:  bit 63 = 1, bits 62..24 = index of its 0xffff page,
 *                 bits 23..0 = number of pages in the chain (the 0xffff
 *                 page and the 0xfffe pages that follow it)
 *   NULL rows hold 0 (the validity bitmap says NULL). */
constexpr uint64_t CJ_DESC_LONG = 1ull << 63;
__host__ __device__ inline uint64_t desc_short(uint64_t off, uint32_t len) {
    return (off << 24) | len;
}
__host__ __device__ inline uint64_t desc_long(uint64_t page, uint32_t chain) {
    return CJ_DESC_LONG | (page << 24) | chain;
}
__host__ __device__ inline bool desc_is_long(uint64_t d) { return (d >> 63) != 0; }
__host__ __device__ inline uint64_t desc_pos(uint64_t d) { return (d >> 24) & ((1ull << 39) - 1); }
__host__ __device__ inline uint32_t desc_len(uint64_t d) { return (uint32_t)(d & 0xFFFFFFu); }

/* Error bits the kernels raise in the device status word. */
enum DevError : uint32_t {
    DEV_ERR_PAGE_HEADER = 1u << 0,   /* n_values > n_rows or page overflow */
    DEV_ERR_VARCHAR_OFFSETS = 1u << 1,
    DEV_ERR_LONG_CHAIN = 1u << 2,    /* 0xfffe page without a 0xffff start */
    DEV_ERR_BAD_PAGE_KIND = 1u << 3, /* 0xffff/0xfffe page in a fixed column */
    DEV_ERR_ROW_COUNT = 1u << 5,     /* pages hold more/fewer rows than the
                                        table declares                       */
    DEV_ERR_STALE = 1u << 6,         /* a prepared batch's counts no longer
                                        match its inputs                     */
    DEV_ERR_INTERNAL = 1u << 31
};

/* What a column's page index leaves on the device. Zero before the launch. */
struct ColumnState {
    unsigned int flags; /* COL_* flags, from the page headers      */
    unsigned int done;  /* blocks of the index that have finished  */
    unsigned int err;   /* DevError bits of this column            */
    unsigned int pad;
};
/* Columns whose state lives in the status block: their errors count only
 * once the plan reads them (Context::sync_status). */
constexpr uint32_t kStatusColumns = 64;

/* Small pinned block the host reads at each synchronisation point. */
struct StatusBlock {
    unsigned int errors;          /* DevError bits                          */
    unsigned int pad;
    unsigned long long counter;   /* match counter of the last probe        */
    unsigned long long table[9];  /* kTableWords of the last unique table   */
    unsigned long long aux;       /* a count on its way to the host (filter) */
    unsigned long long stale[3];  /* DEV_ERR_STALE: check index, count found,
                                     count recorded (one of the mismatches) */
    ColumnState cols[kStatusColumns];
};

/* How a kernel reads one column of a relation: row i of the relation is
 * row rid_b[rid_a[i]] of the decoded base column (each indirection is
 * skipped when its pointer is null). */
struct ColView {
    const void *values;
    const uint32_t *valid;
    const uint64_t *str_desc;
    const uint8_t *pages;
    const uint32_t *rid_a;
    const uint32_t *rid_b;
    int32_t type;
    int32_t null_sentinel; /* INT32: INT32_MIN reads as NULL (value_t) */
    const uint32_t *col_flags; /* device word of COL_* bits from the page
                                  headers; null: unknown (read the decoded
                                  values and validity)                   */
};

/* Column flags, set by the page-row pass. A fixed-width column whose word
 * is 0 has no NULL and every page but the last holds exactly
 * kRowsPerPageInt32 / kRowsPerPage8B rows (the fill of the reference's
 * ColumnInserter): row r is value r % R of page r / R, so it is read from
 * the pages and not decoded at all. */
enum ColFlag : uint32_t {
    COL_HAS_NULLS = 1u,  /* some page stores fewer values than rows      */
    COL_NOT_DIRECT = 2u, /* VARCHAR, or pages not filled as above        */
};

template <typename K> struct Tuple;
template <> struct alignas(8) Tuple<int32_t> {
    int32_t key;
    uint32_t rid;
};
template <> struct alignas(16) Tuple<int64_t> {
    int64_t key;
    uint32_t rid;
    uint32_t pad;
};

/* Directory entry of a table with INT32 keys: the entry word (start of the
 * slot's tuples << 32 | count << 16 | Bloom tags) and the slot's first
 * tuple inline, 16 bytes in one sector: a probe row whose slot holds one
 * tuple needs one random access. Tables with INT64 keys keep 8-byte entries
 * (the word alone). */
struct alignas(16) DirEntry32 {
    uint64_t word;
    int32_t key0;
    uint32_t rid0;
};

template <typename K> struct HashTableView {
    const uint64_t *dir; /* DirEntry32[] for K = int32_t, entry words for int64_t */
    const Tuple<K> *tuples;
    int log2_slots;
};

/* Output of a probe / nested-loop launch. */
struct MatchOut {
    uint32_t *build_rids = nullptr; /* null: not collected (RIGHT_ONLY)  */
    uint32_t *probe_rids = nullptr; /* null: not collected (LEFT_ONLY)   */
    uint8_t *key_pages = nullptr;   /* null, or the join key written straight
                                       into 8 KiB result pages: value pos % R
                                       of page pos / R (R = 1984 or 1007 by
                                       key_bytes); a PageTask with `finish`
                                       adds headers and bitmaps */
    int32_t key_bytes = 4;
    unsigned long long capacity = 0;
    unsigned long long *counter = nullptr;
};

/* Kernels launched by this process (every launcher adds its launches). */
void count_launches(uint64_t n);
uint64_t launches_so_far();

/* ----------------------------------------------------------------------- */
/* Kernel launchers (defined in the .cu files; all enqueue on `s`).         */
/* ----------------------------------------------------------------------- */
struct Launch {
    cudaStream_t stream;
    int num_sms;
    int block_threads; /* 0 = kernel default */
    unsigned int *dev_errors;
    int ctas_per_sm = 0;      /* persistent probe grids: CTAs per SM (0 = as many as fit) */
    int part_ctas_per_sm = 0; /* radix histogram / scatter passes: CTAs per SM (0 = 4)     */
};

/* Tuned launch parameters per size class of a relation's row count (the
 * autotuner's table). Classes split at 2^12, 2^15, 2^18, 2^21 and 2^24
 * rows. A zero entry means "the default". */
constexpr int kTuneClasses = 6;
inline int tune_class(uint64_t rows) {
    int c = 0;
    for (int t : {12, 15, 18, 21, 24})
        if (rows >= (1ull << t)) ++c;
    return c;
}
struct TuneEntry {
    int log2_spp = 0;    /* hash directory slots per radix partition (log2) */
    int part_ctas = 0;   /* radix passes: CTAs per SM                        */
    int probe_ctas = 0;  /* hash probe: CTAs per SM                          */
};
struct Tuning {
    bool loaded = false;
    TuneEntry cls[kTuneClasses];
    const TuneEntry &for_rows(uint64_t rows) const { return cls[tune_class(rows)]; }
};

/* Scan */
size_t scan_temp_bytes(size_t n);
/* out[i] = sum(in[0..i)), out[n] = total; in and out may not alias. */
cudaError_t scan_u32_to_u64(const Launch &L, const uint32_t *in, uint64_t *out,
                            size_t n, void *temp);

/* Decode */
/* One column to index and decode. The index gives row base[p >> 8] + loc[p]
 * as page p's first (page_first_row), the column's COL_* flags, its errors,
 * and a cleared validity bitmap; the decode writes the dense arrays of a
 * column that is not read in place. Rows past `rows` are never written; a
 * page that would write them raises DEV_ERR_ROW_COUNT instead. */
constexpr int kIndexChunk = 256; /* pages per block of the index */
struct ColumnTask {
    const uint8_t *pages;
    uint64_t num_pages;
    uint64_t rows;
    uint32_t *loc;       /* num_pages entries               */
    uint64_t *base;      /* index_blocks(num_pages) entries */
    ColumnState *state;
    unsigned int *err;
    void *values;        /* fixed width                     */
    uint64_t *desc;      /* VARCHAR                         */
    uint32_t *valid;     /* max(1, ceil(rows / 32)) words   */
    int32_t type;
    uint32_t index_base, index_blocks, decode_base, decode_blocks; /* place_columns */
};
constexpr int kColumnArgs = 32; /* tasks passed by value */
struct ColumnGrid {
    uint32_t index = 0, decode = 0; /* blocks of the two launches */
};
uint32_t index_blocks(uint64_t num_pages);
ColumnGrid place_columns(const Launch &L, ColumnTask *tasks, size_t n);
/* Index (or decode) of n columns, a launch per kColumnArgs of them. */
cudaError_t launch_columns(const Launch &L, ColumnTask *tasks, size_t n, bool index);
/* Index and decode of the columns of a batch, placed by place_columns. */
cudaError_t launch_columns_grouped(const Launch &L, const ColumnTask *tasks_dev, uint32_t n, const ColumnGrid &g);

/* Table of unique build keys (k_unique.cu): direct-mapped when their range is
 * at most max_span, else (open_slots > 0) open-addressing, with 8-byte slots
 * for INT32 keys and, for INT64 keys (wide), 16-byte ones and a tag byte each. `slots` holds
 * unique_table_bytes, 16-byte aligned; open_slots is at least twice the build
 * rows and a multiple of 16. `params` (kTableWords words, zero before the build) receives what the
 * device found. */
constexpr uint32_t kArrayEmpty = 0xFFFFFFFFu;
constexpr uint64_t kOpenMaxRows = 1ull << 28;
enum TableWord { /* of params */
    kTableMinC = 0,    /* ~min, max of the non-NULL keys (XOR 2^63: unsigned
                          order is signed order) and their count           */
    kTableMax = 1,
    kTableCount = 2,
    kTableRefused = 3, /* not direct-mapped: a TableRefusal                */
    kTableLo = 4,      /* smallest key, values in the range                */
    kTableSpan = 5,
    kTableDup = 6,     /* the build met a repeated key, or a walk of kMaxWalk
                          slots: the table is unusable                     */
    kTableDone = 7,    /* blocks of the range pass that have finished      */
    kTableEmpty = 8,   /* a key next to the range, that of an empty slot (but
                          for kTableWhole)                                 */
    kTableWords = 9
};
enum TableRefusal : unsigned long long {
    kTableSpread = 1,  /* the keys' range is above max_span           */
    kTableRepeats = 2, /* more keys than values in their range        */
    kTableWhole = 3    /* the keys span all of INT64: no key is free to
                          mark empty slots                            */
};
/* An insert walks at most this many slots of an open-addressing table (at
 * most half full: about one on average); keys whose hashes pile up, on which
 * the walks' sum would be quadratic, go on to the hash table. */
constexpr uint32_t kMaxWalk = 512;
struct UniqueTable {
    void *slots;
    unsigned long long *params;
    uint64_t max_span;
    uint32_t open_slots; /* 0: no open-addressing table */
    uint32_t wide;       /* 16-byte slots: INT64 build keys */
};
inline uint64_t unique_table_bytes(const UniqueTable &t) {
    const uint64_t direct = t.max_span * 4, open = (uint64_t)t.open_slots * (t.wide ? 17 : 8); /* wide: tags last */
    return ((direct > open ? direct : open) + 15) & ~15ull;
}
/* What the params say (host copy or device): 0 unusable, 1 direct-mapped,
 * 2 open-addressing. */
__host__ __device__ inline int table_kind(const unsigned long long *p, uint32_t open_slots) {
    if (p[kTableDup]) return 0;
    if (!p[kTableRefused]) return 1;
    return p[kTableRefused] == kTableSpread && open_slots ? 2 : 0;
}
/* Build */
struct BuildPlan {
    int log2_slots;      /* directory = 2^log2_slots entries + 1          */
    int log2_parts;      /* radix partition bits in all: one pass up to 12
                            bits, two passes above (launch_build)         */
    uint32_t num_rows;   /* rows of the build relation                    */
    bool inline_first = true; /* INT32 keys: 16-byte entries holding the
                                 slot's first tuple (DirEntry32), else the
                                 8-byte word alone                        */
};
/* Directory entry word: start (63..32) | count (31..16, saturated) | tags
 * (15..0); INT32 keys add the first tuple (DirEntry32); one sentinel entry
 * after the last slot. */
inline size_t build_dir_bytes(int log2_slots, int key_bytes, bool inline_first = true) {
    return ((1ull << log2_slots) + 1) * (key_bytes == 4 && inline_first ? sizeof(DirEntry32) : sizeof(uint64_t));
}
size_t build_temp_bytes(const Launch &L, const BuildPlan &bp, int key_bytes);
size_t build_tuple_bytes(int key_bytes);
cudaError_t launch_build(const Launch &L, const BuildPlan &bp, const ColView &key,
                         const uint16_t *bloom, uint64_t *dir, void *tuples,
                         void *temp);

/* Grouped build over the hash joins of one batch level. Each task
 * partitions its own rows into its own part_buf; chunk_base / part_base /
 * cell_base place its chunks, partitions and histogram cells in the global
 * numbering (prefix sums over the tasks). */
struct BuildGeometry {
    uint32_t grid;  /* chunks of the hist / scatter passes */
    uint32_t chunk; /* rows per chunk                      */
    uint64_t cells; /* partitions x chunks                 */
};
BuildGeometry build_geometry(const Launch &L, const BuildPlan &bp);
struct BuildTask {
    ColView key;
    uint32_t n;
    int32_t log2_slots;
    int32_t log2_parts;
    uint32_t grid;
    uint32_t chunk;
    uint32_t chunk_base;
    uint32_t part_base;
    uint64_t cell_base;
    uint64_t *dir;
    void *tuples;
    void *part_buf; /* n tuples of scratch */
    UniqueTable unique; /* nothing is built when this table (params set) is usable */
};
size_t build_grouped_temp_bytes(uint64_t total_cells);
cudaError_t launch_build_grouped(const Launch &L, const BuildTask *tasks_dev, uint32_t ntasks, uint32_t total_chunks,
                                 uint32_t total_parts, uint64_t total_cells, uint32_t max_parts, uint32_t max_slots,
                                 const uint16_t *bloom, void *temp);

cudaError_t launch_unique_build(const Launch &L, const ColView &key, uint32_t n, const UniqueTable &t);

/* The probe's key column: a scan read page by page (base and loc of its page
 * index set; the decoded arrays are not needed), or relation rows through
 * the view (base null). */
struct ProbeKey {
    ColView col;
    const uint64_t *base;
    const uint32_t *loc;
    uint64_t num_pages;
    unsigned int *err; /* errors of the column's pages */
};
/* A fixed-width result column that the probe writes when the device finds
 * that it holds no NULL (else its match row ids are collected). */
struct EmitColumn {
    ColView col; /* rid_a unused: the match row ids */
    uint8_t *pages;
    int32_t from_build;
    int32_t direct_only; /* not beside an open-addressing table: the two would
                            not stay in L2 together                       */
};
constexpr int kEmitColumns = 8;
/* A probe of repeated keys leaves the matches of a row with kRunFrom build
 * rows or more to a kernel that follows it: runs of at most kRunRows of them.
 * Room for capacity / kRunFrom runs is enough: one has that many matches at
 * least, on the mean of its row's. */
constexpr uint32_t kRunFrom = 64, kRunRows = 960;
struct alignas(16) MatchRun {
    int64_t key;
    uint32_t rows, count; /* place in the table's `rows`, matches */
    uint32_t at, probe;   /* first output position, probe row     */
};
struct RunList {
    MatchRun *runs = nullptr; /* null: written by the probe itself */
    unsigned long long *count = nullptr; /* zero before the probe */
    uint64_t capacity = 0;
};
struct UniqueOut {
    MatchOut match;      /* capacity: at least the probe rows         */
    bool need_b, need_p; /* match row ids wanted whatever the columns */
    int n;
    EmitColumn cols[kEmitColumns];
    RunList runs; /* of a probe of repeated keys */
};
/* Probe of a unique table; does nothing when the table is unusable. The
 * match counter must be zero before. */
cudaError_t launch_probe_unique(const Launch &L, const ProbeKey &k, uint32_t n, const UniqueTable &t,
                                const UniqueOut &out);

/* Table of build keys that repeat, over a dense range: entries[key - lo] is
 * the key's build row count (high word) and, for one, the row itself, for
 * more, the end of its rows in `rows` (low word). */
struct MultiTable {
    unsigned long long *entries; /* span + 1 */
    uint32_t *rows;              /* build rows */
    int64_t lo;
    uint32_t span;
};
cudaError_t launch_multi_build(const Launch &L, const ColView &key, uint32_t n, const MultiTable &t);
/* Probe of it; the match counter must be zero before. When the count ends
 * above out.match.capacity the output is incomplete: run again with room. */
cudaError_t launch_probe_multi(const Launch &L, const ProbeKey &k, uint32_t n, const MultiTable &t,
                               const UniqueOut &out);

/* The same over any range that leaves a key free for the empty slots: open
 * addressing, a slot per key with its count and its row or the end of its
 * rows. `found` (zero before the build) receives what the device found. */
struct alignas(16) MultiSlot {
    unsigned long long key;
    uint32_t low, count;
};
struct OpenMultiTable {
    MultiSlot *slots;
    uint32_t *rows;              /* build rows                              */
    uint32_t *slot_of;           /* build rows: scratch of the build        */
    unsigned long long *found;   /* kMultiWords words                       */
    unsigned long long lo, width, empty; /* smallest key, largest - smallest,
                                    the key of an empty slot                */
    uint32_t nslots;             /* at least twice the build rows, a multiple of 8 */
    uint8_t *tags;               /* nslots, zero before the build           */
};
enum MultiWord {
    kMultiKeys = 0,   /* different keys                                      */
    kMultiGaveUp = 1, /* a key's walk reached kMaxWalk: the table is unusable */
    kMultiCursor = 2,
    kMultiMost = 3,   /* most build rows of a key                            */
    kMultiWords = 4
};
/* Estimate of the different keys among n build rows, from those whose hash ends
 * in `shift` zero bits (about kSampleRows rows): each sets a bit of `bits`
 * (kSampleBits, zero before, as *found, the number of bits set). */
constexpr uint32_t kSampleBits = 1u << 20, kSampleRows = 1u << 17;
cudaError_t launch_key_sample(const Launch &L, const ColView &key, uint32_t n, uint32_t *bits, unsigned long long *found,
                              uint32_t *shift);
uint64_t sampled_keys(unsigned long long found, uint32_t shift);

cudaError_t launch_open_multi_build(const Launch &L, const ColView &key, uint32_t n, const OpenMultiTable &t);
cudaError_t launch_probe_open_multi(const Launch &L, const ProbeKey &k, uint32_t n, const OpenMultiTable &t,
                                    const UniqueOut &out);

/* The build for the joins of a batch level: task k owns blocks [key_base,
 * key_base + key_blocks) of the passes over its rows and [fill_base, ...) of
 * the fill. */
struct UniqueBuildTask {
    ColView key;
    UniqueTable table;
    uint32_t n;
    uint32_t key_base, key_blocks, fill_base, fill_blocks; /* place_unique */
};
struct UniqueGrid {
    uint32_t key = 0, fill = 0;
};
UniqueGrid place_unique(const Launch &L, UniqueBuildTask *tasks, size_t n);
cudaError_t launch_unique_build_grouped(const Launch &L, const UniqueBuildTask *tasks_dev, uint32_t n,
                                        const UniqueGrid &g);

/* Probe and nested loop share one tiled kernel; `sched` is scratch of
 * probe_sched_bytes(n_probe) bytes (the tile ticket). */
size_t probe_sched_bytes(uint32_t n_probe);
/* inline_dir: the table was built with BuildPlan::inline_first (INT32
 * keys only; ignored for INT64). */
cudaError_t launch_probe_tiles_hash(const Launch &L, const ColView &pkey, uint32_t n_probe,
                                    int32_t build_key_type, const uint64_t *dir,
                                    const void *tuples, int log2_slots, const uint16_t *bloom,
                                    const MatchOut &out, void *sched, bool inline_dir = true);

/* Nested loop (build side <= 64 rows) */
constexpr uint32_t kNestedLoopMax = 64;
cudaError_t launch_nl_collect(const Launch &L, const ColView &bkey, uint32_t n_build,
                              int64_t *keys, uint32_t *rids, uint32_t *count);
cudaError_t launch_nl_probe_tiles(const Launch &L, const ColView &pkey, uint32_t n_probe,
                                  const int64_t *keys, const uint32_t *rids,
                                  const uint32_t *count, const MatchOut &out, void *sched);

/* Grouped probe over the joins of one batch level. */
struct ProbeTask {
    ColView pkey;
    uint32_t n_probe;
    int32_t kind;           /* 0 hash, 1 nested loop, 2 the direct-mapped table
                               `unique` when it is usable, else hash       */
    int32_t build_key_type; /* hash: CJ_INT32 / CJ_INT64 tuples            */
    int32_t log2_slots;
    const uint64_t *dir;
    const void *tuples;
    const int64_t *nl_keys;
    const uint32_t *nl_rids;
    const uint32_t *nl_count;
    UniqueTable unique;         /* kind 2 (open_slots 0) */
    MatchOut out;               /* out.counter zeroed before launch         */
    uint32_t num_tiles;
    uint32_t tile_base;         /* first global tile of this task           */
};
uint32_t probe_tiles(uint32_t n_probe);
/* `ticket` must be zeroed, and each task's counter. */
cudaError_t launch_probe_grouped(const Launch &L, const ProbeTask *tasks_dev, uint32_t ntasks,
                                 uint32_t total_tiles, unsigned int *ticket, const uint16_t *bloom);
struct NlCollectTask {
    ColView bkey;
    uint32_t n_build;
    int64_t *keys;
    uint32_t *rids;
    uint32_t *count;
};
cudaError_t launch_nl_collect_grouped(const Launch &L, const NlCollectTask *tasks_dev, uint32_t ntasks);

/* Raises DEV_ERR_STALE unless counts[i] == expected[i] for every i < n. */
cudaError_t launch_check_counts(const Launch &L, const unsigned long long *counts,
                                const unsigned long long *expected, uint32_t n,
                                unsigned long long *detail, uint32_t check_id);

/* Intermediates: out[i] = src[idx[i]] */
cudaError_t launch_gather_u32(const Launch &L, const uint32_t *src,
                              const uint32_t *idx, uint64_t n, uint32_t *out);

/* Grouped variants for batches: each task's units are numbered from
 * page_base / chunk_base in a global sequence (prefix sums over tasks). */
constexpr uint64_t kGatherChunk = 8192;
struct GatherTask {
    const uint32_t *src;
    const uint32_t *idx;
    uint32_t *out;
    uint64_t n;
    uint64_t chunk_base;
};
cudaError_t launch_gather_grouped(const Launch &L, const GatherTask *tasks_dev, uint32_t ntasks,
                                  uint64_t total_chunks);
/* One fixed-width result column. `rows` are the rows to write or, with
 * `rows_dev` set, the capacity the pages were sized for while the count
 * itself is read on the device (a match counter the host has not read yet).
 * finish 1: the values are in place already (a NULL-free column written by
 * the probe); headers (n_rows = n_values), zero gaps and all-ones bitmaps
 * only. finish 2: so if the device finds that `col` holds no NULL, else the
 * pages are written through its row ids. */
struct PageTask {
    ColView col;
    uint64_t rows;
    const unsigned long long *rows_dev;
    uint8_t *out;
    int32_t finish;
    const unsigned long long *table; /* finish 2, with the table words set: also
                                        written through the row ids unless the
                                        table is direct-mapped                 */
    uint32_t block_base, blocks; /* place_pages */
};
constexpr int kPageArgs = 24; /* tasks passed by value */
uint32_t place_pages(const Launch &L, PageTask *tasks, size_t n); /* returns the grid */
cudaError_t launch_write_pages(const Launch &L, PageTask *tasks, size_t n);
cudaError_t launch_write_pages_grouped(const Launch &L, const PageTask *tasks_dev, uint32_t n, uint32_t grid);

/* Output pages */
uint32_t rows_per_page_fixed(int32_t type);
/* One VARCHAR result column. launch_varchar with `plan` cuts its rows into
 * pages and leaves their number in *total_pages (done and total_pages zero
 * before); without it the pages are written to `out`, sized by that number. */
struct VarcharTask {
    ColView col;
    uint64_t rows;
    unsigned int *done;
    unsigned long long *total_pages;
    uint8_t *out;
    uint32_t tile_rows, tiles; /* from here on: place_varchar */
    uint32_t *tile_pages, *nseg, *seg, *seg_page;
    uint64_t *tile_base, *row_desc;
    uint32_t tile_first;
};
constexpr int kVarcharArgs = 16; /* tasks passed by value */
size_t varchar_temp_bytes(uint64_t rows, uint32_t tile_rows);
void place_varchar(VarcharTask &t, uint32_t tile_rows, void *temp);
cudaError_t launch_varchar(const Launch &L, const VarcharTask *tasks, size_t n, bool plan);

} // namespace cj
