/*
 * k_unique.cu — joins over unique build keys, and over repeated ones: the
 * tables' builds and a probe that reads the key column's pages and writes the
 * result's pages.
 *
 * The table (launch_unique_build) is direct-mapped when the keys lie densely
 * (slots[key - lo] = build row), else open-addressing, at most half full
 * (slots of 8 bytes, key << 32 | build row, and linear probing from the key's
 * hash; for INT64 keys of 16 bytes, key and build row, in groups of eight with
 * a tag byte per slot). Which one, and whether the keys are unique at all, is
 * decided on the device: `params` says so to the kernels that follow and,
 * at the next synchronisation, to the host. Both kinds share one buffer.
 *
 * The probe (k_probe_unique) takes up to 2,048 probe rows per CTA and step:
 * a page of the key column when the probe side is a scan (NULLs resolved
 * from the page's own bitmap: no decoded copy of the column is written or
 * read back), else 2,048 rows of an intermediate. A lane has eight
 * independent rows: their keys are all requested before any is used, then
 * all their slots, then (for a result column without NULLs) their values.
 * One atomicAdd per step places the matches, and the values of the root's
 * fixed-width columns without NULLs go straight to their places in the
 * result pages: no match row ids are written and read back for them.
 * Columns with NULLs (known on the device only) get their row ids and are
 * written by k_write_pages.
 *
 * Keys that repeat get a table of their own (a count, and the row or where
 * the key's rows lie: per value of a dense range, launch_multi_build, else in
 * an open-addressing slot per key, launch_open_multi_build) and the same probe
 * with room for several matches a row; rows with many are listed and written
 * by a kernel of their own (k_match_runs).
 *
 * Bound: requests from L1 to L2, about one per clock and SM whatever their
 * size (every random slot or value is one), then the 128-byte lines of L1
 * that the requests in flight hold. 64M x 4M rows, 43.9M matches, two
 * 8-byte result columns, direct-mapped: 575 us, where decode, probe and
 * page writers took 945 us (152 + 390 + 403).
 */
#include <algorithm>
#include <atomic>
#include <cmath>

#include "cj_device.cuh"

namespace cj {
namespace {

constexpr unsigned long long kOpenEmpty = ~0ull; /* row 2^32-1 never exists */

/* ---------------- build ---------------- */
constexpr int kUniqueThreads = 256;
constexpr int kUniqueRows = 4; /* build rows a thread has in flight */

/* Smallest / largest key (as unsigned order: XOR 2^63; the smallest as its
 * complement, so that zeroed words are the identity) and count of the
 * non-NULL keys, folded over the block into p[0..2]. */
CJ_DEV void fold_range(const ColView &key, uint64_t first, uint64_t n, uint64_t stride, unsigned long long *p) {
    __shared__ unsigned long long s_lo[32], s_hi[32];
    __shared__ uint32_t s_cnt[32];
    unsigned long long lo = 0, hi = 0;
    uint32_t cnt = 0;
    for (uint64_t i0 = first; i0 < n; i0 += stride * kUniqueRows) {
        int64_t k[kUniqueRows];
        bool v[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            const uint64_t i = i0 + q * stride;
            v[q] = i < n && load_key(key, (uint32_t)i, &k[q]);
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q)
            if (v[q]) {
                const unsigned long long b = (unsigned long long)k[q] ^ (1ull << 63);
                lo = max(lo, ~b);
                hi = max(hi, b);
                ++cnt;
            }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, d));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    const uint32_t warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    if (lane_id() == 0) {
        s_lo[warp] = lo;
        s_hi[warp] = hi;
        s_cnt[warp] = cnt;
    }
    __syncthreads();
    if (warp == 0) {
        lo = lane_id() < nwarps ? s_lo[lane_id()] : 0;
        hi = lane_id() < nwarps ? s_hi[lane_id()] : 0;
        cnt = lane_id() < nwarps ? s_cnt[lane_id()] : 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            lo = max(lo, __shfl_xor_sync(0xffffffffu, lo, d));
            hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
        }
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane_id() == 0 && cnt) {
            atomicMax(p, lo);
            atomicMax(p + 1, hi);
            atomicAdd(p + 2, (unsigned long long)cnt);
        }
    }
}

/* Reads the folded range (from L2: other blocks wrote it) and decides. */
CJ_DEV void decide_table(unsigned long long *p, uint64_t max_span, bool wide) {
    const unsigned long long cnt = __ldcg(p + 2);
    if (cnt == 0) return; /* no non-NULL key: span 0, nothing matches */
    const unsigned long long b = ~__ldcg(p), e = __ldcg(p + 1), width = e - b; /* max - min: the bias cancels */
    p[kTableEmpty] = (e != ~0ull ? e + 1 : b - 1) ^ (1ull << 63);
    if (width >= max_span) p[kTableRefused] = wide && b == 0 && e == ~0ull ? kTableWhole : kTableSpread;
    else if (cnt > width + 1) p[kTableRefused] = kTableRepeats; /* more keys than values in their range */
    p[kTableLo] = b ^ (1ull << 63);
    p[kTableSpan] = width + 1;
}

/* A slot of an open-addressing table of INT64 keys. */
struct alignas(16) WideSlot {
    unsigned long long key;
    uint32_t rid, pad;
};

CJ_DEV uint8_t *wide_tags(const UniqueTable &t) {
    return reinterpret_cast<uint8_t *>(t.slots) + (uint64_t)t.open_slots * sizeof(WideSlot);
}

/* Empty slots are all ones, but for wide ones, whose key is kTableEmpty; their
 * tags are 0. */
CJ_DEV uint64_t table_bytes(const UniqueTable &t) {
    const unsigned long long refused = t.params[kTableRefused];
    if (refused == kTableSpread) return (uint64_t)t.open_slots * (t.wide ? 17 : 8);
    return refused ? 0ull : t.params[kTableSpan] * 4ull;
}
CJ_DEV void fill_table(const UniqueTable &t, uint64_t first, uint64_t stride) {
    const uint64_t bytes = table_bytes(t), n16 = (bytes + 15) / 16; /* the buffer is a multiple of 16 bytes */
    uint4 empty = make_uint4(~0u, ~0u, ~0u, ~0u);
    if (t.wide && t.params[kTableRefused] == kTableSpread) {
        empty.x = (uint32_t)t.params[kTableEmpty];
        empty.y = (uint32_t)(t.params[kTableEmpty] >> 32);
    }
    const bool open = t.params[kTableRefused] == kTableSpread;
    const uint64_t tags = open && t.wide ? (uint64_t)t.open_slots : n16; /* where they begin */
    for (uint64_t i = first; i < n16; i += stride)
        reinterpret_cast<uint4 *>(t.slots)[i] = i < tags ? empty : make_uint4(0u, 0u, 0u, 0u);
}

/* The keys repeat, or pile up. Written once, or nearly: thousands of stores
 * to the one word that every thread also reads took 310 of the insert's 435
 * us (3M rows, a quarter of the keys twice). */
CJ_DEV void flag_once(unsigned long long *word) {
    if (!*reinterpret_cast<volatile unsigned long long *>(word)) *reinterpret_cast<volatile unsigned long long *>(word) = 1ull;
}

/* Each key claims its slot; meeting its own key there means that the keys
 * repeat, and the table cannot be used. kUniqueRows rows per thread and
 * step, their compare-and-swaps all in flight together. */
CJ_DEV void insert_rows(const ColView &key, const UniqueTable &t, uint64_t first, uint64_t n, uint64_t stride) {
    const unsigned long long refused = t.params[kTableRefused];
    if (refused == 0) {
        uint32_t *slots = reinterpret_cast<uint32_t *>(t.slots);
        const uint64_t lo = t.params[kTableLo], span = t.params[kTableSpan];
        for (uint64_t i0 = first; i0 < n; i0 += stride * kUniqueRows) {
            uint64_t off[kUniqueRows];
#pragma unroll
            for (int q = 0; q < kUniqueRows; ++q) {
                const uint64_t i = i0 + q * stride;
                int64_t k;
                off[q] = i < n && load_key(key, (uint32_t)i, &k) ? (uint64_t)k - lo : ~0ull;
            }
            uint32_t was[kUniqueRows];
#pragma unroll
            for (int q = 0; q < kUniqueRows; ++q)
                was[q] = off[q] < span ? atomicCAS(slots + off[q], kArrayEmpty, (uint32_t)(i0 + q * stride))
                                       : kArrayEmpty;
            bool dup = false;
#pragma unroll
            for (int q = 0; q < kUniqueRows; ++q) dup |= was[q] != kArrayEmpty;
            if (dup) flag_once(t.params + kTableDup);
        }
        return;
    }
    if (refused != kTableSpread || !t.open_slots) return;
    if (t.wide) {
        WideSlot *slots = reinterpret_cast<WideSlot *>(t.slots);
        const unsigned long long empty = t.params[kTableEmpty];
        for (uint64_t i = first; i < n; i += stride) {
            if (*reinterpret_cast<volatile unsigned long long *>(t.params + kTableDup)) return;
            int64_t k;
            if (!load_key(key, (uint32_t)i, &k)) continue;
            const TagHash h = tag_hash(k, t.open_slots / 8);
            for (uint32_t step = 0;; ++step) {
                const uint32_t at = tagged_slot(h, step, t.open_slots / 8);
                unsigned long long cur = __ldcg(&slots[at].key);
                if (cur == empty) {
                    cur = atomicCAS(&slots[at].key, empty, (unsigned long long)k);
                    if (cur == empty) {
                        slots[at].rid = (uint32_t)i;
                        wide_tags(t)[at] = (uint8_t)h.tag;
                        break;
                    }
                }
                if (cur == (unsigned long long)k || step == kMaxWalk) {
                    flag_once(t.params + kTableDup);
                    break;
                }
            }
        }
        return;
    }
    unsigned long long *slots = reinterpret_cast<unsigned long long *>(t.slots);
    for (uint64_t i = first; i < n; i += stride) {
        /* a repeat is flagged once; every thread then stops */
        if (*reinterpret_cast<volatile unsigned long long *>(t.params + kTableDup)) return;
        int64_t k;
        if (!load_key(key, (uint32_t)i, &k)) continue;
        const unsigned long long v = ((unsigned long long)(uint32_t)k << 32) | (unsigned long long)i;
        uint32_t h = open_slot(k, t.open_slots);
        for (uint32_t step = 0;; ++step) {
            unsigned long long cur = __ldcg(slots + h); /* slots only fill: a full one is final */
            if (cur == kOpenEmpty) {
                cur = atomicCAS(slots + h, kOpenEmpty, v);
                if (cur == kOpenEmpty) break;
            }
            if ((uint32_t)(cur >> 32) == (uint32_t)k || step == kMaxWalk) {
                flag_once(t.params + kTableDup);
                break;
            }
            if (++h == t.open_slots) h = 0;
        }
    }
}

__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_range(ColView key_arg, uint32_t n, UniqueTable t) {
    const ColView key = resolve_view(key_arg);
    fold_range(key, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, n, (uint64_t)gridDim.x * blockDim.x, t.params);
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(t.params + kTableDone, 1ull) == gridDim.x - 1) {
            __threadfence();
            decide_table(t.params, t.max_span, t.wide);
        }
    }
}

__global__ void __launch_bounds__(kUniqueThreads) k_unique_fill(UniqueTable t) {
    fill_table(t, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, (uint64_t)gridDim.x * blockDim.x);
}

__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_insert(ColView key_arg, uint32_t n, UniqueTable t) {
    const ColView key = resolve_view(key_arg);
    insert_rows(key, t, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, n, (uint64_t)gridDim.x * blockDim.x);
}

/* A small build side: the three passes by one block, one launch. */
constexpr int kSmallThreads = 1024;
constexpr uint32_t kSmallRows = 8192;
__global__ void __launch_bounds__(kSmallThreads)
    k_unique_small(ColView key_arg, uint32_t n, UniqueTable t) {
    const ColView key = resolve_view(key_arg);
    fold_range(key, threadIdx.x, n, kSmallThreads, t.params);
    __syncthreads();
    if (threadIdx.x == 0) decide_table(t.params, t.max_span, t.wide);
    __syncthreads();
    fill_table(t, threadIdx.x, kSmallThreads);
    __syncthreads();
    insert_rows(key, t, threadIdx.x, n, kSmallThreads);
}

/* The three passes for every candidate join of a batch level (one launch
 * less than with a pass of its own for the decision). */
CJ_DEV uint32_t find_build(const UniqueBuildTask *tasks, uint32_t ntasks, uint32_t block, bool fill) {
    uint32_t lo = 0, hi = ntasks;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((fill ? tasks[mid].fill_base : tasks[mid].key_base) <= block) lo = mid;
        else hi = mid;
    }
    return lo;
}
__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_range_grouped(const UniqueBuildTask *__restrict__ tasks, uint32_t ntasks) {
    const UniqueBuildTask &T = tasks[find_build(tasks, ntasks, blockIdx.x, false)];
    const ColView key = resolve_view(T.key);
    const uint64_t b = blockIdx.x - T.key_base;
    fold_range(key, b * blockDim.x + threadIdx.x, T.n, (uint64_t)T.key_blocks * blockDim.x, T.table.params);
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(T.table.params + kTableDone, 1ull) == T.key_blocks - 1) {
            __threadfence();
            decide_table(T.table.params, T.table.max_span, T.table.wide);
        }
    }
}
__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_fill_grouped(const UniqueBuildTask *__restrict__ tasks, uint32_t ntasks) {
    const UniqueBuildTask &T = tasks[find_build(tasks, ntasks, blockIdx.x, true)];
    const uint64_t b = blockIdx.x - T.fill_base;
    fill_table(T.table, b * blockDim.x + threadIdx.x, (uint64_t)T.fill_blocks * blockDim.x);
}
__global__ void __launch_bounds__(kUniqueThreads)
    k_unique_insert_grouped(const UniqueBuildTask *__restrict__ tasks, uint32_t ntasks) {
    const UniqueBuildTask &T = tasks[find_build(tasks, ntasks, blockIdx.x, false)];
    const ColView key = resolve_view(T.key);
    const uint64_t b = blockIdx.x - T.key_base;
    insert_rows(key, T.table, b * blockDim.x + threadIdx.x, T.n, (uint64_t)T.key_blocks * blockDim.x);
}

/* Build of a table of repeated keys: count, place, scatter (launch_multi_build). */
__global__ void __launch_bounds__(kUniqueThreads) k_multi_count(ColView key_arg, uint32_t n, MultiTable t) {
    const ColView key = resolve_view(key_arg);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * kUniqueRows) {
        uint64_t off[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            const uint64_t i = i0 + q * stride;
            int64_t k;
            off[q] = i < n && load_key(key, (uint32_t)i, &k) ? (uint64_t)k - (uint64_t)t.lo : ~0ull;
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q)
            if (off[q] < t.span) atomicAdd(reinterpret_cast<uint32_t *>(t.entries + off[q]) + 1, 1u);
    }
}

/* A place in `rows` for every value with two build rows or more. One
 * atomicAdd per 2,048 values: the places' order does not matter. */
constexpr int kPlaceItems = 8;
__global__ void __launch_bounds__(kUniqueThreads) k_multi_place(MultiTable t) {
    __shared__ uint32_t wbuf[kUniqueThreads / 32 + 1];
    __shared__ uint32_t s_base;
    uint32_t *cursor = reinterpret_cast<uint32_t *>(t.entries + t.span);
    for (uint64_t v0 = (uint64_t)blockIdx.x * kUniqueThreads * kPlaceItems; v0 < t.span;
         v0 += (uint64_t)gridDim.x * kUniqueThreads * kPlaceItems) {
        uint32_t c[kPlaceItems], sum = 0, total;
#pragma unroll
        for (int q = 0; q < kPlaceItems; ++q) {
            const uint64_t v = v0 + q * kUniqueThreads + threadIdx.x;
            c[q] = v < t.span ? (uint32_t)(t.entries[v] >> 32) : 0u;
            if (c[q] > 1) sum += c[q];
        }
        const uint32_t pre = block_exclusive_scan<uint32_t>(sum, wbuf, &total);
        if (threadIdx.x == 0) s_base = total ? atomicAdd(cursor, total) : 0u;
        __syncthreads();
        uint32_t at = s_base + pre;
#pragma unroll
        for (int q = 0; q < kPlaceItems; ++q) {
            const uint64_t v = v0 + q * kUniqueThreads + threadIdx.x;
            if (c[q] < 2) continue;
            *reinterpret_cast<uint32_t *>(t.entries + v) = at;
            at += c[q];
        }
        __syncthreads();
    }
}

/* A single row goes into its entry; rows of a repeated key to their places,
 * which moves the entry's low word on to the end of the key's rows. */
__global__ void __launch_bounds__(kUniqueThreads) k_multi_scatter(ColView key_arg, uint32_t n, MultiTable t) {
    const ColView key = resolve_view(key_arg);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * kUniqueRows) {
        uint64_t off[kUniqueRows];
        uint32_t c[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            const uint64_t i = i0 + q * stride;
            int64_t k;
            off[q] = i < n && load_key(key, (uint32_t)i, &k) ? (uint64_t)k - (uint64_t)t.lo : ~0ull;
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) /* counts no longer change */
            c[q] = off[q] < t.span ? reinterpret_cast<const uint32_t *>(t.entries + off[q])[1] : 0u;
        uint32_t at[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            uint32_t *low = reinterpret_cast<uint32_t *>(t.entries + (c[q] ? off[q] : 0));
            if (c[q] == 1) *low = (uint32_t)(i0 + q * stride);
            else if (c[q]) at[q] = atomicAdd(low, 1u);
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q)
            if (c[q] > 1) t.rows[at[q]] = (uint32_t)(i0 + q * stride);
    }
}

/* Build of the open-addressing one: claim a slot per key and count, place,
 * scatter. The slot of each row is kept for the scatter (4 bytes a row, a
 * walk less). Bound by the random accesses: two to the table per row in the
 * claim (a read and the count's add), two in the scatter. */
__global__ void __launch_bounds__(kUniqueThreads) k_open_multi_fill(OpenMultiTable t) {
    const uint4 empty = make_uint4((uint32_t)t.empty, (uint32_t)(t.empty >> 32), 0u, 0u);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < t.nslots; i += stride) {
        reinterpret_cast<uint4 *>(t.slots)[i] = empty;
        t.tags[i] = 0;
    }
}
__global__ void __launch_bounds__(kUniqueThreads) k_open_multi_claim(ColView key_arg, uint32_t n, OpenMultiTable t) {
    const ColView key = resolve_view(key_arg);
    const uint32_t groups = t.nslots / 8;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * kUniqueRows) {
        unsigned long long k[kUniqueRows], cur[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            const uint64_t i = i0 + q * stride;
            int64_t v;
            k[q] = i < n && load_key(key, (uint32_t)i, &v) ? (unsigned long long)v : t.empty; /* no row's key */
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q)
            cur[q] = k[q] != t.empty ? __ldcg(&t.slots[tagged_slot(tag_hash((int64_t)k[q], groups), 0, groups)].key) : t.empty;
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            uint32_t at = ~0u;
            if (k[q] != t.empty) {
                const TagHash h = tag_hash((int64_t)k[q], groups);
                unsigned long long c = cur[q];
                for (uint32_t step = 0; step <= kMaxWalk; ++step) {
                    const uint32_t s = tagged_slot(h, step, groups);
                    if (step) c = __ldcg(&t.slots[s].key); /* slots only fill: a full one is final */
                    if (c == t.empty) {
                        c = atomicCAS(&t.slots[s].key, t.empty, k[q]);
                        if (c == t.empty) {
                            c = k[q];
                            t.tags[s] = (uint8_t)h.tag;
                        }
                    }
                    if (c == k[q]) {
                        at = s;
                        break;
                    }
                }
                if (at != ~0u) atomicAdd(&t.slots[at].count, 1u);
                else flag_once(t.found + kMultiGaveUp);
            }
            if (i0 + q * stride < n) t.slot_of[i0 + q * stride] = at;
        }
    }
}
__global__ void __launch_bounds__(kUniqueThreads) k_open_multi_place(OpenMultiTable t) {
    __shared__ uint32_t wbuf[kUniqueThreads / 32 + 1];
    __shared__ unsigned long long s_base;
    uint32_t keys = 0, most = 0;
    for (uint64_t v0 = (uint64_t)blockIdx.x * kUniqueThreads * kPlaceItems; v0 < t.nslots;
         v0 += (uint64_t)gridDim.x * kUniqueThreads * kPlaceItems) {
        uint32_t c[kPlaceItems], sum = 0, total;
#pragma unroll
        for (int q = 0; q < kPlaceItems; ++q) {
            const uint64_t v = v0 + q * kUniqueThreads + threadIdx.x;
            c[q] = v < t.nslots ? t.slots[v].count : 0u;
            keys += c[q] > 0;
            most = max(most, c[q]);
            if (c[q] > 1) sum += c[q];
        }
        const uint32_t pre = block_exclusive_scan<uint32_t>(sum, wbuf, &total);
        if (threadIdx.x == 0) s_base = total ? atomicAdd(t.found + kMultiCursor, (unsigned long long)total) : 0ull;
        __syncthreads();
        uint32_t at = (uint32_t)s_base + pre;
#pragma unroll
        for (int q = 0; q < kPlaceItems; ++q) {
            if (c[q] < 2) continue;
            t.slots[v0 + q * kUniqueThreads + threadIdx.x].low = at;
            at += c[q];
        }
        __syncthreads();
    }
    keys = __reduce_add_sync(0xffffffffu, keys);
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane_id() == 0 && keys) {
        atomicAdd(t.found + kMultiKeys, (unsigned long long)keys);
        atomicMax(t.found + kMultiMost, (unsigned long long)most);
    }
}
__global__ void __launch_bounds__(kUniqueThreads) k_open_multi_scatter(uint32_t n, OpenMultiTable t) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * kUniqueRows) {
        uint32_t h[kUniqueRows], c[kUniqueRows], at[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) h[q] = i0 + q * stride < n ? __ldcs(t.slot_of + i0 + q * stride) : ~0u;
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) c[q] = h[q] != ~0u ? t.slots[h[q]].count : 0u; /* no longer change */
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            if (c[q] == 1) t.slots[h[q]].low = (uint32_t)(i0 + q * stride);
            else if (c[q]) at[q] = atomicAdd(&t.slots[h[q]].low, 1u);
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q)
            if (c[q] > 1) t.rows[at[q]] = (uint32_t)(i0 + q * stride);
    }
}

/* Linear counting (Whang, Vander-Zanden and Taylor) of a part of the keys: b of
 * m bits set by hashing say -m ln(1 - b / m) keys, within about a percent here. The
 * keys are sampled by their hash, so that all rows of a key are in or out.
 * Bound by reading the keys and their round trips: 3M rows 29 us. The mixing is
 * MurmurHash3's 32-bit finaliser. */
__global__ void __launch_bounds__(kUniqueThreads)
    k_key_sample(ColView key_arg, uint32_t n, uint32_t shift, uint32_t *bits, unsigned long long *found) {
    const ColView key = resolve_view(key_arg);
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t mine = 0;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * kUniqueRows) {
        int64_t k[kUniqueRows];
        bool v[kUniqueRows];
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            const uint64_t i = i0 + q * stride;
            v[q] = i < n && load_key(key, (uint32_t)i, &k[q]);
        }
#pragma unroll
        for (int q = 0; q < kUniqueRows; ++q) {
            if (!v[q]) continue;
            uint32_t h = (uint32_t)(hash_key(k[q]) >> 32);
            h ^= h >> 16;
            h *= 0x85EBCA6Bu;
            h ^= h >> 13;
            h *= 0xC2B2AE35u;
            h ^= h >> 16;
            if (h & ((1u << shift) - 1u)) continue;
            const uint32_t at = h >> 12, bit = 1u << (at & 31u);
            static_assert(kSampleBits == 1u << 20, "the hash's 20 top bits");
            if (!(__ldcg(bits + at / 32) & bit)) mine += (atomicOr(bits + at / 32, bit) & bit) == 0;
        }
    }
    __shared__ uint32_t s_mine;
    if (threadIdx.x == 0) s_mine = 0;
    __syncthreads();
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane_id() == 0 && mine) atomicAdd(&s_mine, mine);
    __syncthreads();
    if (threadIdx.x == 0 && s_mine) atomicAdd(found, (unsigned long long)s_mine);
}

/* ---------------- probe ---------------- */
/* 256 threads, 48 registers and 10 KB of shared memory: five CTAs per SM.
 * Measured at 64M x 4M rows (probe alone, 575 us since): five 605 us, four
 * with 64 registers 619, six with 40 (spills) 620. */
constexpr int kProbeBlocks = 5;
constexpr int kWideBlocks = 4; /* 64 registers: the codes are 64-bit keys */
/* 80 registers; four with 64, more of them spilled: 1347 us where three take
 * 1314 (30M x 3M INT32 rows, all matching). */
constexpr int kOpenMultiBlocks = 3;
constexpr int kMultiBlocks = 4; /* 64 registers; three with 80 1467 us, five with 48 2343 */
constexpr int kItems = 8;                              /* rows per lane and step       */
constexpr int kProbeThreads = 2048 / kItems;
constexpr int kParts = kProbeThreads / 32;
constexpr uint32_t kWarpRows = 32 * kItems;            /* 256                          */
constexpr uint32_t kTileRows = kWarpRows * kProbeThreads / 32; /* 2048: a full page */

/* A row's key as the table sees it (direct-mapped: key - lo; open
 * addressing: the key's 32 bits), its build row (kArrayEmpty: no match).
 * For INT32 probe keys the table's range is cut to INT32's first, so that a
 * 32-bit difference says all. */
template <typename T> struct DirectLookup {
    const uint32_t *slots;
    int64_t lo;
    uint32_t span; /* at most 2^28 */
    CJ_DEV DirectLookup(const uint32_t *table, int64_t first, uint32_t values) {
        int64_t skip = 0;
        if constexpr (sizeof(T) == 4) {
            const int64_t end = min(first + (int64_t)values, (int64_t)INT32_MAX + 1), cut = max(first, (int64_t)INT32_MIN);
            values = end > cut ? (uint32_t)(end - cut) : 0u;
            skip = values ? cut - first : 0;
        }
        slots = table + skip;
        lo = first + skip;
        span = values;
    }
    using Code = uint32_t;
    static constexpr bool kMask = false; /* a code says by itself whether it may be in the table */
    CJ_DEV uint32_t code(T key, bool present, bool *in) const {
        *in = true;
        uint32_t c;
        if constexpr (sizeof(T) == 4) {
            c = (uint32_t)key - (uint32_t)lo;
        } else {
            const uint64_t off = (uint64_t)key - (uint64_t)lo; /* keys below lo wrap past span */
            c = off < span ? (uint32_t)off : ~0u;
        }
        return present ? c : ~0u;
    }
    CJ_DEV T key_of(uint32_t c) const { return (T)(lo + c); }
    CJ_DEV void find(const uint32_t *c, uint32_t, uint32_t *rid) const {
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            rid[it] = kArrayEmpty;
            if (c[it] < span) rid[it] = __ldg(slots + c[it]);
        }
    }
};

/* Open addressing: the first slots of all of a lane's rows in flight
 * together, then slot by slot (a neighbour is mostly in the sector that just
 * came) until the key or an empty slot. Keys outside the build keys' range
 * are not looked up at all. The bound is the requests that L1 sends out,
 * about one per clock and SM: reading the slot's aligned 32 bytes at once
 * took 858 us where this takes 797 (64M rows, without the range), whatever
 * the table's size between 1.3 and 2 slots a row. */
template <typename T> struct OpenLookup {
    const unsigned long long *slots;
    uint32_t nslots, lo, width; /* of the INT32 build keys */
    CJ_DEV OpenLookup(const UniqueTable &t)
        : slots(reinterpret_cast<const unsigned long long *>(t.slots)), nslots(t.open_slots),
          lo((uint32_t)t.params[kTableLo]), width((uint32_t)(t.params[kTableSpan] - 1)) {}
    using Code = uint32_t;
    static constexpr bool kMask = true;
    CJ_DEV uint32_t code(T key, bool present, bool *in) const {
        /* an INT64 key that is no INT32 value equals no build key */
        *in = present && key == (T)(int32_t)key && (uint32_t)key - lo <= width;
        return (uint32_t)key;
    }
    CJ_DEV T key_of(uint32_t c) const { return (T)(int32_t)c; }
    CJ_DEV void find(const uint32_t *c, uint32_t ok, uint32_t *rid) const {
        unsigned long long v[kItems];
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            v[it] = kOpenEmpty;
            if ((ok >> it) & 1u) v[it] = __ldg(slots + open_slot((int64_t)(int32_t)c[it], nslots));
        }
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            rid[it] = kArrayEmpty;
            uint32_t h = open_slot((int64_t)(int32_t)c[it], nslots);
            for (uint32_t step = 0; v[it] != kOpenEmpty && step < nslots; ++step) {
                if ((uint32_t)(v[it] >> 32) == c[it]) {
                    rid[it] = (uint32_t)v[it];
                    break;
                }
                if (++h == nslots) h = 0;
                v[it] = __ldg(slots + h);
            }
        }
    }
};

/* Lookups in a table of tagged 16-byte slots: the tags of four of a lane's rows
 * in flight together, then the slots that they point to (all eight rows' tags
 * at once spill: 661 us where this takes 605, 30M INT64 rows over 3M keys).
 * What is left, a tag that another key shares (one in 128 per key of the group)
 * or a full group, goes group by group. Bound by the random accesses, one for a
 * row without a match and two for one with. Walking the slots to an empty one
 * instead, unique INT64 keys: 30M probe rows over 3M keys, 97 % of them in the
 * range but no key, 803 us, 416 with tags; 10 % of them outside it 619 and 605;
 * 5M rows over 300K keys 125 and 118. */
struct TaggedTable {
    const ulonglong2 *slots; /* key, payload */
    const unsigned long long *tags;
    uint32_t groups;
    CJ_DEV unsigned long long load_tags(uint32_t g) const { return __ldg(tags + g); }
    CJ_DEV ulonglong2 load(uint32_t s) const { return __ldg(slots + s); }
    /* bytes of `w` that may be the tag: their high bits (a byte above a true
     * one may be set too) */
    CJ_DEV static unsigned long long may_be(unsigned long long w, uint32_t tag) {
        const unsigned long long x = w ^ (tag * 0x0101010101010101ull);
        return (x - 0x0101010101010101ull) & ~x & 0x8080808080808080ull;
    }
    CJ_DEV static bool has_empty(unsigned long long w) { return (~w & 0x8080808080808080ull) != 0; }
    CJ_DEV static uint32_t first(unsigned long long m) { return (uint32_t)(__ffsll((long long)m) - 1) >> 3; }
    template <class P> CJ_DEV void walk(int64_t key, P put) const {
        const TagHash h = tag_hash(key, groups);
        uint32_t g = h.group;
        for (uint32_t k = 0; k < groups; ++k) {
            const unsigned long long w = load_tags(g);
            for (unsigned long long m = may_be(w, h.tag); m; m &= m - 1) {
                const ulonglong2 v = load(g * 8 + first(m));
                if (v.x == (unsigned long long)key) {
                    put(v.y);
                    return;
                }
            }
            if (has_empty(w)) return;
            if (++g == groups) g = 0;
        }
    }
    /* put(it, payload) for each row whose key is there */
    template <typename T, class P> CJ_DEV void find(const T *c, uint32_t ok, P put) const {
#pragma unroll
        for (int it = 0; it < kItems; it += 4) {
            unsigned long long w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                w[j] = 0;
                if ((ok >> (it + j)) & 1u) w[j] = load_tags(tag_hash((int64_t)c[it + j], groups).group);
            }
            ulonglong2 v[4];
            uint32_t some = 0, more = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const TagHash h = tag_hash((int64_t)c[it + j], groups);
                const unsigned long long m = may_be(w[j], h.tag);
                if (m) {
                    v[j] = load(h.group * 8 + first(m));
                    some |= 1u << j;
                }
                if ((m & (m - 1)) || (((ok >> (it + j)) & 1u) && !has_empty(w[j]))) more |= 1u << j;
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (((some >> j) & 1u) && v[j].x == (unsigned long long)(int64_t)c[it + j]) put(it + j, v[j].y);
                else if ((more >> j) & 1u) walk((int64_t)c[it + j], [&](unsigned long long y) { put(it + j, y); });
            }
        }
    }
};

/* Open addressing over INT64 build keys. */
template <typename T> struct WideLookup {
    TaggedTable t;
    unsigned long long lo, width;
    using Code = T;
    static constexpr bool kMask = true;
    CJ_DEV WideLookup(const UniqueTable &u)
        : t{reinterpret_cast<const ulonglong2 *>(u.slots), reinterpret_cast<const unsigned long long *>(wide_tags(u)),
            u.open_slots / 8},
          lo(u.params[kTableLo]), width(u.params[kTableSpan] - 1) {}
    CJ_DEV T code(T key, bool present, bool *in) const {
        *in = present && (unsigned long long)(int64_t)key - lo <= width;
        return key;
    }
    CJ_DEV T key_of(T c) const { return c; }
    CJ_DEV void find(const T *c, uint32_t ok, uint32_t *rid) const {
#pragma unroll
        for (int it = 0; it < kItems; ++it) rid[it] = kArrayEmpty;
        t.find(c, ok, [&](int it, unsigned long long y) { rid[it] = (uint32_t)y; });
    }
};

/* A CTA's step takes one page of an INT32 key column (2,048 rows or fewer at
 * a time), or two of an INT64 one side by side: a full page of 8-byte keys
 * has 1,007 rows, and one page a step left half of the warps without any
 * (300K x 5M INT64 rows, the whole join: 352 us, 306 with two). */
template <typename T> constexpr uint32_t kStepPages = sizeof(T) == 4 ? 1 : 2;
template <typename T> constexpr uint32_t kPageParts = kParts / kStepPages<T>; /* warps of a page */
template <typename T> constexpr uint32_t kPageRows = kTileRows / kStepPages<T>;

/* The keys of 256 rows of a page, from row s0 + part * 256 on, as the table
 * sees them: bit `it` of the result set when row it * 32 + lane of them is
 * non-NULL and may be in the table. The value positions come from the
 * bitmap: the words of rows [s0, s0 + kPageRows), one or two per lane, a warp
 * scan of their popcounts; *before: the page's values before row s0, moved
 * on. */
template <typename T, class LK>
CJ_DEV uint32_t page_keys(const uint8_t *pg, uint32_t nr, uint32_t nv, uint32_t s0, uint32_t part, uint32_t *before,
                          const LK &lk, typename LK::Code *code, unsigned int *err) {
    constexpr uint32_t DB = sizeof(T) == 4 ? 4u : 8u;
    constexpr int kWords = kPageRows<T> / 1024;
    const T *vals = reinterpret_cast<const T *>(pg + DB);
    const uint32_t lane = lane_id(), r0 = s0 + part * kWarpRows + lane;
    uint32_t present = 0;
    T v[kItems];
    if (nr == nv) {
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            v[it] = T(0);
            if (r0 + it * 32 < nr) {
                v[it] = __ldcs(vals + r0 + it * 32);
                present |= 1u << it;
            }
        }
    } else {
        const uint32_t nb = (nr + 7) / 8, bm0 = kPageSize - nb;
        const uint32_t *words = reinterpret_cast<const uint32_t *>(pg);
        uint32_t w[kWords], cnt[kWords];
#pragma unroll
        for (int j = 0; j < kWords; ++j) { /* word s0 / 32 + j * 32 + lane of the bitmap */
            const uint32_t first = s0 + (j * 32 + lane) * 32;
            w[j] = 0;
            if (first < nr) {
                const uint32_t b = bm0 + first / 8, al = b >> 2, sh = (b & 3u) * 8;
                const uint32_t lo = __ldg(words + al), hi = al + 1 < kPageSize / 4 ? __ldg(words + al + 1) : 0u;
                w[j] = __funnelshift_r(lo, hi, sh);
                if (nr - first < 32) w[j] &= (1u << (nr - first)) - 1u;
            }
            cnt[j] = __popc(w[j]);
        }
        /* this part's words and the values before each */
        uint32_t word, pre;
        if constexpr (kWords == 2) { /* lanes of one of the two halves */
            const uint32_t t0 = __reduce_add_sync(0xffffffffu, cnt[0]);
            const bool low = part < kParts / 2;
            const uint32_t mine = low ? cnt[0] : cnt[1];
            word = low ? w[0] : w[1];
            pre = *before + (low ? 0u : t0) + warp_inclusive_scan(mine) - mine;
            if (s0 + kPageRows<T> < nr) *before += t0 + __reduce_add_sync(0xffffffffu, cnt[1]);
        } else {
            word = w[0];
            pre = *before + warp_inclusive_scan(cnt[0]) - cnt[0];
            if (s0 + kPageRows<T> < nr) *before += __reduce_add_sync(0xffffffffu, cnt[0]);
        }
        const uint32_t lt = lanemask_lt(), bit = 1u << lane;
        uint32_t most = 0;
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            const int src = (int)(part * kItems + it) & 31;
            const uint32_t bits = __shfl_sync(0xffffffffu, word, src);
            const uint32_t k = __shfl_sync(0xffffffffu, pre, src) + __popc(bits & lt);
            v[it] = T(0);
            const bool here = (bits & bit) != 0;
            most = max(most, here ? k : 0u);
            if (here && k < nv) {
                v[it] = __ldcs(vals + k);
                present |= 1u << it;
            }
        }
        if (nv && most >= nv) atomicOr(err, DEV_ERR_PAGE_HEADER); /* bitmap holds > n_values bits */
        if (!nv && word) atomicOr(err, DEV_ERR_PAGE_HEADER);
    }
    uint32_t ok = 0;
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        bool in;
        code[it] = lk.code(v[it], (present >> it) & 1u, &in);
        if (LK::kMask && in) ok |= 1u << it;
    }
    return ok;
}

/* 256 consecutive values of a column's full pages touch two pages at most:
 * the first one's values and the place of the run in it are the warp's, a
 * value's offset from there fits 32 bits. */
template <typename T> struct PageRun {
    static constexpr uint32_t R = sizeof(T) == 4 ? kRowsPerPageInt32 : kRowsPerPage8B;
    static constexpr uint32_t kGap = kPageSize - R * (uint32_t)sizeof(T); /* bytes of a page that hold no values */
    uint8_t *base;
    uint32_t k0;
    CJ_DEV PageRun(const uint8_t *pages, uint32_t first) {
        const uint32_t p = first / R;
        k0 = first - p * R;
        base = const_cast<uint8_t *>(pages) + (uint64_t)p * kPageSize + (sizeof(T) == 4 ? 4 : 8);
    }
    CJ_DEV T *at(uint32_t i) const {
        const uint32_t k = k0 + i;
        return reinterpret_cast<T *>(base + (k * (uint32_t)sizeof(T) + (k >= R ? kGap : 0u)));
    }
};

/* A warp's matches, packed: what the columns are written from, by full
 * warps and without predicates on the rows that did not match. Kept small:
 * shared memory is taken from L1, and every random load in flight holds a
 * 128-byte line of L1 until it returns. At 64M rows a variant with 37 KB per
 * CTA ran 880 us at five CTAs per SM and 1587 at six. */
struct WarpMatches {
    uint32_t rid[kWarpRows];
    uint8_t row[kWarpRows];
};
constexpr int kEmit = 3; /* matches a lane has in flight */

/* The values of result column c of the warp's n matches, to their places
 * from output position `at` on. */
template <typename T, class W>
CJ_DEV void emit_column(const EmitColumn &c, bool direct, const W &w, uint32_t n, uint32_t at, uint32_t row0) {
    const PageRun<T> out(c.pages, at);
    const bool in_order = !c.from_build && direct && !c.col.rid_b;
    const PageRun<T> in(c.col.pages, row0); /* used when in_order */
    for (uint32_t i0 = lane_id(); i0 < n; i0 += 32 * kEmit) {
        T v[kEmit];
#pragma unroll
        for (int j = 0; j < kEmit; ++j) {
            const uint32_t i = i0 + j * 32;
            if (i >= n) break;
            if (in_order) {
                v[j] = __ldcs(in.at(w.row[i]));
            } else {
                uint32_t r = c.from_build ? w.rid[i] : row0 + w.row[i];
                if (c.col.rid_b) r = __ldg(c.col.rid_b + r);
                v[j] = direct ? page_value<T>(c.col.pages, r) : __ldg(reinterpret_cast<const T *>(c.col.values) + r);
            }
        }
#pragma unroll
        for (int j = 0; j < kEmit; ++j)
            if (i0 + j * 32 < n) __stcs(out.at(i0 + j * 32), v[j]);
    }
}

/* What the kernel writes, worked out once per warp: the result columns that
 * hold no NULL, and the match row ids that the others need. */
struct EmitPlan {
    uint32_t active = 0, direct = 0;
    bool want_b, want_p;
    CJ_DEV EmitPlan(const UniqueOut &out, bool open) : want_b(out.need_b), want_p(out.need_p) {
        for (int c = 0; c < out.n; ++c) {
            const EmitColumn &e = out.cols[c];
            if (col_null_free(e.col) && !(open && e.direct_only)) {
                active |= 1u << c;
                if (col_direct(e.col)) direct |= 1u << c;
            } else if (e.from_build) {
                want_b = true;
            } else {
                want_p = true;
            }
        }
    }
};

struct StepShared {
    WarpMatches matches[kParts];
    uint32_t count[2][kParts];
    unsigned long long base[2];
};

/* Writes a warp's n packed matches from output position `at` on, but for
 * the key column. */
template <class W>
CJ_DEV void emit_packed(const UniqueOut &out, const EmitPlan &plan, const W &w, uint32_t n, uint32_t at,
                        uint32_t row0) {
    const uint32_t lane = lane_id();
    if (plan.want_b)
        for (uint32_t i = lane; i < n; i += 32) __stcs(out.match.build_rids + at + i, w.rid[i]);
    if (plan.want_p)
        for (uint32_t i = lane; i < n; i += 32) __stcs(out.match.probe_rids + at + i, row0 + w.row[i]);
    for (int c = 0; c < out.n; ++c) {
        if (!((plan.active >> c) & 1u)) continue;
        const EmitColumn &e = out.cols[c];
        if (e.col.type == CJ_INT32) emit_column<int32_t>(e, (plan.direct >> c) & 1u, w, n, at, row0);
        else emit_column<long long>(e, (plan.direct >> c) & 1u, w, n, at, row0);
    }
}

/* A CTA's step: every warp looks up its 256 rows and packs their matches,
 * one atomicAdd reserves the step's output (one per warp instead made the
 * counter the bound: 592 us at 64M rows, 800 us with half the rows per
 * warp), and the warps write it. row0: the relation row of the warp's first;
 * ok: a lane's items to look up; buf alternates between steps. Block-wide. */
template <typename T, class LK>
CJ_DEV void probe_step(const LK &lk, const typename LK::Code *code, uint32_t ok, uint32_t row0, const UniqueOut &out,
                       const EmitPlan &plan, StepShared &sh, uint32_t part, uint32_t buf) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    WarpMatches &w = sh.matches[part];
    uint32_t rid[kItems], n = 0, m = 0;
    uint32_t place[(kItems + 3) / 4] = {}; /* of the lane's matches among the warp's: a byte per item */
    lk.find(code, ok, rid);
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const bool hit = rid[it] != kArrayEmpty;
        const uint32_t b = __ballot_sync(0xffffffffu, hit);
        const uint32_t i = n + __popc(b & lt);
        if (hit) {
            w.rid[i] = rid[it];
            w.row[i] = (uint8_t)(it * 32 + lane);
            m |= 1u << it;
        }
        place[it / 4] |= (i & 0xFFu) << (8 * (it % 4));
        n += __popc(b);
    }
    if (lane == 0) sh.count[buf][part] = n;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
#pragma unroll
        for (int p = 0; p < kParts; ++p) total += sh.count[buf][p];
        sh.base[buf] = total ? atomicAdd(out.match.counter, (unsigned long long)total) : 0ull;
    }
    __syncthreads();
    if (!n) return;
    uint32_t before = 0;
    for (uint32_t p = 0; p < part; ++p) before += sh.count[buf][p];
    /* at most one match per row: positions stay below the probe rows, which
     * the capacity covers */
    const unsigned long long base = sh.base[buf] + before;
    if (base + n > out.match.capacity) return;
    const uint32_t at = (uint32_t)base;
    if (out.match.key_pages) { /* of the probe key's type */
        const PageRun<T> keys(out.match.key_pages, at);
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            T *to = keys.at((place[it / 4] >> (8 * (it % 4))) & 0xFFu);
            if ((m >> it) & 1u) __stcs(to, lk.key_of(code[it]));
        }
    }
    emit_packed(out, plan, w, n, at, row0);
    __syncwarp(); /* done with w before the next step packs */
}

/* The same over a table of repeated keys, of either kind. The matches of rows
 * with up to three are packed and written together, in three parts where they
 * outnumber the room; those of rows with more are listed 32 a step, whichever
 * rows they are of, and written whenever the room is full: all lanes then have
 * loads in flight however many rows the matches come from. Rows with kRunFrom
 * or more are only listed where there is a list (RunList). (In rounds of the
 * j-th matches and, from 33 on, row by row, the 24M matches of 300K x 3M rows,
 * eight a key, took 808 us, 685 so; the whole join, the hash table 1133.)
 * 64M x 4M rows over 3M keys, 58.6M matches: 877 us with one result column of
 * two written beside it (bound by the registers of its many paths: 64, some
 * spilled; 956 with the rounds, which spilled three times as much; a separate
 * function for the rare ones cost more in the common one, 1141; warps without
 * rows of more than three on a path of their own 1150). */
constexpr uint32_t kMultiRoom = 320; /* matches packed at once: 256 rows and a quarter more */
struct MultiMatches {
    uint32_t rid[kMultiRoom]; /* the keys first, then the build rows */
    uint8_t row[kMultiRoom];
};
struct MultiShared {
    MultiMatches matches[kParts];
    unsigned long long count[2][kParts];
    unsigned long long base[2];
};
template <typename T> struct MultiLookup {
    DirectLookup<T> d;
    const unsigned long long *entries;
    const uint32_t *rows;
    using Code = uint32_t;
    static constexpr bool kMask = false;
    static constexpr bool kStage = true; /* codes fit the packed matches: keys are written by full warps */
    CJ_DEV MultiLookup(const MultiTable &t)
        : d(nullptr, t.lo, t.span), entries(t.entries + (d.lo - t.lo)), rows(t.rows) {}
    CJ_DEV uint32_t code(T key, bool present, bool *in) const { return d.code(key, present, in); }
    CJ_DEV T key_of(uint32_t c) const { return d.key_of(c); }
    CJ_DEV void find(const uint32_t *c, uint32_t, uint32_t *low, uint32_t *cnt) const {
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            unsigned long long e = 0;
            if (c[it] < d.span) e = __ldg(entries + c[it]);
            low[it] = (uint32_t)e;
            cnt[it] = (uint32_t)(e >> 32);
        }
    }
};

/* Open addressing; its keys, which need not fit 32 bits, go to their places
 * straight from the lanes. */
template <typename T> struct OpenMultiLookup {
    TaggedTable t;
    const uint32_t *rows;
    unsigned long long lo, width;
    using Code = T;
    static constexpr bool kMask = true;
    static constexpr bool kStage = false;
    CJ_DEV OpenMultiLookup(const OpenMultiTable &m)
        : t{reinterpret_cast<const ulonglong2 *>(m.slots), reinterpret_cast<const unsigned long long *>(m.tags),
            m.nslots / 8},
          rows(m.rows), lo(m.lo), width(m.width) {}
    CJ_DEV T code(T key, bool present, bool *in) const {
        *in = present && (unsigned long long)(int64_t)key - lo <= width;
        return key;
    }
    CJ_DEV T key_of(T c) const { return c; }
    CJ_DEV void find(const T *c, uint32_t ok, uint32_t *low, uint32_t *cnt) const {
#pragma unroll
        for (int it = 0; it < kItems; ++it) low[it] = cnt[it] = 0;
        t.find(c, ok, [&](int it, unsigned long long y) {
            low[it] = (uint32_t)y;
            cnt[it] = (uint32_t)(y >> 32);
        });
    }
};

/* Lists a row's n matches as runs, for k_match_runs. */
CJ_DEV void list_runs(const RunList &l, int64_t key, uint32_t rows, uint32_t n, uint32_t at, uint32_t probe) {
    const uint32_t runs = (n + kRunRows - 1) / kRunRows;
    unsigned long long first = 0;
    if (lane_id() == 0) first = atomicAdd(l.count, (unsigned long long)runs);
    first = __shfl_sync(0xffffffffu, first, 0);
    for (uint32_t k = lane_id(); k < runs && first + k < l.capacity; k += 32) {
        const uint32_t q = k * kRunRows;
        l.runs[first + k] = {key, rows + q, min(kRunRows, n - q), at + q, probe};
    }
}

/* The lanes' items of one packing: item `it`'s matches go to places first(it)
 * on, `count(it)` of them (at most three); the packed total is returned. */
template <class C, class F> CJ_DEV uint32_t pack_few(C count, F put) {
    const uint32_t lt = lanemask_lt();
    uint32_t n = 0;
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const uint32_t c = count(it);
        const uint32_t b0 = __ballot_sync(0xffffffffu, c & 1u), b1 = __ballot_sync(0xffffffffu, c & 2u);
        const uint32_t i = n + __popc(b0 & lt) + 2 * __popc(b1 & lt);
        n += __popc(b0) + 2 * __popc(b1);
        if (c && i + c <= kMultiRoom) put(it, i, c);
    }
    return n;
}
template <typename T, class LK>
CJ_DEV void emit_keys(const LK &lk, const UniqueOut &out, const MultiMatches &w, uint32_t n, uint32_t at) {
    __syncwarp();
    const PageRun<T> keys(out.match.key_pages, at);
    for (uint32_t i = lane_id(); i < n; i += 32) __stcs(keys.at(i), lk.key_of(w.rid[i]));
    __syncwarp();
}

template <typename T, class LK>
CJ_DEV void probe_step(const LK &lk, const typename LK::Code *code, uint32_t ok, uint32_t row0, const UniqueOut &out,
                       const EmitPlan &plan, MultiShared &sh, uint32_t part, uint32_t buf) {
    const uint32_t lane = lane_id(), lt = lanemask_lt();
    MultiMatches &w = sh.matches[part];
    uint32_t low[kItems], cnt[kItems];
    lk.find(code, ok, low, cnt);
    unsigned long long many = 0; /* matches of rows with more than three */
#pragma unroll
    for (int it = 0; it < kItems; ++it)
        if (cnt[it] > 3) many += cnt[it];
    many = warp_sum(many);
    const auto few_of = [&](int it) { return cnt[it] <= 3 ? cnt[it] : 0u; };
    const auto stage = [&](int it, uint32_t i, uint32_t c) {
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j)
            if (j < c) {
                if constexpr (LK::kStage) w.rid[i + j] = code[it];
                w.row[i + j] = (uint8_t)(it * 32 + lane);
            }
    };
    const uint32_t few = pack_few(few_of, stage);
    const bool packed = few <= kMultiRoom;
    const unsigned long long total = few + many;
    if (lane == 0) sh.count[buf][part] = total;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long all = 0;
#pragma unroll
        for (int p = 0; p < kParts; ++p) all += sh.count[buf][p];
        sh.base[buf] = all ? atomicAdd(out.match.counter, all) : 0ull;
    }
    __syncthreads();
    if (!total) return;
    unsigned long long base = sh.base[buf];
    for (uint32_t p = 0; p < part; ++p) base += sh.count[buf][p];
    /* past the capacity nothing is written: the caller runs the probe again
     * with room for the whole count */
    if (base + total > out.match.capacity) return;
    uint32_t at = (uint32_t)base;
    const uint32_t passes = packed ? 1u : 3u;
    for (uint32_t h = 0; few && h < passes; ++h) {
        /* all of them, or those of three items (288 matches at most) */
        const auto part_of = [&](int it) { return packed || (uint32_t)it / 3 == h ? few_of(it) : 0u; };
        const uint32_t n = packed ? few : pack_few(part_of, stage);
        if constexpr (LK::kStage) {
            if (out.match.key_pages) emit_keys<T>(lk, out, w, n, at);
        }
        const PageRun<T> keys(out.match.key_pages, at);
        pack_few(part_of, [&](int it, uint32_t i, uint32_t c) {
            if constexpr (!LK::kStage) {
                if (out.match.key_pages)
                    for (uint32_t j = 0; j < c; ++j) __stcs(keys.at(i + j), lk.key_of(code[it]));
            }
            if (c == 1) {
                w.rid[i] = low[it];
            } else {
                const uint32_t *r = lk.rows + (low[it] - c);
                const uint32_t r0 = __ldg(r), r1 = __ldg(r + 1);
                if (c == 3) w.rid[i + 2] = __ldg(r + 2);
                w.rid[i] = r0;
                w.rid[i + 1] = r1;
            }
        });
        __syncwarp();
        emit_packed(out, plan, w, n, at, row0);
        __syncwarp(); /* done with w before it is packed again */
        at += n;
    }
    if (!many) return;
    uint32_t left = (uint32_t)many, fill = 0; /* below the capacity */
    for (int it = 0; it < kItems; ++it) {
        uint32_t c = 0, lo = 0; /* item `it`, without indexing registers */
        typename LK::Code cd = 0;
#pragma unroll
        for (int q = 0; q < kItems; ++q)
            if (q == it) {
                c = cnt[q];
                lo = low[q];
                cd = code[q];
            }
        if (c <= 3) c = 0;
        if (out.runs.runs) {
            for (uint32_t heavy = __ballot_sync(0xffffffffu, c >= kRunFrom); heavy; heavy &= heavy - 1) {
                const int src = __ffs(heavy) - 1;
                const uint32_t n = __shfl_sync(0xffffffffu, c, src);
                left -= n;
                list_runs(out.runs, (int64_t)lk.key_of(__shfl_sync(0xffffffffu, cd, src)),
                          __shfl_sync(0xffffffffu, lo, src) - n, n, at + fill + left, row0 + it * 32 + src);
            }
            if (c >= kRunFrom) c = 0;
        }
        const uint32_t incl = warp_inclusive_scan(c), all = __shfl_sync(0xffffffffu, incl, 31);
        const uint32_t place = lo - incl; /* of match p of the item's: place + p */
        for (uint32_t p0 = 0; p0 < all || (fill && !left);) { /* the last matches may have been listed before */
            const uint32_t n = min(kMultiRoom - fill, all - p0);
            const PageRun<T> keys(out.match.key_pages, at);
            for (uint32_t i = lane; i < ((n + 31) & ~31u); i += 32) {
                const uint32_t p = p0 + i;
                uint32_t src = 0; /* the first lane whose matches end above p */
#pragma unroll
                for (uint32_t step = 16; step; step >>= 1)
                    if (__shfl_sync(0xffffffffu, incl, src + step - 1) <= p) src += step;
                const uint32_t from = __shfl_sync(0xffffffffu, place, src);
                const typename LK::Code kc = __shfl_sync(0xffffffffu, cd, src);
                if (i >= n) continue;
                w.rid[fill + i] = from + p; /* the place of the build row, until the room is full */
                w.row[fill + i] = (uint8_t)(it * 32 + src);
                if (out.match.key_pages) __stcs(keys.at(fill + i), lk.key_of(kc));
            }
            fill += n;
            left -= n;
            p0 += n;
            if (left && fill < kMultiRoom) continue;
            __syncwarp();
            for (uint32_t i0 = lane; i0 < fill; i0 += 32 * kEmit) {
                uint32_t r[kEmit];
#pragma unroll
                for (int k = 0; k < kEmit; ++k)
                    if (i0 + k * 32 < fill) r[k] = __ldg(lk.rows + w.rid[i0 + k * 32]);
#pragma unroll
                for (int k = 0; k < kEmit; ++k)
                    if (i0 + k * 32 < fill) w.rid[i0 + k * 32] = r[k];
            }
            __syncwarp();
            emit_packed(out, plan, w, fill, at, row0);
            __syncwarp();
            at += fill;
            fill = 0;
        }
    }
}

/* Asks L2 for a warp's part of a page that it reads next: its keys then cost
 * an L2 round trip, not one to HBM. */
template <typename T> CJ_DEV void prefetch_part(const uint8_t *pg, uint32_t part) {
    constexpr uint32_t kLines = kPageSize / 128 / kPageParts<T>;
    if (lane_id() < kLines) asm volatile("prefetch.global.L2 [%0];" ::"l"(pg + (part * kLines + lane_id()) * 128));
}

/* One key of a relation row, typed. */
template <typename T> CJ_DEV bool row_key(const ColView &c, uint32_t i, T *key) {
    int64_t k;
    if (!load_key_stream(c, i, &k)) return false;
    *key = (T)k;
    return true;
}

/* The items of a step that a block takes: all, or every `of`-th where the
 * probe rows are too few to fill the chip and each may have many matches. */
struct Share {
    uint32_t which = 0, of = 1; /* a power of two up to kItems */
    CJ_DEV uint64_t block() const { return blockIdx.x / of; }
    CJ_DEV uint64_t blocks() const { return gridDim.x / of; }
    template <typename T, class LK> CJ_DEV void keep(const LK &lk, typename LK::Code *code, uint32_t *ok) const {
        if (of == 1) return;
#pragma unroll
        for (int it = 0; it < kItems; ++it) {
            bool in;
            if ((it & (of - 1)) == which) continue;
            code[it] = lk.code(T(0), false, &in);
            *ok &= ~(1u << it);
        }
    }
};

/* A step over relation rows t0 ... t0 + 2047. Block-wide. */
template <typename T, class LK, class SH>
CJ_DEV void probe_rows(const ColView &col, uint32_t n, uint64_t t0, const LK &lk, const UniqueOut &out,
                       const EmitPlan &plan, SH &sh, uint32_t part, uint32_t buf, const Share &share) {
    typename LK::Code code[kItems] = {};
    uint32_t ok = 0;
    const uint64_t r0 = t0 + part * kWarpRows;
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const uint64_t i = r0 + it * 32 + lane_id();
        T key = T(0);
        bool in;
        const bool present = i < n && row_key<T>(col, (uint32_t)i, &key);
        code[it] = lk.code(key, present, &in);
        if (LK::kMask && in) ok |= 1u << it;
    }
    share.keep<T>(lk, code, &ok);
    probe_step<T>(lk, code, ok, (uint32_t)r0, out, plan, sh, part, buf);
}

/* The key column's pages, one a step (INT32) or two (INT64). Block-wide. */
template <typename T, class LK, class SH>
CJ_DEV void probe_pages(const ProbeKey &k, uint32_t n, const LK &lk, const UniqueOut &out, const EmitPlan &plan, SH &sh,
                        uint32_t part, const Share &share) {
    uint32_t buf = 0;
    if constexpr (kStepPages<T> == 1) {
        const uint32_t stride = share.blocks();
        for (uint64_t p = share.block(); p < k.num_pages; p += stride) {
            const uint8_t *pg = k.col.pages + p * kPageSize;
            const uint32_t head = __ldg(reinterpret_cast<const uint32_t *>(pg));
            const uint32_t nr = head & 0xFFFFu, nv = head >> 16;
            const uint64_t rs = page_first_row(k.base, k.loc, p);
            if (p + stride < k.num_pages) prefetch_part<T>(pg + (uint64_t)stride * kPageSize, part);
            if (nv > nr || sizeof(T) + sizeof(T) * nv + (nr + 7) / 8 > kPageSize)
                continue; /* the index has raised the error */
            if (rs + nr > n) {
                if (threadIdx.x == 0) atomicOr(k.err, DEV_ERR_ROW_COUNT);
                continue;
            }
            uint32_t before = 0;
            for (uint32_t s0 = 0; s0 < nr; s0 += kPageRows<T>) {
                typename LK::Code code[kItems] = {};
                uint32_t ok = page_keys<T>(pg, nr, nv, s0, part, &before, lk, code, k.err);
                share.keep<T>(lk, code, &ok);
                probe_step<T>(lk, code, ok, (uint32_t)rs + s0 + part * kWarpRows, out, plan, sh, part, buf);
                buf ^= 1u;
            }
        }
    } else {
        const uint64_t stride = share.blocks() * 2;
        const uint32_t ppart = part % kPageParts<T>;
        for (uint64_t p0 = share.block() * 2; p0 < k.num_pages; p0 += stride) {
            const uint64_t p = p0 + part / kPageParts<T>, q = p ^ 1; /* p0 is even */
            const uint8_t *pg = k.col.pages + p * kPageSize;
            uint32_t nr = 0, nv = 0, other = 0;
            uint64_t rs = 0;
            if (q < k.num_pages) other = __ldg(reinterpret_cast<const uint32_t *>(k.col.pages + q * kPageSize)) & 0xFFFFu;
            if (p < k.num_pages) {
                const uint32_t head = __ldg(reinterpret_cast<const uint32_t *>(pg));
                nr = head & 0xFFFFu;
                nv = head >> 16;
                rs = page_first_row(k.base, k.loc, p);
            }
            const uint32_t turns = max(nr, other); /* as many as the page with more rows takes */
            if (p + stride < k.num_pages) prefetch_part<T>(pg + stride * kPageSize, ppart);
            if (nv > nr || sizeof(T) + sizeof(T) * nv + (nr + 7) / 8 > kPageSize) {
                nr = 0; /* the index has raised the error */
            } else if (rs + nr > n) {
                if (lane_id() == 0) atomicOr(k.err, DEV_ERR_ROW_COUNT);
                nr = 0;
            }
            uint32_t before = 0;
            for (uint32_t s0 = 0; s0 < turns; s0 += kPageRows<T>) {
                typename LK::Code code[kItems] = {};
                uint32_t ok = 0;
                if (s0 < nr) {
                    ok = page_keys<T>(pg, nr, nv, s0, ppart, &before, lk, code, k.err);
                } else {
#pragma unroll
                    for (int it = 0; it < kItems; ++it) {
                        bool in;
                        code[it] = lk.code(T(0), false, &in);
                    }
                }
                share.keep<T>(lk, code, &ok);
                probe_step<T>(lk, code, ok, (uint32_t)rs + s0 + ppart * kWarpRows, out, plan, sh, part, buf);
                buf ^= 1u;
            }
        }
    }
}

template <bool kPages, typename T, class LK, class SH>
CJ_DEV void probe_all(const ProbeKey &k, uint32_t n, const LK &lk, const UniqueOut &out, SH &sh,
                      const Share &share = Share()) {
    const EmitPlan plan(out, LK::kMask);
    const uint32_t part = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0); /* warp-uniform */
    if constexpr (kPages) {
        probe_pages<T>(k, n, lk, out, plan, sh, part, share);
    } else {
        const ColView col = resolve_view(k.col);
        uint32_t buf = 0;
        for (uint64_t t0 = share.block() * kTileRows; t0 < n; t0 += share.blocks() * kTileRows) {
            probe_rows<T>(col, n, t0, lk, out, plan, sh, part, buf, share);
            buf ^= 1u;
        }
    }
}

template <bool kPages, typename T>
__global__ void __launch_bounds__(kProbeThreads, kProbeBlocks)
    k_probe_unique(const __grid_constant__ ProbeKey k, uint32_t n, const __grid_constant__ UniqueTable t,
                   const __grid_constant__ UniqueOut out) {
    __shared__ StepShared sh;
    const unsigned long long refused = t.params[kTableRefused];
    if (t.params[kTableDup]) return;
    if (refused == 0) {
        const DirectLookup<T> lk(reinterpret_cast<const uint32_t *>(t.slots), (int64_t)t.params[kTableLo],
                                 (uint32_t)t.params[kTableSpan]);
        probe_all<kPages, T>(k, n, lk, out, sh);
    }
    if (refused == kTableSpread && t.open_slots) probe_all<kPages, T>(k, n, OpenLookup<T>(t), out, sh);
}

/* A table that may have wide slots: a kernel of its own, so that their
 * registers are not the other's. */
template <bool kPages, typename T>
__global__ void __launch_bounds__(kProbeThreads, kWideBlocks)
    k_probe_wide(const __grid_constant__ ProbeKey k, uint32_t n, const __grid_constant__ UniqueTable t,
                 const __grid_constant__ UniqueOut out) {
    __shared__ StepShared sh;
    const unsigned long long refused = t.params[kTableRefused];
    if (t.params[kTableDup]) return;
    if (refused == 0) {
        const DirectLookup<T> lk(reinterpret_cast<const uint32_t *>(t.slots), (int64_t)t.params[kTableLo],
                                 (uint32_t)t.params[kTableSpan]);
        probe_all<kPages, T>(k, n, lk, out, sh);
    }
    if (refused == kTableSpread && t.open_slots) probe_all<kPages, T>(k, n, WideLookup<T>(t), out, sh);
}

/* The matches that a probe of repeated keys listed as runs (list_runs), a
 * warp a run: the build rows come from the table's `rows` side by side, the
 * probe row is one for all of them. 60M matches of 400 a row, 5M x 300K INT64
 * rows of which 3 % match: 1482 us with the probe writing them from its room,
 * whose listing takes seven warp instructions a match, 870 so. A kernel of its
 * own, because these loops beside the probe's spill its registers (64M x 4M
 * rows, at most two matches a row: 1166 us with them, 1007 without). */
template <typename T>
CJ_DEV void emit_run_column(const EmitColumn &c, bool direct, const uint32_t *rows, const MatchRun &run) {
    const PageRun<T> out(c.pages, run.at); /* of one page or two: kRunRows fit one */
    const auto value = [&](uint32_t r) {
        if (c.col.rid_b) r = __ldg(c.col.rid_b + r);
        return direct ? page_value<T>(c.col.pages, r) : __ldg(reinterpret_cast<const T *>(c.col.values) + r);
    };
    if (!c.from_build) {
        const T v = value(run.probe);
        for (uint32_t i = lane_id(); i < run.count; i += 32) __stcs(out.at(i), v);
        return;
    }
    constexpr int kFlight = 4;
    for (uint32_t i0 = lane_id(); i0 < run.count; i0 += 32 * kFlight) {
        T v[kFlight];
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
            if (i0 + j * 32 < run.count) v[j] = value(__ldg(rows + run.rows + i0 + j * 32));
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
            if (i0 + j * 32 < run.count) __stcs(out.at(i0 + j * 32), v[j]);
    }
}
template <typename T>
__global__ void __launch_bounds__(kProbeThreads) k_match_runs(const uint32_t *rows, const __grid_constant__ UniqueOut out) {
    static_assert(kRunRows <= PageRun<T>::R && kRunRows <= PageRun<long long>::R, "a run ends on the next page at most");
    const uint64_t n = min((uint64_t)*out.runs.count, out.runs.capacity);
    if (blockIdx.x * (uint64_t)kParts >= n) return;
    const EmitPlan plan(out, false);
    for (uint64_t k = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32; k < n; k += (uint64_t)gridDim.x * blockDim.x / 32) {
        const MatchRun run = out.runs.runs[k];
        const uint32_t lane = lane_id();
        if (out.match.key_pages) {
            const PageRun<T> keys(out.match.key_pages, run.at);
            for (uint32_t i = lane; i < run.count; i += 32) __stcs(keys.at(i), (T)run.key);
        }
        for (uint32_t i = lane; plan.want_b && i < run.count; i += 32)
            __stcs(out.match.build_rids + run.at + i, __ldg(rows + run.rows + i));
        for (uint32_t i = lane; plan.want_p && i < run.count; i += 32)
            __stcs(out.match.probe_rids + run.at + i, run.probe);
        for (int c = 0; c < out.n; ++c) {
            if (!((plan.active >> c) & 1u)) continue;
            const EmitColumn &e = out.cols[c];
            if (e.col.type == CJ_INT32) emit_run_column<int32_t>(e, (plan.direct >> c) & 1u, rows, run);
            else emit_run_column<long long>(e, (plan.direct >> c) & 1u, rows, run);
        }
    }
}

template <bool kPages, typename T>
__global__ void __launch_bounds__(kProbeThreads, kMultiBlocks)
    k_probe_multi(const __grid_constant__ ProbeKey k, uint32_t n, const __grid_constant__ MultiTable t,
                  const __grid_constant__ UniqueOut out, uint32_t shares) {
    __shared__ MultiShared sh;
    probe_all<kPages, T>(k, n, MultiLookup<T>(t), out, sh, Share{blockIdx.x & (shares - 1), shares});
}

template <bool kPages, typename T>
__global__ void __launch_bounds__(kProbeThreads, kOpenMultiBlocks)
    k_probe_open_multi(const __grid_constant__ ProbeKey k, uint32_t n, const __grid_constant__ OpenMultiTable t,
                       const __grid_constant__ UniqueOut out, uint32_t shares) {
    __shared__ MultiShared sh;
    probe_all<kPages, T>(k, n, OpenMultiLookup<T>(t), out, sh, Share{blockIdx.x & (shares - 1), shares});
}

/* Steps of a probe's CTAs. */
uint64_t probe_tiles(const ProbeKey &k, uint32_t n) {
    if (!k.base) return ((uint64_t)n + kTileRows - 1) / kTileRows;
    return k.col.type == CJ_INT32 ? k.num_pages : (k.num_pages + 1) / 2;
}

/* Blocks that share a step's rows of a probe with several matches a row: as
 * many as the chip holds beside each other and a second wave, up to a block
 * per item. A warp writes the matches of its 256 rows one room after the
 * other, which few probe rows with many matches each leave to a few warps:
 * 50K rows of 40 matches 734 us with a block per step, 290 with eight (the
 * whole join), 300K rows of 200 matches 2938 and, with four, 1360. */
uint32_t shares_of(uint64_t tiles, uint64_t wave) {
    uint32_t s = 1;
    while (s < (uint32_t)kItems && tiles * s <= wave) s *= 2;
    return s;
}

/* Random loads in flight are held in L1: as little of it as possible goes to
 * shared memory (default split 628 us, this one 605, before later gains). Once per kernel and
 * device. */
template <class K> void prefer_l1(K kernel) {
    constexpr int kDevices = 64;
    static std::atomic<const void *> done[kDevices][16];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kDevices) {
        cudaGetLastError();
        return;
    }
    for (auto &slot : done[dev]) {
        const void *seen = slot.load(std::memory_order_acquire);
        if (seen == reinterpret_cast<const void *>(kernel)) return;
        if (seen) continue;
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 25);
        slot.store(reinterpret_cast<const void *>(kernel), std::memory_order_release);
        return;
    }
}

/* After a probe that lists runs: their matches. */
cudaError_t launch_runs(const Launch &L, int32_t key_type, const uint32_t *rows, const UniqueOut &out) {
    if (!out.runs.runs || !out.runs.capacity) return cudaSuccess;
    const unsigned g = (unsigned)std::min<uint64_t>((out.runs.capacity + kParts - 1) / kParts, (uint64_t)L.num_sms * 4);
    const auto kernel = key_type == CJ_INT32 ? k_match_runs<int32_t> : k_match_runs<long long>;
    prefer_l1(kernel);
    kernel<<<g, kProbeThreads, 0, L.stream>>>(rows, out);
    count_launches(1);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_unique_build(const Launch &L, const ColView &key, uint32_t n, const UniqueTable &t) {
    if (n == 0) return cudaSuccess;
    if (t.open_slots && (t.open_slots < 2ull * n || t.open_slots % 16)) return cudaErrorInvalidValue; /* half empty */
    if (reinterpret_cast<uintptr_t>(t.slots) % 16) return cudaErrorInvalidValue;
    if (n <= kSmallRows) {
        k_unique_small<<<1, kSmallThreads, 0, L.stream>>>(key, n, t);
        count_launches(1);
        return cudaGetLastError();
    }
    const uint64_t wave = (uint64_t)L.num_sms * 8;
    const uint64_t rows_per_block = kUniqueThreads * kUniqueRows;
    const unsigned g = (unsigned)std::min<uint64_t>((n + rows_per_block - 1) / rows_per_block, wave);
    k_unique_range<<<g, kUniqueThreads, 0, L.stream>>>(key, n, t);
    const uint64_t most = unique_table_bytes(t) / 16 + 1;
    k_unique_fill<<<(unsigned)std::min<uint64_t>((most + 255) / 256, wave), kUniqueThreads, 0, L.stream>>>(t);
    k_unique_insert<<<g, kUniqueThreads, 0, L.stream>>>(key, n, t);
    count_launches(3);
    return cudaGetLastError();
}

cudaError_t launch_probe_unique(const Launch &L, const ProbeKey &k, uint32_t n, const UniqueTable &t,
                                const UniqueOut &out) {
    if (n == 0) return cudaSuccess;
    const bool pages = k.base != nullptr;
    const uint64_t tiles = probe_tiles(k, n);
    const unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, (uint64_t)L.num_sms * (t.wide ? kWideBlocks : kProbeBlocks)));
    const auto narrow = k.col.type == CJ_INT32 ? (pages ? k_probe_unique<true, int32_t> : k_probe_unique<false, int32_t>)
                                               : (pages ? k_probe_unique<true, long long> : k_probe_unique<false, long long>);
    const auto wide = k.col.type == CJ_INT32 ? (pages ? k_probe_wide<true, int32_t> : k_probe_wide<false, int32_t>)
                                             : (pages ? k_probe_wide<true, long long> : k_probe_wide<false, long long>);
    const auto kernel = t.wide ? wide : narrow;
    prefer_l1(kernel);
    kernel<<<g, kProbeThreads, 0, L.stream>>>(k, n, t, out);
    count_launches(1);
    return cudaGetLastError();
}

UniqueGrid place_unique(const Launch &L, UniqueBuildTask *tasks, size_t n) {
    UniqueGrid g;
    const uint64_t wave = (uint64_t)L.num_sms * 8, rows = kUniqueThreads * kUniqueRows;
    for (size_t k = 0; k < n; ++k) {
        UniqueBuildTask &t = tasks[k];
        const uint64_t most = unique_table_bytes(t.table) / 16 + 1;
        t.key_blocks = (uint32_t)std::min<uint64_t>((t.n + rows - 1) / rows, wave);
        t.key_base = g.key;
        t.fill_blocks = (uint32_t)std::min<uint64_t>((most + kUniqueThreads * 8 - 1) / (kUniqueThreads * 8), wave);
        t.fill_base = g.fill;
        g.key += t.key_blocks;
        g.fill += t.fill_blocks;
    }
    return g;
}

cudaError_t launch_unique_build_grouped(const Launch &L, const UniqueBuildTask *tasks_dev, uint32_t n,
                                        const UniqueGrid &g) {
    if (!n) return cudaSuccess;
    k_unique_range_grouped<<<g.key, kUniqueThreads, 0, L.stream>>>(tasks_dev, n);
    k_unique_fill_grouped<<<g.fill, kUniqueThreads, 0, L.stream>>>(tasks_dev, n);
    k_unique_insert_grouped<<<g.key, kUniqueThreads, 0, L.stream>>>(tasks_dev, n);
    count_launches(3);
    return cudaGetLastError();
}

cudaError_t launch_multi_build(const Launch &L, const ColView &key, uint32_t n, const MultiTable &t) {
    if (!n || !t.span) return cudaErrorInvalidValue;
    const uint64_t wave = (uint64_t)L.num_sms * 8;
    cudaError_t e = cudaMemsetAsync(t.entries, 0, ((uint64_t)t.span + 1) * 8, L.stream);
    if (e != cudaSuccess) return e;
    const uint64_t rows_per_block = kUniqueThreads * kUniqueRows, values_per_block = kUniqueThreads * kPlaceItems;
    const unsigned g = (unsigned)std::min<uint64_t>((n + rows_per_block - 1) / rows_per_block, wave);
    k_multi_count<<<g, kUniqueThreads, 0, L.stream>>>(key, n, t);
    k_multi_place<<<(unsigned)std::min<uint64_t>((t.span + values_per_block - 1) / values_per_block, wave),
                    kUniqueThreads, 0, L.stream>>>(t);
    k_multi_scatter<<<g, kUniqueThreads, 0, L.stream>>>(key, n, t);
    count_launches(3);
    return cudaGetLastError();
}

cudaError_t launch_probe_multi(const Launch &L, const ProbeKey &k, uint32_t n, const MultiTable &t,
                               const UniqueOut &out) {
    if (n == 0) return cudaSuccess;
    const bool pages = k.base != nullptr;
    const uint64_t tiles = probe_tiles(k, n);
    const uint64_t wave = (uint64_t)L.num_sms * kMultiBlocks;
    const uint32_t shares = shares_of(std::max<uint64_t>(tiles, 1), wave);
    const unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, wave)) * shares;
    const auto kernel = k.col.type == CJ_INT32 ? (pages ? k_probe_multi<true, int32_t> : k_probe_multi<false, int32_t>)
                                               : (pages ? k_probe_multi<true, long long> : k_probe_multi<false, long long>);
    prefer_l1(kernel);
    kernel<<<g, kProbeThreads, 0, L.stream>>>(k, n, t, out, shares);
    count_launches(1);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? launch_runs(L, k.col.type, t.rows, out) : e;
}

cudaError_t launch_key_sample(const Launch &L, const ColView &key, uint32_t n, uint32_t *bits, unsigned long long *found,
                              uint32_t *shift) {
    *shift = 0;
    while ((n >> *shift) > kSampleRows) ++*shift; /* at most 15: clear of the bit's place */
    const uint64_t rows_per_block = kUniqueThreads * kUniqueRows;
    const unsigned g = (unsigned)std::min<uint64_t>((n + rows_per_block - 1) / rows_per_block, (uint64_t)L.num_sms * 8);
    k_key_sample<<<g, kUniqueThreads, 0, L.stream>>>(key, n, *shift, bits, found);
    count_launches(1);
    return cudaGetLastError();
}

uint64_t sampled_keys(unsigned long long found, uint32_t shift) {
    const double m = kSampleBits, b = std::min<double>((double)found, m - 1);
    return (uint64_t)std::max(1.0, -m * std::log1p(-b / m) * (double)(1ull << shift));
}

cudaError_t launch_open_multi_build(const Launch &L, const ColView &key, uint32_t n, const OpenMultiTable &t) {
    if (!n || t.nslots < 2ull * n || t.nslots % 8 || reinterpret_cast<uintptr_t>(t.slots) % 16 ||
        reinterpret_cast<uintptr_t>(t.tags) % 8)
        return cudaErrorInvalidValue;
    const uint64_t wave = (uint64_t)L.num_sms * 8;
    const uint64_t rows_per_block = kUniqueThreads * kUniqueRows, slots_per_block = kUniqueThreads * kPlaceItems;
    const unsigned g = (unsigned)std::min<uint64_t>((n + rows_per_block - 1) / rows_per_block, wave);
    const unsigned gs = (unsigned)std::min<uint64_t>((t.nslots + slots_per_block - 1) / slots_per_block, wave);
    k_open_multi_fill<<<gs, kUniqueThreads, 0, L.stream>>>(t);
    k_open_multi_claim<<<g, kUniqueThreads, 0, L.stream>>>(key, n, t);
    k_open_multi_place<<<gs, kUniqueThreads, 0, L.stream>>>(t);
    k_open_multi_scatter<<<g, kUniqueThreads, 0, L.stream>>>(n, t);
    count_launches(4);
    return cudaGetLastError();
}

cudaError_t launch_probe_open_multi(const Launch &L, const ProbeKey &k, uint32_t n, const OpenMultiTable &t,
                                    const UniqueOut &out) {
    if (n == 0) return cudaSuccess;
    const bool pages = k.base != nullptr;
    const uint64_t tiles = probe_tiles(k, n);
    const uint64_t wave = (uint64_t)L.num_sms * kOpenMultiBlocks;
    const uint32_t shares = shares_of(std::max<uint64_t>(tiles, 1), wave);
    const unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(tiles, wave)) * shares;
    const auto kernel = k.col.type == CJ_INT32
                            ? (pages ? k_probe_open_multi<true, int32_t> : k_probe_open_multi<false, int32_t>)
                            : (pages ? k_probe_open_multi<true, long long> : k_probe_open_multi<false, long long>);
    prefer_l1(kernel);
    kernel<<<g, kProbeThreads, 0, L.stream>>>(k, n, t, out, shares);
    count_launches(1);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? launch_runs(L, k.col.type, t.rows, out) : e;
}

} // namespace cj
