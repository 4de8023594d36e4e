/*
 * k_materialize.cu — late materialisation: gather matched rows back into
 * 8 KiB result pages.
 *
 * The reference materialises the root join through per-thread page
 * builders (include/materialization/materialize.h:85-321,
 * page_builders.h:92-391) and non-root joins into 4-byte value_t columns
 * (construct_intermediate.h:121-220). Here non-root joins only gather u32
 * row-id vectors (k_gather_u32); values are read once, by the root's page
 * writers, through up to two row-id indirections.
 *
 * Fixed-width pages (k_write_pages): output page p holds rows
 * [p*R, p*R+R) with R = 1984 (INT32) or 1007 (INT64 / FP64), the fill of
 * ColumnInserter<T> (plan.h:241-250), so every page fits whatever the NULL
 * pattern. One CTA writes one page: all of the page's loads issued at
 * once; a page without NULLs is stored straight from registers (values in
 * row order, header, zero gap, all-ones bitmap); a page with NULLs is built
 * in shared memory (values compacted by one ballot/scan over the validity
 * bits, bitmap at the page end, gap zeroed) and written with 16-byte
 * streaming stores.
 *
 * VARCHAR pages (k_varchar_plan / k_varchar_write): rows are cut into tiles;
 * within a tile pages are packed greedily in row order like
 * ColumnInserter<std::string> (plan.h:340-369): a page takes rows while
 * 4 + 2*n_values + chars + ceil(n_rows/8) <= 8192. A string longer than 8185
 * bytes arrives as a chain of long-string pages and is copied verbatim, as
 * VarcharPageBuilder::copy_long_string_pages does (page_builders.h:345-362).
 * Pass 1 cuts every tile into segments (a page, or a long string's chain) and
 * places the tiles' pages, pass 2 writes a segment per CTA.
 */
#include <algorithm>

#include "cj_device.cuh"

namespace cj {
namespace {

constexpr int kMatThreads = 256;

CJ_DEV uint32_t rows_per_page_dev(int32_t type) { return type == CJ_INT32 ? kRowsPerPageInt32 : kRowsPerPage8B; }

/* out[i] = src[idx[i]] for i = first, first + stride, ...: four rows a thread
 * in flight (one at a time left each waiting for two round trips a row). */
CJ_DEV void gather_rows(const uint32_t *__restrict__ src, const uint32_t *__restrict__ idx, uint32_t *__restrict__ out,
                        uint64_t first, uint64_t n, uint64_t stride) {
    constexpr int kRows = 4;
    for (uint64_t i0 = first; i0 < n; i0 += stride * kRows) {
        uint32_t v[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k)
            if (i0 + k * stride < n) v[k] = __ldcs(idx + i0 + k * stride);
#pragma unroll
        for (int k = 0; k < kRows; ++k)
            if (i0 + k * stride < n) v[k] = __ldg(src + v[k]);
#pragma unroll
        for (int k = 0; k < kRows; ++k)
            if (i0 + k * stride < n) out[i0 + k * stride] = v[k];
    }
}

__global__ void k_gather_u32(const uint32_t *__restrict__ src, const uint32_t *__restrict__ idx,
                             uint64_t n, uint32_t *__restrict__ out) {
    gather_rows(src, idx, out, (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, n, (uint64_t)gridDim.x * blockDim.x);
}

constexpr int kMatMinBlocks = 8; /* page writers: 8 x 256 threads per SM */

struct PageSmem {
    uint4 page[kPageSize / 16]; /* zero between pages: copy-out clears it */
    uint32_t cnt[64];           /* non-NULL rows per (slab, warp), then offsets */
    uint32_t total;
};

/* Builds output page `pg` (rows [pg*R, pg*R+R)) of a fixed-width column in
 * shared memory and stores it. Block-wide; sm.page must be zero on entry and
 * is zero again on return.
 *
 * Thread t takes rows t, t+256, ... of the page (kSlabs of them) and issues
 * all their loads (row ids, then validity words and values) before using
 * any, so a page costs one dependent round trip, not one per 256 rows. One
 * scan over the (slab, warp) counts then places the non-NULL values. */
template <typename T>
CJ_DEV void write_fixed_page(const ColView &col, uint64_t rows, uint32_t R, uint64_t pg, uint8_t *__restrict__ out,
                             PageSmem &sm) {
    constexpr uint32_t DB = sizeof(T) == 4 ? 4u : 8u;
    constexpr int kSlabs = (int)(((sizeof(T) == 4 ? kRowsPerPageInt32 : kRowsPerPage8B) + kMatThreads - 1) / kMatThreads);
    constexpr int kWarps = kMatThreads / 32;
    static_assert(kSlabs * kWarps <= 64, "cnt holds 64 (slab, warp) counts");
    uint8_t *sp = reinterpret_cast<uint8_t *>(sm.page);
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    const uint64_t r0 = pg * R;
    const uint32_t nr = (uint32_t)min((uint64_t)R, rows - r0);


    uint32_t br[kSlabs];
#pragma unroll
    for (int k = 0; k < kSlabs; ++k) {
        const uint32_t r = k * kMatThreads + threadIdx.x;
        br[k] = 0xffffffffu;
        if (r < nr) br[k] = col.rid_a ? __ldcs(col.rid_a + r0 + r) : (uint32_t)(r0 + r);
    }
    if (col.rid_b) {
#pragma unroll
        for (int k = 0; k < kSlabs; ++k)
            if (br[k] != 0xffffffffu) br[k] = __ldg(col.rid_b + br[k]);
    }
    T val[kSlabs];
    uint32_t vm = 0; /* bit k: row of slab k is non-NULL */
    /* a column without NULLs needs no validity loads (one random load per
     * row instead of two when the row ids are random); a direct column is
     * read from its pages */
    const bool all_valid = col_all_valid(col);
    const bool direct = col_direct(col);
#pragma unroll
    for (int k = 0; k < kSlabs; ++k) {
        val[k] = T(0);
        if (br[k] != 0xffffffffu) {
            const bool v = all_valid || valid_bit(col.valid, br[k]);
            val[k] = direct ? page_value<T>(col.pages, br[k]) : __ldg(reinterpret_cast<const T *>(col.values) + br[k]);
            if (v && !(sizeof(T) == 4 && col.null_sentinel && (int32_t)val[k] == INT32_MIN)) vm |= 1u << k;
        }
    }

    const uint32_t bm_bytes = (nr + 7) / 8;

    /* No NULL on this page (always, for a column without NULLs): a value's
     * place is its row, so the page is stored straight from registers, with
     * no compaction, no shared memory and no barrier. Same bytes as below:
     * header, values, zero gap, bitmap of nr ones. */
    uint32_t live = 0;
#pragma unroll
    for (int k = 0; k < kSlabs; ++k)
        if (k * kMatThreads + threadIdx.x < nr) live |= 1u << k;
    const bool null_free_col = all_valid && !(sizeof(T) == 4 && col.null_sentinel);
    if (null_free_col || !__syncthreads_or(vm != live)) {
        uint8_t *dst = out + pg * kPageSize;
        T *dv = reinterpret_cast<T *>(dst + DB);
#pragma unroll
        for (int k = 0; k < kSlabs; ++k) {
            const uint32_t r = k * kMatThreads + threadIdx.x;
            if (r < nr) __stcs(dv + r, val[k]);
        }
        if (threadIdx.x == 0) {
            if (DB == 8) __stcs(reinterpret_cast<unsigned long long *>(dst), (unsigned long long)nr * 0x10001ull);
            else __stcs(reinterpret_cast<unsigned int *>(dst), nr * 0x10001u);
        }
        const uint32_t bm0 = kPageSize - bm_bytes;
        for (uint32_t b = DB + nr * (uint32_t)sizeof(T) + threadIdx.x; b < kPageSize; b += blockDim.x) {
            uint8_t v = 0;
            if (b >= bm0) {
                const uint32_t i = b - bm0;
                v = (i + 1) * 8 <= nr ? 0xFFu : (uint8_t)((1u << (nr - i * 8)) - 1u);
            }
            dst[b] = v;
        }
        return;
    }

    uint8_t *bm = sp + kPageSize - bm_bytes;
#pragma unroll
    for (int k = 0; k < kSlabs; ++k) {
        const uint32_t ball = __ballot_sync(0xffffffffu, (vm >> k) & 1u);
        if (lane == 0) sm.cnt[k * kWarps + warp] = __popc(ball);
        if (lane < 4) {
            const uint32_t byte = (k * kMatThreads + warp * 32) / 8 + lane;
            if (byte < bm_bytes) bm[byte] = (uint8_t)(ball >> (8 * lane));
        }
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t i0 = 2 * lane, i1 = 2 * lane + 1, n = kSlabs * kWarps;
        const uint32_t a = i0 < n ? sm.cnt[i0] : 0u, b = i1 < n ? sm.cnt[i1] : 0u;
        const uint32_t incl = warp_inclusive_scan(a + b);
        if (i0 < n) sm.cnt[i0] = incl - a - b;
        if (i1 < n) sm.cnt[i1] = incl - b;
        if (lane == 31) sm.total = incl;
    }
    __syncthreads();
    T *vals = reinterpret_cast<T *>(sp + DB);
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int k = 0; k < kSlabs; ++k) {
        const uint32_t ball = __ballot_sync(0xffffffffu, (vm >> k) & 1u);
        if ((vm >> k) & 1u) vals[sm.cnt[k * kWarps + warp] + __popc(ball & lt)] = val[k];
    }
    if (threadIdx.x == 0) {
        reinterpret_cast<uint16_t *>(sp)[0] = (uint16_t)nr;
        reinterpret_cast<uint16_t *>(sp)[1] = (uint16_t)sm.total;
    }
    __syncthreads();
    uint4 *dst = reinterpret_cast<uint4 *>(out + pg * kPageSize);
    const uint4 zero = make_uint4(0, 0, 0, 0);
    for (uint32_t k = threadIdx.x; k < kPageSize / 16; k += blockDim.x) {
        __stcs(dst + k, sm.page[k]);
        sm.page[k] = zero;
    }
    __syncthreads();
}

CJ_DEV void zero_page(PageSmem &sm) {
    for (uint32_t k = threadIdx.x; k < kPageSize / 16; k += blockDim.x) sm.page[k] = make_uint4(0, 0, 0, 0);
    __syncthreads();
}

/* Rows to write: `rows`, or, when `rows_dev` is set, the count it holds
 * (at most `rows`, the capacity the pages were sized for). */
CJ_DEV uint64_t live_rows(uint64_t rows, const unsigned long long *rows_dev) {
    if (!rows_dev) return rows;
    const uint64_t n = *rows_dev;
    return n < rows ? n : rows;
}

/* Finishes a page whose values are in place (a NULL-free column written by
 * the probe): header, zero gap after the values, bitmap of nr ones. One warp
 * per page, whole words (byte by byte by a block per page: 54 us for the
 * 110,000 pages of a 43.9M-row result). */
template <typename T> CJ_DEV void finish_dense_page(uint8_t *__restrict__ pages, uint64_t rows, uint64_t pg) {
    constexpr uint32_t R = sizeof(T) == 4 ? kRowsPerPageInt32 : kRowsPerPage8B;
    constexpr uint32_t DB = sizeof(T) == 4 ? 4u : 8u;
    uint32_t *dst = reinterpret_cast<uint32_t *>(pages + pg * kPageSize);
    const uint32_t nr = (uint32_t)min((uint64_t)R, rows - pg * R);
    if (lane_id() < DB / 4) __stcs(dst + lane_id(), lane_id() == 0 ? nr * 0x10001u : 0u);
    const uint32_t bm0 = kPageSize - (nr + 7) / 8;
    for (uint32_t k = (DB + nr * (uint32_t)sizeof(T)) / 4 + lane_id(); k < kPageSize / 4; k += 32) {
        uint32_t v = 0;
        if (4 * k >= bm0 && (4 * k + 4 - bm0) * 8 <= nr) {
            v = ~0u;
        } else if (4 * k + 4 > bm0) {
            for (uint32_t j = 0; j < 4; ++j) {
                if (4 * k + j < bm0) continue;
                const uint32_t i = 4 * k + j - bm0;
                v |= ((i + 1) * 8 <= nr ? 0xFFu : (1u << (nr - i * 8)) - 1u) << (8 * j);
            }
        }
        __stcs(dst + k, v);
    }
}

/* Page writer: the fixed-width result columns of a plan (tasks by value) or
 * of a batch (tasks in device memory) in one launch; task k's blocks stride
 * over its pages. One launch for a plan's columns instead of one each: at
 * C1's size each of those ran 6-10 us for 1-4 us of work. */
CJ_DEV void write_page_blocks(const PageTask &T, uint32_t b, PageSmem &sm) {
    const uint64_t rows = live_rows(T.rows, T.rows_dev);
    const uint32_t R = rows_per_page_dev(T.col.type);
    const uint64_t num_pages = (rows + R - 1) / R;
    if (b >= num_pages) return;
    if (T.finish == 1 || (T.finish == 2 && col_null_free(T.col) && !(T.table && !table_kind(T.table, 0)))) {
        constexpr uint32_t kWarps = kMatThreads / 32;
        for (uint64_t pg = b * kWarps + (threadIdx.x >> 5); pg < num_pages; pg += (uint64_t)T.blocks * kWarps) {
            if (T.col.type == CJ_INT32) finish_dense_page<int32_t>(T.out, rows, pg);
            else finish_dense_page<long long>(T.out, rows, pg);
        }
        return;
    }
    zero_page(sm);
    for (uint64_t pg = b; pg < num_pages; pg += T.blocks) {
        if (T.col.type == CJ_INT32) write_fixed_page<int32_t>(T.col, rows, kRowsPerPageInt32, pg, T.out, sm);
        else write_fixed_page<long long>(T.col, rows, kRowsPerPage8B, pg, T.out, sm);
    }
}

CJ_DEV uint32_t find_pages(const PageTask *tasks, uint32_t ntasks, uint32_t block) {
    uint32_t lo = 0, hi = ntasks;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (tasks[mid].block_base <= block) lo = mid;
        else hi = mid;
    }
    return lo;
}

struct PageArgs {
    PageTask t[kPageArgs];
    uint32_t n;
};

__global__ void __launch_bounds__(kMatThreads, kMatMinBlocks) k_write_pages(const __grid_constant__ PageArgs a) {
    __shared__ PageSmem sm;
    const PageTask &T = a.t[find_pages(a.t, a.n, blockIdx.x)];
    write_page_blocks(T, blockIdx.x - T.block_base, sm);
}

__global__ void __launch_bounds__(kMatThreads, kMatMinBlocks)
    k_write_pages_grouped(const PageTask *__restrict__ tasks, uint32_t ntasks) {
    __shared__ PageSmem sm;
    const PageTask &T = tasks[find_pages(tasks, ntasks, blockIdx.x)];
    write_page_blocks(T, blockIdx.x - T.block_base, sm);
}

/* Grouped row-id gather: task k covers global chunks [chunk_base, ...). */
__global__ void k_gather_grouped(const GatherTask *__restrict__ tasks, uint32_t ntasks, uint64_t total_chunks) {
    __shared__ uint32_t s_task;
    for (uint64_t gc = blockIdx.x; gc < total_chunks; gc += gridDim.x) {
        if (threadIdx.x == 0) {
            uint32_t lo = 0, hi = ntasks;
            while (hi - lo > 1) {
                uint32_t mid = (lo + hi) >> 1;
                if (tasks[mid].chunk_base <= gc) lo = mid;
                else hi = mid;
            }
            s_task = lo;
        }
        __syncthreads();
        const GatherTask &T = tasks[s_task];
        const uint64_t r0 = (gc - T.chunk_base) * kGatherChunk;
        const uint64_t r1 = min(T.n, r0 + kGatherChunk);
        gather_rows(T.src, T.idx, T.out, r0 + threadIdx.x, r1, blockDim.x);
        __syncthreads();
    }
}

/* ---------------- VARCHAR ----------------
 * Weights: a page holds rows a..b-1 when 8 (2 values + characters) + rows <=
 * 8 * 8188, so a row weighs 1, plus 16 and 8 a character when it is not NULL,
 * and a page's rows weigh kPageWeight at most. A long string's row weighs
 * more than a page by itself, which ends the segment before it. */
constexpr uint32_t kPageWeight = 8 * (kPageSize - 4);

CJ_DEV uint32_t row_weight(uint64_t d) {
    if (!d) return 1u;
    return desc_is_long(d) ? kPageWeight + 1u : 17u + 8u * desc_len(d);
}

/* Cuts tile t of a column into segments: the rows' descriptors (through the
 * row ids, eight a thread in flight) go to row_desc in row order, a block
 * scan of the weights to shared memory, and the first warp walks the
 * segments, 32 candidate ends a step. The last tile of the column to finish
 * turns the tiles' page counts into their first pages. Bound by the random
 * descriptor loads (32 bytes of L2 each). 1.8M rows: 20 us, before 60 us
 * with a thread walking 11 dependent steps a segment. */
CJ_DEV void plan_tile(const VarcharTask &T, uint32_t t, uint32_t *s_pre, uint32_t *wbuf, uint64_t *wbuf64,
                      bool *s_last) {
    const uint32_t TR = T.tile_rows;
    const uint64_t r0 = (uint64_t)t * TR;
    const uint32_t nt = (uint32_t)min((uint64_t)TR, T.rows - r0);
    const bool all_valid = col_all_valid(T.col);
    constexpr int kBatch = 8;
    for (uint32_t b0 = threadIdx.x; b0 < nt; b0 += kMatThreads * kBatch) {
        uint32_t br[kBatch];
        uint64_t d[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const uint32_t r = b0 + k * kMatThreads;
            br[k] = (uint32_t)(r0 + r);
            if (r < nt && T.col.rid_a) br[k] = __ldg(T.col.rid_a + br[k]);
        }
        if (T.col.rid_b) {
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (b0 + k * kMatThreads < nt) br[k] = __ldg(T.col.rid_b + br[k]);
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            d[k] = 0;
            if (b0 + k * kMatThreads < nt && (all_valid || valid_bit(T.col.valid, br[k])))
                d[k] = __ldg(T.col.str_desc + br[k]);
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const uint32_t r = b0 + k * kMatThreads;
            if (r >= nt) continue;
            T.row_desc[r0 + r] = d[k];
            s_pre[r] = row_weight(d[k]);
        }
    }
    __syncthreads();
    /* exclusive prefix of the weights, each thread a run of rows */
    const uint32_t per = (nt + kMatThreads - 1) / kMatThreads, q0 = min(threadIdx.x * per, nt), q1 = min(q0 + per, nt);
    uint32_t sum = 0, total;
    for (uint32_t r = q0; r < q1; ++r) sum += s_pre[r];
    uint32_t pre = block_exclusive_scan<uint32_t>(sum, wbuf, &total);
    for (uint32_t r = q0; r < q1; ++r) {
        const uint32_t w = s_pre[r];
        s_pre[r] = pre;
        pre += w;
    }
    if (threadIdx.x == 0) s_pre[nt] = total;
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint32_t lane = lane_id();
        uint32_t *seg = T.seg + (uint64_t)t * (TR + 1), *seg_page = T.seg_page + (uint64_t)t * (TR + 1);
        uint32_t a = 0, ns = 0, np = 0;
        while (a < nt) {
            if (lane == 0) {
                seg[ns] = a;
                seg_page[ns] = np;
            }
            uint32_t end, pages = 1;
            if (s_pre[a + 1] - s_pre[a] > kPageWeight) { /* a long string */
                end = a + 1;
                pages = desc_len(T.row_desc[r0 + a]);
            } else {
                /* the largest end with s_pre[end] - s_pre[a] <= kPageWeight,
                 * at least a + 1 */
                uint32_t lo = a + 1, hi = nt;
                while (lo < hi) {
                    const uint32_t step = (hi - lo + 31) / 32, e = lo + step * (lane + 1);
                    const bool ok = e <= hi && s_pre[e] - s_pre[a] <= kPageWeight;
                    const uint32_t n = __popc(__ballot_sync(0xffffffffu, ok)); /* a prefix of the lanes */
                    const uint32_t next = lo + step * n;
                    hi = min(hi, next + step - 1);
                    lo = next;
                }
                end = lo;
            }
            np += pages;
            ++ns;
            a = end;
        }
        if (lane == 0) {
            seg[ns] = nt;
            T.nseg[t] = ns;
            T.tile_pages[t] = np;
            __threadfence();
            *s_last = atomicAdd(T.done, 1u) == T.tiles - 1;
        }
    }
    __syncthreads();
    if (!*s_last) return;
    __threadfence();
    uint64_t off = 0;
    constexpr uint32_t kRun = 8;
    for (uint32_t c0 = 0; c0 < T.tiles; c0 += kMatThreads * kRun) {
        uint32_t v[kRun];
        uint64_t s = 0, tot;
#pragma unroll
        for (uint32_t k = 0; k < kRun; ++k) {
            const uint32_t c = c0 + threadIdx.x * kRun + k;
            v[k] = c < T.tiles ? __ldcg(T.tile_pages + c) : 0u;
            s += v[k];
        }
        uint64_t e = off + block_exclusive_scan<uint64_t>(s, wbuf64, &tot);
#pragma unroll
        for (uint32_t k = 0; k < kRun; ++k) {
            const uint32_t c = c0 + threadIdx.x * kRun + k;
            if (c < T.tiles) T.tile_base[c] = e;
            e += v[k];
        }
        off += tot;
    }
    if (threadIdx.x == 0) *T.total_pages = off;
}

/* Writes segment g of tile t. Block-wide. */
struct VarcharShared {
    uint4 page[kPageSize / 16];
    uint64_t src[kMatThreads]; /* a string's first character, by row of the chunk */
    uint16_t dst[kMatThreads], len[kMatThreads];
    uint32_t wbuf[kMatThreads / 32 + 1];
};
constexpr uint32_t kCopyLanes = 8;    /* lanes that copy a string together      */
constexpr uint32_t kBlockCopy = 256;  /* longer strings are copied by the block */

/* Characters q .. q + 3 of a string at src (fewer at its end) to shared
 * memory: one or two aligned words, no byte outside the string's words. */
CJ_DEV void copy4(const uint8_t *src, uint8_t *dst, uint32_t q, uint32_t len) {
    const uint32_t n = min(4u, len - q);
    const uintptr_t s = reinterpret_cast<uintptr_t>(src + q);
    const uint32_t sh = (uint32_t)(s & 3u);
    const uint32_t *w = reinterpret_cast<const uint32_t *>(s & ~(uintptr_t)3);
    const uint32_t lo = __ldg(w), hi = sh + n > 4 ? __ldg(w + 1) : 0u;
    const uint32_t v = __funnelshift_r(lo, hi, 8 * sh);
    dst[q] = (uint8_t)v;
    if (n > 1) dst[q + 1] = (uint8_t)(v >> 8);
    if (n > 2) dst[q + 2] = (uint8_t)(v >> 16);
    if (n > 3) dst[q + 3] = (uint8_t)(v >> 24);
}

CJ_DEV void write_segment(const VarcharTask &T, uint32_t t, uint32_t g, VarcharShared &sh) {
    const uint64_t r0 = (uint64_t)t * T.tile_rows, s0 = (uint64_t)t * (T.tile_rows + 1);
    const uint32_t a = T.seg[s0 + g], n = T.seg[s0 + g + 1] - a;
    uint8_t *out = T.out + (T.tile_base[t] + T.seg_page[s0 + g]) * kPageSize;
    const uint64_t *desc = T.row_desc + r0 + a;
    const uint64_t d0 = desc[0];
    if (d0 && desc_is_long(d0)) {
        const uint4 *src = reinterpret_cast<const uint4 *>(T.col.pages + desc_pos(d0) * kPageSize);
        uint4 *dst = reinterpret_cast<uint4 *>(out);
        const uint64_t n16 = (uint64_t)desc_len(d0) * (kPageSize / 16);
        for (uint64_t k = threadIdx.x; k < n16; k += kMatThreads) dst[k] = __ldg(src + k);
        return;
    }
    const uint32_t warp = threadIdx.x >> 5, lane = lane_id();
    uint8_t *sp = reinterpret_cast<uint8_t *>(sh.page);
    /* the number of values says where the characters begin */
    uint32_t mine = 0, nv;
    for (uint32_t j = threadIdx.x; j < n; j += kMatThreads) mine += desc[j] != 0;
    for (uint32_t k = threadIdx.x; k < kPageSize / 16; k += kMatThreads) sh.page[k] = make_uint4(0, 0, 0, 0);
    block_exclusive_scan<uint32_t>(mine, sh.wbuf, &nv);
    const uint32_t chars_at = 4u + 2u * nv, bm_bytes = (n + 7) / 8;
    uint8_t *bm = sp + kPageSize - bm_bytes;
    uint16_t *offs = reinterpret_cast<uint16_t *>(sp + 4);
    uint32_t before = 0; /* characters (low half) and values (high half) of earlier chunks */
    for (uint32_t j0 = 0; j0 < n; j0 += kMatThreads) {
        const uint32_t j = j0 + threadIdx.x;
        const uint64_t d = j < n ? desc[j] : 0ull;
        const uint32_t len = d ? desc_len(d) : 0u;
        uint32_t total;
        /* at most 8188 characters and 4094 values a page: no carry between the halves */
        const uint32_t pre = before + block_exclusive_scan<uint32_t>(len | (d ? 1u << 16 : 0u), sh.wbuf, &total);
        before += total;
        const uint32_t beg = pre & 0xFFFFu;
        if (d) offs[pre >> 16] = (uint16_t)(beg + len);
        sh.src[threadIdx.x] = d ? desc_pos(d) : 0ull;
        sh.dst[threadIdx.x] = (uint16_t)(chars_at + beg);
        sh.len[threadIdx.x] = (uint16_t)len;
        const uint32_t ball = __ballot_sync(0xffffffffu, d != 0);
        if (lane < 4) {
            const uint32_t byte = (j0 + warp * 32) / 8 + lane;
            if (byte < bm_bytes) bm[byte] = (uint8_t)(ball >> (8 * lane));
        }
        const bool long_ones = __syncthreads_or(len > kBlockCopy);
        const uint32_t rows = min((uint32_t)kMatThreads, n - j0);
#pragma unroll 4
        for (uint32_t i = threadIdx.x / kCopyLanes; i < rows; i += kMatThreads / kCopyLanes) {
            const uint32_t l = sh.len[i];
            if (l > kBlockCopy) continue;
            const uint8_t *src = T.col.pages + sh.src[i];
            for (uint32_t q = (threadIdx.x % kCopyLanes) * 4; q < l; q += kCopyLanes * 4)
                copy4(src, sp + sh.dst[i], q, l);
        }
        if (long_ones)
            for (uint32_t i = 0; i < rows; ++i) {
                const uint32_t l = sh.len[i];
                if (l <= kBlockCopy) continue;
                for (uint32_t q = threadIdx.x * 4; q < l; q += kMatThreads * 4)
                    copy4(T.col.pages + sh.src[i], sp + sh.dst[i], q, l);
            }
        __syncthreads();
    }
    if (threadIdx.x == 0) *reinterpret_cast<uint32_t *>(sp) = n | (nv << 16);
    __syncthreads();
    uint4 *dst = reinterpret_cast<uint4 *>(out);
    for (uint32_t k = threadIdx.x; k < kPageSize / 16; k += kMatThreads) __stcs(dst + k, sh.page[k]);
    __syncthreads();
}

/* Columns of a result, by value. Pass 1: a block per tile; pass 2:
 * kSegBlocks blocks per tile, which share its segments (about six at 22
 * bytes a string and 2,048 rows). */
constexpr uint32_t kSegBlocks = 8;
struct VarcharArgs {
    VarcharTask t[kVarcharArgs];
    uint32_t n;
};
CJ_DEV uint32_t find_varchar(const VarcharArgs &a, uint32_t tile) {
    uint32_t c = 0;
    while (c + 1 < a.n && a.t[c + 1].tile_first <= tile) ++c;
    return c;
}

__global__ void __launch_bounds__(kMatThreads) k_varchar_plan(const __grid_constant__ VarcharArgs a) {
    extern __shared__ uint32_t s_pre[];
    __shared__ uint32_t wbuf[kMatThreads / 32 + 1];
    __shared__ uint64_t wbuf64[kMatThreads / 32 + 1];
    __shared__ bool s_last;
    const VarcharTask &T = a.t[find_varchar(a, blockIdx.x)];
    plan_tile(T, blockIdx.x - T.tile_first, s_pre, wbuf, wbuf64, &s_last);
}

/* 1.8M strings of 20 characters on average: 74 us, before 212 us with a
 * block per tile that planned it again and a lane per string, byte by byte. */
__global__ void __launch_bounds__(kMatThreads, 6) k_varchar_write(const __grid_constant__ VarcharArgs a) {
    __shared__ VarcharShared sh;
    const uint32_t tile = blockIdx.x / kSegBlocks;
    const VarcharTask &T = a.t[find_varchar(a, tile)];
    const uint32_t t = tile - T.tile_first, ns = T.nseg[t];
    for (uint32_t g = blockIdx.x % kSegBlocks; g < ns; g += kSegBlocks) write_segment(T, t, g, sh);
}

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

} // namespace

cudaError_t launch_gather_u32(const Launch &L, const uint32_t *src, const uint32_t *idx, uint64_t n,
                              uint32_t *out) {
    if (n == 0) return cudaSuccess;
    uint64_t g = (n + 255) / 256;
    uint64_t cap = (uint64_t)L.num_sms * 8;
    if (g > cap) g = cap;
    k_gather_u32<<<(unsigned)g, 256, 0, L.stream>>>(src, idx, n, out);
    count_launches(1);
    return cudaGetLastError();
}

uint32_t place_pages(const Launch &L, PageTask *tasks, size_t n) {
    uint32_t grid = 0;
    for (size_t k = 0; k < n; ++k) {
        const uint32_t R = rows_per_page_fixed(tasks[k].col.type);
        tasks[k].blocks = (uint32_t)std::min<uint64_t>((tasks[k].rows + R - 1) / R, (uint64_t)L.num_sms * kMatMinBlocks);
        tasks[k].block_base = grid;
        grid += tasks[k].blocks;
    }
    return grid;
}

cudaError_t launch_write_pages(const Launch &L, PageTask *tasks, size_t n) {
    for (size_t k = 0; k < n; k += kPageArgs) {
        PageArgs a;
        a.n = (uint32_t)std::min<size_t>(n - k, kPageArgs);
        const uint32_t grid = place_pages(L, tasks + k, a.n);
        std::copy(tasks + k, tasks + k + a.n, a.t);
        if (!grid) continue;
        k_write_pages<<<grid, kMatThreads, 0, L.stream>>>(a);
        count_launches(1);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_write_pages_grouped(const Launch &L, const PageTask *tasks_dev, uint32_t n, uint32_t grid) {
    if (!grid) return cudaSuccess;
    k_write_pages_grouped<<<grid, kMatThreads, 0, L.stream>>>(tasks_dev, n);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_gather_grouped(const Launch &L, const GatherTask *tasks_dev, uint32_t ntasks,
                                  uint64_t total_chunks) {
    if (!total_chunks) return cudaSuccess;
    uint64_t g = std::min<uint64_t>(total_chunks, (uint64_t)L.num_sms * 8);
    k_gather_grouped<<<(unsigned)g, 256, 0, L.stream>>>(tasks_dev, ntasks, total_chunks);
    count_launches(1);
    return cudaGetLastError();
}

uint32_t rows_per_page_fixed(int32_t type) {
    return type == CJ_INT32 ? kRowsPerPageInt32 : kRowsPerPage8B;
}

/* temp: page counts and first pages of the tiles, segment counts, the
 * segments' first rows and pages, the rows' descriptors */
size_t varchar_temp_bytes(uint64_t rows, uint32_t TR) {
    const uint64_t tiles = (rows + TR - 1) / TR, segs = tiles * (TR + 1ull);
    return align256(tiles * 4) * 2 + align256(tiles * 8) + align256(segs * 4) * 2 + align256(rows * 8);
}

void place_varchar(VarcharTask &t, uint32_t TR, void *temp) {
    const uint64_t tiles = (t.rows + TR - 1) / TR, segs = tiles * (TR + 1ull);
    char *p = reinterpret_cast<char *>(temp);
    auto take = [&](uint64_t bytes) {
        char *q = p;
        p += align256(bytes);
        return q;
    };
    t.tile_rows = TR;
    t.tiles = (uint32_t)tiles;
    t.tile_pages = reinterpret_cast<uint32_t *>(take(tiles * 4));
    t.nseg = reinterpret_cast<uint32_t *>(take(tiles * 4));
    t.tile_base = reinterpret_cast<uint64_t *>(take(tiles * 8));
    t.seg = reinterpret_cast<uint32_t *>(take(segs * 4));
    t.seg_page = reinterpret_cast<uint32_t *>(take(segs * 4));
    t.row_desc = reinterpret_cast<uint64_t *>(take(t.rows * 8));
}

cudaError_t launch_varchar(const Launch &L, const VarcharTask *tasks, size_t n, bool plan) {
    for (size_t k = 0; k < n;) {
        VarcharArgs a;
        a.n = 0;
        uint64_t tiles = 0;
        size_t smem = 0;
        while (k < n && a.n < kVarcharArgs && (tiles + tasks[k].tiles) * kSegBlocks < (1ull << 31)) {
            a.t[a.n] = tasks[k++];
            a.t[a.n].tile_first = (uint32_t)tiles;
            tiles += a.t[a.n].tiles;
            smem = std::max(smem, ((size_t)a.t[a.n].tile_rows + 1) * 4);
            ++a.n;
        }
        if (!a.n) return cudaErrorInvalidValue;
        if (!tiles) continue;
        if (plan) k_varchar_plan<<<(unsigned)tiles, kMatThreads, smem, L.stream>>>(a);
        else k_varchar_write<<<(unsigned)(tiles * kSegBlocks), kMatThreads, 0, L.stream>>>(a);
        count_launches(1);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

} // namespace cj
