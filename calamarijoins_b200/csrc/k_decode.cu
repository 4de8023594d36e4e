/*
 * k_decode.cu — page decode: 8 KiB pages in HBM -> dense device columns.
 *
 * Follows the page format of the reference (include/data_model/plan.h:
 * 75-142, 187-366; README.md "Data format") and its readers:
 *   - row counts per page, long-string pages counting as one row (0xffff)
 *     or none (0xfffe): PageIndex::build (include/data_access/
 *     columnar_reader.h:122-200)
 *   - dense pages (n_rows == n_values) read values in row order without
 *     the bitmap, sparse pages locate a value by popcount of the bitmap
 *     prefix: ColumnarReader::read_dense_int32 / read_sparse
 *     (columnar_reader.h:385-393, 452-474)
 *   - VARCHAR: n_values u16 end offsets at +4, characters after them
 *     (include/materialization/page_builders.h:26-37)
 *
 * One CTA decodes one page at a time (grid-stride over pages); the page's
 * bitmap and its popcount prefix live in shared memory. Value writes are
 * coalesced; the validity bitmap is written with plain stores except for
 * the (at most two) 32-row words a page shares with its neighbours, which
 * use atomicOr on a zeroed bitmap.
 */
#include <algorithm>

#include "cj_device.cuh"

namespace cj {
namespace {

constexpr int kDecodeThreads = 256;
constexpr uint32_t kMaxBitmapWords = 2048; /* 65535 rows */

CJ_DEV uint16_t rd16(const uint8_t *p) { return *reinterpret_cast<const uint16_t *>(p); }

/* Rows a page contributes (n_rows; 1 for a long-string start page, 0 for a
 * continuation) and header checks. */
CJ_DEV uint32_t page_rows_of(const uint8_t *pg, int32_t type, unsigned int *err) {
    uint32_t nr = rd16(pg), nv = rd16(pg + 2);
    uint32_t r = nr;
    if (type == CJ_VARCHAR) {
        if (nr == 0xffff) {
            r = 1;
            if (nv == 0 || nv > kLongChunk) atomicOr(err, DEV_ERR_PAGE_HEADER);
        } else if (nr == 0xfffe) {
            r = 0;
            if (nv == 0 || nv > kLongChunk) atomicOr(err, DEV_ERR_PAGE_HEADER);
        } else if (nv > nr || 4u + 2u * nv + (nr + 7) / 8 > kPageSize) {
            atomicOr(err, DEV_ERR_PAGE_HEADER);
        }
    } else {
        uint32_t w = type == CJ_INT32 ? 4u : 8u;
        if (nv > nr || w + w * nv + (nr + 7) / 8 > kPageSize) atomicOr(err, DEV_ERR_PAGE_HEADER);
    }
    return r;
}

/* COL_* flags of page p of np: COL_HAS_NULLS if a regular page stores
 * fewer values than rows (long-string pages hold one non-NULL row or none);
 * COL_NOT_DIRECT for VARCHAR, or unless every page but the last holds
 * exactly R rows and the last 1..R. */
CJ_DEV uint32_t page_flags(const uint8_t *pg, uint64_t p, uint64_t np, int32_t type) {
    const uint32_t nr = rd16(pg), nv = rd16(pg + 2);
    if (type == CJ_VARCHAR) return COL_NOT_DIRECT | ((nr < 0xfffe && nv < nr) ? COL_HAS_NULLS : 0u);
    const uint32_t R = type == CJ_INT32 ? kRowsPerPageInt32 : kRowsPerPage8B;
    uint32_t f = nv < nr ? COL_HAS_NULLS : 0u;
    if (p + 1 < np ? nr != R : (nr == 0 || nr > R)) f |= COL_NOT_DIRECT;
    return f;
}

/* ---- page index: every column of a plan (or batch) in one launch ----
 * A block owns kIndexChunk consecutive pages of one column, one page per
 * thread: it stores each page's first row relative to the chunk (loc) and
 * the chunk's rows (base), ORs the column's COL_* flags and clears its share
 * of the column's validity bitmap. The last block of a column to finish
 * turns base into the rows before each chunk and checks the column's row
 * count (a mismatch raises DEV_ERR_ROW_COUNT and makes the column
 * NOT_DIRECT, so readers stay inside its decoded arrays).
 *
 * Bound by launch and header latency, not by bytes (one 32-byte sector per
 * 8 KB page). Per column it used to take two launches and two memsets
 * (10-13 us of a plan's time each on the device); now the columns share one
 * launch, and the second pass is folded into readers, which add the two
 * numbers (page_first_row). */
constexpr int kIndexThreads = kIndexChunk;

CJ_DEV void index_chunk(const ColumnTask &T, uint32_t b) {
    __shared__ uint64_t wbuf[kIndexThreads / 32 + 1];
    __shared__ bool s_last;
    const uint64_t np = T.num_pages, p = (uint64_t)b * kIndexThreads + threadIdx.x;
    uint32_t f = 0;
    uint64_t r = 0;
    if (p < np) {
        const uint8_t *pg = T.pages + p * kPageSize;
        r = page_rows_of(pg, T.type, T.err);
        f = page_flags(pg, p, np, T.type);
    }
    f = __reduce_or_sync(0xffffffffu, f);
    if (f && lane_id() == 0) atomicOr(&T.state->flags, f);
    uint64_t tot;
    const uint64_t pre = block_exclusive_scan<uint64_t>(r, wbuf, &tot);
    if (p < np) T.loc[p] = (uint32_t)pre; /* at most 256 * 65535 rows */
    const uint64_t words = T.rows ? (T.rows + 31) / 32 : 1;
    const uint64_t w0 = words * b / T.index_blocks, w1 = words * (b + 1) / T.index_blocks;
    for (uint64_t w = w0 + threadIdx.x; w < w1; w += kIndexThreads) T.valid[w] = 0u;
    if (threadIdx.x == 0) {
        T.base[b] = tot;
        __threadfence();
        s_last = atomicAdd(&T.state->done, 1u) == T.index_blocks - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    uint64_t off = 0;
    for (uint32_t c0 = 0; c0 < T.index_blocks; c0 += kIndexThreads) {
        const uint32_t c = c0 + threadIdx.x;
        const uint64_t v = c < T.index_blocks ? __ldcg(T.base + c) : 0;
        const uint64_t e = block_exclusive_scan<uint64_t>(v, wbuf, &tot);
        if (c < T.index_blocks) T.base[c] = off + e;
        off += tot;
    }
    if (threadIdx.x == 0 && off != T.rows) {
        atomicOr(T.err, DEV_ERR_ROW_COUNT);
        atomicOr(&T.state->flags, COL_NOT_DIRECT);
    }
}

/* Task of a block: the last task whose first block is at most `block`. */
template <bool kIndex> CJ_DEV uint32_t find_column(const ColumnTask *tasks, uint32_t ntasks, uint32_t block) {
    uint32_t lo = 0, hi = ntasks;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if ((kIndex ? tasks[mid].index_base : tasks[mid].decode_base) <= block) lo = mid;
        else hi = mid;
    }
    return lo;
}

/* Tasks travel as a kernel argument (a plan's few columns: no copy to wait
 * for) or in device memory (a batch's hundreds). */
struct ColumnArgs {
    ColumnTask t[kColumnArgs];
    uint32_t n;
};

__global__ void __launch_bounds__(kIndexThreads) k_page_index(const __grid_constant__ ColumnArgs a) {
    const ColumnTask &T = a.t[find_column<true>(a.t, a.n, blockIdx.x)];
    index_chunk(T, blockIdx.x - T.index_base);
}

__global__ void __launch_bounds__(kIndexThreads) k_page_index_grouped(const ColumnTask *tasks, uint32_t n) {
    const ColumnTask &T = tasks[find_column<true>(tasks, n, blockIdx.x)];
    index_chunk(T, blockIdx.x - T.index_base);
}

/* Loads a sparse page's bitmap into s_bm (bits past n_rows cleared) and the
 * exclusive popcount prefix per word into s_pre. Block-wide. */
CJ_DEV void load_page_bitmap(const uint8_t *pg, uint32_t nr, uint32_t *s_bm, uint32_t *s_pre,
                             uint32_t *wbuf) {
    const uint32_t nbytes = (nr + 7) / 8, nwords = (nr + 31) / 32;
    const uint8_t *bmb = pg + kPageSize - nbytes;
    for (uint32_t w = threadIdx.x; w < nwords; w += blockDim.x) {
        uint32_t v = 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            uint32_t bi = w * 4 + b;
            if (bi < nbytes) v |= (uint32_t)bmb[bi] << (8 * b);
        }
        uint32_t live = nr - w * 32;
        if (live < 32) v &= (1u << live) - 1u;
        s_bm[w] = v;
    }
    __syncthreads();
    const uint32_t per = (nwords + blockDim.x - 1) / blockDim.x;
    const uint32_t w0 = threadIdx.x * per;
    uint32_t s = 0;
    for (uint32_t k = 0; k < per; ++k)
        if (w0 + k < nwords) s += __popc(s_bm[w0 + k]);
    uint32_t tot;
    uint32_t pre = block_exclusive_scan<uint32_t>(s, wbuf, &tot);
    for (uint32_t k = 0; k < per; ++k)
        if (w0 + k < nwords) {
            s_pre[w0 + k] = pre;
            pre += __popc(s_bm[w0 + k]);
        }
    __syncthreads();
}

/* Value index of page row i of a sparse page, or -1 if the row is NULL. */
CJ_DEV int value_index(const uint32_t *s_bm, const uint32_t *s_pre, uint32_t i) {
    uint32_t w = i >> 5, b = i & 31;
    uint32_t word = s_bm[w];
    if (!((word >> b) & 1u)) return -1;
    return (int)(s_pre[w] + __popc(word & ((1u << b) - 1u)));
}

/* 32 validity bits of the output word whose first row is page row `off`
 * (off may be negative for the page's first word). */
CJ_DEV uint32_t page_bits(bool dense, const uint32_t *s_bm, uint32_t nr, int64_t off) {
    if (dense) {
        int64_t lo = off < 0 ? -off : 0;
        int64_t hi = (int64_t)nr - off;
        if (hi > 32) hi = 32;
        if (hi <= lo) return 0;
        uint32_t width = (uint32_t)(hi - lo);
        uint32_t m = width >= 32 ? 0xffffffffu : ((1u << width) - 1u);
        return m << lo;
    }
    if (off < 0) return s_bm[0] << (uint32_t)(-off);
    const uint32_t nwords = (nr + 31) / 32;
    uint32_t w0 = (uint32_t)(off >> 5), s = (uint32_t)(off & 31);
    uint32_t lo = w0 < nwords ? s_bm[w0] : 0u;
    uint32_t hi = w0 + 1 < nwords ? s_bm[w0 + 1] : 0u;
    return s ? (lo >> s) | (hi << (32 - s)) : lo;
}

CJ_DEV void write_validity(bool dense, const uint32_t *s_bm, uint32_t nr, uint64_t rs,
                           uint32_t *valid) {
    if (nr == 0) return;
    const uint64_t fw = rs >> 5, lw = (rs + nr - 1) >> 5;
    for (uint64_t ow = fw + threadIdx.x; ow <= lw; ow += blockDim.x) {
        int64_t off = (int64_t)(ow * 32) - (int64_t)rs;
        uint32_t bits = page_bits(dense, s_bm, nr, off);
        if (off >= 0 && off + 32 <= (int64_t)nr)
            valid[ow] = bits;
        else if (bits)
            atomicOr(valid + ow, bits);
    }
}

struct DecodeSmem {
    uint32_t bm[kMaxBitmapWords];
    uint32_t pre[kMaxBitmapWords];
    uint32_t wbuf[kDecodeThreads / 32 + 1];
};

/* Decodes fixed-width page p (of a column whose pages start at `pages`)
 * whose first row is rs. Block-wide. */
template <typename T>
CJ_DEV void decode_fixed_page(const uint8_t *__restrict__ pages, uint64_t p, uint64_t rs, uint64_t max_rows,
                              T *__restrict__ values, uint32_t *__restrict__ valid, unsigned int *err,
                              DecodeSmem &sm) {
    constexpr uint32_t DB = sizeof(T) == 4 ? 4u : 8u;
    const uint8_t *pg = pages + p * kPageSize;
    const uint32_t nr = rd16(pg), nv = rd16(pg + 2);
    if (nv > nr || DB + (uint32_t)sizeof(T) * nv + (nr + 7) / 8 > kPageSize) return;
    if (rs + nr > max_rows) {
        if (threadIdx.x == 0) atomicOr(err, DEV_ERR_ROW_COUNT);
        return;
    }
    const T *vals = reinterpret_cast<const T *>(pg + DB);
    if (nr != nv) {
        load_page_bitmap(pg, nr, sm.bm, sm.pre, sm.wbuf);
        /* Sparse page: a thread takes 4 consecutive rows, whose non-NULL
         * values are consecutive in the page (one bitmap word and its
         * prefix give the first index), and stores the 4 rows at once when
         * the page starts on a multiple of 4 rows. */
        const bool vec = sizeof(T) == 4 && (rs & 3u) == 0;
        for (uint32_t g = threadIdx.x; g * 4 < nr; g += blockDim.x) {
            const uint32_t r = g * 4, w = r >> 5, sh = r & 31u;
            const uint32_t word = sm.bm[w]; /* bits past n_rows are clear */
            uint32_t idx = sm.pre[w] + __popc(word & ((1u << sh) - 1u));
            const uint32_t nib = (word >> sh) & 0xFu;
            T v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = T(0);
                if ((nib >> k) & 1u) {
                    if (idx >= nv) atomicOr(err, DEV_ERR_PAGE_HEADER); /* bitmap holds > n_values bits */
                    else v[k] = __ldcs(vals + idx);
                    ++idx;
                }
            }
            bool done = false;
            if constexpr (sizeof(T) == 4) {
                if (vec && r + 4 <= nr) {
                    *reinterpret_cast<int4 *>(values + rs + r) = make_int4(v[0], v[1], v[2], v[3]);
                    done = true;
                }
            }
            if (!done) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (r + k < nr) values[rs + r + k] = v[k];
            }
        }
        write_validity(false, sm.bm, nr, rs, valid);
        __syncthreads();
        return;
    }
    /* All loads of a chunk are issued before any store: a full page (1984 /
     * 1007 rows) is one chunk, so it costs one DRAM round trip. */
    constexpr int kSlabs =
        (int)(((sizeof(T) == 4 ? kRowsPerPageInt32 : kRowsPerPage8B) + kDecodeThreads - 1) / kDecodeThreads);
    for (uint32_t base = 0; base < nr; base += kSlabs * kDecodeThreads) {
        T v[kSlabs];
#pragma unroll
        for (int k = 0; k < kSlabs; ++k) {
            const uint32_t i = base + k * kDecodeThreads + threadIdx.x;
            v[k] = T(0);
            if (i < nr) v[k] = __ldcs(vals + i);
        }
#pragma unroll
        for (int k = 0; k < kSlabs; ++k) {
            const uint32_t i = base + k * kDecodeThreads + threadIdx.x;
            if (i < nr) values[rs + i] = v[k];
        }
    }
    write_validity(true, sm.bm, nr, rs, valid);
    __syncthreads();
}

CJ_DEV void decode_varchar_page(const uint8_t *__restrict__ pages, uint64_t p, uint64_t np, uint64_t rs,
                                uint64_t max_rows, uint64_t *__restrict__ desc, uint32_t *__restrict__ valid,
                                unsigned int *err, DecodeSmem &sm) {
    const uint8_t *pg = pages + p * kPageSize;
    const uint32_t nr = rd16(pg), nv = rd16(pg + 2);
    if (nr == 0xfffe) {
        if (threadIdx.x == 0) {
            uint32_t prev = p ? rd16(pg - kPageSize) : 0u;
            if (prev != 0xffff && prev != 0xfffe) atomicOr(err, DEV_ERR_LONG_CHAIN);
        }
        return;
    }
    if (nr == 0xffff) {
        if (threadIdx.x == 0 && rs >= max_rows) atomicOr(err, DEV_ERR_ROW_COUNT);
        if (threadIdx.x == 0 && rs < max_rows) {
            uint64_t q = p + 1;
            while (q < np && rd16(pages + q * kPageSize) == 0xfffe) ++q;
            uint64_t chain = q - p;
            if (chain > 0xFFFFFFull) {
                atomicOr(err, DEV_ERR_LONG_CHAIN);
                chain = 0xFFFFFF;
            }
            desc[rs] = desc_long(p, (uint32_t)chain);
            atomicOr(valid + (rs >> 5), 1u << (rs & 31));
        }
        return;
    }
    if (nv > nr || 4u + 2u * nv + (nr + 7) / 8 > kPageSize) return;
    if (rs + nr > max_rows) {
        if (threadIdx.x == 0) atomicOr(err, DEV_ERR_ROW_COUNT);
        return;
    }
    const bool dense = nr == nv;
    if (!dense) load_page_bitmap(pg, nr, sm.bm, sm.pre, sm.wbuf);
    const uint16_t *offs = reinterpret_cast<const uint16_t *>(pg + 4);
    const uint32_t chars_at = 4u + 2u * nv;
    const uint32_t chars_cap = kPageSize - (nr + 7) / 8 - chars_at;
    for (uint32_t i = threadIdx.x; i < nr; i += blockDim.x) {
        int k = dense ? (int)i : value_index(sm.bm, sm.pre, i);
        uint64_t d = 0;
        if (k >= (int)nv) {
            atomicOr(err, DEV_ERR_PAGE_HEADER); /* bitmap holds > n_values bits */
        } else if (k >= 0) {
            uint32_t start = k ? offs[k - 1] : 0u, end = offs[k];
            if (end < start || end > chars_cap) {
                atomicOr(err, DEV_ERR_VARCHAR_OFFSETS);
            } else {
                d = desc_short(p * kPageSize + chars_at + start, end - start);
            }
        }
        desc[rs + i] = d;
    }
    write_validity(dense, sm.bm, nr, rs, valid);
    __syncthreads();
}

/* Decode of every column that is not read in place: task k's blocks stride
 * over its pages; the blocks of a column read in place (flags 0) leave at
 * once. 32 registers and 16 KB of shared memory: 8 CTAs per SM. */
CJ_DEV void decode_blocks(const ColumnTask &T, uint32_t b, DecodeSmem &sm) {
    if (T.type != CJ_VARCHAR && T.state->flags == 0u) return;
    for (uint64_t p = b; p < T.num_pages; p += T.decode_blocks) {
        const uint64_t rs = page_first_row(T.base, T.loc, p);
        if (T.type == CJ_VARCHAR)
            decode_varchar_page(T.pages, p, T.num_pages, rs, T.rows, T.desc, T.valid, T.err, sm);
        else if (T.type == CJ_INT32)
            decode_fixed_page<int32_t>(T.pages, p, rs, T.rows, reinterpret_cast<int32_t *>(T.values), T.valid, T.err,
                                       sm);
        else
            decode_fixed_page<long long>(T.pages, p, rs, T.rows, reinterpret_cast<long long *>(T.values), T.valid,
                                         T.err, sm);
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kDecodeThreads, 8) k_decode(const __grid_constant__ ColumnArgs a) {
    __shared__ DecodeSmem sm;
    const ColumnTask &T = a.t[find_column<false>(a.t, a.n, blockIdx.x)];
    decode_blocks(T, blockIdx.x - T.decode_base, sm);
}

__global__ void __launch_bounds__(kDecodeThreads, 8) k_decode_grouped(const ColumnTask *tasks, uint32_t n) {
    __shared__ DecodeSmem sm;
    const ColumnTask &T = tasks[find_column<false>(tasks, n, blockIdx.x)];
    decode_blocks(T, blockIdx.x - T.decode_base, sm);
}

} // namespace

uint32_t index_blocks(uint64_t np) { return (uint32_t)std::max<uint64_t>((np + kIndexChunk - 1) / kIndexChunk, 1); }

ColumnGrid place_columns(const Launch &L, ColumnTask *tasks, size_t n) {
    ColumnGrid g;
    const uint64_t wave = (uint64_t)L.num_sms * 8;
    for (size_t k = 0; k < n; ++k) {
        ColumnTask &t = tasks[k];
        t.index_blocks = index_blocks(t.num_pages);
        t.index_base = g.index;
        t.decode_blocks = (uint32_t)std::min<uint64_t>(t.num_pages, wave);
        t.decode_base = g.decode;
        g.index += t.index_blocks;
        g.decode += t.decode_blocks;
    }
    return g;
}

cudaError_t launch_columns(const Launch &L, ColumnTask *tasks, size_t n, bool index) {
    for (size_t k = 0; k < n; k += kColumnArgs) {
        ColumnArgs a;
        a.n = (uint32_t)std::min<size_t>(n - k, kColumnArgs);
        const ColumnGrid g = place_columns(L, tasks + k, a.n);
        std::copy(tasks + k, tasks + k + a.n, a.t);
        if (index) k_page_index<<<g.index, kIndexThreads, 0, L.stream>>>(a);
        else if (g.decode) k_decode<<<g.decode, kDecodeThreads, 0, L.stream>>>(a);
        count_launches(index || g.decode ? 1 : 0);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t launch_columns_grouped(const Launch &L, const ColumnTask *tasks_dev, uint32_t n, const ColumnGrid &g) {
    if (!n) return cudaSuccess;
    k_page_index_grouped<<<g.index, kIndexThreads, 0, L.stream>>>(tasks_dev, n);
    if (g.decode) k_decode_grouped<<<g.decode, kDecodeThreads, 0, L.stream>>>(tasks_dev, n);
    count_launches(g.decode ? 2 : 1);
    return cudaGetLastError();
}

} // namespace cj
