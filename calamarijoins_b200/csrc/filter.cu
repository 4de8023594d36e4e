/*
 * filter.cu — scan-side filters on resident tables (cj_table_filter): the
 * GPU form of the predicate evaluation the reference runs while it loads a
 * table, before execute() (src/build_table.cpp:201-367; Comparison and
 * LogicalOperation, include/data_model/statement.h:54-260,
 * src/statement.cpp:47-241, InnerColumn<T>, include/data_model/
 * inner_column.h).
 *
 * The reference evaluates a predicate column-wise into byte bitmaps and
 * copies the selected rows into a new ColumnarTable. Here:
 *   1. each column the predicate or the projection needs is decoded from its
 *      resident pages (page index, then dense values / string descriptors
 *      and a validity bitmap, or read in place when its pages are full and
 *      NULL-free);
 *   2. every comparison node is one kernel writing a u32 word bitmap (one
 *      thread per row, a ballot per 32 rows); AND / OR / NOT nodes combine
 *      word bitmaps, NOT over the table's rows only;
 *   3. the selected rows' ids are compacted in row order (per-word
 *      popcounts, a scan, then each word's set bits written at its offset);
 *   4. each projected column's pages are written by the result page writers
 *      through those row ids, so the new table's pages are exactly
 *      ColumnInserter<T>'s.
 * Semantics kept from the reference: a comparison is false on NULL rows;
 * IS_NULL / IS_NOT_NULL read the validity bit; NOT flips every row (NULL
 * rows included); INT32 columns compare with the literal's low 32 bits
 * (static_cast<int32_t>); VARCHAR compares bytewise as std::string_view;
 * LIKE matches the whole string with '%' = any run of code points and '_' =
 * one code point, neither matching a newline (the RE2 pattern of
 * Comparison::like_match).
 */
#include <algorithm>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

#include "cj_device.cuh"
#include "engine.h"
#include "exec_common.h"

namespace cj {
namespace {

constexpr int kFilterThreads = 256;

/* A VARCHAR value's bytes, short or spread over a long-string page chain. */
struct StrView {
    const uint8_t *pages;
    const uint8_t *p = nullptr; /* short string: its bytes */
    uint32_t len = 0;
    /* long string: chain walking cursor */
    uint64_t first = 0, chain = 0;
    uint64_t cur_page = 0, cur_start = 0;
    uint32_t cur_count = 0;
    bool is_long = false;

    CJ_DEV static uint32_t page_count(const uint8_t *page) { return *reinterpret_cast<const uint16_t *>(page + 2); }

    CJ_DEV void init(const uint8_t *pg, uint64_t desc) {
        pages = pg;
        if (!desc_is_long(desc)) {
            p = pg + desc_pos(desc);
            len = desc_len(desc);
            return;
        }
        is_long = true;
        first = desc_pos(desc);
        chain = desc_len(desc);
        uint64_t total = 0;
        for (uint64_t k = 0; k < chain; ++k) total += page_count(pg + (first + k) * kPageSize);
        len = (uint32_t)total;
        cur_page = 0;
        cur_start = 0;
        cur_count = page_count(pg + first * kPageSize);
    }
    CJ_DEV uint32_t skip_to(uint32_t i, uint32_t, uint32_t) { return i; }
    CJ_DEV uint8_t at(uint32_t i) {
        if (!is_long) return p[i];
        while (i >= cur_start + cur_count && cur_page + 1 < chain) {
            cur_start += cur_count;
            ++cur_page;
            cur_count = page_count(pages + (first + cur_page) * kPageSize);
        }
        while (i < cur_start && cur_page > 0) {
            --cur_page;
            cur_count = page_count(pages + (first + cur_page) * kPageSize);
            cur_start -= cur_count;
        }
        return pages[(first + cur_page) * kPageSize + 4 + (i - cur_start)];
    }
};

/* A short string read forwards and back by bytes: the aligned word around
 * the last byte stays in a register, so a string costs a load per four
 * characters, not one per character looked at (32 lanes' bytes are 32
 * sectors). */
struct ShortStr {
    const uint8_t *p;
    uint32_t len;
    uintptr_t at_word = 0;
    uint32_t word = 0;
    CJ_DEV ShortStr(const uint8_t *pg, uint64_t desc) : p(pg + desc_pos(desc)), len(desc_len(desc)) {}
    CJ_DEV uint32_t aligned(uintptr_t w) {
        if (w != at_word) {
            at_word = w;
            word = __ldg(reinterpret_cast<const uint32_t *>(w));
        }
        return word;
    }
    CJ_DEV uint8_t at(uint32_t i) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p) + i;
        return (uint8_t)(aligned(a & ~(uintptr_t)3) >> (8 * (uint32_t)(a & 3u)));
    }
    /* The first position from i on that a search for byte c followed by byte
     * c2 (256: any, or none) has to look at: skips four positions at once
     * whose characters are ASCII (code points of their own), no newline, and
     * do not begin with c and c2. */
    CJ_DEV uint32_t skip_to(uint32_t i, uint32_t c, uint32_t c2) {
        if (i >= len) return i;
        const uint32_t cc = (c & 0xFFu) * 0x01010101u, cc2 = (c2 & 0xFFu) * 0x01010101u, nl = 0x0A0A0A0Au;
        if (i + 5 <= len) {
            /* one aligned word a step, the same turns for every lane */
            const uintptr_t a = reinterpret_cast<uintptr_t>(p) + i;
            const uint32_t *next = reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3);
            const uint32_t sh = 8 * (uint32_t)(a & 3u);
            uint32_t lo = __ldg(next);
            do {
                const uint32_t hi = __ldg(++next); /* holds byte i + 4 at least */
                const unsigned long long both = ((unsigned long long)hi << 32 | lo) >> sh;
                const uint32_t w = (uint32_t)both, x = w ^ nl;
                /* a zero byte of x (or, of both keys' differences, below), or
                 * a byte above 0x7F */
                uint32_t stop = ((x - 0x01010101u) & ~x) | w;
                if (c < 256) {
                    uint32_t y = w ^ cc;
                    if (c2 < 256) y |= (uint32_t)(both >> 8) ^ cc2;
                    stop |= (y - 0x01010101u) & ~y;
                }
                if (stop & 0x80808080u) return i;
                i += 4;
                lo = hi;
            } while (i + 5 <= len);
        }
        if (i >= len) return i;
        /* the last one to four positions; the second byte has one fewer */
        const uint32_t r = len - i, live = 0x80808080u >> (8 * (4 - r));
        const uint32_t w = tail(i), x = w ^ nl;
        uint32_t stop = (((x - 0x01010101u) & ~x) | w) & live;
        if (c < 256) {
            uint32_t y = w ^ cc, yl = live;
            if (c2 < 256) {
                y |= (w >> 8) ^ cc2;
                yl >>= 8;
            }
            stop |= (y - 0x01010101u) & ~y & yl;
        }
        return stop ? i : len;
    }
    /* The string's last bytes from i on, one to four; what follows them in
     * the word is anything. */
    CJ_DEV uint32_t tail(uint32_t i) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(p) + i, w = a & ~(uintptr_t)3;
        const uint32_t lo = aligned(w);
        const uint32_t hi = w + 4 < reinterpret_cast<uintptr_t>(p) + len ? aligned(w + 4) : 0u;
        return __funnelshift_r(lo, hi, 8 * (uint32_t)(a & 3u));
    }
};

/* Three-way bytewise comparison with the literal (std::string_view order). */
template <class S> CJ_DEV int str_compare(S &s, const uint8_t *lit, uint32_t lit_len) {
    const uint32_t m = s.len < lit_len ? s.len : lit_len;
    for (uint32_t i = 0; i < m; ++i) {
        const uint8_t a = s.at(i), b = lit[i];
        if (a != b) return a < b ? -1 : 1;
    }
    return s.len < lit_len ? -1 : (s.len > lit_len ? 1 : 0);
}

/* Bytes of the UTF-8 code point that starts with byte b (1 for bytes that
 * cannot start one). */
CJ_DEV uint32_t cp_len(uint8_t b) {
    if (b < 0x80) return 1;
    if ((b & 0xE0) == 0xC0) return 2;
    if ((b & 0xF0) == 0xE0) return 3;
    if ((b & 0xF8) == 0xF0) return 4;
    return 1;
}

/* Whole-string LIKE: '%' matches any run of code points and '_' one code
 * point, neither a newline; other pattern bytes match themselves. Greedy
 * with backtracking to the last '%': each '%' extends one code point at a
 * time and never over a newline.
 *
 * Bound by instructions: the lanes of a warp take different turns at every
 * byte (5.6 of 32 active over 10M strings of 20 characters against '%qz%':
 * 1766 us). So after a '%' the lanes skip together, four positions a step,
 * what cannot begin the two bytes that follow it (with one byte a lane of
 * the 32 stopped at nearly every step: 1226 us), the pattern's bytes at j
 * and after the last '%' stay in registers, and a string too short for the
 * rest of the pattern is given up at once: 407 us. */
template <class S> CJ_DEV bool like_match(S &s, const uint8_t *pat, uint32_t m) {
    constexpr uint32_t kEnd = 256; /* past the pattern's last byte */
    const uint32_t n = s.len;
    uint32_t need = 0; /* bytes that the pattern from j on takes at least */
    for (uint32_t k = 0; k < m; ++k) need += pat[k] != '%';
    if (n < need) return false;
    uint32_t i = 0, j = 0, pc = m ? pat[0] : kEnd;
    /* the position after the last '%', its byte and, where both are literal,
     * the next one */
    uint32_t star_j = 0, star_i = 0, star_pc = 0, star_next = kEnd, star_need = 0;
    bool star = false;
    while (i < n) {
        if (pc == '%') {
            star = true;
            star_j = ++j;
            star_i = i;
            star_need = need;
            star_pc = pc = j < m ? pat[j] : kEnd;
            star_next = pc != kEnd && j + 1 < m ? pat[j + 1] : kEnd;
            if (star_next == '%' || star_next == '_') star_next = kEnd;
            if (pc != '%' && pc != '_') i = star_i = s.skip_to(star_i, star_pc, star_next);
            continue;
        }
        const uint8_t c = s.at(i);
        if (pc == '_' ? c != '\n' : pc == c) {
            i += pc == '_' ? cp_len(c) : 1u;
            ++j;
            --need;
            pc = j < m ? pat[j] : kEnd;
            continue;
        }
        if (!star) return false;
        const uint8_t sc = i == star_i ? c : s.at(star_i);
        if (sc == '\n') return false;
        star_i += cp_len(sc);
        if (star_i + star_need > n) return false;
        if (star_pc != '_') star_i = s.skip_to(star_i, star_pc, star_next);
        i = star_i;
        j = star_j;
        pc = star_pc;
        need = star_need;
    }
    while (j < m && pat[j] == '%') ++j;
    return j == m && i == n;
}

struct CmpArgs {
    ColView col;
    uint64_t rows;
    int32_t op;
    int64_t i64;
    double f64;
    const uint8_t *lit;
    uint32_t lit_len;
    uint32_t *out; /* word bitmap */
};

template <typename T> CJ_DEV bool cmp_num(int op, T a, T b) {
    switch (op) {
    case CJ_CMP_EQ: return a == b;
    case CJ_CMP_NEQ: return a != b;
    case CJ_CMP_LT: return a < b;
    case CJ_CMP_GT: return a > b;
    case CJ_CMP_LEQ: return a <= b;
    case CJ_CMP_GEQ: return a >= b;
    default: return false;
    }
}

template <class S> CJ_DEV bool cmp_str(S &s, const CmpArgs &a) {
    if (a.op == CJ_CMP_LIKE) return like_match(s, a.lit, a.lit_len);
    if (a.op == CJ_CMP_NOT_LIKE) return !like_match(s, a.lit, a.lit_len);
    return cmp_num<int>(a.op, str_compare(s, a.lit, a.lit_len), 0);
}

/* Value of base row r of a fixed-width column and whether it is present. */
template <typename T> CJ_DEV bool fixed_value(const ColView &c, uint32_t r, T *v) {
    if (col_direct(c)) {
        *v = page_value<T>(c.pages, r);
        return true;
    }
    if (!valid_bit(c.valid, r)) return false;
    *v = __ldg(reinterpret_cast<const T *>(c.values) + r);
    return true;
}

CJ_DEV bool row_valid(const ColView &c, uint32_t r) { return col_direct(c) || valid_bit(c.valid, r); }

__global__ void __launch_bounds__(kFilterThreads) k_compare(CmpArgs a) {
    const ColView c = resolve_view(a.col);
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < a.rows; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        bool bit = false;
        if (i < a.rows) {
            const uint32_t r = (uint32_t)i;
            if (a.op == CJ_CMP_IS_NULL) {
                bit = !row_valid(c, r);
            } else if (a.op == CJ_CMP_IS_NOT_NULL) {
                bit = row_valid(c, r);
            } else if (c.type == CJ_INT32) {
                int32_t v;
                bit = fixed_value<int32_t>(c, r, &v) && cmp_num<int32_t>(a.op, v, (int32_t)a.i64);
            } else if (c.type == CJ_INT64) {
                long long v;
                bit = fixed_value<long long>(c, r, &v) && cmp_num<long long>(a.op, v, (long long)a.i64);
            } else if (c.type == CJ_FP64) {
                double v;
                bit = fixed_value<double>(c, r, &v) && cmp_num<double>(a.op, v, a.f64);
            }
        }
        const uint32_t w = __ballot_sync(0xffffffffu, bit);
        if (lane_id() == 0 && base + threadIdx.x < a.rows) a.out[(base + threadIdx.x) >> 5] = w;
    }
}

/* A VARCHAR column compared with the literal, for the rows whose bit of `mask`
 * is set (null: all); the bits of other rows are 0. A block takes 32 kTake
 * rows at a time (2,048, or fewer in a table too small to fill the chip with
 * such blocks: text_words), packs those that are non-NULL and in the mask, and
 * its threads compare them side by side: a comparison costs tens of
 * instructions a character step for the whole warp however few of its rows are
 * still in question. 10M strings of 20 characters against '%qz%' beside two conditions
 * that leave a quarter of the rows: the filter 1006 us, 715 so. */
constexpr uint32_t kTextWords = 64;
template <uint32_t kTake>
__global__ void __launch_bounds__(kFilterThreads) k_compare_text(CmpArgs a, const uint32_t *__restrict__ mask) {
    static_assert(kFilterThreads == kTextWords * 4, "a thread lists a byte of the words");
    __shared__ uint32_t s_live[kTextWords], s_pre[kTextWords], s_out[kTextWords];
    __shared__ uint16_t s_row[kTextWords * 32];
    __shared__ uint32_t s_total;
    const ColView c = resolve_view(a.col);
    const uint64_t words = (a.rows + 31) / 32;
    for (uint64_t w0 = (uint64_t)blockIdx.x * kTake; w0 < words; w0 += (uint64_t)gridDim.x * kTake) {
        if (threadIdx.x < 32) {
            uint32_t v[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint64_t w = w0 + 2 * threadIdx.x + j;
                v[j] = 0;
                if (w >= words || (kTake < kTextWords && 2 * threadIdx.x + j >= kTake)) continue;
                v[j] = __ldg(c.valid + w); /* no bits past the last row */
                if (mask) v[j] &= __ldg(mask + w);
            }
            const uint32_t n0 = __popc(v[0]), n = n0 + __popc(v[1]);
            const uint32_t incl = warp_inclusive_scan(n);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                s_live[2 * threadIdx.x + j] = v[j];
                s_pre[2 * threadIdx.x + j] = incl - n + (j ? n0 : 0u);
                s_out[2 * threadIdx.x + j] = 0;
            }
            if (threadIdx.x == 31) s_total = incl;
        }
        __syncthreads();
        {
            const uint32_t w = threadIdx.x >> 2, b0 = (threadIdx.x & 3u) * 8, live = s_live[w];
            uint32_t at = s_pre[w] + __popc(live & ((1u << b0) - 1u));
            for (uint32_t bits = (live >> b0) & 0xFFu; bits; bits &= bits - 1)
                s_row[at++] = (uint16_t)(w * 32 + b0 + __ffs(bits) - 1);
        }
        __syncthreads();
        const uint32_t total = s_total;
        for (uint32_t k = threadIdx.x; k < total; k += kFilterThreads) {
            const uint32_t q = s_row[k];
            const uint64_t d = __ldg(c.str_desc + w0 * 32 + q);
            bool bit;
            if (desc_is_long(d)) {
                StrView s;
                s.init(c.pages, d);
                bit = cmp_str(s, a);
            } else {
                ShortStr s(c.pages, d);
                bit = cmp_str(s, a);
            }
            if (bit) atomicOr(&s_out[q >> 5], 1u << (q & 31u));
        }
        __syncthreads();
        if (threadIdx.x < kTake && w0 + threadIdx.x < words) a.out[w0 + threadIdx.x] = s_out[threadIdx.x];
        __syncthreads();
    }
}

/* out = a op b over `words` words; NOT (b null) keeps only rows < rows. */
__global__ void k_bitmap_logic(const uint32_t *a, const uint32_t *b, uint32_t *out, uint64_t words, uint64_t rows,
                               int kind) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < words; w += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t v;
        if (kind == CJ_PRED_AND) v = a[w] & b[w];
        else if (kind == CJ_PRED_OR) v = a[w] | b[w];
        else {
            v = ~a[w];
            const uint64_t lo = w * 32;
            if (lo + 32 > rows) v &= (rows > lo) ? ((1u << (rows - lo)) - 1u) : 0u;
        }
        out[w] = v;
    }
}

__global__ void k_word_popc(const uint32_t *words, uint64_t n, uint32_t *cnt) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (uint64_t)gridDim.x * blockDim.x)
        cnt[w] = __popc(words[w]);
}

/* Row ids of the set bits, in row order: word w's rows go to off[w]... */
__global__ void k_word_emit(const uint32_t *words, const uint64_t *off, uint64_t n, uint32_t *rids) {
    for (uint64_t w = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t v = words[w];
        uint64_t o = off[w];
        while (v) {
            const int b = __ffs(v) - 1;
            rids[o++] = (uint32_t)(w * 32 + b);
            v &= v - 1;
        }
    }
}

unsigned grid_for(const Context &ctx, uint64_t n, unsigned threads) {
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((n + threads - 1) / threads, (uint64_t)ctx.num_sms * 8));
}

/* Words of rows that a block of k_compare_text takes at a time: halved until
 * the blocks fill the chip, down to a row a thread. 200,000 strings against
 * '%_a_%' (where LIKE cannot skip): the filter 344 us with 64 words, 187
 * with 8; 1,000 strings 209 and 131. */
uint32_t text_words(const Context &ctx, uint64_t words) {
    static_assert(kTextWords == 64 && kFilterThreads == 256, "the kernels of 8 to 64 words");
    uint32_t take = kTextWords;
    while (take > kFilterThreads / 32 && words / take < (uint64_t)ctx.num_sms * 8) take /= 2;
    return take;
}

class Filter {
  public:
    Filter(Context &c, const cj_table &t, const cj_predicate *p) : ctx(c), in(t), pred(p), L(c.launch()) {}

    cj_table *run(uint64_t ncols, const uint64_t *cols, uint64_t *num_rows) {
        validate(ncols, cols);
        const uint64_t rows = in.num_rows;
        if (rows > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "table exceeds 2^32-1 rows");
        const uint64_t words = std::max<uint64_t>((rows + 31) / 32, 1);
        DevPtr sel;
        uint64_t count = rows;
        if (pred && rows) {
            decode(pred_columns());
            DevPtr bits = eval(pred->root, words, 0, nullptr);
            DevPtr cnt = ctx.alloc(words * 4), off = ctx.alloc((words + 1) * 8);
            DevPtr tmp = ctx.alloc(scan_temp_bytes(words));
            k_word_popc<<<grid_for(ctx, words, 256), 256, 0, ctx.stream>>>(bits->as<uint32_t>(), words,
                                                                             cnt->as<uint32_t>());
            count_launches(1);
            check_cuda(cudaGetLastError(), "popc");
            check_cuda(scan_u32_to_u64(L, cnt->as<uint32_t>(), off->as<uint64_t>(), words, tmp->ptr), "scan");
            /* the count goes back with the status block (sync_status copies
             * all of it to the host) */
            check_cuda(cudaMemcpyAsync(&ctx.d_status->aux, off->as<uint64_t>() + words, 8,
                                       cudaMemcpyDeviceToDevice, ctx.stream),
                       "copy");
            ctx.sync_status();
            count = ctx.h_status->aux;
            sel = ctx.alloc(std::max<uint64_t>(count, 1) * 4);
            k_word_emit<<<grid_for(ctx, words, 256), 256, 0, ctx.stream>>>(bits->as<uint32_t>(), off->as<uint64_t>(),
                                                                             words, sel->as<uint32_t>());
            count_launches(1);
            check_cuda(cudaGetLastError(), "emit");
        }
        auto tab = std::make_unique<cj_table>();
        tab->ctx = &ctx;
        tab->num_rows = count;
        const uint32_t TR = 2048;
        if (count) decode(std::set<uint64_t>(cols, cols + ncols));
        for (uint64_t k = 0; k < ncols; ++k) {
            const uint64_t c = cols[k];
            ColumnPages cp;
            cp.type = in.cols[c].type;
            if (count) {
                ColView v = view(c);
                v.rid_a = sel ? sel->as<uint32_t>() : nullptr;
                if (cp.type != CJ_VARCHAR) {
                    const uint32_t R = rows_per_page_fixed(cp.type);
                    cp.num_pages = (count + R - 1) / R;
                    cp.owner = ctx.alloc(cp.num_pages * kPageSize);
                    PageTask pt{};
                    pt.col = v;
                    pt.rows = count;
                    pt.out = cp.owner->as<uint8_t>();
                    check_cuda(launch_write_pages(L, &pt, 1), "write_pages");
                } else {
                    DevPtr temp = ctx.alloc(varchar_temp_bytes(count, TR)), done = ctx.alloc(4);
                    check_cuda(cudaMemsetAsync(done->ptr, 0, 4, ctx.stream), "memset");
                    VarcharTask vt{};
                    vt.col = v;
                    vt.rows = count;
                    vt.done = done->as<unsigned int>();
                    vt.total_pages = &ctx.d_status->aux;
                    place_varchar(vt, TR, temp->ptr);
                    check_cuda(launch_varchar(L, &vt, 1, true), "varchar_plan");
                    ctx.sync_status(); /* brings the page count back in aux */
                    cp.num_pages = ctx.h_status->aux;
                    cp.owner = ctx.alloc(cp.num_pages * kPageSize);
                    vt.out = cp.owner->as<uint8_t>();
                    check_cuda(launch_varchar(L, &vt, 1, false), "varchar_write");
                }
                cp.dev = cp.owner->as<uint8_t>();
            }
            tab->cols.push_back(std::move(cp));
        }
        ctx.sync_status();
        if (num_rows) *num_rows = count;
        return tab.release();
    }

  private:
    Context &ctx;
    const cj_table &in;
    const cj_predicate *pred;
    Launch L;
    std::map<uint64_t, Decoded> decoded;
    std::vector<DevPtr> keep;
    std::vector<int8_t> text_of; /* has_text, by node; -1 not known yet */

    void validate(uint64_t ncols, const uint64_t *cols) {
        if (ncols && !cols) fail(CJ_ERR_INVALID_ARGUMENT, "null column list");
        for (uint64_t k = 0; k < ncols; ++k)
            if (cols[k] >= in.cols.size()) fail(CJ_ERR_INVALID_PLAN, "projected column out of range");
        if (!pred) return;
        if (!pred->nodes || pred->root >= pred->num_nodes) fail(CJ_ERR_INVALID_PLAN, "bad predicate root");
        for (uint64_t i = 0; i < pred->num_nodes; ++i) {
            const cj_pred_node &n = pred->nodes[i];
            if (n.kind == CJ_PRED_CMP) {
                if (n.column >= in.cols.size()) fail(CJ_ERR_INVALID_PLAN, "predicate column out of range");
                if (n.op < CJ_CMP_EQ || n.op > CJ_CMP_IS_NOT_NULL) fail(CJ_ERR_INVALID_PLAN, "unknown comparison");
                if (n.op == CJ_CMP_IS_NULL || n.op == CJ_CMP_IS_NOT_NULL) continue;
                const int32_t t = in.cols[n.column].type;
                const bool like = n.op == CJ_CMP_LIKE || n.op == CJ_CMP_NOT_LIKE;
                if (t == CJ_VARCHAR) {
                    if (n.literal_type != CJ_VARCHAR || (n.str_len && !n.str))
                        fail(CJ_ERR_INVALID_PLAN, "VARCHAR column compared with a non-string literal");
                    if (n.str_len > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "literal too long");
                } else if (like || n.literal_type == CJ_VARCHAR || (t != CJ_FP64 && n.literal_type != CJ_INT64)) {
                    fail(CJ_ERR_INVALID_PLAN, "comparison literal does not fit the column's type");
                }
            } else if (n.kind == CJ_PRED_AND || n.kind == CJ_PRED_OR) {
                if (n.left >= pred->num_nodes || n.right >= pred->num_nodes)
                    fail(CJ_ERR_INVALID_PLAN, "predicate child out of range");
            } else if (n.kind == CJ_PRED_NOT) {
                if (n.left >= pred->num_nodes) fail(CJ_ERR_INVALID_PLAN, "predicate child out of range");
            } else {
                fail(CJ_ERR_INVALID_PLAN, "unknown predicate node");
            }
        }
    }

    /* The columns that the predicate reads. */
    std::set<uint64_t> pred_columns() const {
        std::set<uint64_t> need;
        std::function<void(uint64_t, int)> walk = [&](uint64_t node, int depth) {
            if (depth > (int)pred->num_nodes) fail(CJ_ERR_INVALID_PLAN, "predicate has a cycle");
            const cj_pred_node &n = pred->nodes[node];
            if (n.kind == CJ_PRED_CMP) {
                need.insert(n.column);
                return;
            }
            walk(n.left, depth + 1);
            if (n.kind != CJ_PRED_NOT) walk(n.right, depth + 1);
        };
        walk(pred->root, 0);
        return need;
    }
    /* Indexes and decodes columns, one launch each for all of them. */
    void decode(const std::set<uint64_t> &need) {
        std::vector<ColumnTask> tasks;
        Slab slab;
        for (uint64_t c : need) {
            if (decoded.count(c)) continue;
            Decoded d;
            d.type = in.cols[c].type;
            d.rows = in.num_rows;
            d.src = in.cols[c];
            d.reserve(slab);
            slab.reserve(sizeof(ColumnState));
        }
        if (!slab.size) return;
        slab.open(ctx);
        keep.push_back(slab.mem);
        for (uint64_t c : need) {
            if (decoded.count(c)) continue;
            Decoded d;
            d.type = in.cols[c].type;
            d.rows = in.num_rows;
            d.src = in.cols[c];
            ColumnState *state = slab.take_as<ColumnState>(sizeof(ColumnState));
            check_cuda(cudaMemsetAsync(state, 0, sizeof(ColumnState), ctx.stream), "memset");
            tasks.push_back(column_task(d, slab, state, &ctx.d_status->errors));
            decoded.emplace(c, std::move(d));
        }
        if (tasks.empty()) return;
        check_cuda(launch_columns(L, tasks.data(), tasks.size(), true), "page_index");
        check_cuda(launch_columns(L, tasks.data(), tasks.size(), false), "decode");
    }

    ColView view(uint64_t c) {
        const Decoded &d = decoded.at(c);
        Relation R;
        RelCol rc{d.type, 0, c, -1, false};
        return make_view(d, R, rc, nullptr);
    }

    /* Whether a node's subtree compares text (worked out once a node). */
    bool has_text(uint64_t node, int depth) {
        if (depth > (int)pred->num_nodes) fail(CJ_ERR_INVALID_PLAN, "predicate has a cycle");
        text_of.resize(pred->num_nodes, -1);
        if (text_of[node] < 0) {
            const cj_pred_node &n = pred->nodes[node];
            bool t;
            if (n.kind == CJ_PRED_CMP)
                t = in.cols[n.column].type == CJ_VARCHAR && n.op != CJ_CMP_IS_NULL && n.op != CJ_CMP_IS_NOT_NULL;
            else t = has_text(n.left, depth + 1) || (n.kind != CJ_PRED_NOT && has_text(n.right, depth + 1));
            text_of[node] = t;
        }
        return text_of[node];
    }

    /* The node's bit for the rows whose bit of `mask` is set (null: all); the
     * other rows' bits are anything. Text is compared last: of the children
     * of an AND the one without text comes first, and the second is asked for
     * the rows that the first lets through only. */
    DevPtr eval(uint64_t node, uint64_t words, int depth, const uint32_t *mask) {
        if (depth > (int)pred->num_nodes) fail(CJ_ERR_INVALID_PLAN, "predicate has a cycle");
        const cj_pred_node &n = pred->nodes[node];
        DevPtr out = ctx.alloc(words * 4);
        if (n.kind == CJ_PRED_CMP) {
            CmpArgs a{};
            a.col = view(n.column);
            a.rows = in.num_rows;
            a.op = n.op;
            a.i64 = n.i64;
            a.f64 = n.literal_type == CJ_INT64 ? (double)n.i64 : n.f64;
            a.out = out->as<uint32_t>();
            const bool text = has_text(node, depth);
            if (text) {
                DevPtr lit = ctx.alloc(std::max<uint64_t>(n.str_len, 1));
                if (n.str_len)
                    check_cuda(cudaMemcpyAsync(lit->ptr, n.str, n.str_len, cudaMemcpyHostToDevice, ctx.stream),
                               "literal");
                a.lit = lit->as<uint8_t>();
                a.lit_len = (uint32_t)n.str_len;
                keep.push_back(lit);
            }
            const uint32_t take = text_words(ctx, words);
            const unsigned grid = grid_for(ctx, in.num_rows, text ? take * 32 : kFilterThreads);
            const auto compare_text = take == 64   ? k_compare_text<64>
                                      : take == 32 ? k_compare_text<32>
                                      : take == 16 ? k_compare_text<16>
                                                   : k_compare_text<8>;
            if (text) compare_text<<<grid, kFilterThreads, 0, ctx.stream>>>(a, mask);
            else k_compare<<<grid, kFilterThreads, 0, ctx.stream>>>(a);
            count_launches(1);
            check_cuda(cudaGetLastError(), "compare");
        } else {
            const bool swap = n.kind == CJ_PRED_AND && has_text(n.left, depth + 1) && !has_text(n.right, depth + 1);
            DevPtr l = eval(swap ? n.right : n.left, words, depth + 1, mask);
            DevPtr r;
            if (n.kind != CJ_PRED_NOT)
                r = eval(swap ? n.left : n.right, words, depth + 1, n.kind == CJ_PRED_AND ? l->as<uint32_t>() : mask);
            k_bitmap_logic<<<grid_for(ctx, words, 256), 256, 0, ctx.stream>>>(
                l->as<uint32_t>(), r ? r->as<uint32_t>() : nullptr, out->as<uint32_t>(), words, in.num_rows, n.kind);
            count_launches(1);
            check_cuda(cudaGetLastError(), "bitmap logic");
        }
        return out;
    }
};

} // namespace

cj_table *filter_table(Context &ctx, const cj_table &in, const cj_predicate *pred, uint64_t ncols,
                       const uint64_t *cols, uint64_t *num_rows) {
    Filter f(ctx, in, pred);
    return f.run(ncols, cols, num_rows);
}

} // namespace cj

extern "C" int cj_table_filter(cj_context *ctx, const cj_table *in, const cj_predicate *pred, uint64_t num_columns,
                               const uint64_t *columns, cj_table **out, uint64_t *num_rows) {
    if (!ctx || !in || !out) return cj::set_last_error(CJ_ERR_INVALID_ARGUMENT, "null argument");
    *out = nullptr;
    if (in->ctx != ctx && in->ctx->device != ctx->device)
        return cj::set_last_error(CJ_ERR_INVALID_ARGUMENT, "table of another device");
    cudaSetDevice(ctx->device);
    try {
        *out = cj::filter_table(*ctx, *in, pred, num_columns, columns, num_rows);
    } catch (const cj::Error &e) {
        cudaStreamSynchronize(ctx->stream);
        cudaGetLastError();
        return cj::set_last_error(e.code, e.msg);
    } catch (const std::bad_alloc &) {
        return cj::set_last_error(CJ_ERR_OUT_OF_MEMORY, "host allocation failed");
    }
    cj::clear_last_error();
    return CJ_OK;
}
