/*
 * engine.cpp — plan executor: the depth-first join recursion of the
 * reference (src/execute.cpp:84-325) over device-resident relations.
 *
 * A relation is either a scan (rows are base-table rows) or the output of
 * a join. Join outputs are late-materialised: instead of copying values
 * (construct_intermediate.h:121-220) a join output keeps one u32 row-id
 * vector per contributing base table, and each of its columns names its
 * base column and the vector that reaches it. Values are read only by the
 * kernels that need them: join keys by build/probe, projected columns by
 * the root's page writers.
 */
#include <algorithm>
#include <chrono>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <string>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "engine.h"

#include "exec_common.h"

namespace cj {
namespace {

constexpr uint64_t kMultiSpan = 4; /* values of the range per build row */

/* Repeated keys that are not dense get their open-addressing table from 2.5
 * build rows per key on, else the hash table. A probe row without a match
 * costs the hash table's small kernel less, one with several the other's; with
 * their number known both make room for them and probe once. Random INT32
 * keys, 40 % of the probe rows' in the range but no build key, kernels' sums:
 * 48M x 3M rows, 1.1 a key, 1980 us on the open-addressing table and 1400 on
 * the hash table, two a key 2692 and 1737; all matching, 30M x 1M rows, two a
 * key 1513 and 1287, three 1760 and 2441; 2M x 2M rows, four a key 442 and
 * 471, 40 a key 1621 and 5103. */
constexpr uint64_t kOpenMultiMean2 = 5; /* twice that mean */
/* Probe rows from which the number of keys is estimated before that choice: 15
 * to 30 us and a synchronisation. With fewer, joins of kOpenMultiProbe probe
 * rows or more per build row take the open-addressing table, whose build
 * counts the keys (100K x 1M rows, three a key: 192 us, 204 with the estimate;
 * 300K x 20M rows of 1.1 a key 667 and 546), the others, for whom its dearer
 * build does not pay, the hash table (2M x 2M INT64 rows of 1.1 a key, all
 * matching: 392 us, 367 with the estimate and without a second run, half of
 * them 318 and 349; a five-join star whose last build side is an intermediate
 * of 86K rows against 105K probe rows 828 on the open-addressing table, 766). */
constexpr uint64_t kSampleFrom = 1ull << 22, kSampleFromFew = 1ull << 20;
constexpr uint64_t kOpenMultiProbe = 4;

/* A probe of an open-addressing table reads a build column's values beside
 * it while both stay in L2 (126 MB on two dies, each keeping its own copy of
 * what it reads); a larger pair is read one after the other, through the
 * match row ids: 64 MB of table and 33 MB of values 1513 us together, 1447
 * apart (64M probe rows). A direct-mapped table is 16 MB there. */
constexpr uint64_t kEmitBesideOpen = 48ull << 20;

/* Memory taken for matches that may not come is not asked about up to this
 * size (a query of the free memory takes tens of us). */
constexpr uint64_t kAmpleRoom = 4ull << 30;

/* A result keeps the buffer that its probe wrote, sized for the matches there
 * might have been, unless less than a quarter of it is used and kKeepSpare or
 * more is not: the pages then move to a buffer of their size (64 MB in 20 us). */
constexpr uint64_t kKeepSpare = 32ull << 20;

/* Pages of payload columns that a plan of several joins decodes before the
 * first: a launch less, under which the host prepares that join (a star's
 * 243 MB of them, five joins: 733 us, 747 with the payloads decoded at the root), but
 * for nothing when a join below the root is empty (256 MB: about 100 us). */
constexpr uint64_t kDecodeAhead = 256ull << 20;

/* Probe rows from which a probe of repeated keys gets room for an eighth more
 * than the mean number of matches. */
constexpr uint64_t kSpareEighth = 1ull << 15;

/* Room for matches from which the long runs among them are left to a kernel of
 * their own, where the build found a key with kRunFrom rows or more, and where
 * the host does not know. 240K matches in runs of 400 take 80 us less with it
 * (5K x 20K rows, the whole join 318 and 237 us); without any run its launch
 * and its list cost 5 to 10 us (1,000 x 300K rows over 750 dense keys 199 us,
 * 188 without). */
constexpr uint64_t kRunsFrom = 1ull << 16, kRunsFromBlind = 1ull << 20;

enum Phase { PH_UPLOAD, PH_DECODE, PH_BUILD, PH_PROBE, PH_NL, PH_INTER, PH_MAT, PH_DOWNLOAD, PH_COUNT };
/* NVTX range names of the phases (host-side ranges around the enqueueing of
 * each phase; visible in Nsight Systems timelines). */
constexpr const char *kPhaseNames[PH_COUNT] = {"cj:upload", "cj:decode",       "cj:build",       "cj:probe",
                                               "cj:nested_loop", "cj:intermediate", "cj:materialize",
                                               "cj:download"};

class Executor {
  public:
    Executor(Context &c, const cj_plan_desc &p, uint32_t f) : ctx(c), plan(p), flags(f), L(c.launch()) {}
    ~Executor() {
        /* Pages still being uploaded (an error came first) are freed on the
         * kernel stream: order those frees after the copies. */
        for (auto &kv : prefetched) {
            cudaStreamWaitEvent(ctx.stream, kv.second.done, 0);
            ctx.put_event(kv.second.done);
        }
        for (auto &pe : phase_events) {
            ctx.put_event(pe.a);
            ctx.put_event(pe.b);
        }
    }
    cj_result *run(cj_exec_stats *st);

  private:
    struct PhaseEv {
        int phase;
        cudaEvent_t a, b;
    };
    class PhaseScope {
      public:
        PhaseScope(Executor &e, int ph) : e_(e), ph_(ph) {
            nvtxRangePushA(kPhaseNames[ph]);
            a_ = e.ctx.get_event();
            cudaEventRecord(a_, e.ctx.stream);
        }
        ~PhaseScope() {
            cudaEvent_t b = e_.ctx.get_event();
            cudaEventRecord(b, e_.ctx.stream);
            e_.phase_events.push_back({ph_, a_, b});
            nvtxRangePop();
        }

      private:
        Executor &e_;
        int ph_;
        cudaEvent_t a_;
    };
    /* Per-kernel timing when profiling is on. */
    class KScope {
      public:
        KScope(Executor &e, const char *name) : e_(e) {
            if (!e.ctx.opt.profile_kernels) return;
            auto it = e.ctx.profile_index.find(name);
            if (it == e.ctx.profile_index.end()) {
                slot_ = e.ctx.profile.size();
                e.ctx.profile.push_back({name, 0, 0.0});
                e.ctx.profile_index[name] = slot_;
            } else {
                slot_ = it->second;
            }
            a_ = e.ctx.get_event();
            cudaEventRecord(a_, e.ctx.stream);
            on_ = true;
        }
        ~KScope() {
            if (!on_) return;
            cudaEvent_t b = e_.ctx.get_event();
            cudaEventRecord(b, e_.ctx.stream);
            e_.ctx.pending.push_back({slot_, a_, b});
        }

      private:
        Executor &e_;
        size_t slot_ = 0;
        cudaEvent_t a_ = nullptr;
        bool on_ = false;
    };

    Context &ctx;
    const cj_plan_desc &plan;
    uint32_t flags;
    Launch L;
    std::map<std::pair<uint64_t, uint64_t>, Decoded> decoded;
    /* Host columns whose pages are on their way on the upload stream. */
    struct Prefetched {
        ColumnPages pages;
        cudaEvent_t done = nullptr;
    };
    std::map<std::pair<uint64_t, uint64_t>, Prefetched> prefetched;
    std::vector<PhaseEv> phase_events;
    cj_exec_stats stats{};
    /* The match counter and table words of the status block are zero (they
     * are when a plan starts): nothing to clear before the first join. */
    bool join_words_clear = true;
    void clear_join_words() {
        ck(cudaMemsetAsync(&ctx.d_status->counter, 0, sizeof(ctx.d_status->counter) + sizeof(ctx.d_status->table),
                           ctx.stream),
           "memset");
    }
    uint64_t used_cols = 0;   /* columns of the status block the plan has read */
    bool synced_last = false; /* the last thing enqueued was a synchronisation */
    /* Brings the status block to the host, counting the synchronisation. */
    void sync() {
        ctx.sync_status(used_cols);
        stats.host_syncs++;
    }
    /* A buffer that the plan can do without: null when the memory is out. */
    DevPtr spare(uint64_t bytes) {
        try {
            return ctx.alloc(bytes);
        } catch (const Error &e) {
            if (e.code != CJ_ERR_OUT_OF_MEMORY) throw;
            return nullptr;
        }
    }

    /* `pages` itself, or a buffer of `bytes` that its first bytes move to
     * (kKeepSpare). */
    DevPtr fitted(const DevPtr &pages, uint64_t bytes) {
        if (!pages || bytes > pages->bytes / 4 || pages->bytes - bytes < kKeepSpare) return pages;
        DevPtr fit = spare(bytes);
        if (!fit) return pages;
        ck(cudaMemcpyAsync(fit->ptr, pages->ptr, bytes, cudaMemcpyDeviceToDevice, ctx.stream), "fit pages");
        return fit;
    }
    /* A result written with a device-side row count (materialize with
     * rows_dev): its rows and pages once the count is known. */
    void finish_counted(cj_result &r, uint64_t rows) {
        r.num_rows = rows;
        uint64_t pages = 0;
        bool moved = false;
        std::map<DevPtr, DevPtr> fit; /* columns may share a buffer */
        for (size_t c = 0; c < r.types.size(); ++c) {
            const uint32_t R = rows_per_page_fixed(r.types[c]);
            r.num_pages[c] = (rows + R - 1) / R;
            if (rows) {
                DevPtr &f = fit[r.dev_pages[c]];
                if (!f) f = fitted(r.dev_pages[c], r.num_pages[c] * kPageSize);
                moved |= f != r.dev_pages[c];
                r.dev_pages[c] = f;
            } else {
                r.dev_pages[c].reset();
            }
            pages += r.num_pages[c];
        }
        if (moved) ck(cudaStreamSynchronize(ctx.stream), "fit pages");
        stats.output_rows = rows;
        stats.output_pages = pages;
    }
    /* Whether `bytes` may be taken that the plan can do without: up to
     * kAmpleRoom, above that half of what is left. */
    bool ample(uint64_t bytes) {
        if (bytes <= kAmpleRoom) return true;
        size_t left = 0, total = 0;
        uint64_t used = 0, reserved = 0;
        ck(cudaMemGetInfo(&left, &total), "cudaMemGetInfo");
        ck(cudaMemPoolGetAttribute(ctx.pool, cudaMemPoolAttrUsedMemCurrent, &used), "pool attr");
        ck(cudaMemPoolGetAttribute(ctx.pool, cudaMemPoolAttrReservedMemCurrent, &reserved), "pool attr");
        std::lock_guard<std::mutex> g(ctx.dev_mu); /* frees of other threads touch the cache too */
        return bytes <= (left + (reserved - std::min(reserved, used)) + ctx.dev_cached) / 2;
    }
    /* The same for matches that may not come, under the context's own bound
     * where it has one. A selective join whose matches would fit does not
     * fail for room it would not have used. */
    bool room_for(uint64_t bytes) {
        return ctx.opt.spare_room >= 0 ? bytes <= (uint64_t)ctx.opt.spare_room : ample(bytes);
    }

    const cj_table *resident(uint64_t t) const { return resident_input(plan, t); }
    uint64_t table_rows(uint64_t t) const { return input_rows(plan, t); }
    int32_t column_type(uint64_t t, uint64_t c) const { return input_col_type(plan, t, c); }

    void validate();
    using TC = std::pair<uint64_t, uint64_t>;
    std::map<TC, ColumnPages> upload_small(const std::vector<TC> &order);
    void prefetch();
    void launch_tasks(std::vector<ColumnTask> &tasks, bool index);
    Decoded &indexed(uint64_t t, uint64_t c);
    Decoded &decode(uint64_t t, uint64_t c);
    void decode_all(const std::vector<TC> &cols);
    int streamed_key(std::pair<uint64_t, uint64_t> *col) const;
    Relation resolve(uint64_t node, int depth);
    Relation exec_join(uint64_t node, int depth, bool is_root, cj_result **out);
    ColView view(const Relation &R, const RelCol &c, const uint32_t *rid_a);
    /* An output column of the root: its relation column and the match row
     * ids that select its rows (null for a scan root). Decoded on use. */
    struct OutCol {
        const Relation *rel; /* null: the values are already in `pages` */
        RelCol col;
        const uint32_t *rid_a;
        DevPtr pages; /* result pages written by the probe (with `rel`: if
                         the column holds no NULL)                       */
        bool direct_only = false; /* ... and the table is direct-mapped */
    };
    ColView out_view(const OutCol &oc) { return view(*oc.rel, oc.col, oc.rid_a); }
    cj_result *materialize(const std::vector<OutCol> &cols, const std::vector<int32_t> &types, uint64_t rows,
                           const unsigned long long *rows_dev = nullptr);
    void ck(cudaError_t e, const char *what) { check_cuda(e, what); }
};

void Executor::validate() { validate_plan(ctx, plan); }

/* Host columns that together are small: their pages are gathered in one
 * staging buffer and go up in one copy on the kernel stream, so that they are
 * indexed and decoded like resident ones. Above kSmallUpload the gathering
 * costs more than it saves (copies straight from page-locked pages, each on
 * its way while kernels run, take over). Empty: the columns go one by one. */
std::map<Executor::TC, ColumnPages> Executor::upload_small(const std::vector<TC> &order) {
    constexpr uint64_t kSmallUpload = 1u << 20;
    uint64_t pages = 0;
    std::vector<TC> host;
    for (const TC &tc : order)
        if (!resident(tc.first)) {
            host.push_back(tc);
            pages += plan.inputs[tc.first].columns[tc.second].num_pages;
        }
    std::map<TC, ColumnPages> out;
    if (host.empty() || !pages || pages * kPageSize > std::min<uint64_t>(kSmallUpload, ctx.staging_bytes)) return out;
    PhaseScope ph(*this, PH_UPLOAD);
    DevPtr dev = ctx.alloc(pages * kPageSize);
    ck(cudaEventSynchronize(ctx.staging_ev[0]), "staging wait");
    uint8_t *to = static_cast<uint8_t *>(ctx.staging[0]);
    uint64_t at = 0;
    for (const TC &tc : host) {
        const cj_column_desc &cd = plan.inputs[tc.first].columns[tc.second];
        ColumnPages cp;
        cp.type = cd.type;
        cp.num_pages = cd.num_pages;
        if (cd.num_pages && !cd.pages) fail(CJ_ERR_INVALID_ARGUMENT, "column has pages but no page array");
        if (cd.num_pages) {
            cp.owner = dev;
            cp.dev = dev->as<uint8_t>() + at * kPageSize;
        }
        for (uint64_t k = 0; k < cd.num_pages; ++k, ++at) {
            if (!cd.pages[k]) fail(CJ_ERR_INVALID_ARGUMENT, "null page pointer");
            std::memcpy(to + at * kPageSize, cd.pages[k], kPageSize);
        }
        out.emplace(tc, std::move(cp));
    }
    ck(cudaMemcpyAsync(dev->ptr, to, pages * kPageSize, cudaMemcpyHostToDevice, ctx.stream), "page upload");
    ck(cudaEventRecord(ctx.staging_ev[0], ctx.stream), "event record");
    stats.h2d_bytes += pages * kPageSize;
    return out;
}

/* Starts the upload of every host column the plan will decode, on the
 * context's upload stream, in the order the kernels need them: join keys
 * bottom-up, then the root's outputs. The kernel stream waits for a
 * column's copy only when it decodes that column, so later columns (the
 * payloads) cross PCIe while the joins below the root run.
 *
 * The resident columns among them are indexed here in one launch, and those
 * that the plan is sure to read decoded in another (per column those were two
 * to three launches and two memsets: 212 us of a six-table plan's 1.9 ms):
 * all of a plan of one join, the join keys of a larger one, whose other
 * columns wait for the root (decode_all), since a join below may come out
 * empty; none when a table is empty. (40M probe rows with two payloads that
 * hold NULLs: an empty build side 28 us, 504 with everything decoded; an empty
 * first join of two 358 and 644.) Each column keeps its errors to itself
 * until the plan reads it: a plan that never gets to a malformed column still
 * runs. */
void Executor::prefetch() {
    std::vector<TC> order;
    std::set<TC> seen, keys;
    bool empty = false; /* a table without rows: every join above it is empty too */
    uint64_t joins = 0, ahead = 0; /* pages that are decoded for nothing when a join comes out empty */
    auto add = [&](const TC &tc) {
        if (seen.insert(tc).second) order.push_back(tc);
    };
    std::function<std::vector<TC>(uint64_t, int)> cols = [&](uint64_t node, int depth) -> std::vector<TC> {
        if (depth > (int)plan.num_nodes) fail(CJ_ERR_INVALID_PLAN, "plan has a cycle");
        const cj_plan_node &n = plan.nodes[node];
        std::vector<TC> out;
        if (n.node_type == CJ_NODE_SCAN) {
            empty |= table_rows(n.base_table_id) == 0;
            for (uint64_t a = 0; a < n.num_output_attrs; ++a) out.push_back({n.base_table_id, n.output_attrs[a].index});
            return out;
        }
        ++joins;
        std::vector<TC> both = cols(n.left, depth + 1);
        const std::vector<TC> r = cols(n.right, depth + 1);
        auto add_key = [&](const TC &tc) {
            add(tc);
            keys.insert(tc);
        };
        if (n.left_attr < both.size()) add_key(both[n.left_attr]);
        if (n.right_attr < r.size()) add_key(r[n.right_attr]);
        both.insert(both.end(), r.begin(), r.end());
        for (uint64_t a = 0; a < n.num_output_attrs; ++a)
            if (n.output_attrs[a].index < both.size()) out.push_back(both[n.output_attrs[a].index]);
        return out;
    };
    for (const TC &tc : cols(plan.root, 0)) add(tc);
    ck(cudaMemsetAsync(ctx.d_status, 0, sizeof(StatusBlock), ctx.stream), "memset");
    std::map<TC, ColumnPages> small = upload_small(order);
    std::vector<std::pair<TC, Decoded>> now;
    Slab slab;
    for (const TC &tc : order) {
        const cj_table *r = resident(tc.first);
        const auto up = small.find(tc);
        if (empty || (!r && up == small.end()) || table_rows(tc.first) > 0xFFFFFFFFull || now.size() == kStatusColumns)
            continue;
        Decoded d;
        d.type = column_type(tc.first, tc.second);
        d.rows = table_rows(tc.first);
        d.src = r ? r->cols[tc.second] : up->second;
        d.status_col = (int)now.size();
        d.reserve(slab);
        if (joins > 1 && !keys.count(tc)) ahead += d.src.num_pages * kPageSize;
        now.emplace_back(tc, std::move(d));
    }
    if (!now.empty()) {
        std::vector<ColumnTask> tasks, decodes;
        TC streamed;
        const bool stream = streamed_key(&streamed);
        slab.open(ctx);
        for (auto &kv : now) {
            Decoded &d = kv.second;
            d.mem = slab.mem;
            ColumnState *state = &ctx.d_status->cols[d.status_col];
            tasks.push_back(column_task(d, slab, state, &state->err));
            d.ready = !(stream && kv.first == streamed) && (ahead <= kDecodeAhead || keys.count(kv.first));
            if (d.ready) decodes.push_back(tasks.back());
            decoded.emplace(kv.first, std::move(d));
        }
        PhaseScope ph(*this, PH_DECODE);
        launch_tasks(tasks, true);
        if (!decodes.empty()) launch_tasks(decodes, false);
    }
    cudaEvent_t first = nullptr;
    for (const TC &tc : order) {
        if (resident(tc.first)) continue;
        const auto up = small.find(tc);
        if (up != small.end()) {
            if (decoded.count(tc)) continue;
            Prefetched pf; /* an empty table, or more columns than the status block tracks */
            pf.pages = up->second;
            pf.done = ctx.get_event();
            ck(cudaEventRecord(pf.done, ctx.stream), "event record");
            prefetched.emplace(tc, std::move(pf));
            continue;
        }
        if (!first) {
            first = ctx.get_event();
            ck(cudaEventRecord(first, ctx.h2d_stream), "event record");
        }
        Prefetched pf;
        upload_pages(ctx, plan.inputs[tc.first].columns[tc.second], pf.pages, &stats.h2d_bytes, ctx.h2d_stream);
        pf.done = ctx.get_event();
        ck(cudaEventRecord(pf.done, ctx.h2d_stream), "event record");
        prefetched.emplace(tc, std::move(pf));
    }
    if (first) {
        cudaEvent_t last = ctx.get_event();
        ck(cudaEventRecord(last, ctx.h2d_stream), "event record");
        phase_events.push_back({PH_UPLOAD, first, last});
    }
}

/* Whether the root joins two scans whose probe key column is read by the
 * probe alone, page by page (*col): no other key and no output but the key's
 * own reads it, so it need not be decoded. A rule on what is known before
 * anything runs; a join that goes on to another table decodes it then. */
int Executor::streamed_key(std::pair<uint64_t, uint64_t> *col) const {
    const cj_plan_node &n = plan.nodes[plan.root];
    if (n.node_type != CJ_NODE_HASH_JOIN || ctx.opt.dense_keys <= 0) return 0;
    const cj_plan_node &l = plan.nodes[n.left], &r = plan.nodes[n.right];
    if (l.node_type != CJ_NODE_SCAN || r.node_type != CJ_NODE_SCAN) return 0;
    const uint64_t lrows = table_rows(l.base_table_id), rrows = table_rows(r.base_table_id);
    const bool build_left = lrows <= rrows;
    if ((int64_t)std::min(lrows, rrows) <= ctx.opt.nested_loop_max_build) return 0;
    const cj_plan_node &b = build_left ? l : r, &p = build_left ? r : l;
    const uint64_t battr = build_left ? n.left_attr : n.right_attr, pattr = build_left ? n.right_attr : n.left_attr;
    if (battr >= b.num_output_attrs || pattr >= p.num_output_attrs) return 0;
    *col = {p.base_table_id, p.output_attrs[pattr].index};
    if (*col == std::make_pair(b.base_table_id, b.output_attrs[battr].index)) return 0;
    for (uint64_t a = 0; a < n.num_output_attrs; ++a) {
        const uint64_t i = n.output_attrs[a].index;
        const bool left = i < l.num_output_attrs;
        const cj_plan_node &side = left ? l : r;
        const uint64_t k = left ? i : i - l.num_output_attrs;
        if (k < side.num_output_attrs && &side == &b &&
            *col == std::make_pair(b.base_table_id, b.output_attrs[k].index))
            return 0;
    }
    return 1;
}

void Executor::launch_tasks(std::vector<ColumnTask> &tasks, bool index) {
    KScope k(*this, index ? "page_index" : "decode");
    ck(launch_columns(L, tasks.data(), tasks.size(), index), index ? "page_index" : "decode");
}

/* A column with its page index; its dense arrays may not be written yet. */
Decoded &Executor::indexed(uint64_t t, uint64_t c) {
    auto key = std::make_pair(t, c);
    auto it = decoded.find(key);
    if (it != decoded.end()) {
        if (it->second.status_col >= 0) used_cols |= 1ull << it->second.status_col;
        return it->second;
    }
    Decoded d;
    d.type = column_type(t, c);
    d.rows = table_rows(t);
    if (d.rows > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "table exceeds 2^32-1 rows (u32 row ids)");
    auto pf = prefetched.find(key);
    if (const cj_table *r = resident(t)) {
        d.src = r->cols[c];
    } else if (pf != prefetched.end()) {
        d.src = pf->second.pages;
        ck(cudaStreamWaitEvent(ctx.stream, pf->second.done, 0), "stream wait");
        ctx.put_event(pf->second.done);
        prefetched.erase(pf);
    } else {
        PhaseScope ph(*this, PH_UPLOAD);
        upload_pages(ctx, plan.inputs[t].columns[c], d.src, &stats.h2d_bytes);
    }
    PhaseScope ph(*this, PH_DECODE);
    Slab slab;
    d.reserve(slab);
    slab.reserve(sizeof(ColumnState));
    slab.open(ctx);
    d.mem = slab.mem;
    ColumnState *state = slab.take_as<ColumnState>(sizeof(ColumnState));
    ck(cudaMemsetAsync(state, 0, sizeof(ColumnState), ctx.stream), "memset");
    std::vector<ColumnTask> tasks{column_task(d, slab, state, &ctx.d_status->errors)};
    launch_tasks(tasks, true);
    return decoded.emplace(key, std::move(d)).first->second;
}

Decoded &Executor::decode(uint64_t t, uint64_t c) {
    Decoded &d = indexed(t, c);
    if (!d.ready) {
        PhaseScope ph(*this, PH_DECODE);
        std::vector<ColumnTask> tasks{d.task};
        launch_tasks(tasks, false);
        d.ready = true;
    }
    return d;
}

/* Several columns, in one launch. */
void Executor::decode_all(const std::vector<TC> &cols) {
    std::vector<ColumnTask> tasks;
    for (const TC &tc : cols) {
        Decoded &d = indexed(tc.first, tc.second);
        if (d.ready) continue;
        tasks.push_back(d.task);
        d.ready = true;
    }
    if (tasks.empty()) return;
    PhaseScope ph(*this, PH_DECODE);
    launch_tasks(tasks, false);
}

ColView Executor::view(const Relation &R, const RelCol &c, const uint32_t *rid_a) {
    return make_view(decode(c.input, c.col), R, c, rid_a);
}

Relation Executor::resolve(uint64_t node, int depth) {
    if (depth > (int)plan.num_nodes) fail(CJ_ERR_INVALID_PLAN, "plan has a cycle");
    const cj_plan_node &n = plan.nodes[node];
    if (n.node_type == CJ_NODE_SCAN) return scan_relation(plan, n);
    return exec_join(node, depth, false, nullptr);
}

Relation Executor::exec_join(uint64_t node_idx, int depth, bool is_root, cj_result **out) {
    const cj_plan_node &n = plan.nodes[node_idx];
    Relation Lr = resolve(n.left, depth + 1);
    Relation Rr = resolve(n.right, depth + 1);

    /* select_build_probe_side (join_setup.h:108-136): the smaller relation
     * builds, left wins ties; the plan's build_left hint is not used. */
    const bool build_left = Lr.rows <= Rr.rows;
    Relation &B = build_left ? Lr : Rr;
    Relation &P = build_left ? Rr : Lr;
    const uint64_t battr = build_left ? n.left_attr : n.right_attr;
    const uint64_t pattr = build_left ? n.right_attr : n.left_attr;
    if (battr >= B.cols.size() || pattr >= P.cols.size()) fail(CJ_ERR_INVALID_PLAN, "join key index out of range");
    const RelCol bk = B.cols[battr], pk = P.cols[pattr];
    auto key_ok = [](int32_t t) { return t == CJ_INT32 || t == CJ_INT64; };
    if (!key_ok(bk.type) || !key_ok(pk.type)) fail(CJ_ERR_UNSUPPORTED, "join keys must be INT32 or INT64");
    if (B.rows > 0xFFFFFFFFull || P.rows > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "relation exceeds 2^32-1 rows");

    /* Output columns over (left ++ right) and which match side each needs
     * (determine_collection_mode, join_setup.h:146-173). */
    struct OutRef {
        bool from_build;
        const Relation *rel;
        RelCol col;
        bool from_keys = false; /* root: read from the keys the probe writes */
        DevPtr pages;           /* root: pages the probe writes, if the column has no NULL */
        bool direct_only = false; /* ... and the table is direct-mapped */
    };
    std::vector<OutRef> outs;
    bool need_b = false, need_p = false;
    const uint64_t lsz = Lr.cols.size();
    for (uint64_t a = 0; a < n.num_output_attrs; ++a) {
        const cj_attr &at = n.output_attrs[a];
        if (at.index >= lsz + Rr.cols.size()) fail(CJ_ERR_INVALID_PLAN, "output attribute out of range");
        const Relation *side = at.index < lsz ? &Lr : &Rr;
        RelCol c = side->cols[at.index < lsz ? at.index : at.index - lsz];
        if (c.type != at.type) fail(CJ_ERR_INVALID_PLAN, "output attribute type differs from its column");
        bool fb = side == &B;
        if (key_from_probe_side(fb, c, bk, pk)) {
            fb = false;
            side = &P;
            c = pk;
        }
        need_b |= fb;
        need_p |= !fb;
        outs.push_back({fb, side, c});
    }

    stats.num_joins++;
    stats.probe_rows += P.rows;
    uint64_t M = 0;
    /* At the root, outputs of the probe key (and of the build key, which is
     * read through the probe side) are written by the probe itself, straight
     * into their places in the result pages (matched keys are never NULL):
     * no gather, no copy; every such column shares those pages. */
    bool emit_keys = false;
    if (is_root) {
        need_p = false;
        for (auto &o : outs) {
            if (!o.from_build && o.rel == &P && same_column(o.col, pk)) {
                o.from_keys = true;
                emit_keys = true;
            } else if (!o.from_build) {
                need_p = true;
            }
        }
    }
    const bool collect = need_b || need_p || emit_keys;
    const int32_t key_bytes = pk.type == CJ_INT32 ? 4 : 8;
    DevPtr mb, mp, mk;
    /* The root's result columns: the pages the probe wrote the keys into, or
     * a relation column and the match row ids that select its rows. */
    auto root_columns = [&](std::vector<OutCol> &cols, std::vector<int32_t> &types) {
        for (auto &o : outs) {
            OutCol oc{o.rel, o.col, nullptr, nullptr};
            if (o.from_keys) {
                oc.rel = nullptr;
                oc.pages = mk; /* o.col.type == the probe key's type */
            } else {
                oc.rid_a = o.from_build ? (mb ? mb->as<uint32_t>() : nullptr) : (mp ? mp->as<uint32_t>() : nullptr);
                oc.pages = o.pages;
                oc.direct_only = o.direct_only;
            }
            cols.push_back(oc);
            types.push_back(o.col.type);
        }
    };
    if (B.rows && P.rows) {
        const ColView bv = view(B, bk, nullptr);
        if (is_root) {
            /* The root's other output columns whose pages are already in
             * HBM are indexed (and decoded, if they must be) now, while the
             * kernels above run, rather than after the probe's
             * synchronisation, where the GPU would wait for the host to
             * enqueue them. Columns still uploading stay lazy, so that the
             * result downloads overlap their uploads. */
            std::vector<TC> here;
            for (const auto &o : outs)
                if (!o.from_keys && (resident(o.col.input) || decoded.count({o.col.input, o.col.col})))
                    here.push_back({o.col.input, o.col.col});
            decode_all(here);
        }
        const uint64_t nl_max = std::min<int64_t>(std::max<int64_t>(ctx.opt.nested_loop_max_build, 0), kNestedLoopMax);
        const bool nl = B.rows <= nl_max;
        DevPtr dir, tuples, nlk, nlr, nlc, slots;
        int log2_slots = 0;
        bool inline_dir = true;
        bool unique = false; /* a table of unique keys tried (the device decides) */
        bool multi = false;  /* the table of repeated dense keys */
        MultiTable multi_table{};
        bool open_multi = false; /* multi: the keys are not dense */
        OpenMultiTable open_table{};
        DevPtr multi_rows, runs;
        uint64_t most_rows = ~0ull; /* multi: of a key, where it is known */
        bool words_ready = false; /* multi: the status words are as its probe needs them */
        const bool words_clear = join_words_clear;
        join_words_clear = false; /* every join counts its matches there */
        UniqueTable table{};
        auto build_hash = [&]() {
            BuildPlan bp;
            bp.num_rows = (uint32_t)B.rows;
            bp.log2_slots = std::max(11, ceil_log2(B.rows)); /* hashtable.h:255-264 */
            /* 2^11 directory slots per partition by default (the slot
             * counters of one partition fit shared memory); the partition
             * bits are spread over one radix pass, or two above 12 bits
             * (build sides of more than 2^23 rows) */
            const int log2_spp = std::min(std::min(build_log2_spp(ctx, B.rows), 14), bp.log2_slots);
            bp.log2_parts = bp.log2_slots - log2_spp;
            log2_slots = bp.log2_slots;
            const int kb = bk.type == CJ_INT32 ? 4 : 8;
            const Launch LB = build_launch(ctx, B.rows);
            bp.inline_first = kb == 4 && build_dir_bytes(bp.log2_slots, 4, true) + B.rows * build_tuple_bytes(4) <=
                                             (uint64_t)ctx.opt.inline_dir_max_bytes;
            inline_dir = bp.inline_first;
            dir = ctx.alloc(build_dir_bytes(bp.log2_slots, kb, bp.inline_first));
            tuples = ctx.alloc(B.rows * build_tuple_bytes(kb));
            DevPtr tmp = ctx.alloc(build_temp_bytes(LB, bp, kb));
            KScope k(*this, "build");
            ck(launch_build(LB, bp, bv, ctx.d_bloom, dir->as<uint64_t>(), tuples->ptr, tmp->ptr), "build");
        };
        if (nl) {
            stats.num_nested_loop_joins++;
            PhaseScope ph(*this, PH_NL);
            nlk = ctx.alloc(kNestedLoopMax * 8);
            nlr = ctx.alloc(kNestedLoopMax * 4);
            nlc = ctx.alloc(4);
            KScope k(*this, "nl_collect");
            ck(launch_nl_collect(L, bv, (uint32_t)B.rows, nlk->as<int64_t>(), nlr->as<uint32_t>(),
                                 nlc->as<uint32_t>()),
               "nl_collect");
        } else {
            stats.num_hash_joins++;
            PhaseScope ph(*this, PH_BUILD);
            if (ctx.opt.dense_keys > 0) {
                /* Unique keys spread over at most dense_keys x rows values get
                 * a direct-mapped table: one random access per probe row
                 * instead of a directory entry and a tuple; unique keys that
                 * span more an open-addressing table: one sector. The device
                 * works out the key range and which table it is, if any; the
                 * host learns it at the probe's own synchronisation and then,
                 * if neither, builds another. Direct-mapped: 4 bytes per
                 * slot, at 8 x rows 32 B per build row, at most 2^28 slots (1
                 * GiB); open-addressing: 16 B per build row, 34 for INT64
                 * keys, left out where the memory is short. One buffer serves
                 * both. */
                table.max_span = std::min<uint64_t>((uint64_t)ctx.opt.dense_keys * B.rows, 1ull << 28);
                table.wide = bk.type == CJ_INT64;
                const uint64_t open_slots = std::max<uint64_t>((2 * B.rows + 15) & ~15ull, 1024);
                if (B.rows <= kOpenMaxRows && ample(open_slots * (table.wide ? 17 : 8)))
                    table.open_slots = (uint32_t)open_slots;
                table.params = ctx.d_status->table;
                if (table.open_slots && !(slots = spare(unique_table_bytes(table)))) table.open_slots = 0;
                if (!slots) slots = ctx.alloc(unique_table_bytes(table));
                table.slots = slots->ptr;
                if (!words_clear) clear_join_words();
                KScope k(*this, "unique_build");
                ck(launch_unique_build(L, bv, (uint32_t)B.rows, table), "unique_build");
                unique = true;
            }
            if (!unique) build_hash();
        }
        /* Result pages of an earlier probe: a table that was refused, or a
         * capacity that the matches outgrew. */
        auto drop_pages = [&]() {
            for (auto &o : outs) {
                o.pages.reset();
                o.direct_only = false;
            }
        };
        /* At most: the result pages that a probe with room for `cap` matches
         * writes, the keys' apart. */
        auto beside_bytes = [&](uint64_t cap) {
            uint64_t bytes = 0;
            for (const auto &o : outs)
                if (is_root && !o.from_keys && o.col.type != CJ_VARCHAR) bytes += cap * (o.col.type == CJ_INT32 ? 5 : 9);
            return bytes;
        };
        /* Allocates the match outputs for `cap` pairs and launches the probe
         * of the table built above. */
        uint64_t cap = P.rows;
        bool widened = false; /* cap is above the probe rows on an estimate */
        auto match_arrays = [&](uint64_t cap) {
            /* the key columns' result pages, sized for the capacity */
            const uint32_t key_rpp = rows_per_page_fixed(pk.type);
            mk = emit_keys ? ctx.alloc((cap + key_rpp - 1) / key_rpp * kPageSize) : nullptr;
            mb = need_b ? ctx.alloc(cap * 4) : nullptr;
            mp = need_p ? ctx.alloc(cap * 4) : nullptr;
        };
        auto launch_probe = [&]() {
            drop_pages();
            if (widened) {
                widened = false;
                try {
                    match_arrays(cap);
                } catch (const Error &e) {
                    if (e.code != CJ_ERR_OUT_OF_MEMORY) throw;
                    mk.reset();
                    mb.reset();
                    cap = P.rows;
                    match_arrays(cap);
                }
            } else {
                match_arrays(cap);
            }
            MatchOut mo;
            mo.build_rids = mb ? mb->as<uint32_t>() : nullptr;
            mo.probe_rids = mp ? mp->as<uint32_t>() : nullptr;
            mo.key_pages = mk ? mk->as<uint8_t>() : nullptr;
            mo.key_bytes = key_bytes;
            mo.capacity = collect ? cap : 0;
            mo.counter = &ctx.d_status->counter;
            runs.reset();
            if (unique || multi) {
                /* The root's fixed-width columns whose pages are in HBM are
                 * written by the probe itself where they hold no NULL; row
                 * ids are collected for the others only. */
                UniqueOut uo{};
                uo.match = mo;
                if (multi && most_rows >= kRunFrom && mo.capacity >= (most_rows == ~0ull ? kRunsFromBlind : kRunsFrom) &&
                    (runs = spare(mo.capacity / kRunFrom * sizeof(MatchRun)))) {
                    uo.runs.runs = runs->as<MatchRun>();
                    uo.runs.count = ctx.d_status->table + kTableDone; /* zero: clear_join_words */
                    uo.runs.capacity = mo.capacity / kRunFrom;
                }
                const bool room = room_for(beside_bytes(cap));
                for (auto &o : outs) {
                    if (!is_root || o.from_keys) continue;
                    const auto it = decoded.find({o.col.input, o.col.col});
                    const bool beside = /* the table and the column stay in L2 together */
                        !o.from_build || !multi || it == decoded.end() ||
                        (open_multi ? open_table.nslots * 16ull : multi_table.span * 8ull) + B.rows * 4 +
                                it->second.src.num_pages * kPageSize <= kEmitBesideOpen;
                    if (o.col.type != CJ_VARCHAR && it != decoded.end() && it->second.ready && uo.n < kEmitColumns &&
                        beside && room) {
                        const uint32_t R = rows_per_page_fixed(o.col.type);
                        o.pages = spare((cap + R - 1) / R * kPageSize);
                    }
                    if (o.pages) {
                        o.direct_only = unique && o.from_build && table.open_slots &&
                                        table.open_slots * (table.wide ? 16ull : 8ull) +
                                                        it->second.src.num_pages * kPageSize > kEmitBesideOpen;
                        uo.cols[uo.n++] = {view(*o.rel, o.col, nullptr), o.pages->as<uint8_t>(), o.from_build ? 1 : 0,
                                           o.direct_only ? 1 : 0};
                    } else {
                        (o.from_build ? uo.need_b : uo.need_p) = true;
                    }
                }
                if (!is_root) {
                    uo.need_b = need_b;
                    uo.need_p = need_p;
                }
                ProbeKey key{};
                if (pk.vec < 0) {
                    /* a scan: the probe reads the key's pages themselves */
                    const Decoded &d = indexed(pk.input, pk.col);
                    key.col = make_view(d, P, pk, nullptr);
                    key.base = d.task.base;
                    key.loc = d.task.loc;
                    key.num_pages = d.src.num_pages;
                    key.err = d.task.err;
                } else {
                    key.col = view(P, pk, nullptr);
                }
                PhaseScope ph(*this, PH_PROBE);
                if (multi && open_multi) {
                    KScope k(*this, "probe_open_multi");
                    ck(launch_probe_open_multi(L, key, (uint32_t)P.rows, open_table, uo), "probe_open_multi");
                    return;
                }
                if (multi) {
                    KScope k(*this, "probe_multi");
                    ck(launch_probe_multi(L, key, (uint32_t)P.rows, multi_table, uo), "probe_multi");
                    return;
                }
                KScope k(*this, "probe_unique");
                ck(launch_probe_unique(L, key, (uint32_t)P.rows, table, uo), "probe_unique");
                return;
            }
            const ColView pv = view(P, pk, nullptr);
            DevPtr sched = ctx.alloc(probe_sched_bytes((uint32_t)P.rows));
            {
                PhaseScope ph(*this, nl ? PH_NL : PH_PROBE);
                if (nl) {
                    KScope k(*this, "nl_probe");
                    ck(launch_nl_probe_tiles(L, pv, (uint32_t)P.rows, nlk->as<int64_t>(), nlr->as<uint32_t>(),
                                             nlc->as<uint32_t>(), mo, sched->ptr),
                       "nl_probe");
                } else {
                    KScope k(*this, "probe_hash");
                    ck(launch_probe_tiles_hash(probe_launch(ctx, P.rows), pv, (uint32_t)P.rows, bk.type,
                                               dir->as<uint64_t>(), tuples->ptr, log2_slots, ctx.d_bloom, mo,
                                               sched->ptr, inline_dir),
                       "probe");
                }
            }
        };
        /* The device refused the table of unique keys (its probe did
         * nothing). Keys that repeat get a table of repeated keys: one random
         * access per probe row and one per further match.
         * Over a dense range (64M x 4M rows over 3M keys): hash build, probe
         * and page writers 235 + 1004 + 570 us, 130 + 956 + 344 here, the
         * probe with one of the columns written beside it; 8 bytes per value
         * of the range, at most kMultiSpan values per build row so that it
         * stays near the hash table's 24 bytes per row.
         * Over any other range, open addressing, 42 bytes per build row
         * (30M x 3M INT32 rows, eight a key, half of the probe rows with a
         * match: the whole join 4916 us on the hash table without room for
         * them, 2674 here; 100K x 5K INT64 345 and 248).
         * The hash table is left for keys that hardly repeat
         * (kOpenMultiMean2), few probe rows (kSampleFrom), keys that span all
         * of INT64 or pile up in the table, and for more build rows than fit
         * kOpenMaxRows or the memory. */
        auto replace_unique = [&]() {
            unique = false;
            slots.reset();
            drop_pages();
            PhaseScope ph(*this, PH_BUILD);
            unsigned long long tp[kTableWords];
            std::copy(ctx.h_status->table, ctx.h_status->table + kTableWords, tp);
            /* room for the keys' mean number of rows per match, up to 4, and
             * an eighth more: where every probe row matches, a random half of
             * all results lie just above the mean, and a result above the
             * room runs the probe again (3M x 30M rows, four rows for three
             * keys: 2104 us, 1296 with the eighth; below kSpareEighth the
             * second run is little more than its launch). A server's worker keeps
             * to the probe rows: admission counts on no more, and what one
             * plan takes on a guess another might need. */
            auto widen = [&](uint64_t keys) {
                if (!ctx.owns_pool) return;
                const uint64_t mean =
                    std::min<uint64_t>(P.rows * (uint64_t)tp[kTableCount] / std::max<uint64_t>(keys, 1), 4 * P.rows);
                const uint64_t more = std::min<uint64_t>(mean + (P.rows >= kSpareEighth ? mean / 8 : 0), 0xFFFFFFFFull);
                /* a match: two row ids and a key at most, here */
                if (mean > cap && more > cap && room_for(more * 17)) {
                    cap = more;
                    widened = true;
                }
            };
            if ((!tp[kTableRefused] || tp[kTableRefused] == kTableRepeats) && tp[kTableSpan] <= kMultiSpan * B.rows &&
                (slots = spare((tp[kTableSpan] + 1) * 8)) && (multi_rows = spare(B.rows * 4))) {
                multi = true;
                multi_table.lo = (int64_t)tp[kTableLo];
                multi_table.span = (uint32_t)tp[kTableSpan];
                multi_table.entries = slots->as<unsigned long long>();
                multi_table.rows = multi_rows->as<uint32_t>();
                widen(tp[kTableSpan]);
                clear_join_words();
                words_ready = true;
                KScope k(*this, "multi_build");
                ck(launch_multi_build(L, bv, (uint32_t)B.rows, multi_table), "multi_build");
                return;
            }
            slots.reset();
            multi_rows.reset();
            DevPtr slot_of;
            const uint32_t open_n = (uint32_t)std::max<uint64_t>((2 * std::min(B.rows, kOpenMaxRows) + 7) & ~7ull, 1024);
            const bool many_probes = P.rows / kOpenMultiProbe >= B.rows;
            uint64_t keys = 0; /* different ones, about; 0: not known */
            if (DevPtr bits; P.rows >= (many_probes ? kSampleFrom : kSampleFromFew) && (bits = spare(kSampleBits / 8))) {
                uint32_t shift;
                clear_join_words();
                ck(cudaMemsetAsync(bits->ptr, 0, kSampleBits / 8, ctx.stream), "memset");
                {
                    KScope k(*this, "key_sample");
                    ck(launch_key_sample(L, bv, (uint32_t)B.rows, bits->as<uint32_t>(), ctx.d_status->table, &shift),
                       "key_sample");
                }
                sync();
                keys = std::min<uint64_t>(sampled_keys(ctx.h_status->table[0], shift), tp[kTableCount]);
            }
            if ((keys ? 2 * tp[kTableCount] >= kOpenMultiMean2 * keys : many_probes) && tp[kTableRefused] != kTableWhole &&
                B.rows <= kOpenMaxRows && ample(B.rows * (2 * (sizeof(MultiSlot) + 1) + 8)) &&
                (slots = spare(open_n * (sizeof(MultiSlot) + 1))) && (multi_rows = spare(B.rows * 4)) &&
                (slot_of = spare(B.rows * 4))) {
                open_table.nslots = open_n;
                open_table.lo = tp[kTableLo];
                open_table.width = tp[kTableSpan] - 1;
                open_table.empty = tp[kTableEmpty];
                open_table.found = ctx.d_status->table;
                open_table.slots = slots->as<MultiSlot>();
                open_table.tags = slots->as<uint8_t>() + open_n * sizeof(MultiSlot);
                open_table.rows = multi_rows->as<uint32_t>();
                open_table.slot_of = slot_of->as<uint32_t>();
                clear_join_words();
                {
                    KScope k(*this, "open_multi_build");
                    ck(launch_open_multi_build(L, bv, (uint32_t)B.rows, open_table), "open_multi_build");
                }
                multi = open_multi = true;
                words_ready = true;
                if (!keys) { /* the number of keys, before a probe that might run twice without it */
                    sync();
                    keys = ctx.h_status->table[kMultiKeys];
                    most_rows = ctx.h_status->table[kMultiMost];
                    if (ctx.h_status->table[kMultiGaveUp]) multi = open_multi = false;
                }
                if (multi) {
                    widen(keys);
                    return;
                }
            }
            slots.reset();
            multi_rows.reset();
            slot_of.reset();
            clear_join_words(); /* the match counter, and words no longer read */
            if (keys) widen(keys);
            build_hash();
        };
        auto count_join = [&]() {
            const int kind = table_kind(ctx.h_status->table, table.open_slots);
            stats.num_direct_joins += kind == 1;
            stats.num_open_joins += kind == 2 && !table.wide; /* INT32 keys, as documented */
        };
        bool probed = false; /* the probe has been launched already */
        bool all_fixed = true;
        for (const auto &o : outs) all_fixed &= o.col.type != CJ_VARCHAR;
        if (is_root && unique && collect && all_fixed && (flags & CJ_EXEC_RESULT_ON_DEVICE) && ctx.opt.defer_count &&
            room_for(beside_bytes(cap))) {
            /* Unique build keys at the root, result left in HBM, no VARCHAR
             * output: at most one match per probe row, so the result is sized
             * for P.rows and its pages are written with the match count read
             * on the device. The execution's one host synchronisation comes
             * last; only if the device refused the table does the join go on
             * as below. Without room for the probe rows the count is read
             * first, and the pages sized by it. */
            launch_probe();
            std::vector<OutCol> cols;
            std::vector<int32_t> types;
            root_columns(cols, types);
            std::unique_ptr<cj_result> r;
            try {
                r.reset(materialize(cols, types, cap, &ctx.d_status->counter));
            } catch (const Error &e) {
                if (e.code != CJ_ERR_OUT_OF_MEMORY) throw;
                probed = true; /* the pages of the matches alone may fit */
            }
            if (r) {
                sync();
                if (table_kind(ctx.h_status->table, table.open_slots)) {
                    M = ctx.h_status->counter;
                    finish_counted(*r, M);
                    count_join();
                    stats.matches += M;
                    synced_last = true;
                    *out = r.release();
                    return Relation{};
                }
                r.reset();
                replace_unique();
            }
        }
        for (;; probed = false) {
            if (!probed) {
                if (multi && !words_ready) clear_join_words(); /* the match counter, the number of runs */
                words_ready = false;
                launch_probe();
            }
            sync();
            if (open_multi && ctx.h_status->table[kMultiGaveUp]) { /* walks given up: the table is unusable */
                multi = open_multi = false;
                cap = P.rows;
                widened = false;
                slots.reset();
                multi_rows.reset();
                drop_pages();
                clear_join_words();
                build_hash();
                continue;
            }
            if (unique && !table_kind(ctx.h_status->table, table.open_slots)) {
                replace_unique();
                continue;
            }
            M = ctx.h_status->counter;
            if (M <= cap || !collect) break;
            if (unique) fail(CJ_ERR_INTERNAL, "more matches than probe rows over unique keys");
            if (M > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "join result exceeds 2^32-1 rows");
            stats.probe_reruns++;
            cap = M;
        }
        if (unique) count_join();
    }
    if (M > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "join result exceeds 2^32-1 rows");
    stats.matches += M;

    if (is_root) {
        std::vector<OutCol> cols;
        std::vector<int32_t> types;
        root_columns(cols, types);
        *out = materialize(cols, types, M);
        return Relation{};
    }

    /* Intermediate: one row-id vector per (side, source vector). */
    Relation res;
    res.rows = M;
    std::map<std::pair<int, int>, int> vecmap;
    PhaseScope ph(*this, PH_INTER);
    for (auto &o : outs) {
        const int side = o.from_build ? 0 : 1;
        auto key = std::make_pair(side, o.col.vec);
        auto it = vecmap.find(key);
        int vi;
        if (it != vecmap.end()) {
            vi = it->second;
        } else {
            const DevPtr &match = o.from_build ? mb : mp;
            DevPtr nv;
            if (M == 0) {
                nv = ctx.alloc(0);
            } else if (o.col.vec < 0) {
                nv = match; /* scan side: the match row ids are base rows */
            } else {
                nv = ctx.alloc(M * 4);
                KScope k(*this, "gather_rids");
                ck(launch_gather_u32(L, o.rel->vecs[o.col.vec]->as<uint32_t>(), match->as<uint32_t>(), M,
                                     nv->as<uint32_t>()),
                   "gather");
            }
            vi = (int)res.vecs.size();
            res.vecs.push_back(nv);
            vecmap[key] = vi;
        }
        res.cols.push_back({o.col.type, o.col.input, o.col.col, vi, true});
    }
    return res;
}

/* Writes the root's result pages. For a host result each column's pages
 * go down on the context's download stream as soon as its writer is done,
 * so the copy of one column overlaps the writing of the next. */
cj_result *Executor::materialize(const std::vector<OutCol> &cols, const std::vector<int32_t> &types,
                                 uint64_t rows, const unsigned long long *rows_dev) {
    auto *res = new cj_result;
    std::unique_ptr<cj_result> guard(res);
    res->ctx = &ctx;
    res->num_rows = rows;
    res->types = types;
    const size_t nc = cols.size();
    res->num_pages.assign(nc, 0);
    res->dev_pages.resize(nc);
    res->host_cols.assign(nc, nullptr);
    const bool to_host = !(flags & CJ_EXEC_RESULT_ON_DEVICE);
    if (rows_dev) {
        /* rows is a capacity and the count is on the device: fixed-width
         * columns left in HBM only (their pages do not depend on the count
         * beyond the last one) */
        for (int32_t t : types)
            if (t == CJ_VARCHAR) fail(CJ_ERR_INTERNAL, "device-counted result with a VARCHAR column");
        if (to_host) fail(CJ_ERR_INTERNAL, "device-counted result for the host");
    }
    /* Orders the kernel stream (and so every later free) after the copies
     * issued so far, also when an error leaves this scope early. */
    struct DownloadJoin {
        Context &ctx;
        cudaEvent_t first = nullptr, last = nullptr;
        bool timed = false; /* events handed to the phase timer */
        ~DownloadJoin() {
            if (!first) return;
            if (!last) {
                last = ctx.get_event();
                cudaEventRecord(last, ctx.d2h_stream);
            }
            cudaStreamWaitEvent(ctx.stream, last, 0);
            if (!timed) {
                ctx.put_event(first);
                ctx.put_event(last);
            }
        }
    } dl{ctx};
    constexpr uint64_t kSmallDownload = 4u << 20; /* copied in 80 us; nothing worth overlapping */
    bool small_download = false;
    std::vector<int64_t> alias(nc, -1);
    {
        PhaseScope ph(*this, PH_MAT);
        const uint32_t TR = (uint32_t)std::max<int64_t>(64, std::min<int64_t>(ctx.opt.varchar_tile_rows, 8192));
        std::vector<DevPtr> vtemp;
        std::vector<VarcharTask> vtasks;
        std::vector<int> vtask_of(nc, -1); /* a VARCHAR column's task */
        DevPtr totals;
        size_t nvar = 0;
        for (size_t c = 0; c < nc; ++c)
            if (types[c] == CJ_VARCHAR) ++nvar;
        if (rows && nvar) {
            totals = ctx.alloc(nvar * 12); /* page counts, then finished-tile counts */
            ck(cudaMemsetAsync(totals->ptr, 0, nvar * 12, ctx.stream), "memset");
            for (size_t c = 0; c < nc; ++c) {
                if (types[c] != CJ_VARCHAR) continue;
                const size_t k = vtasks.size();
                vtask_of[c] = (int)k;
                vtemp.push_back(ctx.alloc(varchar_temp_bytes(rows, TR)));
                VarcharTask t{};
                t.col = out_view(cols[c]);
                t.rows = rows;
                t.total_pages = totals->as<unsigned long long>() + k;
                t.done = reinterpret_cast<unsigned int *>(totals->as<unsigned long long>() + nvar) + k;
                place_varchar(t, TR, vtemp.back()->ptr);
                vtasks.push_back(t);
            }
            {
                KScope ks(*this, "varchar_plan");
                ck(launch_varchar(L, vtasks.data(), vtasks.size(), true), "varchar_plan");
            }
            std::vector<unsigned long long> host(nvar);
            ck(cudaMemcpyAsync(host.data(), totals->ptr, nvar * 8, cudaMemcpyDeviceToHost, ctx.stream), "copy");
            sync();
            for (size_t c = 0; c < nc; ++c)
                if (types[c] == CJ_VARCHAR) res->num_pages[c] = host[vtask_of[c]];
        }
        uint64_t total_pages = 0;
        for (size_t c = 0; c < nc; ++c) {
            if (rows && types[c] != CJ_VARCHAR) {
                const uint32_t R = rows_per_page_fixed(types[c]);
                res->num_pages[c] = (rows + R - 1) / R;
            }
            total_pages += res->num_pages[c];
        }
        stats.output_rows = rows;
        stats.output_pages = total_pages;
        /* Columns that share device pages (the join keys written by the
         * probe) share one host copy too: downloaded once. */
        for (size_t c = 0; c < nc; ++c)
            for (size_t k = 0; k < c && alias[c] < 0; ++k)
                if (cols[c].pages && cols[k].pages == cols[c].pages) alias[c] = (int64_t)k;
        uint64_t host_pages = 0;
        for (size_t c = 0; c < nc; ++c)
            if (alias[c] < 0) host_pages += res->num_pages[c];
        if (to_host && host_pages) {
            res->host = ctx.alloc_pinned(host_pages * kPageSize);
            uint8_t *h = static_cast<uint8_t *>(res->host->ptr);
            for (size_t c = 0; c < nc; ++c) {
                if (alias[c] >= 0) {
                    res->host_cols[c] = res->host_cols[alias[c]];
                    continue;
                }
                res->host_cols[c] = h;
                h += res->num_pages[c] * kPageSize;
            }
        }
        /* A host result's columns are written one by one, each downloaded
         * while the next is written (and still uploaded); a result left in
         * HBM, or a small one, has its columns written by one launch of each
         * kind, and a small one is then copied on the kernel stream. */
        const bool overlap = to_host && host_pages * kPageSize > kSmallDownload;
        std::vector<PageTask> ptasks;
        auto write_pages = [&]() {
            KScope ks(*this, "write_pages");
            ck(launch_write_pages(L, ptasks.data(), ptasks.size()), "write_pages");
            ptasks.clear();
        };
        for (size_t c = 0; c < nc; ++c) {
            if (!rows) continue;
            PageTask t{};
            t.rows = rows;
            t.rows_dev = rows_dev;
            if (cols[c].pages) {
                /* values already in place: headers and bitmaps, once per
                 * shared page array */
                if (cols[c].pages->bytes < res->num_pages[c] * kPageSize)
                    fail(CJ_ERR_INTERNAL, "result pages smaller than the result");
                if (alias[c] >= 0) res->dev_pages[c] = res->dev_pages[alias[c]];
                else res->dev_pages[c] = rows_dev ? cols[c].pages : fitted(cols[c].pages, res->num_pages[c] * kPageSize);
                if (cols[c].rel) t.col = out_view(cols[c]);
                else t.col.type = types[c];
                t.finish = cols[c].rel ? 2 : 1;
                if (cols[c].direct_only) t.table = ctx.d_status->table;
            } else {
                /* decoded here, not before the loop: the kernel stream waits
                 * for a column's upload only when its pages are written */
                t.col = out_view(cols[c]);
                res->dev_pages[c] = ctx.alloc(res->num_pages[c] * kPageSize);
            }
            t.out = res->dev_pages[c]->as<uint8_t>();
            if (types[c] == CJ_VARCHAR) {
                VarcharTask &v = vtasks[vtask_of[c]];
                v.out = t.out;
                if (overlap) {
                    KScope ks(*this, "varchar_write");
                    ck(launch_varchar(L, &v, 1, false), "varchar_write");
                }
            } else if (alias[c] < 0) {
                ptasks.push_back(t);
                if (overlap) write_pages();
            }
            const size_t bytes = res->num_pages[c] * kPageSize;
            if (overlap && bytes && alias[c] < 0) {
                cudaEvent_t written = ctx.get_event();
                ck(cudaEventRecord(written, ctx.stream), "event record");
                ck(cudaStreamWaitEvent(ctx.d2h_stream, written, 0), "stream wait");
                ctx.put_event(written);
                if (!dl.first) {
                    dl.first = ctx.get_event();
                    ck(cudaEventRecord(dl.first, ctx.d2h_stream), "event record");
                }
                ck(cudaMemcpyAsync(res->host_cols[c], res->dev_pages[c]->ptr, bytes, cudaMemcpyDeviceToHost,
                                   ctx.d2h_stream),
                   "download");
                stats.d2h_bytes += bytes;
            }
        }
        if (!ptasks.empty()) write_pages();
        if (!overlap && rows && !vtasks.empty()) {
            KScope ks(*this, "varchar_write");
            ck(launch_varchar(L, vtasks.data(), vtasks.size(), false), "varchar_write");
        }
        small_download = to_host && !overlap;
    }
    if (small_download) {
        PhaseScope ph(*this, PH_DOWNLOAD);
        for (size_t c = 0; c < nc; ++c) {
            const size_t bytes = res->num_pages[c] * kPageSize;
            if (!bytes || alias[c] >= 0) continue;
            ck(cudaMemcpyAsync(res->host_cols[c], res->dev_pages[c]->ptr, bytes, cudaMemcpyDeviceToHost, ctx.stream),
               "download");
            stats.d2h_bytes += bytes;
        }
    }
    if (dl.first) {
        dl.last = ctx.get_event();
        ck(cudaEventRecord(dl.last, ctx.d2h_stream), "event record");
        phase_events.push_back({PH_DOWNLOAD, dl.first, dl.last});
        dl.timed = true;
    }
    return guard.release();
}

cj_result *Executor::run(cj_exec_stats *st) {
    auto t0 = std::chrono::steady_clock::now();
    const uint64_t launches0 = launches_so_far();
    validate();
    prefetch();
    cj_result *res = nullptr;
    const cj_plan_node &root = plan.nodes[plan.root];
    if (root.node_type == CJ_NODE_SCAN) {
        /* A scan root (the reference requires a join root) returns the
         * projected table. */
        Relation s = scan_relation(plan, root);
        if (s.rows > 0xFFFFFFFFull) fail(CJ_ERR_LIMIT, "table exceeds 2^32-1 rows");
        std::vector<OutCol> cols;
        std::vector<int32_t> types;
        for (auto &c : s.cols) {
            cols.push_back({&s, c, nullptr, nullptr});
            types.push_back(c.type);
        }
        res = materialize(cols, types, s.rows);
    } else {
        exec_join(plan.root, 0, true, &res);
    }
    std::unique_ptr<cj_result> guard(res);
    if (!synced_last) sync();
    double ph_us[PH_COUNT] = {0};
    for (auto &pe : phase_events) {
        float ms = 0;
        if (cudaEventElapsedTime(&ms, pe.a, pe.b) == cudaSuccess) ph_us[pe.phase] += ms * 1000.0;
    }
    cudaGetLastError();
    if (ctx.opt.profile_kernels) ctx.resolve_profile();
    auto t1 = std::chrono::steady_clock::now();
    stats.upload_us = ph_us[PH_UPLOAD];
    stats.decode_us = ph_us[PH_DECODE];
    stats.build_us = ph_us[PH_BUILD];
    stats.probe_us = ph_us[PH_PROBE];
    stats.nested_loop_us = ph_us[PH_NL];
    stats.intermediate_us = ph_us[PH_INTER];
    stats.materialize_us = ph_us[PH_MAT];
    stats.download_us = ph_us[PH_DOWNLOAD];
    stats.total_us = std::chrono::duration<double, std::micro>(t1 - t0).count();
    stats.kernel_launches = launches_so_far() - launches0;
    if (st) *st = stats;
    return guard.release();
}

} // namespace

cj_result *execute_plan(Context &ctx, const cj_plan_desc &plan, uint32_t flags, cj_exec_stats *stats) {
    struct Range {
        Range() { nvtxRangePushA("cj_execute"); }
        ~Range() { nvtxRangePop(); }
    } range;
    Executor ex(ctx, plan, flags);
    return ex.run(stats);
}

} // namespace cj
