// db_internal.h -- the device-resident database as the runtime translation units see it.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <vector>

#include "host_common.h"
#include "scan_kernel.cuh"

namespace hy {

// Launch shapes. Main scan: int16x2 pairs in groups of MAIN_G lanes with MAIN_R16 query rows per
// lane; int32 items (the long sequences) one full warp each. The band kernel (long items, a winner's
// ends): one warp per band of WIN_G * BAND_FEW_ROWS query rows, or WIN_G * WIN_R in the batched form.
constexpr int MAIN_G = 8;
constexpr int MAIN_R16 = 16;
constexpr int MAIN_G32 = 32;
constexpr int MAIN_R32 = 16;
constexpr int WIN_G = 32;
constexpr int WIN_R = 8;
constexpr int BAND_FEW_ROWS = 4;  // rows per lane of a scan's or a long pair's band
// The batched form's pairs longer than LONG_W columns run one full warp each (LONG_G lanes of
// LONG_R rows) in a class of their own, whose boundary regions the bulk classes then need not
// size for. Plain scans split their pairs by estimated time instead (scan_forms).
constexpr int LONG_G = 32;
constexpr int LONG_R = 8;
constexpr uint32_t LONG_W = 4096;
constexpr uint32_t NO_LONG_SPLIT = 0xffffffffu;
constexpr int BLOCK = 256;
// Rows per lane of the bulk int16x2 kernel for a query of length qlen (passes of MAIN_G * rows): the
// two-column sweep at 8 or 16 rows per lane, 16 unless 8 pads the query to so many fewer rows that it
// wins at 8 rows' rate per padded row (measured 0.853 of 16 rows' rate, 4813 against 5641 GCUPS for
// 1000-residue queries on the protein benchmark: 150 residues take 192 rows at 8 against 256 at 16).
inline int bulk_rows(uint64_t qlen, bool local_ends = false) {
    if (qlen <= 64) return 8;
    if (local_ends) return 16;  // the two-column sweep tracks ends from 12 rows per lane on
    const uint64_t rows8 = (qlen + 63) / 64 * 64, rows16 = (qlen + 127) / 128 * 128;
    return 7 * rows8 < 6 * rows16 ? 8 : 16;
}
// Rows of a pass slice that LayoutChoice::Auto sizes the pair table for.
constexpr int BULK_MAX_RPP = 8 * 32;
constexpr int WIDE_MAX_RPP = 32 * 16;
constexpr size_t BAND_SMEM_BUDGET = 200 * 1024;
// Shared memory of an SM (B200), and what each resident block reserves of it.
constexpr size_t SM_SMEM = 228 * 1024, BLOCK_SMEM_RESERVE = 1024;
// Blocks of one band-kernel cluster at most (the portable cluster size).
constexpr int BAND_CLUSTER_MAX = 8;

// One long pair's BestHit cell on the band kernel (int32 lanes): the query already on the device
// (d_q, m residues), the target on the host (t, tl residues, copied here). Writes the score and the
// 0-based query and target ends (-1 for row or column 0) at index `slot` of d_scores / d_qend /
// d_tend on stream `st` and waits for them; adds the band kernel's time to *kernel_ms.
// Whether a long pair with an m-residue query runs its band passes in one round of one block or
// cluster (band_long_pair's shape); longer queries take the stripe kernel.
bool band_long_pair_fits(uint64_t m, uint64_t al);
hy_status band_long_pair(const uint8_t *d_q, uint64_t m, const uint8_t *t, uint64_t tl, const int32_t *d_matrix,
                         uint64_t al, int32_t go, int32_t ge, int mode, cudaStream_t st, uint32_t slot,
                         int32_t *d_scores, int32_t *d_qend, int32_t *d_tend, double *kernel_ms);
// The same for a lone pair whose query, target and matrix are on the host (align_pair's direct
// path): one copy in, the profile and band kernels, one copy out. out = {score, query end, target
// end}.
hy_status band_single_pair(const uint8_t *q, uint64_t m, const uint8_t *t, uint64_t tl, const int32_t *matrix,
                           uint64_t al, int32_t go, int32_t ge, int mode, int32_t out[3], double *kernel_ms);

struct Partition {
    uint32_t n_items = 0;
    uint64_t n_seqs = 0;
    uint64_t total_cols = 0;
    std::vector<uint64_t> res_prefix;  // host: residues of items [0, i) (both halves of a pair)
    ItemMeta *d_meta = nullptr;
    void *d_res = nullptr;
};

template <class A>
struct ElemSize {
    static constexpr size_t pe = sizeof(typename A::PE);
};

struct QueryPlan {
    int32_t n_passes = 0;
    int32_t vrow0 = 1;
    uint32_t pass_bytes = 0;
};

inline QueryPlan plan(uint64_t qlen, int rpp, uint64_t al, size_t pe) {
    QueryPlan q;
    q.n_passes = (int32_t)((qlen + rpp - 1) / rpp);
    q.vrow0 = (int32_t)qlen - q.n_passes * rpp + 1;
    q.pass_bytes = (uint32_t)((al + 1) * (uint64_t)rpp * pe);
    return q;
}

// The plan of lane arithmetic A (its profile has A::letters(al) letters per table).
template <class A>
inline QueryPlan plan_for(uint64_t qlen, int rpp, uint64_t al) {
    QueryPlan q = plan(qlen, rpp, al, profile_row_bytes<A>());
    q.pass_bytes = (uint32_t)(profile_slice_row_bytes<A>((int64_t)al) * (uint64_t)rpp);
    return q;
}

}  // namespace hy

struct hy_db {
    int device = 0;
    // Largest dynamic shared memory one block may use on the device (opt-in): launch shapes whose
    // query-profile slices exceed it read the profile from global memory instead.
    size_t smem_limit = 48 * 1024;
    uint64_t n_seqs = 0, mql = 0, max_t = 0, al = 0;
    int32_t go = 0, ge = 0, min_e = 0, max_e = 0;
    int mode = 0, search_type = 0, layout = HY_LAYOUT_GATHERED;
    hy_score_width width = HY_WIDTH_I8;
    hy_backend backend = HY_BACKEND_CUDA;
    int32_t *d_matrix = nullptr;
    // Every sequence in int16x2 pairs over the global length order (longest first); the longest
    // ones (those the whole-database proof cannot place in int16) also as int32 singles.
    hy::Partition p16, p32;
    std::vector<uint32_t> pair_w;  // host: longer length of each pair, non-increasing
    uint32_t *d_rank = nullptr;    // device: rank of each global index in the length order
    uint64_t device_bytes = 0;
    // Alignment search type: its budget, and every sequence's residues in db order (sequence k is
    // d_tb_res[tb_off[k] .. tb_off[k+1]]), the targets of the traceback.
    uint64_t tb_max_bytes = 0;
    uint8_t *d_tb_res = nullptr;
    std::vector<uint64_t> tb_off;
};

namespace hy {

// The extents a bounds-checked build (HY_BOUNDS) verifies each item of `part` against: the
// partition's residue columns, `bnd_cols` columns of boundary region, the database's indices and
// the profile letters of lane arithmetic A.
template <class A>
inline void set_extents(ScanParams &p, const hy_db *db, const Partition &part, uint64_t bnd_cols) {
    p.res_cols = part.total_cols;
    p.bnd_cols = bnd_cols;
    p.n_seqs = (uint32_t)db->n_seqs;
    p.letters = (uint32_t)A::letters((int64_t)db->al);
}

// Which items one query runs in which lanes. The width proof is redone with the actual query
// length: pairs [k0, n) fit int16 for this query and run packed; the 2*k0 longest sequences run
// in int32 (always inside the int32 layout, which holds the static int32 set plus one).
struct QuerySplit {
    uint32_t k0 = 0;      // first int16x2 pair item
    uint32_t kl = 0;      // pairs [k0, kl) are long (one warp each), [kl, n) the bulk
    uint32_t n_i32 = 0;   // int32 items [0, n_i32)
};

inline QuerySplit split_for_query(const hy_db *db, uint64_t qlen, uint32_t long_w = NO_LONG_SPLIT) {
    QuerySplit q;
    // Longest target length t whose bound for this query keeps the int16 kernel exact.
    auto fits = [&](uint64_t n) {
        return device_fits_i16(magnitude_bound(db->mode, db->min_e, db->max_e, db->go, db->ge, qlen, n), db->go);
    };
    uint64_t t;
    if (fits(db->max_t)) {
        t = db->max_t;
    } else {
        uint64_t lo = 0, hi = db->max_t;  // fits(lo) may be false only if even length 0 fails
        if (!fits(0)) {
            t = 0;
            lo = hi = 0;
        }
        while (lo < hi) {
            uint64_t mid = lo + (hi - lo + 1) / 2;
            if (fits(mid)) lo = mid; else hi = mid - 1;
        }
        t = lo;
    }
    // First pair whose longer sequence is <= t (pair_w is non-increasing).
    uint32_t a = 0, b = (uint32_t)db->pair_w.size();
    while (a < b) {
        uint32_t mid = a + (b - a) / 2;
        if (db->pair_w[mid] <= t) b = mid; else a = mid + 1;
    }
    q.k0 = a;
    q.n_i32 = (uint32_t)std::min<uint64_t>(2ull * a, db->n_seqs);
    b = (uint32_t)db->pair_w.size();
    while (a < b) {
        uint32_t mid = a + (b - a) / 2;
        if (db->pair_w[mid] <= long_w) b = mid; else a = mid + 1;
    }
    q.kl = a;
    return q;
}

// Which pairs of a scan leave the bulk kernel for forms that finish one item sooner, and the int32
// items' form (host only, from lengths alone). An item is one serial chain: in the bulk kernel on 8
// lanes; in the wide form a warp (16 lanes for queries of at most 64 residues), a quarter of the
// chain; in the band kernel a warp for every 128 query rows. The forms that finish sooner spend more
// instructions a cell, so the split is the one of least estimated time. 50,000 protein sequences, best
// hit with ends: a query of 350 residues 5.7 to 1.7 ms, of 5000 30.1 to 20.6; every target's ends, 500:
// 10.7 to 2.9.
struct ScanForms {
    uint32_t band_end = 0;  // pairs [k0, band_end): the band kernel
    uint32_t wide_end = 0;  // pairs [band_end, wide_end): the wide form; [wide_end, n): the bulk kernel
    int wide_g = 32, wide_r = 8;
    bool band32 = false;  // the int32 items: the band kernel, else a warp each
};

// Lanes and rows per lane of the wide form: one pass of the fewest rows up to 512 rows, longer queries
// in passes of 512 or 256 rows by padded rows at their rates (8 rows 0.853 of 16 rows'). (12 rows
// against 16: a scan of 350 residues x 50,000 proteins 1.62 and 1.81 ms, every target's ends 2.05 and 2.16.)
inline void wide_shape(uint64_t qlen, int *g, int *r) {
    *g = qlen <= 64 ? 16 : 32;
    if (qlen <= 128) *r = 4;
    else if (qlen <= 256) *r = 8;
    else if (qlen <= 384) *r = 12;
    else if (qlen <= 512) *r = 16;
    else *r = 7 * ((qlen + 255) / 256 * 256) < 6 * ((qlen + 511) / 512 * 512) ? 8 : 16;
}

// What the estimate is made of, fitted to measured kernels: a warp's instructions a step (one step of
// two columns of r rows: 292 for 16 rows, 171 for 8; one column 9 a row, 13 with ends; the band's 100),
// cycles an instruction of a scheduler with 4 warps (1.46) and of a lone warp (2.2), and what one more
// kernel and its query profile take (cycles).
struct ScanCost {
    int mode;
    bool ends;
    // Instructions of one item's chain: passes of g * r rows over w columns.
    double chain(uint64_t qlen, int g, int r, double w) const {
        const double passes = (double)((qlen + (uint64_t)(g * r) - 1) / (uint64_t)(g * r));
        if (!scan_two_col_rows(r, mode, ends)) return passes * (w + g) * (50.0 + 13.0 * r);
        return (passes * w / 2 + g) * (mode != MODE_SW ? 55.0 + 14.1 * r : (ends ? 110.0 : 50.0) + 15.1 * r);
    }
};
constexpr double COST_SCHEDULERS = 148 * 4, COST_BUSY = 1.46, COST_ALONE = 2.2, COST_FORM = 16000;
inline double band_chain(uint64_t qlen, double w) {
    return (w / 2 + 51 + 48 * (double)((qlen - 1) / 128)) * 100;
}
// A band's warps hold their places for the whole chain, busy or not: 134 to 152 busy-rate instructions a
// step measured (72 items of 40 passes, 1093 of 3).
inline double band_work(uint64_t qlen, double w) { return (double)((qlen + 127) / 128) * band_chain(qlen, w) * 1.5; }

// Estimated cycles of `work` warp-instructions: the chip at its busy rate, then what is left of the
// bulk's longest chain alone (`warps` bulk warps; `full`: the chain behind one warp a scheduler). The
// other forms start first and their warps, the oldest of a scheduler, run nearly as if alone beside the
// bulk: the longest of those bounds it, at 2.35 cycles an instruction (int32 chains of 12.1 M took 14.5
// ms) or, a warp a pair, at 3.0 (blocks of 8 warps) or 3.7 (of 16: 4.0 M took 7.5 ms).
struct ScanLoad {
    double work = 0, bulk_warps = 0, bulk_chain = 0, full = 0, side_warps = 0, side_chain = 0, forms = 0;  // side_chain: cycles
    double time() const {
        const double busy = work / COST_SCHEDULERS * COST_BUSY;
        const double rate = std::max(COST_ALONE, COST_BUSY * std::min(4.0, (bulk_warps + side_warps) / COST_SCHEDULERS));
        const double bulk = std::max(busy, full * COST_ALONE) + std::max(0.0, bulk_chain - std::max(busy / rate, full)) * COST_ALONE;
        const double side = side_chain * std::max(1.0, COST_BUSY / 2.35 * std::min(4.0, side_warps / COST_SCHEDULERS));
        return std::max(bulk, side) + forms * COST_FORM;
    }
};

// hold, hold32: what bands of pairs and of int32 items take beyond band_work, at least 1.
inline ScanForms scan_forms(const hy_db *db, const QuerySplit &split, uint64_t qlen, bool ends, int bulk_r,
                            int wide_g, int wide_r, int wide_threads, double hold, double hold32) {
    ScanForms f;
    f.wide_g = wide_g;
    f.wide_r = wide_r;
    const ScanCost cost{db->mode, ends};
    const uint32_t k0 = split.k0, n = db->p16.n_items;
    f.band_end = f.wide_end = k0;
    if (qlen == 0 || (k0 >= n && split.n_i32 == 0)) return f;
    auto width = [&](uint32_t i) { return i < n ? (double)db->pair_w[i] : 0.0; };
    auto mean = [&](uint32_t a, uint32_t b) {  // mean columns of pairs [a, b)
        return b > a ? (double)(db->p16.res_prefix[b] - db->p16.res_prefix[a]) / 2 / (b - a) : 0.0;
    };
    // The int32 items: chains and work of both forms (their widths are the longest pairs').
    const double w32 = split.n_i32 ? width(0) : 0.0, mean32 = mean(0, (split.n_i32 + 1) / 2);
    auto time = [&](uint32_t band, uint32_t wide, bool band32) {
        ScanLoad l;
        auto side = [&](double count, double lanes, double each, double longest, double rate) {
            if (count <= 0) return;
            l.work += count * each * lanes / 32;
            l.side_warps += count * lanes / 32;
            l.side_chain = std::max(l.side_chain, longest * rate);
            l.forms += 1;
        };
        if (band32) side(split.n_i32, 32, band_work(qlen, mean32), band_chain(qlen, w32), 2.35);
        else side(split.n_i32, 32, cost.chain(qlen, 32, MAIN_R32, mean32), cost.chain(qlen, 32, MAIN_R32, w32), 2.35);
        side(band - k0, 32, band_work(qlen, mean(k0, band)), band_chain(qlen, width(k0)), 2.35);
        side(wide - band, f.wide_g, cost.chain(qlen, f.wide_g, f.wide_r, mean(band, wide)),
             cost.chain(qlen, f.wide_g, f.wide_r, width(band)), wide_threads > BLOCK ? 3.7 : 3.0);
        if (wide < n) {
            const double count = n - wide;
            l.work += count * cost.chain(qlen, MAIN_G, bulk_r, mean(wide, n)) * MAIN_G / 32;
            l.bulk_warps = count * MAIN_G / 32;
            l.bulk_chain = cost.chain(qlen, MAIN_G, bulk_r, width(wide));
            const uint32_t i = wide + (uint32_t)COST_SCHEDULERS * (32 / MAIN_G);
            if (i < n) l.full = cost.chain(qlen, MAIN_G, bulk_r, width(i));
            l.forms += 1;
        }
        return l.time();
    };
    // Candidate splits: none, then pairs longer than 0.8^i of the longest, then all.
    uint32_t cand[24];
    int n_cand = 0;
    double w = width(k0);
    for (cand[n_cand++] = k0; n_cand < 23 && k0 < n; ++n_cand) {
        w *= 0.8;
        cand[n_cand] = (uint32_t)(std::partition_point(db->pair_w.begin() + k0, db->pair_w.end(),
                                                       [&](uint32_t x) { return (double)x > w; }) -
                                  db->pair_w.begin());
    }
    cand[n_cand++] = n;
    double best = time(k0, k0, false);
    // The int32 items' form, then the wide split, then the band split under it, then the wide one again.
    if (split.n_i32) {
        const double t = time(k0, k0, true);
        if (t < best) best = t, f.band32 = true;
    }
    for (int round = 0; round < 2; ++round) {
        for (int i = 0; i < n_cand; ++i) {
            if (cand[i] < f.band_end) continue;
            const double t = time(f.band_end, cand[i], f.band32);
            if (t < best) best = t, f.wide_end = cand[i];
        }
        if (round == 0)
            for (int i = 0; i < n_cand; ++i) {
                const double t = time(cand[i], std::max(cand[i], f.wide_end), f.band32);
                if (t < best) best = t, f.band_end = cand[i];
            }
        f.wide_end = std::max(f.wide_end, f.band_end);
    }
    if (split.n_i32) {
        const double t = time(f.band_end, f.wide_end, !f.band32);
        if (t < best) f.band32 = !f.band32;
    }
    // Bands whose blocks leave a scheduler few warps stay only where they are still the sooner form of the
    // items they took, by themselves.
    auto alone = [](double count, double work, double chain) {
        return std::max(count * work / COST_SCHEDULERS * COST_BUSY, chain);
    };
    if (f.band32 && hold32 > 1.0 &&
        alone(split.n_i32, band_work(qlen, mean32) * hold32, band_chain(qlen, w32) * 2.35) >
            alone(split.n_i32, cost.chain(qlen, 32, MAIN_R32, mean32), cost.chain(qlen, 32, MAIN_R32, w32) * 2.35))
        f.band32 = false;
    const double bands = f.band_end - k0, mean16 = mean(k0, f.band_end);
    if (bands > 0 && hold > 1.0 &&
        alone(bands, band_work(qlen, mean16) * hold, band_chain(qlen, width(k0)) * 2.35) >
            alone(bands, cost.chain(qlen, f.wide_g, f.wide_r, mean16) * f.wide_g / 32,
                  cost.chain(qlen, f.wide_g, f.wide_r, width(k0)) * (wide_threads > BLOCK ? 3.7 : 3.0)))
        f.band_end = k0;
    return f;
}

}  // namespace hy

