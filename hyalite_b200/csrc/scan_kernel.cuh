// scan_kernel.cuh -- the device side of the inter-sequence database scan.
//
// One "item" is either a PAIR of database sequences packed into the two int16 halves of every
// 32-bit register (Pair16), or ONE sequence in int32 lanes (Single32). A group of G consecutive
// lanes of a warp runs one item: lane L owns R consecutive query rows of the current pass and
// sweeps the item's columns one step behind lane L-1 (an anti-diagonal wavefront); the H and F
// values of a lane's last row move to the next lane with one shuffle each per step. A pass covers
// G*R query rows; the last row of a pass is handed to the next pass through a boundary row in
// global memory. The query profile of the current pass is staged into shared memory by a TMA bulk
// copy (cp.async.bulk) with an mbarrier, double-buffered across passes.
//
// The recurrence is the Gotoh recurrence of the scalar oracle (src/kernel.rs:168-217):
//   E[i][j] = max(E[i][j-1] - ge, H[i][j-1] - go)
//   F[i][j] = max(F[i-1][j] - ge, H[i-1][j] - go)
//   H[i][j] = max(H[i-1][j-1] + sub(q_i, t_j), E[i][j], F[i][j])   (SW: also max with 0)
// carried as G = H - go, with the profile holding P = sub + go so that G_diag + P = H_diag + sub:
//   E = max(E + (-ge), G_left)           __viaddmax            (ALU pipe)
//   F = max(F + (-ge), G_up)             __viaddmax            (ALU)
//   d = G_diag + P                       __vadd2 (x2 for the two Gathered tables)   (FMA pipe)
//   H = max(d, E, F)                     __vimax3 (SW: __vimax3_relu)               (ALU)
//   G = H + (-go)                        __vadd2               (FMA)
// For SW scores the row-to-row chain is shortened to one op (see sweep_step).
// Width safety: the host routes a sequence to Pair16 only when its magnitude bound plus gap_open
// fits int16 (bound + go <= 32767), which keeps every intermediate above exactly representable,
// so the packed arithmetic never wraps on a real cell and the results equal the i32 oracle.
//
// Rows: the query is padded at the FRONT so the last query row always sits in the last slot of
// the last lane of the last pass. Virtual rows (index <= 0) reproduce the border row 0 exactly:
// left border 0 and a profile value of `go` (free top border) or 0 (penalised top border).
// Columns: in a Pair16 item the shorter sequence is padded with a symbol whose profile value is
// the most negative representable; padded columns never feed a real cell and are excluded from
// every answer region (or, for SW, can only tie a real cell at a larger column).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace hy {

enum { MODE_SW = 0, MODE_NW = 1, MODE_HW = 2, MODE_OV = 3, MODE_SHW = 4 };

// Flags::for_mode (src/kernel.rs:43-98).
template <int MODE>
struct ModeFlags {
    static constexpr bool top_free = MODE == MODE_SW || MODE == MODE_HW || MODE == MODE_OV;
    static constexpr bool left_free = MODE == MODE_SW || MODE == MODE_OV || MODE == MODE_SHW;
    static constexpr bool last_row = MODE == MODE_HW || MODE == MODE_OV;
    static constexpr bool last_col = MODE == MODE_OV || MODE == MODE_SHW;
    static constexpr bool local = MODE == MODE_SW;
    static constexpr bool corner = MODE == MODE_NW;
};

struct ItemMeta {
    uint64_t col_off;  // first column of the item in the residue / boundary arrays
    uint32_t w;        // columns swept (the longer length of the pair)
    uint32_t n[2];     // sequence lengths; a lone sequence has n[1] = 0 and idx[1] = NO_INDEX
    uint32_t idx[2];   // global db indices
    uint32_t pad_;
};
static constexpr uint32_t NO_INDEX = 0xffffffffu;

struct ScanParams {
    const ItemMeta *meta;
    uint32_t item_base;        // first item of the launch: items [item_base, n_items) run
    uint32_t n_items;
    const uint32_t *item_ptr;  // when set: run the single item *item_ptr (NO_INDEX: nothing)
    const void *res;           // Pair16: uint16 (lo | hi << 8); Single32: uint8
    const uint8_t *profile;    // pass-major profile slices, pass_bytes each
    uint32_t pass_bytes;
    int32_t n_passes;
    int32_t vrow0;  // grid row of pass 0, lane 0, slot 0 (<= 1)
    int32_t qlen;
    int32_t go, ge;
    int32_t sentinel;
    void *boundary;     // 2 values (G, F) per column, starting at column bnd_col0
    uint64_t bnd_col0;  // first column the boundary region covers
    int32_t *scores;    // per-target outputs by global index (may be null: best key only)
    int32_t *qend;
    int32_t *tend;
    unsigned long long *best_key;
    int *err;
    // Band recovery only: when set, the winner named by *best_key is written here as {score,
    // query end, target end} instead of to scores / qend / tend.
    int32_t *ends_out;
    uint32_t wait_polls;  // polls a wait for a profile copy makes before it gives up
    uint32_t row_polls;   // polls a band block waits for its neighbour's rows, or for ring space there
    // Extents the bounds-checked build (HY_BOUNDS) verifies every item against before use.
    uint64_t res_cols;  // columns of the residue array
    uint64_t bnd_cols;  // columns the boundary region holds, from bnd_col0
    uint32_t n_seqs;    // db indices are below this
    uint32_t letters;   // profile letters per table (the last is the padding symbol)
};

// Error words a kernel leaves in ScanParams::err: a bounded wait gave up, or (bounds-checked
// build) an item failed its check and was skipped.
enum { ERR_WAIT = 1, ERR_BOUNDS = 2 };

// ---- lane arithmetic -----------------------------------------------------------------------
//
// Per cell the recurrence issues three ops on the ALU pipe (two __viaddmax for E and F, one
// __vimax3 for H) and, for int16x2, three on the FMA pipe (__vadd2 for the diagonal's two profile
// words and for G = H - go); the two half-rate pipes run in parallel.

struct Pair16 {
    typedef uint32_t V;
    // Profile words: a low-half table holding (P, 0) and a high-half table holding (0, P), so the
    // two sequences' substitution values are merged by per-halfword adds on the FMA pipe.
    typedef uint32_t PE;
    typedef uint16_t RES;
    static constexpr int NH = 2;
    static constexpr int EPV = 4;     // profile words per 16-byte vector
    static constexpr int TABLES = 2;  // per pass slice: the low-half table, then the high-half one
    static constexpr int32_t VMIN = -32768, VMAX = 32767;
    __device__ __forceinline__ static V splat(int64_t x) {
        x = x < VMIN ? VMIN : (x > VMAX ? VMAX : x);
        uint32_t h = (uint16_t)(int16_t)x;
        return h | (h << 16);
    }
    // splat of a value that fits.
    __device__ __forceinline__ static V pack(int32_t x) { return __byte_perm((uint32_t)x, 0, 0x1010); }
    __device__ __forceinline__ static V addmax(V a, V b, V c) { return __viaddmax_s16x2(a, b, c); }
    __device__ __forceinline__ static V vmax(V a, V b) { return __vmaxs2(a, b); }
    __device__ __forceinline__ static V vmax3(V a, V b, V c) { return __vimax3_s16x2(a, b, c); }
    __device__ __forceinline__ static V vmax3_relu(V a, V b, V c) { return __vimax3_s16x2_relu(a, b, c); }
    __device__ __forceinline__ static V vadd(V a, V b) { return __vadd2(a, b); }
    __device__ __forceinline__ static V diag(V g, V pa, V pb) { return __vadd2(__vadd2(g, pa), pb); }
    __device__ __forceinline__ static int32_t get(V v, int h) {
        return h ? (int32_t)(int16_t)(v >> 16) : (int32_t)(int16_t)(v & 0xffffu);
    }
    // Running maximum; up[h] is set where x is strictly greater than best in half h.
    __device__ __forceinline__ static V bmax(V best, V x, bool &up0, bool &up1) {
        bool ph, pl;
        V r = __vibmax_s16x2(best, x, &ph, &pl);
        up0 = !pl;
        up1 = !ph;
        return r;
    }
    __device__ __forceinline__ static void residues(RES r, int &a, int &b) {
        a = r & 0xff;
        b = r >> 8;
    }
    // Chunk k (EPV rows) of the profile for letters (a, b): prof_lo is the low-half table used by
    // the low sequence, prof_hi the high-half table used by the high sequence.
    template <int R, int G>
    __device__ __forceinline__ static void load_chunk(const uint8_t *prof_lo, const uint8_t *prof_hi,
                                                      int a, int b, int lane, int k, V (&pa)[EPV],
                                                      V (&pb)[EPV]) {
        constexpr int KCH = R / EPV;
        const uint4 A = reinterpret_cast<const uint4 *>(prof_lo)[((size_t)a * KCH + k) * G + lane];
        const uint4 B = reinterpret_cast<const uint4 *>(prof_hi)[((size_t)b * KCH + k) * G + lane];
        pa[0] = A.x; pa[1] = A.y; pa[2] = A.z; pa[3] = A.w;
        pb[0] = B.x; pb[1] = B.y; pb[2] = B.z; pb[3] = B.w;
    }
    // The profile word of value v in table t (0: low half, 1: high half).
    __host__ __device__ __forceinline__ static PE word(int64_t v, int t) {
        const uint32_t h = (uint16_t)(int16_t)v;
        return t ? (h << 16) : h;
    }
    // Profile letters of an alphabet of `al` symbols (the padding symbol included).
    static constexpr bool PAIRTAB = false;
    __host__ __device__ static constexpr int64_t letters(int64_t al) { return al + 1; }
    // Residue code of a pair column (low sequence's symbol lo, high sequence's hi).
    __host__ __device__ static constexpr uint32_t code(uint32_t lo, uint32_t hi, uint32_t) { return lo | (hi << 8); }
    // The padding column's residue code, of a profile of `letters` letters.
    __host__ __device__ static constexpr uint32_t pad_code(uint32_t letters) { return (letters - 1) * 0x101u; }
};

// The int16x2 arithmetic with a half-size query profile, for kernels whose groups each keep their
// own profile in shared memory (the pair kernel): each table holds 16-bit entries, and a row's
// word is assembled from the two tables' entries by one byte permute instead of merging two 32-bit
// words by an add. The same values; half the shared memory, so twice the groups fit on an SM.
struct Pair16H : Pair16 {
    typedef uint16_t PE;
    __device__ __forceinline__ static V diag(V g, V p, V) { return __vadd2(g, p); }
    template <int R, int G>
    __device__ __forceinline__ static void load_chunk(const uint8_t *prof_lo, const uint8_t *prof_hi,
                                                      int a, int b, int lane, int k, V (&pa)[EPV],
                                                      V (&pb)[EPV]) {
        constexpr int KCH = R / EPV;
        const uint2 A = reinterpret_cast<const uint2 *>(prof_lo)[((size_t)a * KCH + k) * G + lane];
        const uint2 B = reinterpret_cast<const uint2 *>(prof_hi)[((size_t)b * KCH + k) * G + lane];
        // Row 2i: the low entries of both tables' word i; row 2i + 1: the high entries.
        pa[0] = __byte_perm(A.x, B.x, 0x5410);
        pa[1] = __byte_perm(A.x, B.x, 0x7632);
        pa[2] = __byte_perm(A.y, B.y, 0x5410);
        pa[3] = __byte_perm(A.y, B.y, 0x7632);
        pb[0] = pb[1] = pb[2] = pb[3] = 0;
    }
    __host__ __device__ __forceinline__ static PE word(int64_t v, int) { return (uint16_t)(int16_t)v; }
};

// The Precomputed layout (src/inter.rs:317-330: "a precomputed score table, so each cell's
// substitution vector is a direct load with no gather"), restated for the device: the database
// stores each pair column as one code c = lo * (al + 1) + hi, and the pass's profile is a single
// table indexed by (c, query row) whose word already holds both halves' substitution values. A
// cell pair then costs one profile load and one add instead of two of each; the table has
// (al + 1)^2 letters, so it is compact for small alphabets only. Arithmetic as Pair16.
struct PairTab16 : Pair16 {
    static constexpr int TABLES = 1;
    static constexpr bool PAIRTAB = true;
    __host__ __device__ static constexpr int64_t letters(int64_t al) { return (al + 1) * (al + 1); }
    __host__ __device__ static constexpr uint32_t code(uint32_t lo, uint32_t hi, uint32_t al) {
        return lo * (al + 1) + hi;
    }
    __host__ __device__ static constexpr uint32_t pad_code(uint32_t letters) { return letters - 1; }
    __device__ __forceinline__ static V diag(V g, V p, V) { return __vadd2(g, p); }
    __device__ __forceinline__ static void residues(RES r, int &a, int &b) {
        a = r;
        b = 0;
    }
    template <int R, int G>
    __device__ __forceinline__ static void load_chunk(const uint8_t *prof, const uint8_t *, int c,
                                                      int, int lane, int k, V (&pa)[EPV],
                                                      V (&pb)[EPV]) {
        constexpr int KCH = R / EPV;
        const uint4 A = reinterpret_cast<const uint4 *>(prof)[((size_t)c * KCH + k) * G + lane];
        pa[0] = A.x; pa[1] = A.y; pa[2] = A.z; pa[3] = A.w;
        pb[0] = pb[1] = pb[2] = pb[3] = 0;
    }
    // The word of a pair code's two values (low half: the low sequence's).
    __host__ __device__ __forceinline__ static PE pair_word(int64_t lo, int64_t hi) {
        return (uint32_t)(uint16_t)(int16_t)lo | ((uint32_t)(uint16_t)(int16_t)hi << 16);
    }
};

struct Single32 {
    typedef int32_t V;
    typedef int32_t PE;
    typedef uint8_t RES;
    static constexpr int NH = 1;
    static constexpr int EPV = 4;
    static constexpr int TABLES = 1;
    static constexpr int64_t VMIN = INT32_MIN, VMAX = INT32_MAX;
    __device__ __forceinline__ static V splat(int64_t x) {
        return (V)(x < VMIN ? VMIN : (x > VMAX ? VMAX : x));
    }
    __device__ __forceinline__ static V pack(int32_t x) { return x; }
    __device__ __forceinline__ static V addmax(V a, V b, V c) { return __viaddmax_s32(a, b, c); }
    __device__ __forceinline__ static V vmax(V a, V b) { return max(a, b); }
    __device__ __forceinline__ static V vmax3(V a, V b, V c) { return __vimax3_s32(a, b, c); }
    __device__ __forceinline__ static V vmax3_relu(V a, V b, V c) { return __vimax3_s32_relu(a, b, c); }
    __device__ __forceinline__ static V vadd(V a, V b) { return a + b; }
    __device__ __forceinline__ static V diag(V g, V pa, V) { return g + pa; }
    __device__ __forceinline__ static int32_t get(V v, int) { return v; }
    __device__ __forceinline__ static V bmax(V best, V x, bool &up0, bool &up1) {
        bool p;
        V r = __vibmax_s32(best, x, &p);
        up0 = !p;
        up1 = false;
        return r;
    }
    __device__ __forceinline__ static void residues(RES r, int &a, int &b) {
        a = r;
        b = r;
    }
    template <int R, int G>
    __device__ __forceinline__ static void load_chunk(const uint8_t *prof, const uint8_t *, int a,
                                                      int, int lane, int k, V (&pa)[EPV],
                                                      V (&pb)[EPV]) {
        constexpr int KCH = R / EPV;
        const int4 A = reinterpret_cast<const int4 *>(prof)[((size_t)a * KCH + k) * G + lane];
        pa[0] = A.x; pa[1] = A.y; pa[2] = A.z; pa[3] = A.w;
        pb[0] = pb[1] = pb[2] = pb[3] = 0;
    }
    __host__ __device__ __forceinline__ static PE word(int64_t v, int) { return (PE)v; }
    static constexpr bool PAIRTAB = false;
    __host__ __device__ static constexpr int64_t letters(int64_t al) { return al + 1; }
    __host__ __device__ static constexpr uint32_t pad_code(uint32_t letters) { return letters - 1; }
};

// Profile bytes per (letter, query row) of one lane arithmetic: every table's word.
template <class A>
__host__ __device__ constexpr size_t profile_row_bytes() {
    return A::TABLES * sizeof(typename A::PE);
}

// Profile bytes of one query row of a pass slice: every letter of every table.
template <class A>
__host__ __device__ constexpr size_t profile_slice_row_bytes(int64_t al) {
    return (size_t)A::letters(al) * profile_row_bytes<A>();
}

// ---- small helpers -------------------------------------------------------------------------

// gap_penalty (src/kernel.rs:103-109).
__device__ __forceinline__ int64_t gap_pen(int32_t go, int32_t ge, int64_t len) {
    return len <= 0 ? 0 : (int64_t)go + (len - 1) * (int64_t)ge;
}

// Answer candidate under the tie-break of Best::consider (src/kernel.rs:113-129): higher score,
// then smaller grid column, then smaller grid row.
struct Cand {
    int32_t s;
    int32_t col;
    int32_t row;
};
__device__ __forceinline__ bool better(const Cand &a, const Cand &b) {
    return a.s > b.s || (a.s == b.s && (a.col < b.col || (a.col == b.col && a.row < b.row)));
}
__device__ __forceinline__ void consider(Cand &b, int32_t s, int32_t col, int32_t row) {
    Cand c = {s, col, row};
    if (better(c, b)) b = c;
}

// Best border-cell candidate of the mode's answer region (reduce_answer, src/kernel.rs:223-260,
// restricted to row 0 and column 0), for query length m and target length n.
template <int MODE>
__device__ __forceinline__ Cand border_seed(int32_t m, int32_t n, int32_t go, int32_t ge) {
    const Cand none = {INT32_MIN, INT32_MAX, INT32_MAX};
    switch (MODE) {
    case MODE_SW: return {0, 0, 0};
    case MODE_NW:
        if (m == 0) return {(int32_t)-gap_pen(go, ge, n), n, 0};
        if (n == 0) return {(int32_t)-gap_pen(go, ge, m), 0, m};
        return none;
    case MODE_HW:
        if (m == 0) return {0, 0, 0};
        return {(int32_t)-gap_pen(go, ge, m), 0, m};
    case MODE_SHW:
        if (n == 0) return {0, 0, 0};
        return {(int32_t)-gap_pen(go, ge, n), n, 0};
    default: /* OV */
        if (m == 0 || n == 0) return {0, 0, 0};
        return {0, 0, m};
    }
}

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// Issue one TMA bulk copy global -> shared whose completion is tracked by `bar`.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, "
        "0, p;\n}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: gives up after `polls` polls (each poll may itself suspend briefly).
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, uint32_t parity, uint32_t polls) {
    for (uint32_t it = 0; it < polls; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// After a wait gave up (one thread of the block): records the timeout and lets the copies still
// in flight into the block's shared memory land before the block exits (bounded again, by the
// default number of polls; the block's shared memory stays allocated while this thread runs).
// `pending` holds the barriers with a copy outstanding (bit b: bars[b]) and `phase` the parity
// each waits for. Out of line: the scan kernels' hot loops keep their register allocation.
static __device__ __noinline__ void wait_gave_up(int *err, uint64_t *bars, uint32_t pending, uint32_t phase) {
    atomicExch(err, ERR_WAIT);
    for (int b = 0; b < 2; ++b)
        if ((pending >> b) & 1u) mbar_wait_bounded(&bars[b], (phase >> b) & 1u, 1u << 24);
}

// ---- thread-block clusters (the band kernel's blocks) -----------------------------------------
// A block not launched as part of a cluster is a cluster of one: rank 0 of 1.
__device__ __forceinline__ int cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return (int)r;
}
__device__ __forceinline__ int cluster_size() {
    uint32_t n;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
    return (int)n;
}
// Every thread of every block of the cluster; orders memory at cluster scope (release, acquire).
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The 32-bit word at the address of `p` in the shared memory of block `rank` of the cluster.
__device__ __forceinline__ uint32_t ld_cluster_u32(const void *p, int rank) {
    uint32_t a, v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
// The address of `p` in the shared memory of block `rank` of the cluster.
__device__ __forceinline__ uint32_t cluster_addr(const void *p, int rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
// 16 bytes to another block's shared memory, counted by an mbarrier there (both cluster addresses).
__device__ __forceinline__ void st_async_v4(uint32_t dst, const uint4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(dst),
                 "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// Bounded wait on an mbarrier that another block of the cluster completes.
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t *bar, uint32_t parity, uint32_t polls) {
    for (uint32_t it = 0; it < polls; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, "
            "1, 0, p;\n}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}
// Whether `v` holds in any block of the cluster (`v` block-uniform; every thread calls it).
// `flag` is a shared word of this block; no block returns before every block has read the others'.
__device__ __forceinline__ bool cluster_any(const bool v, uint32_t *flag, const int csize) {
    if (csize == 1) return v;
    if (threadIdx.x == 0) *flag = v ? 1u : 0u;
    cluster_barrier();
    const uint32_t o = (int)threadIdx.x < csize ? ld_cluster_u32(flag, (int)threadIdx.x) : 0u;
    const bool any = __syncthreads_or(o != 0);
    cluster_barrier();
    return any;
}

__device__ __forceinline__ unsigned long long hit_key(int32_t score, uint32_t idx) {
    return ((unsigned long long)((uint32_t)score ^ 0x80000000u) << 32) | (uint32_t)(~idx);
}

// ---- one pass of the wavefront -------------------------------------------------------------
//
// Sweeps the item's columns for the G*R query rows of one pass. Steps are warp-uniform (every
// lane of the warp shuffles every step). Lane L works on column j = s - L + 1 at step s; the G and
// F values of its last row at column j reach lane L+1 at step s+1. Lane 0 reads the row above the
// pass from the boundary row (or the top border in the first pass); lane G-1 writes the pass's
// last row to the boundary row unless this is the last pass. The state lives in a Sweep so a
// pass can be run in windows of steps.
template <class A, int R>
struct Sweep {
    typename A::V Gp[R], E[R];  // G (= H - go) of the previous column and E, per row slot
    typename A::V diag;         // G of the row above at the previous column (row slot 0)
    typename A::V botG, botF;   // this lane's last row at its current column, for lane L+1
    // SW end tracking within a pass: the running per-half maximum of G (= H - go) and the cell id
    // (column * R + slot) where it was first reached; column-major order inside the lane means
    // the first strict improvement is the smallest (column, row).
    typename A::V pbest;
    int32_t pid0, pid1;
    typename A::V botM;  // column maxima (COLMAX): G maximum of this column down to this lane's rows
};

// Where a COLMAX sweep writes its column maxima: per half, the pair's array indexed by target
// position (H of the column's best cell, so >= 0 in local mode); `atomic` when several passes
// combine into one array.
struct ColMaxOut {
    int32_t *p[2];
    bool atomic;
};

template <class A, int R, int MODE>
__device__ __forceinline__ void sweep_begin(Sweep<A, R> &sw, const int32_t row0, const int32_t go,
                                            const int32_t ge, const typename A::V Sv) {
    typedef ModeFlags<MODE> Fl;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int32_t row = row0 + r;
        const int64_t lb = (row <= 0 || Fl::left_free) ? 0 : -gap_pen(go, ge, row);
        sw.Gp[r] = A::splat(lb - go);
        sw.E[r] = Sv;
    }
    const int32_t row = row0 - 1;
    const int64_t lb = (row <= 0 || Fl::left_free) ? 0 : -gap_pen(go, ge, row);
    sw.diag = A::splat(lb - go);
    sw.botG = A::splat(0);
    sw.botF = A::splat(0);
    sw.pbest = A::splat(INT32_MIN);
    sw.pid0 = -1;
    sw.pid1 = -1;
}

// Constants of a sweep that do not change from step to step.
template <class A>
struct SweepConst {
    typename A::V negge, neggo, Sv;
    typename A::V top_free_g;  // G of the free top border row (H = 0)
};

// One step s of one lane. CHECKED steps test whether the lane's column is inside [1, w]; the
// caller runs unchecked steps only where every lane of the warp is live.
// With PRE the step's residue code and (lane 0) boundary-row values come from the caller, which
// loaded them one step ahead.
template <class A, int G, int R, int MODE, bool ENDS, bool CHECKED, bool PRE = false, bool COLMAX = false>
__device__ __forceinline__ void sweep_step(Sweep<A, R> &sw, const int s, const int lane,
                                           const int32_t w, const uint32_t (&n)[2],
                                           const typename A::RES *__restrict__ res,
                                           const uint8_t *prof_a, const uint8_t *prof_b,
                                           const int32_t row0, const bool first_pass,
                                           const bool last_pass, typename A::V *bnd,
                                           const int32_t qlen, const int32_t go, const int32_t ge,
                                           const SweepConst<A> &k, typename A::V &best,
                                           Cand (&cand)[2], const typename A::RES pre_r = 0,
                                           const typename A::V pre_g = 0, const typename A::V pre_f = 0,
                                           const ColMaxOut *cmo = nullptr) {
    typedef typename A::V V;
    typedef ModeFlags<MODE> Fl;
    static_assert(!COLMAX || (Fl::local && !ENDS), "column maxima are a local score-only sweep");
    const V negge = k.negge, neggo = k.neggo;
    {
        const int32_t j = s - lane + 1;
        V upG = __shfl_up_sync(0xffffffffu, sw.botG, 1, G);
        V upF = __shfl_up_sync(0xffffffffu, sw.botF, 1, G);
        // COLMAX: the column's maximum over the rows of the lanes above (lane 0: none this pass).
        V upM;
        if constexpr (COLMAX) {
            upM = __shfl_up_sync(0xffffffffu, sw.botM, 1, G);
            if (lane == 0) upM = neggo;
        }
        const bool live = !CHECKED || (j >= 1 && j <= w);
        if (lane == 0) {
            if (first_pass) {
                upG = Fl::top_free ? k.top_free_g : A::splat(-gap_pen(go, ge, j) - go);
                upF = k.Sv;
            } else if (live) {
                upG = PRE ? pre_g : bnd[2 * (j - 1)];
                upF = PRE ? pre_f : bnd[2 * (j - 1) + 1];
            }
        }
        if (live) {
            int a, b;
            A::residues(PRE ? pre_r : res[j - 1], a, b);
            V pa[A::EPV], pb[A::EPV];
            V g_up = upG, f = upF, gd = sw.diag, hprev = A::splat(0), hlast = A::splat(0);
            V xprev = A::splat(0);
            V cm;  // COLMAX: this column's G maximum, down to this lane's rows
            if constexpr (COLMAX) cm = upM;
            const int32_t jR = j * R;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (r % A::EPV == 0)
                    A::template load_chunk<R, G>(prof_a, prof_b, a, b, lane, r / A::EPV, pa, pb);
                sw.E[r] = A::addmax(sw.E[r], negge, sw.Gp[r]);
                V h;
                if (Fl::local) {
                    // SW, with a one-op dependency chain from row to row: with x = max(d, E, 0) -
                    // go, G = max(F - go, x) and, since go >= ge, F of the next row = max(F - ge,
                    // G) = max(F - ge, x). x >= -go, so nothing leaves int16. h here is G; the
                    // running maximum (and with ENDS the tracked best cell) is kept in G, go added
                    // at the end.
                    f = A::addmax(f, negge, r == 0 ? g_up : xprev);
                    const V d = A::diag(gd, pa[r % A::EPV], pb[r % A::EPV]);
                    const V x = A::vadd(A::vmax3_relu(d, sw.E[r], d), neggo);
                    xprev = x;
                    h = A::addmax(f, neggo, x);
                    gd = sw.Gp[r];
                    sw.Gp[r] = h;
                    g_up = h;
                } else {
                    f = A::addmax(f, negge, g_up);
                    const V d = A::diag(gd, pa[r % A::EPV], pb[r % A::EPV]);
                    h = Fl::local ? A::vmax3_relu(d, sw.E[r], f) : A::vmax3(d, sw.E[r], f);
                    gd = sw.Gp[r];
                    const V g = A::vadd(h, neggo);
                    sw.Gp[r] = g;
                    g_up = g;
                }
                if (Fl::local) {
                    if (ENDS) {
                        bool u0, u1;
                        sw.pbest = A::bmax(sw.pbest, h, u0, u1);
                        if (u0) sw.pid0 = jR + r;
                        if (u1) sw.pid1 = jR + r;
                    } else if (COLMAX) {
                        if (r & 1)
                            cm = A::vmax3(cm, hprev, h);
                        else
                            hprev = h;
                    } else {
                        if (r & 1)
                            best = A::vmax3(best, hprev, h);
                        else
                            hprev = h;
                    }
                }
                if (r == R - 1) hlast = h;
            }
            if (Fl::local && !ENDS && (R & 1)) {
                if (COLMAX)
                    cm = A::vmax(cm, hprev);
                else
                    best = A::vmax(best, hprev);
            }
            if constexpr (COLMAX) {
                // The last lane holds the column's maximum over the pass: H = G + go.
                sw.botM = cm;
                if (lane == G - 1) {
#pragma unroll
                    for (int h = 0; h < A::NH; ++h) {
                        if (j <= (int32_t)n[h]) {
                            const int32_t v = A::get(cm, h) + go;
                            if (cmo->atomic)
                                atomicMax(cmo->p[h] + (j - 1), v);
                            else
                                cmo->p[h][j - 1] = v;
                        }
                    }
                }
            }
            sw.botG = g_up;
            sw.botF = f;
            sw.diag = upG;
            if (lane == G - 1 && !last_pass) {
                bnd[2 * (j - 1)] = sw.botG;
                bnd[2 * (j - 1) + 1] = sw.botF;
            }
            // Last query row (grid row qlen): slot R-1 of lane G-1 in the last pass.
            if ((Fl::last_row || Fl::corner) && last_pass && lane == G - 1) {
#pragma unroll
                for (int h = 0; h < A::NH; ++h) {
                    const int32_t nh = (int32_t)n[h];
                    if (Fl::last_row ? (j <= nh) : (j == nh)) consider(cand[h], A::get(hlast, h), j, qlen);
                }
            }
            // Last column of each sequence (grid column n): every real row of this lane.
            if (Fl::last_col) {
#pragma unroll
                for (int h = 0; h < A::NH; ++h) {
                    if (j == (int32_t)n[h]) {
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            if (row0 + r >= 1) consider(cand[h], A::get(sw.Gp[r], h) + go, j, row0 + r);
                    }
                }
            }
        }
    }
}

// Steps [s_begin, s_end) of one lane. `w_min` is the smallest item width in the warp: steps in
// [G-1, w_min) have every lane of the warp on a real column and skip the per-lane checks. All
// bounds are warp-uniform.
// The unchecked steps load the next step's residue code and boundary-row values one step ahead (the
// boundary row was written by an earlier, completed pass).
template <class A, int G, int R, int MODE, bool ENDS, bool COLMAX = false>
__device__ __forceinline__ void sweep_run(Sweep<A, R> &sw, const int s_begin, const int s_end,
                                          const int w_min, const int lane, const int32_t w,
                                          const uint32_t (&n)[2],
                                          const typename A::RES *__restrict__ res,
                                          const uint8_t *prof_a, const uint8_t *prof_b,
                                          const int32_t row0, const bool first_pass,
                                          const bool last_pass, typename A::V *bnd,
                                          const int32_t qlen, const int32_t go, const int32_t ge,
                                          const typename A::V Sv, typename A::V &best,
                                          Cand (&cand)[2], const ColMaxOut *cmo = nullptr) {
    SweepConst<A> k;
    k.negge = A::splat(-(int64_t)ge);
    k.neggo = A::splat(-(int64_t)go);
    k.Sv = Sv;
    k.top_free_g = A::splat(-(int64_t)go);
    const int fast_lo = max(s_begin, G - 1);
    const int fast_hi = max(fast_lo, min(s_end, w_min));
    const int head_end = min(s_end, fast_lo);
    for (int s = s_begin; s < head_end; ++s)
        sweep_step<A, G, R, MODE, ENDS, true, false, COLMAX>(sw, s, lane, w, n, res, prof_a, prof_b, row0,
                                                             first_pass, last_pass, bnd, qlen, go, ge, k,
                                                             best, cand, 0, 0, 0, cmo);
    if (fast_lo < fast_hi) {
        typedef typename A::V V;
        // Every lane of the warp is inside its item in [fast_lo, fast_hi): the indices below
        // (step s - lane, clamped to the range) are real columns.
        typename A::RES r_cur = res[fast_lo - lane];
        V g_cur = 0, f_cur = 0;
        if (lane == 0 && !first_pass) {
            g_cur = bnd[2 * (fast_lo - lane)];
            f_cur = bnd[2 * (fast_lo - lane) + 1];
        }
        for (int s = fast_lo; s < fast_hi; ++s) {
            const int sn = min(s + 1, fast_hi - 1);
            const typename A::RES r_next = res[sn - lane];
            V g_next = g_cur, f_next = f_cur;
            if (lane == 0 && !first_pass) {
                g_next = bnd[2 * (sn - lane)];
                f_next = bnd[2 * (sn - lane) + 1];
            }
            sweep_step<A, G, R, MODE, ENDS, false, true, COLMAX>(sw, s, lane, w, n, res, prof_a, prof_b,
                                                                 row0, first_pass, last_pass, bnd, qlen,
                                                                 go, ge, k, best, cand, r_cur, g_cur,
                                                                 f_cur, cmo);
            r_cur = r_next;
            g_cur = g_next;
            f_cur = f_next;
        }
    }
    for (int s = max(fast_hi, head_end); s < s_end; ++s)
        sweep_step<A, G, R, MODE, ENDS, true, false, COLMAX>(sw, s, lane, w, n, res, prof_a, prof_b, row0,
                                                             first_pass, last_pass, bnd, qlen, go, ge, k,
                                                             best, cand, 0, 0, 0, cmo);
}

// The lane's tracked best cell of the pass as a candidate (local mode: pbest holds G = H - go).
template <class A, int R, int MODE, bool ENDS>
__device__ __forceinline__ void sweep_end(const Sweep<A, R> &sw, const int32_t row0, const int32_t go,
                                          Cand (&cand)[2]) {
    if (ModeFlags<MODE>::local && ENDS) {
        if (sw.pid0 >= 0) consider(cand[0], A::get(sw.pbest, 0) + go, sw.pid0 / R, row0 + sw.pid0 % R);
        if (A::NH > 1 && sw.pid1 >= 0)
            consider(cand[1], A::get(sw.pbest, 1) + go, sw.pid1 / R, row0 + sw.pid1 % R);
    }
}

// One whole pass: begin, every step, end.
template <class A, int G, int R, int MODE, bool ENDS, bool COLMAX = false>
__device__ __forceinline__ void sweep_pass(const int lane, const int steps, const int w_min,
                                           const int32_t w, const uint32_t (&n)[2],
                                           const typename A::RES *__restrict__ res,
                                           const uint8_t *prof_a, const uint8_t *prof_b,
                                           const int32_t row0, const bool first_pass,
                                           const bool last_pass, typename A::V *bnd,
                                           const int32_t qlen, const int32_t go, const int32_t ge,
                                           const typename A::V Sv, typename A::V &best,
                                           Cand (&cand)[2], const ColMaxOut *cmo = nullptr) {
    Sweep<A, R> sw;
    sweep_begin<A, R, MODE>(sw, row0, go, ge, Sv);
    if constexpr (COLMAX) sw.botM = A::splat(-(int64_t)go);
    sweep_run<A, G, R, MODE, ENDS, COLMAX>(sw, 0, steps, w_min, lane, w, n, res, prof_a, prof_b,
                                                 row0, first_pass, last_pass, bnd, qlen, go, ge, Sv,
                                                 best, cand, cmo);
    sweep_end<A, R, MODE, ENDS>(sw, row0, go, cand);
}

// ---- two columns per step: the sweep of int16x2 pairs and int32 items ---------------------------
//
// Lane L works on columns j0 = 2(s - L) + 1 and j1 = j0 + 1 at step s, R rows each: the per-step
// work (shuffles, residue and boundary loads, loop control) is spread over 2R rows of work while a
// lane keeps only R rows of state, and the F chains of the two columns (column j1 one row behind
// column j0) give the scheduler two independent dependency chains. Long form of the recurrence
// (E, F, H = max(d, E, F), in local mode also max with 0, G = H - go); the running maximum is kept on
// G. The modes that answer in the last row track it once a step; those that answer in a sequence's last
// column do so in checked steps, which every step is that may hold one.

// The residue codes of two adjacent columns as one load: two 16-bit pair codes (int16x2 pairs) or
// two 8-bit residues (int32 items). OK: the lane arithmetic has a two-column form.
template <class A>
struct TwoCodes {
    static constexpr bool OK = (A::NH == 2 && sizeof(typename A::RES) == 2) || (A::NH == 1 && sizeof(typename A::RES) == 1);
    static constexpr int BITS = 8 * (int)sizeof(typename A::RES);
    typedef typename std::conditional<sizeof(typename A::RES) == 2, uint32_t, uint16_t>::type W;
};

template <class A, int R>
struct Sweep2 {
    typename A::V Gp[R], E[R];        // G of the previous column and E, per row slot
    typename A::V diag;               // G of the row above the lane at the column before j0
    typename A::V botG[2], botF[2];   // this lane's last row at columns j0, j1, for lane L + 1
    // End tracking: a value that this lane's cells must exceed to be the answer, and per half the first
    // of the two columns that last did (-1: none this pass).
    typename A::V pbest;
    int32_t pcol[2];
    typename A::V lastG;  // the last query row's running maximum (lane G - 1, last pass)
};

// End tracking (local mode) costs a comparison a step. A cell can be the answer only if it exceeds every earlier
// column of its lane, and is no worse than the cells of the lanes above up to the step's columns (equal:
// it may win by its column) and of the passes before. Where a step has such a cell in some half, both
// columns' rows are copied to shared memory (`copy`: the lane's uint4s `stride` apart, R / 2 a half), and
// the cell is looked up in the copy at the pass's end. (scan_all of 50,000 protein sequences, a query of
// 900: 26.1 ms with a predicate and two selects a cell on 8 lanes a pair, 6.4 with the length forms and a
// comparison a column, 5.6 so.)
template <class A, int R>
__device__ __forceinline__ void sweep2_track(Sweep2<A, R> &sw, const typename A::V (&g0)[R], const typename A::V (&g1)[R],
                                             const typename A::V cm, const int32_t j, uint4 *copy, const int stride) {
    if (cm == sw.pbest) return;
#pragma unroll
    for (int h = 0; h < A::NH; ++h) {
        const uint32_t mask = A::NH == 1 ? 0xffffffffu : h ? 0xffff0000u : 0xffffu;
        if (((uint32_t)cm ^ (uint32_t)sw.pbest) & mask) {
#pragma unroll
            for (int c = 0; c < R / 4; ++c) {
                copy[(h * (R / 2) + c) * stride] = make_uint4((uint32_t)g0[4 * c], (uint32_t)g0[4 * c + 1],
                                                              (uint32_t)g0[4 * c + 2], (uint32_t)g0[4 * c + 3]);
                copy[(h * (R / 2) + R / 4 + c) * stride] = make_uint4((uint32_t)g1[4 * c], (uint32_t)g1[4 * c + 1],
                                                                      (uint32_t)g1[4 * c + 2], (uint32_t)g1[4 * c + 3]);
            }
            sw.pcol[h] = j;
        }
    }
    sw.pbest = cm;
}

// The lane's tracked cells of a pass whose first row of this lane is row0, as candidates: the first
// column's rows, then the second's, so the first cell with the copy's maximum.
template <class A, int R>
__device__ __forceinline__ void sweep2_tracked(const Sweep2<A, R> &sw, const int32_t row0, const int32_t go,
                                               const uint4 *copy, const int stride, Cand (&cand)[2]) {
#pragma unroll
    for (int h = 0; h < A::NH; ++h) {
        if (sw.pcol[h] < 0) continue;
        int32_t best = INT32_MIN;
        int at = 0;
        for (int c = 0; c < R / 2; ++c) {
            const uint4 v = copy[(h * (R / 2) + c) * stride];
            const int32_t g[4] = {A::get(v.x, h), A::get(v.y, h), A::get(v.z, h), A::get(v.w, h)};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (g[e] > best) best = g[e], at = 4 * c + e;
        }
        consider(cand[h], best + go, sw.pcol[h] + at / R, row0 + at % R);
    }
}

// One column of R rows: E, F, H, G in place; returns the last row's G and F.
template <class A, int G, int R, bool LOCAL>
__device__ __forceinline__ void sweep2_column(Sweep2<A, R> &sw, const int a, const int b, const int lane,
                                              const uint8_t *prof_a, const uint8_t *prof_b,
                                              typename A::V g_up, typename A::V f, typename A::V gd,
                                              const typename A::V negge, const typename A::V neggo,
                                              typename A::V &best, typename A::V &outG,
                                              typename A::V &outF) {
    typedef typename A::V V;
    V pa[A::EPV], pb[A::EPV];
    V hprev = A::splat(0);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r % A::EPV == 0) A::template load_chunk<R, G>(prof_a, prof_b, a, b, lane, r / A::EPV, pa, pb);
        sw.E[r] = A::addmax(sw.E[r], negge, sw.Gp[r]);
        f = A::addmax(f, negge, g_up);
        const V d = A::diag(gd, pa[r % A::EPV], pb[r % A::EPV]);
        const V h = LOCAL ? A::vmax3_relu(d, sw.E[r], f) : A::vmax3(d, sw.E[r], f);
        const V g = A::vadd(h, neggo);
        gd = sw.Gp[r];
        sw.Gp[r] = g;
        g_up = g;
        if (LOCAL) {
            if (r & 1)
                best = A::vmax3(best, hprev, g);
            else
                hprev = g;
        }
    }
    if (LOCAL && (R & 1)) best = A::vmax(best, hprev);
    outG = g_up;
    outF = f;
}

// Both columns of a step, interleaved one row apart (row r of column j0 with row r - 1 of column
// j1, which needs rows r - 1 of column j0 only): the same values as sweep2_column twice, with the
// two columns' dependency chains side by side in the instruction stream. With TRACK column j0's G is kept
// in g0.
template <class A, int G, int R, bool LOCAL, bool TRACK>
__device__ __forceinline__ void sweep2_both(Sweep2<A, R> &sw, const int a0, const int b0, const int a1,
                                            const int b1, const int lane, const uint8_t *prof_a,
                                            const uint8_t *prof_b, const typename A::V upG0,
                                            const typename A::V upF0, const typename A::V upG1,
                                            const typename A::V upF1, const typename A::V negge,
                                            const typename A::V neggo, typename A::V &best,
                                            typename A::V (&g0)[R]) {
    typedef typename A::V V;
    V p0a[A::EPV], p0b[A::EPV], p1a[A::EPV], p1b[A::EPV];
    V g_up0 = upG0, f0 = upF0, gd0 = sw.diag, hprev0 = A::splat(0);
    V g_up1 = upG1, f1 = upF1, gd1 = upG0, hprev1 = A::splat(0);
#pragma unroll
    for (int t = 0; t <= R; ++t) {
        if (t < R) {  // column j0, row t
            const int r = t;
            if (r % A::EPV == 0) A::template load_chunk<R, G>(prof_a, prof_b, a0, b0, lane, r / A::EPV, p0a, p0b);
            sw.E[r] = A::addmax(sw.E[r], negge, sw.Gp[r]);
            f0 = A::addmax(f0, negge, g_up0);
            const V d = A::diag(gd0, p0a[r % A::EPV], p0b[r % A::EPV]);
            const V h = LOCAL ? A::vmax3_relu(d, sw.E[r], f0) : A::vmax3(d, sw.E[r], f0);
            const V g = A::vadd(h, neggo);
            gd0 = sw.Gp[r];
            sw.Gp[r] = g;
            if (TRACK) g0[r] = g;
            g_up0 = g;
            if (LOCAL) {
                if (r & 1)
                    best = A::vmax3(best, hprev0, g);
                else
                    hprev0 = g;
            }
        }
        if (t >= 1) {  // column j1, row t - 1
            const int r = t - 1;
            if (r % A::EPV == 0) A::template load_chunk<R, G>(prof_a, prof_b, a1, b1, lane, r / A::EPV, p1a, p1b);
            sw.E[r] = A::addmax(sw.E[r], negge, sw.Gp[r]);
            f1 = A::addmax(f1, negge, g_up1);
            const V d = A::diag(gd1, p1a[r % A::EPV], p1b[r % A::EPV]);
            const V h = LOCAL ? A::vmax3_relu(d, sw.E[r], f1) : A::vmax3(d, sw.E[r], f1);
            const V g = A::vadd(h, neggo);
            gd1 = sw.Gp[r];
            sw.Gp[r] = g;
            g_up1 = g;
            if (LOCAL) {
                if (r & 1)
                    best = A::vmax3(best, hprev1, g);
                else
                    hprev1 = g;
            }
        }
    }
    if (LOCAL && (R & 1)) best = A::vmax3(best, hprev0, hprev1);
    sw.botG[0] = g_up0;
    sw.botF[0] = f0;
    sw.botG[1] = g_up1;
    sw.botF[1] = f1;
}

// Step s of one lane (see above), whose first row is row0. The residue codes of columns j0, j1 come as
// one 32-bit word (`codes`) and, for lane 0 after the first pass, the boundary values of both columns
// as one 16-byte word (`up`: G, F of j0, then of j1). CHECKED steps test each column against [1, w].
template <class A, int G, int R, int MODE, bool CHECKED, bool ENDS>
__device__ __forceinline__ void sweep2_step(Sweep2<A, R> &sw, const ScanParams &p, const int s, const int lane,
                                            const int32_t w, const uint32_t (&n)[2], const uint8_t *prof_a,
                                            const uint8_t *prof_b, const int32_t row0, const bool first_pass,
                                            const bool last_pass, typename A::V *bnd, const SweepConst<A> &k,
                                            typename A::V &best, Cand (&cand)[2], const uint32_t codes, const uint4 up,
                                            uint4 *copy) {
    typedef typename A::V V;
    typedef ModeFlags<MODE> Fl;
    constexpr bool TRACK = Fl::local && ENDS;
    constexpr int CODE_BITS = TwoCodes<A>::BITS;
    constexpr uint32_t CODE_MASK = (1u << CODE_BITS) - 1u;
    const int32_t j0 = 2 * (s - lane) + 1;
    V upG0 = __shfl_up_sync(0xffffffffu, sw.botG[0], 1, G);
    V upF0 = __shfl_up_sync(0xffffffffu, sw.botF[0], 1, G);
    V upG1 = __shfl_up_sync(0xffffffffu, sw.botG[1], 1, G);
    V upF1 = __shfl_up_sync(0xffffffffu, sw.botF[1], 1, G);
    const bool live0 = !CHECKED || (j0 >= 1 && j0 <= w);
    const bool live1 = !CHECKED || (j0 + 1 >= 1 && j0 + 1 <= w);
    if (lane == 0) {
        if (first_pass) {
            if (Fl::top_free) {
                upG0 = upG1 = k.top_free_g;
            } else {
                // G of H(0, j) = -go - (j - 1) ge (columns past the item may wrap: never used).
                upG0 = A::pack(-2 * p.go - (j0 - 1) * p.ge);
                upG1 = A::vadd(upG0, k.negge);
            }
            upF0 = upF1 = k.Sv;
        } else {
            upG0 = up.x;
            upF0 = up.y;
            upG1 = up.z;
            upF1 = up.w;
        }
    }
    int a, b;
    if (TRACK) {
        const V upB = __shfl_up_sync(0xffffffffu, sw.pbest, 1, G);
        if (lane > 0) sw.pbest = A::vmax(sw.pbest, A::vadd(upB, A::splat(-1)));
        best = sw.pbest;
    }
    const bool last_lane = last_pass && lane == G - 1;
    V g0[R];
    if (!CHECKED) {
        // Both columns live: interleaved (measured 0.6% faster than one after the other).
        int a1, b1;
        A::residues((typename A::RES)(codes & CODE_MASK), a, b);
        A::residues((typename A::RES)(codes >> CODE_BITS), a1, b1);
        sweep2_both<A, G, R, Fl::local, TRACK>(sw, a, b, a1, b1, lane, prof_a, prof_b, upG0, upF0, upG1, upF1, k.negge,
                                               k.neggo, best, g0);
        if (TRACK) sweep2_track<A, R>(sw, g0, sw.Gp, best, j0, copy, (int)blockDim.x);
        if (Fl::last_row && last_lane) {
            const V m = A::vmax3(sw.lastG, sw.botG[0], sw.botG[1]);
            if (m != sw.lastG) {
#pragma unroll
                for (int h = 0; h < A::NH; ++h) {
                    if (j0 <= (int32_t)n[h]) consider(cand[h], A::get(sw.botG[0], h) + p.go, j0, p.qlen);
                    if (j0 + 1 <= (int32_t)n[h]) consider(cand[h], A::get(sw.botG[1], h) + p.go, j0 + 1, p.qlen);
                }
                sw.lastG = m;
            }
        }
    } else {
        // Candidates of column j, whose rows are in Gp and last row's G is g.
        auto answers = [&](const int32_t j, const V g) {
            if ((Fl::last_row || Fl::corner) && last_lane) {
                sw.lastG = A::vmax(sw.lastG, g);
#pragma unroll
                for (int h = 0; h < A::NH; ++h) {
                    const int32_t nh = (int32_t)n[h];
                    if (Fl::last_row ? (j <= nh) : (j == nh)) consider(cand[h], A::get(g, h) + p.go, j, p.qlen);
                }
            }
            if (Fl::last_col) {
#pragma unroll
                for (int h = 0; h < A::NH; ++h) {
                    if (j == (int32_t)n[h]) {
#pragma unroll
                        for (int r = 0; r < R; ++r)
                            if (row0 + r >= 1) consider(cand[h], A::get(sw.Gp[r], h) + p.go, j, row0 + r);
                    }
                }
            }
        };
        if (live0) {
            A::residues((typename A::RES)(codes & CODE_MASK), a, b);
            sweep2_column<A, G, R, Fl::local>(sw, a, b, lane, prof_a, prof_b, upG0, upF0, sw.diag, k.negge, k.neggo,
                                              best, sw.botG[0], sw.botF[0]);
            answers(j0, sw.botG[0]);
            if (TRACK) {
#pragma unroll
                for (int r = 0; r < R; ++r) g0[r] = sw.Gp[r];
            }
        }
        if (live1) {
            A::residues((typename A::RES)(codes >> CODE_BITS), a, b);
            sweep2_column<A, G, R, Fl::local>(sw, a, b, lane, prof_a, prof_b, upG1, upF1, upG0, k.negge, k.neggo, best,
                                              sw.botG[1], sw.botF[1]);
            answers(j0 + 1, sw.botG[1]);
        }
        // (A dead second column leaves the first one's rows in Gp.)
        if (TRACK && live0) sweep2_track<A, R>(sw, g0, sw.Gp, best, j0, copy, (int)blockDim.x);
    }
    if (live0) sw.diag = live1 ? upG1 : upG0;
    if (lane == G - 1 && !last_pass && live0)
        *reinterpret_cast<uint4 *>(bnd + 2 * (j0 - 1)) = make_uint4(sw.botG[0], sw.botF[0], sw.botG[1], sw.botF[1]);
}

// Every pass of one item's two-column sweep, the passes back to back. With W column pairs a pass
// (warp-uniform), lane L works virtual column pair v = s - L at step s, that is pass v / W at
// column pair v % W: when lane 0 has finished a pass it starts the next one while lanes 1..G-1
// finish theirs, so the G - 1 fill and drain steps of the wavefront are paid once per item, not
// once per pass. A pass p >= 1 begins with G - 1 transition steps (lanes L <= t at column pair
// t - L of pass p, the others at W + t - L of pass p - 1), then its interior steps (every lane in
// pass p; the ones with both columns of every lane inside its item run unchecked, with the next
// step's codes and boundary values loaded one step ahead).
//
// Shared memory: pass p's profile slice is in buffer p % 2. After the transition into pass p no
// lane of the block reads pass p - 1's slice any more: the block barrier there (one per pass, in
// every warp) frees that buffer for pass p + 1's copy, issued by thread 0. The boundary row: lane
// G-1 writes column pair c of pass p at step pW + c + G - 1, lane 0 reads it for pass p + 1 at
// step (p + 1)W + c (one step earlier with the prefetch). W >= 2G keeps every such read at least G
// steps after its write; the warp barrier at the start of each transition orders the writes the
// transition's reads need, and the block barrier after it orders the rest.
//
// Every thread of the block calls it with the block's `phase` (see scan_unit). Returns false if a
// profile copy did not arrive in time (the error flag is then set and the block must stop).
template <class A, int G, int R, int MODE, bool ENDS>
__device__ __forceinline__ bool sweep2_item(const ScanParams &p, const int lane, const int W, const int wfast,
                                            const int32_t w, const uint32_t (&n)[2],
                                            const typename A::RES *__restrict__ res,
                                            typename A::V *bnd, uint8_t *smem, uint64_t *bars,
                                            uint32_t &phase, const typename A::V Sv, typename A::V &best,
                                            Cand (&cand)[2]) {
    typedef typename A::V V;
    typedef ModeFlags<MODE> Fl;
    constexpr bool TRACK = Fl::local && ENDS;
    typedef typename TwoCodes<A>::W W2;
    const int n_passes = p.n_passes;
    const uint32_t hi_off = (A::TABLES - 1) * (p.pass_bytes / A::TABLES);
    SweepConst<A> k;
    k.negge = A::splat(-(int64_t)p.ge);
    k.neggo = A::splat(-(int64_t)p.go);
    k.Sv = Sv;
    k.top_free_g = A::splat(-(int64_t)p.go);
    Sweep2<A, R> sw;
    auto row0_of = [&](int pass) { return p.vrow0 + pass * (G * R) + lane * R; };
    // A lane's state at the start of a pass: the left border.
    auto reset = [&](int pass) {
        const int32_t row0 = row0_of(pass);
        auto left = [&](int32_t row) {
            return Fl::left_free ? k.top_free_g : A::splat((row <= 0 ? 0 : -gap_pen(p.go, p.ge, row)) - p.go);
        };
#pragma unroll
        for (int r = 0; r < R; ++r) {
            sw.Gp[r] = left(row0 + r);
            sw.E[r] = Sv;
        }
        sw.diag = left(row0 - 1);
        sw.pcol[0] = sw.pcol[1] = -1;
        // In a later pass a cell as good as the passes before may still win, by its column.
        if (TRACK) sw.pbest = A::vmax(k.neggo, A::vadd(sw.pbest, A::splat(-1)));
    };
    sw.pbest = k.neggo;  // H = 0: only a cell above the border's 0 is tracked
    sw.lastG = A::splat(A::VMIN);
    uint4 *copy = reinterpret_cast<uint4 *>(reinterpret_cast<uint8_t *>(bars) + 16) + threadIdx.x;
    // This lane is done with pass `pass`.
    auto tracked = [&](int pass) {
        if constexpr (TRACK) sweep2_tracked<A, R>(sw, row0_of(pass), p.go, copy, (int)blockDim.x, cand);
    };
    reset(0);
    sw.botG[0] = sw.botG[1] = sw.botF[0] = sw.botF[1] = A::splat(0);
    const W2 *res2 = reinterpret_cast<const W2 *>(res);  // codes of columns (2i+1, 2i+2)
    const uint4 *bnd4 = reinterpret_cast<const uint4 *>(bnd);          // boundary of the same pair
    const uint4 none = make_uint4(0, 0, 0, 0);
    // Loads for column pair c of this lane (-1: no column; a dead pair's values are never used).
    auto codes_at = [&](int c) -> uint32_t { return (c >= 0 && 2 * c < w) ? res2[c] : 0u; };
    auto up_at = [&](int c, bool first) -> uint4 {
        return (lane == 0 && !first && c >= 0 && 2 * c < w) ? bnd4[c] : none;
    };
    // One checked step of this lane at column pair c of pass lp (lp < 0 or c < 0: no column).
    auto checked = [&](int lp, int c) {
        const uint8_t *pa = smem + (size_t)(lp & 1) * p.pass_bytes;
        if (lp < 0) c = -1;
        sweep2_step<A, G, R, MODE, true, ENDS>(sw, p, c + lane, lane, w, n, pa, pa + hi_off, row0_of(lp), lp == 0,
                                               lp == n_passes - 1, bnd, k, best, cand, codes_at(c), up_at(c, lp == 0), copy);
    };
    for (int pass = 0; pass < n_passes; ++pass) {
        const int buf = pass & 1;
        const bool ok = mbar_wait_bounded(&bars[buf], (phase >> buf) & 1u, p.wait_polls);
        phase ^= 1u << buf;
        if (W > 0) {
            __syncwarp();
            for (int t = 0; t < G - 1; ++t) {
                const bool fresh = lane <= t;  // this lane has entered pass `pass`
                if (fresh && lane == t && pass > 0) tracked(pass - 1), reset(pass);
                checked(fresh ? pass : pass - 1, fresh ? t - lane : W + t - lane);
            }
            if (lane == G - 1 && pass > 0) tracked(pass - 1), reset(pass);  // lane G-1 enters at the first interior step
        }
        if (__syncthreads_or(!ok)) {
            // This pass's copy and, in the first pass, the second one are still outstanding.
            if (threadIdx.x == 0)
                wait_gave_up(p.err, bars, (1u << buf) | (pass == 0 && n_passes > 1 ? 2u : 0u), phase ^ (1u << buf));
            return false;
        }
        if (threadIdx.x == 0 && pass >= 1 && pass + 1 < n_passes)
            bulk_load(smem + (size_t)(buf ^ 1) * p.pass_bytes, p.profile + (size_t)(pass + 1) * p.pass_bytes,
                      p.pass_bytes, &bars[buf ^ 1]);
        if (W == 0) continue;
        const uint8_t *pa = smem + (size_t)buf * p.pass_bytes, *pb = pa + hi_off;
        const bool first = pass == 0, last = pass == n_passes - 1;
        const int32_t row0 = row0_of(pass);
        const int fast_hi = max(G - 1, wfast);
        if (G - 1 < fast_hi) {
            // Two steps an iteration with two sets of registers for the one-step-ahead loads (only
            // lane 0 reads the boundary row: the other lanes' copies are never used).
            const bool up_lane = lane == 0 && !first;
            uint32_t c_a = res2[G - 1 - lane], c_b = 0;
            uint4 u_a = none, u_b = none;
            if (up_lane) u_a = bnd4[G - 1];
            int s = G - 1;
            for (; s + 1 < fast_hi; s += 2) {
                c_b = res2[s + 1 - lane];
                if (up_lane) u_b = bnd4[s + 1];
                sweep2_step<A, G, R, MODE, false, ENDS>(sw, p, s, lane, w, n, pa, pb, row0, first, last, bnd, k, best, cand,
                                                        c_a, u_a, copy);
                const int s2 = min(s + 2, fast_hi - 1);
                c_a = res2[s2 - lane];
                if (up_lane) u_a = bnd4[s2];
                sweep2_step<A, G, R, MODE, false, ENDS>(sw, p, s + 1, lane, w, n, pa, pb, row0, first, last, bnd, k, best, cand,
                                                        c_b, u_b, copy);
            }
            if (s < fast_hi)
                sweep2_step<A, G, R, MODE, false, ENDS>(sw, p, s, lane, w, n, pa, pb, row0, first, last, bnd, k, best, cand,
                                                        c_a, u_a, copy);
        }
        for (int s = fast_hi; s < W; ++s) checked(pass, s - lane);
    }
    // The last pass's drain: lanes L > t finish their columns W + t - L.
    if (W > 0)
        for (int t = 0; t < G - 1; ++t) checked(lane > t ? n_passes - 1 : -1, W + t - lane);
    if (n_passes > 0) tracked(n_passes - 1);
    __syncthreads();  // both profile buffers are free for the block's next unit
    return true;
}

// Group reduction of the per-lane candidates, border seeds, output and best-key fold. Every lane
// of the warp must call it (it shuffles).
template <class A, int G, int MODE, bool ENDS>
__device__ __forceinline__ void finish_item(const int lane, const bool active, const ItemMeta &meta,
                                            const int32_t qlen, const int32_t go, const int32_t ge,
                                            const typename A::V best, Cand (&cand)[2],
                                            int32_t *scores, int32_t *qend, int32_t *tend,
                                            unsigned long long *best_key) {
    typedef ModeFlags<MODE> Fl;
    if (Fl::local && !ENDS) {
#pragma unroll
        for (int h = 0; h < A::NH; ++h) cand[h].s = A::get(best, h) + go;  // best is kept in G
    }
#pragma unroll
    for (int h = 0; h < A::NH; ++h) {
#pragma unroll
        for (int off = G / 2; off > 0; off >>= 1) {
            Cand o;
            o.s = __shfl_xor_sync(0xffffffffu, cand[h].s, off, G);
            o.col = __shfl_xor_sync(0xffffffffu, cand[h].col, off, G);
            o.row = __shfl_xor_sync(0xffffffffu, cand[h].row, off, G);
            if (Fl::local && !ENDS) {
                if (o.s > cand[h].s) cand[h] = o;
            } else if (better(o, cand[h])) {
                cand[h] = o;
            }
        }
    }
    unsigned long long key = 0;
    if (active && lane == 0) {
#pragma unroll
        for (int h = 0; h < A::NH; ++h) {
            const uint32_t idx = meta.idx[h];
            if (idx == NO_INDEX) continue;
            Cand c = border_seed<MODE>(qlen, (int32_t)meta.n[h], go, ge);
            if (Fl::local && !ENDS) {
                if (cand[h].s > c.s) c.s = cand[h].s;
            } else if (better(cand[h], c)) {
                c = cand[h];
            }
            if (scores) scores[idx] = c.s;
            if (ENDS) {
                qend[idx] = c.row - 1;
                tend[idx] = c.col - 1;
            }
            const unsigned long long k = hit_key(c.s, idx);
            key = k > key ? k : key;
        }
    }
    if (best_key) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
            key = o > key ? o : key;
        }
        if ((threadIdx.x & 31) == 0 && key != 0) atomicMax(best_key, key);
    }
}

// Rows per lane the two-column sweep takes: up to 16; tracking ends in local mode from 12 on (with
// fewer rows the comparison a step outweighs what the second column saves: 64-residue queries against
// 5,000 reads 77 us a call with one column a step, 90 with two).
__host__ __device__ constexpr bool scan_two_col_rows(int rows, int mode, bool ends) {
    return rows <= 16 && (mode != MODE_SW || !ends || rows >= 12);
}

// Whether a scan launch shape runs the two-column sweep. Measured on the protein benchmark (SW scores):
// for the pairs as fast as one column of 32 rows, with half the per-lane state and 10% faster on
// 64-residue DNA queries; for the int32 items of a 5000-residue query 1014 against 594 GCUPS (two
// independent column chains per lane for their latency-bound warps).
// ONE_COL: the form with one column all the same.
template <class A, int R, int MODE, bool ENDS, bool GPROF, bool ONE_COL = false>
__host__ __device__ constexpr bool two_col_form() {
    return TwoCodes<A>::OK && !GPROF && !ONE_COL && scan_two_col_rows(R, MODE, ENDS);
}

#ifdef HY_BOUNDS
// The bounds-checked build: before an item is used, every index its metadata and residue codes
// can produce is checked against the extents in `p` (residue columns, boundary region, db
// indices, profile letters). All G lanes of a group call it for their group's item (`active`:
// the group has one); returns whether the item may be swept.
template <class A, int G>
__device__ bool item_in_bounds(const ScanParams &p, const ItemMeta &m, const int lane, const bool active) {
    bool ok = true;
    if (active) {
        ok = m.col_off + m.w <= p.res_cols && m.n[0] <= m.w && m.n[1] <= m.w &&
             (m.idx[0] == NO_INDEX || m.idx[0] < p.n_seqs) && (m.idx[1] == NO_INDEX || m.idx[1] < p.n_seqs) &&
             (A::NH == 2 || m.idx[1] == NO_INDEX) &&
             (p.n_passes <= 1 || (m.col_off >= p.bnd_col0 && m.col_off - p.bnd_col0 + m.w <= p.bnd_cols));
        if (ok) {
            const typename A::RES *res = reinterpret_cast<const typename A::RES *>(p.res) + m.col_off;
            for (uint32_t j = lane; j < m.w; j += G) {
                int a, b;
                A::residues(res[j], a, b);
                if ((uint32_t)a >= p.letters || (uint32_t)b >= p.letters) ok = false;
            }
        }
    }
#pragma unroll
    for (int off = G / 2; off > 0; off >>= 1) ok &= __shfl_xor_sync(0xffffffffu, (int)ok, off, G) != 0;
    return ok;
}
#endif

// ---- the database scan kernel ---------------------------------------------------------------
//
// All groups of a block step through the passes together: the pass's query profile is one
// contiguous slice, brought into shared memory by a TMA bulk copy while the previous pass runs.

// Initialise the block's two profile mbarriers (thread 0; the caller synchronises the block).
__device__ __forceinline__ void init_profile_bars(uint64_t *bars) {
    if (threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
}

// One unit of work for one block: group g of the block runs item `item_first + g` if that is
// below `item_end`, through every pass of the query in `p`. The block's two profile buffers and
// mbarriers live in `smem` / `bars`; `phase` holds the parity each barrier waits for next (bit b
// for barrier b) and is carried from unit to unit by a persistent caller. Every thread of the
// block must call it with the same arguments. Returns false if a profile copy did not arrive in
// time (the error flag is then set and the block must stop). With GPROF the lanes read the pass
// slices straight from the profile in global memory (through L1) instead of shared memory: the
// form for alphabets whose slices do not fit in shared memory; `smem` and `bars` are then unused.
template <class A, int G, int R, int MODE, bool ENDS, bool GPROF = false, bool ONE_COL = false>
__device__ __forceinline__ bool scan_unit(const ScanParams &p, const uint32_t item_first,
                                          const uint32_t item_end, uint8_t *smem, uint64_t *bars,
                                          uint32_t &phase) {
    typedef typename A::V V;
    constexpr int RPP = G * R;
    static_assert(R % A::EPV == 0, "rows per lane must fill whole profile vectors");
    static_assert(32 % G == 0, "groups must tile a warp");
    const uint8_t *prof_buf[2] = {smem, smem + p.pass_bytes};

    const int lane = threadIdx.x % G;
    const uint32_t item = item_first == NO_INDEX ? NO_INDEX : item_first + threadIdx.x / G;
    bool active = item != NO_INDEX && item < item_end;
    ItemMeta meta;
    if (active) meta = p.meta[item];
#ifdef HY_BOUNDS
    if (!item_in_bounds<A, G>(p, meta, lane, active)) {
        if (lane == 0) atomicExch(p.err, ERR_BOUNDS);
        active = false;
    }
#endif
    if (!active) {
        meta.col_off = p.bnd_col0;
        meta.w = 0;
        meta.n[0] = meta.n[1] = 0;
        meta.idx[0] = meta.idx[1] = NO_INDEX;
    }
    const V Sv = A::splat(p.sentinel);
    const typename A::RES *res = reinterpret_cast<const typename A::RES *>(p.res) + meta.col_off;
    V *bnd = reinterpret_cast<V *>(p.boundary) + 2 * (meta.col_off - p.bnd_col0);
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, meta.w);
    const int w_min = (int)__reduce_min_sync(0xffffffffu, meta.w);
    const int steps = wmax == 0 ? 0 : (int)wmax + G - 1;

    V best = A::splat(ModeFlags<MODE>::local && !ENDS ? -(int64_t)p.go : 0);
    Cand cand[2] = {{INT32_MIN, INT32_MAX, INT32_MAX}, {INT32_MIN, INT32_MAX, INT32_MAX}};

    if (!GPROF && threadIdx.x == 0 && p.n_passes > 0) {
        bulk_load(smem, p.profile, p.pass_bytes, &bars[0]);
        if (p.n_passes > 1) bulk_load(smem + p.pass_bytes, p.profile + p.pass_bytes, p.pass_bytes, &bars[1]);
    }
    if constexpr (two_col_form<A, R, MODE, ENDS, GPROF, ONE_COL>()) {
        // Column pairs a pass: at least 2G (the boundary row's read-after-write distance), and with one
        // pass the G - 1 of the fill.
        const int W = wmax == 0 ? 0 : max((int)(wmax + 1) / 2, p.n_passes > 1 ? 2 * G : G - 1);
        // Steps before this column pair hold no sequence's last column where the mode answers there.
        int wfast = min(W, w_min / 2);
        if constexpr (ModeFlags<MODE>::last_col || ModeFlags<MODE>::corner) {
            const uint32_t n_low = meta.idx[1] == NO_INDEX ? meta.n[0] : min(meta.n[0], meta.n[1]);
            wfast = min(wfast, max((int)__reduce_min_sync(0xffffffffu, n_low) - 1, 0) / 2);
        }
        if (!sweep2_item<A, G, R, MODE, ENDS>(p, lane, W, wfast, (int32_t)meta.w, meta.n, res, bnd, smem, bars, phase,
                                              Sv, best, cand))
            return false;
    } else {
        for (int pass = 0; pass < p.n_passes; ++pass) {
            const int buf = pass & 1;
            const uint8_t *prof;
            if (GPROF) {
                prof = p.profile + (size_t)pass * p.pass_bytes;
            } else {
                const bool ok = mbar_wait_bounded(&bars[buf], (phase >> buf) & 1u, p.wait_polls);
                phase ^= 1u << buf;
                if (__syncthreads_or(!ok)) {
                    // This pass's copy and, if issued, the next pass's are still outstanding.
                    if (threadIdx.x == 0)
                        wait_gave_up(p.err, bars, (1u << buf) | (pass + 1 < p.n_passes ? 1u << (buf ^ 1) : 0u),
                                     phase ^ (1u << buf));
                    return false;
                }
                prof = prof_buf[buf];
            }
            sweep_pass<A, G, R, MODE, ENDS>(lane, steps, w_min, (int32_t)meta.w, meta.n, res, prof,
                                            prof + (A::TABLES - 1) * (p.pass_bytes / A::TABLES),
                                            p.vrow0 + pass * RPP + lane * R, pass == 0, pass == p.n_passes - 1,
                                            bnd, p.qlen, p.go, p.ge, Sv, best, cand);
            __syncthreads();  // the profile buffer and boundary row are free again
            if (!GPROF && threadIdx.x == 0 && pass + 2 < p.n_passes)
                bulk_load(smem + (size_t)buf * p.pass_bytes, p.profile + (size_t)(pass + 2) * p.pass_bytes,
                          p.pass_bytes, &bars[buf]);
        }
    }
    finish_item<A, G, MODE, ENDS>(lane, active, meta, p.qlen, p.go, p.ge, best, cand, p.scores,
                                  p.qend, p.tend, p.best_key);
    return true;
}

// Threads a block of a launch shape may have: 512 for the pairs a warp each with 16 rows per lane,
// whose two slices of a large alphabet leave an SM one block.
template <class A, int G, int R>
constexpr int scan_max_threads() {
    return A::NH == 2 && G == 32 && R == 16 ? 512 : 256;
}

// Resident 256-thread blocks per SM each launch shape is compiled for (its register budget).
// The two-column sweep of 16 rows per lane is compiled for two blocks (measured faster than three
// with the spills three would need).
template <class A, int G, int R, bool TWO_COL = false>
constexpr int scan_min_blocks() {
    return A::NH == 1                                       ? 2
           : (G == 8 && R == 8) || R == 4                   ? 4
           : (G == 8 && R == 32) || (TWO_COL && R == 16 && G == 8) ? 2
           : scan_max_threads<A, G, R>() == 512             ? 1
           : R == 12                                        ? 2
                                                            : 3;
}

// Shared memory of a scan block besides its pass slices: the mbarriers and, where the two-column sweep
// tracks ends, each lane's copied columns.
inline size_t scan_extra_smem(int halves, int rows, int mode, bool ends, int threads) {
    return 16 + (mode == MODE_SW && ends && scan_two_col_rows(rows, mode, ends) ? (size_t)halves * 2 * rows * 4 * threads : 0);
}

// Pass slices a launch keeps in shared memory.
__host__ __device__ inline uint32_t scan_slices(int32_t n_passes) { return n_passes > 1 ? 2 : 1; }

template <class A, int G, int R, int MODE, bool ENDS, bool GPROF = false, bool ONE_COL = false>
__global__ void __launch_bounds__((scan_max_threads<A, G, R>()), (scan_min_blocks<A, G, R, two_col_form<A, R, MODE, ENDS, GPROF, ONE_COL>()>()))
    scan_kernel(const ScanParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + (GPROF ? 0 : scan_slices(p.n_passes) * (size_t)p.pass_bytes));
    const int gpb = blockDim.x / G;
    uint32_t first, end;
    if (p.item_ptr) {
        // One item, run by group 0 of block 0.
        const uint32_t want = *p.item_ptr;
        first = blockIdx.x == 0 ? want : NO_INDEX;
        end = (first == NO_INDEX || first >= p.n_items) ? first : first + 1;
    } else {
        first = p.item_base + blockIdx.x * gpb;
        end = p.n_items;
    }
    init_profile_bars(bars);
    __syncthreads();
    uint32_t phase = 0;
    scan_unit<A, G, R, MODE, ENDS, GPROF, ONE_COL>(p, first, end, smem, bars, phase);
}

// ---- the block-cooperative band kernel (long items, with end positions) ----------------------
//
// Runs one item (the winner of a scan, a long pair) on a whole block or thread-block cluster, with
// position tracking. Every warp is one 32-lane group running one pass (a band of 32*R query rows),
// two columns a step: lane L works columns 2(s - L) and 2(s - L) + 1 (from 0) at step s. The warps
// take the passes in rounds of W * (blocks). Inside a round warp g runs BAND_LAG * g steps behind
// the block's warp 0, with a block barrier every BAND_K steps: lane 31 of the warp above writes column
// pair c at its step c + 31, and the window of steps [s0, s0 + BAND_K) here reads pairs s0 .. s0 +
// BAND_K - 1, all written before the window's barrier since BAND_LAG >= BAND_K + 31. Between blocks
// the last warp stores its row into the next block's ring (st.async, counted by an mbarrier per
// BAND_K pairs there), which gives each ring block back once read; the blocks share no other step
// (no cluster barrier a window).
//
// A wait between blocks that gives up ends its side of that link: a block that did not get its row
// arms and gives back no more ring blocks, one that got no space sends none from that ring block on
// (it has sent whole ring blocks then). Both sweep on, on rows that no one uses, so that every block
// comes to the next cluster barrier, and there all stop: the error word is set, no result is written,
// and before the barrier that lets the blocks exit a block waits for the ring blocks that were sent
// to it and that it has not read, so that no row lands in the shared memory of a block that is gone.
//
// What bounds it is one warp's step: a lone warp issues a chain of dependent instructions with
// nothing beside it. So a step has two columns whose chains are independent but for a row's lag, and as few other instructions
// as it can: residue codes lie in a strip of shared memory that is refilled every 32 steps, the row
// above in a ring there that the warp above writes (warp 0 fills its own a window at a time, from the
// border or from the boundary row in global memory), both read at constant offsets; a step's codes are
// loaded two steps and its profile words one step ahead. 93 instructions and 258 cycles for a step of two
// columns, over the chain of 1,751 steps of a 2000 x 2000 int32 pair on four blocks: 0.47 ms with one
// column a step to 0.23, 5000 x 5000 1.45 to 0.67. Local mode takes the short row chain (sweep_step) and
// tracks the best cell once a step: the columns' maximum against the running one, its place looked up
// only where that improves.
constexpr int BAND_K = 16;
constexpr int BAND_LAG = 48;
constexpr int BAND_RING = 64;  // column pairs a ring holds: at least the lag plus a window
static_assert(BAND_LAG >= BAND_K + 31 && BAND_LAG % BAND_K == 0 && 32 % BAND_K == 0, "a window's row above must be written before it");
static_assert(BAND_RING >= BAND_LAG + BAND_K && BAND_RING % BAND_K == 0, "the ring must hold every pair not yet read");

// Where a step improves a lane's best cell, the form with 4 rows per lane copies the step's two
// columns to shared memory (predicated stores, no branch: 0.425 to 0.350 ms for a 2000 x 2000 pair) and
// finds the row in them after the sweep; the form with 8 rows finds it there and then.
template <int R>
__host__ __device__ constexpr bool band_copies() {
    return R <= 4;
}

// Shared memory of a band warp besides its pass slice: its last row (G, F of both columns) by
// column pair, the residue codes of 66 column pairs (32 before a block of 32 steps, 32 in it, and the
// two loaded ahead), and the lanes' copied columns (two halves). A
// block has one more ring, for the row above warp 0.
constexpr size_t BAND_RING_BYTES = BAND_RING * 16;
constexpr size_t BAND_STRIP_BYTES = (66 * 4 + 15) / 16 * 16;
__host__ __device__ constexpr size_t band_warp_bytes(int rows) {
    return BAND_RING_BYTES + BAND_STRIP_BYTES + (rows <= 4 ? (size_t)2 * 2 * rows * 4 * 32 : 0);
}

// The block's mbarriers: the profile copy's, then per ring block (BAND_K pairs) one that counts the
// bytes of the row above and one by which the next block gives its ring block back.
constexpr int BAND_SLOTS = BAND_RING / BAND_K;
constexpr int BAND_BARS = 1 + 2 * BAND_SLOTS;

// Shared memory of a band block of `warps` warps with pass slices of `slice` bytes (0: in global
// memory): the slices, the rings (at the end the warps' candidates in their place), the rest of the
// warps' bytes, the mbarriers, two words. All of it dynamic, so that the host's sum is what a block takes.
constexpr size_t BAND_TAIL_BYTES = BAND_BARS * 8 + 8;
__host__ __device__ inline size_t band_smem_bytes(size_t warps, size_t slice, int rows) {
    return warps * (slice + band_warp_bytes(rows)) + BAND_RING_BYTES + BAND_TAIL_BYTES;
}
static_assert(BAND_RING_BYTES >= 2 * sizeof(Cand), "a warp's candidates must fit in its ring");

// A band lane's state: a Sweep's, with the last row of both columns.
template <class A, int R>
struct Band : Sweep<A, R> {
    typename A::V botG1, botF1;
};

// The first of a lane's R rows whose G in half h is b, or R.
template <class A, int R>
__device__ __forceinline__ int band_row(const typename A::V (&col)[R], const int h, const int32_t b) {
    int row = R;
#pragma unroll
    for (int r = R - 1; r >= 0; --r)
        if (A::get(col[r], h) == b) row = r;
    return row;
}

// Local mode: the columns j and j + 1 (their G in g0, g1) raise the lane's running best to cm in
// some halves. Either the best cell's id, or (band_copies) a copy of both columns in `copy`, the
// lane's uint4s 32 apart, and j as the id.
template <class A, int R>
__device__ __forceinline__ void band_improve(Band<A, R> &sw, const typename A::V (&g0)[R], const typename A::V (&g1)[R],
                                             const int32_t j, const typename A::V cm0, const typename A::V cm, uint4 *copy) {
    if constexpr (band_copies<R>()) {
#pragma unroll
        for (int h = 0; h < A::NH; ++h) {
            const uint32_t mask = A::NH == 1 ? 0xffffffffu : h ? 0xffff0000u : 0xffffu;
            if (((uint32_t)cm ^ (uint32_t)sw.pbest) & mask) {
#pragma unroll
                for (int c = 0; c < R / 4; ++c) {
                    copy[((2 * h) * (R / 4) + c) * 32] = make_uint4((uint32_t)g0[4 * c], (uint32_t)g0[4 * c + 1], (uint32_t)g0[4 * c + 2], (uint32_t)g0[4 * c + 3]);
                    copy[((2 * h + 1) * (R / 4) + c) * 32] = make_uint4((uint32_t)g1[4 * c], (uint32_t)g1[4 * c + 1], (uint32_t)g1[4 * c + 2], (uint32_t)g1[4 * c + 3]);
                }
                (h ? sw.pid1 : sw.pid0) = j;
            }
        }
        sw.pbest = cm;
    } else if (cm != sw.pbest) {
        // In the first column unless the second is higher.
#pragma unroll
        for (int h = 0; h < A::NH; ++h) {
            const int32_t b = A::get(cm, h);
            if (b != A::get(sw.pbest, h)) {
                const bool first = b == A::get(cm0, h);
                (h ? sw.pid1 : sw.pid0) = first ? j * R + band_row<A, R>(g0, h, b) : (j + 1) * R + band_row<A, R>(g1, h, b);
            }
        }
        sw.pbest = cm;
    }
}

// The lane's best cell of the pass as a candidate (see band_improve).
template <class A, int R, int MODE>
__device__ __forceinline__ void band_end(Band<A, R> &sw, const int32_t row0, const int32_t go, const uint4 *copy,
                                         Cand (&cand)[2]) {
    if constexpr (ModeFlags<MODE>::local && band_copies<R>()) {
#pragma unroll
        for (int h = 0; h < A::NH; ++h) {
            int32_t &id = h ? sw.pid1 : sw.pid0;
            if (id < 0) continue;
            const int32_t b = A::get(sw.pbest, h);
            typename A::V g[2][R];
#pragma unroll
            for (int col = 0; col < 2; ++col)
#pragma unroll
                for (int c = 0; c < R / 4; ++c) {
                    const uint4 v = copy[((2 * h + col) * (R / 4) + c) * 32];
                    g[col][4 * c] = v.x;
                    g[col][4 * c + 1] = v.y;
                    g[col][4 * c + 2] = v.z;
                    g[col][4 * c + 3] = v.w;
                }
            const int r0 = band_row<A, R>(g[0], h, b);
            id = r0 < R ? id * R + r0 : (id + 1) * R + band_row<A, R>(g[1], h, b);
        }
    }
    sweep_end<A, R, MODE, true>(sw, row0, go, cand);
}

// Both columns j, j + 1 (1-based) of a step of one lane's R rows, the profile words and the row above
// given, the second column one row behind the first in the instruction stream. `lastG`: the running
// best of the last query row (modes that answer there, lane 31 of the last pass); columns past a
// half's end are never considered, so its running best may run ahead of its candidate there. END:
// one of the columns may be a half's last one (modes that answer there).
template <class A, int R, int MODE, bool END>
__device__ __forceinline__ void band_columns(Band<A, R> &sw, const int32_t j, const uint32_t (&n)[2],
                                             const typename A::V (&pa)[2][R], const typename A::V (&pb)[2][R],
                                             const int32_t row0, const bool last_lane, const typename A::V upG0, const typename A::V upF0,
                                             const typename A::V upG1, const typename A::V upF1, const int32_t qlen,
                                             const int32_t go, const SweepConst<A> &k, typename A::V &lastG,
                                             Cand (&cand)[2], uint4 *copy) {
    typedef typename A::V V;
    typedef ModeFlags<MODE> Fl;
    static_assert(R % 2 == 0, "rows are folded into the columns' maxima in twos");
    V f0 = upF0, f1 = upF1, c0 = upG0, c1 = upG1, g0[R], g1[R], cm0 = sw.pbest, cm1 = k.neggo;
#pragma unroll
    for (int t = 0; t <= R; ++t) {
#pragma unroll
        for (int col = 0; col < 2; ++col) {
            const int r = t - col;
            if (r < 0 || r >= R) continue;
            V &f = col ? f1 : f0, &chain = col ? c1 : c0;
            V(&g)[R] = col ? g1 : g0;
            // Column j's diagonal and left neighbours are the column before it; column j + 1's are j's.
            const V left = col ? g0[r] : sw.Gp[r];
            const V diag = r == 0 ? (col ? upG0 : sw.diag) : (col ? g0[r > 0 ? r - 1 : 0] : sw.Gp[r > 0 ? r - 1 : 0]);
            sw.E[r] = A::addmax(sw.E[r], k.negge, left);
            const V d = A::diag(diag, pa[col][r], pb[col][r]);
            f = A::addmax(f, k.negge, chain);
            if (Fl::local) {
                const V x = A::vadd(A::vmax3_relu(d, sw.E[r], d), k.neggo);
                chain = x;  // F of the next row from x: see sweep_step
                g[r] = A::addmax(f, k.neggo, x);
                if (r & 1) {
                    if (col)
                        cm1 = A::vmax3(cm1, g[r - 1], g[r]);
                    else
                        cm0 = A::vmax3(cm0, g[r - 1], g[r]);
                }
            } else {
                chain = g[r] = A::vadd(A::vmax3(d, sw.E[r], f), k.neggo);
            }
        }
    }
    sw.diag = upG1;
    sw.botG = g0[R - 1];
    sw.botF = f0;
    sw.botG1 = g1[R - 1];
    sw.botF1 = f1;
    if (Fl::local) {
        band_improve<A, R>(sw, g0, g1, j, cm0, A::vmax(cm0, cm1), copy);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) sw.Gp[r] = g1[r];
    if (Fl::last_row && last_lane) {
        const V m = A::vmax3(lastG, sw.botG, sw.botG1);
        if (m != lastG) {
#pragma unroll
            for (int h = 0; h < A::NH; ++h) {
                const int32_t nh = (int32_t)n[h];
                if (j <= nh) consider(cand[h], A::get(sw.botG, h) + go, j, qlen);
                if (j + 1 <= nh) consider(cand[h], A::get(sw.botG1, h) + go, j + 1, qlen);
            }
            lastG = m;
        }
    }
    if constexpr (END && (Fl::last_col || Fl::corner)) {
#pragma unroll
        for (int h = 0; h < A::NH; ++h)
#pragma unroll
            for (int col = 0; col < 2; ++col) {
                if (j + col != (int32_t)n[h]) continue;
                const V(&g)[R] = col ? g1 : g0;
                if (Fl::corner) {
                    if (last_lane) consider(cand[h], A::get(g[R - 1], h) + go, j + col, qlen);
                } else {
#pragma unroll
                    for (int r = 0; r < R; ++r)
                        if (row0 + r >= 1) consider(cand[h], A::get(g[r], h) + go, j + col, row0 + r);
                }
            }
    }
}

// A band warp's profile words of one residue code: row r's in pa[r] (and pb[r], two tables).
template <class A, int R>
__device__ __forceinline__ void band_words(const uint8_t *prof, const uint8_t *prof_hi, const uint32_t code,
                                           const int lane, typename A::V (&pa)[R], typename A::V (&pb)[R]) {
    int a, b;
    A::residues((typename A::RES)code, a, b);
#pragma unroll
    for (int c = 0; c < R / A::EPV; ++c) {
        typename A::V qa[A::EPV], qb[A::EPV];
        A::template load_chunk<R, 32>(prof, prof_hi, a, b, lane, c, qa, qb);
#pragma unroll
        for (int e = 0; e < A::EPV; ++e) {
            pa[c * A::EPV + e] = qa[e];
            pb[c * A::EPV + e] = qb[e];
        }
    }
}

// The sweep of item `item` (a valid item of p.meta) by the whole block, or by every block of a
// thread-block cluster: block b's warps take the passes b * W .. b * W + W - 1 of a round. `bar` is
// an initialised mbarrier whose next wait parity is `phase` (a cluster's blocks: BAND_BARS of them,
// not yet used); the block's dynamic shared memory (`smem`) holds W = blockDim/32 pass slices and
// what band_smem_bytes adds. Every thread of every block must call it. With GPROF (single blocks only)
// the warps read their pass slices from the profile in global memory; `bar` is then unused and `smem` holds the rings and strips alone.
template <class A, int R, int MODE, bool GPROF = false>
__device__ __forceinline__ void band_item(const ScanParams &p, const uint32_t item, uint8_t *smem,
                                          uint64_t *bar, uint32_t &phase) {
    typedef typename A::V V;
    typedef typename A::RES RES;
    typedef ModeFlags<MODE> Fl;
    constexpr int G = 32;
    constexpr int RPP = G * R;
    // The residue codes of a column pair as one load: two 16-bit or two 8-bit codes.
    typedef typename TwoCodes<A>::W W2;
    constexpr int CODE_BITS = TwoCodes<A>::BITS;
    constexpr uint32_t CODE_MASK = (1u << CODE_BITS) - 1u;
    static_assert(R % A::EPV == 0, "rows per lane must fill whole profile vectors");
    const int W = blockDim.x / G;
    const int warp = threadIdx.x / G, lane = threadIdx.x % G;
    const int crank = cluster_rank(), csize = cluster_size();
    const int WT = W * csize;          // warps of the cluster
    const int gw = crank * W + warp;   // this warp's index in the cluster
    const ItemMeta meta = p.meta[item];
#ifdef HY_BOUNDS
    // Every warp checks the item (the same answer in all of them), so all skip it together.
    if (!item_in_bounds<A, G>(p, meta, lane, true)) {
        if (threadIdx.x == 0) atomicExch(p.err, ERR_BOUNDS);
        return;
    }
#endif
    const int32_t w = (int32_t)meta.w;
    const RES *res = reinterpret_cast<const RES *>(p.res) + meta.col_off;
    const W2 *res2 = reinterpret_cast<const W2 *>(res);
    uint4 *bnd = reinterpret_cast<uint4 *>(reinterpret_cast<uint2 *>(p.boundary) + (meta.col_off - p.bnd_col0));
    // Ring `warp` holds the row above this warp (ring 0: filled by warp 0 itself), ring warp + 1
    // this warp's last row.
    uint8_t *rings = smem + (GPROF ? 0 : (size_t)W * p.pass_bytes);
    uint4 *in = reinterpret_cast<uint4 *>(rings + (size_t)warp * BAND_RING_BYTES);
    uint4 *out = in + BAND_RING;
    uint8_t *own = rings + (size_t)(W + 1) * BAND_RING_BYTES + (size_t)warp * (band_warp_bytes(R) - BAND_RING_BYTES);
    W2 *strip = reinterpret_cast<W2 *>(own);
    uint32_t *words = reinterpret_cast<uint32_t *>(rings + (size_t)(W + 1) * BAND_RING_BYTES +
                                                   (size_t)W * (band_warp_bytes(R) - BAND_RING_BYTES) + BAND_BARS * 8);
    uint32_t &s_flag = words[0];
    uint32_t &s_sent = words[1];  // ring blocks of the round that this block has sent
    uint4 *copy = reinterpret_cast<uint4 *>(own + BAND_STRIP_BYTES) + lane;
    SweepConst<A> k;
    k.negge = A::splat(-(int64_t)p.ge);
    k.neggo = A::splat(-(int64_t)p.go);
    k.Sv = A::splat(p.sentinel);
    k.top_free_g = k.neggo;
    Cand cand[2] = {{INT32_MIN, INT32_MAX, INT32_MAX}, {INT32_MIN, INT32_MAX, INT32_MAX}};
    const int pairs = (w + 1) / 2;  // column pairs
    const int pass_steps = pairs + G - 1;
    // Between blocks: ring blocks of BAND_K pairs, those of one slot in turn.
    uint64_t *full = bar + 1, *empty = full + BAND_SLOTS;
    const int n_blk = (pairs + BAND_K - 1) / BAND_K;
    uint32_t full_ph = 0, empty_ph = 0;  // per slot: parity of its next wait at the round's start
    auto blk_bytes = [&](int blk) { return 16u * (uint32_t)min(BAND_K, pairs - blk * BAND_K); };
    // The ring block at which this warp gave up on the row above or on space for its own row.
    constexpr int NEVER = INT32_MAX;
    int recv_end = NEVER, send_end = NEVER;
    bool gave = false;           // any warp of the block has
    // The wait for the rows still on their way to this block (every block's sweep is over).
    auto drain = [&]() {
        if (threadIdx.x == 0 && recv_end != NEVER) {
            const int sent = (int)ld_cluster_u32(&s_sent, crank - 1);
            for (int blk = recv_end; blk < sent; ++blk)
                mbar_wait_cluster(full + blk % BAND_SLOTS, ((full_ph >> (blk % BAND_SLOTS)) + (uint32_t)(blk / BAND_SLOTS)) & 1u,
                                  1u << 24);
        }
        __syncwarp();
    };
    const int rounds = (p.n_passes + WT - 1) / WT;
    for (int round = 0; round < rounds; ++round) {
        const int first = round * WT;
        const int cnt = min(WT, p.n_passes - first);          // warps of the cluster with a pass
        const int bcnt = max(0, min(W, cnt - crank * W));      // ... of this block
        if (!GPROF) {
            bool fail = false;
            if (bcnt > 0) {
                if (threadIdx.x == 0)
                    bulk_load(smem, p.profile + (size_t)(first + crank * W) * p.pass_bytes,
                              (uint32_t)bcnt * p.pass_bytes, bar);
                const bool ok = mbar_wait_bounded(bar, phase & 1u, p.wait_polls);
                phase ^= 1u;
                fail = __syncthreads_or(!ok);
            }
            if (csize > 1 && threadIdx.x == 0 && crank > 0 && bcnt > 0 && w > 0 && !gave)
                for (int blk = 0; blk < min(BAND_SLOTS, n_blk); ++blk) mbar_expect(full + blk, blk_bytes(blk));
            if (cluster_any(fail || gave, &s_flag, csize)) {
                if (threadIdx.x == 0 && fail) wait_gave_up(p.err, bar, 1u, phase ^ 1u);  // the round's copy
                if (csize > 1) {
                    drain();
                    cluster_barrier();
                }
                return;
            }
        }
        const int pass = first + gw;
        const bool mine = gw < cnt && w > 0;
        const bool first_pass = pass == 0, last_pass = pass == p.n_passes - 1;
        const bool last_lane = last_pass && lane == G - 1;
        // Where the row above warp 0 comes from and where a block's last row goes.
        const bool from_block = warp == 0 && crank > 0;
        const bool to_block = warp == W - 1 && gw + 1 < cnt;
        const bool to_bnd = !last_pass && gw + 1 == cnt;  // the round's last row: for the next round
        auto wait_cluster = [&](uint64_t *b, uint32_t parity) -> bool {
            const bool ok = mbar_wait_cluster(b, parity & 1u, p.row_polls);
            if (!ok) atomicExch(p.err, ERR_WAIT);
            return __all_sync(0xffffffffu, ok);
        };
        const int32_t row0 = p.vrow0 + pass * RPP + lane * R;
        const uint8_t *prof = GPROF ? p.profile + (size_t)min(pass, p.n_passes - 1) * p.pass_bytes
                                    : smem + (size_t)warp * p.pass_bytes;
        const uint8_t *prof_hi = prof + (A::TABLES - 1) * (p.pass_bytes / A::TABLES);
        Band<A, R> sw;
        sweep_begin<A, R, MODE>(sw, row0, p.go, p.ge, k.Sv);
        sw.botG1 = sw.botF1 = sw.botG;
        sw.pbest = k.neggo;  // H = 0: only a cell above the border's 0 is tracked
        V lastG = A::splat(A::VMIN);
        // Codes of column pair c >= 0. An odd item's last pair holds the padding symbol in its second
        // column, whose cells never exceed a real one in local mode and are never considered in others.
        const uint32_t pad = A::pad_code(p.letters);
        auto code_at = [&](int c) -> W2 {
            const uint32_t v = 2 * c < w ? (uint32_t)res2[c] : pad;
            return (W2)(2 * c + 1 < w ? v : (v & CODE_MASK) | (pad << CODE_BITS));
        };
        // This lane's pair of the 32 pairs before the strip's base, from it on, and after those.
        W2 c_prev = 0, c_cur = 0, c_next = 0;  // (0: a valid letter)
        V pa[2][R], pb[2][R];  // profile words of the coming step
        uint32_t code = 0;     // residue codes of the step after it
        auto prof_words = [&](const uint32_t cc, V (&a)[2][R], V (&b)[2][R]) {
            band_words<A, R>(prof, prof_hi, cc & CODE_MASK, lane, a[0], b[0]);
            band_words<A, R>(prof, prof_hi, cc >> CODE_BITS, lane, a[1], b[1]);
        };
        if (mine) {
            c_cur = code_at(lane);
            c_next = code_at(G + lane);
            strip[lane] = 0;
            strip[G + lane] = c_cur;
            __syncwarp();
            prof_words(strip[G - lane], pa, pb);
            code = strip[G + 1 - lane];
        }
        // Step s = s0 + i of the window at s0: `up` the row above at lane 0's pair, `cp` the strip at
        // this lane's pair of step s0, `op` the ring slot of lane 31's pair. EDGE: lanes may not have
        // started, be done (the row above is not defined past the item), or be at a half's last column.
        auto step = [&](auto EDGE, const int s0, const int i, const uint4 up, const W2 *cp, uint4 *op) {
            V upG0 = __shfl_up_sync(0xffffffffu, sw.botG, 1, G);
            V upF0 = __shfl_up_sync(0xffffffffu, sw.botF, 1, G);
            V upG1 = __shfl_up_sync(0xffffffffu, sw.botG1, 1, G);
            V upF1 = __shfl_up_sync(0xffffffffu, sw.botF1, 1, G);
            if (lane == 0) {
                upG0 = (V)up.x;
                upF0 = (V)up.y;
                upG1 = (V)up.z;
                upF1 = (V)up.w;
            }
            V na[2][R], nb[2][R];
            prof_words(code, na, nb);
            code = cp[i + 2];
            constexpr bool edge = decltype(EDGE)::value;
            const int c = s0 + i - lane;
            if (!edge || (c >= 0 && c < pairs))
                band_columns<A, R, MODE, edge>(sw, 2 * c + 1, meta.n, pa, pb, row0, last_lane, upG0, upF0, upG1, upF1,
                                               p.qlen, p.go, k, lastG, cand, copy);
            if (lane == G - 1)
                *op = make_uint4((uint32_t)sw.botG, (uint32_t)sw.botF, (uint32_t)sw.botG1, (uint32_t)sw.botF1);
#pragma unroll
            for (int col = 0; col < 2; ++col)
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    pa[col][r] = na[col][r];
                    pb[col][r] = nb[col][r];
                }
        };
        // Whether a half's last column lies among the window's (modes that answer there).
        auto ends_in = [&](int s0) {
            if (!Fl::last_col && !Fl::corner) return false;
            bool in_window = false;
#pragma unroll
            for (int h = 0; h < A::NH; ++h) {
                const int c = ((int)meta.n[h] - 1) >> 1;  // the pair of half h's last column
                in_window |= c > s0 - G && c < s0 + BAND_K;
            }
            return in_window;
        };
        const int total = bcnt > 0 ? pass_steps + BAND_LAG * (bcnt - 1) : 0;
        for (int t0 = 0; t0 < total; t0 += BAND_K) {
            const int s0 = t0 - BAND_LAG * warp;
            if (mine && s0 >= 0 && s0 < pass_steps) {
                if (from_block) {
                    // Block b - 1's last warp writes the row above: the ring block read a window ago
                    // goes back to it, and the next one must have arrived.
                    const int blk = s0 / BAND_K, old = blk - 1;
                    if (recv_end == NEVER) {
                        if (old >= 0 && old + BAND_SLOTS < n_blk && lane == 0) {
                            mbar_expect(full + old % BAND_SLOTS, blk_bytes(old + BAND_SLOTS));
                            mbar_arrive_cluster(cluster_addr(empty + old % BAND_SLOTS, crank - 1));
                        }
                        if (blk < n_blk &&
                            !wait_cluster(full + blk % BAND_SLOTS, (full_ph >> (blk % BAND_SLOTS)) + (uint32_t)(blk / BAND_SLOTS)))
                            recv_end = blk;
                    }
                } else if (warp == 0 && lane < BAND_K) {
                    // The row above of the window's pairs: the top border, or the boundary row that
                    // the round before wrote.
                    const int c = s0 + lane;
                    uint4 v = make_uint4(0, 0, 0, 0);
                    if (first_pass) {
                        auto top = [&](int j) {
                            return (uint32_t)(Fl::top_free ? k.top_free_g : A::splat(-gap_pen(p.go, p.ge, j) - p.go));
                        };
                        v = make_uint4(top(2 * c + 1), (uint32_t)k.Sv, top(2 * c + 2), (uint32_t)k.Sv);
                    } else if (c < pairs) {
                        v = __ldcg(bnd + c);
                    }
                    in[c % BAND_RING] = v;
                }
                __syncwarp();  // no lane reads the strip's old codes any more
                if (s0 % G == 0) {
                    strip[lane] = c_prev;
                    strip[G + lane] = c_cur;
                    if (lane < 2) strip[2 * G + lane] = c_next;
                    c_prev = c_cur;
                    c_cur = c_next;
                    c_next = code_at(s0 + 2 * G + lane);
                }
                __syncwarp();
                const uint4 *ip = in + s0 % BAND_RING;
                const W2 *cp = strip + G + s0 % G - lane;
                // Lane 31 is at pair s - 31: slots 1 .. K - 1 of the ring's block at s0 - 32, then slot
                // 0 of the next block.
                uint4 *op = out + (s0 + BAND_RING - G) % BAND_RING + 1;
                uint4 *op_last = out + (s0 + BAND_RING - G + BAND_K) % BAND_RING;
                uint4 up = ip[0];
                auto window = [&](auto EDGE) {
                    for (int i0 = 0; i0 < BAND_K; i0 += 4) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint4 next = ip[i + 1];
                            step(EDGE, s0 + i0, i, up, cp, i == 3 && i0 == BAND_K - 4 ? op_last : op + i);
                            up = next;
                        }
                        ip += 4;
                        cp += 4;
                        op += 4;
                    }
                };
                if (s0 >= G && s0 + BAND_K <= pairs && !ends_in(s0))
                    window(std::false_type());
                else
                    window(std::true_type());
                if (to_bnd || to_block) {
                    static_assert(G == 2 * BAND_K, "a window's last pair begins a ring block");
                    __syncwarp();
                    const int c = s0 - (G - 1) + lane;
                    const bool has = lane < BAND_K && c >= 0 && c < pairs;
                    if (to_bnd) {
                        if (has) bnd[c] = out[c % BAND_RING];
                    } else {
                        // Pairs s0 - 31 .. s0 - 16, the last one the first of its ring block, whose
                        // earlier pairs the next block must have read.
                        const int blk = s0 / BAND_K - 1;
                        if (send_end == NEVER && blk >= BAND_SLOTS && blk < n_blk &&
                            !wait_cluster(empty + blk % BAND_SLOTS,
                                          (empty_ph >> (blk % BAND_SLOTS)) + (uint32_t)(blk / BAND_SLOTS - 1)))
                            send_end = blk;
                        if (has && c / BAND_K < send_end)
                            st_async_v4(cluster_addr(in - (size_t)warp * BAND_RING + c % BAND_RING, crank + 1), out[c % BAND_RING],
                                        cluster_addr(full + (c / BAND_K) % BAND_SLOTS, crank + 1));
                    }
                }
            }
            __syncthreads();
        }
        if (to_block && lane == 0) s_sent = (uint32_t)min(send_end, n_blk);
        if (mine) band_end<A, R, MODE>(sw, row0, p.go, copy, cand);
        gave = __syncthreads_or(recv_end != NEVER || send_end != NEVER);  // the slices and rings may be refilled
        if (gave) continue;  // (the phases stay those of the round that gave up)
        for (int k2 = 0; k2 < BAND_SLOTS; ++k2) {
            const int uses = n_blk > k2 ? (n_blk - k2 + BAND_SLOTS - 1) / BAND_SLOTS : 0;
            full_ph ^= (uint32_t)(uses & 1) << k2;
            empty_ph ^= (uint32_t)(max(uses - 1, 0) & 1) << k2;
        }
    }
    // Reduce every lane's candidates: inside each warp, then across warps in shared memory.
    Cand(*s_cand)[2] = reinterpret_cast<Cand(*)[2]>(rings);  // (the last round's rings have been read)
    __syncthreads();
#pragma unroll
    for (int h = 0; h < A::NH; ++h) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            Cand o;
            o.s = __shfl_xor_sync(0xffffffffu, cand[h].s, off);
            o.col = __shfl_xor_sync(0xffffffffu, cand[h].col, off);
            o.row = __shfl_xor_sync(0xffffffffu, cand[h].row, off);
            if (better(o, cand[h])) cand[h] = o;
        }
        if (lane == 0) s_cand[warp][h] = cand[h];
    }
    if (csize > 1)
        cluster_barrier();  // every block's candidates are in its shared memory
    else
        __syncthreads();
    if (csize > 1) drain();
    if (threadIdx.x == 0 && crank == 0) {
        // A block of the cluster that gave up has set the error word before the barrier.
        const int err = csize > 1 ? *(volatile int *)p.err : 0;
        for (int h = 0; h < A::NH; ++h) {
            const uint32_t idx = meta.idx[h];
            if (idx == NO_INDEX) continue;
            Cand c = border_seed<MODE>(p.qlen, (int32_t)meta.n[h], p.go, p.ge);
            for (int b = 0; b < csize; ++b)
                for (int k = 0; k < W; ++k) {
                    Cand o = s_cand[k][h];
                    if (b > 0) {
                        o.s = (int32_t)ld_cluster_u32(&s_cand[k][h].s, b);
                        o.col = (int32_t)ld_cluster_u32(&s_cand[k][h].col, b);
                        o.row = (int32_t)ld_cluster_u32(&s_cand[k][h].row, b);
                    }
                    if (better(o, c)) c = o;
                }
            if (err) continue;
            if (p.ends_out) {
                if (idx == ~(uint32_t)(*p.best_key & 0xffffffffu)) {
                    p.ends_out[0] = c.s;
                    p.ends_out[1] = c.row - 1;
                    p.ends_out[2] = c.col - 1;
                }
            } else {
                p.scores[idx] = c.s;
                p.qend[idx] = c.row - 1;
                p.tend[idx] = c.col - 1;
                if (p.best_key) atomicMax(p.best_key, hit_key(c.s, idx));
            }
        }
    }
    if (csize > 1) cluster_barrier();  // block 0 has read every block's candidates
}

// Warps of a band block at most: 128 registers a thread. (The sweep of two columns needs 110 to 124 with
// 4 rows per lane; at 64, for 32 warps, 8 rows spilled 0.4 to 2 KB a thread and took twice as long.)
constexpr int BAND_WARPS = 16;

template <class A, int R, int MODE, bool GPROF = false>
__global__ void __launch_bounds__(32 * BAND_WARPS, 1) band_kernel(const ScanParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    // The item *item_ptr, or an item a cluster.
    const uint32_t item = p.item_ptr ? *p.item_ptr : p.item_base + blockIdx.x / (uint32_t)cluster_size();
    if (item == NO_INDEX || item >= p.n_items) return;  // the same for every thread of the cluster
    const int W = blockDim.x / 32;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + band_smem_bytes(W, GPROF ? 0 : p.pass_bytes, R) - BAND_TAIL_BYTES);
    if (threadIdx.x == 0) {
        for (int i = 0; i < BAND_BARS; ++i) mbar_init(bar + i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t phase = 0;
    band_item<A, R, MODE, GPROF>(p, item, smem, bar, phase);
}

// ---- the batched pairwise kernel (align_pairs) -----------------------------------------------
//
// Every item carries its own queries (one per half, of equal length), so each group builds the
// profile slice of its own pass in its own region of shared memory, then sweeps it. Groups of a
// warp run their items' passes in step; there is no block-wide synchronisation.
struct PairParams {
    const ItemMeta *meta;  // n[h]: target lengths; idx[h]: pair indices
    const uint32_t *qlen;  // per item
    const uint64_t *qoff;  // per item and half: offset of the query residues in q_res
    uint32_t item_base;    // items [item_base, n_items) run
    uint32_t n_items;
    const uint8_t *q_res;
    const void *res;       // packed target residues, as in the scan
    const int32_t *matrix;
    int32_t al;
    int32_t lim;
    int32_t go, ge;
    int32_t sentinel;
    int top_free;
    uint32_t group_bytes;  // shared memory per group (both halves of one pass slice)
    void *boundary;
    int32_t *scores;
    int32_t *qend;
    int32_t *tend;
    // Global-memory-profile form (alphabets whose group profiles do not fit in shared memory):
    // group g of block b builds and reads its profile at gprof + (b * groups_per_block + g) *
    // group_bytes.
    uint8_t *gprof;
    // Column-maxima form (align_pair_position_max): pair half h of item i writes the maximum of H
    // over each target column to colmax + toff[2 * i + h] + column.
    int32_t *colmax;
    const uint64_t *toff;
};

template <class A, int G, int R>
__device__ __forceinline__ void build_group_profile(uint8_t *dst, const uint8_t *q, int32_t qlen,
                                                    int32_t row_base, const int32_t *matrix,
                                                    int32_t al, int32_t lim, int32_t go,
                                                    int top_free, int lane, int table) {
    static_assert(R % A::EPV == 0 && R >= A::EPV, "rows per lane must fill whole profile vectors");
    constexpr int KCH = R / A::EPV;
    typename A::PE *out = reinterpret_cast<typename A::PE *>(dst);
    const int64_t pad = -(int64_t)lim - 1 + go;
    for (int letter = 0; letter <= al; ++letter) {
#pragma unroll
        for (int k = 0; k < KCH; ++k) {
#pragma unroll
            for (int e = 0; e < A::EPV; ++e) {
                const int32_t row = row_base + lane * R + k * A::EPV + e;
                int64_t v;
                if (row <= 0) {
                    v = top_free ? go : 0;
                } else if (letter == al) {
                    v = pad;
                } else {
                    int64_t sub = matrix[(int32_t)q[row - 1] * al + letter];
                    if (sub < -(int64_t)lim - 1) sub = -(int64_t)lim - 1;
                    if (sub > lim) sub = lim;
                    v = sub + go;
                }
                out[(((size_t)letter * KCH + k) * G + lane) * A::EPV + e] = A::word(v, table);
            }
        }
    }
}

template <class A, int G, int R, int MODE, bool ENDS, bool GPROF = false, bool COLMAX = false>
__global__ void __launch_bounds__(256) pairs_kernel(const PairParams p) {
    typedef typename A::V V;
    constexpr int RPP = G * R;
    extern __shared__ __align__(128) uint8_t smem[];
    const int lane = threadIdx.x % G;
    const int gib = threadIdx.x / G;
    const uint32_t item = p.item_base + blockIdx.x * (blockDim.x / G) + gib;
    const bool active = item < p.n_items;
    ItemMeta meta;
    int32_t qlen = 0;
    if (active) {
        meta = p.meta[item];
        qlen = (int32_t)p.qlen[item];
    } else {
        meta.col_off = 0;
        meta.w = 0;
        meta.n[0] = meta.n[1] = 0;
        meta.idx[0] = meta.idx[1] = NO_INDEX;
    }
    const int32_t n_passes = (qlen + RPP - 1) / RPP;
    const int32_t vrow0 = qlen - n_passes * RPP + 1;
    const uint8_t *qa = active ? p.q_res + p.qoff[2 * (size_t)item] : p.q_res;
    const uint8_t *qb = (active && A::NH > 1 && meta.idx[1] != NO_INDEX) ? p.q_res + p.qoff[2 * (size_t)item + 1] : qa;
    // The group's region: the low-half table of query a, then (int16x2) the high-half table of b.
    uint8_t *gprof_a = GPROF ? p.gprof + ((size_t)blockIdx.x * (blockDim.x / G) + gib) * p.group_bytes
                             : smem + (size_t)gib * p.group_bytes;
    uint8_t *gprof_b = gprof_a + (A::TABLES - 1) * (p.group_bytes / A::TABLES);
    const V Sv = A::splat(p.sentinel);
    const typename A::RES *res = reinterpret_cast<const typename A::RES *>(p.res) + meta.col_off;
    V *bnd = reinterpret_cast<V *>(p.boundary) + 2 * meta.col_off;
    const uint32_t wmax = __reduce_max_sync(0xffffffffu, meta.w);
    const int steps = wmax == 0 ? 0 : (int)wmax + G - 1;
    const int32_t pmax = (int32_t)__reduce_max_sync(0xffffffffu, (uint32_t)n_passes);
    ColMaxOut cmo;
    if constexpr (COLMAX) {
        cmo.p[0] = cmo.p[1] = p.colmax;
        if (active) {
            cmo.p[0] = p.colmax + p.toff[2 * (size_t)item];
            cmo.p[1] = p.colmax + p.toff[2 * (size_t)item + 1];
        }
        cmo.atomic = n_passes > 1;
    }

    V best = A::splat(ModeFlags<MODE>::local && !ENDS ? -(int64_t)p.go : 0);
    Cand cand[2] = {{INT32_MIN, INT32_MAX, INT32_MAX}, {INT32_MIN, INT32_MAX, INT32_MAX}};
    for (int pass = 0; pass < pmax; ++pass) {
        const bool mine = pass < n_passes;
        const int32_t row_base = vrow0 + pass * RPP;
        if (mine) {
            build_group_profile<A, G, R>(gprof_a, qa, qlen, row_base, p.matrix, p.al, p.lim, p.go,
                                         p.top_free, lane, 0);
            if (A::TABLES > 1)
                build_group_profile<A, G, R>(gprof_b, qb, qlen, row_base, p.matrix, p.al, p.lim,
                                             p.go, p.top_free, lane, 1);
        }
        __syncwarp();
        // `steps` stays warp-uniform; a group past its last pass sweeps zero columns.
        const int w_here = mine ? (int)meta.w : 0;
        const int w_min = (int)__reduce_min_sync(0xffffffffu, (uint32_t)w_here);
        sweep_pass<A, G, R, MODE, ENDS, COLMAX>(lane, steps, w_min, w_here, meta.n, res, gprof_a,
                                                gprof_b, row_base + lane * R, pass == 0,
                                                pass == n_passes - 1, bnd, qlen, p.go, p.ge, Sv, best,
                                                cand, COLMAX ? &cmo : nullptr);
        __syncwarp();
    }
    if constexpr (!COLMAX)
        finish_item<A, G, MODE, ENDS>(lane, active, meta, qlen, p.go, p.ge, best, cand, p.scores,
                                      p.qend, p.tend, nullptr);
}

// ---- query profile ----------------------------------------------------------------------------
//
// Layout of one pass slice: [table < TABLES][letter 0..al][chunk k < R/EPV][lane < G][EPV words],
// word e of chunk k of lane L being grid row vrow0 + pass*G*R + L*R + k*EPV + e. Letter `al` is the
// padding symbol. Values are P = clamp(sub, -(lim+1), lim) + go; virtual rows (<= 0) get go (free
// top border) or 0 (penalised top border); the padding symbol gets -(lim+1) + go. For int16x2 the
// first table holds each value in the low half of its word, the second in the high half.
// Words [first, total) in steps of `stride` of the profile described above.
template <class A, int G, int R>
__device__ __forceinline__ void build_profile_words(const uint8_t *q, const int32_t *matrix,
                                                    int32_t al, int32_t go, int32_t lim,
                                                    int top_free, int32_t vrow0, int32_t n_passes,
                                                    typename A::PE *out, int64_t first,
                                                    int64_t stride) {
    static_assert(R % A::EPV == 0 && R >= A::EPV, "rows per lane must fill whole profile vectors");
    constexpr int KCH = R / A::EPV;
    const int64_t per_table = A::letters(al) * G * R;
    const int64_t per_pass = per_table * A::TABLES;
    const int64_t total = per_pass * n_passes;
    for (int64_t i = first; i < total; i += stride) {
        const int64_t pass = i / per_pass;
        const int table = (int)((i % per_pass) / per_table);
        int64_t rem = i % per_table;
        const int e = (int)(rem % A::EPV);
        rem /= A::EPV;
        const int lane = (int)(rem % G);
        rem /= G;
        const int k = (int)(rem % KCH);
        const int letter = (int)(rem / KCH);
        const int64_t row = vrow0 + pass * (G * R) + (int64_t)lane * R + k * A::EPV + e;
        const int64_t pad = -(int64_t)lim - 1 + go;
        // Profile value of target symbol l at this row.
        auto value = [&](int l) -> int64_t {
            if (row <= 0) return top_free ? go : 0;
            if (l == al) return pad;
            int64_t sub = matrix[(int64_t)q[row - 1] * al + l];
            if (sub < -(int64_t)lim - 1) sub = -(int64_t)lim - 1;
            if (sub > lim) sub = lim;
            return sub + go;
        };
        if constexpr (A::PAIRTAB)
            out[i] = A::pair_word(value(letter / (al + 1)), value(letter % (al + 1)));
        else
            out[i] = A::word(value(letter), table);
    }
}

template <class A, int G, int R>
__global__ void build_profile_kernel(const uint8_t *q, int32_t qlen, const int32_t *matrix,
                                     int32_t al, int32_t go, int32_t lim, int top_free,
                                     int32_t vrow0, int32_t n_passes, typename A::PE *out) {
    (void)qlen;
    build_profile_words<A, G, R>(q, matrix, al, go, lim, top_free, vrow0, n_passes, out,
                                 blockIdx.x * (int64_t)blockDim.x + threadIdx.x,
                                 (int64_t)gridDim.x * blockDim.x);
}

}  // namespace hy
