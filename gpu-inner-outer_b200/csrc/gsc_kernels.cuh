// gsc_kernels.cuh -- launch wrappers shared between the kernel files and the C ABI layer.
#pragma once

#include <algorithm>
#include <cstdint>
#include <mutex>
#include <set>
#include <utility>

#include <cuda_runtime.h>

#include "gsc_common.cuh"

namespace gsc_b200 {

// Launch of `k` that may begin while the kernel queued before it on `st`
// drains (programmatic stream serialization); `k` starts with pdl_wait().
// Under stream capture the dependency becomes a programmatic graph edge.
template <typename... KArgs, typename... Args>
cudaError_t launch_pdl(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, static_cast<KArgs>(args)...);
}

// Opts `k` in to kFusedSmemOptIn bytes of dynamic shared memory on the current
// device, once per device.  Launches may come from several host threads (a
// server's loop and the caller's); setting the attribute twice is harmless.
constexpr size_t kFusedSmemOptIn = 220 * 1024;
template <typename... KArgs>
cudaError_t allow_smem(void (*k)(KArgs...)) {
    static std::mutex mu;
    static std::set<std::pair<int, const void*>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (done.count({dev, reinterpret_cast<const void*>(k)})) return cudaSuccess;
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kFusedSmemOptIn));
    if (e == cudaSuccess) done.insert({dev, reinterpret_cast<const void*>(k)});
    return e;
}

// ---- abstraction (resident nominal successors) ------------------------------------------
// xn[xy_plane(i2, i3, j)*n0 + i0] = nominal x after K Euler substeps (model.hpp:26-46),
// yn likewise over i1.  cosT/sinT[(i2*mw + jw)*K + k], vseq[(i3*ma + ja)*K + k].
cudaError_t launch_nominal_xy(const GridInfo& g, const double* cosT, const double* sinT, const double* vseq,
                              double* xn, double* yn, cudaStream_t st);

// ---- query preparation ------------------------------------------------------------------
struct MaskArgs {
    const double* obstacles;  // [n][8] device
    uint8_t* valid;           // [S]
    uint8_t* cand;            // [S]
    int build_valid;          // 0: valid already filled by the caller's mask
    int build_cand;
    const uint8_t* safe;      // caller's constraint mask (rank 2 or 4), or null: use the constraint kind
    int safe_rank;
    // Bit-sliced sets to fill too (or null): valid, candidate, unsafe (by
    // cmp_safe; none where that is null), valid and safe.
    bword *validb, *candb, *unsafeb, *srcb;
    const uint8_t* cmp_safe;  // safety at the centres (rank cmp_rank), to count cells whose validity differs
    int cmp_rank;
    unsigned long long* counts;  // [0] valid, [1] candidate, [2] candidate-not-valid, [4] valid != safe
};
cudaError_t launch_masks(const GridInfo& g, const QueryInfo& q, const MaskArgs& a, cudaStream_t st);
cudaError_t launch_safe2(const GridInfo& g, const QueryInfo& q, uint8_t* safe2, cudaStream_t st);

// Per-axis quantised boxes.  xt/yt: [xy_plane][n0|n1], zt: [n2][mw], wt: [n3][ma], packed
// lo | hi << 16 or kReject.  flags |= 1 if an accepted non-wrap interval is empty (hi < lo),
// |= 2 if one is wider than 32 cells.  flags[1] |= 1 << p for every accepted y interval of
// 2^p .. 2^(p+1) - 1 cells, flags[2] |= 1 << (ny - 1) for one of ny; flags |= 4 if an x interval is wider
// than 17 cells.
// shorts (or null): per plane its x and y boxes in short, {hx, hy, yr, xr}: hx = b - a + 1 | a << 8 of the x boxes
// [i + a, i + b], with kBoxX where they are alike, |a|, |b| < 32, and the cells with one (xr: first |
// end << 16) are in a row, and kBoxY likewise for the y boxes (hy, yr).
constexpr uint32_t kBoxX = 1u << 16, kBoxY = 1u << 17;
cudaError_t launch_axis_tables(const GridInfo& g, const QueryInfo& q, const double* xn, const double* yn,
                               const double* thf, const double* vf, uint32_t* xt, uint32_t* yt, uint32_t* zt,
                               uint32_t* wt, uint4* shorts, unsigned int* flags, cudaStream_t st);

// Bit-sliced sets: g.sw words per (theta, v) slice, of which word y*W + w
// holds cells 32*w .. 32*w + 31 of row y.
cudaError_t launch_unpack_bits(const GridInfo& g, const bword* bits, uint8_t* out, cudaStream_t st);
// n words from src to dst by one small kernel (dst may be pinned host memory
// mapped into the device's address space).
cudaError_t launch_store_words(const uint32_t* src, uint32_t* dst, uint32_t n, cudaStream_t st);

// ---- 4-D inclusive prefix tables (int32, zero first plane per dimension) -----------------
// mode 0: valid; 1: valid && !reach (b = reach); 2: !safe (4-D safe mask).
// Built in two passes (x-y per (theta, v) slice, then theta-v per (x tile,
// y)) when a slice and a theta-v plane fit shared memory, else one pass per
// dimension.  ev (optional, prefix4_launches(g) events): ev[k] is recorded
// after pass k + 1.
cudaError_t launch_prefix4(const GridInfo& g, int mode, const uint8_t* a, const uint8_t* b, int32_t* table,
                           const FixControl* ctl, cudaStream_t st, cudaEvent_t* ev = nullptr);
// Kernels launch_prefix4 launches for this grid.
uint32_t prefix4_launches(const GridInfo& g);
// 2-D prefix of !safe2 over (x, y): (n0+1)*(n1+1) entries, stride n0+1.
cudaError_t launch_prefix2_unsafe(const GridInfo& g, const uint8_t* safe2, int32_t* table, cudaStream_t st);

// ---- stored per-pair boxes --------------------------------------------------------------
// Box widths present in a problem: theta widths kval[0..nk) and v widths
// lval[0..nl), ascending; combo (ki, li) indexes the dilated copies.
constexpr int kMaxDilate = 8;
struct DilateArgs {
    uint32_t nk, nl;
    uint32_t kval[kMaxDilate];
    uint32_t lval[kMaxDilate];
};
// Box table of the stored method: a set ORed over every (y, theta, v) box
// width in use, as overlapping 32-bit words (word h of a row covers x cells
// 16 h .. 16 h + 31), so that any box of at most 17 x cells is one word and a
// mask of it.  Copy c = (y width's rank * nk + k) * nl + l, words
// kBoxTableHead + ((c * slices + slice) * n1 + y) * hw + h; the head is all ones.
constexpr uint32_t kBoxTableHead = 4, kBoxBits = 17;
struct StoredBits {
    uint32_t copies;    // 0: prefix counts instead
    uint32_t ywidths;   // bit ny - 1 for every y width ny
    uint32_t nk, nl;
    uint32_t hw;        // words a row
    uint32_t rows, tiles, smem;   // rows a block, blocks a slice, and its shared memory
};
struct StoredBuildArgs {
    const uint32_t *xt, *yt, *zt, *wt;
    const uint8_t* safe;      // rank 2 or 4
    int safe_rank;
    const int32_t* unsafe2;   // rank 2 prefix
    const int32_t* unsafe4;   // rank 4 prefix
    const int32_t* pvalid;    // 4-D valid prefix
    StoredBits bits;          // with copies: boxes hold {word, mask} of the box table, vbits the valid set's
    const uint32_t* vbits;
    const uint8_t *kidx, *lidx;
    uint2* boxes;             // [M][S_pad]: one byte per bound (every dimension <= 255 cells)
    uint64_t S_pad;
    uint4* boxes16;           // [M][S]: 16 bits per bound, when a dimension has more than 255 cells
    int wide;                 // 1: boxes16 in use
    unsigned long long* valid_pairs;   // abstraction-valid pairs (before the V(box) > 0 fold)
};
cudaError_t launch_stored_build(const GridInfo& g, const StoredBuildArgs& a, cudaStream_t st);

// Reference-format abstraction (pair = s * M + j), abstraction.hpp:161-209.
struct ExportArgs {
    const uint32_t *xt, *yt, *zt, *wt;
    const uint8_t* safe;
    int safe_rank;
    const int32_t* unsafe2;
    const int32_t* unsafe4;
    uint32_t* min_flat;
    uint32_t* max_flat;
    uint8_t* valid;
    uint64_t pair_begin, pair_count;
};
cudaError_t launch_export(const GridInfo& g, const ExportArgs& a, cudaStream_t st);

// ---- fixpoint ---------------------------------------------------------------------------
struct StoredFixArgs {
    StoredBits bits;          // with copies: boxes, dbits and table in place of pd
    DilateArgs dil;
    bword* dbits;             // D = valid && !reachable, bit-sliced
    const bword *validb, *candb;
    uint32_t* table;          // its box table, rebuilt every iteration
    const uint2* boxes;
    uint64_t S_pad;
    const uint4* boxes16;     // wide grids: {lo0 | lo1 << 16, lo2 | lo3 << 16, hi0 | hi1 << 16, hi2 | hi3 << 16}
    int wide;
    int32_t* pd;              // D-prefix table
    const uint8_t* valid;
    const uint8_t* cand;
    uint8_t* reach;
    uint32_t* controller;
    uint32_t* reach_step;
    FixControl* fc;
    unsigned long long* stats;   // [stats_cap][kStatsCols]
    cudaGraphConditionalHandle cond;
    int use_cond;
    // Host-loop solves: a word of page-locked host memory, mapped for the
    // device, that receives iter | stop << 32 after each iteration's stop
    // rules (write_mirror), or nullptr.
    unsigned long long* mirror;
};
// The box table of a bit-sliced set, and its sizes for the widths in use
// (copies 0 where they are too many).
cudaError_t launch_box_table(const GridInfo& g, const bword* set, uint32_t* table, const StoredBits& b,
                             const DilateArgs& d, const FixControl* fc, cudaStream_t st);
StoredBits stored_bits_of(const GridInfo& g, const DilateArgs& d, uint32_t ywidths);
inline uint64_t box_table_words(const GridInfo& g, const StoredBits& b) {
    return kBoxTableHead + static_cast<uint64_t>(b.copies) * g.slices * g.n[1] * b.hw;
}
// Kernels of one iteration, and those of them that rebuild the table.
uint32_t stored_passes(const GridInfo& g, const StoredBits& b);
inline uint32_t stored_launches(const GridInfo& g, const StoredBits& b) {
    return stored_passes(g, b) + (b.copies ? 1u : 2u);
}
cudaError_t launch_stored_init(const GridInfo& g, const StoredFixArgs& a, cudaStream_t st);
// ev (optional, kProfileEvents events): [0] before the table's rebuild, [1..n]
// after its n passes (stored_passes; events n+1 .. 4 are not recorded), [5]
// after the satisfaction kernel, [6] after the control kernel, where there is
// one.
constexpr int kProfileEvents = 8;
cudaError_t launch_stored_iteration(const GridInfo& g, const StoredFixArgs& a, cudaStream_t st, uint32_t* launches,
                                    cudaEvent_t* ev = nullptr);
// One thread that holds the stream for about `ns` nanoseconds (bounded by
// the global timer and by an iteration cap), so that what the host queues
// behind it meanwhile runs back to back: profiled phases then time the
// kernels rather than the host's enqueueing.
cudaError_t launch_hold(cudaStream_t st, uint64_t ns);

// y levels: a copy of level p ORs the 2^p rows from each row on, so that any
// y interval of 2^p .. 2^(p+1) - 1 rows is the OR of two rows of it.
constexpr int kYLevels = 6;   // fused boxes span at most 32 rows
// How one launch brings the dilated copies up to date: the y levels in use
// (bit mask; copy (level, k, l) at ((level's rank * nk + k) * nl + l) * slices * sw)
// and the rows of a slice that one block takes, plus the rows its highest
// level reads beyond them.
struct DilateTile {
    uint32_t levels, rows, tiles, smem;
};

// Set-up plan of a problem, written by k_plan and copied to the host once:
// the mask counts and axis-table flags, the largest number of representative
// accelerations in one omega column, and the theta / v box widths in use.
struct PlanRecord {
    unsigned long long counts[8];
    uint32_t flags;
    uint32_t max_reps;
    uint32_t ylevels;          // y levels in use (bit mask)
    uint32_t ywidths;          // y widths in use: bit ny - 1 (up to 32 cells)
    uint32_t width_overflow;   // more widths than kMaxDilate, or a v width above kMaxDilate
    uint32_t fused;            // 1 when the fused tables were planned
    DilateArgs dil;
    uint32_t slice_reps;            // most representatives of one slice
    unsigned long long reps;        // representatives of all slices
    unsigned long long rep_rows;    // (theta, v) cells of their windows, summed
};

// Words of the dilated copies of a set for these widths and y levels (level 0
// where there are none).
inline uint64_t dilated_words(const GridInfo& g, const DilateArgs& d, uint32_t levels) {
    return static_cast<uint64_t>(d.nk) * d.nl * __builtin_popcount(levels ? levels : 1u) * g.slices * g.sw;
}
// Whether a set may have dilated copies: offsets into them (SliceRep::off,
// ylev) are 32-bit.
inline bool dilated_offsets_fit(const GridInfo& g, const DilateArgs& d, uint32_t levels) {
    return dilated_words(g, d, levels) < 0xFFFFFFFFull;
}
// Whether the satisfaction test reads a representative's (theta, v) window
// of D' itself (nz * nv words per staged word), rather than one word of a
// dilated copy that a kernel of its own brings up to date every iteration.
// Directly where the windows' further words, over all representatives, are
// few: up to 17 MB, and up to 32 MB for windows of four cells.  Measured, us a
// solve with copies and directly (MB): 20x20x16x10 50.0 and 43.1 (0.4);
// hyperbolic 30x30x16x6 71 and 62 (1.2); 200x64x20x6 630 and 543 (6.2);
// 256x40x20x10 787 and 659 (8.3); 47x83x29x17 487 and 419 (12); hyperbolic
// 45x41x30x9 860 and 824 (14), 60x60x30x10 with obstacles 1,480 and 1,361 (16),
// 20x20x63x13 209 and 216 (17), 80x80x30x8 1,756 and 1,912 (22), 70x70x63x13
// 737 and 1,182 (177); 128x128x72x48 9,291 and 13,452 (725); of four cells
// 65x65x38x25 717 and 645 (16), 128x128x40x20 1,408 and 1,200 (18), but
// 48x48x16x8 x 192 inputs 163 and 175 (13).  With tests of few states an
// iteration direct reads stay ahead for longer (64x64x72x48 x 36: 2,179 and
// 1,839 at 71).
// batched: the instances of a batch or server keep the line at four cells: the
// dilations of all of them are one launch a step, which callers count among its
// launches (32 small instances 7.8 ms a call so, 7.4 with the wider line; a
// served burst's runs differ by more).
inline bool reads_windows_directly(const GridInfo& g, const PlanRecord& pl, bool batched) {
    if (!dilated_offsets_fit(g, pl.dil, pl.ylevels)) return true;
    const uint64_t further = (pl.rep_rows - pl.reps) * g.sw * sizeof(bword);
    return (!batched && further <= 17ull << 20) || (pl.rep_rows <= 4 * pl.reps && further <= 32ull << 20);
}

// A representative input of a (theta, v) slice: the lowest of the inputs
// whose boxes coincide for every state of the slice (all x and y rows, the
// theta box and the v box).
struct __align__(16) SliceRep {
    uint32_t j;     // the input
    uint32_t zw;    // theta window: first cell | cells << 16 (wraps)
    uint32_t vw;    // v window: first cell | cells << 16 (at most kMaxDilate) | 1 << 31 when some row is
                    // marked in needv
    uint32_t off;   // word offset of the window's copy in dzw: with kBoxY of the box's first row for row 0,
                    // in the y level in use, else of row 0 in level 0's place
    // Its plane's x and y boxes in short (launch_axis_tables), so that a plane
    // whose boxes are all alike needs no table; with kBoxY (launch_rep_offsets)
    // hy also has the words from the first to the second row of the level << 16,
    // and yr the number of rows in place of their end:
    uint32_t hx, hy, yr, xr;
};

// Launch shape of k_slice: threads a block, rows of a slice a block takes (a
// multiple of 8, or all of them), and whether it is the kernel for few slices
// (more registers a thread; the only one that splits slices).
struct SliceShape {
    uint32_t threads, part_rows, wide;
    uint32_t parts(uint32_t n1) const { return (n1 + part_rows - 1) / part_rows; }
};

struct FusedFixArgs {
    const uint32_t *xt, *yt;
    const bword* validb;
    const bword* unsafeb;
    const bword* srcb;         // valid && source-safe
    const bword* candb;
    bword* dp[2];              // D': iteration k (from 0) reads dp[k & 1] and writes the other
    bword* reach0;             // updated in place
    bword* active;
    uint32_t* controller;
    uint32_t* reach_step;
    FixControl* fc;
    unsigned long long* stats;
    const bword* xcls;         // per-plane x-box classes (launch_x_classes)
    uint32_t cls_words;        // 32-bit words per class record
    const SliceRep* reps;      // [slices][M]: each slice's representatives, in input order
    const uint32_t* nreps;     // [slices]
    uint32_t pass;             // representatives whose records and changed rows are in shared memory at a time
    SliceShape shape;          // of k_slice
    uint32_t direct;           // 1: D' windows are read from D' itself, 0: from dzw
    bword* dzw;                // (y, theta, v)-dilated copies of D' (DilateTile), brought up to date each iteration
    uint32_t ylev[kYLevels];   // word offset of each y level in dzw
    DilateTile tile;
    uint32_t* rowlost;         // [2][rl_words] bit per x-row: the row lost a D' cell in the iteration before
                               // (W1 = ceil(n1 / 32) words per (theta, v) slice, bit y % 32 of word y / 32):
                               // iteration k reads [k & 1] and writes the other
    uint32_t rl_words;         // slices * W1 + 1
    // When validity is more than safety:
    const bword* vzw;          // the dilated copies of the valid set (or null with direct: validb itself is read)
    const uint32_t* needv;     // [slices][M][W1] bit per representative and row: some state's box may hold no
                               // valid cell
    DilateArgs dil;
    // Sharded solve (one rank of several): the launch covers slices
    // [shard_begin, shard_begin + shard_slices) only, reads dp[0], and the
    // stop rules are left to the host, which applies them with the counts of
    // every rank (gsc_problem_shard_control).  shard_slices == 0: not sharded.
    uint32_t shard_begin;
    uint32_t shard_slices;
    cudaGraphConditionalHandle cond;
    int use_cond;
    unsigned long long* mirror;   // as StoredFixArgs::mirror
};

constexpr int kShiftMax = 8;   // most shifts d of a plane's shift-mask record
// Which problems the fused method takes, and which launch shapes a batch may
// use, is a rule on the shared memory that a task of max_reps representative
// accelerations once staged (fused_admission_bytes at most kFusedSmemMax).  A
// slice's task takes less (fused_smem_bytes); the rule stays because it decides
// which calls by method or launch shape are refused.
constexpr size_t kFusedSmemMax = 200 * 1024;
size_t fused_admission_bytes(const GridInfo& g, int need_valid, uint32_t max_reps);
// Representatives kept in shared memory at a time, and the shared memory of a
// slice's task (k_slice, k_batch_slice).
constexpr uint32_t kPackedRows = 8192;   // more rows a slice than this are all tested
constexpr uint32_t kHitNotes = 384;      // (row, representative) hits noted at a time
uint32_t fused_pass(const GridInfo& g, uint32_t slice_reps);
size_t fused_smem_bytes(const GridInfo& g, uint32_t pass, uint32_t rows);
DilateTile dilate_tile_of(const GridInfo& g, const DilateArgs& d, uint32_t levels);
// Most threads of a satisfaction block: at most kSliceThreadsMax at 48
// registers (40 warps an SM), or, where few slices share an SM (wide),
// kSliceThreadsWide at 64 (32 warps).
constexpr uint32_t kSliceThreadsMax = 256, kSliceThreadsWide = 512;
// For a launch over `slices` slices of at most slice_reps representatives.
inline SliceShape slice_shape(const GridInfo& g, uint32_t slices, uint32_t slice_reps) {
    SliceShape s{};
    s.part_rows = g.n[1];
    const uint64_t items = static_cast<uint64_t>(g.n[1]) * std::max(1u, slice_reps);
    // Few slices with much to test each: parts of at least 16 rows, two a slice
    // or as many as give two blocks an SM.
    // Measured, us a solve with one block a slice and so: 16x400x12x6 57.7 and
    // 53.6, 16x1000x8x4 57.6 and 47.1, 48x48x16x8 x 192 inputs 189 and 156,
    // 60x60x30x10 x 36 1,477 and 1,379, 100x100x30x10 x 36 1,590 and 1,495.  But
    // with little to test (100x100x20x12, 4 representatives) 357 and 363 in two
    // parts, and above 300 slices (47x83x29x17) 439 and 460.
    if (slices <= 300 && items * g.W > 2048) {
        const uint32_t parts = std::max(2u, 288u / slices);
        s.part_rows = std::min(g.n[1], std::max(16u, ((g.n[1] + parts - 1) / parts + 7) & ~7u));
    }
    if (s.part_rows < g.n[1]) {
        s.wide = 1;
        // Every block resident at once (1,024 threads an SM at 64 registers), up
        // to 384 threads.  Measured, us a solve with 110,000 threads in all, which
        // left a second wave of a few blocks at 149 to 184 slices, and so:
        // hyperbolic 64x64x24x7 x 36 inputs 876 and 745, 108x46x24x7 x 35 1,122 and
        // 1,030, 48x96x20x8 x 36 617 and 529, 45x41x30x9 x 36 2,077 and 2,020.
        const uint32_t per_sm = (slices * s.parts(g.n[1]) + 147) / 148;
        const uint64_t each = static_cast<uint64_t>(s.part_rows) * std::max(1u, slice_reps);
        s.threads = static_cast<uint32_t>(
            std::min<uint64_t>({384, kSliceThreadsWide * 2 / per_sm & ~31u, (each + 31) & ~uint64_t(31)}));
        return s;
    }
    // A packed row of the slice per thread, for several representatives side
    // by side.  As wide as lets every slice's block be resident at once (a
    // second wave of a few blocks doubles an iteration), and at least 128.
    const uint32_t per_sm = (slices + 147) / 148;
    uint32_t most = per_sm <= 2 ? kSliceThreadsWide / per_sm * 2 : per_sm <= 10 ? 40 / per_sm * 32 : 128;
    most = std::min(per_sm <= 2 ? kSliceThreadsWide : kSliceThreadsMax, std::max(128u, most));
    s.threads = static_cast<uint32_t>(std::min<uint64_t>(most, (items + 31) & ~31ull));
    s.wide = s.threads > kSliceThreadsMax;
    return s;
}

// Dilated copies of src into dst.  With fc and rowlost (during a fixpoint,
// after its first iteration) only tiles whose windows hold a row that lost a
// D' cell are recomputed, and src is src0 or src1 by the iteration's parity.
cudaError_t launch_dilate(const GridInfo& g, const bword* src0, const bword* src1, bword* dst, const DilateArgs& d,
                          const DilateTile& t, const FixControl* fc, const uint32_t* rowlost, uint32_t rl_words,
                          cudaStream_t st);
// Fills a PlanRecord from the counts, flags and (when xrep is set) the
// theta / v tables and plane representatives; writes kidx / lidx.
cudaError_t launch_plan(const GridInfo& g, const uint32_t* zt, const uint32_t* wt, bool fused,
                        const unsigned long long* counts, const unsigned int* flags, uint8_t* kidx, uint8_t* lidx,
                        PlanRecord* out, cudaStream_t st);
// One instance of a batched solve (or of the serving loop), resident in
// device memory and indexed by slot.
struct InstanceDesc {
    GridInfo g;
    FusedFixArgs a;
    const uint8_t* cand;
    const unsigned long long* counts;
    uint32_t max_iterations;
    uint32_t stats_cap;
    uint32_t words;       // slices * sw
};

// The instances one launch works on: slot[k] and, per task kind, the prefix
// offsets of their tasks (off[0] = 0, off[n] = total).  A satisfaction task
// is a slice; a dilate task is a tile (none for an instance that reads D'
// itself); an init task `chunk` words, states and
// stats entries.
struct WorkList {
    const uint32_t* slot;
    const uint32_t* sat_off;
    const uint32_t* dil_off;
    const uint32_t* ini_off;
    uint32_t n;
    uint32_t chunk;
    FixControl* status;   // [n]: copy of each instance's FixControl after the iteration (optional)
    uint32_t* running;    // instances still running after the iteration (optional)
};

// Consecutive instances [begin, end) of a work list whose rows have W words:
// one launch of the satisfaction kernel compiled for W.  smem: the largest
// instance's task.
struct BatchClass {
    uint32_t W, begin, end, tasks;
    size_t smem;
};

// Launch shapes of the batched kernels.
struct BatchShape {
    uint32_t sat_threads;   // threads per satisfaction block
    uint32_t sat_blocks;    // persistent satisfaction blocks (0 = one per task)
    uint32_t chunk;         // word positions per init task
    uint32_t warp;          // 1: one satisfaction task per warp (smem per task, sat_threads / 32 of them)
};

// Host-side task counts of one list (matching WorkList's offsets).
struct WorkTotals {
    uint32_t sat, dil, ini;
    uint32_t dil_smem;   // shared memory of the largest dilate task
};

// An instance of a batch that keeps the GPU busy on its own (at least
// kBigPairs state-input pairs per iteration) iterates with the one-problem
// kernels, whose row width is a compile-time constant and whose arguments
// stay in the constant bank.  Smaller instances gain more from sharing the
// batched kernels' launches than they lose to their run-time row width.
constexpr uint64_t kBigPairs = 1ull << 28;
inline bool is_big_instance(const GridInfo& g) { return g.S * g.M >= kBigPairs; }

// A big instance of a batch: its grid and its fixpoint arguments (without a
// graph condition; the batch's status kernel sets that).
struct BigInstance {
    GridInfo g;
    FusedFixArgs a;
};

cudaError_t launch_batch_init(const InstanceDesc* descs, const WorkList& wl, const WorkTotals& tot, int sms,
                              cudaStream_t st);
// One fixpoint iteration of a batch: each of the nbig big instances with the
// one-problem kernels, the instances of `small` with the batched kernels (a
// dilation where one needs it, then one satisfaction launch per row width:
// `classes`), then the status kernel over `all` (every instance, big and
// small, in the order its status records use), which also sets the graph
// condition when use_cond.
cudaError_t launch_batch_step(const InstanceDesc* descs, const WorkList& small, const WorkTotals& tot_small,
                              const BatchClass* classes, uint32_t nclasses, const WorkList& all,
                              const BigInstance* big, uint32_t nbig, const BatchShape& sh, int sms,
                              cudaGraphConditionalHandle cond, int use_cond, cudaStream_t st, uint32_t* launches);
// Shift-mask record words per plane: a 16-byte header + (kShiftMax + 1) * W
// masks, up to a multiple of 4.
__host__ __device__ inline uint32_t class_words(const GridInfo& g) { return (4 + (kShiftMax + 1) * g.W + 3) & ~3u; }
// Per (slice, input) plane, the x boxes [i0 + a, i0 + b] of its states as
// shift masks: M_d = the states whose box holds i0 + d, for the nd shifts
// d = dmin .. dmin + nd - 1 (nd <= kShiftMax), and OK = the states with a
// box.  A state is blocked by a row F exactly when bit i0 of
// OR_d ((F >> d) & M_d) is set.  Header word 0: byte 0 = nd (0xFF: the plane
// is irregular and tested state by state), byte 1 = dmin (int8), byte 2 = 1
// when every state with a box has all nd shifts (M_d = OK); then M_d
// for each d (W words each) at word 4 + (d - dmin) * W, and OK at word
// 4 + kShiftMax * W.  |a|, |b| < 32.
cudaError_t launch_x_classes(const GridInfo& g, const uint32_t* xt, const uint4* shorts, bword* xcls,
                             cudaStream_t st);
// Per plane (slice, j = ja + ma * jw): the lowest ja' of the same omega column
// whose x row, y row and v box equal those of ja, so the two inputs test every
// state alike (with one Euler substep the x and y successors do not depend on
// the acceleration at all).
// Also raises *max_reps to the most representatives of one omega column.
cudaError_t launch_plane_reps(const GridInfo& g, const uint32_t* xt, const uint32_t* yt, const uint32_t* wt,
                              const uint4* shorts, uint8_t* xrep, uint32_t* max_reps, cudaStream_t st);
// Each slice's representatives: of the accelerations that launch_plane_reps
// keeps, in input order, those whose theta box, v box and rows equal no
// earlier one's of the slice.  Raises plan->slice_reps, reps and rep_rows.
cudaError_t launch_slice_reps(const GridInfo& g, const uint32_t* xt, const uint32_t* yt, const uint32_t* zt,
                              const uint32_t* wt, const uint4* shorts, const uint8_t* xrep, SliceRep* reps,
                              uint32_t* nreps, PlanRecord* plan, cudaStream_t st);
// The offset and the level's rows of every representative (after the plan:
// kidx, lidx, nl, a.ylev).
cudaError_t launch_rep_offsets(const GridInfo& g, const uint8_t* kidx, const uint8_t* lidx, uint32_t nl,
                               const FusedFixArgs& a, SliceRep* reps, cudaStream_t st);
// When validity is more than safety: the rows (needv) with a state whose box
// under a representative holds no valid cell, marked in the representative
// when there are any; rowvoid: [slices * W1] scratch.  A box with no D' cell
// and a row without a void cell (invalid yet safe) in its y, theta and v
// ranges holds a valid one, since none of that row's cells is unsafe; only
// the others are looked at cell by cell.
cudaError_t launch_need_valid(const GridInfo& g, const FusedFixArgs& a, uint32_t* rowvoid, SliceRep* reps,
                              uint32_t* needv, cudaStream_t st);
cudaError_t launch_fused_init(const GridInfo& g, const FusedFixArgs& a, const uint8_t* cand, cudaStream_t st);
// One iteration is one launch (k_slice, whose last block applies the stop
// rules), after the dilation unless a.direct.
// ev (optional, kProfileEvents events): [0] before the dilation, [1] after
// it, [5] and [6] after the satisfaction kernel.
cudaError_t launch_fused_iteration(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st, uint32_t* launches,
                                   cudaEvent_t* ev = nullptr);

inline uint32_t fused_launches(bool direct) { return direct ? 1u : 2u; }

// Sharded solve: one iteration of the shard's slices without the stop rules;
// dp[0] then holds the shard's new D'.
cudaError_t launch_shard_iteration(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st);
// Stop rules of a sharded solve's iteration fc->iter + 1 with the counts of
// every rank; the next iteration is never incremental.
cudaError_t launch_shard_control(FixControl* fc, unsigned long long* stats, unsigned long long new_reachable,
                                 unsigned long long new_certified, cudaStream_t st);

// Resets the control block and zeroes the per-iteration counters.
cudaError_t launch_fix_init(FixControl* fc, uint32_t max_iterations, uint32_t stats_cap,
                            const unsigned long long* counts, unsigned long long* stats, cudaStream_t st);

// Sets the graph condition from the control block (first node of a graph solve).
cudaError_t launch_set_condition(const FixControl* fc, cudaGraphConditionalHandle cond, cudaStream_t st);

}  // namespace gsc_b200
