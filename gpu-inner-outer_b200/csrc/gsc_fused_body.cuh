// gsc_fused_body.cuh -- device bodies of the fused fixpoint, shared by the
// one-problem kernels (gsc_fused.cu) and the batched kernels (gsc_batch.cu),
// so that a problem computes the same bits alone and inside a batch.
//
// Semantics are those of reachability.hpp:53-153 (Jacobi update, lowest
// satisfied input, reach_step = iteration, stop rules in the reference's
// order).
#pragma once

#include "gsc_kernels.cuh"

namespace gsc_b200 {
namespace fused {

// Bits [lx, hx] of the row F (hx - lx < 32), in the low bits.
template <int W>
__device__ __forceinline__ bword extract_bits(const bword (&F)[W], uint32_t lx, uint32_t hx) {
    const uint32_t wi = lx / kBits, sh = lx % kBits, len = hx - lx + 1;
    bword lo = 0, hi = 0;
#pragma unroll
    for (int w = 0; w < W; ++w) {
        if (static_cast<uint32_t>(w) == wi) lo = F[w];
        if (static_cast<uint32_t>(w) == wi + 1) hi = F[w];
    }
    const bword v = __funnelshift_r(lo, hi, sh);
    return len >= kBits ? v : (v & ((bword(1) << len) - 1));
}

// Word w (0 <= w <= WMAX) of the row F moved by d (|d| < 32): bit j of the
// result is bit 32 w + j + d of F, with F zero outside its WMAX words.
template <int WMAX>
__device__ __forceinline__ bword moved_word(const bword (&F)[WMAX], int w, int d) {
    const bword fm1 = (w >= 1 && w - 1 < WMAX) ? F[w - 1] : 0u;
    const bword f0 = (w < WMAX) ? F[w] : 0u;
    const bword fp1 = (w + 1 < WMAX) ? F[w + 1] : 0u;
    const bool up = d >= 0;
    return __funnelshift_r(up ? f0 : fm1, up ? fp1 : f0, static_cast<uint32_t>(d) & 31u);
}

// The bits of word w of a row at cell x and beyond (PTX shl gives 0 for a
// shift of 32 or more; C++ leaves that open).
__device__ __forceinline__ bword bits_from(uint32_t x, int w) {
    const int s = max(static_cast<int>(x) - w * kBits, 0);
#ifdef __CUDA_ARCH__
    bword m;
    asm("shl.b32 %0, %1, %2;" : "=r"(m) : "r"(0xFFFFFFFFu), "r"(s));
    return m;
#else
    return s < kBits ? 0xFFFFFFFFu << s : 0u;   // (a test on the CPU)
#endif
}

// The states m of a row (from state srow on) satisfied by input j: a state is
// satisfied in one iteration only, so its controller entry, still empty,
// takes the lowest input by atomicMin.
template <int W>
__device__ __forceinline__ void take_hits(const FusedFixArgs& a, uint64_t srow, uint32_t j, bword* hits,
                                          const bword (&m)[W]) {
#pragma unroll
    for (int w = 0; w < W; ++w) {
        if (!m[w]) continue;
        atomicOr(hits + w, m[w]);
        for (bword t = m[w]; t; t &= t - 1) atomicMin(a.controller + srow + w * kBits + __ffs(t) - 1, j);
    }
}

// Initial sets of word e: reachable = candidate, active = valid && safe
// source, D' = (valid && !candidate) || unsafe.
__device__ __forceinline__ void init_word(const FusedFixArgs& a, uint64_t e) {
    const bword c = a.candb[e];
    a.reach0[e] = c;
    a.active[e] = a.srcb[e];
    const bword d = (a.validb[e] & ~c) | a.unsafeb[e];
    a.dp[0][e] = d;
    a.dp[1][e] = d;
}

__device__ __forceinline__ void init_state(const FusedFixArgs& a, const uint8_t* cand, uint64_t s) {
    a.controller[s] = kInvalid32;
    a.reach_step[s] = cand[s] ? 0u : kInvalid32;
}

// FixControl at the start of a solve (counts: [0] valid, [1] candidates).
__device__ __forceinline__ void init_control(FixControl* fc, uint32_t max_iterations, uint32_t stats_cap,
                                             const unsigned long long* counts) {
    fc->iter = 0;
    fc->ticket = 0;
    fc->last_new = 0;
    fc->max_iterations = max_iterations;
    fc->stats_cap = stats_cap;
    fc->valid_count = counts[0];
    fc->candidate_count = counts[1];
    fc->certified = 0;
    fc->reachable = counts[1];
    fc->converged = 0;
    fc->stop = (max_iterations == 0) ? 1u : 0u;
    fc->message = (max_iterations == 0) ? 3u : 0u;
}

// Words [first, first + words) of slice (z, v) of src ORed over theta cells
// z .. z+k-1 (wrapped) and v cells v .. v+l-1 for every width k and l, into
// smem [(ki * nl + li) * words]; 0 where the v window leaves the grid (lfit: v
// cells that stay inside it).  By the whole block; the theta ORs are extended
// incrementally.
__device__ __forceinline__ void window_copies(const GridInfo& g, const bword* src, const DilateArgs& d, uint32_t z,
                                              uint32_t v, uint32_t kmax, uint32_t lfit, uint32_t first, uint32_t words,
                                              bword* smem) {
    const uint32_t n2 = g.n[2];
    for (uint32_t e = threadIdx.x; e < words; e += blockDim.x) {
        bword zor[kMaxDilate];
#pragma unroll
        for (uint32_t j = 0; j < kMaxDilate; ++j) zor[j] = 0;
        uint32_t ki = 0, zz = z;
#pragma unroll 2
        for (uint32_t i = 0; i < kmax; ++i) {
#pragma unroll
            for (uint32_t j = 0; j < kMaxDilate; ++j)
                if (j < lfit) zor[j] |= __ldg(src + static_cast<uint64_t>(zz + n2 * (v + j)) * g.sw + first + e);
            zz = (zz + 1 == n2) ? 0 : zz + 1;
            if (i + 1 == d.kval[ki]) {
                bword acc = 0;
                uint32_t li = 0;
#pragma unroll
                for (uint32_t j = 0; j < kMaxDilate; ++j) {
                    acc |= zor[j];
                    if (li < d.nl && j + 1 == d.lval[li]) {
                        smem[(ki * d.nl + li) * words + e] = (j < lfit) ? acc : 0u;
                        ++li;
                    }
                }
                ++ki;
            }
        }
    }
}

// Dilated copies of one tile (rows [y0, y0 + t.rows) of one slice), by the
// whole block: for every theta width k in d.kval and v width l in d.lval, the
// OR of src over theta cells z .. z+k-1 (wrapped) and v cells v .. v+l-1
// (copies whose v window leaves the grid are never read and are left 0), and
// of that over the 2^p rows from each row on for every y level p in use.  The
// y ORs read shared memory.
// With `lost` (the rows that lost a D' cell since the last dilation) the tile
// is left as it is when no row that it reads did.
__device__ __forceinline__ void dilate_tile(const GridInfo& g, const bword* __restrict__ src, bword* __restrict__ dst,
                                            const DilateArgs& d, const DilateTile& t, uint32_t task,
                                            const uint32_t* __restrict__ lost, bword* smem) {
    const uint32_t n1 = g.n[1], n2 = g.n[2], n3 = g.n[3], W = g.W;
    const uint32_t pos = g.slices * g.sw;
    const uint32_t kmax = d.kval[d.nk - 1], lmax = d.lval[d.nl - 1];
    const uint32_t slice = task / t.tiles, y0 = (task - slice * t.tiles) * t.rows;
    const uint32_t z = slice % n2, v = slice / n2;
    const uint32_t lfit = min(lmax, n3 - v);   // v windows that stay inside the grid
    const uint32_t halo = (1u << (31 - __clz(t.levels))) - 1;
    const uint32_t y1 = min(n1, y0 + t.rows), y2 = min(n1, y1 + halo);
    if (lost) {
        // The row-lost words hold W1 = ceil(n1 / 32) words per (theta, v)
        // slice, bit y % 32 of word y / 32 for row y.
        const uint32_t W1 = (n1 + 31) / 32, w0 = y0 >> 5, nwin = kmax * lfit, ny = ((y2 - 1) >> 5) - w0 + 1;
        uint32_t hit = 0;
        for (uint32_t e = threadIdx.x; e < nwin * ny; e += blockDim.x) {
            const uint32_t yw = w0 + e / nwin, q = e % nwin, j = q / kmax;
            uint32_t zz = z + (q - j * kmax);
            if (zz >= n2) zz -= n2;
            uint32_t m = lost[(zz + n2 * (v + j)) * W1 + yw];
            if (yw == w0) m &= 0xFFFFFFFFu << (y0 & 31);
            if (yw == (y2 - 1) >> 5) m &= 0xFFFFFFFFu >> (31 - ((y2 - 1) & 31));
            hit |= m;
        }
        if (!__syncthreads_or(hit != 0)) return;
    }
    const uint32_t words = (y2 - y0) * W, ncombo = d.nk * d.nl;
    window_copies(g, src, d, z, v, kmax, lfit, y0 * W, words, smem);
    __syncthreads();
    const uint32_t out = (y1 - y0) * W;
    bword* base = dst + static_cast<uint64_t>(slice) * g.sw + y0 * W;
    for (uint32_t p = 0, rank = 0; p < kYLevels; ++p) {
        if (!((t.levels >> p) & 1u)) continue;
        for (uint32_t c = 0; c < ncombo; ++c) {
            const bword* s = smem + c * words;
            bword* o = base + static_cast<uint64_t>(rank * ncombo + c) * pos;
            for (uint32_t e = threadIdx.x; e < out; e += blockDim.x) {
                bword acc = s[e];
                for (uint32_t i = 1, q = e + W; i < (1u << p) && q < words; ++i, q += W) acc |= s[q];
                o[e] = acc;
            }
        }
        ++rank;
    }
}

// The group that runs one slice: the whole block, or one warp
// (WARP), with its barrier and its barrier-with-OR.
template <bool WARP>
__device__ __forceinline__ void group_sync() {
    if (WARP)
        __syncwarp();
    else
        __syncthreads();
}

template <bool WARP>
__device__ __forceinline__ int group_sync_or(int p) {
    if (WARP) {
        __syncwarp();
        return __any_sync(0xFFFFFFFFu, p);
    }
    return __syncthreads_or(p);
}

// An iteration runs incrementally when the previous one added at most one
// state per kIncrementalRows x-rows.  A sharded solve sets last_new to
// 2^32 - 1, which no threshold of 1 or more admits.
constexpr unsigned long long kIncrementalRows = 4;

// The W words of a row (rows of 2 words are 8-byte and rows of 4 or 8 words
// 16-byte aligned: one or two wide loads).
template <int W>
__device__ __forceinline__ void load_row(bword (&out)[W], const bword* row) {
    if constexpr (W == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(row);
        out[0] = v.x;
        out[1] = v.y;
    } else if constexpr (W % 4 == 0) {
#pragma unroll
        for (int w = 0; w < W; w += 4) {
            const uint4 v = *reinterpret_cast<const uint4*>(row + w);
            out[w] = v.x;
            out[w + 1] = v.y;
            out[w + 2] = v.z;
            out[w + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) out[w] = row[w];
    }
}

// Y = X | X >> s over a row of W words (s < 32).
template <int W>
__device__ __forceinline__ void or_shifted(const bword (&X)[W], bword (&Y)[W], uint32_t s) {
#pragma unroll
    for (int w = 0; w < W; ++w) Y[w] = X[w] | __funnelshift_r(X[w], w + 1 < W ? X[w + 1] : 0u, s);
}

// T = the OR of X >> 0 .. nd - 1 (nd <= 32; X itself for nd = 0).
template <int W>
__device__ __forceinline__ void or_range(const bword (&X)[W], bword (&T)[W], uint32_t nd) {
    or_shifted<W>(X, T, nd > 1 ? 1u : 0u);
    if (nd <= 2) return;
    if (nd > 4) {
        // By twos up to nd - 1 or nd - 2, then the rest at once.
        for (uint32_t i = 2; i + 2 < nd; i += 2) {
            bword u[W];
            or_shifted<W>(T, u, 2u);
#pragma unroll
            for (int w = 0; w < W; ++w) T[w] = u[w];
        }
    }
    bword u[W];
    or_shifted<W>(T, u, nd <= 4 ? nd - 2 : (nd & 1u) ? 1u : 2u);
#pragma unroll
    for (int w = 0; w < W; ++w) T[w] = u[w];
}

// Any bits of X in each state's x box: U = OR_d ((X >> d) & M_d) over the
// plane's shifts (launch_x_classes; masks at rec, W words each), without the
// masks where every state with a box has all the shifts.  G is X moved by
// dmin, one word longer, so every shift is a right funnel shift by d - dmin
// in [0, kShiftMax).
template <int W>
__device__ __forceinline__ void in_x_box(const bword (&X)[W], bword (&U)[W], bword hdr, const bword* rec) {
    const int dmin = static_cast<int8_t>((hdr >> 8) & 0xFFu);
    const uint32_t nd = hdr & 0xFFu;
    bword G[W + 1];
#pragma unroll
    for (int w = 0; w <= W; ++w) G[w] = moved_word<W>(X, w, dmin);
    if (hdr & 0x10000u) {
#pragma unroll
        for (int w = 0; w < W; ++w) U[w] = nd ? G[w] : 0u;
        for (uint32_t i = 1; i < nd; ++i) {
#pragma unroll
            for (int w = 0; w < W; ++w) U[w] |= __funnelshift_r(G[w], G[w + 1], i);
        }
    } else {
#pragma unroll
        for (int w = 0; w < W; ++w) U[w] = 0;
        for (uint32_t i = 0; i < nd; ++i) {
#pragma unroll
            for (int w = 0; w < W; ++w) U[w] |= __funnelshift_r(G[w], G[w + 1], i) & __ldg(rec + i * W + w);
        }
    }
}

// Of the states m of a row, those whose x box (xrow: the row's box per cell)
// is there and holds no cell of X.
template <int W>
__device__ __noinline__ void without_cell(const uint32_t* xrow, const bword (&X)[W], bword (&m)[W]) {
    for (int w = 0; w < W; ++w) {
        for (bword t = m[w]; t; t &= t - 1) {
            const uint32_t bit = __ffs(t) - 1;
            const uint32_t xe = __ldg(xrow + w * kBits + bit);
            if (xe == kReject || extract_bits<W>(X, lo16(xe), hi16(xe)) != 0) m[w] &= ~(bword(1) << bit);
        }
    }
}

// The OR of two rows `d` words apart.
template <int W>
__device__ __forceinline__ void two_rows(const bword* row, uint32_t d, bword (&F)[W]) {
    bword t[W];
    load_row<W>(F, row);
    load_row<W>(t, row + d);
#pragma unroll
    for (int w = 0; w < W; ++w) F[w] |= t[w];
}

// Row i1's box rows of the dilated copies Z under a representative (offset
// off, boxes in short hx, hy; ye: its y box where those are not alike).
template <int W>
__device__ __forceinline__ void box_rows(const FusedFixArgs& a, const bword* Z, uint32_t off, uint32_t hx, uint32_t hy,
                                         uint32_t i1, uint32_t ye, bword (&F)[W]) {
    if (hx & kBoxY) {
        two_rows<W>(Z + (off + i1 * W), hy >> 16, F);
    } else {
        const uint32_t ylo = lo16(ye), ny = hi16(ye) - ylo + 1, p = 31 - __clz(ny);
        two_rows<W>(Z + (a.ylev[p] + off + ylo * W), (ny - (1u << p)) * W, F);
    }
}

// Rows of the valid set in a representative's (theta, v) window, ORed: row by
// row, out of line and in few registers, since only grids without dilated
// copies of the valid set come here.
template <int W>
__device__ __noinline__ void valid_window(const GridInfo& g, const bword* validb, uint4 rp, uint32_t ylo, uint32_t ny,
                                          bword (&V)[W]) {
#pragma unroll
    for (int w = 0; w < W; ++w) V[w] = 0;
    uint32_t z = lo16(rp.y);
#pragma unroll 1
    for (uint32_t i = 0; i < hi16(rp.y); ++i) {
#pragma unroll 1
        for (uint32_t v = 0; v < (hi16(rp.z) & 0x7FFFu); ++v) {
            const bword* row = validb + static_cast<uint64_t>(z + g.n[2] * (lo16(rp.z) + v)) * g.sw + ylo * W;
#pragma unroll 1
            for (uint32_t e = 0; e < ny * W; e += W) {
#pragma unroll
                for (int w = 0; w < W; ++w) V[w] |= row[e + w];
            }
        }
        z = (z + 1 == g.n[2]) ? 0 : z + 1;
    }
}

// Row i1's box rows of the valid set under a representative (as box_rows): from
// its dilated copies, or from the set itself where it has none, which is only
// where D' is read directly (DIRECT: as a.direct; 2 = decided at run time).
// Copies beside direct reads: 65x65x38x25 x 36 inputs with obstacles takes 629
// us with them and 679 without.
template <int W, int DIRECT>
__device__ __forceinline__ void valid_rows(const GridInfo& g, const FusedFixArgs& a, uint4 rp, uint32_t hx, uint32_t hy,
                                           uint32_t i1, uint32_t ye, bword (&V)[W]) {
    if (DIRECT == 0 || a.vzw) {
        box_rows<W>(a, a.vzw, rp.w, hx, hy, i1, ye, V);
        return;
    }
    const uint32_t ylo = hx & kBoxY ? i1 + static_cast<int8_t>(hy >> 8) : lo16(ye);
    valid_window<W>(g, a.validb, rp, ylo, hx & kBoxY ? hy & 0xFFu : hi16(ye) - ylo + 1, V);
}

// Of the states m of row i1 of a slice, those whose box under the slice's
// representative number `index` holds a valid cell: the x test on the valid
// set (valid_rows).  Only rows marked in needv (launch_need_valid) have a state
// whose box does not.
template <int W, int DIRECT>
__device__ __noinline__ void keep_valid(const GridInfo& g, const FusedFixArgs& a, uint4 rp, uint4 bx, uint32_t slice,
                                        uint32_t index, uint32_t i1, bword (&m)[W]) {
    const uint32_t W1 = (g.n[1] + 31) / 32;
    if (!((__ldg(a.needv + (static_cast<uint64_t>(slice) * g.M + index) * W1 + (i1 >> 5)) >> (i1 & 31)) & 1u)) return;
    const uint64_t pl = xy_plane(g, slice % g.n[2], slice / g.n[2], rp.x);
    bword V[W], none[W];
    valid_rows<W, DIRECT>(g, a, rp, bx.x, bx.y, i1, bx.x & kBoxY ? 0u : __ldg(a.yt + pl * g.n[1] + i1), V);
    if (bx.x & kBoxX) {
        bword T[W];
        or_range<W>(V, T, bx.x & 0xFFu);
        const int dmin = static_cast<int8_t>(bx.x >> 8);
#pragma unroll
        for (int w = 0; w < W; ++w) m[w] &= moved_word<W>(T, w, dmin);
        return;
    }
#pragma unroll
    for (int w = 0; w < W; ++w) none[w] = m[w];
    without_cell<W>(a.xt + pl * g.n[0], V, none);
#pragma unroll
    for (int w = 0; w < W; ++w) m[w] &= ~none[w];
}

// D' cells of rows [ylo, ylo + ny) in a representative's (theta, v) window,
// ORed, from D' itself.
template <int W>
__device__ __forceinline__ void window_rows(const GridInfo& g, const bword* cur, uint4 rp, uint32_t ylo, uint32_t ny,
                                            bword (&F)[W]) {
    const uint32_t n2 = g.n[2], z0 = lo16(rp.y), nz = hi16(rp.y), v0 = lo16(rp.z), nv = hi16(rp.z) & 0x7FFFu;
#pragma unroll
    for (int w = 0; w < W; ++w) F[w] = 0;
    for (uint32_t v = v0; v < v0 + nv; ++v) {
        for (uint32_t i = 0; i < nz; i += 2) {
            // Two theta cells at a time (the last one twice when there is no second).
            uint32_t za = z0 + i, zb = za + (i + 1 < nz ? 1u : 0u);
            if (za >= n2) za -= n2;
            if (zb >= n2) zb -= n2;
            const bword* A = cur + static_cast<uint64_t>(za + n2 * v) * g.sw + ylo * W;
            const bword* B = cur + static_cast<uint64_t>(zb + n2 * v) * g.sw + ylo * W;
#pragma unroll 2
            for (uint32_t y = 0; y < ny; ++y) {
                bword s[W], t[W];
                load_row<W>(s, A + y * W);
                load_row<W>(t, B + y * W);
#pragma unroll
                for (int w = 0; w < W; ++w) F[w] |= s[w] | t[w];
            }
        }
    }
}

// One (theta, v) slice of one iteration, or with PARTS one part of its rows
// (SliceShape::part_rows), by one group: the satisfaction test of every active
// state against every representative input, the lowest satisfied input, and
// the state update.  A row's states are updated by its own group alone and D'
// is double-buffered (this iteration reads dp[iter & 1] and writes its rows of
// the other), so the update needs no further kernel, and an iteration is one
// launch (two with the dilation).
//
// A thread takes a row of the slice and every kpar-th of its representatives
// (launch_slice_reps).  For each, F = D' ORed over the box's y, theta and v
// ranges (from a y level of the dilated copies two rows, which cover the y
// range; from D' itself, direct, every row of the window), then the x test, 32 states per word: a state whose x box
// is [i0 + a, i0 + b] is blocked when F has a bit in it, i.e. bit i0 of
// OR_{d=a..b} (F >> d); with the plane's shift masks M_d (launch_x_classes)
// that is bit i0 of OR_d ((F >> d) & M_d); a plane whose boxes are alike needs
// no masks (SliceRep::hx), one with boxes of more than kShiftMax shifts is
// tested state by state.  When validity is more than safety, the box must also
// hold a valid cell (keep_valid; few rows have a box that may not).
// In incremental iterations a representative's rows that lost a D' cell in
// the last iteration are gathered first, and a (representative, row) item
// with none in its y range is left out: its states failed, and nothing they
// wait for changed.
// Then the words with a hit: D' loses the hit bits (a hit state is valid and
// safe, so its bit is 1 exactly while it is not reachable: the newly reachable
// are hit & D', the newly certified candidates hit & ~D'), and the rows that
// lost one are recorded for the next iteration.
//
// Bound: latency and issue, with every slice's block resident at once
// (slice_shape).  Rows are read from L2 straight into registers: staged
// in shared memory in chunks of representatives, three block barriers a chunk
// and 45 M warp instructions took 85 us an iteration on the published demo; so,
// 16 M take 51 us, where one block per (slice, omega column) with a kernel of
// its own for the update took 88.  Hits are noted and taken after the loop: taken in it, by
// one lane while its warp waits, the same iteration took 76 us.  Loading two
// or four representatives ahead costs registers (resident warps) and was no
// faster (55 to 58 us).
//
// Returns 0 once the solve has stopped, 2 when the group counted a hit, else 1.
// Every early return is taken by the whole group.  s_meta: [0] iteration |
// incremental << 31, or all ones once stopped, [1] rows packed, [2] hits noted.
// SHARED: the slice has one x / y plane (xy_plane); DIRECT: as a.direct; 2 =
// decided at run time.
template <int W, int SHARED, int DIRECT, bool WARP, bool PDL, bool PARTS>
__device__ __forceinline__ int slice_task(const GridInfo& g, const FusedFixArgs& a, uint32_t slice, uint32_t part,
                                           bword* smem, uint32_t* s_meta) {
    const uint32_t n0 = g.n[0], n1 = g.n[1], n2 = g.n[2];
    const uint32_t sw = g.sw, W1 = (n1 + 31) / 32;
    // Rows [y0, y0 + np1), whose row-lost bits are in the words from yw0 on.
    const uint32_t y0 = PARTS ? part * a.shape.part_rows : 0u, np1 = PARTS ? min(a.shape.part_rows, n1 - y0) : n1;
    const uint32_t yw0 = PARTS ? y0 >> 5 : 0u, W1p = PARTS ? ((y0 + np1 + 31) >> 5) - yw0 : W1;
    const uint32_t i2 = slice % n2, i3 = slice / n2;
    const uint64_t wbase = static_cast<uint64_t>(slice) * sw + y0 * W;   // of row y0
    const uint32_t tid = WARP ? (threadIdx.x & 31u) : threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t bd = WARP ? 32u : blockDim.x;
    const bool shared_xy = SHARED == 2 ? g.xy_planes == 1 : SHARED == 1;
    const bool direct = DIRECT == 2 ? a.direct != 0 : DIRECT == 1;
    const uint32_t pass = a.pass;
    uint4* reps = reinterpret_cast<uint4*>(smem);            // [pass][2] SliceRep
    bword* hits = smem + 8 * pass;                           // [np1 * W] states satisfied now
    uint32_t* rowchg = hits + np1 * W;                        // [pass][W1]
    uint32_t* lostown = rowchg + pass * W1;                  // [W1p] rows of this slice that lost a cell
    uint32_t* lostnew = lostown + W1p;                       // [W1p] that lose one now
    uint32_t* notes = lostnew + W1p;                         // [kHitNotes][W + 1] hits: row | representative << 16, states
    uint16_t* rows = reinterpret_cast<uint16_t*>(notes + kHitNotes * (W + 1));   // [np1] rows with an active state, up to kPackedRows

    // Tables that no iteration changes, before waiting for the last one.
    const uint32_t nrep = a.nreps[slice];
    const uint4* list = reinterpret_cast<const uint4*>(a.reps) + static_cast<uint64_t>(slice) * g.M * 2;
    for (uint32_t r = tid; r < 2 * min(pass, nrep); r += bd) reps[r] = list[r];
    for (uint32_t e = tid; e < np1 * W; e += bd) hits[e] = 0;
    if (tid == 0) s_meta[1] = s_meta[2] = 0;
    group_sync<WARP>();
    if (PDL) pdl_wait();

    const FixControl* fc = a.fc;
    const uint32_t it = fc->iter;
    if (tid == 0) {
        const bool inc = it > 0 && static_cast<unsigned long long>(fc->last_new) * kIncrementalRows <= g.rows;
        s_meta[0] = fc->stop ? 0xFFFFFFFFu : (it | (inc ? 0x80000000u : 0u));
    }
    // The rows with an active state, packed (in no particular order), so that
    // every thread of the group has as many items.
    const bool packed = np1 <= kPackedRows;
    int any = 0;
    for (uint32_t yb = tid & ~31u; yb < np1; yb += bd) {
        const uint32_t y = yb + lane;   // (from y0)
        bword v[W], o = 0;
        if (y < np1) {
            load_row<W>(v, a.active + wbase + y * W);
#pragma unroll
            for (int w = 0; w < W; ++w) o |= v[w];
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, o != 0);
        any |= m != 0;
        if (packed && m) {
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(s_meta + 1, __popc(m));
            at = __shfl_sync(0xFFFFFFFFu, at, 0);
            if (o) rows[at + __popc(m & ((1u << lane) - 1))] = static_cast<uint16_t>(y);
        }
    }
    const uint32_t* rl = a.rowlost + static_cast<uint64_t>(it & 1u) * a.rl_words;
    uint32_t* rlnext = a.rowlost + static_cast<uint64_t>((it + 1) & 1u) * a.rl_words;
    const bool odd = !a.shard_slices && (it & 1u);
    const bword* cur = odd ? a.dp[1] : a.dp[0];
    // Changed rows of `n` staged representatives' windows (unless this is the
    // first iteration, which has no record of any).
    auto changed_rows = [&](uint32_t n) {
        for (uint32_t e = tid; e < n * W1; e += bd) {
            const uint32_t r = e / W1, yw = e - r * W1;
            const uint4 rp = reps[2 * r];
            const uint32_t z0 = lo16(rp.y), nz = hi16(rp.y), v0 = lo16(rp.z), nv = hi16(rp.z) & 0x7FFFu;
            const auto at = [&](uint32_t z, uint32_t v) { return rl[static_cast<uint64_t>(z + n2 * v) * W1 + yw]; };
            uint32_t m = 0;
            if (nz <= 2 && nv <= 2) {
                const uint32_t z1 = nz < 2 ? z0 : (z0 + 1 == n2 ? 0 : z0 + 1), v1 = v0 + nv - 1;
                m = at(z0, v0) | at(z0, v1) | at(z1, v0) | at(z1, v1);
            } else {
                uint32_t z = z0;
                for (uint32_t i = 0; i < nz; ++i) {
#pragma unroll 4
                    for (uint32_t v = v0; v < v0 + nv; ++v) m |= at(z, v);
                    z = (z + 1 == n2) ? 0 : z + 1;
                }
            }
            rowchg[e] = m;
        }
    };
    if (it) changed_rows(min(pass, nrep));
    for (uint32_t e = tid; e < W1p; e += bd) {
        lostown[e] = it ? rl[static_cast<uint64_t>(slice) * W1 + yw0 + e] : 0u;
        lostnew[e] = 0;
    }
    any = group_sync_or<WARP>(any);
    const uint32_t ctl = s_meta[0];
    if (ctl == 0xFFFFFFFFu) return 0;
    const bool incremental = (ctl >> 31) != 0;
    // Threads = rows x kpar; a group smaller than the rows strides over them.
    const uint32_t nrows = packed ? s_meta[1] : np1;
    const uint32_t kpar = any && nrows < bd ? bd / nrows : 1u;
    const uint32_t kk = any && nrows < bd ? tid / nrows : 0u;
    unsigned long long ntest = 0;
    int hit_any = 0;   // of the group, once a pass is through
    for (uint32_t p0 = 0; any && p0 < nrep; p0 += pass) {
        const uint32_t np = min(pass, nrep - p0);
        if (p0) {
            group_sync<WARP>();
            for (uint32_t r = tid; r < 2 * np; r += bd) reps[r] = list[2 * p0 + r];
            group_sync<WARP>();
            if (incremental) {
                changed_rows(np);
                group_sync<WARP>();
            }
        }
        for (uint32_t row = tid - kk * nrows; row < nrows && kk < kpar; row += bd) {
            const uint32_t ir = packed ? rows[row] : row, i1 = y0 + ir;
            bword open[W], anyo = 0;
            load_row<W>(open, a.active + wbase + ir * W);
            uint32_t states = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                anyo |= open[w];
                states += __popc(open[w]);
            }
            if (!anyo) continue;
            const uint64_t base_pl = xy_plane(g, i2, i3, 0);
            uint32_t tested = 0;
            for (uint32_t k = kk; k < np; k += kpar) {
                const uint4 rp = reps[2 * k], bx = reps[2 * k + 1];
                uint32_t ye = 0;
                if (bx.x & kBoxY) {
                    if (i1 - lo16(bx.z) >= hi16(bx.z)) continue;
                } else {
                    ye = __ldg(a.yt + (shared_xy ? base_pl : base_pl + rp.x) * g.n[1] + i1);
                    if (ye == kReject) continue;
                }
                bword F[W];
                if (incremental || direct || !(bx.x & kBoxY)) {
                    const uint32_t ylo = bx.x & kBoxY ? i1 + static_cast<int8_t>(bx.y >> 8) : lo16(ye);
                    const uint32_t ny = bx.x & kBoxY ? bx.y & 0xFFu : hi16(ye) - lo16(ye) + 1;
                    if (incremental) {
                        // Bits [ylo, ylo + ny) of the representative's changed-row
                        // mask (fused boxes span at most 32 rows): one funnel shift.
                        const uint32_t* rc = rowchg + k * W1;
                        const uint32_t wl = ylo >> 5, wh = (ylo + ny - 1) >> 5;
                        const uint32_t bits = __funnelshift_r(rc[wl], wh != wl ? rc[wh] : 0u, ylo & 31);
                        if (!(bits << (32u - ny))) continue;
                    }
                    if (direct) window_rows<W>(g, cur, rp, ylo, ny, F);
                }
                if (!direct) box_rows<W>(a, a.dzw, rp.w, bx.x, bx.y, i1, ye, F);
                tested += states;
                bword sm[W], anys = 0;
                if (bx.x & kBoxX) {
                    // T = the OR of F >> 0 .. b - a (bits that come in from
                    // beyond the row belong to no state with a box), moved by a.
                    bword T[W];
                    or_range<W>(F, T, bx.x & 0xFFu);
                    const int dmin = static_cast<int8_t>(bx.x >> 8);
                    const uint32_t x0 = lo16(bx.w), x1 = hi16(bx.w);
#pragma unroll
                    for (int w = 0; w < W; ++w) {
                        sm[w] = open[w] & ~moved_word<W>(T, w, dmin) & bits_from(x0, w) & ~bits_from(x1, w);
                        anys |= sm[w];
                    }
                } else {
                    const uint64_t pl = shared_xy ? base_pl : base_pl + rp.x;
                    const bword* rec = a.xcls + pl * a.cls_words;
                    const bword hdr = __ldg(rec);
                    if ((hdr & 0xFFu) != 0xFFu) {
                        bword U[W];
                        in_x_box<W>(F, U, hdr, rec + 4);
#pragma unroll
                        for (int w = 0; w < W; ++w) sm[w] = open[w] & __ldg(rec + 4 + kShiftMax * W + w) & ~U[w];
                    } else {
                        bword x[W], y[W];
#pragma unroll
                        for (int w = 0; w < W; ++w) {
                            x[w] = F[w];
                            y[w] = open[w];
                        }
                        without_cell<W>(a.xt + pl * n0, x, y);
#pragma unroll
                        for (int w = 0; w < W; ++w) sm[w] = y[w];
                    }
#pragma unroll
                    for (int w = 0; w < W; ++w) anys |= sm[w];
                }
                if (!anys) continue;
                if (rp.z >> 31) {
                    bword x[W];
#pragma unroll
                    for (int w = 0; w < W; ++w) x[w] = sm[w];
                    keep_valid<W, DIRECT>(g, a, rp, bx, slice, p0 + k, i1, x);
#pragma unroll
                    for (int w = 0; w < W; ++w) sm[w] = x[w];
                }
                // Noted for later, so that a warp does not stop for each of its
                // lanes' hits (at once when the list is full).
                hit_any = 1;
                const uint32_t at = atomicAdd(s_meta + 2, 1u);
                if (at < kHitNotes) {
                    uint32_t* note = notes + at * (W + 1);
                    note[0] = ir | (k << 16);
#pragma unroll
                    for (int w = 0; w < W; ++w) note[1 + w] = sm[w];
                } else {
                    take_hits<W>(a, (static_cast<uint64_t>(slice) * n1 + i1) * n0, rp.x, hits + ir * W, sm);
                }
                anyo = 0;
                states = 0;
#pragma unroll
                for (int w = 0; w < W; ++w) {
                    open[w] &= ~sm[w];
                    anyo |= open[w];
                    states += __popc(open[w]);
                }
                if (!anyo) break;
            }
            ntest += tested;
        }
        // The noted hits (of this pass: its representatives are still staged).
        hit_any = group_sync_or<WARP>(hit_any);
        if (hit_any) {
            const uint32_t n = min(s_meta[2], kHitNotes);
            for (uint32_t e = tid; e < n; e += bd) {
                const uint32_t* note = notes + e * (W + 1);
                const uint32_t ir = note[0] & 0xFFFFu;
                bword sm[W];
#pragma unroll
                for (int w = 0; w < W; ++w) sm[w] = note[1 + w];
                take_hits<W>(a, (static_cast<uint64_t>(slice) * n1 + y0 + ir) * n0, reps[2 * (note[0] >> 16)].x,
                             hits + ir * W, sm);
            }
            group_sync<WARP>();
            if (tid == 0) s_meta[2] = 0;
            // The next pass tests the states that this one left, which it reads
            // from the active set: `hits` may be written at once by a thread of
            // a pass while another, with a lower input, begins the same row.
            if (p0 + pass < nrep) {
                for (uint32_t e = tid; e < np1 * W; e += bd)
                    if (hits[e]) a.active[wbase + e] &= ~hits[e];
            }
        }
    }
    // The update: words with a hit, and D' rows whose other buffer is behind.
    bword* next = odd ? a.dp[0] : a.dp[1];
    unsigned long long nr = 0, nc = 0;
    const uint32_t step = it + 1;
    for (uint32_t e = tid; e < np1 * W; e += bd) {
        const uint32_t y = y0 + e / W, yw = (y >> 5) - yw0, yb = 1u << (y & 31);
        const bword h = hit_any ? hits[e] : 0u;
        if (!h && !(lostown[yw] & yb)) continue;
        const bword d = cur[wbase + e];
        next[wbase + e] = d & ~h;
        if (!h) continue;
        a.active[wbase + e] &= ~h;
        a.reach0[wbase + e] |= h;
        const bword fresh = h & d;
        nr += __popc(fresh);
        nc += __popc(h & ~d);
        if (fresh) {
            atomicOr(lostnew + yw, yb);
            const uint64_t srow = (static_cast<uint64_t>(slice) * n1 + y) * n0 + (e % W) * kBits;
            for (bword m = fresh; m; m &= m - 1) a.reach_step[srow + __ffs(m) - 1] = step;
        }
    }
    if (hit_any) group_sync<WARP>();
    if (PARTS) {
        // A part's rows are whole bytes of the row-lost words, the last part's to the end.
        uint8_t* bytes = reinterpret_cast<uint8_t*>(rlnext + static_cast<uint64_t>(slice) * W1);
        const uint32_t end = y0 + np1 == n1 ? 4 * W1 : (y0 + np1) >> 3;
        for (uint32_t e = (y0 >> 3) + tid; e < end; e += bd)
            bytes[e] = static_cast<uint8_t>(lostnew[(e >> 2) - yw0] >> (8 * (e & 3u)));
    } else {
        for (uint32_t e = tid; e < W1; e += bd) rlnext[static_cast<uint64_t>(slice) * W1 + e] = lostnew[e];
    }
    if (any) {   // else nothing was tested
        unsigned long long* row = a.stats + kStatsCols * step;
        for (int off = 16; off > 0; off >>= 1) ntest += __shfl_down_sync(0xFFFFFFFFu, ntest, off);
        if (lane == 0 && ntest) atomicAdd(row + 2, ntest);
        if (tid == 0) atomicAdd(row + 3, static_cast<unsigned long long>(nrep));
        if (hit_any) {
            for (int off = 16; off > 0; off >>= 1) {
                nr += __shfl_down_sync(0xFFFFFFFFu, nr, off);
                nc += __shfl_down_sync(0xFFFFFFFFu, nc, off);
            }
            if (lane == 0) {
                if (nr) atomicAdd(row, nr);
                if (nc) atomicAdd(row + 1, nc);
            }
        }
    }
    return hit_any ? 2 : 1;
}

// iter | stop << 32 of the control record into the host's mirror word, for
// a host loop that polls it instead of copying the record back.  One 8-byte
// store, with no fence after it: the host needs nothing else from the word's
// iteration, and a system fence held the iteration's end for 2 us.
__device__ __forceinline__ void write_mirror(unsigned long long* mirror, const FixControl* fc) {
    *reinterpret_cast<volatile unsigned long long*>(mirror) =
        fc->iter | (static_cast<unsigned long long>(fc->stop ? 1u : 0u) << 32);
}

// The stop rules after iteration `it` (reachability.hpp:133-144), by one
// thread once every counter of the iteration is in.
// Its loads are one round, from L2 (where the other blocks' counter atomics
// were performed).
__device__ __forceinline__ void control_step(FixControl* fc, unsigned long long* row, uint32_t it) {
    const unsigned long long tnr = __ldcg(row);
    const unsigned long long tnc = __ldcg(row + 1);
    const unsigned long long certified = __ldcg(&fc->certified) + tnc;
    const unsigned long long reachable = __ldcg(&fc->reachable) + tnr;
    const unsigned long long candidates = __ldcg(&fc->candidate_count);
    const uint32_t max_iterations = __ldcg(&fc->max_iterations);
    const uint32_t stats_cap = __ldcg(&fc->stats_cap);
    fc->certified = certified;
    fc->reachable = reachable;
    fc->iter = it;
    fc->last_new = tnr > 0xFFFFFFFFull ? 0xFFFFFFFFu : static_cast<uint32_t>(tnr);
    if (certified == candidates) {
        fc->converged = 1;
        fc->message = 1;
        fc->stop = 1;
    } else if (tnr == 0 && tnc == 0) {
        fc->message = 2;
        fc->stop = 1;
    } else if (it >= max_iterations || it + 1 >= stats_cap) {
        fc->message = 3;
        fc->stop = 1;
    }
}

// Largest k in [0, n) with off[k] <= t, given off[0] <= t < off[n].
__device__ __forceinline__ uint32_t find_task(const uint32_t* __restrict__ off, uint32_t n, uint32_t t) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (off[mid] <= t)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// Every task t = first, first + step, ... of the slices of the instances
// [kb, ke) of a list, by one group.  The instance of the current task is
// copied to shared memory (sd) when it changes.
template <int W, bool WARP>
__device__ __forceinline__ void batch_slices(const InstanceDesc* __restrict__ descs, const WorkList& wl, uint32_t kb,
                                             uint32_t ke, uint32_t first, uint32_t step, bword* smem, InstanceDesc& sd,
                                             uint32_t* s_meta) {
    const uint32_t total = wl.sat_off[ke];
    const uint32_t rank = WARP ? (threadIdx.x & 31u) : threadIdx.x;
    const uint32_t gsize = WARP ? 32u : blockDim.x;
    uint32_t cur = 0xFFFFFFFFu;
    bool stopped = false;
    for (uint32_t t = wl.sat_off[kb] + first; t < total; t += step) {
        const uint32_t k = kb + find_task(wl.sat_off + kb, ke - kb, t);
        const uint32_t slot = wl.slot[k];
        if (slot != cur) {
            // (A thread may still read the last record's stop flag.)
            group_sync<WARP>();
            const uint32_t* src = reinterpret_cast<const uint32_t*>(descs + slot);
            uint32_t* dst = reinterpret_cast<uint32_t*>(&sd);
            for (uint32_t i = rank; i < sizeof(InstanceDesc) / 4; i += gsize) dst[i] = src[i];
            group_sync<WARP>();
            cur = slot;
            // An instance's stop flag changes only after its last task, so the
            // tasks of a stopped instance are skipped without a look.
            stopped = __ldcg(&sd.a.fc->stop) != 0;
        }
        if (stopped) continue;
        const int done = slice_task<W, 2, 2, WARP, false, false>(sd.g, sd.a, t - wl.sat_off[k], 0, smem, s_meta);
        // The counters are atomics; the barrier orders the group's before its
        // first thread's fence (cumulative) and ticket.
        group_sync<WARP>();
        if (rank == 0 && done) {
            FixControl* fc = sd.a.fc;
            if (done == 2) __threadfence();
            if (atomicAdd(&fc->ticket, 1u) == wl.sat_off[k + 1] - wl.sat_off[k] - 1) {
                __threadfence();
                fc->ticket = 0;
                const uint32_t it = __ldcg(&fc->iter) + 1;
                control_step(fc, sd.a.stats + kStatsCols * it, it);
            }
        }
        group_sync<WARP>();
    }
}

}  // namespace fused
}  // namespace gsc_b200
