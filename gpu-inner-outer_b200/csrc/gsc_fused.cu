// gsc_fused.cu -- the FUSED fixpoint method: boxes recomputed from per-axis
// tables inside the satisfaction kernel, sets bit-sliced.
//
// Semantics are those of reachability.hpp:53-153 (Jacobi update, lowest
// satisfied input, reach_step = iteration, stop rules in the reference's
// order), as in the stored method.
//
// Data: every set is a bit slice, one 32-bit word per 32 x-cells of a
// (y, theta, v) row.  D' = (valid && !reachable) || unsafe.  A pair is
// satisfied when its box holds no D' cell (so every cell is safe, and every
// valid cell already reachable) and, when validity is more than safety, at
// least one valid cell.
//
// One iteration is one launch: k_slice, one block per (theta, v) slice (or part
// of its rows, where slices are few), tests every active state of the slice
// against the slice's representative inputs and updates the slice (slice_task);
// its last block applies the stop rules.
// Where the boxes' (theta, v) windows are wide, k_dilate first brings the
// dilated copies of D' up to date, and k_slice reads one word of those in
// place of a window of D'.
#include <algorithm>
#include <atomic>

#include "gsc_fused_body.cuh"

namespace gsc_b200 {

namespace {

inline unsigned int blocks_for(uint64_t n, int threads) {
    uint64_t b = (n + threads - 1) / threads;
    if (b == 0) b = 1;
    return static_cast<unsigned int>(b);
}

using namespace fused;

__global__ void k_fused_init(GridInfo g, FusedFixArgs a, const uint8_t* __restrict__ cand) {
    const uint64_t words = static_cast<uint64_t>(g.slices) * g.sw;
    for (uint64_t e = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; e < words;
         e += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        init_word(a, e);
    for (uint64_t s = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; s < g.S;
         s += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        init_state(a, cand, s);
}

// Dilated copies of a bit-sliced set, one block per tile (dilate_tile).
__global__ void __launch_bounds__(256) k_dilate(GridInfo g, const bword* src0, const bword* src1,
                                                bword* __restrict__ dst, DilateArgs d, DilateTile t,
                                                const FixControl* fc, const uint32_t* rowlost, uint32_t rl_words) {
    extern __shared__ __align__(16) bword smem[];
    pdl_wait();
    if (fc && fc->stop) return;
    const uint32_t c = fc ? fc->iter : 0;
    const uint32_t* lost = (rowlost && c > 0) ? rowlost + static_cast<uint64_t>(c & 1) * rl_words : nullptr;
    dilate_tile(g, (c & 1) ? src1 : src0, dst, d, t, blockIdx.x, lost, smem);
}

// The set-up plan (one block): which theta widths (wrapped lengths of the
// omega columns' theta boxes) and v widths (of the accelerations' v boxes)
// occur, numbered in increasing order.  out->max_reps (zeroed before, then
// raised by k_plane_reps) becomes at least 1.
__global__ void __launch_bounds__(256) k_plan(GridInfo g, const uint32_t* __restrict__ zt,
                                              const uint32_t* __restrict__ wt, uint32_t fused,
                                              const unsigned long long* __restrict__ counts,
                                              const unsigned int* __restrict__ flags, uint8_t* __restrict__ kidx,
                                              uint8_t* __restrict__ lidx, PlanRecord* __restrict__ out) {
    __shared__ uint32_t kbits[2048], lbits[2048];   // widths 1 .. 65535
    __shared__ DilateArgs s_dil;
    const uint32_t tid = threadIdx.x;
    if (tid < 8) out->counts[tid] = counts[tid];
    if (tid == 0) {
        out->flags = flags[0];
        out->ylevels = flags[1];
        out->ywidths = flags[2];
        out->fused = fused;
    }
    if (!kidx) {
        if (tid == 0) out->width_overflow = 1;
        return;
    }
    const uint32_t n2 = g.n[2], n3 = g.n[3];
    for (uint32_t i = tid; i < 2048; i += blockDim.x) kbits[i] = lbits[i] = 0;
    __syncthreads();
    for (uint32_t e = tid; e < n2 * g.mw; e += blockDim.x) {
        const uint32_t ze = zt[e];
        const uint32_t lz = lo16(ze), hz = hi16(ze);
        const uint32_t k = (lz <= hz) ? hz - lz + 1 : n2 - lz + hz + 1;
        atomicOr(&kbits[k >> 5], 1u << (k & 31));
    }
    for (uint32_t e = tid; e < n3 * g.ma; e += blockDim.x) {
        const uint32_t we = wt[e];
        if (we == kReject || hi16(we) < lo16(we)) continue;
        const uint32_t l = hi16(we) - lo16(we) + 1;
        atomicOr(&lbits[l >> 5], 1u << (l & 31));
    }
    __syncthreads();
    if (tid == 0) {
        DilateArgs d{};
        uint32_t over = 0;
        for (uint32_t k = 1; k <= n2; ++k) {
            if (!((kbits[k >> 5] >> (k & 31)) & 1u)) continue;
            if (d.nk == kMaxDilate) {
                over = 1;
                break;
            }
            d.kval[d.nk++] = k;
        }
        for (uint32_t l = 1; l <= n3; ++l) {
            if (!((lbits[l >> 5] >> (l & 31)) & 1u)) continue;
            if (d.nl == kMaxDilate || l > static_cast<uint32_t>(kMaxDilate)) {
                over = 1;
                break;
            }
            d.lval[d.nl++] = l;
        }
        if (d.nk == 0 || d.nl == 0) over = 1;
        s_dil = d;
        out->dil = d;
        out->width_overflow = over;
        out->max_reps = max(out->max_reps, 1u);   // raised by k_plane_reps
    }
    __syncthreads();
    for (uint32_t k = tid; k <= n2; k += blockDim.x) {
        uint32_t slot = 0xFF;
        for (uint32_t i = 0; i < s_dil.nk; ++i)
            if (s_dil.kval[i] == k) slot = i;
        kidx[k] = static_cast<uint8_t>(slot);
    }
    for (uint32_t l = tid; l <= n3; l += blockDim.x) {
        uint32_t slot = 0xFF;
        for (uint32_t i = 0; i < s_dil.nl; ++i)
            if (s_dil.lval[i] == l) slot = i;
        lidx[l] = static_cast<uint8_t>(slot);
    }
}

// SliceRep::off (kslot * nl + lslot) * slices * sw + (lz + n2 * lw) * sw and,
// where its y boxes are alike, the level's rows; one warp per slice.  Offsets
// are sums modulo 2^32 (below it with a row's when the dilated copies are used).
__global__ void __launch_bounds__(256) k_rep_offsets(const __grid_constant__ GridInfo g,
                                                     const uint8_t* __restrict__ kidx,
                                                     const uint8_t* __restrict__ lidx, uint32_t nl,
                                                     const __grid_constant__ FusedFixArgs a, SliceRep* reps) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < g.slices; s += (gridDim.x * blockDim.x) >> 5) {
        SliceRep* list = reps + static_cast<uint64_t>(s) * g.M;
        const uint32_t n = a.nreps[s];
        for (uint32_t k = lane; k < n; k += 32) {
            SliceRep rp = list[k];
            rp.off = (kidx[hi16(rp.zw)] * nl + lidx[hi16(rp.vw)]) * (g.slices * g.sw) +
                     (lo16(rp.zw) + g.n[2] * lo16(rp.vw)) * g.sw;
            if (rp.hx & kBoxY) {
                const uint32_t ny = rp.hy & 0xFFu;
                if (ny) {
                    const uint32_t p = 31 - __clz(ny);
                    const int first = static_cast<int8_t>(rp.hy >> 8);
                    rp.off += a.ylev[p] + static_cast<uint32_t>(first * static_cast<int>(g.W));
                    rp.hy |= ((ny - (1u << p)) * g.W) << 16;
                }
                rp.yr = pack16(lo16(rp.yr), hi16(rp.yr) - lo16(rp.yr));
            }
            list[k] = rp;
        }
    }
}

// Rows with a void (invalid yet safe) cell, one warp per 32 rows of a slice.
__global__ void k_row_void(GridInfo g, const bword* __restrict__ validb, const bword* __restrict__ unsafeb,
                           uint32_t* __restrict__ rowvoid) {
    const uint32_t W1 = (g.n[1] + 31) / 32, lane = threadIdx.x & 31;
    const uint64_t total = static_cast<uint64_t>(g.slices) * W1;
    for (uint64_t t = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5; t < total;
         t += (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5) {
        const uint64_t slice = t / W1;
        const uint32_t y = static_cast<uint32_t>(t - slice * W1) * 32 + lane;
        bool any = false;
        for (uint32_t w = 0; w < g.W && y < g.n[1]; ++w) {
            const uint64_t e = slice * g.sw + y * g.W + w;
            const uint32_t cells = min(32u, g.n[0] - w * kBits);
            const bword in = cells == 32 ? ~0u : (1u << cells) - 1;
            any |= (~validb[e] & ~unsafeb[e] & in) != 0;
        }
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, any);
        if (lane == 0) rowvoid[t] = m;
    }
}

// needv, one warp per (slice, representative), lanes over the rows.
template <int W>
__global__ void __launch_bounds__(256) k_need_valid(const __grid_constant__ GridInfo g,
                                                    const __grid_constant__ FusedFixArgs a,
                                                    const uint32_t* __restrict__ rowvoid, SliceRep* reps,
                                                    uint32_t* __restrict__ needv) {
    const uint32_t n1 = g.n[1], n2 = g.n[2], W1 = (n1 + 31) / 32, lane = threadIdx.x & 31;
    const uint64_t total = static_cast<uint64_t>(g.slices) * g.M;
    for (uint64_t t = (blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x) >> 5; t < total;
         t += (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5) {
        const uint32_t s = static_cast<uint32_t>(t / g.M), k = static_cast<uint32_t>(t - static_cast<uint64_t>(s) * g.M);
        if (k >= a.nreps[s]) continue;
        const SliceRep rp = reps[t];
        const uint64_t pl = xy_plane(g, s % n2, s / n2, rp.j);
        auto void_word = [&](uint32_t q) {
            uint32_t m = 0xFFFFFFFFu, z = lo16(rp.zw);
            for (uint32_t i = 0; i < hi16(rp.zw) && m; ++i) {
                for (uint32_t v = 0; v < hi16(rp.vw); ++v)
                    m &= rowvoid[static_cast<uint64_t>(z + n2 * (lo16(rp.vw) + v)) * W1 + q];
                z = (z + 1 == n2) ? 0 : z + 1;
            }
            return m;
        };
        // Void rows of the window, a word a lane; usually there are none.
        bool some = false;
        uint32_t mine = 0;
        for (uint32_t q = lane; q < W1; q += 32) {
            mine |= void_word(q);
            needv[t * W1 + q] = 0;
        }
        if (!__any_sync(0xFFFFFFFFu, mine != 0)) continue;
        __syncwarp();
        for (uint32_t q = 0; q < W1; ++q) {
            const uint32_t y = q * 32 + lane;
            const uint32_t ye = y < n1 ? a.yt[pl * g.n[1] + y] : kReject;
            bool need = false;
            if (ye != kReject) {
                const uint32_t ylo = lo16(ye), yhi = hi16(ye), wl = ylo >> 5, wh = yhi >> 5;
                const uint32_t lo = void_word(wl), hi = wh != wl ? void_word(wh) : 0u;
                if (!(~__funnelshift_r(lo, hi, ylo & 31) << (31u - (yhi - ylo)))) {
                    bword V[W], m[W];
                    valid_rows<W, 2>(g, a, make_uint4(rp.j, rp.zw, rp.vw, rp.off), rp.hx, rp.hy, y, ye, V);
                    const bword* src = a.srcb + static_cast<uint64_t>(s) * g.sw + y * W;
#pragma unroll
                    for (int w = 0; w < W; ++w) m[w] = src[w];
                    if (rp.hx & kBoxX) {
                        bword T[W];
                        or_range<W>(V, T, rp.hx & 0xFFu);
                        const int dmin = static_cast<int8_t>(rp.hx >> 8);
#pragma unroll
                        for (int w = 0; w < W; ++w)
                            m[w] &= ~moved_word<W>(T, w, dmin) & bits_from(lo16(rp.xr), w) & ~bits_from(hi16(rp.xr), w);
                    } else {
                        without_cell<W>(a.xt + pl * g.n[0], V, m);   // drops states without a box too
                    }
#pragma unroll
                    for (int w = 0; w < W; ++w) need |= m[w] != 0;
                }
            }
            const uint32_t bits = __ballot_sync(0xFFFFFFFFu, need);
            if (lane == 0 && bits) needv[t * W1 + q] = bits;
            some |= bits != 0;
        }
        if (some && lane == 0) reps[t].vw = rp.vw | 0x80000000u;
    }
}

// One block per (theta, v) slice (slice_task), or per part of its rows with WIDE
// (blockIdx.y); a sharded solve launches the shard's slices only.  The last block to finish applies the stop rules
// (reachability.hpp:133-144), except in a sharded solve.
template <int W, int SHARED, int DIRECT, bool WIDE>
__global__ void __launch_bounds__(WIDE ? kSliceThreadsWide : kSliceThreadsMax, WIDE ? 2 : 5)
    k_slice(const __grid_constant__ GridInfo g, const __grid_constant__ FusedFixArgs a) {
    extern __shared__ __align__(16) bword smem[];
    __shared__ uint32_t s_meta[3];
    FixControl* fc = a.fc;
    const int done =
        slice_task<W, SHARED, DIRECT, false, true, WIDE>(g, a, blockIdx.x + a.shard_begin, blockIdx.y, smem, s_meta);
    if (!done) {
        // Already stopped (e.g. max_iterations == 0): the graph loop must still end.
        const bool first = blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0;
        if (a.use_cond && first) cudaGraphSetConditional(a.cond, 0u);
        if (a.mirror && first) write_mirror(a.mirror, fc);
        return;
    }
    if (a.shard_slices) return;
    // The counters are device-scope atomics; the barrier orders a block's
    // atomics before its first thread's fence (cumulative) and ticket, and a
    // block without any has nothing to order.  Nothing else the last block
    // reads was written by this kernel's others.
    if (done == 2) __syncthreads();
    if (threadIdx.x != 0) return;
    if (done == 2) __threadfence();
    if (atomicAdd(&fc->ticket, 1u) != gridDim.x * gridDim.y - 1) return;
    __threadfence();
    fc->ticket = 0;
    const uint32_t it = __ldcg(&fc->iter) + 1;
    control_step(fc, a.stats + kStatsCols * it, it);
    if (a.use_cond) cudaGraphSetConditional(a.cond, fc->stop ? 0u : 1u);
    if (a.mirror) write_mirror(a.mirror, fc);
}

// Stop rules of a sharded iteration with the summed counts of every rank.
__global__ void k_shard_control(FixControl* fc, unsigned long long* stats, unsigned long long nr,
                                unsigned long long nc) {
    if (fc->stop) return;
    const uint32_t it = fc->iter + 1;
    unsigned long long* row = stats + kStatsCols * it;
    row[0] = nr;
    row[1] = nc;
    control_step(fc, row, it);
    fc->last_new = 0xFFFFFFFFu;   // every iteration of a sharded solve tests every pair
}

template <int W, int SHARED, int DIRECT, bool WIDE>
cudaError_t launch_slice_v(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st) {
    const cudaError_t e = allow_smem(k_slice<W, SHARED, DIRECT, WIDE>);
    if (e != cudaSuccess) return e;
    const uint32_t slices = a.shard_slices ? a.shard_slices : g.slices;
    return launch_pdl(k_slice<W, SHARED, DIRECT, WIDE>, dim3(slices, WIDE ? a.shape.parts(g.n[1]) : 1u),
                      dim3(a.shape.threads), fused_smem_bytes(g, a.pass, a.shape.part_rows), st, g, a);
}

template <int W, int SHARED, int DIRECT>
cudaError_t launch_slice_t(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st) {
    return a.shape.wide ? launch_slice_v<W, SHARED, DIRECT, true>(g, a, st)
                                            : launch_slice_v<W, SHARED, DIRECT, false>(g, a, st);
}

template <int W>
cudaError_t launch_slice_w(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st) {
    if (g.xy_planes == 1) return a.direct ? launch_slice_t<W, 1, 1>(g, a, st) : launch_slice_t<W, 1, 0>(g, a, st);
    return a.direct ? launch_slice_t<W, 0, 1>(g, a, st) : launch_slice_t<W, 0, 0>(g, a, st);
}

}  // namespace

size_t fused_admission_bytes(const GridInfo& g, int need_valid, uint32_t max_reps) {
    // The rows, class records and y tables of a column's representatives, in
    // slots of 16 bytes three words longer or word by word, whichever is more.
    auto r4 = [](uint64_t x) { return (x + 3) & ~uint64_t(3); };
    const uint64_t nw = static_cast<uint64_t>(g.n[1]) * g.W, nv = need_valid ? 2 : 1, mr = max_reps;
    const uint64_t cw = 4 + (kShiftMax + 1) * g.W, n1 = g.n[1], w1 = (n1 + 31) / 32, ma = g.ma;
    const uint64_t words = nw + mr * nv * nw + mr * nw + mr * cw + mr * n1 + 3 * ma + mr * w1;
    uint64_t bulk = r4(r4(nw) + mr * nv * r4(nw + 3) + mr * nw) + mr * r4(cw + 3) + mr * r4(n1 + 3) + 3 * ma + mr * w1;
    bulk = ((bulk + ma + 1) & ~uint64_t(1)) + 2;
    return static_cast<size_t>(sizeof(bword) * std::max(words, bulk));
}

size_t fused_smem_bytes(const GridInfo& g, uint32_t pass, uint32_t rows) {
    const uint64_t w1 = (g.n[1] + 31) / 32;
    const uint64_t words = 8ull * pass + static_cast<uint64_t>(rows) * g.W + (pass + 2) * w1 + kHitNotes * (g.W + 1) +
                           (rows <= kPackedRows ? (rows + 1) / 2 : 0);
    return sizeof(bword) * static_cast<size_t>((words + 3) & ~3ull);
}

uint32_t fused_pass(const GridInfo& g, uint32_t slice_reps) {
    // Up to 256 representatives, and 4 KB of changed rows.
    const uint32_t w1 = (g.n[1] + 31) / 32;
    return std::min(std::max(1u, slice_reps), std::max(1u, std::min(256u, 1024u / w1)));
}

DilateTile dilate_tile_of(const GridInfo& g, const DilateArgs& d, uint32_t levels) {
    DilateTile t{};
    t.levels = levels ? levels : 1u;
    uint32_t halo = 0;
    for (uint32_t p = 0; p < static_cast<uint32_t>(kYLevels); ++p)
        if ((t.levels >> p) & 1u) halo = (1u << p) - 1;
    // A tile's (theta, v) copies take at most 40 KB of shared memory.
    const uint32_t row = d.nk * d.nl * g.W * 4;
    const uint32_t fit = std::max<uint32_t>(1u, 40u * 1024u / row);
    t.rows = std::min(g.n[1], fit > halo ? std::max<uint32_t>(fit - halo, 1u) : 1u);
    // Few slices leave the chip idle at a block each: several tiles a slice, up
    // to four blocks an SM, of at least 128 words (their windows' rows overlap).
    // Measured, us an iteration with one tile a slice and with this rule:
    // 16x400x12x6 36.2 and 30.3, 16x1000x8x4 33.6 and 28.5, 256x40x20x10 23.8 and
    // 21.1, 100x100x30x10 34.0 and 31.9; but at 60x60x30x10 (two of 60 words) 25.2
    // and 25.5, at 128x128x72x48 (3,456 slices) 143.9 and 151.8 with two tiles.
    const uint32_t tiles = std::min(600u / g.slices, g.n[1] * g.W / 128u);
    if (tiles > 1) t.rows = std::min(t.rows, (g.n[1] + tiles - 1) / tiles);
    t.tiles = (g.n[1] + t.rows - 1) / t.rows;
    t.smem = std::min(g.n[1], t.rows + halo) * row;
    return t;
}

cudaError_t launch_plan(const GridInfo& g, const uint32_t* zt, const uint32_t* wt, bool fused,
                        const unsigned long long* counts, const unsigned int* flags, uint8_t* kidx, uint8_t* lidx,
                        PlanRecord* out, cudaStream_t st) {
    if (kidx && (g.n[2] > 65535 || g.n[3] > 65535)) return cudaErrorInvalidValue;
    k_plan<<<1, 256, 0, st>>>(g, zt, wt, fused ? 1u : 0u, counts, flags, kidx, lidx, out);
    return cudaGetLastError();
}

cudaError_t launch_dilate(const GridInfo& g, const bword* src0, const bword* src1, bword* dst, const DilateArgs& d,
                          const DilateTile& t, const FixControl* fc, const uint32_t* rowlost, uint32_t rl_words,
                          cudaStream_t st) {
    cudaError_t e = allow_smem(k_dilate);
    if (e != cudaSuccess) return e;
    return launch_pdl(k_dilate, dim3(g.slices * t.tiles), dim3(256), t.smem, st, g, src0, src1, dst, d, t, fc, rowlost,
                      rl_words);
}

template <int W>
cudaError_t launch_need_valid_t(const GridInfo& g, const FusedFixArgs& a, const uint32_t* rowvoid, SliceRep* reps,
                                uint32_t* needv, cudaStream_t st) {
    const uint64_t b = std::min<uint64_t>(148ull * 32, (static_cast<uint64_t>(g.slices) * g.M + 7) / 8);
    k_need_valid<W><<<static_cast<unsigned int>(b), 256, 0, st>>>(g, a, rowvoid, reps, needv);
    return cudaGetLastError();
}

cudaError_t launch_need_valid(const GridInfo& g, const FusedFixArgs& a, uint32_t* rowvoid, SliceRep* reps,
                              uint32_t* needv, cudaStream_t st) {
    const uint64_t words = static_cast<uint64_t>(g.slices) * ((g.n[1] + 31) / 32);
    k_row_void<<<blocks_for(words * 32, 256), 256, 0, st>>>(g, a.validb, a.unsafeb, rowvoid);
    switch (g.W) {
        case 1: return launch_need_valid_t<1>(g, a, rowvoid, reps, needv, st);
        case 2: return launch_need_valid_t<2>(g, a, rowvoid, reps, needv, st);
        case 3: return launch_need_valid_t<3>(g, a, rowvoid, reps, needv, st);
        case 4: return launch_need_valid_t<4>(g, a, rowvoid, reps, needv, st);
        case 5: return launch_need_valid_t<5>(g, a, rowvoid, reps, needv, st);
        case 6: return launch_need_valid_t<6>(g, a, rowvoid, reps, needv, st);
        case 7: return launch_need_valid_t<7>(g, a, rowvoid, reps, needv, st);
        default: return launch_need_valid_t<8>(g, a, rowvoid, reps, needv, st);
    }
}

cudaError_t launch_rep_offsets(const GridInfo& g, const uint8_t* kidx, const uint8_t* lidx, uint32_t nl,
                               const FusedFixArgs& a, SliceRep* reps, cudaStream_t st) {
    k_rep_offsets<<<blocks_for(static_cast<uint64_t>(g.slices) * 32, 256), 256, 0, st>>>(g, kidx, lidx, nl, a, reps);
    return cudaGetLastError();
}

cudaError_t launch_fused_init(const GridInfo& g, const FusedFixArgs& a, const uint8_t* cand, cudaStream_t st) {
    k_fused_init<<<blocks_for(g.S, 256), 256, 0, st>>>(g, a, cand);
    return cudaGetLastError();
}

cudaError_t launch_shard_iteration(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st) {
    cudaError_t e = launch_fused_iteration(g, a, st, nullptr, nullptr);
    if (e != cudaSuccess) return e;
    // The ranks exchange dp[0]: the shard's new D' goes there.
    const uint64_t sw = g.sw, first = a.shard_begin * sw;
    return cudaMemcpyAsync(a.dp[0] + first, a.dp[1] + first, a.shard_slices * sw * sizeof(bword),
                           cudaMemcpyDeviceToDevice, st);
}

cudaError_t launch_shard_control(FixControl* fc, unsigned long long* stats, unsigned long long new_reachable,
                                 unsigned long long new_certified, cudaStream_t st) {
    k_shard_control<<<1, 1, 0, st>>>(fc, stats, new_reachable, new_certified);
    return cudaGetLastError();
}

// Device time of an iteration, against three launches (dilation, a block per
// slice and omega column, update) before:
//   65x65x38x25 x 100     38 -> 17 us       published demo   88 -> 54 us
//   128x128x72x48 x 144  518 -> 135 us      47x83x29x17 x 63  24 -> 17 us
cudaError_t launch_fused_iteration(const GridInfo& g, const FusedFixArgs& a, cudaStream_t st, uint32_t* launches,
                                   cudaEvent_t* ev) {
    if (ev) cudaEventRecord(ev[0], st);
    cudaError_t err = cudaSuccess;
    if (!a.direct) {
        // A sharded solve reads dp[0] and dilates the whole grid every
        // iteration: the other ranks' D' slabs arrive without row-lost records.
        err = launch_dilate(g, a.dp[0], a.shard_slices ? a.dp[0] : a.dp[1], a.dzw, a.dil, a.tile, a.fc,
                            a.shard_slices ? nullptr : a.rowlost, a.rl_words, st);
        if (err != cudaSuccess) return err;
    }
    if (ev) cudaEventRecord(ev[1], st);
    switch (g.W) {
        case 1: err = launch_slice_w<1>(g, a, st); break;
        case 2: err = launch_slice_w<2>(g, a, st); break;
        case 3: err = launch_slice_w<3>(g, a, st); break;
        case 4: err = launch_slice_w<4>(g, a, st); break;
        case 5: err = launch_slice_w<5>(g, a, st); break;
        case 6: err = launch_slice_w<6>(g, a, st); break;
        case 7: err = launch_slice_w<7>(g, a, st); break;
        default: err = launch_slice_w<8>(g, a, st); break;
    }
    if (launches) *launches += fused_launches(a.direct != 0);
    if (ev) cudaEventRecord(ev[5], st);
    if (ev) cudaEventRecord(ev[6], st);
    return err;
}

}  // namespace gsc_b200
